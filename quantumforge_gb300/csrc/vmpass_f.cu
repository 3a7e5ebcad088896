// vmpass_f.cu — register-tile passes, instantiations for float2.
#include "vmpass.cuh"

namespace qf {
int vm_run_f(qf_sv *psi, const Plan &plan) { return vm::run<float2, false>(psi, nullptr, plan, nullptr); }
}  // namespace qf
