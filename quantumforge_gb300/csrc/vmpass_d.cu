// vmpass_d.cu — register-tile passes, instantiations for double2.
#include "vmpass.cuh"

namespace qf {
int vm_run_d(qf_sv *psi, const Plan &plan) { return vm::run<double2, false>(psi, nullptr, plan, nullptr); }
}  // namespace qf
