// vmpass_d2.cu — register-tile passes, instantiations for double2 with psi and lambda.
#include "vmpass.cuh"

namespace qf {
int vm_run_d2(qf_sv *psi, qf_sv *lam, const Plan &plan, double *d_slot_sums) {
    return vm::run<double2, true>(psi, lam, plan, d_slot_sums);
}
}  // namespace qf
