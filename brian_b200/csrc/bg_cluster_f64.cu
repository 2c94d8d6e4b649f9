// bg_cluster_f64.cu -- the cluster kernel's instances for double state.
#include "bg_cluster_inst.cuh"

const void *bg_cluster_kernel_f64(int nvar, int npt, bool diag, bool multi, int pat) {
    return cluster_instance<double>(nvar, npt, diag, multi, pat);
}
