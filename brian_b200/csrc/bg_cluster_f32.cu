// bg_cluster_f32.cu -- the cluster kernel's instances for float state.
#include "bg_cluster_inst.cuh"

const void *bg_cluster_kernel_f32(int nvar, int npt, bool diag, bool multi, int pat) {
    return cluster_instance<float>(nvar, npt, diag, multi, pat);
}
