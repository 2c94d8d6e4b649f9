// bg_cluster_inst.cuh -- selection among the cluster kernel's instances: any
// variables and update with PAT 0 (1-4 variables), the constant forms for two
// and three variables with the DIAG update.
#pragma once
#include "bg_cluster_host.h"

namespace {

template <typename T, int NV, bool DIAG, int PAT>
const void *cluster_of(int npt, bool multi) {
    if (multi)
        return npt == 1 ? (const void *)bg::k_cluster<T, NV, 1, DIAG, true, PAT>
             : npt == 2 ? (const void *)bg::k_cluster<T, NV, 2, DIAG, true, PAT>
                        : (const void *)bg::k_cluster<T, NV, 4, DIAG, true, PAT>;
    return npt == 1 ? (const void *)bg::k_cluster<T, NV, 1, DIAG, false, PAT>
         : npt == 2 ? (const void *)bg::k_cluster<T, NV, 2, DIAG, false, PAT>
                    : (const void *)bg::k_cluster<T, NV, 4, DIAG, false, PAT>;
}

template <typename T>
const void *cluster_instance(int nvar, int npt, bool diag, bool multi, int pat) {
    if (diag && nvar == 3 && pat == 1) return cluster_of<T, 3, true, 1>(npt, multi);
    if (diag && nvar == 3 && pat == 2) return cluster_of<T, 3, true, 2>(npt, multi);
    if (diag && nvar == 3 && pat == 3) return cluster_of<T, 3, true, 3>(npt, multi);
    if (diag && nvar == 2 && pat == 2) return cluster_of<T, 2, true, 2>(npt, multi);
    if (diag && nvar == 2 && pat == 3) return cluster_of<T, 2, true, 3>(npt, multi);
    switch (nvar) {
    case 1: return cluster_of<T, 1, false, 0>(npt, multi);
    case 2: return cluster_of<T, 2, false, 0>(npt, multi);
    case 3: return cluster_of<T, 3, false, 0>(npt, multi);
    default: return cluster_of<T, 4, false, 0>(npt, multi);
    }
}

}  // namespace
