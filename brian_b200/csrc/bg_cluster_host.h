// bg_cluster_host.h -- host side of the cluster kernel (bg_cluster.cuh).
#pragma once
#include "bg_cluster.cuh"

// Bytes of a block's shared memory left to the kernel's own variables.
constexpr int kClusterStaticSmem = 512;

// The built-in instance for 1-4 variables and 1, 2 or 4 neurons per thread;
// multi: several blocks; pat: cluster_body's PAT (an instance without it
// takes PAT 0).
const void *bg_cluster_kernel(int precision, int nvar, int npt, bool diag, bool multi, int pat);
const void *bg_cluster_kernel_f64(int nvar, int npt, bool diag, bool multi, int pat);
const void *bg_cluster_kernel_f32(int nvar, int npt, bool diag, bool multi, int pat);
// Whether one cluster of `blocks` blocks with `smem` bytes each can run; raises
// the kernel's limits.  `generated`: an NVRTC kernel in place of `kernel`.
bool bg_cluster_fits(const void *kernel, cudaKernel_t generated, int blocks, size_t smem);
cudaError_t bg_cluster_launch(const void *kernel, const void *args, int blocks, size_t smem, cudaStream_t s);
