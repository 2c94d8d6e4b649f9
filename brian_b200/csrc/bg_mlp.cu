// bg_mlp.cu -- the learned proposal network for model fitting: a 4-layer MLP
// (64 -> 512 -> 512 -> 512 -> 10, ReLU) whose output is a diagonal Gaussian
// over the fitted parameters (5 means, 5 log standard deviations), trained by
// Gaussian negative log-likelihood with Adam.
//
// Every matrix product runs on the tensor cores (tcgen05) with BF16 operands
// and FP32 accumulation, in three launches (bg_mlpchain.cuh):
//
//   forward   H_l = relu(H_{l-1} W_l^T + b_l)     128 batch rows through all layers
//   backward  G_l = (G_{l+1} W_{l+1}) * [H_l > 0]  likewise
//   weights   dW_l = G_l^T H_{l-1}                 all four, with the bias sums
//
// The chains write each activation and gradient once, row-major; the weight
// gradients read them as MN-major operands, so there are no transposed copies
// of them.  The weights exist as FP32 master copies plus BF16 copies in both
// layouts, written by the Adam kernel.  The output layer is padded from 10 to
// 64 rows (zero rows, zero gradients) so every K is a multiple of 64.  Weight
// gradients split the batch reduction eight ways and the slices are summed in
// a fixed order by the Adam kernel (deterministic).  A training step is six
// launches: gather, forward, loss, backward, weight gradients, Adam (16384
// rows: 351 -> 173 us a step with one product per launch before).
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "bg_common.cuh"
#include "bg_deviceonce.h"
#include "bg_mlpchain.cuh"
#include "../../include/brian_b200.h"

namespace {

int fail(int code, const std::string &m) { return bg_internal_fail(code, m.c_str()); }

#define MCK(call)                                                                            \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return fail(BG_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_));       \
    } while (0)

constexpr int kIn = 64, kHid = 512, kOutPad = 64, kNLayer = 4;
constexpr int kSplits = 8;

typedef __nv_bfloat16 bf16;

// ------------------------------------------------------------------ kernels
// Batch rows of the normalised training set -> X (bf16), Y.  Row b of the batch
// is row order[base + b], base = B * batch_index (a device counter, so the
// gather can sit in a captured graph; null: 0).  Eight threads a row, 32 rows a
// block: each thread two 16-byte loads and one 16-byte store, where one block a
// row was bound by the launch of its blocks (16384 rows: 12.5 -> 5.8 us).
__global__ void __launch_bounds__(256) k_gather(const float *Xall, const float *Yall, const int64_t *order,
                                                const int64_t *batch_index, int B, int ydim, bf16 *X, float *Y) {
    umma::pdl_launch_dependents();
    umma::pdl_wait();
    const int b = blockIdx.x * 32 + (threadIdx.x >> 3), j = (threadIdx.x & 7) * 8;
    if (b >= B) return;
    const int64_t r = order[(batch_index ? *batch_index * B : 0) + b];
    const float4 lo = *reinterpret_cast<const float4 *>(Xall + r * kIn + j);
    const float4 hi = *reinterpret_cast<const float4 *>(Xall + r * kIn + j + 4);
    __nv_bfloat162 h[4] = {__floats2bfloat162_rn(lo.x, lo.y), __floats2bfloat162_rn(lo.z, lo.w),
                           __floats2bfloat162_rn(hi.x, hi.y), __floats2bfloat162_rn(hi.z, hi.w)};
    *reinterpret_cast<uint4 *>(X + (int64_t)b * kIn + j) = *reinterpret_cast<const uint4 *>(h);
    for (int q = threadIdx.x & 7; q < ydim; q += 8) Y[(int64_t)b * ydim + q] = Yall[r * ydim + q];
}

// Gaussian NLL per sample, mean over the batch:
//   sum_d 0.5 ((y_d - mu_d) e^{-s_d})^2 + s_d,  s = clamp(log sigma, -7, 7)
// gradients (already divided by B) into dOUT (bf16; the padded columns stay
// zero from allocation) and per-block column sums of the
// bf16 gradients into colsum[blockIdx.x][64] (the output bias gradient).
__global__ void __launch_bounds__(256) k_nll(const float *OUT, const float *Y, int B, int ydim, bf16 *dO,
                                             float *colsum, float *loss_sum) {
    umma::pdl_launch_dependents();
    umma::pdl_wait();
    constexpr int kMaxY = kOutPad / 2;
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __shared__ float red[8][kOutPad];
    __shared__ float lred[8];
    float l = 0.f;
    const float inv_b = 1.0f / (float)B;
    // (chunks of kYc outputs, so that their loads and the shuffles of their sums
    // overlap; every index below is a constant of the unrolled code)
    constexpr int kYc = 5;
    for (int j0 = 0; j0 < ydim; j0 += kYc) {
        float mu[kYc], sr[kYc], y[kYc], gm[kYc], gs[kYc];
#pragma unroll
        for (int q = 0; q < kYc; ++q) {
            const int j = j0 + q;
            const bool on = b < B && j < ydim && j < kMaxY;
            mu[q] = on ? OUT[(int64_t)b * kOutPad + j] : 0.f;
            sr[q] = on ? OUT[(int64_t)b * kOutPad + ydim + j] : 0.f;
            y[q] = on ? Y[(int64_t)b * ydim + j] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < kYc; ++q) {
            const int j = j0 + q;
            gm[q] = gs[q] = 0.f;
            if (b < B && j < ydim && j < kMaxY) {
                const float s = fminf(fmaxf(sr[q], -7.f), 7.f);
                const float r = (y[q] - mu[q]) * expf(-s);
                l += 0.5f * r * r + s;
                const bf16 g = __float2bfloat16_rn(-r * expf(-s) * inv_b);                                        // d/d mu
                const bf16 gg = __float2bfloat16_rn((sr[q] > -7.f && sr[q] < 7.f) ? (1.f - r * r) * inv_b : 0.f);  // d/d log sigma
                dO[(int64_t)b * kOutPad + j] = g;
                dO[(int64_t)b * kOutPad + ydim + j] = gg;
                gm[q] = __bfloat162float(g);
                gs[q] = __bfloat162float(gg);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int q = 0; q < kYc; ++q) {
                gm[q] += __shfl_xor_sync(0xffffffffu, gm[q], off);
                gs[q] += __shfl_xor_sync(0xffffffffu, gs[q], off);
            }
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < kYc; ++q)
                if (j0 + q < ydim) {
                    red[warp][j0 + q] = gm[q];
                    red[warp][ydim + j0 + q] = gs[q];
                }
    }
    float lv = l;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) lv += __shfl_xor_sync(0xffffffffu, lv, off);
    if (lane == 0) lred[warp] = lv;
    __syncthreads();
    if ((int)threadIdx.x < 2 * ydim) {
        float v = 0.f;
        for (int w = 0; w < 8; ++w) v += red[w][threadIdx.x];
        colsum[(int64_t)blockIdx.x * kOutPad + threadIdx.x] = v;
    }
    if (threadIdx.x == 0) {
        float v = 0.f;
        for (int w = 0; w < 8; ++w) v += lred[w];
        atomicAdd(loss_sum, v / (float)B);
    }
}

__global__ void k_to_bf16(const float *W, int rows, int cols, bf16 *Wb, bf16 *WbT) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (int64_t)rows * cols) return;
    const int r = (int)(i / cols), c = (int)(i % cols);
    const bf16 h = __float2bfloat16_rn(W[i]);
    Wb[i] = h;
    if (WbT) WbT[(int64_t)c * rows + r] = h;
}

// Adam over every parameter tensor of the network in one launch: segment k
// of the flat index space is tensor k (W0, b0, W1, b1, ...), whose gradient
// is the sum of `splits` partial slices.  The step count t comes from device
// memory (the step runs as a captured graph), c1 = 1 - b1^t, c2 = 1 - b2^t.
struct AdamSeg {
    float *P, *m, *v; const float *grad; int splits; int64_t split_stride; int rows, cols, rows_train;
    bf16 *Pb, *PbT;
};
struct AdamAll {
    AdamSeg seg[2 * kNLayer];
    int64_t off[2 * kNLayer + 1];
    int blk0[2 * kNLayer + 1];     // first block of each segment: 32 x 32 tiles of a weight, 256 entries of a bias
    const int64_t *step;
    float lr, b1, b2, eps;
    float scale;                   // gradient multiplier (1: exact; 1/ranks after a summing all-reduce)
};
// The sum of entry i's partial slices, in slice order.
__device__ __forceinline__ float sum_slices(const AdamSeg &sg, int64_t i) {
    float g = 0.f;
    if (sg.splits == kSplits) {
#pragma unroll
        for (int s = 0; s < kSplits; ++s) g += sg.grad[s * sg.split_stride + i];
    } else {
        for (int s = 0; s < sg.splits; ++s) g += sg.grad[s * sg.split_stride + i];
    }
    return g;
}
__device__ __forceinline__ float adam_entry(const AdamAll &a, const AdamSeg &sg, int64_t i, float c1, float c2) {
    const float g = sum_slices(sg, i) * a.scale;
    const float mi = a.b1 * sg.m[i] + (1.f - a.b1) * g;
    const float vi = a.b2 * sg.v[i] + (1.f - a.b2) * g * g;
    sg.m[i] = mi;
    sg.v[i] = vi;
    const float p = sg.P[i] - a.lr * (mi / c1) / (sqrtf(vi / c2) + a.eps);
    sg.P[i] = p;
    return p;
}
// Bound by the 28 bytes an entry moves plus 4 per partial slice.  A block updates a
// 32 x 32 tile of one weight, so that its bf16 copy and (through shared memory) the
// transposed one are written in whole rows by the same launch: 13.6 us and 5.7 us
// of a second one before, 13.2 us now.
__global__ void __launch_bounds__(256) k_adam_all(const __grid_constant__ AdamAll a) {
    umma::pdl_launch_dependents();
    umma::pdl_wait();
    __shared__ float corr[2];
    __shared__ bf16 tile[32][33];
    if (threadIdx.x < 2) corr[threadIdx.x] = 1.f - powf(threadIdx.x ? a.b2 : a.b1, (float)*a.step);
    __syncthreads();
    int k = 0;
#pragma unroll
    for (int q = 1; q < 2 * kNLayer; ++q) k += (int)blockIdx.x >= a.blk0[q] ? 1 : 0;
    const AdamSeg &sg = a.seg[k];
    const int blk = (int)blockIdx.x - a.blk0[k];
    const float c1 = corr[0], c2 = corr[1];
    if (!sg.Pb) {
        const int i = blk * 256 + (int)threadIdx.x;
        if (i < sg.rows_train) adam_entry(a, sg, i, c1, c2);
        return;
    }
    const int tcols = sg.cols / 32, r0 = (blk / tcols) * 32, c0 = (blk % tcols) * 32;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const int r = r0 + ty + j;
        const int64_t i = (int64_t)r * sg.cols + c0 + tx;
        const bf16 p = __float2bfloat16_rn(r < sg.rows_train ? adam_entry(a, sg, i, c1, c2) : sg.P[i]);
        sg.Pb[i] = p;
        tile[ty + j][tx] = p;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 32; j += 8) sg.PbT[(int64_t)(c0 + ty + j) * sg.rows + r0 + tx] = tile[tx][ty + j];
}
static_assert(kIn % 32 == 0 && kHid % 32 == 0 && kOutPad % 32 == 0, "Adam's tiles are whole");

// The gradient of every tensor as one flat vector in the optimiser's segment
// order (W0, b0, W1, b1, ...): each entry the sum of its partial slices in
// the order Adam sums them, so an update from the flat vector (scale 1)
// equals the fused one.  Data-parallel training all-reduces this vector.
__global__ void k_grad_flat(const __grid_constant__ AdamAll a, float *flat) {
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 >= a.off[2 * kNLayer]) return;
    int k = 0;
#pragma unroll
    for (int q = 1; q < 2 * kNLayer; ++q) k += i0 >= a.off[q] ? 1 : 0;
    const AdamSeg &sg = a.seg[k];
    const int64_t i = i0 - a.off[k];
    flat[i0] = sum_slices(sg, i);
}

// The bookkeeping of a step whose gradients come from outside: the batch index
// within the epoch and the optimiser step (a training step's own are advanced by
// the weight-gradient kernel).
__global__ void k_step_advance(int64_t *batch_index, int64_t *opt_step) {
    umma::pdl_launch_dependents();
    umma::pdl_wait();
    *batch_index += 1;
    *opt_step += 1;
}

// The epoch's batch order: rows sorted by a Philox draw keyed (seed, epoch, row).
__global__ void k_perm_keys(uint64_t seed, int64_t epoch, int64_t n, unsigned long long *keys, int64_t *vals) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t c[4] = {(uint32_t)i, (uint32_t)((uint64_t)i >> 32), (uint32_t)epoch, (uint32_t)((uint64_t)epoch >> 32)};
        bg_philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
        keys[i] = ((unsigned long long)c[0] << 32) | c[1];
        vals[i] = i;
    }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no
// link against the driver library); null when unavailable.
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
                        q == cudaDriverEntryPointSuccess;
        cudaGetLastError();
        return ok ? (EncodeTiledFn)p : nullptr;
    }();
    return fn;
}

// A device and its multiprocessors.
struct Device { int id, sms; };
Device device_of(int id) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, id) != cudaSuccess || n <= 0) n = 148;
    return {id, n};
}

// The dynamic shared memory that a kernel may take, raised once per device
// (the attribute belongs to the kernel on the current device `dev`; handles on
// several devices and threads share the kernels).
int raise_smem(int dev, const void *kernel, size_t bytes) {
    static DeviceOnce once;
    cudaError_t e = cudaSuccess;
    if (!once(dev, kernel, [&] {
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            return e == cudaSuccess;
        }))
        return fail(BG_ECUDA, std::string("mlp: shared memory of a kernel: ") + cudaGetErrorString(e));
    return BG_OK;
}

// 2-D map of a row-major bf16 matrix [rows][ld] over its first `cols`
// columns, zero fill past the edges: boxes of 8 columns x box_rows rows
// (no swizzle), or with sw128 of 64 columns (one 128-byte line) x box_rows
// rows landing in the 128-byte swizzled layout.
bool tile_map(CUtensorMap *m, const bf16 *base, int rows, int cols, int ld, int box_rows, bool sw128 = false) {
    EncodeTiledFn f = encode_tiled();
    if (!f || ((uintptr_t)base & 15) || ((size_t)ld * 2) % 16 || cols % (sw128 ? 64 : 8)) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {sw128 ? 64u : 8u, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)base, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, sw128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT, bool TMA>
int launch_gemm_as(const umma::GemmArgs &g, int splits, const Device &dev, cudaStream_t st, const CUtensorMap &ta,
                   const CUtensorMap &tb) {
    constexpr size_t smem = umma::smem_bytes<NT>();
    if (int rc = raise_smem(dev.id, (const void *)(umma::k_gemm<NT, TMA>), smem)) return rc;
    dim3 grid((unsigned)((g.M + umma::kM - 1) / umma::kM), (unsigned)((g.N + NT - 1) / NT), (unsigned)splits);
    umma::k_gemm<NT, TMA><<<grid, umma::kThreads, smem, st>>>(g, ta, tb);
    MCK(cudaGetLastError());
    return BG_OK;
}

// Launch with programmatic stream serialization: the kernel may start while
// the previous one in the stream finishes; it waits (griddepcontrol.wait)
// before reading anything that one wrote.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// The persistent warp-specialised kernel over all tiles of the product.
template <int NT>
int launch_gemm_persistent(const umma::GemmArgs &g, int splits, const Device &dev, cudaStream_t st, const CUtensorMap &ta,
                           const CUtensorMap &tb) {
    constexpr size_t smem = umma::psmem_bytes<NT>();
    if (int rc = raise_smem(dev.id, (const void *)umma::k_gemm_p<NT>, smem)) return rc;
    const int tiles_m = (g.M + umma::kM - 1) / umma::kM, tiles_n = (g.N + NT - 1) / NT;
    const int ntiles = tiles_m * tiles_n * splits;
    const int grid = std::max(1, std::min(ntiles, dev.sms));
    MCK(launch_pdl(umma::k_gemm_p<NT>, dim3(grid), dim3(umma::kPThreads), smem, st, g, ta, tb, tiles_m, tiles_n,
                   splits));
    return BG_OK;
}

// TMA-fed persistent kernel when both operands allow a tensor map (16-byte
// aligned rows, K a multiple of 8) and every split has K-chunks, else the
// one-tile-per-CTA kernel with cp.async stages.
template <int NT>
int launch_gemm(const umma::GemmArgs &g, int splits, const Device &dev, cudaStream_t st) {
    CUtensorMap ta, tb;
    memset(&ta, 0, sizeof ta);
    memset(&tb, 0, sizeof tb);
    if (g.k_per_split >= umma::kKc && g.k_per_split % umma::kKc == 0 && (long long)g.k_per_split * splits == g.K &&
        tile_map(&ta, g.A, g.M, g.K, g.lda, umma::kM, true) && tile_map(&tb, g.B, g.N, g.K, g.ldb, NT, true))
        return launch_gemm_persistent<NT>(g, splits, dev, st, ta, tb);
    memset(&ta, 0, sizeof ta);
    memset(&tb, 0, sizeof tb);
    return launch_gemm_as<NT, false>(g, splits, dev, st, ta, tb);
}

template <bool BWD>
int launch_chain(const umma::ChainArgs &g, const umma::ChainMaps &m, const Device &dev, cudaStream_t st) {
    constexpr size_t smem = umma::chain_smem_bytes();
    if (int rc = raise_smem(dev.id, (const void *)umma::k_mlp_chain<BWD>, smem)) return rc;
    const int grid = std::max(1, std::min(g.rows / umma::kM, dev.sms));
    MCK(launch_pdl(umma::k_mlp_chain<BWD>, dim3(grid), dim3(umma::kPThreads), smem, st, g, m));
    return BG_OK;
}

int launch_weight_gradients(const umma::DwArgs &g, const umma::DwMaps &m, const Device &dev, cudaStream_t st) {
    constexpr size_t smem = sizeof(umma::DwSmem);
    if (int rc = raise_smem(dev.id, (const void *)umma::k_weight_gradients, smem)) return rc;
    const int grid = std::max(1, std::min(g.units, dev.sms));
    MCK(launch_pdl(umma::k_weight_gradients, dim3(grid), dim3(umma::kPThreads), smem, st, g, m));
    return BG_OK;
}

umma::GemmArgs gemm_args(const bf16 *A, int lda, const bf16 *B, int ldb, int M, int N, int K, int *err) {
    umma::GemmArgs g;
    memset(&g, 0, sizeof g);
    g.A = A;
    g.B = B;
    g.M = M;
    g.N = N;
    g.K = K;
    g.lda = lda;
    g.ldb = ldb;
    g.k_per_split = K;
    g.err = err;
    return g;
}

template <typename T>
void dfree(T *&p) {
    if (p) cudaFree((void *)p);
    p = nullptr;
}

template <typename T>
int dalloc(T **p, size_t n) {
    dfree(*p);
    if (n == 0) return BG_OK;
    if (cudaMalloc((void **)p, n * sizeof(T)) != cudaSuccess) return fail(BG_ENOMEM, "mlp: cudaMalloc failed");
    cudaMemset(*p, 0, n * sizeof(T));
    return BG_OK;
}

}  // namespace

struct bg_mlp {
    int device = 0;
    Device dev = {0, 148};
    int ydim = 5;
    cudaStream_t stream = nullptr;
    int *err = nullptr;
    // parameters: layer l has W[l] [rows][cols] (fp32 master), b[l]
    int rows[kNLayer] = {kHid, kHid, kHid, kOutPad};
    int cols[kNLayer] = {kIn, kHid, kHid, kHid};
    float *W[kNLayer] = {}, *b[kNLayer] = {}, *mW[kNLayer] = {}, *vW[kNLayer] = {}, *mb[kNLayer] = {},
          *vb[kNLayer] = {};
    bf16 *Wb[kNLayer] = {}, *WbT[kNLayer] = {};
    float *gW = nullptr;                  // weight-gradient scratch: per layer, kSplits partial slices
    float *gWl[kNLayer] = {};             //   layer l's region of gW
    int64_t *dBatchIdx = nullptr;         // device counters of a training step: batch within the epoch,
    int64_t *dOptStep = nullptr;          //   optimiser step
    // epoch order: Philox keys sorted with their row indices
    unsigned long long *pkeys = nullptr, *pkeys_out = nullptr; int64_t *pvals = nullptr, *perm = nullptr;
    void *sort_tmp = nullptr; size_t sort_tmp_bytes = 0;
    // one training step captured as a graph (rebuilt when the batch size changes)
    cudaGraphExec_t step_graph = nullptr; int graph_batch = 0; float graph_lr = 0.f;
    float *cs[kNLayer] = {};              // bias-gradient partials per layer [row blocks][512]
    float *gbias = nullptr;               // their sums, [kNLayer][512]
    int64_t step = 0;
    // the launches' arguments over the batch buffers (plan_batch)
    umma::ChainArgs fwd, bwd;
    umma::ChainMaps fwd_maps, bwd_maps;
    umma::DwArgs dw;
    umma::DwMaps dw_maps;
    // batch buffers
    int B = 0;
    bf16 *X = nullptr, *H[3] = {}, *G[3] = {}, *dO = nullptr;
    uint32_t *mask[3] = {};               // nonzero bits of the hidden activations, [B][16]
    float *OUT = nullptr, *Y = nullptr;
    float *loss = nullptr;                // one allocation with err: read back in one copy
    int64_t *idx = nullptr;
    // training set
    int64_t nset = 0;
    float *Xall = nullptr, *Yall = nullptr;
    float last_forward_ms = 0;
    float *gflat = nullptr; int64_t nflat = 0;   // flat gradient (data-parallel steps)
};

namespace {

// Bias-gradient partials of layer l: per-block column sums written by the
// loss kernel (output layer, blocks of 256 rows, 64 columns) or by the
// ReLU-gradient epilogue that produced G[l] (blocks of 32 rows).
void bias_partials(const bg_mlp *h, int l, int B, const float **p, int *nblk, int *ld) {
    *p = h->cs[l];
    if (l == kNLayer - 1) {
        *nblk = (B + 255) / 256;
        *ld = kOutPad;
    } else {
        *nblk = 4 * ((B + umma::kM - 1) / umma::kM);
        *ld = kHid;
    }
}

// Arguments and tensor maps of the chains and the weight gradients over batch
// buffers of B rows (a multiple of 128).
int plan_batch(bg_mlp *h, int B) {
    memset(&h->fwd, 0, sizeof h->fwd);
    memset(&h->bwd, 0, sizeof h->bwd);
    memset(&h->dw, 0, sizeof h->dw);
    h->fwd.layers = kNLayer;
    h->bwd.layers = kNLayer - 1;
    h->fwd.rows = h->bwd.rows = B;
    h->fwd.err = h->bwd.err = h->dw.err = h->err;
    bool ok = tile_map(&h->fwd_maps.in, h->X, B, kIn, kIn, umma::kM, true) &&
              tile_map(&h->bwd_maps.in, h->dO, B, kOutPad, kOutPad, umma::kM, true);
    for (int l = 0; l < kNLayer; ++l) {
        umma::ChainLayer &L = h->fwd.L[l];
        L.K = h->cols[l];
        L.N = h->rows[l];
        L.bias = h->b[l];
        if (l < 3) {
            L.keep = 1;
            L.mask = h->mask[l];
            ok = ok && tile_map(&h->fwd_maps.out[l], h->H[l], B, kHid, kHid, umma::kM, true);
        } else {
            L.C = h->OUT;
        }
        ok = ok && tile_map(&h->fwd_maps.w[l], h->Wb[l], L.N, L.K, L.K, std::min(L.N, umma::kChainN), true);
    }
    for (int q = 0; q < kNLayer - 1; ++q) {
        const int l = 3 - q;                 // through W_l into hidden layer l - 1
        umma::ChainLayer &L = h->bwd.L[q];
        L.K = h->rows[l];
        L.N = h->cols[l];
        L.keep = 1;
        L.mask = h->mask[l - 1];
        L.colsum = h->cs[l - 1];
        ok = ok && tile_map(&h->bwd_maps.out[q], h->G[l - 1], B, kHid, kHid, umma::kM, true);
        ok = ok && tile_map(&h->bwd_maps.w[q], h->WbT[l], L.N, L.K, L.K, umma::kChainN, true);
    }
    // the weight gradients need whole 64-row chunks in each split (the training
    // calls ask for it; the buffers of a forward call may have any 128 rows)
    if (B % (kSplits * umma::kKc) == 0) {
        h->dw.splits = kSplits;
        h->dw.nk = B / kSplits / umma::kKc;
        const int order[kNLayer] = {2, 1, 3, 0};             // the widest units first
        for (int q = 0; q < kNLayer; ++q) {
            const int l = order[q];
            umma::DwProduct &p = h->dw.p[q];
            p.M = h->rows[l];
            p.N = h->cols[l];
            p.nt = p.N == kHid ? umma::kDwN : 64;
            p.tiles_m = (p.M + umma::kM - 1) / umma::kM;
            p.tiles_n = p.N / p.nt;
            p.unit0 = h->dw.units;
            h->dw.units += p.tiles_m * p.tiles_n * kSplits;
            p.C = h->gWl[l];
            p.split_stride = (long long)p.M * p.N;
            ok = ok && tile_map(&h->dw_maps.a[q], l == 3 ? h->dO : h->G[l], B, p.M, p.M, umma::kKc, true);
            ok = ok && tile_map(&h->dw_maps.b[q], l > 0 ? h->H[l - 1] : h->X, B, p.N, p.N, umma::kKc, true);
        }
        umma::BiasRed &r = h->dw.bias;
        for (int l = 0; l < kNLayer; ++l) {
            bias_partials(h, l, B, &r.p[l], &r.nblk[l], &r.ld[l]);
            r.rows[l] = h->rows[l];
            r.blk0[l + 1] = r.blk0[l] + (r.rows[l] + 31) / 32;
        }
        r.out = h->gbias;
    }
    return ok ? BG_OK : fail(BG_ECUDA, "mlp: tensor map");
}

int ensure_batch(bg_mlp *h, int B) {
    if (B == h->B) return BG_OK;
    // the batch buffers move: a captured training step holds their addresses
    if (h->step_graph) {
        cudaStreamSynchronize(h->stream);
        cudaGraphExecDestroy(h->step_graph);
        h->step_graph = nullptr;
        h->graph_batch = 0;
    }
    int rc = 0;
    h->B = 0;
    if ((rc = dalloc(&h->X, (size_t)B * kIn))) return rc;
    for (int l = 0; l < 3; ++l) {
        if ((rc = dalloc(&h->H[l], (size_t)B * kHid))) return rc;
        if ((rc = dalloc(&h->G[l], (size_t)B * kHid))) return rc;
        if ((rc = dalloc(&h->mask[l], (size_t)B * (kHid / 32)))) return rc;
    }
    if ((rc = dalloc(&h->dO, (size_t)B * kOutPad))) return rc;
    if ((rc = dalloc(&h->OUT, (size_t)B * kOutPad))) return rc;
    if ((rc = dalloc(&h->Y, (size_t)B * h->ydim))) return rc;
    if ((rc = dalloc(&h->idx, (size_t)B))) return rc;
    for (int l = 0; l < kNLayer; ++l)
        if ((rc = dalloc(&h->cs[l], (size_t)((B + 31) / 32) * kHid))) return rc;
    if (!h->gbias && (rc = dalloc(&h->gbias, (size_t)kNLayer * kHid))) return rc;
    if ((rc = plan_batch(h, B))) return rc;
    MCK(cudaStreamSynchronize(nullptr));     // the buffers are cleared before h->stream writes them
    h->B = B;
    return BG_OK;
}

// forward of the batch in h->X -> h->OUT, and (keep) the hidden activations -> h->H
int forward(bg_mlp *h, bool keep) {
    umma::ChainArgs g = h->fwd;
    if (!keep)
        for (int l = 0; l < 3; ++l) { g.L[l].keep = 0; g.L[l].mask = nullptr; }
    return launch_chain<false>(g, h->fwd_maps, h->dev, h->stream);
}

// backward from the loss gradient in h->dO: the hidden layers' gradients -> h->G
// with the column-sum partials of their bias gradients, then the weight gradients'
// partial slices -> h->gWl and the bias gradients -> h->gbias.  `advance`: also
// count the training step.
int backward(bg_mlp *h, bool advance) {
    int rc = launch_chain<true>(h->bwd, h->bwd_maps, h->dev, h->stream);
    if (rc) return rc;
    umma::DwArgs g = h->dw;
    if (advance) {
        g.batch_index = (long long *)h->dBatchIdx;
        g.opt_step = (long long *)h->dOptStep;
    }
    return launch_weight_gradients(g, h->dw_maps, h->dev, h->stream);
}

// Adam's tensor descriptors: gradients from the partial slices of a batch
// of B rows, or (flat != null) from a flat gradient vector
AdamAll adam_desc(bg_mlp *h, int B, float lr, const float *flat, float scale) {
    AdamAll a;
    memset(&a, 0, sizeof a);
    int64_t off = 0;
    for (int l = 0; l < kNLayer; ++l) {
        const int rows_train = l == 3 ? 2 * h->ydim : h->rows[l];
        AdamSeg &w = a.seg[2 * l];
        w.P = h->W[l]; w.m = h->mW[l]; w.v = h->vW[l]; w.grad = h->gWl[l]; w.splits = kSplits;
        w.split_stride = (int64_t)h->rows[l] * h->cols[l]; w.rows = h->rows[l]; w.cols = h->cols[l];
        w.rows_train = rows_train; w.Pb = h->Wb[l]; w.PbT = h->WbT[l];
        a.off[2 * l] = off;
        off += (int64_t)h->rows[l] * h->cols[l];
        AdamSeg &bb = a.seg[2 * l + 1];
        bb.P = h->b[l]; bb.m = h->mb[l]; bb.v = h->vb[l];
        bb.grad = h->gbias + (int64_t)l * kHid; bb.splits = 1; bb.split_stride = 0;   // the weight-gradient kernel's sums
        bb.rows = h->rows[l]; bb.cols = 1; bb.rows_train = rows_train;
        a.off[2 * l + 1] = off;
        off += h->rows[l];
    }
    a.off[2 * kNLayer] = off;
    for (int k = 0; k < 2 * kNLayer; ++k)
        a.blk0[k + 1] = a.blk0[k] + (a.seg[k].Pb ? (a.seg[k].rows / 32) * (a.seg[k].cols / 32) : (a.seg[k].rows + 255) / 256);
    a.step = h->dOptStep;
    a.lr = lr; a.b1 = 0.9f; a.b2 = 0.999f; a.eps = 1e-8f; a.scale = scale;
    if (flat)
        for (int k = 0; k < 2 * kNLayer; ++k) { a.seg[k].grad = flat + a.off[k]; a.seg[k].splits = 1; a.seg[k].split_stride = 0; }
    return a;
}

// Adam on every tensor in one launch (the step count is read on the device)
int adam_all(bg_mlp *h, int B, float lr, const float *flat = nullptr, float scale = 1.f) {
    const AdamAll a = adam_desc(h, B, lr, flat, scale);
    MCK(launch_pdl(k_adam_all, dim3((unsigned)a.blk0[2 * kNLayer]), dim3(256), 0, h->stream, a));
    return BG_OK;
}

int gather(bg_mlp *h, const int64_t *order, const int64_t *batch_index) {
    MCK(launch_pdl(k_gather, dim3((unsigned)((h->B + 31) / 32)), dim3(256), 0, h->stream, (const float *)h->Xall,
                   (const float *)h->Yall, order, batch_index, h->B, h->ydim, h->X, h->Y));
    return BG_OK;
}

int loss_gradient(bg_mlp *h) {
    MCK(launch_pdl(k_nll, dim3((h->B + 255) / 256), dim3(256), 0, h->stream, (const float *)h->OUT, (const float *)h->Y, h->B,
                   h->ydim, h->dO, h->cs[kNLayer - 1], h->loss));
    return BG_OK;
}

// one training step on batch `*dBatchIdx` of h->perm: gather, forward, loss,
// backward, Adam, counters
int train_step(bg_mlp *h, int B, float lr) {
    int rc = gather(h, h->perm, h->dBatchIdx);
    if (rc || (rc = forward(h, true))) return rc;
    if ((rc = loss_gradient(h))) return rc;
    // Adam's step count t is the step being taken (1 for the first)
    if ((rc = backward(h, true))) return rc;
    return adam_all(h, B, lr);
}

// the epoch order buffers and the sort's scratch, kept for later calls
int ensure_perm(bg_mlp *h) {
    if (h->perm) return BG_OK;
    int rc;
    if ((rc = dalloc(&h->pkeys, (size_t)h->nset)) || (rc = dalloc(&h->pkeys_out, (size_t)h->nset)) ||
        (rc = dalloc(&h->pvals, (size_t)h->nset)) || (rc = dalloc(&h->perm, (size_t)h->nset)))
        return rc;
    size_t bytes = 0;
    MCK(cub::DeviceRadixSort::SortPairs(nullptr, bytes, h->pkeys, h->pkeys_out, h->pvals, h->perm, (int)h->nset));
    MCK(cudaMalloc(&h->sort_tmp, bytes));
    h->sort_tmp_bytes = bytes;
    return BG_OK;
}

// the epoch's order: rows sorted by Philox keys (seed, epoch, row)
int epoch_perm(bg_mlp *h, uint64_t seed, int64_t ep) {
    k_perm_keys<<<(unsigned)std::min<int64_t>((h->nset + 255) / 256, 4096), 256, 0, h->stream>>>(
        seed, ep, h->nset, h->pkeys, h->pvals);
    MCK(cudaGetLastError());
    MCK(cub::DeviceRadixSort::SortPairs(h->sort_tmp, h->sort_tmp_bytes, h->pkeys, h->pkeys_out, h->pvals, h->perm,
                                        (int)h->nset, 0, 64, h->stream));
    return BG_OK;
}

int check_err(bg_mlp *h) {
    int e = 0;
    MCK(cudaMemcpy(&e, h->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) return fail(BG_ETIMEOUT, "mlp: a tensor-core wait gave up");
    return BG_OK;
}

}  // namespace

extern "C" {

BG_API int bg_mlp_create(bg_mlp **out, int device, int ydim) {
    if (!out || ydim <= 0 || 2 * ydim > kOutPad) return fail(BG_EINVAL, "mlp: bad arguments");
    *out = nullptr;
    MCK(cudaSetDevice(device));
    bg_mlp *h = new bg_mlp();
    h->device = device;
    h->dev = device_of(device);
    h->ydim = ydim;
    int rc = 0;
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess) rc = fail(BG_ECUDA, "mlp: stream");
    for (int l = 0; l < kNLayer && !rc; ++l) {
        const size_t n = (size_t)h->rows[l] * h->cols[l];
        if (!rc) rc = dalloc(&h->W[l], n);
        if (!rc) rc = dalloc(&h->mW[l], n);
        if (!rc) rc = dalloc(&h->vW[l], n);
        if (!rc) rc = dalloc(&h->b[l], (size_t)h->rows[l]);
        if (!rc) rc = dalloc(&h->mb[l], (size_t)h->rows[l]);
        if (!rc) rc = dalloc(&h->vb[l], (size_t)h->rows[l]);
        if (!rc) rc = dalloc(&h->Wb[l], n);
        if (!rc) rc = dalloc(&h->WbT[l], n);
    }
    {
        size_t tot = 0;
        for (int l = 0; l < kNLayer; ++l) tot += (size_t)kSplits * h->rows[l] * h->cols[l];
        if (!rc) rc = dalloc(&h->gW, tot);
        size_t o = 0;
        for (int l = 0; l < kNLayer && !rc; ++l) { h->gWl[l] = h->gW + o; o += (size_t)kSplits * h->rows[l] * h->cols[l]; }
    }
    if (!rc) rc = dalloc(&h->dBatchIdx, 1);
    if (!rc) rc = dalloc(&h->dOptStep, 1);
    if (!rc) rc = dalloc(&h->loss, 2);
    if (!rc) h->err = reinterpret_cast<int *>(h->loss + 1);
    if (rc) {
        bg_mlp_destroy(h);
        return rc;
    }
    *out = h;
    return BG_OK;
}

BG_API int bg_mlp_destroy(bg_mlp *h) {
    if (!h) return BG_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (int l = 0; l < kNLayer; ++l) {
        dfree(h->W[l]); dfree(h->b[l]); dfree(h->mW[l]); dfree(h->vW[l]); dfree(h->mb[l]); dfree(h->vb[l]);
        dfree(h->Wb[l]); dfree(h->WbT[l]);
    }
    for (int l = 0; l < 3; ++l) { dfree(h->H[l]); dfree(h->G[l]); dfree(h->mask[l]); }
    dfree(h->X); dfree(h->dO); dfree(h->OUT); dfree(h->Y); dfree(h->idx);
    for (int l = 0; l < kNLayer; ++l) dfree(h->cs[l]);
    dfree(h->gW); dfree(h->gbias); dfree(h->gflat); dfree(h->loss); dfree(h->Xall); dfree(h->Yall);
    dfree(h->dBatchIdx); dfree(h->dOptStep); dfree(h->pkeys); dfree(h->pkeys_out); dfree(h->pvals); dfree(h->perm);
    if (h->sort_tmp) cudaFree(h->sort_tmp);
    if (h->step_graph) cudaGraphExecDestroy(h->step_graph);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return BG_OK;
}

BG_API int bg_mlp_set_params(bg_mlp *h, int layer, const float *W, const float *b) {
    if (!h || layer < 0 || layer >= kNLayer || !W || !b) return fail(BG_EINVAL, "mlp: bad parameter set");
    MCK(cudaSetDevice(h->device));
    const size_t n = (size_t)h->rows[layer] * h->cols[layer];
    MCK(cudaMemcpy(h->W[layer], W, n * sizeof(float), cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(h->b[layer], b, (size_t)h->rows[layer] * sizeof(float), cudaMemcpyHostToDevice));
    MCK(cudaMemset(h->mW[layer], 0, n * sizeof(float)));
    MCK(cudaMemset(h->vW[layer], 0, n * sizeof(float)));
    MCK(cudaMemset(h->mb[layer], 0, (size_t)h->rows[layer] * sizeof(float)));
    MCK(cudaMemset(h->vb[layer], 0, (size_t)h->rows[layer] * sizeof(float)));
    k_to_bf16<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>(h->W[layer], h->rows[layer], h->cols[layer],
                                                                    h->Wb[layer], h->WbT[layer]);
    MCK(cudaGetLastError());
    MCK(cudaMemsetAsync(h->dOptStep, 0, sizeof(int64_t), h->stream));
    MCK(cudaStreamSynchronize(h->stream));
    h->step = 0;
    return BG_OK;
}

BG_API int bg_mlp_get_params(bg_mlp *h, int layer, float *W, float *b) {
    if (!h || layer < 0 || layer >= kNLayer) return fail(BG_EINVAL, "mlp: bad layer");
    MCK(cudaSetDevice(h->device));
    MCK(cudaStreamSynchronize(h->stream));
    if (W) MCK(cudaMemcpy(W, h->W[layer], (size_t)h->rows[layer] * h->cols[layer] * sizeof(float),
                          cudaMemcpyDeviceToHost));
    if (b) MCK(cudaMemcpy(b, h->b[layer], (size_t)h->rows[layer] * sizeof(float), cudaMemcpyDeviceToHost));
    return BG_OK;
}

BG_API int bg_mlp_forward(bg_mlp *h, const float *X, int64_t n, float *out) {
    if (!h || !X || n <= 0 || !out) return fail(BG_EINVAL, "mlp: bad forward call");
    MCK(cudaSetDevice(h->device));
    const int B = (int)((n + 127) / 128 * 128);
    int rc = ensure_batch(h, B);
    if (rc) return rc;
    std::vector<bf16> xb((size_t)B * kIn, __float2bfloat16_rn(0.f));
    for (int64_t r = 0; r < n; ++r)
        for (int j = 0; j < kIn; ++j) xb[(size_t)r * kIn + j] = __float2bfloat16_rn(X[r * kIn + j]);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, h->stream);
    MCK(cudaMemcpyAsync(h->X, xb.data(), xb.size() * sizeof(bf16), cudaMemcpyHostToDevice, h->stream));
    if ((rc = forward(h, false))) return rc;
    std::vector<float> o((size_t)B * kOutPad);
    MCK(cudaMemcpyAsync(o.data(), h->OUT, o.size() * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    cudaEventRecord(e1, h->stream);
    MCK(cudaStreamSynchronize(h->stream));
    cudaEventElapsedTime(&h->last_forward_ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if ((rc = check_err(h))) return rc;
    for (int64_t r = 0; r < n; ++r)
        for (int j = 0; j < 2 * h->ydim; ++j) out[r * 2 * h->ydim + j] = o[(size_t)r * kOutPad + j];
    return BG_OK;
}

BG_API int bg_mlp_last_forward_ms(bg_mlp *h, float *ms) {
    if (!h || !ms) return fail(BG_EINVAL, "mlp: bad arguments");
    *ms = h->last_forward_ms;
    return BG_OK;
}

BG_API int bg_mlp_set_data(bg_mlp *h, const float *X, const float *Y, int64_t n) {
    if (!h || !X || !Y || n <= 0) return fail(BG_EINVAL, "mlp: bad training set");
    MCK(cudaSetDevice(h->device));
    MCK(cudaStreamSynchronize(h->stream));
    // the training set moves: the epoch-order buffers and the captured step
    // (which holds its addresses) are rebuilt by the next bg_mlp_train
    dfree(h->pkeys); dfree(h->pkeys_out); dfree(h->pvals); dfree(h->perm);
    if (h->sort_tmp) { cudaFree(h->sort_tmp); h->sort_tmp = nullptr; h->sort_tmp_bytes = 0; }
    if (h->step_graph) { cudaGraphExecDestroy(h->step_graph); h->step_graph = nullptr; h->graph_batch = 0; }
    int rc = dalloc(&h->Xall, (size_t)n * kIn);
    if (!rc) rc = dalloc(&h->Yall, (size_t)n * h->ydim);
    if (rc) return rc;
    MCK(cudaMemcpy(h->Xall, X, (size_t)n * kIn * sizeof(float), cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(h->Yall, Y, (size_t)n * h->ydim * sizeof(float), cudaMemcpyHostToDevice));
    h->nset = n;
    return BG_OK;
}

BG_API int bg_mlp_train(bg_mlp *h, int epochs, int batch, float lr, uint64_t seed, float *epoch_loss,
                        float *gpu_ms) {
    if (!h || epochs < 0 || batch < 128 || batch % 128 != 0 || (batch / kSplits) % umma::kKc != 0)
        return fail(BG_EINVAL, "mlp: batch must be a multiple of 512 (128 rows x 8 batch splits of 64)");
    if (h->nset < batch) return fail(BG_ESTATE, "mlp: training set smaller than one batch");
    MCK(cudaSetDevice(h->device));
    int rc = ensure_batch(h, batch);
    if (rc) return rc;
    const int64_t steps = h->nset / batch;
    if ((rc = ensure_perm(h))) return rc;
    cudaEvent_t e0, e1;
    MCK(cudaEventCreate(&e0));
    MCK(cudaEventCreate(&e1));
    MCK(cudaEventRecord(e0, h->stream));
    for (int ep = 0; ep < epochs && !rc; ++ep) {
        if ((rc = epoch_perm(h, seed, ep))) break;
        MCK(cudaMemsetAsync(h->loss, 0, sizeof(float), h->stream));
        MCK(cudaMemsetAsync(h->dBatchIdx, 0, sizeof(int64_t), h->stream));
        for (int64_t s = 0; s < steps && !rc; ++s) {
            if (h->step_graph && h->graph_batch == batch && h->graph_lr == lr) {
                MCK(cudaGraphLaunch(h->step_graph, h->stream));
            } else if (s == 0) {
                // the first step runs directly (kernel attributes, tensor maps)
                rc = train_step(h, batch, lr);
            } else {
                // capture one step and replay it for the rest of training
                if (h->step_graph) { cudaGraphExecDestroy(h->step_graph); h->step_graph = nullptr; }
                cudaGraph_t graph = nullptr;
                MCK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
                rc = train_step(h, batch, lr);
                cudaError_t ce = cudaStreamEndCapture(h->stream, &graph);
                if (!rc && ce != cudaSuccess) rc = fail(BG_ECUDA, std::string("mlp: step capture: ") + cudaGetErrorString(ce));
                if (!rc && cudaGraphInstantiate(&h->step_graph, graph, 0) != cudaSuccess)
                    rc = fail(BG_ECUDA, "mlp: step graph instantiation failed");
                if (graph) cudaGraphDestroy(graph);
                if (rc) break;
                h->graph_batch = batch;
                h->graph_lr = lr;
                MCK(cudaGraphLaunch(h->step_graph, h->stream));
            }
        }
        h->step += steps;
        float ls = 0;
        cudaMemcpyAsync(&ls, h->loss, sizeof(float), cudaMemcpyDeviceToHost, h->stream);
        cudaError_t e = cudaStreamSynchronize(h->stream);
        if (!rc && e != cudaSuccess) rc = fail(BG_ECUDA, std::string("mlp: training failed: ") + cudaGetErrorString(e));
        if (!rc) rc = check_err(h);
        if (epoch_loss) epoch_loss[ep] = ls / (float)steps;
    }
    cudaEventRecord(e1, h->stream);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    if (gpu_ms) *gpu_ms = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
}

BG_API int bg_mlp_epoch_order(bg_mlp *h, uint64_t seed, int64_t epoch) {
    if (!h || epoch < 0) return fail(BG_EINVAL, "mlp: bad epoch");
    if (h->nset <= 0) return fail(BG_ESTATE, "mlp: no training set");
    MCK(cudaSetDevice(h->device));
    int rc = ensure_perm(h);
    if (!rc) rc = epoch_perm(h, seed, epoch);
    if (!rc) MCK(cudaStreamSynchronize(h->stream));
    return rc;
}

BG_API int bg_mlp_step_gradients(bg_mlp *h, int batch, int64_t row0, float *loss, void **grad, int64_t *ngrad) {
    if (!h || batch < 128 || batch % 128 != 0 || (batch / kSplits) % umma::kKc != 0)
        return fail(BG_EINVAL, "mlp: batch must be a multiple of 512 (128 rows x 8 batch splits of 64)");
    if (!h->perm) return fail(BG_ESTATE, "mlp: no epoch order (bg_mlp_epoch_order)");
    if (row0 < 0 || row0 % batch != 0 || row0 + batch > h->nset) return fail(BG_EINVAL, "mlp: rows outside the epoch");
    MCK(cudaSetDevice(h->device));
    int rc = ensure_batch(h, batch);
    if (rc) return rc;
    const int64_t nflat = adam_desc(h, batch, 0.f, nullptr, 1.f).off[2 * kNLayer];
    if (h->nflat != nflat) {
        if ((rc = dalloc(&h->gflat, (size_t)nflat))) return rc;
        h->nflat = nflat;
    }
    const int64_t bidx = row0 / batch;
    MCK(cudaMemcpyAsync(h->dBatchIdx, &bidx, sizeof(int64_t), cudaMemcpyHostToDevice, h->stream));
    MCK(cudaMemsetAsync(h->loss, 0, sizeof(float), h->stream));
    if ((rc = gather(h, h->perm, h->dBatchIdx)) || (rc = forward(h, true)) || (rc = loss_gradient(h)) ||
        (rc = backward(h, false)))
        return rc;
    const AdamAll a = adam_desc(h, batch, 0.f, nullptr, 1.f);
    k_grad_flat<<<(unsigned)((nflat + 255) / 256), 256, 0, h->stream>>>(a, h->gflat);
    MCK(cudaGetLastError());
    float out[2];                        // the loss and the error flag
    MCK(cudaMemcpyAsync(out, h->loss, sizeof out, cudaMemcpyDeviceToHost, h->stream));
    MCK(cudaStreamSynchronize(h->stream));
    int e;
    memcpy(&e, &out[1], sizeof e);
    if (e) return fail(BG_ETIMEOUT, "mlp: a tensor-core wait gave up");
    if (loss) *loss = out[0];
    if (grad) *grad = h->gflat;
    if (ngrad) *ngrad = nflat;
    return BG_OK;
}

BG_API int bg_mlp_apply_gradients(bg_mlp *h, const void *grad, float lr, float scale) {
    if (!h || !grad) return fail(BG_EINVAL, "mlp: no gradient");
    if (!h->gflat || h->B <= 0) return fail(BG_ESTATE, "mlp: no step gradients yet");
    MCK(cudaSetDevice(h->device));
    // Adam's step count t is the step being taken (1 for the first)
    MCK(launch_pdl(k_step_advance, dim3(1), dim3(1), 0, h->stream, h->dBatchIdx, h->dOptStep));
    int rc = adam_all(h, h->B, lr, (const float *)grad, scale);
    if (rc) return rc;
    MCK(cudaStreamSynchronize(h->stream));
    h->step += 1;
    return BG_OK;
}

// One forward + backward on the first `n` rows of the training set (no
// update), for gradient checks: loss, dW_l (summed) and db_l of every layer.
BG_API int bg_mlp_gradients(bg_mlp *h, int batch, float *loss, float *const *dW, float *const *db) {
    if (!h || batch < 128 || batch % 512 != 0 || h->nset < batch) return fail(BG_EINVAL, "mlp: bad gradient call");
    MCK(cudaSetDevice(h->device));
    int rc = ensure_batch(h, batch);
    if (rc) return rc;
    std::vector<int64_t> idx(batch);
    for (int i = 0; i < batch; ++i) idx[i] = i;
    MCK(cudaMemcpyAsync(h->idx, idx.data(), batch * sizeof(int64_t), cudaMemcpyHostToDevice, h->stream));
    MCK(cudaMemsetAsync(h->loss, 0, sizeof(float), h->stream));
    if ((rc = gather(h, h->idx, nullptr)) || (rc = forward(h, true)) || (rc = loss_gradient(h)) || (rc = backward(h, false)))
        return rc;
    const int splits = kSplits;
    for (int l = 3; l >= 0; --l) {
        const size_t n = (size_t)h->rows[l] * h->cols[l];
        std::vector<float> part((size_t)splits * n);
        MCK(cudaMemcpyAsync(part.data(), h->gWl[l], part.size() * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
        MCK(cudaStreamSynchronize(h->stream));
        if (dW && dW[l])
            for (size_t i = 0; i < n; ++i) {
                float s = 0;
                for (int z = 0; z < splits; ++z) s += part[(size_t)z * n + i];
                dW[l][i] = s;
            }
        if (db && db[l]) {
            // the bias gradient: fixed-order sum of the column-sum partials
            const float *bp;
            int nblk, ld;
            bias_partials(h, l, batch, &bp, &nblk, &ld);
            std::vector<float> cp((size_t)nblk * ld);
            MCK(cudaMemcpy(cp.data(), bp, cp.size() * sizeof(float), cudaMemcpyDeviceToHost));
            for (int r = 0; r < h->rows[l]; ++r) {
                float s = 0;
                for (int z = 0; z < nblk; ++z) s += r < ld ? cp[(size_t)z * ld + r] : 0.f;
                db[l][r] = s;
            }
        }
    }
    if (loss) MCK(cudaMemcpy(loss, h->loss, sizeof(float), cudaMemcpyDeviceToHost));
    MCK(cudaStreamSynchronize(h->stream));
    return check_err(h);
}

// Plain GEMM on device buffers: C[M][N] = A[M][K] . B[N][K]^T (bf16 in,
// fp32 out), K a multiple of 64.  k_gemm_p (or k_gemm where no tensor map is
// allowed) serves this entry point alone: the network's layers are chains.
BG_API int bg_gemm_bf16(int64_t M, int64_t N, int64_t K, const void *A, const void *B, float *C, void *stream) {
    if (M <= 0 || N <= 0 || K <= 0 || K % 64 != 0 || !A || !B || !C) return fail(BG_EINVAL, "gemm: bad shape");
    // the error flag of the tensor-core waits: one per device, kept for the process
    static int *flags[64] = {nullptr};
    int dev = 0;
    MCK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(BG_EINVAL, "gemm: device index");
    if (!flags[dev]) MCK(cudaMalloc((void **)&flags[dev], sizeof(int)));
    int *err = flags[dev];
    cudaStream_t st = (cudaStream_t)stream;
    MCK(cudaMemsetAsync(err, 0, sizeof(int), st));
    umma::GemmArgs g = gemm_args((const bf16 *)A, (int)K, (const bf16 *)B, (int)K, (int)M, (int)N, (int)K, err);
    g.C = C;
    g.ldc = (int)N;
    int rc = launch_gemm<128>(g, 1, device_of(dev), st);
    cudaError_t e = cudaStreamSynchronize(st);
    int ev = 0;
    cudaMemcpy(&ev, err, sizeof(int), cudaMemcpyDeviceToHost);
    if (rc) return rc;
    if (e != cudaSuccess) return fail(BG_ECUDA, std::string("gemm: ") + cudaGetErrorString(e));
    if (ev) return fail(BG_ETIMEOUT, "gemm: a tensor-core wait gave up");
    return BG_OK;
}

}  // extern "C"
