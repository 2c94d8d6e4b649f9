// bg_stdplazy.cuh -- STDP on a dense connection with the postsynaptic updates
// applied when a weight is next needed.
//
// The rule changes w[i,j] (+)= A_pre[i] at every spike of target j and
// w[i,j] (+)= A_post[j] at every spike of source i, each followed by the clip
// (stdp.py:395-408).  A weight is only read when its source spikes, so its
// postsynaptic updates can wait: per step the targets' spikes are kept as one
// bit per column and the sources' traces as one value per row, for up to
// kLazySteps steps.  When source i spikes its row takes the pending updates
// -- the same additions, in the same order, each rounded and clipped -- before
// it is propagated; and every 32 steps, and at the end of a run, one pass
// over the matrix applies what is pending everywhere (k_stdp_flush).  Results
// are those of updating every step, bit for bit (the sign of a zero and special
// values included: lazy_update).
//
// Updating every step moved the whole matrix each way every step once about
// half of the targets spike (10 000 x 4096: 328 MB, 52.7 us, at 0.95 of the
// measured memory rate; with the other kernels 73 us a step).  The pass every
// 32 steps moves it once; it is bound by the updates' arithmetic (20 M a step:
// an integer pipe at 0.76 and the conversion pipe at 0.37 of their peaks at
// 303 us a pass, before the clip became a minimum and a maximum and the sign
// was taken out: 400 -> 303 -> 203 us).  A step of that network takes
// 26 us, of which the pass is a quarter and the three launches' latency the
// rest; 2000 x 1000: 23 -> 18 us, 1000 x 64: 19 -> 16 us.
//
// Everything else of a step of the rule -- trace decay, propagation, the
// presynaptic update, the targets' trace jump -- needs one row or one column
// at a time, so it is one launch (k_stdp_step) where it was three.
#pragma once
#include "bg_kernels.cuh"

namespace bg {

constexpr int kLazySteps = 64;         // pending steps the masks and the trace records hold
constexpr int kLazyCols = 32;          // columns of a k_stdp_step block (one per lane)
constexpr int kLazyThreads = 1024;     // and 32 rows at a time (one per warp)
constexpr int kLazyList = 2048;        // spiking rows listed at a time
constexpr int kFlushThreads = 256;
constexpr int kFlushRows = 8;

struct LazyCtl { long long base; int win; unsigned int done; };   // first pending step, mask buffer in use

template <typename T> struct StdpStepArgs {
    DevCtl *ctl; LazyCtl *lz;
    // sources' and targets' spike histories
    const uint32_t *hist; int depth; int64_t nwords; int delay; int64_t so, sn;
    const uint32_t *thist; int tdepth; int64_t tnwords; int post_delay; int64_t to, tn;
    T *sv; const T *mod; void *w;
    double *A_pre, *A_post; double a_pre, c_pre, a_post, c_post, Ap, Am; int pre_set, post_set;
    double wmin, wmax, wx; int pre_mode, post_mode;
    double *rec;                            // [sn][kLazySteps]: A_pre at the end of the pending steps
    unsigned long long *rowmask, *colmask;  // [2][sn], [2][tn]: pending steps in which row / column spiked
    unsigned long long *events;
    int last;
};

// One postsynaptic update of a weight, as stdp_w_val.  FAST (additive, FP32
// weights, bounds 0 <= lo <= hi with lo finite and not -0): the weight's bits
// placed in a double are w * 2^-896 exactly (zeros and subnormals too), so one
// FMA gives w + add with the one rounding of the double sum, where widening w
// takes a conversion on a pipe a quarter as wide as the FP64 one; the clip is a
// minimum and a maximum.  Both hold for weights in [+0, 2^120) and
// lazy_plain_add only:
//  - a weight with its sign bit set (-0 among them), infinite or NaN is another
//    number in that place;
//  - a NaN sum would leave a minimum and maximum as a bound, where the
//    comparisons of stdp_w_val keep it; weights below 2^120 and additions of at
//    most 2^100 make no infinity in kLazySteps additions either;
//  - a sum that rounds to -0 would leave them as +0.  A weight >= 0 gets there
//    by a negative addition of at most 2^-96 only: past that it must cancel a
//    weight above 2^-97, and the sum is then a multiple of 2^-148, which is 0
//    (+0) or too large to round to zero.
template <typename WT, bool FAST>
__device__ __forceinline__ WT lazy_update(WT w, double add, float flo, float fhi, double wmin, double wmax, int mode, double wx) {
    if constexpr (FAST && sizeof(WT) == 4) {
        const uint32_t u = __float_as_uint((float)w);
        const double d = __hiloint2double((int)(u >> 3), (int)(u << 29));
        return (WT)fminf(fmaxf(__double2float_rn(__fma_rn(d, 0x1p896, add)), flo), fhi);
    } else {
        return stdp_w_val<WT>(w, add, wmin, wmax, mode, wx);
    }
}
__device__ __forceinline__ bool lazy_plain_add(double add) {
    const double m = fabs(add);
    return m <= 0x1p100 && !(__double2hiint(add) < 0 && m <= 0x1p-96);
}

__device__ __forceinline__ bool spike_bit(const uint32_t *H, int64_t i) { return (H[i >> 5] >> (i & 31)) & 1u; }

template <typename T, typename WT>
__global__ void __launch_bounds__(kLazyThreads) k_stdp_step(const StdpStepArgs<T> a) {
    __shared__ int32_t list[kLazyList];
    __shared__ int wsum[33];
    __shared__ double tr[32][kLazySteps];      // trace records of the rows at hand
    __shared__ T wsm[32][kLazyCols + 1];       // their weights as propagated
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long t = a.ctl->nstep;
    const int n = (int)(t - a.lz->base);       // pending steps before this one, < kLazySteps
    const int win = a.lz->win;
    const unsigned long long before = (1ull << n) - 1ull;
    unsigned long long *rowmask = a.rowmask + (int64_t)win * a.sn, *colmask = a.colmask + (int64_t)win * a.tn;
    const bool on = t >= a.delay;
    const uint32_t *H = a.hist + (int64_t)(on ? (int)((t - a.delay) % a.depth) : 0) * a.nwords;
    // ---- the sources' traces: decay, the jump of those that spike, the record.
    // (Other blocks may read rowmask meanwhile: they look at earlier bits only.)
    for (int64_t i = (int64_t)blockIdx.x * kLazyThreads + tid; i < a.sn; i += (int64_t)gridDim.x * kLazyThreads) {
        double x = __dadd_rn(__dmul_rn(a.a_pre, a.A_pre[i]), a.c_pre);
        if (on && spike_bit(H, a.so + i)) {
            x = a.pre_set ? a.Ap : __dadd_rn(x, a.Ap);
            atomicOr(rowmask + i, 1ull << n);
        }
        a.A_pre[i] = x;
        a.rec[i * kLazySteps + n] = x;
    }
    // ---- this block's columns
    const int64_t j = (int64_t)blockIdx.x * kLazyCols + lane;
    const bool act = j < a.tn;
    const unsigned long long cm = act ? colmask[j] : 0ull;
    double ap = act ? __dadd_rn(__dmul_rn(a.a_post, a.A_post[j]), a.c_post) : 0.0;
    T acc = act && warp == 0 ? a.sv[j] : T(0);
    const float flo = __double2float_rn(a.wmin), fhi = __double2float_rn(a.wmax);
    WT *W = (WT *)a.w;
    long long nspk = 0;
    if (on) {
        const int64_t end = a.so + a.sn, w0 = a.so >> 5, w1 = (end + 31) >> 5;
        for (int64_t cw = w0; cw < w1; cw += kLazyThreads) {
            const int64_t wi = cw + tid;
            const uint32_t word = wi < w1 ? masked_word(H, wi, a.so, end) : 0u;
            int incl = __popc(word);
            const int pc = incl;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
            if (lane == 31) wsum[warp] = incl;
            __syncthreads();
            if (warp == 0) {
                const int v0 = wsum[lane];
                int v = v0;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) { const int x = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += x; }
                wsum[lane] = v - v0;
                if (lane == 31) wsum[32] = v;
            }
            __syncthreads();
            const int total = wsum[32], off = wsum[warp] + incl - pc;
            nspk += total;
            for (int b0 = 0; b0 < total; b0 += kLazyList) {
                uint32_t wd = word;
                int o = off - b0;
                while (wd) {
                    const int b = __ffs(wd) - 1;
                    wd &= wd - 1;
                    if (o >= 0 && o < kLazyList) list[o] = (int32_t)(((wi << 5) + b) - a.so);
                    ++o;
                }
                __syncthreads();
                const int cnt = min(kLazyList, total - b0);
                for (int r0 = 0; r0 < cnt; r0 += 32) {
                    // ---- warp r takes row r0 + r: its pending updates, its
                    // weights for the propagation, the presynaptic update
                    if (r0 + warp < cnt) {
                        const int64_t i = list[r0 + warp];
                        const unsigned long long rm = *(volatile unsigned long long *)(rowmask + i) & before;
                        const int lo = rm ? 63 - __clzll((long long)rm) : 0;   // the row is current up to step lo
                        if (lane >= lo && lane < n) tr[warp][lane] = a.rec[i * kLazySteps + lane];
                        if (lane + 32 >= lo && lane + 32 < n) tr[warp][lane + 32] = a.rec[i * kLazySteps + lane + 32];
                        WT w = act ? W[i * a.tn + j] : WT(0);
                        __syncwarp();
                        unsigned long long m = cm & before & ~((1ull << lo) - 1ull);
                        while (m) {
                            const int s = __ffsll((long long)m) - 1;
                            m &= m - 1;
                            w = stdp_w_val<WT>(w, tr[warp][s], a.wmin, a.wmax, a.post_mode, a.wx);
                        }
                        if (act) {
                            T wv = (T)w;
                            if (a.mod) wv = rn<T>::mul(wv, a.mod[i]);
                            wsm[warp][lane] = wv;
                            W[i * a.tn + j] = stdp_w_val<WT>(w, ap, a.wmin, a.wmax, a.pre_mode, a.wx);
                        }
                    }
                    __syncthreads();
                    // ---- propagation, rows ascending (connection.py:256-262)
                    if (warp == 0) {
                        const int rows = min(32, cnt - r0);
                        for (int r = 0; r < rows; ++r) acc = rn<T>::add(acc, wsm[r][lane]);
                    }
                    __syncthreads();
                }
            }
            __syncthreads();
        }
    }
    // every warp has read the columns' masks and traces
    __syncthreads();
    if (warp == 0 && act) {
        if (nspk) a.sv[j] = acc;
        if (t >= a.post_delay && spike_bit(a.thist + (int64_t)((int)((t - a.post_delay) % a.tdepth)) * a.tnwords, a.to + j)) {
            ap = a.post_set ? a.Am : __dadd_rn(ap, a.Am);
            colmask[j] = cm | (1ull << n);
        }
        a.A_post[j] = ap;
    }
    if (blockIdx.x == 0 && tid == 0 && nspk && a.events) atomicAdd(a.events, (unsigned long long)nspk * (unsigned long long)a.tn);
    bg_finish_step(a.ctl, a.last);
}

struct StdpFlushArgs {
    DevCtl *ctl; LazyCtl *lz;
    int64_t sn, tn; void *w;
    double wmin, wmax, wx; int mode;
    const double *rec;
    unsigned long long *rowmask, *colmask;
};

// Applies every pending update to the whole matrix.  A block takes bands of
// kFlushRows rows: their trace records go to shared memory, with -0 for the
// steps a row has taken already (w + -0 is w, and such a row was clipped by its
// presynaptic update since; the instance for the other rules skips them), then a
// thread takes one column of the band at a time and walks the column's spikes,
// all rows of the band side by side.  Warps whose 32 columns have no spikes skip
// them.
template <typename WT, bool FAST>
__global__ void __launch_bounds__(kFlushThreads) k_stdp_flush(const StdpFlushArgs a) {
    __shared__ double tab[kFlushRows][kLazySteps];
    __shared__ int from[kFlushRows];               // first step a row has not taken (not FAST)
    const int tid = threadIdx.x;
    const int n = (int)(a.ctl->nstep - a.lz->base), win = a.lz->win;
    const unsigned long long *rowmask = a.rowmask + (int64_t)win * a.sn, *colmask = a.colmask + (int64_t)win * a.tn;
    const float flo = __double2float_rn(a.wmin), fhi = __double2float_rn(a.wmax);
    WT *W = (WT *)a.w;
    // the other buffers of the masks start the next window empty
    for (int64_t k = (int64_t)blockIdx.x * kFlushThreads + tid; k < a.sn; k += (int64_t)gridDim.x * kFlushThreads)
        a.rowmask[(int64_t)(win ^ 1) * a.sn + k] = 0ull;
    for (int64_t k = (int64_t)blockIdx.x * kFlushThreads + tid; k < a.tn; k += (int64_t)gridDim.x * kFlushThreads)
        a.colmask[(int64_t)(win ^ 1) * a.tn + k] = 0ull;
    const int64_t nb = n > 0 ? (a.sn + kFlushRows - 1) / kFlushRows : 0;
    for (int64_t b = blockIdx.x; b < nb; b += gridDim.x) {
        const int64_t i0 = b * kFlushRows;
        const int rows = (int)min((int64_t)kFlushRows, a.sn - i0);
        int fits = 1;                              // the band's additions keep the fast form exact
        for (int k = tid; k < kFlushRows * kLazySteps; k += kFlushThreads) {
            const int r = k / kLazySteps, s = k % kLazySteps;
            double x = -0.0;
            if (r < rows && s < n) {
                const unsigned long long rm = rowmask[i0 + r];
                const int lo = rm ? 63 - __clzll((long long)rm) : 0;
                if (!FAST && s == 0) from[r] = lo;
                if (s >= lo) { x = a.rec[(i0 + r) * kLazySteps + s]; fits &= lazy_plain_add(x); }
            }
            tab[r][s] = x;
        }
        const bool band = __syncthreads_and(fits) != 0;
        for (int64_t c0 = 0; c0 < a.tn; c0 += kFlushThreads) {
            const int64_t j = c0 + tid;
            unsigned long long m = j < a.tn ? colmask[j] : 0ull;
            if (!__any_sync(0xffffffffu, m != 0ull)) continue;
            if (!m) continue;
            WT w[kFlushRows];
            bool plain = FAST && band;
            int signs = 0;                         // (one unsigned comparison a row made a pass after one step 13 us longer)
#pragma unroll
            for (int r = 0; r < kFlushRows; ++r) {
                w[r] = r < rows ? W[(i0 + r) * a.tn + j] : WT(0);
                plain = plain && w[r] < WT(0x1p120);
                signs |= __float_as_int((float)w[r]);
            }
            if (plain && signs >= 0) {
                do {
                    const int s = __ffsll((long long)m) - 1;
                    m &= m - 1;
#pragma unroll
                    for (int r = 0; r < kFlushRows; ++r)
                        w[r] = lazy_update<WT, FAST>(w[r], tab[r][s], flo, fhi, a.wmin, a.wmax, a.mode, a.wx);
                } while (m);
            } else {
                do {
                    const int s = __ffsll((long long)m) - 1;
                    m &= m - 1;
#pragma unroll
                    for (int r = 0; r < kFlushRows; ++r)
                        if (FAST || s >= from[r]) w[r] = lazy_update<WT, false>(w[r], tab[r][s], flo, fhi, a.wmin, a.wmax, a.mode, a.wx);
                } while (m);
            }
#pragma unroll
            for (int r = 0; r < kFlushRows; ++r)
                if (r < rows) W[(i0 + r) * a.tn + j] = w[r];
        }
        __syncthreads();
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&a.lz->done, 1u) == gridDim.x - 1) {
            // every block has read base and win
            a.lz->done = 0;
            a.lz->base = a.ctl->nstep;
            a.lz->win = win ^ 1;
            __threadfence();
        }
    }
}

}  // namespace bg
