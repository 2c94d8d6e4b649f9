// bg_synpersist.cuh -- one cooperative launch runs many steps of a single
// linear group whose Synapses (event path, static variables, one additive
// presynaptic statement each, one common target range) connect it to
// itself: CUBA through Synapses.
//
// Block b owns neurons [1024 b, 1024 b + 1024) for the whole launch, state in
// registers (512 threads, neurons tid and tid + 512), and bin b: the events
// of every object that reach those neurons, in a ring of dmax + 2 slots by the
// step that applies them.  A step t is
//   A: update + threshold; the block's spike words into the history (and the
//      monitor words); kSPParts warps per spike and object take all the source's
//      synapses, whatever their delay, and put each event -- a key in the
//      pull's order (target, object, delay descending, source, rank) and the
//      statement's term, read as one 16-byte record by source -- into the bin
//      of its target in slot t + d;
//   arrive at step t (release), wait for every block's arrival (acquire);
//   C: bin b of slot t applied to the registers in key order -- the additions
//      of the pull, in its order -- and emptied; the resets of step t;
//      StateMonitors ('end').
// One wait per step: a block in A(t+2) has passed the wait of step t+1, so every
// block has finished C(t), where it empties its bin of slot t, which A(t+2) may
// push into again.  A bin that more events reached than it holds is delivered by
// the pull's test for its targets, object by object.  The ring outlives a launch; after a
// reinit, a loaded state or changed terms it is filled again from the spike
// history (k_synp_refill).  Every wait is bounded; on timeout the block raises
// BG_DERR_TIMEOUT and leaves the loop.
//
// What bounds it: the chain of a step's dependent round trips (record, bin
// slot, store, arrival, count and entries).  Pushing a spike's events for all
// delays at once reads its row once and coalesced, by the block that found it;
// walking the spike lists of every past step and each delay's part of the rows
// again, dealt over the blocks, took two more round trips (list entry, delay
// offsets) and gathered records one by one: 12.3 -> 5.4 us a step at 32768
// neurons of in-degree 160.  Ordering a target's few events where they arrive
// (kSPTab each) leaves the counting sort to the busy bins.
#pragma once
#include "bg_persist.cuh"

namespace bg {

constexpr int kSPTh = kSynBinThreads;            // threads per block
constexpr int kSPNpt = kSynTPT;                  // neurons per thread
constexpr int kSPBn = kSPTh * kSPNpt;            // neurons per block
static_assert(kSPBn == kSynBin, "a block's neurons are one bin of targets");
constexpr int kSPTab = kSynBinCap / kSPBn;       // events of one target ordered without a sort
constexpr int kSPParts = 4;                      // warps per source: a few records a lane, loaded at once
constexpr int64_t kSPRing = (int64_t)2 << 30;    // bytes of the ring of bins; kSynBinCap entries a bin if that fits

// One synapse, rows by source.  x: target within its bin (10 bits), object (2),
// 255 - delay (8), the target's bin (24; the source takes its place in an
// event's key), place in the source's row (20).  y: the statement's term.
using SynRec = ulonglong2;

struct SynPersistObj {
    SynEvArgs e;                                 // rows by source, pull columns, terms
    const SynRec *rec;                           // [nsyn] by source
    int var, sub;                                // the statement: var += term (sub: var -= term)
};

struct SynPersistArgs {
    DevCtl *ctl;
    double *S; int64_t n, npad;
    double A[kMaxVars * kMaxVars]; double C[kMaxVars];
    uint64_t anz; uint32_t cnz;
    int thr_kind, thr_var, thr_var2; double thr_val;
    int reset_kind, reset_var, reset_var2; double reset_val;
    uint32_t *hist; int depth; int64_t nwords;
    int nobj; SynPersistObj o[kSynEvMerge];
    // the objects' common bins: [ring][nbins], [ring][nbins][cap]
    int *bin_cnt; SynRec *bin_ev; int ring, cap;
    int nbins, blk0; int64_t tn;                 // bin 0 is block blk0's; targets of the range
    unsigned long long *spikes;
    unsigned int *arrived;                       // [4] arrivals per step mod 4 (zeroed before the launch)
    int nsteps;
    uint32_t *mon_words; int64_t mon_stride;     // spike monitors: the words of each step of the launch
    unsigned int spin_limit;
    int hold_block;                              // test hook: this block never publishes its arrivals (-1: none)
    int nrec; RecDev rec[kMaxRec];               // StateMonitors; blk_lo holds this kernel's block ranges
};

// the events of source i (relative to the object's range) of step slot `now`
// (step mod ring) into the bins: of records [r0, r1), every `stride`-th from the
// lane's own on, four at a time (loads, then slots, then stores); only those of
// delay dmin or more
__device__ __forceinline__ void synp_push(const SynPersistArgs &a, const SynRec *rec, int64_t i, int64_t r0, int64_t r1, int now,
                                          int lane, int stride, int dmin) {
    for (int64_t p0 = r0 + lane; p0 < r1; p0 += 4 * stride) {
        SynRec v[4];
        int at[4], slot[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            at[u] = -1;
            if (p0 + u * stride < r1) v[u] = __ldg(rec + p0 + u * stride);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (p0 + u * stride < r1) {
                const int d = 255 - (int)((v[u].x >> 44) & 255u);
                if (d < dmin) continue;
                int row = now + d;
                row -= row >= a.ring ? a.ring : 0;
                at[u] = row * a.nbins + (int)((v[u].x >> 20) & 0xffffffu);
                slot[u] = atomicAdd(a.bin_cnt + at[u], 1);
            }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (at[u] < 0) continue;
            if (slot[u] >= a.cap) continue;              // (the count tells)
            v[u].x = (v[u].x & ~(0xffffffull << 20)) | ((unsigned long long)i << 20);
            __stcg(a.bin_ev + (int64_t)at[u] * a.cap + slot[u], v[u]);
        }
    }
}

// the records of an object's synapses (a warp per source)
static __global__ void __launch_bounds__(256) k_synp_records(const SynEvArgs e, int k, SynRec *rec) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t i = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); i < e.sn; i += nw) {
        const int64_t r0 = e.srcptr[i], r1 = e.srcptr[i + 1];
        for (int64_t p = r0 + lane; p < r1; p += 32) {
            const unsigned long long j = (unsigned long long)e.stgt[p];
            SynRec v;
            v.x = ((j % kSynBin) << 54) | ((unsigned long long)k << 52) | ((unsigned long long)(255 - e.sd[p]) << 44) |
                  ((j / kSynBin) << 20) | (unsigned long long)(p - r0);
            v.y = (unsigned long long)__double_as_longlong(e.term[e.sq[p]]);
            rec[p] = v;
        }
    }
}

// the (emptied) ring filled with the events still to come of the spikes in the
// history: blocks of one object's (step back, word) pairs, a warp per pair
static __global__ void __launch_bounds__(256) k_synp_refill(const __grid_constant__ SynPersistArgs a, int k) {
    const SynEvArgs &e = a.o[k].e;
    const long long nstep = a.ctl->nstep;
    const int lane = threadIdx.x & 31;
    const int64_t w0 = e.so >> 5, nw = ((e.so + e.sn + 31) >> 5) - w0;
    for (int64_t x = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); x < nw * e.dmax;
         x += (int64_t)gridDim.x * (blockDim.x / 32)) {
        const int back = 1 + (int)(x / nw);
        const int64_t wi = w0 + x % nw;
        if (nstep < back) continue;
        uint32_t word = masked_word(a.hist + (int64_t)(((int)nstep - back) % a.depth) * a.nwords, wi, e.so, e.so + e.sn);
        for (; word; word &= word - 1) {
            const int64_t i = (wi << 5) + (__ffs(word) - 1) - e.so;
            synp_push(a, a.o[k].rec, i, e.srcptr[i], e.srcptr[i + 1], (int)((nstep - back) % a.ring), lane, 32, back);
        }
    }
}

template <int NV>
__device__ __forceinline__ void synp_apply(const SynPersistArgs &a, double (&s)[kSPNpt][NV], int u, int k, double t) {
    const int v = a.o[k].var;
    const bool sub = a.o[k].sub != 0;
#pragma unroll
    for (int uu = 0; uu < kSPNpt; ++uu)
        if (uu == u) uset<double, NV>(s[uu], v, sub ? __dsub_rn(uget<double, NV>(s[uu], v), t) : __dadd_rn(uget<double, NV>(s[uu], v), t));
}

// C(t) for this block's bin (block-uniform call; synchronises).  tcnt is zero
// and `over` false at entry, and again on return.
template <int NV>
__device__ __forceinline__ void synp_bins(const SynPersistArgs &a, long long t, int now,
                                          double (&s)[kSPNpt][NV], int (&tcnt)[kSynBin], int &over) {
    extern __shared__ __align__(16) unsigned char syn_smem[];
    SynRec *tab = reinterpret_cast<SynRec *>(syn_smem);                          // [kSPTab][kSPBn]
    unsigned long long *key = reinterpret_cast<unsigned long long *>(syn_smem);  // or the bin in order
    double *tv = reinterpret_cast<double *>(key + kSynBinCap);
    __shared__ int wsum[kSPTh / 32], maxc;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int bin = (int)blockIdx.x - a.blk0;
    if (bin < 0 || bin >= a.nbins) return;
    const int64_t jb = (int64_t)bin * kSynBin;
    int *cnt = a.bin_cnt + now * a.nbins + bin;
    const SynRec *gev = a.bin_ev + ((int64_t)now * a.nbins + bin) * a.cap;
    // the first kSPTh entries loaded beside the count (those beyond it unused)
    const SynRec e0 = __ldcg(gev + tid);
    const int n = __ldcg(cnt);
    if (n > a.cap) {
        // the pull's test for every target of the bin, object by object
        const int row0 = (int)t % a.depth;
#pragma unroll
        for (int u = 0; u < kSPNpt; ++u) {
            const int64_t j = jb + u * kSPTh + tid;
            if (j >= a.tn) continue;
            for (int k = 0; k < a.nobj; ++k) {
                const SynEvArgs &e = a.o[k].e;
                for (int64_t q = e.colptr[j]; q < e.colptr[j + 1]; ++q) {
                    const uint32_t wd = e.word[q];
                    const int lag = (int)(wd >> 24) - 1;
                    if (lag < 0 || t < lag) continue;
                    const int64_t src = e.so + (int64_t)(wd & 0xFFFFFFu);
                    int row = row0 - lag;
                    row += row < 0 ? a.depth : 0;
                    if (!((__ldcg(a.hist + (int64_t)row * a.nwords + (src >> 5)) >> (src & 31)) & 1u)) continue;
                    synp_apply<NV>(a, s, u, k, e.term[q]);
                }
            }
        }
    } else if (n > 0) {
        // each event beside the others of its target, in the order of arrival
        for (int e = tid; e < n; e += kSPTh) {
            const SynRec v = e == tid ? e0 : __ldcg(gev + e);
            const int j = (int)(v.x >> 54);
            const int pos = atomicAdd(&tcnt[j], 1);
            if (pos < kSPTab) tab[pos * kSPBn + j] = v;
            else over = 1;
        }
        __syncthreads();
        if (!over) {                                             // uniform
            // a target's few events by ascending key
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u) {
                const int j = u * kSPTh + tid, c = tcnt[j];
                if (!c) continue;
                tcnt[j] = 0;
                unsigned long long from = 0;
                for (int r = 0; r < c; ++r) {
                    SynRec best = tab[j];
                    bool have = best.x >= from;
                    for (int q = 1; q < c; ++q) {
                        const SynRec v = tab[q * kSPBn + j];
                        if (v.x >= from && (!have || v.x < best.x)) { best = v; have = true; }
                    }
                    synp_apply<NV>(a, s, u, (int)((best.x >> 52) & 3u), __longlong_as_double((long long)best.y));
                    from = best.x + 1;
                }
            }
        } else {
        if (tid == 0) maxc = 0;
        __syncthreads();
        int cu[kSPNpt], c = 0, cmax = 0;
#pragma unroll
        for (int u = 0; u < kSPNpt; ++u) { cu[u] = tcnt[u * kSPTh + tid]; c += cu[u]; cmax = max(cmax, cu[u]); }
        if (cmax) atomicMax(&maxc, cmax);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += v; }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            int v = lane < kSPTh / 32 ? wsum[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int x = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += x; }
            if (lane < kSPTh / 32) wsum[lane] = v;
        }
        __syncthreads();
        const int beg = (warp ? wsum[warp - 1] : 0) + incl - c;
        if (maxc <= kSynSegMax) {                                // uniform
            {
                int b = beg;
#pragma unroll
                for (int u = 0; u < kSPNpt; ++u) { tcnt[u * kSPTh + tid] = b; b += cu[u]; }
            }
            __syncthreads();
            for (int e = tid; e < n; e += kSPTh) {
                const SynRec v = e == tid ? e0 : __ldcg(gev + e);
                const int pos = atomicAdd(&tcnt[(int)(v.x >> 54)], 1);
                key[pos] = v.x;
                tv[pos] = __longlong_as_double((long long)v.y);
            }
            __syncthreads();
            int sb = beg;
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u) {
                const int cc = cu[u];
                if (cc) {
                    for (int v = sb + 1; v < sb + cc; ++v) {
                        const unsigned long long kk = key[v];
                        const double tt = tv[v];
                        int w = v - 1;
                        while (w >= sb && key[w] > kk) { key[w + 1] = key[w]; tv[w + 1] = tv[w]; --w; }
                        key[w + 1] = kk;
                        tv[w + 1] = tt;
                    }
                    for (int e = sb; e < sb + cc; ++e) synp_apply<NV>(a, s, u, (int)((key[e] >> 52) & 3u), tv[e]);
                }
                sb += cc;
            }
        } else {
            int m = 1;
            while (m < n) m <<= 1;
            for (int e = tid; e < m; e += kSPTh) {
                if (e < n) { const SynRec v = __ldcg(gev + e); key[e] = v.x; tv[e] = __longlong_as_double((long long)v.y); }
                else { key[e] = ~0ull; tv[e] = 0.0; }
            }
            __syncthreads();
            for (int k = 2; k <= m; k <<= 1) {
                for (int jj = k >> 1; jj > 0; jj >>= 1) {
                    for (int e = tid; e < m; e += kSPTh) {
                        const int o = e ^ jj;
                        if (o > e) {
                            const bool up = (e & k) == 0;
                            const unsigned long long ka = key[e], kb = key[o];
                            if ((ka > kb) == up) {
                                key[e] = kb; key[o] = ka;
                                const double x = tv[e]; tv[e] = tv[o]; tv[o] = x;
                            }
                        }
                    }
                    __syncthreads();
                }
            }
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u) {
                if (!cu[u]) continue;
                const unsigned long long want = (unsigned long long)(u * kSPTh + tid);
                int l = 0, h = n;
                while (l < h) { const int mm = (l + h) >> 1; if ((key[mm] >> 54) < want) l = mm + 1; else h = mm; }
                for (int e = l; e < n && (key[e] >> 54) == want; ++e)
                    synp_apply<NV>(a, s, u, (int)((key[e] >> 52) & 3u), tv[e]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kSPNpt; ++u) tcnt[u * kSPTh + tid] = 0;
        }
    }
    __syncthreads();                     // every thread has read the count; shared memory free
    // the slot takes pushes again in A(t+2) (delay dmax): the clear must stay before
    // this block's arrival of step t+1, which A(t+2) of every block has waited for
    if (tid == 0) { *cnt = 0; over = 0; }
}

template <int NV, bool DIAG>
__global__ void __launch_bounds__(kSPTh, 2) k_syn_persist(const __grid_constant__ SynPersistArgs a) {
    extern __shared__ __align__(16) unsigned char syn_smem[];
    // row starts of the block's neurons as sources, relative to the first one's
    uint32_t *rows = reinterpret_cast<uint32_t *>(syn_smem + (size_t)kSynBinCap * sizeof(SynRec));   // [nobj][kSPBn + 1]
    __shared__ int64_t row0[kSynEvMerge];
    __shared__ uint16_t fired[kSPBn];            // the step's spikes, and how many
    __shared__ int nfired;
    __shared__ int tcnt[kSynBin], over;          // synp_bins
    __shared__ int abort_flag;
    __shared__ double stash[kSPBn];              // StateMonitor values of the block's neurons
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int base = blockIdx.x * kSPBn;         // neuron counts < 2^31
    const int nvalid = (int)min((int64_t)kSPBn, a.n - (int64_t)base);
    const unsigned int G = gridDim.x;
    const long long t0 = a.ctl->nstep;          // step counters are below 2^31 (checked by the host)
    if (tid == 0) { abort_flag = 0; nfired = 0; over = 0; }
#pragma unroll
    for (int u = 0; u < kSPNpt; ++u) tcnt[u * kSPTh + tid] = 0;
    for (int k = 0; k < a.nobj; ++k) {
        const SynEvArgs &e = a.o[k].e;
        auto start = [&](int64_t li) {           // (neurons outside the object's sources have empty rows)
            const int64_t i = (int64_t)base + li - e.so;
            return e.srcptr[i < 0 ? 0 : (i > e.sn ? e.sn : i)];
        };
        const int64_t r0 = start(0);
        if (tid == 0) row0[k] = r0;
        for (int li = tid; li <= kSPBn; li += kSPTh) rows[k * (kSPBn + 1) + li] = (uint32_t)(start(li) - r0);
    }
    int now = (int)(t0 % a.ring);                // the step's slot
    double s[kSPNpt][NV];
#pragma unroll
    for (int u = 0; u < kSPNpt; ++u) {
        const int li = u * kSPTh + tid;
#pragma unroll
        for (int k = 0; k < NV; ++k) s[u][k] = li < nvalid ? a.S[k * a.npad + base + li] : 0.0;
    }
    unsigned long long my_spikes = 0;
    __syncthreads();

    for (int st = 0; st < a.nsteps; ++st, now = now + 1 == a.ring ? 0 : now + 1) {
        const long long t = t0 + st;
        // ---- A(t): update (x = A s + C, the order of linear_row), threshold
        {
            double x[kSPNpt][NV];
            if constexpr (DIAG) {
#pragma unroll
                for (int u = 0; u < kSPNpt; ++u) {
                    double acc = 0.0;
#pragma unroll
                    for (int k = 0; k < NV; ++k) acc = __dadd_rn(acc, __dmul_rn(a.A[k], s[u][k]));
                    x[u][0] = acc;
#pragma unroll
                    for (int j = 1; j < NV; ++j) x[u][j] = __dadd_rn(0.0, __dmul_rn(a.A[j * NV + j], s[u][j]));
                }
                if (a.cnz & 1u) {
#pragma unroll
                    for (int u = 0; u < kSPNpt; ++u) x[u][0] = __dadd_rn(x[u][0], a.C[0]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < NV; ++j) {
#pragma unroll
                    for (int u = 0; u < kSPNpt; ++u) x[u][j] = 0.0;
#pragma unroll
                    for (int k = 0; k < NV; ++k)
                        if (a.anz & (1ull << (j * NV + k))) {
                            const double c = a.A[j * NV + k];
#pragma unroll
                            for (int u = 0; u < kSPNpt; ++u) x[u][j] = __dadd_rn(x[u][j], __dmul_rn(c, s[u][k]));
                        }
                    if (a.cnz & (1u << j)) {
#pragma unroll
                        for (int u = 0; u < kSPNpt; ++u) x[u][j] = __dadd_rn(x[u][j], a.C[j]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u)
#pragma unroll
                for (int j = 0; j < NV; ++j) s[u][j] = x[u][j];
        }
        unsigned int spk_bits = 0;
#pragma unroll
        for (int u = 0; u < kSPNpt; ++u) {
            const int li = u * kSPTh + tid;
            bool spk = false;
            if (a.thr_kind == 1) spk = uget<double, NV>(s[u], a.thr_var) > a.thr_val;
            else if (a.thr_kind == 2) spk = uget<double, NV>(s[u], a.thr_var) > uget<double, NV>(s[u], a.thr_var2);
            spk = spk && li < nvalid;
            spk_bits |= (spk ? 1u : 0u) << u;
            const uint32_t ball = __ballot_sync(0xffffffffu, spk);
            if (ball) {
                int at = 0;
                if (lane == 0) at = atomicAdd(&nfired, __popc(ball));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (spk) fired[at + __popc(ball & ((1u << lane) - 1u))] = (uint16_t)li;
            }
            if (lane == 0) {
                const int w = u * (kSPTh / 32) + warp;
                a.hist[(int64_t)((int)t % a.depth) * a.nwords + (base >> 5) + w] = ball;
                if (a.mon_words) a.mon_words[(int64_t)st * a.mon_stride + (base >> 5) + w] = ball;
                my_spikes += __popc(ball);
            }
        }
        __syncthreads();
        for (int q = warp; q < nfired * a.nobj * kSPParts; q += kSPTh / 32) {
            const int part = q % kSPParts, qo = q / kSPParts, k = qo % a.nobj, li = fired[qo / a.nobj];
            const uint32_t *rw = rows + k * (kSPBn + 1) + li;
            synp_push(a, a.o[k].rec, (int64_t)base + li - a.o[k].e.so, row0[k] + rw[0], row0[k] + rw[1], now, part * 32 + lane,
                      32 * kSPParts, 0);
        }
        // ---- arrive at step t; wait for every block's arrival
        __syncthreads();
        if (tid == 0) nfired = 0;
        if (tid == 0 && (int)blockIdx.x != a.hold_block) red_release_add(a.arrived + (st & 3), 1u);
        if (tid == 32) {
            const unsigned int *ctr = a.arrived + (st & 3);
            const unsigned int target = (unsigned int)((st >> 2) + 1) * G;
            unsigned int it = 0;
            while (ld_acquire_u32(ctr) < target) {
                if (++it > a.spin_limit) { abort_flag = 1; bg_raise(a.ctl, BG_DERR_TIMEOUT, t); break; }
                __nanosleep(32);
            }
        }
        __syncthreads();
        if (abort_flag) break;
        // ---- C(t): this block's bin, then the resets of step t
        synp_bins<NV>(a, t, now, s, tcnt, over);
        if (a.reset_kind == 1) {
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u)
                if ((spk_bits >> u) & 1u) uset<double, NV>(s[u], a.reset_var, a.reset_val);
        } else if (a.reset_kind) {
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u)
                if ((spk_bits >> u) & 1u) uset<double, NV>(s[u], a.reset_var, uget<double, NV>(s[u], a.reset_var2));
        }
        // StateMonitors ('end' slot, after the resets)
        for (int r = 0; r < a.nrec; ++r) {
            const RecDev &m = a.rec[r];
            const long long rel = t - m.start;
            if (rel < 0 || rel % m.timestep) continue;           // block-uniform
#pragma unroll
            for (int u = 0; u < kSPNpt; ++u) stash[u * kSPTh + tid] = uget<double, NV>(s[u], m.var);
            __syncthreads();
            const long long row = rel / m.timestep - *m.row_base;
            const int e0 = m.blk_lo[blockIdx.x], e1 = m.blk_lo[blockIdx.x + 1];
            for (int e = e0 + tid; e < e1; e += kSPTh) ((double *)m.buf)[row * m.nidx + m.pos[e]] = stash[m.idx[e] - base];
            __syncthreads();
        }
    }
#pragma unroll
    for (int u = 0; u < kSPNpt; ++u) {
        const int li = u * kSPTh + tid;
        if (li < nvalid) {
#pragma unroll
            for (int k = 0; k < NV; ++k) a.S[k * a.npad + base + li] = s[u][k];
        }
    }
    block_count(a.spikes, my_spikes);
}

}  // namespace bg
