// bg_cluster.cuh -- the persistent kernel of small networks: one thread-block
// cluster (or one block) holds the whole network, so a step needs no round
// trip through L2.
//
// The topology is bg_persist.cuh's (one group, shared-weight DelayConnections
// or zero-delay Connections onto itself), for groups of up to 16 blocks of
// 512 threads whose count rings fit in shared memory; the update, threshold
// and reset may also be a generated model's (head_body's policy M).
//
// Each block owns BN = 512 x NPT consecutive neurons: their state in
// registers, the count-ring columns of those neurons and the row starts of
// their outgoing synapses in its shared memory (for zero-delay networks the
// synapses themselves, 16 bits each, when they fit).  A step is
//   update -> threshold -> every warp pushes its own spikes straight into the
//   target's ring -> block barrier -> ring delivery, reset, StateMonitors.
// With one block the pushes are shared-memory atomics and that barrier is all.
//
// With several, a push is a red.async on the owner's shared memory that counts
// its bytes on the owner's mbarrier of the step, and a 17th warp, which owns
// no neurons, sends every block one arrival per step with the number of bytes
// pushed to it (arrive.expect_tx); a block's step is complete when all blocks
// arrived and all their bytes landed.  (red and a cluster barrier with release
// semantics take 900 cycles a step at 8 blocks, this 630: the release waits
// about 400 cycles in every warp, and the reductions are fenced before it.)
// With every delay at least one step the row delivered at step t holds pushes
// of steps <= t-1 only, so the block waits for step t-1 after its pushes of
// step t and the latency passes behind a step.
//
// Reuse of a ring row.  The arrivals are relaxed; after each one the 17th
// warp runs a cluster fence, so the arrival of step t+2 publishes everything
// the block did before its barrier of step t+1, its reads and clearing of the
// rows of step t among them, and the fence's latency passes beside the other
// warps' step.  A block pushes at step t' after waiting for all arrivals of
// step t'-1 (split: t'-2), so a row delivered at step t may be pushed to from
// step t+3 (split: t+4) on: a zero-delay ring has 3 rows, a delay ring at
// least dmax + 4.  A step's mbarrier (t mod 4) is used again four steps
// later, when every block has long passed the wait on it.
//
// Every wait is bounded, by polls and by time (a poll may suspend its warp for
// as long as the hardware sees fit).  A thread that gives up raises
// BG_DERR_TIMEOUT and has no more spikes, its block leaves the loop at the next
// block barrier, and the others follow as their waits run out.  Pushes of
// theirs may still be on their way then, so no block may leave the kernel on
// the cluster barrier alone: cluster_land waits until all of them have landed.
//
// What bounds it: the step's chain and the instructions of its 4 to 8 warps a
// scheduler.  Us per step, FP64, in-degree 80 without delays (n = 1000 / 4000
// / 16000 / 32000): 0.71 / 0.97 / 1.54 / 2.19, in-degree 200 with delays of 1
// to 50 steps (4000 / 10007 / 16384): 0.88 / 1.16 / 1.21; the persistent
// kernel, whose chain goes through L2 four times and a polled counter: 2.64 /
// 3.17 / 3.43 / 3.35 and 2.24 / 2.32 / 2.28.  4000 neurons of a generated
// conductance model: 1.24, on the stepped launches 14.  (The waits' time limit,
// since then, costs up to 1 % of a step.)
#pragma once
#include "bg_kernels.cuh"

namespace bg {

constexpr int kClusterThreads = 512;           // threads that own neurons
constexpr int kClusterMaxBlocks = 16;          // non-portable above 8
constexpr int kClusterMaxConn = 2;
// synapses into one block: a step's pushes stay below the 2^20 - 1 bytes an
// mbarrier's transaction count holds
constexpr int kClusterMaxInto = 262143;

template <typename T> struct ClusterConn {
    int so, sn, to, tn;                        // source and target ranges in the group
    int var, direct;                           // target variable; 1: Connection (w per event)
    int md, emd;                               // ring rows here, and of the engine's ring
    int tablen;                                // DelayConnection: entries of the k-fold sums
    int off_ring, off_rows, off_syn, off_tab;  // shared memory (bytes): ring, row starts, 16-bit synapses or -1, table or -1
    T w;                                       // the shared weight
    const T *table;
    const int64_t *rowptr; const uint32_t *packed;   // target | delay << 24 per synapse
    uint16_t *cring; int64_t tnp;              // DelayConnection: the engine's count ring, kept in shared memory for the launch
    unsigned long long *events;
};
template <typename T> struct ClusterArgs {
    DevCtl *ctl;
    T *S; int n; int64_t npad;
    T A[kMaxVars * kMaxVars]; T C[kMaxVars]; uint64_t anz; uint32_t cnz;
    int linear; double dt;
    int thr_kind, thr_var, thr_var2; T thr_val;
    int reset_kind, reset_var, reset_var2; T reset_val;
    int nconn; ClusterConn<T> conn[kClusterMaxConn];   // in delivery order: zero-delay Connections, then DelayConnections
    int split;                                 // every delay >= 1: a step waits for the step before it
    unsigned long long *spikes;
    int nsteps;
    unsigned int spin_limit;                   // polls, and microseconds, of a wait before it gives up
    int hold_block;                            // test hook: this block never publishes its arrivals (-1: none)
    uint32_t *mon_words; int mon_stride;       // spike words per step of the launch, or null
    int nrec; RecDev rec[kMaxRec]; int off_rec;   // StateMonitors; first entry of each neuron [nrec][BN + 1]
};

// the hardware cluster barrier, release/acquire
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t block) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(block));
    return r;
}
// *addr += v in a block's shared memory, counted as 4 bytes on its mbarrier
__device__ __forceinline__ void cluster_push(uint32_t addr, uint32_t v, uint32_t mbar) {
    asm volatile("red.async.relaxed.cluster.shared::cluster.mbarrier::complete_tx::bytes.add.u32 [%0], %1, [%2];"
                 :: "r"(addr), "r"(v), "r"(mbar) : "memory");
}
__device__ __forceinline__ void cluster_arrive_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" :: "r"(mbar), "r"(bytes) : "memory");
}
// the bytes without the arrival
__device__ __forceinline__ void cluster_expect_tx(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cluster.shared::cluster.b64 [%0], %1;" :: "r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool cluster_try(uint32_t mbar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                 " selp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// A thread's wait for a phase of an mbarrier; false when it gave up.  (The time
// is looked at every 64 polls of a loop that is not unrolled: a timed loop behind
// a few plain polls cost 4 to 6 % of a step.)
__device__ __forceinline__ bool cluster_wait(uint32_t mbar, uint32_t parity, unsigned int limit) {
    unsigned long long until = 0;
#pragma unroll 1
    for (unsigned int i = 0; i <= limit; ++i) {
        if (cluster_try(mbar, parity)) return true;
        if ((i & 63) == 63) {
            const unsigned long long t = global_ns();
            if (!until) until = t + 1000ull * limit;
            else if (t > until) return false;
        }
    }
    return false;
}

// After a wait has run out somewhere in the cluster, and a cluster barrier:
// called by one warp of every block, it returns when all pushes into the block
// have landed.  `count`: arrivals each block sent every block, by mbarrier.  Each
// push's bytes were announced, so a phase completes when its bytes have landed and
// its arrivals are there; the missing arrivals of the last, incomplete phase are
// made up here.
__device__ __forceinline__ void cluster_land(uint32_t mb0, uint32_t count, int blocks, int lane, unsigned int limit) {
    for (int i = 0; i < 4; ++i) {
        uint32_t sent = 0;
        if (lane < blocks)
            asm volatile("ld.relaxed.cluster.shared::cluster.u32 %0, [%1];" : "=r"(sent) : "r"(cluster_addr(count + 4 * i, lane)) : "memory");
        sent = __reduce_add_sync(0xffffffffu, sent);
        const uint32_t phases = (sent + blocks - 1) / blocks;
        if (lane == 0)
            for (uint32_t k = sent; k < phases * blocks; ++k)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(mb0 + 8 * i) : "memory");
        __syncwarp();
        if (phases) cluster_wait(mb0 + 8 * i, (phases - 1) & 1, limit);
        __syncwarp();
    }
}

// 1 << var where the compiler cannot see that one bit is set: a chain of tests
// on its bits stays a chain of uniform branches over the state registers,
// where one on the index is turned into an indexed access that puts the whole
// state into local memory.
__device__ __forceinline__ uint32_t one_hot(int var) {
    uint32_t m;
    asm volatile("shl.b32 %0, 1, %1;" : "=r"(m) : "r"(var));
    return m;
}
template <typename T, int NV>
__device__ __forceinline__ T pick_var(const T (&s)[NV], uint32_t mask) {
    T v = s[0];
#pragma unroll
    for (int k = 1; k < NV; ++k)
        if ((mask >> k) & 1u) v = s[k];
    return v;
}

// PAT, the delivered variable of connection d as a constant: 1: d + 1 (CUBA's
// ge and gi), 2: 1, 3: 0 (delta synapses), each with the built-in threshold
// and reset being constants on variable 0; 0: whatever the arguments say.  A
// step is bound by the instructions of its 4 to 8 warps per scheduler, and
// the general tests cost it half again as many.
template <int PAT> __device__ __forceinline__ constexpr int cluster_var(int d) { return PAT == 1 ? d + 1 : (PAT == 2 ? 1 : 0); }

template <typename T, int NV, int NPT, bool DIAG, bool MULTI, int PAT, class M>
__device__ __forceinline__ void cluster_body(const ClusterArgs<T> &a) {
    constexpr int TH = kClusterThreads, BN = TH * NPT;
    constexpr int SHIFT = NPT == 1 ? 9 : (NPT == 2 ? 10 : 11);
    static_assert(BN == 1 << SHIFT, "neurons per block");
    extern __shared__ __align__(16) unsigned char csm[];
    __shared__ __align__(8) unsigned long long mbars[4];     // arrivals and bytes of the steps t mod 4
    __shared__ uint32_t sent[2][kClusterMaxBlocks];          // pushes of this block to each block, steps t mod 2
    __shared__ uint32_t count[4];                            // arrivals sent to every block, by mbarrier
    __shared__ uint32_t failed;                              // a wait has run out in some block
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nth = blockDim.x;
    const int blocks = gridDim.x;                  // the grid is one cluster: block rank = block index
    const int base = blockIdx.x * BN;
    const int nvalid = max(0, min(BN, a.n - base));
    const long long t0 = a.ctl->nstep;
    const long long cs0 = t0 + a.ctl->clock_off;
    const uint32_t sm0 = (uint32_t)__cvta_generic_to_shared(csm);
    const uint32_t mb0 = (uint32_t)__cvta_generic_to_shared(mbars);
    if (MULTI) {
        if (tid == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(mb0 + 8 * i), "r"(blocks) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int k = tid; k < 2 * kClusterMaxBlocks; k += nth) sent[k / kClusterMaxBlocks][k % kClusterMaxBlocks] = 0;
        if (tid == 0) failed = 0;
    }
    // ---- staging: rings (row k: due at step t0 + k), row starts (relative to
    // the block's first), synapses, tables
    const uint32_t *syn0[kClusterMaxConn] = {nullptr, nullptr};   // the block's first synapse
    bool pact[kClusterMaxConn] = {false, false};   // the connection's sources meet this block
#pragma unroll
    for (int c = 0; c < kClusterMaxConn; ++c) {
        if (c >= a.nconn) break;
        const ClusterConn<T> &q = a.conn[c];
        pact[c] = q.so < base + nvalid && q.so + q.sn > base;
        const int lo = min(max(base - q.so, 0), q.sn), hi = min(max(base + BN - q.so, 0), q.sn);
        const int64_t r0 = q.rowptr[lo], r1 = q.rowptr[hi];
        syn0[c] = q.packed + r0;
        uint32_t *rows = reinterpret_cast<uint32_t *>(csm + q.off_rows);
        for (int j = tid; j <= BN; j += nth) {
            const int r = min(max(base + j - q.so, 0), q.sn);
            rows[j] = (uint32_t)(q.rowptr[r] - r0);
        }
        uint16_t *ring = reinterpret_cast<uint16_t *>(csm + q.off_ring);
        const int e0 = q.direct ? 0 : (int)(t0 % q.emd);
        for (int k = tid; k < q.md * BN; k += nth) {
            const int row = k >> SHIFT, i = base + (k & (BN - 1)) - q.to;   // target of this column
            uint16_t v = 0;
            if (!q.direct && row < q.emd && i >= 0 && i < q.tn) {
                const int er = e0 + row >= q.emd ? e0 + row - q.emd : e0 + row;
                v = q.cring[(int64_t)er * q.tnp + i];
            }
            ring[k] = v;
        }
        if (q.off_syn >= 0) {
            uint16_t *sy = reinterpret_cast<uint16_t *>(csm + q.off_syn);
            const int m = (int)(r1 - r0);
            for (int k = tid; k < m; k += nth) sy[k] = (uint16_t)(__ldg(syn0[c] + k) + (uint32_t)q.to);
        }
        if (q.off_tab >= 0) {
            T *tab = reinterpret_cast<T *>(csm + q.off_tab);
            for (int k = tid; k < q.tablen; k += nth) tab[k] = q.table[k];
        }
    }
    // StateMonitors: first entry (of the monitor's ascending indices) at or
    // past each neuron; steps until the next record, and its row
    int rnext[kMaxRec]; long long rrow[kMaxRec]; uint32_t rvar[kMaxRec];
#pragma unroll
    for (int r = 0; r < kMaxRec; ++r) {
        rnext[r] = 0; rrow[r] = 0; rvar[r] = 0;
        if (r >= a.nrec) continue;
        const RecDev &m = a.rec[r];
        rvar[r] = one_hot(m.var);
        int *first = reinterpret_cast<int *>(csm + a.off_rec) + r * (BN + 1);
        for (int j = tid; j <= BN; j += nth) {
            int lo = 0, hi = m.nidx;
            while (lo < hi) { const int mid = (lo + hi) >> 1; if (m.idx[mid] < base + j) lo = mid + 1; else hi = mid; }
            first[j] = lo;
        }
        const long long rel = t0 - m.start;
        rnext[r] = rel < 0 ? (int)-rel : (int)((m.timestep - rel % m.timestep) % m.timestep);
        rrow[r] = (rel + rnext[r]) / m.timestep - *m.row_base;
    }
    __syncthreads();
    if (MULTI) cluster_sync();                     // every block's rings and mbarriers are ready

    if (MULTI && warp == TH / 32) {
        // ---- the 17th warp: one arrival per block and step
        const bool held = (int)blockIdx.x == a.hold_block;
        int st = 0;
        uint32_t extra = 0;
        for (; st < a.nsteps; ++st) {
            const bool stop = __syncthreads_or(0);
            const uint32_t n = lane < blocks ? sent[st & 1][lane] : 0;
            // (a block that stops has pushed only where a thread's last wait did not run out)
            if (stop && !__any_sync(0xffffffffu, n != 0)) break;
            if (lane < blocks) {
                sent[st & 1][lane] = 0;            // next used at step st + 2, past the barrier of step st + 1
                const uint32_t mbar = cluster_addr(mb0 + 8 * (st & 3), lane);
                if (held) cluster_expect_tx(mbar, 4u * n);
                else cluster_arrive_tx(mbar, 4u * n);
            }
            __syncwarp();
            asm volatile("fence.acq_rel.cluster;" ::: "memory");
            if (stop) { extra = 1; break; }
        }
        if (lane < 4) count[lane] = held ? 0 : (uint32_t)(st + extra + 3 - lane) / 4;     // steps lane, lane + 4, ...
        __syncwarp();
        cluster_sync();
        if (failed) {                              // uniform over the cluster
            cluster_land(mb0, (uint32_t)__cvta_generic_to_shared(count), blocks, lane, a.spin_limit);
            __syncwarp();
            cluster_sync();                        // every block's counts are read
        }
        return;
    }

    T s[NPT][NV];
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
        const int li = u * TH + tid;
#pragma unroll
        for (int k = 0; k < NV; ++k) s[u][k] = li < nvalid ? a.S[k * a.npad + base + li] : T(0);
    }
    unsigned long long my_spikes = 0, my_events[kClusterMaxConn] = {0, 0};
    // per connection: row of the current step, as an index and as the address
    // of the thread's first column in it
    int cur[kClusterMaxConn] = {0, 0};
    uint32_t at[kClusterMaxConn] = {0, 0};
#pragma unroll
    for (int c = 0; c < kClusterMaxConn; ++c)
        if (c < a.nconn) at[c] = (uint32_t)a.conn[c].off_ring + 2u * tid;
    // PAT 0: delivered, threshold and reset variables, one bit each
    uint32_t dvar[kClusterMaxConn] = {0, 0}, thr1 = 0, thr2 = 0, rst1 = 0, rst2 = 0;
    if (PAT == 0) {
#pragma unroll
        for (int c = 0; c < kClusterMaxConn; ++c)
            if (c < a.nconn) dvar[c] = one_hot(a.conn[c].var);
        thr1 = one_hot(a.thr_var); thr2 = one_hot(a.thr_var2); rst1 = one_hot(a.reset_var); rst2 = one_hot(a.reset_var2);
    }
    // spike words of the thread's warp, written by its first lane
    uint32_t *mon = a.mon_words ? a.mon_words + ((base + warp * 32) >> 5) : nullptr;
    uint32_t monmask = 0;
#pragma unroll
    for (int u = 0; u < NPT; ++u)
        if (mon && lane == 0 && ((base + u * TH + warp * 32) >> 5) < a.mon_stride) monmask |= 1u << u;
    bool gave_up = false;
    int live = nvalid;                             // neurons that may spike: none once the thread has given up
    int st = 0;
    for (; st < a.nsteps; ++st) {
        const double tm = __dmul_rn((double)(cs0 + st), a.dt);   // time of the step (generated models)
        // ---- update and threshold
        if constexpr (M::custom_update) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) M::template update<T, NV>(s[u], tm);
        } else if (a.linear) {
            linear_update<T, NV, NPT, DIAG>(a.A, a.C, a.anz, a.cnz, s);
        }
        bool spk[NPT];
#pragma unroll
        for (int u = 0; u < NPT; ++u) spk[u] = false;
        if constexpr (M::custom_threshold) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) spk[u] = M::template threshold<T, NV>(s[u], tm);
        } else if (PAT) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) spk[u] = s[u][0] > a.thr_val;
        } else if (a.thr_kind == 1) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) spk[u] = pick_var<T, NV>(s[u], thr1) > a.thr_val;
        } else if (a.thr_kind == 2) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) spk[u] = pick_var<T, NV>(s[u], thr1) > pick_var<T, NV>(s[u], thr2);
        }
        // ---- the warp's spikes into the targets' rings (counts commute, so no order is needed)
        const uint32_t mbar = mb0 + 8 * (st & 3);
        uint32_t *snt = sent[st & 1];
        auto push = [&](uint32_t ring, uint32_t row, uint32_t tgt) {
            const uint32_t col = tgt & (BN - 1), at = ring + 2u * ((row << SHIFT) + (col & ~1u)), one = 1u << ((col & 1u) << 4);
            if (MULTI) {
                const uint32_t b = tgt >> SHIFT;
                atomicAdd(snt + b, 1u);
                cluster_push(cluster_addr(at, b), one, cluster_addr(mbar, b));
            } else {
                atomicAdd(reinterpret_cast<uint32_t *>(csm + (at - sm0)), one);
            }
        };
#pragma unroll
        for (int u = 0; u < NPT; ++u) {
            const int wb = u * TH + warp * 32;     // neuron of bit 0 within the block
            spk[u] = spk[u] && wb + lane < live;
            const uint32_t ball = __ballot_sync(0xffffffffu, spk[u]);
            if ((monmask >> u) & 1u) mon[u * (TH / 32)] = ball;
            if (!ball) continue;                   // warp-uniform
            if (lane == 0) my_spikes += __popc(ball);
#pragma unroll
            for (int c = 0; c < kClusterMaxConn; ++c) {
                if (c >= a.nconn) break;
                if (!pact[c]) continue;            // block-uniform
                const ClusterConn<T> &q = a.conn[c];
                const uint32_t *rows = reinterpret_cast<const uint32_t *>(csm + q.off_rows);
                const uint32_t ring = sm0 + (uint32_t)q.off_ring;
                uint32_t mask = ball;
                while (mask) {
                    const int j = wb + __ffs(mask) - 1;
                    mask &= mask - 1;
                    const uint32_t k0 = rows[j], k1 = rows[j + 1];
                    if (lane == 0) my_events[c] += k1 - k0;
                    if (q.off_syn >= 0) {
                        const uint16_t *sy = reinterpret_cast<const uint16_t *>(csm + q.off_syn);
                        for (uint32_t k = k0 + lane; k < k1; k += 32) push(ring, cur[c], sy[k]);
                    } else {
                        // from L2: eight synapses in flight per lane
                        for (uint32_t k = k0 + lane; k < k1; k += 256) {
                            uint32_t w8[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) w8[i] = k + 32 * i < k1 ? __ldg(syn0[c] + k + 32 * i) : 0xffffffffu;
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                if (w8[i] == 0xffffffffu) continue;
                                const int r = cur[c] + (int)(w8[i] >> 24);
                                push(ring, r >= q.md ? r - q.md : r, (w8[i] & 0xffffffu) + (uint32_t)q.to);
                            }
                        }
                    }
                }
            }
        }
        // ---- the rows due now are complete
        if (MULTI) {
            if (__syncthreads_or(gave_up)) break;  // uniform over the block
            if (!a.split) gave_up = !cluster_wait(mbar, (st >> 2) & 1, a.spin_limit);
            else if (st > 0) gave_up = !cluster_wait(mb0 + 8 * ((st - 1) & 3), ((st - 1) >> 2) & 1, a.spin_limit);
            if (gave_up) live = 0;
        } else {
            __syncthreads();
        }
        // ---- delivery in the reference's order, reset, StateMonitors
        if (mon) mon += a.mon_stride;
        int cnt[kClusterMaxConn][NPT];
#pragma unroll
        for (int d = 0; d < kClusterMaxConn; ++d) {
            if (d >= a.nconn) break;
            uint16_t *ring = reinterpret_cast<uint16_t *>(csm + at[d]);
#pragma unroll
            for (int u = 0; u < NPT; ++u) cnt[d][u] = ring[u * TH];
#pragma unroll
            for (int u = 0; u < NPT; ++u)
                if (cnt[d][u]) ring[u * TH] = 0;
            const bool wrap = cur[d] + 1 == a.conn[d].md;
            cur[d] = wrap ? 0 : cur[d] + 1;
            at[d] = wrap ? (uint32_t)a.conn[d].off_ring + 2u * tid : at[d] + 2u * BN;
        }
#pragma unroll
        for (int d = 0; d < kClusterMaxConn; ++d) {
            if (d >= a.nconn) break;
            const ClusterConn<T> &q = a.conn[d];
            // A DelayConnection adds its row's 0 where no event is due, too: that
            // makes +0 of a -0, which a linear update does not leave behind but a
            // generated one may.
            const int i0 = base + tid - q.to;
            if constexpr (PAT != 0) {
                constexpr int NVd = NV;
                const int k = cluster_var<PAT>(d);
                if (q.direct) {
                    // one event at most, nearly always: no branch on the lane's count
                    int most = 0;
#pragma unroll
                    for (int u = 0; u < NPT; ++u) {
                        const int n = cnt[d][u];
                        most = max(most, n);
                        const T x = rn<T>::add(s[u][k < NVd ? k : 0], q.w);
                        s[u][k < NVd ? k : 0] = n ? x : s[u][k < NVd ? k : 0];
                    }
                    if (__any_sync(0xffffffffu, most > 1)) {
#pragma unroll
                        for (int u = 0; u < NPT; ++u)
                            for (int i = 1; i < cnt[d][u]; ++i) s[u][k < NVd ? k : 0] = rn<T>::add(s[u][k < NVd ? k : 0], q.w);
                    }
                } else {
                    const T *tab = q.off_tab >= 0 ? reinterpret_cast<const T *>(csm + q.off_tab) : q.table;
#pragma unroll
                    for (int u = 0; u < NPT; ++u)
                        if (M::custom_update ? (unsigned)(i0 + u * TH) < (unsigned)q.tn : cnt[d][u] != 0)
                            s[u][k < NVd ? k : 0] = rn<T>::add(s[u][k < NVd ? k : 0], tab[cnt[d][u]]);
                }
            } else {
                const T *tab = q.off_tab >= 0 ? reinterpret_cast<const T *>(csm + q.off_tab) : q.table;
#pragma unroll
                for (int u = 0; u < NPT; ++u) {
                    const int n = cnt[d][u];
                    if (!n && !(M::custom_update && !q.direct && (unsigned)(i0 + u * TH) < (unsigned)q.tn)) continue;
                    T x = pick_var<T, NV>(s[u], dvar[d]);
                    if (q.direct) {
                        for (int i = 0; i < n; ++i) x = rn<T>::add(x, q.w);
                    } else {
                        x = rn<T>::add(x, tab[n]);
                    }
#pragma unroll
                    for (int k = 0; k < NV; ++k)
                        if ((dvar[d] >> k) & 1u) s[u][k] = x;
                }
            }
        }
        if (PAT && !M::custom_reset) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) s[u][0] = spk[u] ? a.reset_val : s[u][0];
        } else if (M::custom_reset || a.reset_kind) {
#pragma unroll
            for (int u = 0; u < NPT; ++u) {
                if (!spk[u]) continue;
                if constexpr (M::custom_reset) M::template reset<T, NV>(s[u], tm);
                else {
                    const T x = a.reset_kind == 1 ? a.reset_val : pick_var<T, NV>(s[u], rst2);
#pragma unroll
                    for (int k = 0; k < NV; ++k)
                        if ((rst1 >> k) & 1u) s[u][k] = x;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kMaxRec; ++r) {
            if (r >= a.nrec) break;
            if (rnext[r]) { --rnext[r]; continue; }        // uniform
            const RecDev &m = a.rec[r];
            rnext[r] = m.timestep - 1;
            const int *first = reinterpret_cast<const int *>(csm + a.off_rec) + r * (BN + 1);
#pragma unroll
            for (int u = 0; u < NPT; ++u) {
                const int li = u * TH + tid;
                for (int e = first[li]; e < first[li + 1]; ++e)
                    ((T *)m.buf)[rrow[r] * m.nidx + m.pos[e]] = pick_var<T, NV>(s[u], rvar[r]);
            }
            ++rrow[r];
        }
    }
    if (MULTI) {
        // the others' pushes of the last step have landed here; no block
        // leaves while another may still send to it
        if (a.split && !gave_up && st == a.nsteps && st > 0)
            gave_up = !cluster_wait(mb0 + 8 * ((st - 1) & 3), ((st - 1) >> 2) & 1, a.spin_limit);
        if (__any_sync(0xffffffffu, gave_up)) {
            bg_raise(a.ctl, BG_DERR_TIMEOUT, t0 + st);
            if (lane < blocks)
                asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;"
                             :: "r"(cluster_addr((uint32_t)__cvta_generic_to_shared(&failed), lane)), "r"(1u) : "memory");
        }
        __syncwarp();
        cluster_sync();
        if (failed) cluster_sync();                // (cluster_land, by the 17th warp)
    } else {
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < NPT; ++u) {
        const int li = u * TH + tid;
        if (li < nvalid) {
#pragma unroll
            for (int k = 0; k < NV; ++k) a.S[k * a.npad + base + li] = s[u][k];
        }
    }
#pragma unroll
    for (int c = 0; c < kClusterMaxConn; ++c) {
        if (c >= a.nconn) break;
        const ClusterConn<T> &q = a.conn[c];
        if (q.direct) continue;
        // due at step t0 + st + k: row (st + k) mod md here, (t0 + st + k) mod emd there
        const uint16_t *ring = reinterpret_cast<const uint16_t *>(csm + q.off_ring);
        const int e0 = (int)((t0 + st) % q.emd);
        for (int k = tid; k < q.emd * BN; k += TH) {
            const int row = k >> SHIFT, li = k & (BN - 1), i = base + li - q.to;
            if (i < 0 || i >= q.tn) continue;
            const int r = cur[c] + row >= q.md ? cur[c] + row - q.md : cur[c] + row;
            const int er = e0 + row >= q.emd ? e0 + row - q.emd : e0 + row;
            q.cring[(int64_t)er * q.tnp + i] = ring[(r << SHIFT) + li];
        }
    }
    if (lane == 0) {
        if (my_spikes) atomicAdd(a.spikes, my_spikes);
#pragma unroll
        for (int c = 0; c < kClusterMaxConn; ++c)
            if (c < a.nconn && my_events[c]) atomicAdd(a.conn[c].events, my_events[c]);
    }
}

template <typename T, int NV, int NPT, bool DIAG, bool MULTI, int PAT>
__global__ void __launch_bounds__(kClusterThreads + (MULTI ? 32 : 0), 1) k_cluster(const __grid_constant__ ClusterArgs<T> a) {
    cluster_body<T, NV, NPT, DIAG, MULTI, PAT, BuiltinModel>(a);
}

}  // namespace bg
