// bg_mlpchain.cuh -- the proposal network's layers in one kernel per direction,
// and all its weight gradients in one.
//
// A CTA takes 128 rows of the batch through all layers.  Its activations stay
// in shared memory (128 x 512 bf16, K-major in the 128-byte swizzled layout:
// the A operand of the next product) and the accumulators of a whole layer in
// tensor memory (128 x 512 fp32, all of it); only the weights stream, one
// stage of 64 K-elements x 256 output rows at a time.
//
//   forward   H_l = relu(H_{l-1} W_l^T + b_l), l = 1..3; OUT = H_3 W_4^T + b_4
//   backward  G_l = (G_{l+1} W_{l+1}) * [H_l > 0], l = 3..1, G_4 = dOUT
//
// Roles, as in the persistent GEMM: warp 0 loads (TMA), warp 1 issues the
// MMAs, warps 2-9 are the epilogue, two per tensor-memory lane quarter with
// half of the columns each: one pass reads the accumulators 32 columns at a
// time, applies bias and ReLU (or the ReLU's mask), and writes the bf16 results
// to shared memory and, row-major, to the copy the weight gradients read.  A
// layer takes all of tensor memory, so the next one's MMAs start when its
// epilogue is done with a half.
//
// What bounds it: the weights, 1.15 MB per CTA at the 45 bytes a cycle that
// one SM's TMA brings in (a 32 KB stage in 725 cycles, its MMAs in 512), and
// the epilogues between the layers.  One product per launch read every
// activation tile eight times and wrote each activation twice (row-major and
// transposed for the weight gradients, which now read it as it is).  At 16384
// rows the forward chain takes 42 us and the backward one 41 (cold caches); with
// the weight gradients below a training step went from 351 us to 173.
#pragma once

#include "bg_umma.cuh"

namespace umma {

constexpr int kChainWidth = 512;                 // hidden width
constexpr int kChainStages = 3;
constexpr int kChainN = 256;                     // output columns per MMA
constexpr int kChainWide = 4;                    // K-chunks per stage of a 64-column layer (a stage of 32 KB either way)
constexpr int kChainLayers = 4;

struct ChainLayer {
    int K, N;                    // 64 or 512; 64 or 512
    const float *bias;           // forward
    int keep;                    // store the result through its map (ChainMaps::out)
    uint32_t *mask;              // [rows][16]: bit b of word w, column 32 w + b of the ReLU's result is not 0;
                                 // written forward (or null), read backward
    float *C;                    // fp32 result of a 64-wide layer, [rows][64]
    float *colsum;               // backward: column sums over each 32 rows, [rows / 32][512]
};
struct ChainArgs {
    ChainLayer L[kChainLayers];
    int layers, rows;            // rows: a multiple of 128
    int *err;
};
struct alignas(64) ChainMaps {
    CUtensorMap in;              // [rows][64], boxes of 64 x 128
    CUtensorMap w[kChainLayers]; // [N][K], boxes of 64 x min(N, 256)
    CUtensorMap out[kChainLayers];   // [rows][512] row-major results, boxes of 64 x 128
};

struct ChainSmem {
    alignas(1024) unsigned char a[kChainWidth / kKc][kM * kKc * 2];
    alignas(1024) unsigned char w[kChainStages][kChainN * kKc * 2];
    alignas(8) unsigned long long full[kChainStages], empty[kChainStages];
    alignas(8) unsigned long long in_full, in_free;      // the tile's input landed; its last layer has left the buffer
    alignas(8) unsigned long long acc_full[2];           // MMAs of a column half done
    alignas(8) unsigned long long ready[2];              // that half is out of tensor memory and, but for a last
                                                         // layer, the next one's operand in shared memory
    alignas(8) unsigned long long done;
    uint32_t tmem_base;
    int failed;
    alignas(16) float bias[2][kChainN];                  // of the layer at hand, per column half
};
// the whole of a block's shared memory: the dynamic part starts at the
// 1024-byte boundary the swizzled layout needs (checked by the kernel)
constexpr size_t chain_smem_bytes() { return sizeof(ChainSmem); }
static_assert(sizeof(ChainSmem) <= 227 * 1024, "chain shared memory");

// One 2-D box from shared memory (the swizzled layout) to a tensor map.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];\n" ::"l"(reinterpret_cast<uint64_t>(map)),
                 "r"(src), "r"(x), "r"(y)
                 : "memory");
}

// 32 columns of the warp's 32 TMEM lanes, without waiting
__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
          "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

// The sums over a warp's 32 rows of its 16 columns: at each level a lane
// keeps half of its columns and adds the partner's values of them, which is
// the butterfly's tree (16, 8, 4, 2, 1) in 16 shuffles instead of 80.  The
// lane ends with the sum of column 8 b4 + 4 b3 + 2 b2 + b1 of its bits.
__device__ __forceinline__ float column_sums16(float (&v)[16], int lane) {
#pragma unroll
    for (int n = 8; n >= 1; n >>= 1) {
        const bool up = (lane & (2 * n)) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The conjunction of `p` over the 128 threads of named barrier `bar`.
__device__ __forceinline__ bool all_of_half(int p, int bar) {
    int r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.b32 p, %1, 0;\n barrier.red.and.pred q, %2, 128, p;\n selp.b32 %0, 1, 0, q;\n}\n"
        : "=r"(r)
        : "r"(p), "r"(bar)
        : "memory");
    return r != 0;
}

template <bool BWD>
__global__ void __launch_bounds__(kPThreads, 1) k_mlp_chain(const ChainArgs g, const __grid_constant__ ChainMaps maps) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    ChainSmem &sm = *reinterpret_cast<ChainSmem *>(smem_raw);
    if (smem_u32(smem_raw) & 1023u) {                    // uniform
        if (threadIdx.x == 0 && g.err) atomicExch(g.err, 2);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = g.rows / kM;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < kChainStages; ++s) {
            mbar_init(smem_u32(&sm.full[s]), 1);
            mbar_init(smem_u32(&sm.empty[s]), 1);
        }
        mbar_init(smem_u32(&sm.in_full), 1);
        mbar_init(smem_u32(&sm.in_free), 8);
        for (int h = 0; h < 2; ++h) {
            mbar_init(smem_u32(&sm.acc_full[h]), 1);
            mbar_init(smem_u32(&sm.ready[h]), 4);
        }
        mbar_init(smem_u32(&sm.done), 1);
        sm.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sm.tmem_base;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            // ---- producer: the tile's input, then every layer's weight stages
            long long it = 0;
            int tiles = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++tiles) {
                if (tiles && !mbar_wait(smem_u32(&sm.in_free), (uint32_t)((tiles - 1) & 1))) { ok = false; break; }
                mbar_expect_tx(smem_u32(&sm.in_full), kM * kKc * 2);
                tma_load_2d(smem_u32(sm.a[0]), &maps.in, 0, t * kM, smem_u32(&sm.in_full));
                for (int l = 0; l < g.layers && ok; ++l) {
                    const int K = g.L[l].K, N = g.L[l].N, box = N < kChainN ? N : kChainN;
                    const int step = N < kChainN ? min(K, kChainWide * kKc) : kKc;     // K of a stage
                    for (int n0 = 0; n0 < N && ok; n0 += box)
                        for (int k0 = 0; k0 < K; k0 += step, ++it) {
                            const int st = (int)(it % kChainStages);
                            const long long use = it / kChainStages;
                            if (use >= 1 && !mbar_wait(smem_u32(&sm.empty[st]), (uint32_t)((use - 1) & 1))) { ok = false; break; }
                            if (*(volatile int *)&sm.failed) { ok = false; break; }
                            mbar_expect_tx(smem_u32(&sm.full[st]), (uint32_t)(box * step * 2));
                            for (int k = 0; k < step; k += kKc)
                                tma_load_2d(smem_u32(sm.w[st]) + (uint32_t)(k * box * 2), &maps.w[l], k0 + k, n0, smem_u32(&sm.full[st]));
                        }
                }
            }
            if (!ok) atomicExch(&sm.failed, 1);
            // the boxes in flight have landed before the CTA leaves
            if (tiles) mbar_wait(smem_u32(&sm.in_full), (uint32_t)((tiles - 1) & 1));
            for (long long j = (it > kChainStages ? it - kChainStages : 0); j < it; ++j)
                mbar_wait(smem_u32(&sm.full[j % kChainStages]), (uint32_t)((j / kChainStages) & 1));
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issue
            long long it = 0;
            int tiles = 0, inst = 0;                     // inst: layers done so far, over all tiles
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++tiles) {
                if (!mbar_wait(smem_u32(&sm.in_full), (uint32_t)(tiles & 1))) { ok = false; break; }
                for (int l = 0; l < g.layers && ok; ++l, ++inst) {
                    const int K = g.L[l].K, N = g.L[l].N, box = N < kChainN ? N : kChainN;
                    const int step = N < kChainN ? min(K, kChainWide * kKc) : kKc;
                    const uint32_t idesc = box == kChainN ? idesc_bf16(kM, kChainN) : idesc_bf16(kM, 64);
                    // the previous layer's halves (each barrier is passed once a layer)
                    bool have[2] = {inst == 0, inst == 0};
                    auto need = [&](int h) {
                        if (have[h] || !ok) return;
                        have[h] = true;
                        if (!mbar_wait(smem_u32(&sm.ready[h]), (uint32_t)((inst - 1) & 1))) ok = false;
                    };
                    for (int n0 = 0; n0 < N && ok; n0 += box) {
                        need(n0 ? 1 : 0);
                        for (int k0 = 0; k0 < K && ok; k0 += step, ++it) {
                            need(k0 >= kChainN ? 1 : 0);
                            const int st = (int)(it % kChainStages);
                            if (!ok || !mbar_wait(smem_u32(&sm.full[st]), (uint32_t)((it / kChainStages) & 1))) { ok = false; break; }
                            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                            for (int k = 0; k < step; k += kKc) {
                                const uint32_t a_addr = smem_u32(sm.a[(k0 + k) / kKc]), b_addr = smem_u32(sm.w[st]) + (uint32_t)(k * box * 2);
#pragma unroll
                                for (int j = 0; j < kKc / 16; ++j)
                                    umma_bf16(tmem + (uint32_t)n0, smem_desc_sw128(a_addr + j * 32), smem_desc_sw128(b_addr + j * 32),
                                              idesc, (k0 + k > 0 || j > 0) ? 1u : 0u);
                            }
                            umma_commit(smem_u32(&sm.empty[st]));
                        }
                        if (ok) umma_commit(smem_u32(&sm.acc_full[n0 ? 1 : 0]));
                    }
                    need(0);
                    need(1);
                    // a layer of one half completes both barriers
                    if (ok && N <= kChainN) umma_commit(smem_u32(&sm.acc_full[1]));
                }
            }
            if (!ok) atomicExch(&sm.failed, 1);
            umma_commit(smem_u32(&sm.done));             // arrives once every MMA issued above has finished
            if (!mbar_wait(smem_u32(&sm.done), 0u)) atomicExch(&sm.failed, 1);
        }
    } else {
        // ---- epilogue: lanes 32 quarter .. +31, columns 256 half .. +255
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        const uint32_t tq = tmem + ((uint32_t)(quarter * 32) << 16);
        const int c0 = half * kChainN;
        const bool storer = quarter == 0 && lane == 0;          // the half's thread for the stores
        int inst = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            for (int l = 0; l < g.layers && ok; ++l, ++inst) {
                const ChainLayer &L = g.L[l];
                const int r = quarter * 32 + lane, row = t * kM + r;
                const bool narrow = L.N < kChainN;
                // the last layer's stores have read the buffer, and its warps the bias
                if (storer) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                asm volatile("bar.sync %0, 128;\n" ::"r"(1 + half) : "memory");
                if (!BWD) {
                    const int k = (quarter * 32 + lane) * 2;
                    if (!narrow || (half == 0 && k < 64))
                        *reinterpret_cast<float2 *>(&sm.bias[half][k]) = __ldg(reinterpret_cast<const float2 *>(L.bias + c0 + k));
                }
                uint32_t *mrow = L.mask ? L.mask + (long long)row * (kChainWidth / 32) + half * (kChainN / 32) : nullptr;
                uint32_t mnext = BWD ? mrow[0] : 0u;         // a word ahead of its use
                // (both halves write the buffer that the MMAs of both read; the half's
                // warps agree on a wait that gave up, so all of them leave together)
                const int waited = mbar_wait(smem_u32(&sm.acc_full[0]), (uint32_t)(inst & 1)) &&
                                   mbar_wait(smem_u32(&sm.acc_full[1]), (uint32_t)(inst & 1)) && !*(volatile int *)&sm.failed;
                ok = all_of_half(waited, 1 + half);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                if (narrow) {
                    // a 64-wide fp32 layer
                    if (half == 0)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            float v[16];
                            tmem_ld16(tq + (uint32_t)(16 * q), v);
                            float *d = L.C + (long long)row * 64 + 16 * q;
#pragma unroll
                            for (int i = 0; i < 16; i += 4) {
                                const float4 b4 = *reinterpret_cast<const float4 *>(&sm.bias[0][16 * q + i]);
                                reinterpret_cast<float4 *>(d)[i / 4] =
                                    make_float4(v[i] + b4.x, v[i + 1] + b4.y, v[i + 2] + b4.z, v[i + 3] + b4.w);
                            }
                        }
                } else {
                    uint32_t raw[32];
                    tmem_ld32_nowait(tq + (uint32_t)c0, raw);
#pragma unroll 1
                    for (int q = 0; q < kChainN / 32; ++q) {
                        const int col = c0 + 32 * q;
                        uint32_t pk[16];
                        uint32_t m = mnext;
                        if (BWD && q + 1 < kChainN / 32) mnext = mrow[q + 1];
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float x[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) x[e] = __uint_as_float(raw[4 * i + e]);
                            if (BWD) {
#pragma unroll
                                for (int e = 0; e < 4; ++e) x[e] = (m >> (4 * i + e)) & 1u ? x[e] : 0.f;
                            } else {
                                const float4 b4 = *reinterpret_cast<const float4 *>(&sm.bias[half][32 * q + 4 * i]);
                                x[0] += b4.x; x[1] += b4.y; x[2] += b4.z; x[3] += b4.w;
#pragma unroll
                                for (int e = 0; e < 4; ++e) x[e] = x[e] > 0.f ? x[e] : 0.f;
                            }
                            const __nv_bfloat162 h0 = __floats2bfloat162_rn(x[0], x[1]), h1 = __floats2bfloat162_rn(x[2], x[3]);
                            pk[2 * i] = *reinterpret_cast<const uint32_t *>(&h0);
                            pk[2 * i + 1] = *reinterpret_cast<const uint32_t *>(&h1);
                        }
                        if (q + 1 < kChainN / 32) {
                            tmem_ld32_nowait(tq + (uint32_t)(col + 32), raw);
                        }
                        {
                            // the next layer's operand, 16-byte pieces of the swizzled rows
                            unsigned char *d = sm.a[col / kKc] + r * 128;
                            const int p = (col % kKc) / 8;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                *reinterpret_cast<uint4 *>(d + (((p + i) ^ (r & 7)) << 4)) =
                                    make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
                        }
                        if (!BWD && mrow) {
                            m = 0;
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                m |= (((pk[i] & 0xffffu) ? 1u : 0u) | ((pk[i] >> 16) ? 2u : 0u)) << (2 * i);
                            mrow[q] = m;
                        }
                        if (BWD && L.colsum) {
#pragma unroll
                            for (int hh = 0; hh < 2; ++hh) {
                                float v[16];
#pragma unroll
                                for (int i = 0; i < 8; ++i) {
                                    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162 *>(&pk[8 * hh + i]);
                                    v[2 * i] = __low2float(h);
                                    v[2 * i + 1] = __high2float(h);
                                }
                                const float sum = column_sums16(v, lane);
                                if (!(lane & 1))
                                    L.colsum[(long long)(4 * t + quarter) * kChainWidth + col + 16 * hh + (lane >> 1 & 1) +
                                             (lane >> 2 & 1) * 2 + (lane >> 3 & 1) * 4 + (lane >> 4 & 1) * 8] = sum;
                            }
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                }
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sm.ready[half]));
                if (L.keep) {
                    // the half's four chunks to the row-major copy
                    asm volatile("bar.sync %0, 128;\n" ::"r"(1 + half) : "memory");
                    if (storer) {
#pragma unroll
                        for (int c = 0; c < kChainN / kKc; ++c)
                            tma_store_2d(&maps.out[l], smem_u32(sm.a[c0 / kKc + c]), c0 + c * kKc, t * kM);
                        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                    }
                }
                if (l + 1 == g.layers) {
                    if (storer) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sm.in_free));
                }
            }
        if (storer) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
        if (!ok && lane == 0) atomicExch(&sm.failed, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (sm.failed && tid == 0 && g.err) atomicExch(g.err, 1);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
}

// ---------------------------------------------------------------------------
// Every weight gradient in one launch: dW_l = G_l^T H_{l-1}, in `splits` partial
// sums over the batch.  Both operands are read as the chains left them, K (the
// batch row) being the memory row: MN-major tiles.  A unit is a 128 x nt tile of
// one product and one split; a persistent CTA walks the units, the widest
// products first.  While its first loads are under way the epilogue warps sum the
// bias gradients' partials (which depend on the same kernel before this one), so
// that reduction costs no launch and no time of its own.
//
// What bounds it: the operand tiles through one SM's TMA, 48 KB per 64 batch rows
// of a 128 x 256 unit, read 4 + 2 times in all (128-wide tiles: 4 + 4, and
// four launches of one to two uneven waves, 74 us in all at 16384 rows): 39 us, with
// the bias sums (8.7 us) and the step's counters (3.3 us) inside.
constexpr int kDwN = 256;                        // columns of a wide unit
constexpr int kDwStages = 4;
struct DwProduct {
    int M, N, nt;                // nt: kDwN or 64 columns per unit
    int tiles_m, tiles_n, unit0; // first unit
    float *C;                    // [splits][M][N]
    long long split_stride;
};
// The bias gradients, each the sum of its layer's column-sum partials (one per 32
// or 256 batch rows), in one fixed order: block b sums 32 columns of one layer,
// warp w the partials w, w + 8, ... of them (coalesced rows), and warp 0 adds the
// eight warp sums in warp order.
struct BiasRed {
    const float *p[kChainLayers]; int nblk[kChainLayers], ld[kChainLayers], rows[kChainLayers];
    int blk0[kChainLayers + 1];  // first block of each layer
    float *out;                  // [kChainLayers][kChainWidth]
};
struct DwArgs {
    DwProduct p[kChainLayers];
    int units, splits, nk;       // nk: K-chunks per split
    BiasRed bias;
    long long *batch_index, *opt_step;   // counters of a training step, advanced (or null)
    int *err;
};
struct alignas(64) DwMaps {
    CUtensorMap a[kChainLayers], b[kChainLayers];   // boxes of 64 columns x 64 batch rows
};
struct DwSmem {
    alignas(1024) unsigned char a[kDwStages][kM * kKc * 2];
    alignas(1024) unsigned char b[kDwStages][kDwN * kKc * 2];
    alignas(8) unsigned long long full[kDwStages], empty[kDwStages];
    alignas(8) unsigned long long acc_full[2], acc_empty[2];
    alignas(8) unsigned long long done;
    uint32_t tmem_base;
    int failed;
    float red[8][32];
};
static_assert(sizeof(DwSmem) <= 227 * 1024, "weight-gradient shared memory");

struct DwUnit { int q, m0, n0, z; };
__device__ __forceinline__ DwUnit dw_unit(const DwArgs &g, int u) {
    DwUnit r;
    r.q = 0;
#pragma unroll
    for (int i = 1; i < kChainLayers; ++i) r.q += u >= g.p[i].unit0 ? 1 : 0;
    const DwProduct &p = g.p[r.q];
    int mt, nt;
    tile_coords(u - p.unit0, p.tiles_m, p.tiles_n, mt, nt, r.z);
    r.m0 = mt * kM;
    r.n0 = nt * p.nt;
    return r;
}

__device__ __forceinline__ void bias_sums(const BiasRed &r, float (&red)[8][32], int warp, int lane) {
    for (int b = blockIdx.x; b < r.blk0[kChainLayers]; b += gridDim.x) {
        int l = 0;
        while (l + 1 < kChainLayers && b >= r.blk0[l + 1]) ++l;
        const int i = (b - r.blk0[l]) * 32 + lane;
        float g = 0.f;
        if (i < r.rows[l]) {
#pragma unroll 8
            for (int s = warp; s < r.nblk[l]; s += 8) g += r.p[l][(long long)s * r.ld[l] + i];
        }
        red[warp][lane] = g;
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        if (warp == 0 && i < r.rows[l]) {
            float t = red[0][lane];
#pragma unroll
            for (int w = 1; w < 8; ++w) t += red[w][lane];
            r.out[l * kChainWidth + i] = t;
        }
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
    }
}

__global__ void __launch_bounds__(kPThreads, 1) k_weight_gradients(const __grid_constant__ DwArgs g,
                                                                   const __grid_constant__ DwMaps maps) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    DwSmem &sm = *reinterpret_cast<DwSmem *>(smem_raw);
    if (smem_u32(smem_raw) & 1023u) {                    // uniform
        if (threadIdx.x == 0 && g.err) atomicExch(g.err, 2);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid == 0) {
        for (int s = 0; s < kDwStages; ++s) {
            mbar_init(smem_u32(&sm.full[s]), 1);
            mbar_init(smem_u32(&sm.empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&sm.acc_full[b]), 1);
            mbar_init(smem_u32(&sm.acc_empty[b]), 8);
        }
        mbar_init(smem_u32(&sm.done), 1);
        sm.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = sm.tmem_base;
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            // ---- producer
            long long it = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
                const DwUnit w = dw_unit(g, u);
                const int na = min(kM, g.p[w.q].M - w.m0) / 64, nb = g.p[w.q].nt / 64;
                for (int c = 0; c < g.nk; ++c, ++it) {
                    const int st = (int)(it % kDwStages);
                    const long long use = it / kDwStages;
                    if (use >= 1 && !mbar_wait(smem_u32(&sm.empty[st]), (uint32_t)((use - 1) & 1))) { ok = false; break; }
                    if (*(volatile int *)&sm.failed) { ok = false; break; }
                    const uint32_t fb = smem_u32(&sm.full[st]);
                    mbar_expect_tx(fb, (uint32_t)((na + nb) * kKc * 128));
                    const int kx = (w.z * g.nk + c) * kKc;
                    // (a product of 64 rows leaves the other half of its A tile as it was: rows of the
                    // accumulator that are not stored)
                    for (int i = 0; i < na; ++i) tma_load_2d(smem_u32(sm.a[st]) + i * kKc * 128, &maps.a[w.q], w.m0 + 64 * i, kx, fb);
                    for (int i = 0; i < nb; ++i) tma_load_2d(smem_u32(sm.b[st]) + i * kKc * 128, &maps.b[w.q], w.n0 + 64 * i, kx, fb);
                }
            }
            if (!ok) atomicExch(&sm.failed, 1);
            // the last boxes issued into each stage have landed before the CTA leaves
            for (long long j = (it > kDwStages ? it - kDwStages : 0); j < it; ++j)
                mbar_wait(smem_u32(&sm.full[j % kDwStages]), (uint32_t)((j / kDwStages) & 1));
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issue
            long long it = 0;
            int ti = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < g.units && ok; u += gridDim.x, ++ti) {
                const int buf = ti & 1, use = ti >> 1;
                if (use >= 1 && !mbar_wait(smem_u32(&sm.acc_empty[buf]), (uint32_t)((use - 1) & 1))) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t acc = tmem + (uint32_t)(buf * kDwN);
                const uint32_t idesc = g.p[dw_unit(g, u).q].nt == kDwN ? idesc_bf16(kM, kDwN, true) : idesc_bf16(kM, 64, true);
                for (int c = 0; c < g.nk; ++c, ++it) {
                    const int st = (int)(it % kDwStages);
                    if (!mbar_wait(smem_u32(&sm.full[st]), (uint32_t)((it / kDwStages) & 1))) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t a_addr = smem_u32(sm.a[st]), b_addr = smem_u32(sm.b[st]);
#pragma unroll
                    for (int j = 0; j < kKc / 16; ++j)
                        umma_bf16(acc, smem_desc_mn(a_addr + j * 2048), smem_desc_mn(b_addr + j * 2048), idesc,
                                  (c > 0 || j > 0) ? 1u : 0u);
                    umma_commit(smem_u32(&sm.empty[st]));
                }
                if (!ok) break;
                umma_commit(smem_u32(&sm.acc_full[buf]));
            }
            if (!ok) atomicExch(&sm.failed, 1);
            umma_commit(smem_u32(&sm.done));             // arrives once every MMA issued above has finished
            if (!mbar_wait(smem_u32(&sm.done), 0u)) atomicExch(&sm.failed, 1);
        }
    } else {
        // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31, the columns of its half
        if (blockIdx.x == 0 && warp == 2 && lane == 0 && g.opt_step) {
            *g.batch_index += 1;
            *g.opt_step += 1;
        }
        bias_sums(g.bias, sm.red, warp - 2, lane);
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        int ti = 0;
        for (int u = blockIdx.x; u < g.units; u += gridDim.x, ++ti) {
            const int buf = ti & 1, use = ti >> 1;
            const DwUnit w = dw_unit(g, u);
            const DwProduct &p = g.p[w.q];
            const int row = w.m0 + quarter * 32 + lane, cols = p.nt / 2;
            bool ok = mbar_wait(smem_u32(&sm.acc_full[buf]), (uint32_t)(use & 1));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok || *(volatile int *)&sm.failed) { if (lane == 0) atomicExch(&sm.failed, 1); break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            float *d = p.C + (long long)w.z * p.split_stride + (long long)row * p.N + w.n0 + half * cols;
            const uint32_t t0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kDwN + half * cols);
            for (int c = 0; c < cols; c += 32) {
                uint32_t raw[32];
                tmem_ld32_nowait(t0 + (uint32_t)c, raw);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (row < p.M) {
#pragma unroll
                    for (int i = 0; i < 32; i += 4)
                        *reinterpret_cast<float4 *>(d + c + i) =
                            make_float4(__uint_as_float(raw[i]), __uint_as_float(raw[i + 1]), __uint_as_float(raw[i + 2]),
                                        __uint_as_float(raw[i + 3]));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sm.acc_empty[buf]));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (sm.failed && tid == 0 && g.err) atomicExch(g.err, 1);
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
}

}  // namespace umma
