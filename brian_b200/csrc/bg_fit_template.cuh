// bg_fit_template.cuh -- source of the batched fitting kernel, compiled at
// run time by NVRTC for sm_100a once the model is known.
//
// One thread simulates one candidate (particle x target x slice) over its own
// duration and counts coincidences with its target spike train online: the
// semantics of the reference's `runsim` template
// (library/modelfitting/gpu_modelfitting.py:39-116) and its exclusive and
// inclusive coincidence algorithms (gpu_modelfitting.py:118-156):
//
//   I = input[T + I_offset]; state update; is_refractory = T <= next_allowed;
//   has_spiked = threshold && !is_refractory; spikes counted from `onset`;
//   reset while spiking or refractory; next_allowed = T + refractory;
//   the coincidence test uses Tspike = T + spike delay against the last and
//   next target spikes, then the target pointer moves on once Tspike has
//   reached the next target spike.
//
// Differences from the reference template, all by design:
//   * each simulation has its own number of steps (uneven durations);
//   * the target pointer stops at the train's final sentinel instead of
//     reading past the end of the train;
//   * candidates are visited in `order` (longest first, candidates of one
//     target side by side) so a warp shares its input row and its length;
//   * every simulation's state, pointer and flags are loaded once and stored
//     once per launch (the whole run is normally one launch).
//
// Scheduling: simulations are grouped into warp tasks of 32 consecutive
// entries of `order` (longest first, one target's candidates together, so a
// task shares its length and its input row).  The tasks form a queue of
// classes, class k holding the k-th longest nsm tasks (nsm: the device's
// SMs), and a fixed number of resident warps pull from it.  A warp starts
// with a task of the class of its place on its SM (the first block's warps 0
// .. 3 on classes 0 .. 3, the second block's the other way round, and so
// on), so that every SM, and every scheduler of it, begins with one of the
// longest tasks and one of the shorter ones; after that it takes the longest
// task left (greedy longest-processing-time).  One queue for all left that
// to the order in which the blocks' first warps came: with more than two
// blocks an SM some SMs drew only long tasks and the SMs were busy half of the
// time (64 targets x 1024 candidates of 1-20 s, FP32, ms with 2 / 3 / 4 / 8
// blocks: 9.0 / 11.7 / 14.8 / 14.9 with one queue, 9.0 / 9.1 / 9.1 / 9.1 so).
// No warp waits on another; where a block sits changes only the order of the
// tasks.
//
// Latency: the state update is a chain of dependent operations per step, so
// the hot loop carries nothing else: per step it integrates, tests the
// threshold and refractoriness, applies the reset as selects and shifts the
// spike into a 32-bit word.  Everything that only changes at a model spike or
// at a target-pointer move -- the coincidence test, the spike count from
// onset, the record, the pointer itself -- is replayed once per block of 32
// steps, in step order, from that word and the next target time: per step T
// the spike's coincidence test comes first, then the pointer moves at most
// once, exactly as in the reference's per-step loop.  The input of step T+1
// is loaded while step T computes.
//
// The host prepends `typedef <float|double> scalar;`, BG_DT (double),
// BG_DELTA (steps), BG_EXCLUSIVE (0/1) and a `struct Model`
// holding the state registers with load/store/update/threshold/reset members.
#pragma once

// Division by a divisor b fixed for the whole run, given y = RN(1/b), in the
// scalar type itself (P. Markstein, IBM J. Res. Dev. 34(1), 1990; N.
// Brisebarre, J.-M. Muller and S. K. Raina, IEEE Trans. Comput. 53(8), 2004,
// for divisors known in advance): q = RN(a*y), r = b*q - a (exact with one
// FMA), RN(q - r*y) is RN(a/b) while nothing under- or overflows.  bg_rcp_set
// fixes the dividends for which that holds: |a| in [lo, hi], with b, a and
// a/b far enough from the ends of the exponent range that r is exact.  A zero
// dividend gives r = +0 and, for b > 0, -r*y = -0, so the sum keeps the sign
// of q, which is the one IEEE division gives; with b < 0 a zero dividend
// counts as out of range.  BgSeen collects the dividends of a block of steps.
// When one may have been out of range the kernel redoes the block with the
// wide form, which also takes infinite, NaN and every zero dividend (the
// quotient is a*y itself): a swarm without bounds sends candidates to
// negative time constants, whose potential runs off to infinity and stays
// there, and their blocks went through IEEE division one and all (2 targets x
// 1000 candidates, FP64: 4.8 ms an evaluation, against 1.5 ms without).  A
// block that is still suspect is redone with IEEE division; a divisor out of
// range sends the whole simulation there (bg_exact).
//
// The update is a chain of dependent operations, so the division is three of
// them (12 cycles in FP32).  A product in double (two conversions and a
// multiplication on the FP64 pipe) in their place made a step of the adaptive
// LIF, one warp alone in FP32, 71 ns; this form with the samples loaded eight
// steps ahead makes it 36 ns.  The range tests hang off the chain;
// the double's are integer tests on the high word, since a comparison on the
// FP64 pipe costs as much issue as a multiplication.
//
// The five-argument forms are for update code written by hand against the
// interface (reciprocal in double, dividend bound): the float one relies on
// RN32(RN64(a * RN64(1/b))) = RN32(a/b) for normal a and a/b (a/b lies at
// least 2^-49 away from every rounding midpoint of binary32, the double
// product within 2^-52 of a/b).
static const char kFitHelperSource[] = R"BGFIT(
__device__ __forceinline__ float bg_div_fast(const float a, const float b, const double y, const float thr,
                                             bool &suspect) {
    suspect |= (fabsf(a) < thr) && (a != 0.0f);
    return __double2float_rn(__dmul_rn((double)a, y));
}
__device__ __forceinline__ double bg_div_fast(const double a, const double b, const double y, const double thr,
                                              bool &suspect) {
    const double m = fabs(a);
    suspect |= !(m >= thr && m <= 0x1p+900) && (a != 0.0);
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-b, q, a);
    const double q1 = __fma_rn(r, y, q);
    return a == 0.0 ? q : q1;
}
template <typename S> struct BgRcp;
template <> struct BgRcp<float> { float y; int zadj; };  // zadj: -1, or 0 when zero dividends are out of range
template <> struct BgRcp<double> { double y; bool zero; };       // zero: zero dividends are in range
// What a block of steps saw of its divisions: whether some dividend may have
// been out of range.
template <typename S> struct BgSeen;
template <> struct BgSeen<float> {
    // smallest nonzero and largest |dividend| over all divisions (the bits of
    // the first doubled, which drops the sign, and less one, which makes zero
    // the largest): three integer and min/max operations a division, where
    // comparing each with its bounds took four that depend on one another
    unsigned small = 0xffffffffu;
    float large = 0.0f;
    __device__ __forceinline__ void operator()(const float a, const BgRcp<float> &c) {
        small = min(small, 2u * (unsigned)__float_as_int(a) + (unsigned)c.zadj);
        large = fmaxf(large, fabsf(a));
    }
    // lo, hi: the tightest bounds of the simulation's divisors (NaN dividends
    // need no test: either division returns NaN)
    __device__ __forceinline__ bool suspect(const float lo, const float hi) const {
        return small < 2u * (unsigned)__float_as_int(lo) - 1u || large > hi;
    }
};
template <> struct BgSeen<double> {
    bool bad = false;
    __device__ __forceinline__ void operator()(const double a, const BgRcp<double> &c) {
        // exponents 2^-900 .. 2^900 by the high word
        const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
        bad |= !((h - 0x07b00000u < 0x78300000u - 0x07b00000u) || ((h | (unsigned)__double2loint(a)) == 0u && c.zero));
    }
    __device__ __forceinline__ bool suspect(const double, const double) const { return bad; }
};
// The reciprocal of one divisor; lo and hi tighten to its dividends' range.
__device__ __forceinline__ void bg_rcp_set(BgRcp<float> &c, const float b, float &lo, float &hi, bool &exact) {
    const float m = fabsf(b);
    if (!(m >= 0x1p-100f && m <= 0x1p+100f)) exact = true;
    c.y = 1.0f / b;
    c.zadj = b > 0.0f ? -1 : 0;
    lo = fmaxf(lo, fmaxf(0x1p-100f, 0x1p-120f * m));
    hi = fminf(hi, fminf(0x1p+100f, 0x1p+120f * m));
}
__device__ __forceinline__ void bg_rcp_set(BgRcp<double> &c, const double b, double &, double &, bool &exact) {
    const double m = fabs(b);
    if (!(m >= 0x1p-100 && m <= 0x1p+100)) exact = true;
    c.y = 1.0 / b;
    c.zero = b > 0.0;
}
template <typename S> __device__ __forceinline__ S bg_quotient(const S a, const S b, const S y, const S q);
template <> __device__ __forceinline__ float bg_quotient(const float a, const float b, const float y, const float q) {
    return __fmaf_rn(__fmaf_rn(b, q, -a), -y, q);
}
template <> __device__ __forceinline__ double bg_quotient(const double a, const double b, const double y, const double q) {
    return __fma_rn(__fma_rn(b, q, -a), -y, q);
}
// The wide form's record: `bad` when a dividend was out of range, `special`
// when one was infinite, NaN or a zero that BgSeen would not take.
template <typename S> struct BgWide {
    S lo, hi;
    bool bad, special;
    __device__ __forceinline__ BgWide(const S l, const S h) : lo(l), hi(h), bad(false), special(false) {}
    __device__ __forceinline__ bool suspect(const S, const S) const { return bad; }
    // true: the dividend is in range; false: the quotient is a*y or the block is bad
    __device__ __forceinline__ bool operator()(const float a, const BgRcp<float> &c) {
        const float m = fabsf(a);
        const bool in = m >= lo && m <= hi, odd = !(m > 0.0f && m < __int_as_float(0x7f800000));
        bad |= !in && !odd;
        special |= odd && (m != 0.0f || c.zadj == 0);
        return in;
    }
    __device__ __forceinline__ bool operator()(const double a, const BgRcp<double> &c) {
        const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu, l = (unsigned)__double2loint(a);
        const bool in = h - 0x07b00000u < 0x78300000u - 0x07b00000u, zero = (h | l) == 0u, big = h >= 0x7ff00000u;
        bad |= !in && !zero && !big;
        special |= big || (zero && !c.zero);
        return in;
    }
};
template <typename S>
__device__ __forceinline__ S bg_div_fast(const S a, const S b, const BgRcp<S> &c, BgSeen<S> &seen) {
    seen(a, c);
    return bg_quotient<S>(a, b, c.y, a * c.y);
}
template <typename S>
__device__ __forceinline__ S bg_div_fast(const S a, const S b, const BgRcp<S> &c, BgWide<S> &wide) {
    const bool in = wide(a, c);
    const S q = a * c.y, q1 = bg_quotient<S>(a, b, c.y, q);
    return in ? q1 : q;
}
)BGFIT";

static const char kFitKernelSource[] = R"BGFIT(
struct FitArgs {
    scalar *S;                  // [nstate][ns] state, SoA
    const scalar *I;            // concatenated input traces
    const long long *I_off;     // first input sample of each simulation
    const int *nsteps;          // length of each simulation (steps)
    const int *spk;             // concatenated target trains (steps), sentinel-framed
    const long long *spk_end;   // one past the last entry of each simulation's train
    long long *spk_idx;         // current position in the train
    const int *delay;           // spike delay (steps)
    const int *refr;            // refractory period (steps)
    int *next_allowed;          // last refractory step
    int *ncoinc;
    int *nspikes;
    unsigned char *flags;       // bit 0 last_spike_allowed, bit 1 next_spike_allowed
    const int *order;           // thread -> simulation
    int *rec;                   // optional spike record [ns][rec_cap]
    int *rec_n;
    int *queue;                 // tasks taken of each class, then blocks seen per SM; zero at launch
    long long ns;
    int Tstart, Tend, onset, rec_cap, nsm;
};
#define BG_CLASSES 64           // the last class holds every task past the others
#define BG_SM_SLOTS 256         // block counters per SM (an SM id beyond them shares one: only the balance is at stake)

#define BG_NO_SPIKE 0x7fffffff

struct Sim {
    Model m;
    const int *spk;
    long long idx, last_idx;
    int last_spike, next_spike, next2_spike;
    bool last_allowed, next_allowed;
    int ncoinc, nspikes, spikedelay, refractory, next_allowed_T, onset;
    int *rec;
    int nrec, rec_cap;

    __device__ __forceinline__ int train_at(long long k) const {
        return k <= last_idx ? __ldg(spk + k) : BG_NO_SPIKE;
    }

    // update, threshold, refractoriness and reset of step T; true on a spike.
    // FAST selects the update with reciprocal divisions (sets `suspect` when
    // one of them may differ from IEEE division).  REFR false: no step of the
    // block can be refractory (no refractory period and none pending), so
    // next_allowed_T is left to the caller.
    template <bool FAST, bool REFR, class SEEN>
    __device__ __forceinline__ bool step(const int T, const scalar I_in, bool &suspect, SEEN &seen) {
        const scalar t = (scalar)((double)T * BG_DT);
        if (FAST) m.update_fast(I_in, t, suspect, seen);
        else m.update(I_in, t);
        if (!REFR) {
            const bool has_spiked = m.threshold(I_in, t);
            m.reset(I_in, t, has_spiked);
            return has_spiked;
        }
        const bool is_refractory = (T <= next_allowed_T);
        const bool has_spiked = m.threshold(I_in, t) && !is_refractory;
        m.reset(I_in, t, has_spiked || is_refractory);
        next_allowed_T = has_spiked ? T + refractory : next_allowed_T;
        return has_spiked;
    }

    // Samples T .. T+7 of the input (the last sample for steps past Tlast).
    static __device__ __forceinline__ void load8(scalar (&v)[8], const scalar *Iin, const int T, const int Tlast) {
        if (T + 7 <= Tlast) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __ldg(Iin + T + j);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __ldg(Iin + min(T + j, Tlast));
        }
    }

    // Eight steps from T on the fast update, their spikes at constant bits.
    template <bool REFR, class SEEN>
    __device__ __forceinline__ unsigned steps8(const int T, const scalar (&I)[8], bool &suspect, SEEN &seen) {
        unsigned b = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (step<true, REFR, SEEN>(T + j, I[j], suspect, seen)) b |= 1u << j;
        return b;
    }

    // The 32 steps of a whole block on the fast update.  Ia holds the samples
    // of its first eight steps and leaves with those of the eight steps after
    // it: every sample is loaded eight steps (some 500 cycles) before its
    // use, where loading it one step ahead left a third of the issue slots
    // waiting for it (one warp in FP32: 51 against 36 ns a step).
    template <bool REFR, class SEEN>
    __device__ __forceinline__ unsigned block(const int T0, const int Tlast, const scalar *Iin, scalar (&Ia)[8],
                                              bool &suspect, SEEN &seen) {
        unsigned bits = 0;
        scalar Ib[8];
#pragma unroll 1
        for (int k = 0; k < 32; k += 16) {
            load8(Ib, Iin, T0 + k + 8, Tlast);
            bits |= steps8<REFR, SEEN>(T0 + k, Ia, suspect, seen) << k;
            load8(Ia, Iin, T0 + k + 16, Tlast);
            bits |= steps8<REFR, SEEN>(T0 + k + 8, Ib, suspect, seen) << (k + 8);
        }
        return bits;
    }

    // block() with the refractory test when some step of it can be refractory;
    // without it next_allowed_T only records the last spike.
    template <class SEEN>
    __device__ __forceinline__ unsigned fast_block(const bool refr, const int T0, const int Tlast, const scalar *Iin,
                                                   scalar (&Ia)[8], bool &suspect, SEEN &seen) {
        if (refr) return block<true, SEEN>(T0, Tlast, Iin, Ia, suspect, seen);
        const unsigned bits = block<false, SEEN>(T0, Tlast, Iin, Ia, suspect, seen);
        if (bits) next_allowed_T = T0 + 31 - __clz(bits) + refractory;
        return bits;
    }

    // The rare forms of a block, on a copy of the simulation and out of line
    // (inline they cost the fast form a quarter of its speed: 45 against 36 ns
    // a step of one warp).  The wide form: bit 0 of `flags` when the block is
    // still suspect, bit 1 when the next one should start with this form too.
    // It leaves Ia to the caller.
    static __device__ __noinline__ unsigned wide_block(Sim &s, const int T0, const int Tlast, const scalar *Iin,
                                                       unsigned &flags) {
        BgWide<scalar> seen(s.m.bg_lo, s.m.bg_hi);
        bool suspect = false;
        scalar Ia[8];
        load8(Ia, Iin, T0, Tlast);
        const unsigned bits = s.block<true, BgWide<scalar>>(T0, Tlast, Iin, Ia, suspect, seen);
        flags = (suspect || seen.bad ? 1u : 0u) | (suspect || seen.bad || seen.special ? 2u : 0u);
        return bits;
    }
    // n steps with IEEE division.
    static __device__ __noinline__ unsigned exact_block(Sim &s, const int T0, const int n, const scalar *Iin) {
        unsigned bits = 0;
        bool unused = false;
        BgSeen<scalar> unseen;
        for (int k = 0; k < n; ++k)
            bits |= (s.step<false, true>(T0 + k, __ldg(Iin + T0 + k), unused, unseen) ? 1u : 0u) << k;
        return bits;
    }

    // Steps T0 .. T0+n-1 have run; bit k of `bits` is the spike of step T0+k.
    __device__ __forceinline__ void replay(const int T0, const int n, unsigned bits) {
        const int Tn = T0 + n;
        if (bits) {
            const int c = onset - T0;
            const unsigned counted = c <= 0 ? 0xffffffffu : (c >= 32 ? 0u : (0xffffffffu << c));
            nspikes += __popc(bits & counted);
            if (rec) {
                for (unsigned b = bits; b; b &= b - 1) {
                    if (nrec < rec_cap) rec[nrec] = T0 + __ffs(b) - 1;
                    ++nrec;
                }
            }
        }
        int Tc = T0;                        // first step whose pointer test is pending
        for (;;) {
            const long long ta = (long long)next_spike - spikedelay;
            const int Tadv = ta <= Tc ? Tc : (ta >= Tn ? Tn : (int)ta);
            const int Tsp = bits ? T0 + __ffs(bits) - 1 : Tn;
            const int Te = min(Tadv, Tsp);
            if (Te >= Tn) break;
            const int Tspike = Te + spikedelay;
            if (Te == Tsp) {
                bits &= bits - 1;
#if BG_EXCLUSIVE
                const bool near_last = last_spike + BG_DELTA >= Tspike;
                const bool near_next = next_spike - BG_DELTA <= Tspike;
                const bool ml = near_last && last_allowed, mn = near_next && next_allowed;
                ncoinc += (ml || mn) ? 1 : 0;
                last_allowed = last_allowed && !near_last;
                next_allowed = (next_allowed && !near_next) || (ml && mn);
#else
                ncoinc += ((last_spike + BG_DELTA >= Tspike) || (next_spike - BG_DELTA <= Tspike)) ? 1 : 0;
#endif
            }
            if (Tspike >= next_spike) {
                ++idx;
                last_spike = next_spike;
                next_spike = next2_spike;
                next2_spike = train_at(idx + 2);
#if BG_EXCLUSIVE
                last_allowed = next_allowed;
                next_allowed = true;
#endif
            }
            Tc = Te + 1;
        }
    }
};

__device__ __forceinline__ void run_sim(const FitArgs &a, const long long i)
{
    Sim s;
    s.m.load(a.S, a.ns, i);
    const scalar *Iin = a.I + a.I_off[i];
    s.spk = a.spk;
    s.idx = a.spk_idx[i];
    s.last_idx = a.spk_end[i] - 1;
    s.last_spike = s.train_at(s.idx);
    s.next_spike = s.train_at(s.idx + 1);
    s.next2_spike = s.train_at(s.idx + 2);
    const unsigned char fl = a.flags[i];
    s.last_allowed = (fl & 1) != 0;
    s.next_allowed = (fl & 2) != 0;
    s.ncoinc = a.ncoinc[i];
    s.nspikes = a.nspikes[i];
    s.spikedelay = a.delay[i];
    s.refractory = a.refr[i];
    s.next_allowed_T = a.next_allowed[i];
    s.onset = a.onset;
    s.rec = a.rec ? a.rec + i * (long long)a.rec_cap : (int *)0;
    s.nrec = a.rec ? a.rec_n[i] : 0;
    s.rec_cap = a.rec_cap;
    const int Tend = min(a.Tend, a.nsteps[i]);
    if (a.Tstart < Tend) {
        // loads clamp to the last step, so every address stays inside this
        // simulation's input
        const int Tlast = Tend - 1;
        scalar Ia[8];
        Sim::load8(Ia, Iin, a.Tstart, Tlast);
        int T0 = a.Tstart;
        const bool fast_ok = !s.m.bg_exact;
        bool wide = false;                  // start the block with the wide form: the last one needed it
        while (T0 < Tend) {
            const int n = min(32, Tend - T0);
            // checkpoint: a block with a suspect division runs again
            const Model m0 = s.m;
            const int na0 = s.next_allowed_T;
            unsigned bits = 0;
            bool done = false;
            if (fast_ok && n == 32 && !wide) {
                BgSeen<scalar> seen;
                bool suspect = false;
                bits = s.fast_block(s.refractory > 0 || na0 >= T0, T0, Tlast, Iin, Ia, suspect, seen);
                done = !(suspect || seen.suspect(s.m.bg_lo, s.m.bg_hi));
            }
            // the lanes here decide together: every form gives the same results,
            // and a warp that splits over two of them runs both
            const unsigned lanes = __activemask();
            if (!__all_sync(lanes, done)) {
                // a suspect block, one after such a block, a simulation whose
                // divisors need IEEE division, or the steps after the last whole block
                Sim r = s;
                r.m = m0;
                r.next_allowed_T = na0;
                unsigned flags = 1;
                if (fast_ok && n == 32) {
                    bits = Sim::wide_block(r, T0, Tlast, Iin, flags);
                    wide = (flags & 2) != 0;
                    if (flags & 1) {
                        r.m = m0;
                        r.next_allowed_T = na0;
                    }
                }
                if (flags & 1) bits = Sim::exact_block(r, T0, n, Iin);
                s.m = r.m;
                s.next_allowed_T = r.next_allowed_T;
                Sim::load8(Ia, Iin, T0 + n, Tlast);
                wide = __any_sync(lanes, wide);
            }
            s.replay(T0, n, bits);
            T0 += n;
        }
    }
    s.m.store(a.S, a.ns, i);
    a.spk_idx[i] = s.idx;
    a.flags[i] = (unsigned char)((s.last_allowed ? 1 : 0) | (s.next_allowed ? 2 : 0));
    a.ncoinc[i] = s.ncoinc;
    a.nspikes[i] = s.nspikes;
    a.next_allowed[i] = s.next_allowed_T;
    if (a.rec) a.rec_n[i] = s.nrec;
}

extern "C" __global__ void __launch_bounds__(128) bg_fit_sim(const FitArgs a)
{
    __shared__ int slot_s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        unsigned sm;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
        slot_s = atomicAdd(a.queue + BG_CLASSES + (sm % BG_SM_SLOTS), 1);
    }
    __syncthreads();
    const int slot = slot_s;
    const long long ntasks = (a.ns + 31) / 32;
    const int nclass = (int)min((ntasks + a.nsm - 1) / a.nsm, (long long)BG_CLASSES);
    // this warp's first class; a warp beyond the classes has nothing to start
    // with and leaves (the first block of an SM starts class 0, and whoever
    // starts empties the queue)
    const int first = slot * 4 + ((slot & 1) ? 3 - warp : warp);
    if (first >= nclass) return;
    int c = first, lo = 0;
    for (;;) {
        const long long c0 = (long long)c * a.nsm;
        const long long left = ntasks - c0;
        const int size = (int)(c == BG_CLASSES - 1 ? left : min(left, (long long)a.nsm));
        int idx = 0;
        if (lane == 0) idx = atomicAdd(a.queue + c, 1);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx < size) {
            const long long g = (c0 + idx) * 32 + lane;
            if (g < a.ns) run_sim(a, a.order[g]);
            __syncwarp();
        } else if (c == lo) {
            ++lo;                           // this class is empty, and stays so
        }
        if (lo >= nclass) break;
        c = lo;
    }
}
)BGFIT";
