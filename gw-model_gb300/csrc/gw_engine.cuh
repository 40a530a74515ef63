// gw_engine.cuh -- the cluster-resident multi-step engine kernel and its launcher.
// Included by gw_kernel_fp64.cu and gw_kernel_fp32.cu, which instantiate one precision each.
//
// CTA = ssa_warps + kOdeWarps warps.  In a cell's leader CTA the last kOdeWarps warps run the
// global step as the lane program of gw_ode_program.h; in the other CTAs of the cell every warp
// runs SSA.  The CTAs of a cell are held together only by their data, which travel by st.async
// and complete per-parity mbarriers of the receiver (no cluster barrier inside the launch):
//   SSA warps : wait for sv[s&1] (the CTA's mbarrier), run the SSA of step s on the CTA's CRU tile, and
//               push their flux partials into their slots in the leader's shared memory.  FP64: one
//               CRU per lane at a time, the ones with events on four lanes each.  FP32: group_steps
//               (few CRUs) or split_steps.
//   ODE warps : wait for the warp partials of step s-1 (the leader's mbarrier), reduce them,
//               increments and Euler update (globals s -> s+1), transcendental phases of the new
//               state (an idle lane forms the stimulus of step s+1), push sv[(s+1)&1]; phases the
//               SSA does not need run after the push.
#pragma once

#include <type_traits>

#include "gw_kernel.cuh"
#include "gw_math64.cuh"
#include "gw_ode_program.h"

namespace gw {
namespace dev {

// Flux partial of a warp: the sums over its CRUs of JLCC, Jxfer, Jtr and the open ClCh count.
template <bool FP64>
struct alignas(16) Partial;
template <>
struct alignas(16) Partial<true> {
    double v[4];
};
// FP32: each sum in three integers, of the cell's units (SsaConsts::flux_exp) and of 2^-23 and 2^-46 of them,
// the latter two from 0 to 2^28; or, with the last one's top bit set, an FP64 number in the first two.
// Jtr's last two words lie apart (CtaView::part_tail), which keeps the others' stride at 32 bytes.
template <>
struct alignas(16) Partial<false> {
    int jh;
    uint32_t jl, jm;
    int cl;
    int xh;
    uint32_t xl, xm;
    int th;
};
struct alignas(8) PartialTail {
    uint32_t tl, tm;
};
constexpr uint32_t kWideSum = 0x80000000u;
// Bytes of a warp's partial.
template <bool FP64>
constexpr int kPartBytes = (int)sizeof(Partial<FP64>) + (FP64 ? 0 : (int)sizeof(PartialTail));
// A term has to stay below kMaxFluxUnits units.  Then 32 bits hold a warp's first words (2^19 a term, and
// whatever warp takes how many, the CTA's CRUs once each) and a lane's other words (2^22 a term: at most two
// quiet passes over all CRUs of the CTA, or one event in each batch of eight).
constexpr int kMaxFluxUnits = 1 << 19;
constexpr int kMostCtaCrus = 232448 / (int)(sizeof(TileRec<float>) + 4);  // in 227 KB of shared memory
static_assert((int64_t)kMostCtaCrus * (kMaxFluxUnits + 1) < (1ll << 31) && (int64_t)(kMostCtaCrus / 8 + 1) * (1 << 22) < (1ll << 31) &&
              2 * (kMostCtaCrus / 32 + 1) <= kMostCtaCrus / 8, "FP32 flux sums in 32 bits");

struct OdeShared {
    double g[kNumGlobals];  // the cell's globals (FP64 state)
    double sums[4];         // JLCC, ClCh, Jtr, Jxfer sums of the last reduced step (FP64)
    int status;
    int pad;
};

constexpr int kMaxThreads = 512;  // SSA warps + ODE warps per CTA (128 registers per thread)
constexpr int kMaxThreadsFp64 = 256;  // FP64 instance: at most 4 SSA warps, up to 255 registers
constexpr int kMaxWarps = kMaxThreads / 32;

struct SmemLayout {
    size_t cc, sv, ode, x, math, svs, rtab, part, mbar, fq, tile, total;
};

// FP64: CRUs of a CTA whose first iteration of a step waits for the four-lane pass (the queue
// holds their tile indices; a CTA with more such CRUs in a step runs the rest on their own lanes).
constexpr int kEngQCap = 256;

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

template <typename R, typename T>
__host__ __device__ inline SmemLayout smem_layout(int tile_cap, int max_cta_cell) {
    SmemLayout L;
    size_t o = 0;
    L.cc = o;
    o += align16(sizeof(SsaConsts<R>));
    L.sv = o;
    o += align16(2 * kSvCount * sizeof(R));
    L.ode = o;
    o += align16(sizeof(OdeShared));
    L.x = o;
    o += align16(kOdeMaxSlots * sizeof(T));
    L.math = o;  // exp / log tables of the FP64 global step
    o += align16(sizeof(math64::Tables));
    L.svs = o;   // staging of the per-step SSA values before the push
    o += align16(kSvCount * sizeof(R));
    L.rtab = o;  // the CTA's subunit rate tables (FP32 SSA), one per step parity
    o += align16((size_t)2 * kRateTab * sizeof(float2));
    L.part = o;  // [parity][rank in cell][warp]: warp partials (written by the cell's CTAs)
    o += (size_t)2 * max_cta_cell * kMaxWarps * kPartBytes<sizeof(R) == 8>;
    L.mbar = o;  // mbarriers: the warp partials of steps of parity 0 and 1 (leader CTA), then the
    o += 80;     // per-step SSA values of parity 0 and 1 (every CTA); FP32: the quiet warps', the event
                 // warps' and the queue's of parity 0 and 1
    L.fq = o;    // the event queue: FP64: four counters, then kEngQCap tile indices; FP32: eight counters,
                 // then two queues of a 16-bit tile index for every CRU of the CTA
    o += sizeof(R) == 8 ? align16((size_t)(4 + kEngQCap) * sizeof(int)) : align16(32 + (size_t)4 * tile_cap);
    L.tile = o;  // TileRec<R> per CRU
    o += align16((size_t)tile_cap * sizeof(TileRec<R>));
    L.total = o;
    return L;
}

__device__ __forceinline__ bool finite_bits(double x) {
    return ((__double_as_longlong(x) >> 52) & 0x7FF) != 0x7FF;
}

__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// barrier of the ODE warps (named barrier 1, kOdeLanes threads)
__device__ __forceinline__ void ode_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kOdeLanes) : "memory"); }
// barrier of a CTA's SSA warps (named barrier 2, n threads: the CTA's SSA threads 0 .. n-1)
__device__ __forceinline__ void ssa_bar(int n) { asm volatile("bar.sync 2, %0;" ::"r"(n) : "memory"); }
// barrier of a CTA's quiet warps after a record (split_steps; named barrier 3, n threads)
__device__ __forceinline__ void rec_bar(int n) { asm volatile("bar.sync 3, %0;" ::"r"(n) : "memory"); }
// named barrier `id` of n threads that also returns the OR of v over them: a decision that every
// participating thread takes the same way (a bounded wait's outcome, which is per thread)
__device__ __forceinline__ bool bar_or(int id, int n, bool v) {
    int r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((int)v), "r"(id), "r"(n)
        : "memory");
    return r != 0;
}

// A cell's stimulus protocol in registers.
struct Stim {
    int mode;
    double start, period, dur, amp;
    const double *samples;
    int64_t n;
    __device__ __forceinline__ explicit Stim(const CellDyn &d)
        : mode(d.stim_mode), start(d.stim_start), period(d.stim_period), dur(d.stim_dur), amp(d.stim_amp),
          samples(d.stim_samples), n(d.stim_n) {}
    __device__ __forceinline__ double sample(int64_t ri) const {
        return mode == STIM_SAMPLES && ri >= 0 && ri < n ? samples[ri] : 0.0;
    }
    // Pulse train at time t.  Uses explicit round-to-nearest operations so the host's evaluation of the
    // same pulse train gives the same values (within the first period the quotient truncates to 0).
    __device__ __forceinline__ double pulse(double t) const {
        if (mode == STIM_PULSE) {
            double tb = __dsub_rn(t, start);
            if (tb >= 0.0) {
                if (period > 0.0 && tb >= period) tb = __dsub_rn(tb, __dmul_rn(period, trunc(div_rn(tb, period))));
                if (tb < dur) return amp;
            }
        }
        return 0.0;
    }
};

// Branch of the gate rates (common.hpp:176-218): 0 for V >= -40, 2 for V == -47.13, 1 otherwise
// (NaN included), from integer compares on the bit pattern (no FP64 issue slots).
__device__ __forceinline__ int v_regime(double V) {
    const long long b = __double_as_longlong(V);
    if (b >= 0) return (unsigned long long)b > 0x7FF0000000000000ull ? 1 : 0;  // +NaN: 1
    const unsigned long long u = (unsigned long long)b;
    if (u <= 0xC044000000000000ull) return 0;  // -40 <= V <= -0
    return u == 0xC04790A3D70A3D71ull ? 2 : 1;  // V == -47.13
}

// !(x > 0) for a concentration, from the bit pattern (non-positive or NaN).
__device__ __forceinline__ bool not_positive(double x) {
    const long long b = __double_as_longlong(x);
    return b <= 0 || (unsigned long long)b > 0x7FF0000000000000ull;
}

__device__ __forceinline__ double o_exp(double x, const math64::Tables &M) { return math64::exp(x, M); }
__device__ __forceinline__ float o_exp(float x, const math64::Tables &) { return expf(x); }
__device__ __forceinline__ double o_log(double x, const math64::Tables &M) { return math64::log(x, M); }
__device__ __forceinline__ float o_log(float x, const math64::Tables &) { return logf(x); }
__device__ __forceinline__ double o_sqrt(double x) { return sqrt_rn(x); }
__device__ __forceinline__ float o_sqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double o_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float o_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// x with its sign flipped where bit 31 of w is set
__device__ __forceinline__ double flip(double x, uint32_t w) {
    return __hiloint2double(__double2hiint(x) ^ (int)(w & 0x80000000u), __double2loint(x));
}
__device__ __forceinline__ float flip(float x, uint32_t w) { return __uint_as_float(__float_as_uint(x) ^ (w & 0x80000000u)); }

// The FP32 pair (hi, lo) of an FP64 value for the SSA: hi = (float)d, lo = (float)(d - hi); for an
// FP64 SSA the value itself and 0.  By integer operations where hi and lo are normal (the two
// conversions and the subtraction would take the FP64 pipe, of every warp that meets them predicated).
__device__ __forceinline__ void stage_pair(float *st, int ihi, int ilo, double d) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const uint32_t e = (uint32_t)(b >> 52) & 0x7FFu, sign = (uint32_t)(b >> 32) & 0x80000000u;
    float hi, lo;
    if (e - 960u < 180u) {
        // significand 2^52 + f: its upper 24 bits rounded to nearest even, the rest a signed 30-bit integer
        const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
        const unsigned long long r = m + 0x0FFFFFFFull + ((m >> 29) & 1ull);
        const uint32_t h = (uint32_t)(r >> 29);  // 2^23 .. 2^24
        const int rest = (int)((long long)m - (long long)((unsigned long long)h << 29));
        hi = __uint_as_float(sign | (((e - 897u) << 23) + h));
        // rest 2^(e - 1075): rounded to 24 bits by the conversion, then scaled by a normal power of two
        const float l = __fmul_rn((float)rest, __uint_as_float((e - 948u) << 23));
        lo = __uint_as_float(__float_as_uint(l) ^ sign);
    } else {
        hi = (float)d;
        lo = (float)(d - (double)hi);
    }
    st[ihi] = hi;
    st[ilo] = lo;
}
__device__ __forceinline__ void stage_pair(double *st, int ihi, int ilo, double d) {
    st[ihi] = d;
    st[ilo] = 0.0;
}

// One op of the lane program in registers: the operand slots as byte offsets into X (a sign bit on
// top of 15 bits), so that a step spends no loads on the program.
struct LaneOp {
    uint32_t w[7];   // a[0..13], two to a word
    uint32_t meta;   // kind | width << 8 | output slot (byte offset; a global's index for OK_DOT) << 16
    int stage;       // 1 + the sv index an op's output is staged to, or 0
    __device__ __forceinline__ int kind() const { return (int)(meta & 0xFFu); }
    __device__ __forceinline__ int width() const { return (int)((meta >> 8) & 0xFFu); }
    __device__ __forceinline__ uint32_t out() const { return meta >> 16; }
    __device__ __forceinline__ uint32_t off(int k) const { return (w[k >> 1] >> (16 * (k & 1))) & 0x7FFFu; }
    __device__ __forceinline__ uint32_t sign(int k) const { return (k & 1) ? w[k >> 1] : w[k >> 1] << 16; }
};

// The cell's global step by the kOdeLanes ODE threads (t = 0 .. kOdeLanes-1), thread t running op t
// of each phase.  Every warp holds one op kind per phase, so the kinds do not diverge.
//   increments()  phase E up to the flux sums: this thread's row sum (rows of up to 8 lanes, shuffles
//                 in the first warp only), with update()'s other operands already loaded
//   update()      after a barrier: the flux-sum terms and the Euler update by the rows' first lanes
//   terms()       phase A of the new state (reloads the ops where V changed its regime)
//   powers()      phase P (general Jup exponents only)
//   quotients()   phase B
// Each is followed by a barrier of the ODE threads (after powers() only when has_powers()).  An op
// whose output is a per-step SSA value also writes it, in the SSA's precision, to the staging row;
// Cai and CaNSR are staged by the caller.
// What bounds it: the latency of three phases, each one op: 4 FP64 instructions (64 cycles each) and
// a three-level shuffle tree, an integer exp / log / square root between two FP64 instructions
// (gw_math64.cuh, gw_div64.cuh), and an integer division behind three FP64 instructions.
template <typename T, typename R>
struct OdeLane {
    unsigned char *X;
    R *stage;
    OdeShared *os;
    const math64::Tables *M;
    const OdeProgram *P;  // global memory
    int t, reg;
    LaneOp e, a, b;

    __device__ __forceinline__ T &x(uint32_t off) const { return *reinterpret_cast<T *>(X + off); }
    __device__ __forceinline__ T arg(const LaneOp &o, int k) const { return x(o.off(k)); }
    __device__ __forceinline__ T *slots() const { return reinterpret_cast<T *>(X); }
    __device__ __forceinline__ bool has_powers() const { return P->n_phases == 4; }

    __device__ __forceinline__ void load(LaneOp &o, int q) const {
        const int b0 = P->phase_begin[q];
        o = LaneOp{};
        if (t >= P->phase_begin[q + 1] - b0) return;
        const int i = b0 + t, ai = P->alt_idx[i];
        const OdeOp *op = reg > 0 && ai != 255 ? &P->alt[reg - 1][ai] : &P->ops[i];
        const uint32_t *src = reinterpret_cast<const uint32_t *>(op);
        const uint32_t m = src[0];
        const bool dot = (m & 0xFFu) == (uint32_t)OK_DOT;
        o.meta = (m & 0xFFFFu) | ((m >> 16) * (dot ? 1u : (uint32_t)sizeof(T)) << 16);
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const uint32_t v = src[1 + k];
            o.w[k] = (v & 0x80008000u) | ((v & 0x7FFF7FFFu) * (uint32_t)sizeof(T));
        }
        o.stage = P->sv_stage[i];
    }
    __device__ __forceinline__ void load_all() {
        load(e, 0);
        load(a, 1);
        load(b, P->push_phase);
    }

    // A row's first lane after increments(): its sum, and what update() will need that does not depend
    // on the flux sums.
    struct Row {
        T v, s, c0, c1;
        double g;
        bool first;
    };
    __device__ __forceinline__ Row increments() const {
        Row r{};
        if (t >= 64) return r;
        T v = flip(arg(e, 1), e.sign(1)) * arg(e, 2);
        v = o_fma(flip(arg(e, 3), e.sign(3)), arg(e, 4), v);
        v = o_fma(flip(arg(e, 5), e.sign(5)), arg(e, 6), v);
        v = o_fma(flip(arg(e, 7), e.sign(7)), arg(e, 8), v);
        if (t < 32) {
            // rows of `width` lanes (a power of two, rows aligned to it): tree over offsets 1, 2, 4
            const int wm = e.kind() == OK_DOT ? e.width() - 1 : 0;
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) {
                const T o = __shfl_down_sync(0xffffffffu, v, off);
                if ((t & wm) + off <= wm && (t & (2 * off - 1)) == 0) v += o;
            }
        }
        r.first = e.kind() == OK_DOT && (t & (e.width() - 1)) == 0;
        r.v = v;
        r.s = arg(e, 0);
        r.c0 = arg(e, 9);
        r.c1 = arg(e, 11);
        r.g = os->g[r.first ? e.out() : 0u];
        return r;
    }
    __device__ __forceinline__ void update(const Row &r) const {
        if (!r.first) return;
        T v = r.v;
        if (t < 32) v = o_fma(r.c1, arg(e, 12), o_fma(r.c0, arg(e, 10), v));
        const int out = (int)e.out();
        const double ng = sizeof(T) == 8 ? __fma_rn((double)r.s, (double)v, r.g) : r.g + (double)(r.s * v);
        os->g[out] = ng;
        slots()[XS_G + out] = (T)ng;
        if (!finite_bits(ng)) atomicCAS(&os->status, 0, (int)GW_ERR_NONFINITE);  // first error of the cell
    }
    __device__ __forceinline__ void put(const LaneOp &o, T v) const {
        x(o.out()) = v;
        if (o.stage) stage[o.stage - 1] = (R)v;
    }
    __device__ __forceinline__ void exp_op(const LaneOp &o) const {
        put(o, o_fma(arg(o, 0), o_exp(o_fma(arg(o, 1), arg(o, 2), arg(o, 3)), *M), arg(o, 4)));
    }
    __device__ __forceinline__ void terms() {
        const int r = v_regime(os->g[0]);
        if (r != reg) {
            reg = r;
            load_all();
        }
        switch (a.kind()) {
        case OK_EXP: exp_op(a); break;
        case OK_LOG:
            put(a, o_fma(arg(a, 4), o_log(o_fma(arg(a, 1), arg(a, 5), arg(a, 0)), *M), arg(a, 2) + arg(a, 3)));
            break;
        case OK_POW: {
            const T s = o_sqrt(arg(a, 2)), c = arg(a, 0) * arg(a, 1);
            put(a, o_fma(c, a.width() == 2 ? s * o_sqrt(s) : s, arg(a, 3)));
            break;
        }
        default: break;
        }
    }
    __device__ __forceinline__ void powers() const {
        LaneOp o;
        load(o, 2);
        if (o.kind() == OK_EXP) exp_op(o);
    }
    __device__ __forceinline__ void quotients() const {
        if (b.kind() == OK_QUOT)
            put(b, quot(arg(b, 0) * o_fma(arg(b, 2), arg(b, 3), arg(b, 1)), o_fma(arg(b, 5), arg(b, 6), arg(b, 4))));
        else if (b.kind() == OK_SUM3)
            put(b, o_fma(arg(b, 4), arg(b, 5), o_fma(arg(b, 2), arg(b, 3), arg(b, 0) * arg(b, 1))));
    }
};

// Sums {JLCC, ClCh, Jtr, Jxfer} of the n warp partials of one slot (n <= 16 CTAs x kMaxWarps), quantity
// `warp` by ODE warp `warp`.
constexpr int kSlotsPerLane = 16 * kMaxWarps / 32;
// FP32: integer sums, the lanes' through REDUX (s in three pieces), hence exact: s units of 2^-23 of the
// flux unit 2^u, and f < 2^23 per lane of 2^-46 of it; rounded once to FP64 (sums of 2^40 and more of the
// former, 2^17 flux units, without the latter: 2^-40 of them).
__device__ __forceinline__ double fixed_total(long long s, uint32_t f, int u) {
    const uint32_t lo = (uint32_t)s;
    const int h = __reduce_add_sync(0xffffffffu, (int)(s >> 32));
    const uint32_t l1 = __reduce_add_sync(0xffffffffu, lo >> 16), l0 = __reduce_add_sync(0xffffffffu, lo & 0xFFFFu);
    f = __reduce_add_sync(0xffffffffu, f);
    s = ((long long)h << 32) + ((long long)l1 << 16) + (long long)l0 + (long long)(f >> 23);
    u -= 23;
    if ((unsigned long long)(s + (1ll << 40)) < (2ull << 40)) {
        s = s * 8388608ll + (long long)(f & 0x7FFFFFu);
        u -= 23;
    }
    const unsigned long long m = s < 0 ? 0ull - (unsigned long long)s : (unsigned long long)s;
    if (m == 0ull) return 0.0;
    const uint32_t mh = (uint32_t)(m >> 32);
    const int z = mh ? __clz((int)mh) : 32 + __clz((int)(uint32_t)m);
    const unsigned long long d = math64::pack(m << z, 63 - z + u);
    return __longlong_as_double((long long)(s < 0 ? d | 0x8000000000000000ull : d));
}
template <typename T>
__device__ __forceinline__ void reduce_partials(const Partial<false> *slot, const PartialTail *tail, const int *flux_exp,
                                                int n, int warp, int lane, double *out, T *X) {
    // the words of {jh, jl, jm, cl, xh, xl, xm, th} and {tl, tm} that are this warp's sum
    const int *const first = reinterpret_cast<const int *>(slot) + (warp == 0 ? 0 : (warp == 1 ? 3 : (warp == 2 ? 7 : 4)));
    const uint32_t *const next = reinterpret_cast<const uint32_t *>(warp == 2 ? reinterpret_cast<const int *>(tail) : first + 1);
    const int step = warp == 2 ? 2 : 8;
    double r;
    if (warp == 1) {
        int c = 0;
#pragma unroll
        for (int k = 0; k < kSlotsPerLane; ++k) {
            const int i = lane + 32 * k;
            c += i < n ? first[8 * i] : 0;
        }
        r = (double)__reduce_add_sync(0xffffffffu, c);
    } else {
        const int unit = flux_exp[warp == 0 ? 0 : (warp == 2 ? 2 : 1)];
        long long s = 0;
        uint32_t l = 0, m = 0, any = 0;  // (the sums of eight slots fit)
#pragma unroll
        for (int k = 0; k < kSlotsPerLane; ++k) {
            const int i = lane + 32 * k;
            const uint32_t mi = i < n ? next[step * i + 1] : 0u;
            s += i < n ? first[8 * i] : 0;
            l += i < n ? next[step * i] : 0u;
            m += mi;
            any |= mi;
        }
        if (!__any_sync(0xffffffffu, any & kWideSum)) {
            r = fixed_total(s * 8388608ll + (long long)(l + (m >> 23)), m & 0x7FFFFFu, unit);
        } else {
            // some warp had a term beyond the integers' range (or a NaN): FP64 sums
            r = 0.0;
#pragma unroll 1
            for (int i = lane; i < n; i += 32) {
                const int h = first[8 * i];
                const uint32_t l = next[step * i], m = next[step * i + 1];
                r += m & kWideSum ? __hiloint2double(h, (int)l)
                                  : ldexp((double)h + (double)l * 0x1p-23 + (double)m * 0x1p-46, unit);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
        }
    }
    if (lane == 0) {
        out[warp] = r;
        X[XS_SUMS + warp] = (T)r;
    }
}
template <typename T>
__device__ __forceinline__ void reduce_partials(const Partial<true> *slot, const PartialTail *, const int *, int n, int warp,
                                                int lane, double *out, T *X) {
    const int src = warp == 0 ? 0 : (warp == 1 ? 3 : (warp == 2 ? 2 : 1));  // of {JLCC, Jxfer, Jtr, ClCh}
    const int nk = (n + 31) >> 5;
    double a = 0.0;
    for (int k = 0; k < nk; ++k) {
        const int i = lane + 32 * k;
        if (i < n) a += slot[i].v[src];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) {
        out[warp] = a;
        X[XS_SUMS + warp] = (T)a;
    }
}

// Per-step SSA values of the new state to every CTA of the cell: the staging row (written by the
// ops that produce the values, see OdeLane, and visible after the phase's barrier) pushed in
// 16-byte words (CTA, word) by all kOdeLanes threads, as asynchronous stores that count themselves
// off the receiving CTA's mbarrier of this slot.  The addresses are formed once per launch.
template <bool FP64>
struct SvPush {
    using R = typename std::conditional<FP64, double, float>::type;
    static constexpr int kWords = kSvCount * (int)sizeof(R) / 16;  // 16-byte words of one slot
    static constexpr int kMost = (kWords * kMaxClusterCtas + kOdeLanes - 1) / kOdeLanes;
    static_assert(kSvCount * sizeof(R) % 16 == 0, "sv slot in 16-byte words");
    const uint4 *src[kMost];
    uint32_t dst[kMost], bar[kMost];  // of slot 0 (slot 1: kSvCount values and 8 bytes on); dst 0: none
    __device__ __forceinline__ SvPush(void *svbuf, const void *stage, uint32_t mbar, const CtaWork &w, int t) {
#pragma unroll
        for (int k = 0; k < kMost; ++k) {
            const int idx = t + k * kOdeLanes, r = idx / kWords, i = idx - r * kWords;
            src[k] = reinterpret_cast<const uint4 *>(stage) + i;
            dst[k] = bar[k] = 0u;
            if (r < w.n_cta_cell) {
                const uint32_t rank = (uint32_t)(w.first + r);
                dst[k] = map_rank(reinterpret_cast<uint4 *>(svbuf) + i, rank);
                bar[k] = map_rank_addr(mbar, rank);
            }
        }
    }
    __device__ __forceinline__ void operator()(int slot) const {
#pragma unroll
        for (int k = 0; k < kMost; ++k)
            if (bar[k])
                st_async(dst[k] + (uint32_t)slot * (uint32_t)(kSvCount * sizeof(R)), *src[k], bar[k] + 8u * (uint32_t)slot);
    }
};

// Ca in 2^-40 mM fixed point (exact, order-independent sums of the record-time CRU sums).
__device__ __forceinline__ long long fix40(float x) { return __float2ll_rn(x * 0x1p40f); }
__device__ __forceinline__ long long fix40(double x) { return __double2ll_rn(x * 0x1p40); }

// The RyR states of subunit j as the int16 code of the reference's reduced-memory trace
// (utils.py:8-22): a negative count in a lumped pair (3/4, 5/6) moves the pair's total into the
// pair's first state; code = n1 + 6 n2 + 36 n3 + 216 n4 + 1296 n5.
__device__ __forceinline__ uint32_t ryr_code16(const uint32_t (&ry)[6], int j) {
    const int r0 = byte_s(ry[0], j), r1 = byte_s(ry[1], j), r2 = byte_s(ry[2], j);
    const int r3 = byte_s(ry[3], j), r4 = byte_s(ry[4], j), r5 = byte_s(ry[5], j);
    const bool n34 = r2 < 0 || r3 < 0, n56 = r4 < 0 || r5 < 0;
    const int q2 = n34 ? r2 + r3 : r2, q3 = n34 ? 0 : r3, q4 = n56 ? r4 + r5 : r4;
    return (uint32_t)(uint16_t)(int16_t)(r0 + 6 * r1 + 36 * q2 + 216 * q3 + 1296 * q4);
}

// Record step, by one warp over its CRUs [beg, end) of the tile after the step's SSA: the trace
// cell's CRU records (planes or the reduced-memory codec) and every cell's CRU sums (warp sums
// added to the record's int64 counters; integer adds, so the totals do not depend on order).
template <typename R>
__device__ __forceinline__ void record_pass(const KernelArgs &a, const CtaWork &w, int cell, int64_t r_idx, int beg,
                                            int end, int lane, const TileRec<R> *tile) {
    constexpr bool FP64 = sizeof(R) == 8;
    const bool crus = cell == a.tr_cell;
    const bool sums = a.tr_sums != nullptr;
    long long v[kSumFields] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int m = beg + lane; m < end; m += 32) {
        Cru<R> c;
        tile_get(c, tile[m]);
        const uint32_t lcc = c.lcc, fl = c.flags;
        const uint32_t(&ry)[6] = c.ryr;
        const R(&cs)[4] = c.cass;
        const R jsr = c.cajsr;
        if (sums) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int st = byte_u(lcc, j);
                const bool open = st == 6 || st == 12;
                const bool cond = open && ((fl >> j) & 1u);
                const long long f = fix40(cs[j]);
                v[0] += open;
                v[1] += cond;
                v[2] += cond ? f : 0;
                v[3] += byte_s(ry[2], j) + byte_s(ry[3], j);
                v[5] += f;
            }
            v[4] += __popc((fl >> 4) & 0xFu);
            v[6] += fix40(jsr) + (FP64 ? 0ll : fix40(c.cajsr_lo));
            v[7] += 1;
        }
        if (crus) {
            const int64_t cm = w.cru_begin + m;
            if (a.tr_mode == 0) {
                const int64_t st = a.tr_cru_stride;
                a.tr_lcc[r_idx * st + cm] = lcc;
                a.tr_flags[r_idx * st + cm] = fl;
#pragma unroll
                for (int k = 0; k < 6; ++k) a.tr_ryr[(r_idx * 6 + k) * st + cm] = ry[k];
#pragma unroll
                for (int j = 0; j < 4; ++j) reinterpret_cast<R *>(a.tr_cass)[(r_idx * 4 + j) * st + cm] = cs[j];
                reinterpret_cast<R *>(a.tr_cajsr)[r_idx * st + cm] = jsr;
            } else {
                const int64_t o = r_idx * a.tr_ncru + cm;
                a.tr_lcc[o] = lcc;
                a.tr_gate[o] = ((fl & 0xFu) * 0x00204081u) & 0x01010101u;
                a.tr_clch[o] = (((fl >> 4) & 0xFu) * 0x00204081u) & 0x01010101u;
                a.tr_ryrc[2 * o] = ryr_code16(ry, 0) | (ryr_code16(ry, 1) << 16);
                a.tr_ryrc[2 * o + 1] = ryr_code16(ry, 2) | (ryr_code16(ry, 3) << 16);
                reinterpret_cast<float4 *>(a.tr_cass_f)[o] =
                    make_float4((float)cs[0], (float)cs[1], (float)cs[2], (float)cs[3]);
                a.tr_cajsr_f[o] = (float)jsr;  // FP32: the compensated value rounds to its leading part
            }
        }
    }
    if (sums) {
#pragma unroll
        for (int f = 0; f < kSumFields; ++f) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[f] += __shfl_xor_sync(0xffffffffu, v[f], o);
        }
        if (lane == 0) {
            unsigned long long *dst = a.tr_sums + ((int64_t)cell * a.rec_cap + r_idx) * kSumFields;
#pragma unroll
            for (int f = 0; f < kSumFields; ++f)
                if (v[f] != 0) atomicAdd(dst + f, (unsigned long long)v[f]);
        }
    }
}


// Per-lane flux accumulators and their warp sum as a Partial (all lanes hold it).
template <bool FP64>
struct FluxAcc;
template <>
struct FluxAcc<true> {
    double dj = 0, dx = 0, dtr = 0;
    int acl = 0;
    __device__ __forceinline__ void add(double j, double x, double t, int cl) {
        dj += j;
        dx += x;
        dtr += t;
        acl += cl;
    }
    __device__ __forceinline__ Partial<true> warp_total(PartialTail &) {
        Partial<true> pv;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dj += __shfl_xor_sync(0xffffffffu, dj, o);
            dx += __shfl_xor_sync(0xffffffffu, dx, o);
            dtr += __shfl_xor_sync(0xffffffffu, dtr, o);
            acl += __shfl_xor_sync(0xffffffffu, acl, o);
        }
        pv.v[0] = dj;
        pv.v[1] = dx;
        pv.v[2] = dtr;
        pv.v[3] = (double)acl;
        return pv;
    }
};
// FP32: fixed-point sums, so that they do not depend on which lane of which warp took a CRU, or when (the
// split between quiet and event warps depends on the launch's start).  A term v is scaled to the cell's
// units (SsaConsts::flux_scale, from its JLCC_const, rxfer and rtr) and rounded to a multiple of them by
// adding 1.5 * 2^23, whose float's low bits are then the multiple (less the constant's); what is left goes
// the same way to multiples of 2^-23 and 2^-46 of a unit.  All differences are exact.  So a term of 2^-23 units or
// more is summed whole (at the model's parameters down to 2.3e-10, 3.7e-9 and 7.3e-12 mM/ms of JLCC, Jxfer and
// Jtr, and in proportion to those three), a smaller one rounded to 2^-46 units.
// (Two words, the last at 2^-34 to 2^-40 mM/ms whatever the parameters, took 15 fewer of ~710 instructions per
// pass, but a warp's Jxfer sum at rest was off by up to 9.4e-8 of itself at rxfer = 200 and 3.5e-5 at 0.2, an FP32
// tree's by 5.9e-8 and 1.2e-7; these by nothing.  1,024 cells 20.0 -> 20.8 ms per 50 steps, 256 amid the release
// 11.4 -> 11.8 per 100, one 12,500-CRU cell 10.6 -> 10.8 per 1,000.  Not taken: the terms converted to 64-bit
// integers, 21.8 ms; a branch on the range instead of the maximum and the float sums, 21.2.)
// With a term out of range the warp sends its plain float sums.
template <>
struct FluxAcc<false> {
    int jh = 0, jl = 0, jm = 0, xh = 0, xl = 0, xm = 0, th = 0, tl = 0, tm = 0, acl = 0;
    float jf = 0.f, xf = 0.f, tf = 0.f;
    float largest = 0.f;  // term, in its units
    const SsaConsts<float> &c;
    __device__ __forceinline__ explicit FluxAcc(const SsaConsts<float> &cc) : c(cc) {}
    __device__ __forceinline__ static void split(float a, int &h, int &l, int &m) {
        constexpr uint32_t Mb = 0x4B400000u;
        constexpr float M = 12582912.f, S = 8388608.f;
        const float t = __fadd_rn(a, M), r = __fsub_rn(a, __fsub_rn(t, M));
        const float u = __fmaf_rn(r, S, M), w = __fmaf_rn(__fmaf_rn(r, S, __fsub_rn(M, u)), S, M);
        h += (int)(__float_as_uint(t) - Mb);
        l += (int)(__float_as_uint(u) - Mb);
        m += (int)(__float_as_uint(w) - Mb);
    }
    // the largest of |a|, |b| and |c|, or NaN
    __device__ __forceinline__ static float max3(float a, float b, float c) {
        float r;
        asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
        return r;
    }
    __device__ __forceinline__ void add(float j, float x, float t, int cl) {
        const float aj = __fmul_rn(j, c.flux_scale[0]), ax = __fmul_rn(x, c.flux_scale[1]), at = __fmul_rn(t, c.flux_scale[2]);
        largest = max3(max3(largest, aj, ax), at, at);
        split(aj, jh, jl, jm);
        split(ax, xh, xl, xm);
        split(at, th, tl, tm);
        jf += j;
        xf += x;
        tf += t;
        acl += cl;
    }
    // The warp's sum: the lower words' carries go up in every lane, which leaves them from 0 to 2^23.
    __device__ __forceinline__ static void total(bool floats, float f, int &h, int &l, int &m) {
        if (floats) {
            double v = (double)f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            h = __double2hiint(v);
            l = __double2loint(v);
            m = (int)kWideSum;
        } else {
            l += m >> 23;
            h = __reduce_add_sync(0xffffffffu, h + (l >> 23));
            l = (int)__reduce_add_sync(0xffffffffu, (uint32_t)l & 0x7FFFFFu);
            m = (int)__reduce_add_sync(0xffffffffu, (uint32_t)m & 0x7FFFFFu);
        }
    }
    __device__ __forceinline__ Partial<false> warp_total(PartialTail &tail) {
        const bool floats = __any_sync(0xffffffffu, !(largest < (float)kMaxFluxUnits));
        total(floats, jf, jh, jl, jm);
        total(floats, xf, xh, xl, xm);
        total(floats, tf, th, tl, tm);
        tail = PartialTail{(uint32_t)tl, (uint32_t)tm};
        return Partial<false>{jh, (uint32_t)jl, (uint32_t)jm, (int)__reduce_add_sync(0xffffffffu, acl),
                              xh, (uint32_t)xl, (uint32_t)xm, th};
    }
};

// A CTA's view of its work item and of the shared-memory layout, rebuilt from the kernel
// arguments by each of the kernel's parts.
template <bool FP64, bool ODE64>
struct CtaView {
    using R = typename std::conditional<FP64, double, float>::type;
    using T = typename std::conditional<ODE64, double, float>::type;
    CtaWork w;
    int nw, warp, lane, ot, n_ssa;
    bool active, leader, ode_thread;
    SsaConsts<R> *cc;
    R *svbuf;
    OdeShared *os;
    T *X;
    math64::Tables *M;
    void *svstage;
    Partial<FP64> *part;
    PartialTail *part_tail;  // FP32
    float2 *rtab;
    int *fq;        // FP64: by parity, entries queued; FP32: by step mod 3, entries reserved << 16 | written, and
                    // claimed, then the split by parity; then the queues, by parity
    uint32_t mbar;  // shared address of the partials' mbarrier of parity 0 (parity 1 at +8); the
                    // SSA values' mbarriers of parity 0 and 1 at +16 and +24; FP32: the quiet warps'
                    // at +32 and +40, the event warps' at +48 and +56, the queue's (cleared for the
                    // step) at +64 and +72
    bool grouped;   // FP32: few enough CRUs for group_steps
    TileRec<R> *tile;

    __device__ __forceinline__ explicit CtaView(const KernelArgs &a) {
        extern __shared__ __align__(16) unsigned char smem[];
        nw = a.ssa_warps;  // SSA warps of a leader CTA; the other CTAs have nw + kOdeWarps
        warp = (int)(threadIdx.x >> 5);
        lane = (int)(threadIdx.x & 31);
        ot = (int)threadIdx.x - nw * 32;  // ODE thread index 0 .. kOdeLanes-1
        w = a.work[blockIdx.x];
        active = w.cell >= 0;
        leader = active && w.rank_in_cell == 0;
        ode_thread = leader && warp >= nw;
        n_ssa = (leader ? nw : nw + kOdeWarps) * 32;  // SSA threads of this CTA
        grouped = !FP64 && w.cru_count <= (n_ssa == 32 * kMaxWarps && w.n_cta_cell > 2 ? kGroupCrusSpread : kGroupCrus) * (n_ssa >> 5);
        const SmemLayout L = smem_layout<R, T>(a.tile_cap, a.max_cta_cell);
        cc = reinterpret_cast<SsaConsts<R> *>(smem + L.cc);
        svbuf = reinterpret_cast<R *>(smem + L.sv);
        os = reinterpret_cast<OdeShared *>(smem + L.ode);
        X = reinterpret_cast<T *>(smem + L.x);
        M = reinterpret_cast<math64::Tables *>(smem + L.math);
        svstage = smem + L.svs;
        part = reinterpret_cast<Partial<FP64> *>(smem + L.part);
        part_tail = reinterpret_cast<PartialTail *>(part + 2 * a.max_cta_cell * kMaxWarps);
        rtab = reinterpret_cast<float2 *>(smem + L.rtab);
        fq = reinterpret_cast<int *>(smem + L.fq);
        mbar = smem_addr(smem + L.mbar);
        tile = reinterpret_cast<TileRec<R> *>(smem + L.tile);
    }
};

// The leader CTA's ODE warps over a launch: the transcendental phases of the initial state and
// the push of sv[0], then per global step s the increments up to the flux sums, the wait for and the
// reduction of the warp partials of step s-1 (one quantity per warp), the global step s -> s+1 and the
// push of sv[(s+1)&1], and the carry back to the cell block at the end.  A function of its own (not inlined
// into the kernel), so that its register allocation and schedule do not depend on the SSA code.
template <bool FP64, bool ODE64>
__device__ __noinline__ void ode_warps(const KernelArgs &a, uint64_t step0) {
    using T = typename std::conditional<ODE64, double, float>::type;
    using R = typename std::conditional<FP64, double, float>::type;
    const CtaView<FP64, ODE64> v(a);
    OdeShared &os = *v.os;
    T *X = v.X;
    const int ot = v.ot, lane = v.lane, cell = v.w.cell, warp = ot >> 5;
    const int pslot = a.max_cta_cell * kMaxWarps;  // warp partials per parity slot
    R *stage = reinterpret_cast<R *>(v.svstage);
    const CellStatic &C = a.cs[cell];
    const CellDyn &d0 = a.dyn[cell];
    const Stim stim(d0);
    OdeLane<T, R> L;
    L.X = reinterpret_cast<unsigned char *>(X);
    L.stage = stage;
    L.os = &os;
    L.M = v.M;
    L.P = a.prog;
    L.t = ot;
    for (int i = ot; i < kOdeMaxSlots; i += kOdeLanes) X[i] = (T)0;
    math64::load_tables(*v.M, ot, kOdeLanes);
    ode_bar();
    if (ot == 0) {
        X[XS_ONE] = (T)1;
        X[XS_MONE] = (T)-1;
        os.sums[0] = d0.sum_jlcc;
        os.sums[1] = d0.sum_clch;
        os.sums[2] = d0.sum_jtr;
        os.sums[3] = d0.sum_jxfer;
        os.status = 0;
        X[XS_DT] = (T)a.dt;
        for (int i = 0; i < 4; ++i) X[XS_SUMS + i] = (T)os.sums[i];
    }
    for (int i = ot; i < kNumGlobals; i += kOdeLanes) {
        os.g[i] = d0.g[i];
        X[XS_G + i] = (T)d0.g[i];
    }
    for (int i = ot; i < kOdeConstCap; i += kOdeLanes) X[XS_FIRST_FREE + i] = (T)C.ode_consts[i];
    // The accumulated time, and the stimulus of the next step, by a lane that has no increment (t_{s+1} =
    // t_s + dt, as the reference accumulates it).  A sampled stimulus is read a step before its use.
    const bool clock = ot == 2 * 32;
    double time = d0.t, next_time = d0.t, next_stim = 0.0, ahead = 0.0;
    if (clock) {
        ahead = stim.sample(a.run_step0 + 1);
        X[XS_ISTIM] = (T)(stim.mode == STIM_SAMPLES ? stim.sample(a.run_step0) : stim.pulse(time));
    }
    ode_bar();
    // staging row: the constant SSA values once per launch, Cai and CaNSR of the initial state
    // (the other values are staged by the ops that compute them)
    if (ot < kSvCount && ot != SV_CAI && ot != SV_CANSR && ot != SV_CAI_LO && ot != SV_CANSR_LO) {
        const int src = a.prog->sv_src[ot];
        if (src < XS_FIRST_FREE + kOdeMaxConsts) stage[ot] = (R)X[src];
    }
    const SvPush<FP64> push(v.svbuf, v.svstage, v.mbar + 16u, v.w, ot);
    L.reg = v_regime(os.g[0]);
    L.load_all();
    const bool powers = L.has_powers();
    // Cai and CaNSR of the state with their FP32 remainders, by two lanes of the last warp in phase B
    const int pair = ot == kOdeLanes - 1 ? 0 : (ot == kOdeLanes - 2 ? 1 : -1);
    auto phases = [&]() {  // the new state's phases, each with its barrier
        L.terms();
        ode_bar();
        if (powers) {
            L.powers();
            ode_bar();
        }
        L.quotients();
        if (pair == 0) stage_pair(stage, SV_CAI, SV_CAI_LO, os.g[3]);
        if (pair == 1) stage_pair(stage, SV_CANSR, SV_CANSR_LO, os.g[4]);
    };
    phases();
    ode_bar();
    // (the SSA warps wait for these bytes in step 0: the host launches 1..steps_per_launch
    // steps, never 0, so no CTA exits while they may be in flight)
    push(0);
    // bytes of the cell's warp partials per step
    const uint32_t part_bytes =
        (uint32_t)kPartBytes<FP64> * (uint32_t)(v.nw + (v.w.n_cta_cell - 1) * (v.nw + kOdeWarps));
    bool stopped = false;  // a wait ran out (the same on every ODE thread)
    int s_stop = -1;       // the step whose wait (for the partials of step s_stop - 1) ran out
    for (int s = 0; s < a.n_steps; ++s) {
        const int par = s & 1;
        const int64_t ri = a.run_step0 + s;
        const bool rec = a.record_every > 0 && (ri % a.record_every) == 0;
        const int64_t r_idx = rec ? ri / a.record_every - a.rec_base : -1;
        const bool rec_ok = rec && r_idx >= 0 && r_idx < a.rec_cap;
        // After a wait has run out the cell stops for the rest of the launch (no waits, no
        // declarations, no pushes): its CTAs then run out their own waits and stop too, so the
        // launch ends within about a second per CTA and few stray bytes land on any mbarrier.
        if (stopped) continue;
        // the partials of step s will complete the next phase of mbarrier par (the previous one,
        // step s-2's, completed before the wait of step s-1)
        if (ot == 0)
            mbar_arrive_expect_tx(v.mbar + 8u * (uint32_t)par,
                                  part_bytes + (s == (a.test_extra_first ? 0 : a.n_steps - 1) ? (uint32_t)a.test_extra_tx : 0u));
        if (ot == 0 && (not_positive(os.g[1]) || not_positive(os.g[2])) && os.status == 0)
            os.status = GW_ERR_NERNST;
        // the increments up to the flux sums (warps 0 and 1), the next stimulus (warp 2), and the sums of
        // step s-1 (step 0 uses the carry)
        const typename OdeLane<T, R>::Row row = L.increments();
        if (clock) {
            next_time = time + a.dt;
            next_stim = stim.mode == STIM_SAMPLES ? ahead : stim.pulse(next_time);
            ahead = stim.sample(ri + 2);
        }
        bool ok = true;
        if (s > 0) {
            ok = mbar_wait_warp(v.mbar + 8u * (uint32_t)(par ^ 1), (uint32_t)((s - 1) >> 1) & 1u);
            __syncwarp();
            // (a warp's lanes may find different outcomes; whatever is summed after a wait that ran out
            // is not used)
            reduce_partials(v.part + (par ^ 1) * pslot, v.part_tail + (par ^ 1) * pslot, v.cc->flux_exp,
                            v.w.n_cta_cell * kMaxWarps, warp, lane, os.sums, X);
        }
        if (bar_or(1, kOdeLanes, !ok)) {  // the same decision on all ODE threads
            if (ot == 0) atomicCAS(&os.status, 0, (int)GW_ERR_SYNC_TIMEOUT);
            stopped = true;
            s_stop = s;
            continue;
        }
        L.update(row);
        if (clock) {
            time = next_time;
            X[XS_ISTIM] = (T)next_stim;
        }
        ode_bar();
        if (rec_ok) {
            double *dst = a.tr_glob + ((int64_t)cell * a.rec_cap + r_idx) * kNumGlobals;
            for (int i = ot; i < kNumGlobals; i += kOdeLanes) dst[i] = os.g[i];
            if (clock && (cell == 0 || (a.tr_cell >= 0 && cell == a.tr_cell))) a.tr_t[r_idx] = time;
        }
        phases();
        ode_bar();
        // (no push after the launch's last step: no one would wait for those bytes, and a CTA
        // must not exit while stores into its shared memory may still be in flight)
        if (s + 1 < a.n_steps)
            push(par ^ 1);
    }
    // carry of the last step's fluxes, globals and counters back to the cell block
    if (a.n_steps > 0 && !stopped) {
        const bool ok =
            mbar_wait(v.mbar + 8u * (uint32_t)((a.n_steps - 1) & 1), (uint32_t)((a.n_steps - 1) >> 1) & 1u);
        if (bar_or(1, kOdeLanes, !ok) && ot == 0) atomicCAS(&os.status, 0, (int)GW_ERR_SYNC_TIMEOUT);
    }
    // After a wait ran out in step s_stop, warp partials of steps s_stop - 1 and s_stop may still
    // land here (the cell's CTAs send step s + 1 only after the SSA values of step s + 1, which the
    // leader pushes only after the partials of step s - 1): thread 0 waits, bounded, for both
    // declared phases, so that no store into this CTA is in flight when it exits (an st.async
    // completes only on its mbarrier; the closing cluster barrier does not order it).
    if (stopped && ot == 0 && s_stop >= 1) {
        mbar_wait(v.mbar + 8u * (uint32_t)((s_stop - 1) & 1), (uint32_t)((s_stop - 1) >> 1) & 1u);
        mbar_wait(v.mbar + 8u * (uint32_t)(s_stop & 1), (uint32_t)(s_stop >> 1) & 1u);
    }
    if (a.n_steps > 0)
        reduce_partials(v.part + ((a.n_steps - 1) & 1) * pslot, v.part_tail + ((a.n_steps - 1) & 1) * pslot, v.cc->flux_exp,
                        v.w.n_cta_cell * kMaxWarps, warp, lane, os.sums, X);
    ode_bar();
    CellDyn &d = a.dyn[cell];
    for (int i = ot; i < kNumGlobals; i += kOdeLanes) d.g[i] = os.g[i];
    if (clock) d.t = time;
    if (ot == 0) {
        d.sum_jlcc = os.sums[0];
        d.sum_clch = os.sums[1];
        d.sum_jtr = os.sums[2];
        d.sum_jxfer = os.sums[3];
        d.step = step0 + (uint64_t)a.n_steps;
        if (os.status != 0) atomicCAS(&a.status[cell], 0, os.status);
    }
    // the launch's one closing cluster barrier (every thread of every CTA of the cluster)
    cluster_arrive();
    cluster_wait();
}

// A warp's flux partial of a step of parity par, pushed by lane 0 straight into the leader's slot (rank,
// warp) by asynchronous stores that count themselves off the leader's mbarrier of this parity
// (the warp goes on without waiting for them to land); the leader sums the cell's warp partials.
template <bool FP64, bool ODE64>
__device__ __forceinline__ void send_partial(const KernelArgs &a, const CtaView<FP64, ODE64> &v, int par, int pslot,
                                             FluxAcc<FP64> &acc) {
    PartialTail tail;
    const Partial<FP64> pv = acc.warp_total(tail);
    if (v.lane != 0) return;
    const int slot = par * pslot + v.w.rank_in_cell * kMaxWarps + v.warp;
    const uint32_t rd = map_rank(v.part + slot, (uint32_t)v.w.first);
    const uint32_t rm = map_rank_addr(v.mbar + 8u * (uint32_t)par, (uint32_t)v.w.first);
    if constexpr (FP64) {
        st_async(rd, make_uint4(lo_of(pv.v[0]), hi_of(pv.v[0]), lo_of(pv.v[1]), hi_of(pv.v[1])), rm);
        st_async(rd + 16u, make_uint4(lo_of(pv.v[2]), hi_of(pv.v[2]), lo_of(pv.v[3]), hi_of(pv.v[3])), rm);
    } else {
        st_async(rd, make_uint4((uint32_t)pv.jh, pv.jl, pv.jm, (uint32_t)pv.cl), rm);
        st_async(rd + 16u, make_uint4((uint32_t)pv.xh, pv.xl, pv.xm, (uint32_t)pv.th), rm);
        st_async8(map_rank(v.part_tail + slot, (uint32_t)v.w.first), make_uint2(tail.tl, tail.tm), rm);
    }
}

// The step of the CRUs held by a warp's eight groups of four lanes (m < 0: none), from begin().
__device__ __forceinline__ void group_run(const KernelArgs &a, const SsaConsts<float> &cc, TileRec<float> *tile, int m,
                                          Cru<float> &c, SsaLane<float, false> &sl, Stream &rng, const float *sv,
                                          const float2 *rtab, uint32_t tag, FluxAcc<false> &acc,
                                          unsigned long long &my_events, int &my_err) {
    while (__any_sync(0xffffffffu, m >= 0)) {
        int err = 0;
        const bool done = sl.iterate_group(m >= 0, c, cc, sv, rtab, rng, (float)a.dt, a.event_cap, err);
        if (m >= 0 && done) {
            if ((threadIdx.x & 3u) == 0u) {
                tile_put(tile[m], c, tag);
                my_events += (unsigned long long)sl.ev;
                my_err |= err;
                acc.add(c.jlcc[0] + c.jlcc[1] + c.jlcc[2] + c.jlcc[3], sl.jxfer_sum, sl.jtr,
                        __popc((c.flags >> 4) & 0xFu));
            }
            m = -1;
        }
    }
}

// The FP32 SSA of a CTA with few CRUs (v.grouped), each warp with a contiguous range of them and nothing shared
// between the warps.  With up to eight to a warp every CRU goes on four lanes at once: one pass, 2.0 k cycles
// without an event and 5.3 k with one, and the global step beside it sets the time (3.2 us per step at rest
// for a cell of 777 CRUs over 9 to 16 CTAs).  With more, up to 32, one CRU goes on each lane through all its
// iterations (SsaLane::iterate): the warp runs as many as its CRU with the most jumps, the first one together
// with the quiet CRUs' only one.  It is bound by latency: 2.7 k cycles an iteration, 5.5 k with an event in it,
// most of it instruction fetch.  (A quiet pass first and then the CRUs with a jump eight at a time on four lanes did the
// first iteration twice and kept more code in flight.  us per step at rest and amid the release, this and that,
// and last a lane that takes the warp's next CRU, beside the global step of that time:
// 300 cells of 20 to 60 CRUs, two SSA warps: 4.4 and 8.4; 7.0 and 10.1; 7.0 and 7.3 (a whole beat of 400 ms: this
// 5.7, the last 7.0).
// 256 cells of 100, four warps: 5.4 and 8.6; 7.1 and 10.0; 7.1 and 9.2.
// 100 cells of 50 to 200, twelve warps: 4.2 and 6.6; 4.6 and 6.9; 6.2 and 6.6.)
// split_steps shares quiet passes and events between warps.  It needs enough events: with few, one warp has them, a
// batch of 8 to 10 k cycles after the quiet pass, and the next step's passes over those CRUs wait for it.  So CTAs of
// fewer than 16 warps and those of cells over one or two CTAs are split above 32 CRUs per warp, the others above 16.
// us per step at rest and amid the release, line at 16 and at 32: 76 cells of 385 to 760 CRUs over two CTAs 7.4 and
// 11.3, 4.4 and 7.3; 198 of 373 to 711 19.0 and 29.2, 12.5 and 20.3; but 38 of 672 to 989 over four 8.4 and 11.9,
// 7.8 and 13.3; one of 5,000 over 16 5.0 and 6.8, 4.1 and 7.0.
template <bool ODE64>
__device__ __forceinline__ void group_steps(const KernelArgs &a, const CtaView<false, ODE64> &v, uint64_t step0,
                                            unsigned long long &my_events, int &my_err, int &s_stop) {
    const CtaWork &w = v.w;
    const int warp = v.warp, lane = v.lane, cell = w.cell;
    const SsaConsts<float> &cc = *v.cc;
    TileRec<float> *tile = v.tile;
    const int pslot = a.max_cta_cell * kMaxWarps;
    const uint32_t rcell = (uint32_t)(a.cell_base + cell);
    // (a leader takes CRUs on its first lead_warps warps only, possibly none)
    const int nwu = max(1, v.leader ? w.lead_warps : v.n_ssa >> 5);
    const bool direct = w.cru_count <= 8 * nwu;
    const int nse = direct ? max(1, (w.cru_count + 7) >> 3) : nwu;
    const int beg = warp < nse ? (int)((int64_t)w.cru_count * warp / nse) : w.cru_count;
    const int end = warp < nse ? (int)((int64_t)w.cru_count * (warp + 1) / nse) : w.cru_count;
    for (int s = 0; s < a.n_steps; ++s) {
        const int par = s & 1;
        const int64_t ri = a.run_step0 + s;
        const bool rec = a.record_every > 0 && (ri % a.record_every) == 0;
        const int64_t r_idx = rec ? ri / a.record_every - a.rec_base : -1;
        const bool rec_ok = rec && r_idx >= 0 && r_idx < a.rec_cap;
        if (my_err & 2) continue;
        // (as in split_steps; the first two warps, or the only one, wait and build the rate table)
        const uint32_t svm = v.mbar + 16u + 8u * (uint32_t)par;
        if (threadIdx.x == 0) mbar_arrive_expect_tx(svm, (uint32_t)(kSvCount * sizeof(float)));
        const float *sv = v.svbuf + par * kSvCount;
        float2 *rtab = v.rtab + par * kRateTab;
        bool bad = false;
        if (warp < 2) {
            bad = !mbar_wait_warp(svm, (uint32_t)(s >> 1) & 1u);
            for (int e = (int)threadIdx.x; e < kRateTab; e += min(64, v.n_ssa)) build_rate_entry<float>(rtab, cc, sv, e);
        }
        if (bar_or(2, v.n_ssa, bad)) {
            my_err |= 2;
            s_stop = s;
            continue;
        }
        FluxAcc<false> acc(cc);
        if (beg < end) {
            // (a group or lane without a CRU computes along on the range's last)
            const int i = beg + (direct ? lane >> 2 : lane), m = min(i, end - 1);
            Cru<float> c;
            SsaLane<float, false> sl;
            Stream rng;
            tile_get(c, tile[m]);
            rng.open(a.seed, rcell, (uint32_t)(w.cru_begin + m), step0 + s, 0);
            sl.begin(c, cc);
            if (direct) {
                group_run(a, cc, tile, i < end ? m : -1, c, sl, rng, sv, rtab, 0u, acc, my_events, my_err);
            } else {
                StepDraw draw;
                draw.open(a.seed, rcell, step0 + s, 0);
                float u0 = Stream::u24_of(draw.word((uint32_t)(w.cru_begin + m)));
                bool live = i < end;
                int err = 0;
                while (__any_sync(0xffffffffu, live))
                    if (sl.iterate(live, c, cc, sv, rtab, rng, u0, (float)a.dt, a.event_cap, err)) live = false;
                if (i < end) {
                    tile_put(tile[m], c);
                    my_events += (unsigned long long)sl.ev;
                    my_err |= err;
                    acc.add(c.jlcc[0] + c.jlcc[1] + c.jlcc[2] + c.jlcc[3], sl.jxfer_sum, sl.jtr,
                            __popc((c.flags >> 4) & 0xFu));
                }
            }
        }
        __syncwarp();  // (the CRUs of this step are stored)
        if (rec_ok && (cell == a.tr_cell || a.tr_sums != nullptr))
            record_pass<float>(a, w, cell, r_idx, beg, end, lane, tile);
        send_partial<false, ODE64>(a, v, par, pslot, acc);
    }
}

// The FP32 SSA of a CTA with more CRUs, split by the kind of work.
//
// Quiet passes, on the first nq warps, in groups of 32 of the CTA's CRUs: every CRU through the step as
// if it had no jump (SsaLane::quiet), 32 at a time with full lanes.  A CRU that may have a
// jump is left untouched, tagged with the step and put in the CTA's queue.
// Events, on the other warps: the queued CRUs through all their iterations, in batches that a warp claims
// as they are queued: eight, each on four lanes.
// The split follows the load (quiet_warps): warp 0 sets nq of step s + 1 from the events up to step s - 2.
//
// (With both kinds in one loop, one or two lanes of a warp with an event made the other thirty walk
// through the event code, in most passes: 17 of 32 lanes active during the release.  A pass takes 2.4 k
// cycles beside eleven others, a batch 5.5 k to 8 k.  us per step, one loop before: a 12,500-CRU cell over 16
// CTAs 6.7 at rest, 10.6 amid the release, now 5.9 and 8.9; 256 mixed cells amid the release 132, now 116.
// A queue per warp run at its end costs about as much as one loop, its few lanes' event code being as long
// as all the quiet passes; one CRU per lane for the events takes twice the latency.)
//
// The quiet passes do not wait for the events of the step before: the CRUs of step s's queue are skipped
// by their tag at step s + 1 and taken last, in the queue's order, once the events of step s are through.
// Buffers: the SSA values, the rate table and the split of step s are used until the warps send their
// partials of step s, and rewritten for step s + 2, whose SSA values the leader sends only after those
// partials.  The queue of step s is used by its events, and until the quiet passes of step s + 1 are through;
// m_quiet of step s + 1 takes every warp's arrival from after both, so warp 0 has its counters, one of three
// sets, cleared in step s + 2 (for step s + 3), and its entries, one of two arrays, rewritten from then on.
// m_quiet(s): every warp arrives when its quiet passes of step s are through, its queue entries written;
// m_event(s): when it finds no more events of step s.  Two of each, by parity: the phase of step s + 2
// takes every warp's arrival in step s + 2, so a waiter is at most one phase behind and the parity tells
// the two apart.
//
// The split: of nw warps, as many take events as make the rounds of quiet passes plus the event batches per
// warp shortest, a batch counting as kBatchCost passes, for load / 8 events; the present one (nq quiet
// warps) stays unless it is an eighth longer, since a warp that comes back from the events holds the quiet
// passes up.
__device__ __forceinline__ int quiet_warps(int nw, int n_crus, int load, int lane, int nq) {
    const int groups = (n_crus + 31) / 32 + (load + 255) / 256;
    const int ne = min(lane + 1, nw >> 1);  // one choice per lane
    const int cost = 8 * ((groups + nw - ne - 1) / (nw - ne)) + kBatchCost * max(8, (load + (load >> 2)) / (8 * ne));
    const unsigned best = __reduce_min_sync(0xffffffffu, ((unsigned)cost << 5) | (unsigned)ne);
    const int now = __shfl_sync(0xffffffffu, cost, max(nw - nq - 1, 0));
    return nq > 0 && now <= (int)(best >> 5) * 9 / 8 ? nq : nw - (int)(best & 31u);
}
template <bool ODE64>
__device__ __forceinline__ void split_steps(const KernelArgs &a, const CtaView<false, ODE64> &v, uint64_t step0,
                                            unsigned long long &my_events, int &my_err, int &s_stop) {
    const CtaWork &w = v.w;
    const int warp = v.warp, lane = v.lane, cell = w.cell, nw = v.n_ssa >> 5, n_crus = w.cru_count;
    const SsaConsts<float> &cc = *v.cc;
    TileRec<float> *tile = v.tile;
    const int pslot = a.max_cta_cell * kMaxWarps;
    const float dt = (float)a.dt;
    const uint32_t rcell = (uint32_t)(a.cell_base + cell);
    uint16_t *const queues = reinterpret_cast<uint16_t *>(v.fq + 8);
    int load = n_crus >> 2;  // (warp 0) eight times the recent events per step; until known, one in 32 CRUs
    int nq = quiet_warps(nw, n_crus, load, lane, 0);
    bool bad = false;  // a wait ran out
    int slot = 0;      // s mod 3
    for (int s = 0; s < a.n_steps; ++s) {
        const int par = s & 1;
        const uint32_t ph = (uint32_t)(s >> 1) & 1u, ph_prev = (uint32_t)((s - 1) >> 1) & 1u;
        const uint32_t bars = v.mbar + 8u * (uint32_t)par, bars_prev = v.mbar + 8u * (uint32_t)(par ^ 1);
        constexpr uint32_t kSv = 16u, kQuiet = 32u, kEvent = 48u, kClear = 64u;
        if (my_err & 2) continue;
        const float *sv = v.svbuf + par * kSvCount;
        float2 *rtab = v.rtab + par * kRateTab;
        const uint32_t tag = (uint32_t)s + 2u;
        const int slot_prev = slot == 0 ? 2 : slot - 1, slot_next = slot == 2 ? 0 : slot + 1;
        uint16_t *q = queues + par * a.tile_cap;
        int *const q_put = v.fq + 2 * slot, *const q_got = q_put + 1;
        const bool quiet_warp = warp < nq;
        FluxAcc<false> acc(cc);
        int nq_next;
        if (!quiet_warp) {
            // (each of these waits for itself: they may be in different steps, the set changing with nq)
            // Whether the CTA stops is warp 0's decision, passed on as a split of 0: a warp that gave up by its own
            // clock while the quiet warps went on would be missing from a later step's bar_or.  So this wait is
            // longer than all that warp 0 may wait through before it arrives (four waits).
            if (lane == 0) mbar_arrive(bars + kQuiet);
            const bool told = mbar_wait_warp(bars + kClear, ph, 8 * kWaitCycles);
            nq_next = told ? v.fq[6 + (par ^ 1)] : 0;
            if (nq_next == 0) {
                my_err |= 2;
                continue;
            }
        } else {
            // The SSA values of step s arrive by st.async from the leader's ODE warps and complete this
            // CTA's mbarrier of parity par (thread 0 declares the bytes; that mbarrier's previous phase,
            // step s-2's, completed before this CTA's waits of step s-2).  The quiet warps meet at named
            // barrier 2 (bar_or below) and take the waits' outcome together: after a wait has run out
            // the CTA stops for the rest of the launch (no more sends), so that its partners stop too.
            if (threadIdx.x == 0) mbar_arrive_expect_tx(bars + kSv, (uint32_t)(kSvCount * sizeof(float)));
            // (the first warp alone waits and builds the rate table: a waiting warp's polling takes issue
            // slots, a warp at a named barrier none)
            if (warp == 0) {
                bad |= !mbar_wait_warp(bars + kSv, ph);
                // (with the split a group may pass to another warp, and its last one may take events now)
                if (s > 0) bad |= !mbar_wait_warp(bars_prev + kQuiet, ph_prev);
                // the split of step s + 1, from the events of step s - 2
                const int n_events = v.fq[2 * slot_next] & 0xFFFF;
                load = s < 2 ? load : (s == 2 ? 8 * n_events : load + n_events - (load >> 3));
                const int nq1 = quiet_warps(nw, n_crus, load, lane, s <= 2 ? 0 : nq);
                __syncwarp();
                if (lane == 0) v.fq[6 + (par ^ 1)] = nq1;
                if (lane == 0) v.fq[2 * slot_next] = v.fq[2 * slot_next + 1] = 0;
                for (int e = lane; e < kRateTab; e += 32) build_rate_entry<float>(rtab, cc, sv, e);
            }
            const bool stop = bar_or(2, nq * 32, bad);
            if (threadIdx.x == 0) {
                if (stop) v.fq[6 + (par ^ 1)] = 0;
                mbar_arrive(bars + kClear);  // to the event warps
            }
            if (stop) {
                my_err |= 2;
                s_stop = s;
                continue;
            }
            nq_next = v.fq[6 + (par ^ 1)];
            StepDraw draw;
            draw.open(a.seed, rcell, step0 + s, 0);
            // The CTA's groups of 32, without the CRUs of step s-1's queue, then the groups of those, in turn
            // to the quiet warps.
            const int n_own = (n_crus + 31) >> 5, n_late = s > 0 ? v.fq[2 * slot_prev] & 0xFFFF : 0;
            const uint16_t *q_prev = queues + (par ^ 1) * a.tile_cap;
            bool waited = false;
            for (int g = warp; g < n_own + ((n_late + 31) >> 5); g += nq) {
                const bool late = g >= n_own;
                int m = 32 * g + lane;
                if (late) {
                    if (!waited) bad |= !mbar_wait_warp(bars_prev + kEvent, ph_prev);
                    waited = true;
                    m -= 32 * n_own;
                    m = m < n_late ? (int)q_prev[m] : -1;
                } else if (m >= n_crus) {
                    m = -1;
                }
                // (a lane without a CRU computes along on the CTA's first: no branch in the pass)
                Cru<float> c;
                SsaLane<float, false> sl;
                TileRec<float> &rec_m = tile[max(m, 0)];
                tile_get(c, rec_m);
                // (its group's pass may reach a CRU of step s-1's queue before or after that was taken here)
                const bool valid = m >= 0 && (late || tile_tag(rec_m) < tag - 1u);
                sl.begin(c, cc);
                const bool quiet = sl.quiet(c, cc, sv, rtab, draw.word((uint32_t)(w.cru_begin + m)), dt);
                const bool done = valid && quiet, jumps = valid && !quiet;
                if (done) tile_put_quiet(rec_m, c, late ? tag - 1u : 0u);
                acc.add(done ? c.jlcc[0] + c.jlcc[1] + c.jlcc[2] + c.jlcc[3] : 0.f, done ? sl.jxfer_sum : 0.f,
                        done ? sl.jtr : 0.f, done ? __popc((c.flags >> 4) & 0xFu) : 0);
                const unsigned em = __ballot_sync(0xffffffffu, jumps);
                if (em == 0u) continue;
                // into the queue: slots reserved, written, then counted as written
                const int ne = __popc(em);
                int q0 = 0;
                if (lane == 0) q0 = atomicAdd(q_put, ne << 16) >> 16;
                q0 = __shfl_sync(0xffffffffu, q0, 0);
                if (jumps) {
                    tile_tag(rec_m) = tag;
                    q[q0 + __popc(em & ((1u << lane) - 1u))] = (uint16_t)m;
                }
                __threadfence_block();
                __syncwarp();
                if (lane == 0) atomicAdd(q_put, ne);
            }
            // the warp's queue entries and CRUs are stored
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + kQuiet);
        }
        while (!quiet_warp) {
            // The next batch, claimed by lane 0 for the warp (bounded: the quiet warps arrive, or their own
            // wait ran out).  Every lane polls, with the loop's branches on votes: see mbar_wait_warp.
            int h = -1, n = 0;
            const long long t0 = clock64();
            for (;;) {
                const bool fin = __all_sync(0xffffffffu, mbar_test(bars + kQuiet, ph));
                if (lane == 0) {
                    const int word = *(volatile int *)q_put, head = *(volatile int *)q_got;
                    const int written = (word & 0xFFFF) == (word >> 16) ? word & 0xFFFF : 0;
                    n = written - head;
                    n = n >= 8 || fin ? min(n, 8) : 0;
                    if (n > 0 && atomicCAS(q_got, head, head + n) == head) h = head;
                }
                h = __shfl_sync(0xffffffffu, h, 0);
                n = __shfl_sync(0xffffffffu, n, 0);
                if (h >= 0 || (fin && n <= 0)) break;
                if (n <= 0) __nanosleep(20);
                if (__any_sync(0xffffffffu, clock64() - t0 > (1ll << 32))) {
                    bad = true;
                    break;
                }
            }
            if (h < 0) break;
            __threadfence_block();
            // (a group without a CRU holds, and computes along on, the batch's last)
            const int i = lane >> 2;
            int m = q[h + min(i, n - 1)];
            Cru<float> c;
            SsaLane<float, false> sl;
            Stream rng;
            tile_get(c, tile[m]);
            rng.open(a.seed, rcell, (uint32_t)(w.cru_begin + m), step0 + s, 0);
            sl.begin(c, cc);
            if (i >= n) m = -1;
            group_run(a, cc, tile, m, c, sl, rng, sv, rtab, tag, acc, my_events, my_err);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bars + kEvent);
        const int64_t ri = a.run_step0 + s;
        if (quiet_warp && a.record_every > 0 && (ri % a.record_every) == 0 && (cell == a.tr_cell || a.tr_sums != nullptr)) {
            // records of this step, from the warp's part of the tile at the end of the step
            const int64_t r_idx = ri / a.record_every - a.rec_base;
            if (r_idx >= 0 && r_idx < a.rec_cap) {
                bad |= !mbar_wait_warp(bars + kEvent, ph);
                const int beg = (int)((int64_t)n_crus * warp / nq), end = (int)((int64_t)n_crus * (warp + 1) / nq);
                record_pass<float>(a, w, cell, r_idx, beg, end, lane, tile);
                // The quiet warps meet again: one that takes events in step s + 1 is not in that step's bar_or,
                // and nothing else keeps the first writes of step s + 1 (which come after warp 0's arrival there,
                // those of event warps by m_clear) behind its reads.  All of them are here: the record step and
                // the split are the same for the CTA's quiet warps.  A barrier of its own, since a warp that
                // turns quiet may be waiting in the next bar_or already; no two uses of it overlap, because a
                // warp comes to the next one only through a bar_or that warp 0 is in.
                rec_bar(nq * 32);
            }
        }
        send_partial<false, ODE64>(a, v, par, pslot, acc);
        nq = nq_next;
        slot = slot_next;
    }
    if (bad) my_err |= 2;
}

// The SSA warps over a launch (every warp of a CTA that is not a leader's ODE warp, and every
// warp of an idle CTA, which only keeps the closing cluster barrier): per global step the SSA of
// the warp's CRUs, the record pass and the flux partials (FP32: group_steps or split_steps), and the
// tile back to the cell's planes at the end.  Inlined into the kernel (out of line it spills).
template <bool FP64, bool ODE64>
__device__ __forceinline__ void ssa_warps(const KernelArgs &a, uint64_t step0) {
    using R = typename std::conditional<FP64, double, float>::type;
    const CtaView<FP64, ODE64> v(a);
    const CtaWork &w = v.w;
    const int warp = v.warp, lane = v.lane, cell = w.cell, n_ssa = v.n_ssa;
    const SsaConsts<R> &cc = *v.cc;
    TileRec<R> *tile = v.tile;
    const int pslot = a.max_cta_cell * kMaxWarps;  // warp partials per parity slot
    const R dt = (R)a.dt;
    unsigned long long my_events = 0;
    int my_err = 0;  // bit 0: a CRU hit the event cap; bit 1: a wait for the SSA values ran out
    int s_stop = -1;  // the step whose wait ran out
    if constexpr (FP64) {
        for (int s = 0; s < a.n_steps; ++s) {
            const int par = s & 1;
            const int64_t ri = a.run_step0 + s;
            const bool rec = a.record_every > 0 && (ri % a.record_every) == 0;
            const int64_t r_idx = rec ? ri / a.record_every - a.rec_base : -1;
            const bool rec_ok = rec && r_idx >= 0 && r_idx < a.rec_cap;
            if (v.active && !(my_err & 2)) {
                // The SSA values of step s arrive by st.async from the leader's ODE warps and complete
                // this CTA's mbarrier of parity par (thread 0 declares the bytes; that mbarrier's
                // previous phase, step s-2's, completed before this CTA's waits of step s-2).  The
                // CTA's SSA threads then meet at named barrier 2 (bar_or below; the CTAs of a cell are
                // held together only by their data) and take the wait's outcome together: after a
                // wait has run out the CTA stops for the rest of the launch (no more sends), so that
                // its partners stop too.
                const uint32_t svm = v.mbar + 16u + 8u * (uint32_t)par;
                if (threadIdx.x == 0) mbar_arrive_expect_tx(svm, (uint32_t)(kSvCount * sizeof(R)));
                const bool ok = mbar_wait_warp(svm, (uint32_t)(s >> 1) & 1u);
                const R *sv = v.svbuf + par * kSvCount;
                // Float copies of the step's SSA values for the screen, in the rate-table area of this
                // parity (floats 0..kSvCount-1), before bar_or(2) of step s, which publishes them.  No reader
                // of that area (step s-2's) can remain: every SSA thread passed bar_or of step s-1 after its
                // last iteration of step s-2.  A warp still in step s-1 reads the other one.
                float2 *rtab = v.rtab + par * kRateTab;
                float *svf = reinterpret_cast<float *>(rtab);
                const float *sk = reinterpret_cast<const float *>(v.rtab) + 64;
                for (int e = (int)threadIdx.x; e < kSvCount; e += n_ssa) svf[e] = (float)sv[e];
                if (bar_or(2, n_ssa, !ok)) {
                    my_err |= 2;
                    s_stop = s;
                    continue;
                }
                const int nsw = n_ssa >> 5;
                // This warp's CRUs [beg, end), four lanes each (grouped) or one.
                // (a leader takes CRUs on its first lead_warps SSA warps only, possibly none)
                const bool grouped = w.cru_count <= kGroupCrusFp64;
                const int per = grouped ? 8 : 32;
                // (no more warps than the rounds take: they share the sub-partitions' FP64 pipes)
                const int fills = (w.cru_count + per - 1) / per, nwu = max(1, v.leader ? w.lead_warps : nsw);
                const int rounds = max(1, (fills + nwu - 1) / nwu);
                const int nse = grouped ? max(1, (fills + rounds - 1) / rounds) : max(1, min(nwu, fills));
                const int beg = warp < nse ? (int)((int64_t)w.cru_count * warp / nse) : w.cru_count;
                const int end = warp < nse ? (int)((int64_t)w.cru_count * (warp + 1) / nse) : w.cru_count;
                FluxAcc<FP64> acc;
                Cru<R> c;
                SsaLane<R, true> sl;
                Stream rng;
                const int jq = lane & 3, base = lane & ~3;
                auto load = [&](int mm) {
                    tile_get(c, tile[mm]);
                    rng.open(a.seed, (uint32_t)(a.cell_base + cell), (uint32_t)(w.cru_begin + mm), step0 + s, 0);
                    sl.begin_group(c, cc);
                };
                auto store = [&](int mm, int err) {  // (a group's on its first lane)
                    tile_put(tile[mm], c);
                    my_events += (unsigned long long)sl.ev;
                    my_err |= err;
                    acc.add(c.jlcc[0] + c.jlcc[1] + c.jlcc[2] + c.jlcc[3], sl.jxfer_sum, sl.jtr,
                            __popc((c.flags >> 4) & 0xFu));
                };
                {
                    // Pass 1: the warp's CRUs.  One whose first iteration the FP32 screen shows to be the step's
                    // last runs without the FP64 rates (finish); the others (an event in the step) go,
                    // untouched in the tile, to the CTA's queue.
                    int *qn = v.fq + par;
                    int *q = v.fq + 4;
                    if (threadIdx.x == 0) v.fq[par ^ 1] = 0;  // step s-1's count: every reader has passed
                                                              // bar_or(2) of this step
                    for (int b = beg; grouped && b < end; b += 8) {
                        // (a group without a CRU holds, and computes along on, the range's last)
                        const int mb = b + (lane >> 2), m = min(mb, end - 1);
                        load(m);
                        const bool last = sl.surely_last_group(c, cc, sk, svf, rng, dt) && mb < end;
                        sl.finish_group(last, c, cc, sv, rng, dt);
                        if (last && jq == 0) store(m, 0);
                        int qs = 0;
                        if (!last && mb < end && jq == 0) {
                            qs = atomicAdd(qn, 1);
                            if (qs < kEngQCap) q[qs] = m;
                        }
                        bool more = __shfl_sync(0xffffffffu, qs, base) >= kEngQCap;
                        while (__any_sync(0xffffffffu, more)) {  // the queue is full
                            int err = 0;
                            if (sl.iterate_group(more, c, cc, sv, rng, dt, a.event_cap, err) && more) {
                                if (jq == 0) store(m, err);
                                more = false;
                            }
                        }
                    }
                    // One per lane: a lane whose CRU is done takes the warp's next one.
                    int m = grouped ? -2 : -1;  // CRU of this lane; -1 none yet, -2 none left
                    int cursor = beg;
                    bool fresh = false;
                    while (!grouped) {
                        const unsigned need = __ballot_sync(0xffffffffu, m == -1);
                        if (need) {
                            const int nm = cursor + __popc(need & ((1u << lane) - 1u));
                            cursor += __popc(need);
                            if (m == -1) {
                                if (nm < end) {
                                    m = nm;
                                    tile_get(c, tile[m]);
                                    rng.open(a.seed, (uint32_t)(a.cell_base + cell), (uint32_t)(w.cru_begin + m),
                                             step0 + s, 0);
                                    sl.begin(c, cc);
                                    fresh = true;
                                } else {
                                    m = -2;
                                }
                            }
                        }
                        if (!__any_sync(0xffffffffu, m >= 0)) break;
                        if (m >= 0) {
                            int err = 0;
                            bool done = false;
                            if (sl.surely_last(c, cc, sk, svf, rng, dt)) {
                                sl.finish(c, cc, sv, rng, dt);
                                done = true;
                            } else {
                                const int qs = fresh ? atomicAdd(qn, 1) : kEngQCap;
                                if (qs < kEngQCap) {
                                    q[qs] = m;
                                    m = -1;
                                } else {  // the queue is full, or the CRU is past its first iteration
                                    done = sl.iterate(c, cc, sv, rng, dt, a.event_cap, err);
                                }
                            }
                            fresh = false;
                            if (done) {
                                store(m, err);
                                m = -1;
                            }
                        }
                    }
                    // Pass 2: the queued CRUs on four lanes each, eight per warp at a time, over the CTA's SSA
                    // warps.
                    ssa_bar(n_ssa);
                    const int nq = min(*qn, kEngQCap);
                    const int nw2 = min(nsw, (nq + 7) >> 3);
                    if (warp < nw2) {
                        int qc = (int)((int64_t)nq * warp / nw2);
                        const int qe = (int)((int64_t)nq * (warp + 1) / nw2);
                        m = -1;  // the group's CRU
                        bool first = false;
                        for (;;) {
                            const unsigned need = __ballot_sync(0xffffffffu, m == -1 && jq == 0);
                            if (need) {
                                const int nm = qc + __popc(need & ((1u << base) - 1u));
                                qc += __popc(need);
                                const Cru<R> c0 = c;
                                const SsaLane<R, true> sl0 = sl;
                                const Stream rng0 = rng;
                                const int mq = q[min(nm, qe - 1)];
                                load(mq);  // (a group without one holds the range's last)
                                if (m == -1) {
                                    first = true;
                                    m = nm < qe ? mq : -2;
                                } else {
                                    c = c0;
                                    sl = sl0;
                                    rng = rng0;
                                }
                            }
                            if (!__any_sync(0xffffffffu, m >= 0)) break;
                            int err = 0;
                            const bool last = sl.surely_last_group(c, cc, sk, svf, rng, dt) && m >= 0 && !first;
                            bool done = last;
                            if (__any_sync(0xffffffffu, last)) sl.finish_group(last, c, cc, sv, rng, dt);
                            const bool more = m >= 0 && !last;
                            if (__any_sync(0xffffffffu, more))
                                done |= sl.iterate_group(more, c, cc, sv, rng, dt, a.event_cap, err) && more;
                            first = false;
                            if (done) {
                                if (jq == 0) store(m, err);
                                m = -1;
                            }
                        }
                    }
                    // the records read the warps' tile ranges, which pass 2 may have written elsewhere
                    if (rec_ok && (cell == a.tr_cell || a.tr_sums != nullptr)) ssa_bar(n_ssa);
                }
                // Records of this step, from the warp's part of the tile (now at the end of the step)
                if (rec_ok && (cell == a.tr_cell || a.tr_sums != nullptr))
                    record_pass<R>(a, w, cell, r_idx, beg, end, lane, tile);
                send_partial<FP64, ODE64>(a, v, par, pslot, acc);
            }
        }
    } else if (v.active) {
        if (v.grouped)
            group_steps<ODE64>(a, v, step0, my_events, my_err, s_stop);
        else
            split_steps<ODE64>(a, v, step0, my_events, my_err, s_stop);
    }
    // A CTA that stopped at step s_stop may still receive the SSA values of steps s_stop and
    // s_stop + 1, stores the leader issued before it stopped in turn (it pushes step s + 2 only
    // after this CTA's partials of step s, which a stopped CTA does not send).  Nothing orders the
    // landing of an st.async with the closing cluster barrier; its completion shows only on the
    // receiving mbarrier.  So thread 0 waits, bounded, for those two phases before the barrier
    // (declaring the bytes of step s_stop + 1, whose phase was not declared yet): no store into
    // this CTA's shared memory is in flight when it exits.
    if ((my_err & 2) && threadIdx.x == 0 && s_stop >= 0) {
        const uint32_t m0 = v.mbar + 16u + 8u * (uint32_t)(s_stop & 1);
        mbar_wait(m0, (uint32_t)(s_stop >> 1) & 1u);
        if (s_stop + 1 < a.n_steps) {
            const uint32_t m1 = v.mbar + 16u + 8u * (uint32_t)((s_stop + 1) & 1);
            mbar_arrive_expect_tx(m1, (uint32_t)(kSvCount * sizeof(R)));
            mbar_wait(m1, (uint32_t)((s_stop + 1) >> 1) & 1u);
        }
    }
    // the launch's one closing cluster barrier (every thread of every CTA of the cluster)
    cluster_arrive();
    cluster_wait();
    if (!v.active) return;
    // the tile back to the cell's planes
    R *g_cass = reinterpret_cast<R *>(a.cass);
    R *g_jlcc = reinterpret_cast<R *>(a.jlcc);
    R *g_cajsr = reinterpret_cast<R *>(a.cajsr);
    const int64_t base = a.slot0[cell] + w.cru_begin;
    for (int m = (int)threadIdx.x; m < w.cru_count; m += n_ssa) {
        const int64_t gs = base + m;
        Cru<R> c;
        tile_get(c, tile[m]);
        a.lcc[gs] = c.lcc;
        a.flags[gs] = c.flags;
#pragma unroll
        for (int k = 0; k < 6; ++k) a.ryr[k * a.n_slots + gs] = c.ryr[k];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            g_cass[j * a.n_slots + gs] = c.cass[j];
            g_jlcc[j * a.n_slots + gs] = c.jlcc[j];
        }
        g_cajsr[gs] = c.cajsr;
        if (!FP64) a.cajsr_lo[gs] = c.cajsr_lo;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        my_events += __shfl_xor_sync(0xffffffffu, my_events, o);
        my_err |= __shfl_xor_sync(0xffffffffu, my_err, o);
    }
    if (lane == 0) {
        if (my_events) atomicAdd(a.events, my_events);
        if (my_err) atomicCAS(&a.status[cell], 0, (my_err & 2) ? (int)GW_ERR_SYNC_TIMEOUT : (int)GW_ERR_EVENT_CAP);
    }
}

// The engine kernel: every CTA of a cluster initialises its mbarriers and waits for the whole
// cluster to be resident (it writes into the other CTAs' shared memory from its first global step
// on), loads its CRU tile and the cell's SSA constants, then splits into the ODE warps of a leader
// CTA and the SSA warps.  Both parts end with one more cluster barrier, so that no CTA exits
// while another may still write into its shared memory.
template <bool FP64, bool ODE64>
__global__ void __launch_bounds__(FP64 ? kMaxThreadsFp64 : kMaxThreads, 1) engine_kernel(const __grid_constant__ KernelArgs a) {
    using R = typename std::conditional<FP64, double, float>::type;
    const CtaView<FP64, ODE64> v(a);
    // The partials' mbarriers (one arrival per phase: the ODE thread's expect_tx) are initialised
    // before the cluster barrier that every CTA passes before its first remote write.
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 4; ++i) mbar_init(v.mbar + 8u * i, 1);
        if (!FP64) {
            for (uint32_t i = 0; i < 2; ++i) {
                mbar_init(v.mbar + 32u + 8u * i, (uint32_t)(v.n_ssa >> 5));
                mbar_init(v.mbar + 48u + 8u * i, (uint32_t)(v.n_ssa >> 5));
                mbar_init(v.mbar + 64u + 8u * i, 1);
            }
        }
        mbar_fence_init();
    }
    cluster_arrive();
    cluster_wait();
    uint64_t step0 = 0;
    if (v.active) {
        const int cell = v.w.cell;
        if (threadIdx.x == 0) {
            load_ssa_consts<R>(*v.cc, a.cs[cell]);
            // FP64: the screen's constants (SsaLane::surely_last) in the rate-table area, which the
            // FP64 lane does not otherwise use: floats 64.. of parity 0's table
            if (FP64) {
                load_screen_consts(reinterpret_cast<float *>(v.rtab) + 64, a.cs[cell]);
                v.fq[0] = 0;
                v.fq[1] = 0;
            }
        }
        if (!FP64 && threadIdx.x < 8) v.fq[threadIdx.x] = 0;
        // The leader's warp-partial slots start at zero (slots of warps a CTA does not have stay
        // so); the cell's CTAs write them only after the first cluster barrier of the steps.
        if (v.leader) {
            uint4 *pz = reinterpret_cast<uint4 *>(v.part);
            const int nz = 2 * a.max_cta_cell * kMaxWarps * kPartBytes<FP64> / 16;
            for (int i = (int)threadIdx.x; i < nz; i += (int)blockDim.x) pz[i] = make_uint4(0u, 0u, 0u, 0u);
        }
        step0 = a.dyn[cell].step;
        if (!v.ode_thread) {
            R *g_cass = reinterpret_cast<R *>(a.cass);
            R *g_jlcc = reinterpret_cast<R *>(a.jlcc);
            R *g_cajsr = reinterpret_cast<R *>(a.cajsr);
            const int64_t base = a.slot0[cell] + v.w.cru_begin;
            for (int m = (int)threadIdx.x; m < v.w.cru_count; m += v.n_ssa) {
                const int64_t gs = base + m;
                Cru<R> c;
                c.lcc = a.lcc[gs];
                c.flags = a.flags[gs];
#pragma unroll
                for (int k = 0; k < 6; ++k) c.ryr[k] = a.ryr[k * a.n_slots + gs];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    c.cass[j] = g_cass[j * a.n_slots + gs];
                    c.jlcc[j] = g_jlcc[j * a.n_slots + gs];
                }
                c.cajsr = g_cajsr[gs];
                c.cajsr_lo = FP64 ? 0.f : a.cajsr_lo[gs];
                tile_put(v.tile[m], c);
            }
        }
    }
    __syncthreads();
    if (v.ode_thread)
        ode_warps<FP64, ODE64>(a, step0);
    else
        ssa_warps<FP64, ODE64>(a, step0);
}

// Random initial CRU state (GW_utils.tpp:5-64) from stream 1, one thread per CRU, in the same
// draw order as the oracle's orc_sample_initial_crus.
template <bool FP64>
__global__ void init_crus_kernel(const KernelArgs a, int cell, int ncru) {
    using R = typename std::conditional<FP64, double, float>::type;
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= ncru) return;
    Stream s;
    s.open(a.seed, (uint32_t)(a.cell_base + cell), (uint32_t)i, 0, 1);
    uint32_t k = 0;
    auto pick = [&](const double *w, int n) {
        const double u = FP64 ? s.u53(k) : (double)s.u24(k);
        ++k;
        double cum = w[0];
        int idx = 0;
        while (cum < u && idx < n - 1) {
            ++idx;
            cum += w[idx];
        }
        return idx;
    };
    const double wl[3] = {0.958, 0.038, 0.004};
    const double wi[2] = {0.9425, 0.0575};
    const double wr[3] = {0.609, 0.5 * 0.391, 0.5 * 0.391};
    const double wc[2] = {0.998, 0.002};
    const int lcc_of[3] = {1, 2, 7};
    const int ryr_of[3] = {0, 4, 5};
    uint32_t lcc = 0, flags = 0, ryr[6] = {0, 0, 0, 0, 0, 0};
    for (int j = 0; j < 4; ++j) lcc = byte_set(lcc, j, lcc_of[pick(wl, 3)]);
    for (int j = 0; j < 4; ++j)
        if (pick(wi, 2) == 0) flags |= (1u << j);
    for (int j = 0; j < 4; ++j)
        for (int q = 0; q < 5; ++q) {
            const int st = ryr_of[pick(wr, 3)];
#pragma unroll
            for (int z = 0; z < 6; ++z)
                if (z == st) ryr[z] = byte_add(ryr[z], j, 1);
        }
    for (int j = 0; j < 4; ++j)
        if (pick(wc, 2) == 1) flags |= (1u << (4 + j));
    const int64_t gs = a.slot0[cell] + i;
    a.lcc[gs] = lcc;
    a.flags[gs] = flags;
    for (int z = 0; z < 6; ++z) a.ryr[z * a.n_slots + gs] = ryr[z];
    R *cass = reinterpret_cast<R *>(a.cass);
    R *jlcc = reinterpret_cast<R *>(a.jlcc);
    for (int j = 0; j < 4; ++j) {
        cass[j * a.n_slots + gs] = (R)1.45370e-4;
        jlcc[j * a.n_slots + gs] = (R)0;
    }
    reinterpret_cast<R *>(a.cajsr)[gs] = (R)0.908408;
    if (!FP64) a.cajsr_lo[gs] = (float)(0.908408 - (double)(float)0.908408);
}

template <bool FP64, bool ODE64>
inline cudaError_t set_attrs(size_t smem) {
    auto k = engine_kernel<FP64, ODE64>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

inline cudaLaunchConfig_t launch_cfg(const LaunchShape &s, void *stream, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)s.ctas, 1, 1);
    cfg.blockDim = dim3((unsigned)s.threads, 1, 1);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = (cudaStream_t)stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <bool FP64>
inline int launch_engine(const KernelArgs &a, const LaunchShape &s, void *stream, bool ode64) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = launch_cfg(s, stream, attr);
    cudaError_t e;
    if constexpr (FP64) {
        (void)ode64;
        e = set_attrs<true, true>(s.smem);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, engine_kernel<true, true>, a);
    } else if (ode64) {
        e = set_attrs<false, true>(s.smem);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, engine_kernel<false, true>, a);
    } else {
        e = set_attrs<false, false>(s.smem);
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, engine_kernel<false, false>, a);
    }
    return (int)e;
}

template <bool FP64>
inline int max_active_clusters(const LaunchShape &s, bool ode64, int *out) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = launch_cfg(s, nullptr, attr);
    cudaError_t e;
    if constexpr (FP64) {
        (void)ode64;
        e = set_attrs<true, true>(s.smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(out, engine_kernel<true, true>, &cfg);
    } else if (ode64) {
        e = set_attrs<false, true>(s.smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(out, engine_kernel<false, true>, &cfg);
    } else {
        e = set_attrs<false, false>(s.smem);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(out, engine_kernel<false, false>, &cfg);
    }
    return (int)e;
}

}  // namespace dev
}  // namespace gw
