// gw_ode_program.h -- the global step (GW_model::euler_step, GW.tpp:237-272) as a SIMT "lane
// program" for the ODE warps of a cell's leader CTA.
//
// GB300 runs an FP64 instruction in ~34 ns per warp whether 1 or 32 lanes are active, so the
// reference's ~1400 scalar FP64 operations per step cannot be run by one thread.  The step is
// instead split into dependency phases; every op of a phase evaluates the same formula shape on
// operands picked from a slot array X[] by per-op indices, one op per lane (128 lanes = 4 warps).
// Three phases: the increments with the Euler update, the transcendental terms of the new state, and
// quotients and rate sums of those; an increment is a sum of products of two slots, so that the
// product of two quotients, or of a quotient and a driving force, needs no phase of its own.
// Reassociation changes results at the level of a few ulp, far inside the 1e-12 relative FP64 parity
// bound.
#pragma once

#include <cstdint>

#include "gw_internal.h"

namespace gw {

enum OdeKind : uint8_t {
    OK_NOP = 0,
    OK_LOG,   // out = (X[a2] + X[a3]) + X[a4] * log(X[a0] + X[a1]*X[a5])
    OK_EXP,   // out = X[a4] + X[a0] * exp(X[a1]*X[a2] + X[a3])
    OK_POW,   // out = X[a3] + X[a0]*X[a1] * X[a2]^(1/2), or ^(3/4) when width = 2
    OK_QUOT,  // out = X[a0] * (X[a1] + X[a2]*X[a3]) / (X[a4] + X[a5]*X[a6])
    OK_SUM3,  // out = X[a0]*X[a1] + X[a2]*X[a3] + X[a4]*X[a5]
    OK_DOT,   // row of `width` lanes: the increment of global `out` is X[a0] times the sum over lanes and
              // t < 4 of s_t X[a(1+2t)] X[a(2+2t)], s_t = -1 where bit 15 of a(1+2t) is set; the row's
              // first lane adds X[a9]*X[a10] + X[a11]*X[a12] (the flux sums) and, once every row has
              // read the old globals, updates g[out] (FP64 state) and X[XS_G + out]
};
constexpr uint16_t kOdeNeg = 0x8000;  // sign bit of an OK_DOT factor

struct OdeOp {
    uint8_t kind;
    uint8_t width;   // OK_DOT: lanes in the row (1, 2, 4 or 8), the row's first lane writes; OK_POW: see there
    uint16_t out;
    uint16_t a[14];
};
static_assert(sizeof(OdeOp) == 32, "OdeOp layout");

constexpr int kOdeWarps = 4;
constexpr int kOdeLanes = 32 * kOdeWarps;
constexpr int kOdeMaxPhases = 8;
constexpr int kOdeMaxOps = 448;
constexpr int kOdeMaxAlt = 24;
constexpr int kOdeMaxSlots = 640;
constexpr int kOdeMaxConsts = kOdeConstCap;

// Fixed slots of X[].
enum OdeSlot : uint16_t {
    XS_ZERO = 0,
    XS_ONE = 1,
    XS_MONE = 2,
    XS_G = 3,                        // 36 globals (gw_globals order)
    XS_SUMS = XS_G + kNumGlobals,    // JLCC, ClCh, Jtr, Jxfer sums of the previous step
    XS_ISTIM = XS_SUMS + 4,
    XS_DT = XS_ISTIM + 1,
    XS_FIRST_FREE = XS_DT + 1,
};

// Per-step SSA values pushed to the CTAs (sv[]) that come from the program, by sv index.
struct alignas(16) OdeProgram {
    int n_phases;
    int phase_begin[kOdeMaxPhases + 1];  // ops [phase_begin[p], phase_begin[p+1]) of phase p (<= 128)
    int upd_phase;                       // phase of the increments and the update (OK_DOT rows): 0
    int push_phase;                      // sv are pushed after this phase (the last one)
    int n_slots;
    int const_begin, n_consts;           // per-cell constants occupy X[const_begin, +n_consts)
    int n_alt;
    uint16_t sv_src[kSvCount];           // X slot of each sv value (XS_ZERO if not produced)
    uint8_t alt_idx[kOdeMaxOps];         // 255, or index of the op's variant in alt[regime-1]
    uint8_t sv_stage[kOdeMaxOps];        // 1 + the sv index an op's output is staged to for the push, or 0
    OdeOp ops[kOdeMaxOps];               // regime 0: V >= -40
    OdeOp alt[2][kOdeMaxAlt];            // regime 1: V < -40;  regime 2: V == -47.13
};
static_assert(sizeof(OdeProgram) % 16 == 0, "OdeProgram is copied in 16-byte words");

// Builds the program shared by all cells (pow_fast: all cells have Hf == Hr == 0.75, so the
// Jup powers are taken with square roots; else a fourth phase exponentiates their logarithms) and the
// per-cell constant values.
bool ode_program_build(const CellStatic &cs, bool pow_fast, OdeProgram *prog, double *consts);

// Host evaluation of one global step (FP64) in the device's operation order.
void ode_program_step_host(const OdeProgram &P, const double *consts, double *g, const double *sums,
                           double Istim, double dt, double *sv);

}  // namespace gw
