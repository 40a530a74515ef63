// gw_ode_program.cpp -- builds the SIMT lane program of the global step (see gw_ode_program.h).
//
// Every term below restates GW_model::euler_step (GW.tpp:237-272) and the functions it calls
// (update_V_and_concentration_derivatives GW.tpp:171-212, update_QKr/QKv GW.tpp:26-44/65-123,
// update_*_derivatives GW.tpp:127-168, the currents of common.hpp:70-218 and GW_utils.hpp:273-375,
// and the per-step constants of GW_model::SSA GW.tpp:216-221), rearranged into
//   phase E  DOT  : increments of the 36 globals (sums of products of two slots) and the Euler update
//                   g += dg (FP64) by each row's first lane, once every row has read the old globals
//   phase A  LOG | EXP | POW : transcendental terms of the new globals, each with its scale and offset
//                   (driving forces V - E, denominators 1 + exp(..), LCC rates)
//   phase P  EXP  : (only with general Jup exponents) exp(H log(Ca / K))
//   phase B  QUOT | SUM3 : quotients of those (conductances, gate rates, inactivation rates, JLCC
//                   factor) and sums of three products (rate times coefficient, total outgoing rates
//                   of the Markov states)
// The per-step SSA values are pushed after phase B.  Three V regimes select the branches of the
// gate rates (common.hpp:176-218): 0: V >= -40, 1: V < -40, 2: V == -47.13.
#include "gw_ode_program.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <utility>
#include <string>
#include <vector>

namespace gw {
namespace {

constexpr double kF = 96.5;  // common.hpp:9

struct Builder {
    const CellStatic &C;
    const gw_params &p;
    bool fast;
    int regime;
    double *consts;
    int const_begin;
    int nconst = 0;
    int next = XS_FIRST_FREE + kOdeMaxConsts;  // intermediates after the constant block
    std::vector<std::vector<OdeOp>> ph;
    std::vector<int> cursor;
    uint16_t sv_src[kSvCount];

    Builder(const CellStatic &c, bool f, int r, double *k)
        : C(c), p(c.p), fast(f), regime(r), consts(k), const_begin(XS_FIRST_FREE) {
        for (auto &s : sv_src) s = XS_ZERO;
    }

    // per-cell constant (allocated in call order, identical for every cell and regime)
    uint16_t K(double v) {
        const int i = nconst++;
        if (consts && i < kOdeMaxConsts) consts[i] = v;
        return (uint16_t)(const_begin + i);
    }
    // literal constant (same value for every cell): shared slot
    std::vector<std::pair<double, uint16_t>> lits;
    uint16_t KL(double v) {
        for (auto &l : lits)
            if (l.first == v) return l.second;
        const uint16_t s = K(v);
        lits.push_back({v, s});
        return s;
    }
    uint16_t S() { return (uint16_t)next++; }
    uint16_t G(int i) const { return (uint16_t)(XS_G + i); }
    void phase(int n) {
        ph.assign(n, {});
        cursor.assign(n, 0);
    }
    // start a new kind group at the next warp boundary of phase q
    void warp_align(int q) {
        auto &v = ph[q];
        while (v.size() % 32 != 0) v.push_back(OdeOp{OK_NOP, 1, 0, {}});
    }
    void emit(int q, uint8_t kind, uint16_t out, std::initializer_list<uint16_t> args, int width = 1) {
        auto &v = ph[q];
        while (v.size() % width != 0) v.push_back(OdeOp{OK_NOP, 1, 0, {}});
        OdeOp op{};
        op.kind = kind;
        op.width = (uint8_t)width;
        op.out = out;
        int i = 0;
        for (uint16_t a : args) op.a[i++] = a;
        for (; i < 14; ++i) op.a[i] = XS_ZERO;
        v.push_back(op);
    }
    // DOT row: increment of global out = s0 * sum(+-x * y), terms padded to 4 per lane, the terms of
    // the flux sums (at most two, with constant or phase-B factors) apart
    struct Term {
        uint16_t x, y;
    };
    void row(int q, uint16_t out, uint16_t s0, std::vector<Term> terms, std::vector<Term> sums = {}) {
        int width = 1;
        while (width * 4 < (int)terms.size()) width *= 2;
        auto &v = ph[q];
        while (v.size() % width != 0) v.push_back(OdeOp{OK_NOP, 1, 0, {}});
        for (int l = 0; l < width; ++l) {
            OdeOp op{};
            op.kind = OK_DOT;
            op.width = (uint8_t)width;
            op.out = out;
            op.a[0] = s0;
            for (int t = 0; t < 4; ++t) {
                const int k = l * 4 + t;
                const Term tm = k < (int)terms.size() ? terms[k] : Term{XS_ZERO, XS_ZERO};
                op.a[1 + 2 * t] = tm.x;
                op.a[2 + 2 * t] = tm.y;
            }
            for (int t = 0; t < 2; ++t) {
                const Term tm = l == 0 && t < (int)sums.size() ? sums[t] : Term{XS_ZERO, XS_ZERO};
                op.a[9 + 2 * t] = tm.x;
                op.a[10 + 2 * t] = tm.y;
            }
            v.push_back(op);
        }
    }
};

enum { PH_E = 0, PH_A, PH_P, PH_B, PH_COUNT };

uint16_t neg(uint16_t slot) { return (uint16_t)(slot | kOdeNeg); }

void build(Builder &b) {
    const CellStatic &C = b.C;
    const gw_params &p = b.p;
    const int r = b.regime;
    const bool r0 = r == 0;  // V >= -40
    b.phase(PH_COUNT);
    const uint16_t ONE = XS_ONE, ZERO = XS_ZERO, DT = XS_DT;
    enum { iV = 0, iNai, iKi, iCai, iCaNSR, iCaL, iCaH, im, ih, ij, ixKs, iKr = 11, iKv43 = 16, iKv14 = 26 };
    const uint16_t V = b.G(iV), Nai = b.G(iNai), Ki = b.G(iKi), Cai = b.G(iCai), NSR = b.G(iCaNSR);
    const uint16_t SJLCC = XS_SUMS + 0, SClCh = XS_SUMS + 1, SJtr = XS_SUMS + 2, SJxfer = XS_SUMS + 3;
    auto S = [&]() { return b.S(); };
    auto K = [&](double v) { return b.K(v); };
    // phase A
    const uint16_t VmENa = S(), VmEK = S(), VmECa = S(), VmEKs = S(), argf = S(), argr = S();
    const uint16_t NaS = S(), KiS = S(), pf = S(), pr = S(), opf = S(), Na2 = S(), mm = S(), hj = S(), xKs2 = S();
    const uint16_t OME = S(), KXE = S(), ECL = S(), JEXP = S(), E1C = S(), E12C = S(), D12 = S(), D01 = S(), DKr = S(),
                   DKp = S();
    const uint16_t Q01 = S(), Q10 = S(), Q23 = S(), Q24 = S(), Q32 = S(), Q34 = S(), Q43 = S(), Q42 = S();
    uint16_t kv[2][4];  // [Kv14, Kv43][aa, ai, ba, bi]
    for (auto &c : kv)
        for (auto &x : c) x = S();
    const uint16_t DAM = S(), E_bm = S(), E_ah = S(), E_bh1 = S(), E_bh2 = S(), E_aj1 = S(), E_aj2 = S(), D_aj = S(),
                   E_bj1 = S(), D_bj = S(), DXI = S(), DT1 = S(), DT2 = S(), EK1 = S();
    const uint16_t OPY = S(), OPY6 = S(), Y4 = S(), OPT = S(), T460 = S(), U = S();
    uint16_t al[8], be[8];  // 4a 3a 2a a and those times a; b 2b 3b 4b and those times 1/b
    for (auto &x : al) x = S();
    for (auto &x : be) x = S();
    // phase B
    const uint16_t qKr = S(), qKp = S(), qNaK = S(), qNaK3 = S(), qNaK2 = S(), qNaKS = S(), NaCa1 = S(), NaCa2 = S(),
                   qKv14 = S(), qIto2 = S(), qK1 = S(), qIpCa = S(), am = S(), bh = S(), bj = S(), aj1 = S(), aj2 = S(),
                   xinf = S(), t1 = S(), t2 = S(), qf = S(), qr = S(), sCai = S(), JMUL = S(), IN0 = S(), IN1 = S(),
                   gm3 = S();
    const uint16_t sNa = S(), A1 = S(), nL = S(), nH = S(), omj = S(), omh = S(), gKs = S(), gKv43 = S(), hjV = S();

    const double RT_F = C.RT_F, F_RT = C.F_RT;
    // ---------------- phase A: LOG | EXP | POW ----------------
    {
        const int q = PH_A;
        // V - E = (V + RT/F log(1/Xo)) + RT/F log(Xi); ECa is the reference's (Ki / Ko with valence 2)
        auto lg = [&](uint16_t out, uint16_t v, double off, double scale, uint16_t x, uint16_t c, uint16_t y) {
            b.emit(q, OK_LOG, out, {x, c, v, K(off), K(scale), y});
        };
        lg(VmENa, V, -RT_F * std::log(p.Nao), RT_F, Nai, ZERO, ZERO);
        lg(VmEK, V, -RT_F * std::log(p.Ko), RT_F, Ki, ZERO, ZERO);
        lg(VmECa, V, -0.5 * RT_F * std::log(p.Ko), 0.5 * RT_F, Ki, ZERO, ZERO);
        lg(VmEKs, V, -RT_F * std::log(p.Ko + 0.01833 * p.Nao), RT_F, Ki, K(0.01833), Nai);
        if (!b.fast) {
            lg(argf, ZERO, -p.Hf * std::log(p.Kmf), p.Hf, Cai, ZERO, ZERO);
            lg(argr, ZERO, -p.Hr * std::log(p.Kmr), p.Hr, NSR, ZERO, ZERO);
        }
        b.warp_align(q);
        // out = off + c exp(a V + b)
        auto ex = [&](uint16_t out, uint16_t c, uint16_t a, uint16_t bb, uint16_t off) {
            b.emit(q, OK_EXP, out, {c, a, V, bb, off});
        };
        const uint16_t mF = K(-F_RT), MONE = XS_MONE;
        ex(OME, MONE, mF, ZERO, ONE);
        ex(KXE, K(p.Ko + 0.02 * p.Nao), mF, ZERO, ZERO);
        ex(ECL, K(p.Clcyto), mF, ZERO, K(-p.Clo));
        ex(JEXP, ONE, K(2.0 * F_RT), ZERO, ZERO);
        ex(E1C, K(C.INaCa_const * p.Cao), K(p.eta * F_RT), ZERO, ZERO);
        const uint16_t cEta1 = K((p.eta - 1.0) * F_RT);
        ex(E12C, K(C.INaCa_const * C.Nao3), cEta1, ZERO, ZERO);
        ex(D12, K(p.ksat), cEta1, ZERO, ONE);
        ex(D01, K(0.1245), K(-0.1 * F_RT), ZERO, K(1.0 + 0.0365 * C.sigma));
        ex(DKr, K(1.4945), K(0.0446), ZERO, ONE);
        ex(DKp, ONE, K(-1.0 / 5.98), K(7.488 / 5.98), ONE);
        ex(Q01, K(0.0069), K(0.0272), ZERO, ZERO);
        ex(Q10, K(0.0227), K(-0.0431), ZERO, ZERO);
        ex(Q23, K(0.0218), K(0.0262), ZERO, ZERO);
        ex(Q24, K(1.29e-5), K(2.71e-6), ZERO, ZERO);
        ex(Q32, K(0.0009), K(-0.0269), ZERO, ZERO);
        ex(Q34, K(0.0622), K(0.0120), ZERO, ZERO);
        ex(Q43, K(0.0059), K(-0.0443), ZERO, ZERO);
        // Q42 = Q32 Q43 Q24 / (Q23 Q34)
        ex(Q42, K(0.0009 * 0.0059 * 1.29e-5 / (0.0218 * 0.0622)), K(-0.0269 - 0.0443 + 2.71e-6 - 0.0262 - 0.0120), ZERO, ZERO);
        ex(kv[0][0], K(p.alphaa0Kv14), K(p.aaKv14), ZERO, ZERO);
        ex(kv[1][0], K(p.alphaa0Kv43), K(p.aaKv43), ZERO, ZERO);
        ex(kv[0][1], K(p.alphai0Kv14), K(-p.aiKv14), ZERO, ZERO);
        ex(kv[1][1], K(p.alphai0Kv43), K(-p.aiKv43), ZERO, ZERO);
        ex(kv[0][2], K(p.betaa0Kv14), K(-p.baKv14), ZERO, ZERO);
        ex(kv[1][2], K(p.betaa0Kv43), K(-p.baKv43), ZERO, ZERO);
        ex(kv[0][3], K(p.betai0Kv14), K(p.biKv14), ZERO, ZERO);
        ex(kv[1][3], K(p.betai0Kv43), K(p.biKv43), ZERO, ZERO);
        // gate rates (common.hpp:176-218; GW_utils.hpp:358-362); constants allocated for every
        // regime so that the slot layout does not depend on it
        const uint16_t c0135 = K(0.135), c_ah = K(-1.0 / 6.8), c_ahb = K(-80.0 / 6.8);
        const uint16_t c_bh0a = K(-1.0 / 11.1), c_bh0b = K(-10.66 / 11.1);
        const uint16_t c356 = K(3.56), c0079 = K(0.079), c31e5 = K(3.1e5), c035 = K(0.35);
        const uint16_t c127 = K(-127140.0), c2444 = K(0.2444), c3474 = K(-3.474e-5), c04391 = K(-0.04391);
        const uint16_t c0311 = K(0.311), c0311b = K(0.311 * 79.23);
        const uint16_t c03 = K(0.3), c2535 = K(-2.535e-7), c01212 = K(0.1212), c01052 = K(-0.01052);
        const uint16_t cm01 = K(-0.1), cm32 = K(-3.2), c1378 = K(-0.1378), c1378b = K(-0.1378 * 40.14);
        ex(DAM, MONE, cm01, K(-4.713), ONE);
        ex(E_bm, K(0.08), K(-1.0 / 11.0), ZERO, ZERO);
        if (r0) {
            ex(E_ah, ZERO, ZERO, ZERO, ZERO);
            ex(E_bh1, ONE, c_bh0a, c_bh0b, ONE);  // the denominator of bh
            ex(E_bh2, ZERO, ZERO, ZERO, ZERO);
            ex(E_aj1, ZERO, ZERO, ZERO, ONE);     // (aj is zero: its row does not use them)
            ex(E_aj2, ZERO, ZERO, ZERO, ONE);
            ex(D_aj, ZERO, ZERO, ZERO, ONE);
            ex(E_bj1, c03, c2535, ZERO, ZERO);
            ex(D_bj, ONE, cm01, cm32, ONE);
        } else {
            ex(E_ah, c0135, c_ah, c_ahb, ZERO);
            ex(E_bh1, c356, c0079, ZERO, ZERO);
            ex(E_bh2, c31e5, c035, ZERO, ZERO);
            ex(E_aj1, c127, c2444, ZERO, ZERO);
            ex(E_aj2, c3474, c04391, ZERO, ZERO);
            ex(D_aj, ONE, c0311, c0311b, ONE);
            ex(E_bj1, c01212, c01052, ZERO, ZERO);
            ex(D_bj, ONE, c1378, c1378b, ONE);
        }
        ex(DXI, ONE, K(-1.0 / 13.6), K(24.7 / 13.6), ONE);
        ex(DT1, MONE, K(-0.148), K(1.48), ONE);
        ex(DT2, ONE, K(0.0687), K(-0.687), MONE);
        ex(EK1, ONE, K(1.5 * F_RT), ZERO, ZERO);
        const uint16_t cy = K(0.2), cyb = K(2.5), ct = K(1.0 / 12.0);
        ex(OPY, ONE, cy, cyb, ONE);
        ex(OPY6, K(0.6), cy, cyb, ONE);
        ex(Y4, K(0.4), cy, cyb, ZERO);
        ex(OPT, ONE, ct, cyb, ONE);
        ex(T460, K(60.0), ct, cyb, K(400.0));
        b.emit(q, OK_EXP, U, {Cai, ZERO, ZERO, ZERO, K(p.KCMDN)});  // KCMDN + Cai exp(0)
        // LCC rates of update_LCC_rates (GW_utils.tpp:118-186) at this V
        const uint16_t ca = K(0.012), cab = K(-0.42), cb = K(-0.05), cbb = K(1.75);
        for (int k = 0; k < 8; ++k) {
            ex(al[k], K(2.0 * (4 - k % 4) * (k < 4 ? 1.0 : C.a)), ca, cab, ZERO);
            ex(be[k], K(0.0882 * (1 + k % 4) * (k < 4 ? 1.0 : C.binv)), cb, cbb, ZERO);
        }
        while (b.ph[q].size() < 96) b.ph[q].push_back(OdeOp{OK_NOP, 1, 0, {}});
        // (KmNai/Nai)^1.5 = KmNai^1.5 / (Nai sqrt(Nai)); exp(1.5 F/RT (V - EK)) = exp(1.5 F/RT V) *
        // (Ki/Ko)^1.5 (EK = RT/F log(Ko/Ki)); products of two globals through sqrt(1)
        auto pw = [&](uint16_t out, uint16_t c, uint16_t y, uint16_t x, int w, uint16_t off) {
            b.emit(q, OK_POW, out, {c, y, x, off});
            b.ph[q].back().width = (uint8_t)w;
        };
        pw(NaS, ONE, Nai, Nai, 1, ZERO);
        pw(KiS, K(std::pow(p.Ko, -1.5)), Ki, Ki, 1, ZERO);
        if (b.fast) {
            const uint16_t cf = K(std::pow(p.Kmf, -0.75)), cr = K(std::pow(p.Kmr, -0.75));
            pw(pf, cf, ONE, Cai, 2, ZERO);
            pw(pr, cr, ONE, NSR, 2, ZERO);
            pw(opf, cf, ONE, Cai, 2, ONE);
        }
        pw(Na2, Nai, Nai, ONE, 1, ZERO);
        pw(mm, b.G(im), b.G(im), ONE, 1, ZERO);
        pw(hj, b.G(ih), b.G(ij), ONE, 1, ZERO);
        pw(xKs2, b.G(ixKs), b.G(ixKs), ONE, 1, ZERO);
    }
    // ---------------- phase P: general Jup exponents ----------------
    if (!b.fast) {
        b.emit(PH_P, OK_EXP, pf, {ONE, ONE, argf, ZERO, ZERO});
        b.emit(PH_P, OK_EXP, pr, {ONE, ONE, argr, ZERO, ZERO});
        b.emit(PH_P, OK_EXP, opf, {ONE, ONE, argf, ZERO, ONE});
    }
    // ---------------- phase B: QUOT | SUM3 ----------------
    const uint16_t MONE = XS_MONE;
    const uint16_t kpL = K(p.kLTRPNp), kpH = K(p.kHTRPNp);
    uint16_t kvp[2][22], kvd[2][10], krd[5];
    {
        const int q = PH_B;
        // out = c (x + y z) / (d0 + d1 d2)
        auto quot = [&](uint16_t out, std::initializer_list<uint16_t> a) { b.emit(q, OK_QUOT, out, a); };
        quot(qKr, {K(p.GKr * C.sqrtKo * 0.5), b.G(iKr + 3), ZERO, ZERO, DKr});
        quot(qKp, {K(p.GKp), ONE, ZERO, ZERO, DKp});
        const uint16_t dNaK = K(-0.0365 * C.sigma);  // 1 + 0.1245 e01 + 0.0365 sigma e, e = 1 - OME
        quot(qNaK, {K(C.INaK_const), ONE, ZERO, ZERO, D01, dNaK, OME});
        quot(qNaK3, {K(3.0 * C.INaK_const), ONE, ZERO, ZERO, D01, dNaK, OME});
        quot(qNaK2, {K(-2.0 * C.INaK_const), ONE, ZERO, ZERO, D01, dNaK, OME});
        quot(qNaKS, {ONE, NaS, ZERO, ZERO, K(std::pow(p.KmNai, 1.5)), ONE, NaS});
        quot(NaCa1, {E1C, ZERO, Na2, Nai, D12});
        quot(NaCa2, {E12C, Cai, ZERO, ZERO, D12});
        quot(qKv14, {b.G(iKv14 + 4), ZERO, K(C.PKv14_Csc * kF * F_RT * 1.0e9), V, OME});
        quot(qIto2, {ECL, ZERO, K(C.Ito2_const * F_RT), V, OME});  // -Ito2 per open ClCh
        quot(qK1, {K(p.GK1 * C.IK1_const), ONE, ZERO, ZERO, K(2.0), EK1, KiS});
        quot(qIpCa, {K(p.IpCamax), Cai, ZERO, ZERO, K(p.KmpCa), ONE, Cai});
        const uint16_t c032 = K(0.32), c4713 = K(47.13), c32 = K(3.2);
        if (r == 2)
            quot(am, {c32, ONE, ZERO, ZERO, ONE});
        else
            quot(am, {c032, c4713, V, ONE, DAM});
        const uint16_t c013 = K(1.0 / 0.13);
        if (r0)
            quot(bh, {c013, ONE, ZERO, ZERO, E_bh1});
        else
            quot(bh, {ONE, E_bh1, E_bh2, ONE, ONE});
        quot(bj, {E_bj1, ONE, ZERO, ZERO, D_bj});
        const uint16_t c3778 = K(37.78), cm10 = K(-10.0);
        quot(aj1, {E_aj1, c3778, V, ONE, D_aj});
        quot(aj2, {E_aj2, c3778, V, ONE, D_aj});
        quot(xinf, {ONE, ONE, ZERO, ZERO, DXI});
        quot(t1, {K(0.0000719), cm10, V, ONE, DT1});
        quot(t2, {K(0.000131), cm10, V, ONE, DT2});
        quot(qf, {ONE, pf, ZERO, ZERO, opf, ONE, pr});
        quot(qr, {ONE, pr, ZERO, ZERO, opf, ONE, pr});
        quot(sCai, {DT, ZERO, U, U, K(C.CMDN_const), U, U});  // dt / (1 + CMDN / (KCMDN + Cai)^2)
        quot(JMUL, {K(C.JLCC_const * F_RT), V, ZERO, ZERO, MONE, ONE, JEXP});
        // yinf / tau and (1 - yinf) / tau, with yinf = 0.4 / (1 + Ey) + 0.6 and
        // 1 / tau = (1 + Et) / (400 + 60 Et)
        quot(IN0, {OPT, OPY6, ZERO, ZERO, ZERO, OPY, T460});
        quot(IN1, {OPT, Y4, ZERO, ZERO, ZERO, OPY, T460});
        quot(gm3, {K(p.GNa), ZERO, mm, b.G(im), ONE});
        b.warp_align(q);
        auto sum3 = [&](uint16_t out, std::initializer_list<uint16_t> a) { b.emit(q, OK_SUM3, out, a); };
        sum3(sNa, {DT, K(-C.CSA_FVcyto)});
        sum3(A1, {Ki, ONE, Nai, K(0.02)});
        sum3(nL, {kpL, Cai, K(p.kLTRPNm), ONE});
        sum3(nH, {kpH, Cai, K(p.kHTRPNm), ONE});
        sum3(omj, {ONE, ONE, MONE, b.G(ij)});
        sum3(omh, {ONE, ONE, MONE, b.G(ih)});
        sum3(gKs, {K(p.GKs), xKs2});
        sum3(gKv43, {K(p.GKv43), b.G(iKv43 + 4)});
        sum3(hjV, {hj, VmENa});
        // total outgoing rates of the IKr states (update_QKr, GW.tpp:26-44)
        for (int i = 1; i < 5; ++i) krd[i] = S();
        const uint16_t cKf = K(p.Kf), cKb = K(p.Kb);
        sum3(krd[1], {ONE, Q10, cKf, ONE});
        sum3(krd[2], {cKb, ONE, ONE, Q23, ONE, Q24});
        sum3(krd[3], {ONE, Q32, ONE, Q34});
        sum3(krd[4], {ONE, Q42, ONE, Q43});
        krd[0] = Q01;
        // the Kv1.4 and Kv4.3 generators (update_QKv, GW.tpp:65-123): coefficient times rate for the
        // entries whose coefficient is not 1, and the total outgoing rate of every state
        for (int ch = 0; ch < 2; ++ch) {
            const double f[5] = {1.0, ch == 0 ? p.f1Kv14 : p.f1Kv43, ch == 0 ? p.f2Kv14 : p.f2Kv43,
                                 ch == 0 ? p.f3Kv14 : p.f3Kv43, ch == 0 ? p.f4Kv14 : p.f4Kv43};
            const double g[5] = {1.0, ch == 0 ? p.b1Kv14 : p.b1Kv43, ch == 0 ? p.b2Kv14 : p.b2Kv43,
                                 ch == 0 ? p.b3Kv14 : p.b3Kv43, ch == 0 ? p.b4Kv14 : p.b4Kv43};
            const uint16_t aa = kv[ch][0], ai = kv[ch][1], ba = kv[ch][2], bi = kv[ch][3];
            for (auto &x : kvp[ch]) x = ZERO;
            auto prod = [&](int k, double c, uint16_t x) {
                kvp[ch][k] = S();
                sum3(kvp[ch][k], {K(c), x});
            };
            for (int i = 0; i < 4; ++i) {
                if (i < 3) prod(i, 4.0 - i, aa);                       // 0..2: i -> i + 1 (3 -> 4: aa itself)
                if (i > 0) prod(2 + i, 1.0 + i, ba);                    // 3..5: i + 1 -> i (1 -> 0: ba itself)
                prod(6 + i, (4.0 - i) * g[i + 1] / g[i], aa);           // 6..9: 5 + i -> 6 + i
                prod(10 + i, (1.0 + i) * f[i] / f[i + 1], ba);          // 10..13: 6 + i -> 5 + i
                prod(14 + i, f[i + 1], bi);                             // 14..17: i + 1 -> 6 + i (0 -> 5: bi)
                prod(18 + i, 1.0 / g[i + 1], ai);                       // 18..21: 6 + i -> i + 1 (5 -> 0: ai)
            }
            for (int i = 0; i < 10; ++i) kvd[ch][i] = S();
            for (int i = 0; i < 5; ++i) {
                sum3(kvd[ch][i], {K(4.0 - i), aa, K((double)i), ba, K(f[i]), bi});
                sum3(kvd[ch][5 + i], {K(i < 4 ? (4.0 - i) * g[i + 1] / g[i] : 0.0), aa, K(i > 0 ? i * f[i - 1] / f[i] : 0.0), ba,
                                      K(1.0 / g[i]), ai});
            }
        }
    }
    // ---------------- phase E: increments and update (DOT rows) ----------------
    {
        const int q = PH_E;
        const double CSA = C.CSA_FVcyto;
        // dV (GW.tpp:211)
        b.row(q, iV, DT,
              {{XS_ISTIM, ONE}, {neg(gm3), hjV}, {neg(qKr), VmEK}, {neg(gKs), VmEKs}, {neg(qKv14), A1}, {qKv14, KXE},
               {neg(gKv43), VmEK}, {neg(qK1), VmEK}, {neg(qKp), VmEK}, {neg(qNaK), qNaKS}, {neg(NaCa1), ONE}, {NaCa2, ONE},
               {neg(qIpCa), ONE}, {K(-p.GCab), VmECa}, {K(-p.GNab), VmENa}},
              {{K(-C.ICaL_const), SJLCC}, {qIto2, SClCh}});
        // dNai, dKi (GW.tpp:201-202)
        const uint16_t c3 = K(3.0);
        b.row(q, iNai, sNa, {{gm3, hjV}, {K(p.GNab), VmENa}, {c3, NaCa1}, {neg(c3), NaCa2}, {qNaK3, qNaKS}});
        b.row(q, iKi, sNa,
              {{qKr, VmEK}, {gKs, VmEKs}, {qKv14, A1}, {neg(qKv14), KXE}, {gKv43, VmEK}, {qK1, VmEK}, {qKp, VmEK}, {qNaK2, qNaKS}});
        // dCai, dCaNSR (GW.tpp:203-204)
        const uint16_t cC = K(CSA), L0 = K(p.kLTRPNp * p.LTRPNtot), H0 = K(p.kHTRPNp * p.HTRPNtot);
        const uint16_t gCai = b.G(iCai), gL = b.G(iCaL), gH = b.G(iCaH);
        b.row(q, iCai, sCai,
              {{K(-0.5 * CSA * p.GCab), VmECa}, {K(-0.5 * CSA), qIpCa}, {cC, NaCa1}, {neg(cC), NaCa2}, {K(-p.Vmaxf), qf},
               {K(p.Vmaxr), qr}, {neg(L0), gCai}, {nL, gL}, {neg(H0), gCai}, {nH, gH}},
              {{K(C.VSS_Vcyto * C.CRU_factor), SJxfer}});
        b.row(q, iCaNSR, DT, {{K(C.Vcyto_VNSR * p.Vmaxf), qf}, {K(-C.Vcyto_VNSR * p.Vmaxr), qr}},
              {{K(-C.VJSR_VNSR * C.CRU_factor), SJtr}});
        b.warp_align(q);  // the rows above take shuffles or flux sums, those below neither
        b.row(q, iCaL, DT, {{L0, gCai}, {neg(nL), gL}});
        b.row(q, iCaH, DT, {{H0, gCai}, {neg(nH), gH}});
        // gates (GW.tpp:163-168)
        b.row(q, im, DT, {{am, ONE}, {neg(am), b.G(im)}, {neg(E_bm), b.G(im)}});
        b.row(q, ih, DT, {{E_ah, omh}, {neg(bh), b.G(ih)}});
        if (r0)
            b.row(q, ij, DT, {{neg(bj), b.G(ij)}});
        else
            b.row(q, ij, DT, {{aj1, omj}, {aj2, omj}, {neg(bj), b.G(ij)}});
        b.row(q, ixKs, DT, {{t1, xinf}, {t2, xinf}, {neg(t1), b.G(ixKs)}, {neg(t2), b.G(ixKs)}});
        // IKr Markov chain (update_Kr_derivatives, GW.tpp:127-133)
        const uint16_t cKf = K(p.Kf), cKb = K(p.Kb);
        auto kr = [&](int i) { return b.G(iKr + i); };
        b.row(q, iKr + 0, DT, {{Q10, kr(1)}, {neg(krd[0]), kr(0)}});
        b.row(q, iKr + 1, DT, {{Q01, kr(0)}, {cKb, kr(2)}, {neg(krd[1]), kr(1)}});
        b.row(q, iKr + 2, DT, {{cKf, kr(1)}, {Q32, kr(3)}, {Q42, kr(4)}, {neg(krd[2]), kr(2)}});
        b.row(q, iKr + 3, DT, {{Q23, kr(2)}, {Q43, kr(4)}, {neg(krd[3]), kr(3)}});
        b.row(q, iKr + 4, DT, {{Q24, kr(2)}, {Q34, kr(3)}, {neg(krd[4]), kr(4)}});
        // Kv1.4 and Kv4.3 10-state chains (update_Kv_derivatives, GW.tpp:136-160)
        for (int ch = 0; ch < 2; ++ch) {
            const int base = ch == 0 ? iKv14 : iKv43;
            const uint16_t aa = kv[ch][0], ai = kv[ch][1], ba = kv[ch][2], bi = kv[ch][3];
            const uint16_t *P = kvp[ch], *D = kvd[ch];
            auto x = [&](int i) { return b.G(base + i); };
            for (int i = 0; i < 10; ++i) {
                std::vector<Builder::Term> in;
                if (i < 5) {
                    if (i > 0) in.push_back({i < 4 ? P[i - 1] : aa, x(i - 1)});
                    if (i < 4) in.push_back({i > 0 ? P[3 + i - 1] : ba, x(i + 1)});
                    in.push_back({i > 0 ? P[18 + i - 1] : ai, x(5 + i)});
                } else {
                    const int k = i - 5;
                    if (k > 0) in.push_back({P[6 + k - 1], x(i - 1)});
                    if (k < 4) in.push_back({P[10 + k], x(i + 1)});
                    in.push_back({k > 0 ? P[14 + k - 1] : bi, x(k)});
                }
                in.push_back({neg(D[i]), x(i)});
                b.row(q, (uint16_t)(base + i), DT, in);
            }
        }
    }
    // per-step SSA values
    b.sv_src[SV_ZERO] = ZERO;
    for (int k = 0; k < 4; ++k) {
        b.sv_src[SV_A4 + k] = al[k];
        b.sv_src[SV_A4a + k] = al[4 + k];
        b.sv_src[SV_B1 + k] = be[k];
        b.sv_src[SV_B1bi + k] = be[4 + k];
    }
    b.sv_src[SV_F] = b.K(p.f); b.sv_src[SV_G] = b.K(p.g); b.sv_src[SV_OM] = b.K(C.omega);
    b.sv_src[SV_OMB1] = b.K(C.omega_b); b.sv_src[SV_OMB2] = b.K(C.omega_b2);
    b.sv_src[SV_OMB3] = b.K(C.omega_b3); b.sv_src[SV_OMB4] = b.K(C.omega_b4);
    b.sv_src[SV_F1] = b.K(p.f1); b.sv_src[SV_G1] = b.K(p.g1);
    b.sv_src[SV_INACT0] = IN0; b.sv_src[SV_INACT1] = IN1;
    b.sv_src[SV_JMUL] = JMUL; b.sv_src[SV_JEXP] = JEXP;
    b.sv_src[SV_CAI] = Cai; b.sv_src[SV_CANSR] = NSR;
}

int regime_of(double V, bool) { return V >= -40.0 ? 0 : (V == -47.13 ? 2 : 1); }

bool same_op(const OdeOp &a, const OdeOp &b) { return std::memcmp(&a, &b, sizeof a) == 0; }

}  // namespace

bool ode_program_build(const CellStatic &cs, bool pow_fast, OdeProgram *prog, double *consts) {
    Builder v[3] = {Builder(cs, pow_fast, 0, consts), Builder(cs, pow_fast, 1, nullptr),
                    Builder(cs, pow_fast, 2, nullptr)};
    for (auto &b : v) build(b);
    if (v[0].nconst > kOdeMaxConsts || v[0].next > kOdeMaxSlots) {
        if (prog) { prog->n_consts = v[0].nconst; prog->n_slots = v[0].next; }
        return false;
    }
    if (!prog) return true;
    std::memset(prog, 0, sizeof *prog);
    int n = 0;
    prog->n_phases = 0;
    for (int q = 0; q < PH_COUNT; ++q) {
        if (v[0].ph[q].empty()) continue;
        for (int k = 1; k < 3; ++k)
            if (v[k].ph[q].size() != v[0].ph[q].size()) {
                fprintf(stderr, "ode program: phase %d size differs in regime %d (%zu vs %zu)\n", q, k, v[k].ph[q].size(), v[0].ph[q].size());
                return false;
            }
        if (q == PH_E) prog->upd_phase = prog->n_phases;
        if (q == PH_B) prog->push_phase = prog->n_phases;
        prog->phase_begin[prog->n_phases++] = n;
        for (size_t j = 0; j < v[0].ph[q].size(); ++j) {
            if (n >= kOdeMaxOps) { fprintf(stderr, "ode program: too many ops\n"); return false; }
            prog->ops[n] = v[0].ph[q][j];
            prog->alt_idx[n] = 255;
            if (!same_op(v[1].ph[q][j], v[0].ph[q][j]) || !same_op(v[2].ph[q][j], v[0].ph[q][j])) {
                if (prog->n_alt >= kOdeMaxAlt) { fprintf(stderr, "ode program: too many variants\n"); return false; }
                prog->alt[0][prog->n_alt] = v[1].ph[q][j];
                prog->alt[1][prog->n_alt] = v[2].ph[q][j];
                prog->alt_idx[n] = (uint8_t)prog->n_alt++;
            }
            ++n;
        }
    }
    prog->phase_begin[prog->n_phases] = n;
    // Each warp of a phase must hold one op kind (in every regime): the device switches on it once
    // per warp.
    for (int q = 0; q < prog->n_phases; ++q) {
        const int b0 = prog->phase_begin[q], nq = prog->phase_begin[q + 1] - b0;
        if (nq > kOdeLanes) {
            fprintf(stderr, "ode program: phase %d has %d ops (max %d)\n", q, nq, kOdeLanes);
            return false;
        }
        for (int w = 0; w < kOdeWarps; ++w) {
            int kind = OK_NOP;
            for (int l = 32 * w; l < std::min(32 * w + 32, nq); ++l) {
                const OdeOp *cand[3] = {&prog->ops[b0 + l], nullptr, nullptr};
                if (prog->alt_idx[b0 + l] != 255) {
                    cand[1] = &prog->alt[0][prog->alt_idx[b0 + l]];
                    cand[2] = &prog->alt[1][prog->alt_idx[b0 + l]];
                }
                for (const OdeOp *op : cand) {
                    if (!op || op->kind == OK_NOP) continue;
                    if (kind != OK_NOP && kind != op->kind) {
                        fprintf(stderr, "ode program: phase %d warp %d mixes op kinds\n", q, w);
                        return false;
                    }
                    kind = op->kind;
                }
            }
        }
    }
    prog->n_slots = v[0].next;
    prog->const_begin = XS_FIRST_FREE;
    prog->n_consts = v[0].nconst;
    for (int i = 0; i < kSvCount; ++i) prog->sv_src[i] = v[0].sv_src[i];
    // The ops whose outputs are per-step SSA values stage them for the push themselves (Cai and
    // CaNSR are staged by their updates, constant values once per launch).
    for (int i = 0; i < kSvCount; ++i) {
        if (i == SV_CAI || i == SV_CANSR || i == SV_CAI_LO || i == SV_CANSR_LO) continue;
        const int src = prog->sv_src[i];
        if (src < XS_FIRST_FREE + kOdeMaxConsts) continue;  // fixed or constant slot
        for (int j = 0; j < n; ++j) {
            const bool writes = prog->ops[j].kind != OK_NOP && prog->ops[j].out == src;
            const bool alt_writes = prog->alt_idx[j] != 255 && (prog->alt[0][prog->alt_idx[j]].out == src ||
                                                                prog->alt[1][prog->alt_idx[j]].out == src);
            if (!writes && !alt_writes) continue;
            if (prog->sv_stage[j] != 0 && prog->sv_stage[j] != i + 1) {
                fprintf(stderr, "ode program: slot %d staged to two sv values\n", src);
                return false;
            }
            prog->sv_stage[j] = (uint8_t)(i + 1);
        }
    }
    return true;
}

// Host evaluation of one global step with the device's operation order (FP64): g[36] in/out,
// sums {JLCC, ClCh, Jtr, Jxfer}; sv receives the per-step SSA values of the updated state.
void ode_program_step_host(const OdeProgram &P, const double *consts, double *g, const double *sums,
                           double Istim, double dt, double *sv) {
    std::vector<double> X(kOdeMaxSlots, 0.0);  // (a slot index of 15 bits: see kOdeNeg)
    X[XS_ZERO] = 0.0;
    X[XS_ONE] = 1.0;
    X[XS_MONE] = -1.0;
    for (int i = 0; i < P.n_consts; ++i) X[P.const_begin + i] = consts[i];
    for (int i = 0; i < kNumGlobals; ++i) X[XS_G + i] = g[i];
    for (int i = 0; i < 4; ++i) X[XS_SUMS + i] = sums[i];
    X[XS_ISTIM] = Istim;
    X[XS_DT] = dt;
    auto regime = [&]() { const double V = g[0]; return V >= -40.0 ? 0 : (V == -47.13 ? 2 : 1); };
    auto run_phase = [&](int q, int reg) {
        const int b0 = P.phase_begin[q], n = P.phase_begin[q + 1] - b0;
        std::vector<double> val(n, 0.0);
        std::vector<const OdeOp *> ops(n);
        for (int j = 0; j < n; ++j) {
            const OdeOp *op = &P.ops[b0 + j];
            if (reg > 0 && P.alt_idx[b0 + j] != 255) op = &P.alt[reg - 1][P.alt_idx[b0 + j]];
            ops[j] = op;
            const uint16_t *a = op->a;
            double v = 0.0;
            switch (op->kind) {
            case OK_LOG: v = (X[a[2]] + X[a[3]]) + X[a[4]] * std::log(X[a[0]] + X[a[1]] * X[a[5]]); break;
            case OK_EXP: v = X[a[4]] + X[a[0]] * std::exp(X[a[1]] * X[a[2]] + X[a[3]]); break;
            case OK_POW: {
                const double t = std::sqrt(X[a[2]]);
                v = X[a[3]] + X[a[0]] * X[a[1]] * (op->width == 2 ? t * std::sqrt(t) : t);
                break;
            }
            case OK_QUOT: v = X[a[0]] * (X[a[1]] + X[a[2]] * X[a[3]]) / (X[a[4]] + X[a[5]] * X[a[6]]); break;
            case OK_SUM3: v = X[a[0]] * X[a[1]] + X[a[2]] * X[a[3]] + X[a[4]] * X[a[5]]; break;
            case OK_DOT:
                for (int t = 0; t < 4; ++t) {
                    const double x = X[a[1 + 2 * t] & (uint16_t)~kOdeNeg];
                    v += ((a[1 + 2 * t] & kOdeNeg) ? -x : x) * X[a[2 + 2 * t]];
                }
                break;
            default: break;
            }
            val[j] = v;
        }
        // DOT rows: lane tree (offsets 1, 2, 4) as the device's shuffles, then the flux sums and the update
        for (int off = 1; off < 8; off <<= 1)
            for (int j = 0; j < n; ++j)
                if (ops[j]->kind == OK_DOT && (j % ops[j]->width) + off < ops[j]->width && (j % (2 * off)) == 0)
                    val[j] += val[j + off];
        for (int j = 0; j < n; ++j) {
            const OdeOp *op = ops[j];
            if (op->kind == OK_NOP) continue;
            if (op->kind == OK_DOT) {
                if (j % op->width == 0) {
                    const double v = val[j] + X[op->a[9]] * X[op->a[10]] + X[op->a[11]] * X[op->a[12]];
                    g[op->out] += X[op->a[0]] * v;
                    X[XS_G + op->out] = g[op->out];
                }
            } else {
                X[op->out] = val[j];
            }
        }
    };
    // the transcendental phases of the current state (run before the loop on the device)
    for (int q = P.upd_phase + 1; q < P.n_phases; ++q) run_phase(q, regime());
    // the step: increments and update, then the new state's phases
    for (int q = 0; q < P.n_phases; ++q) run_phase(q, q <= P.upd_phase ? regime_of(g[0], true) : regime());
    for (int i = 0; i < kSvCount; ++i) sv[i] = X[P.sv_src[i]];
}

}  // namespace gw
