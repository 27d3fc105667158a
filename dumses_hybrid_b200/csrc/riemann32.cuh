// FP32 HLLD/HLLD solves of two cells at a time (k_riemann32): the solvers of solvers.cuh
// (hlld1d_f, hlld2d_f; solver.f90:618-836, solver_magnetic.f90:362-548) on pairs of values, with the
// chip's two-lane FP32 instructions (__fadd2_rn, __fmul2_rn, __ffma2_rn).
//
// k_riemann3d, one cell per thread, is bound by issue slots (2800 instructions a cell).  A thread here
// takes the cells c and c + 1 of the trace core, c even: an addition or product of both is one
// instruction, a field of both one 8-byte load (rows of cells start at even places: an even nx), and
// index arithmetic is shared.  Minima, roots, reciprocals and the choice of a zone stay one per cell.
// 1800 instructions a cell; bound now by the latency of its loads at 16 warps per SM.
#pragma once
#include "step_impl.cuh"

namespace dg {
namespace f32 {
namespace {

using V2 = float2;
__device__ __forceinline__ V2 operator+(V2 a, V2 b) { return add2(a, b); }
__device__ __forceinline__ V2 operator*(V2 a, V2 b) { return mul2(a, b); }
__device__ __forceinline__ V2 operator*(float a, V2 b) { return mul2(s2(a), b); }
__device__ __forceinline__ V2 operator-(V2 a, V2 b) { return fma2(b, s2(-1.0f), a); }
template <class F> __device__ __forceinline__ V2 each(V2 a, F f) { return p2(f(a.x), f(a.y)); }
template <class F> __device__ __forceinline__ V2 each(V2 a, V2 b, F f) { return p2(f(a.x, b.x), f(a.y, b.y)); }
__device__ __forceinline__ V2 rcp2(V2 a) { return p2(1.0f / a.x, 1.0f / a.y); }
__device__ __forceinline__ V2 rsq2(V2 a) { return p2(rsqrtf(a.x), rsqrtf(a.y)); }
__device__ __forceinline__ V2 root2(V2 a) { return p2(sqrtf(a.x), sqrtf(a.y)); }
__device__ __forceinline__ V2 abs2(V2 a) { return p2(fabsf(a.x), fabsf(a.y)); }
__device__ __forceinline__ V2 max2(V2 a, V2 b) { return p2(fmaxf(a.x, b.x), fmaxf(a.y, b.y)); }
__device__ __forceinline__ V2 min2(V2 a, V2 b) { return p2(fminf(a.x, b.x), fminf(a.y, b.y)); }
__device__ __forceinline__ V2 floor2(float small, V2 a) { return p2(floored(small, a.x), floored(small, a.y)); }
// a b + c d
__device__ __forceinline__ V2 dot2(V2 a, V2 b, V2 c, V2 d) { return fma2(a, b, mul2(c, d)); }

// the values of core field f at cells c and c + 1, c even (one block of the core, 8-byte aligned);
// kShift: at c - 1 and c
template <bool kShift>
__device__ __forceinline__ V2 pair_at(const float *core, int f, long long c) {
    const float *p = core + core_base(c, kCore3) + f * kCoreLane;
    const V2 v = chk(p, 8) ? __ldg((const float2 *)p) : p2(0.0f, 0.0f);
    if constexpr (kShift) return p2(ld(core + core_base(c - 1, kCore3) + f * kCoreLane), v.x);
    return v;
}

struct State2 {
    V2 r, p, u, v, w, b, c;  // density, pressure, normal and transverse velocities and fields
};

// the states of two cells on their plus (sgn = 1) or minus side in direction d, and the field there;
// load(f): their values of core field f
template <int d, int sgn, class Load>
__device__ __forceinline__ State2 face_side(Load load, float smallp, V2 &bn) {
    int f[15];
    face_fields(d, sgn, 3, f);
    auto at = [&](int n, int m) { return sgn > 0 ? load(f[n]) + load(f[m]) : load(f[n]) - load(f[m]); };
    constexpr int ln = 1 + d, t1 = d == 0 ? 2 : 1, t2 = d == 2 ? 2 : 3;  // positions of the velocities
    State2 s;
    s.r = floor2((float)kSmallr, at(0, 5));
    s.p = floor2(smallp, at(4, 9));
    s.u = at(ln, 5 + ln);
    s.v = at(t1, 5 + t1);
    s.w = at(t2, 5 + t2);
    s.b = at(12, 10);
    s.c = at(13, 11);
    bn = load(f[14]);
    return s;
}

// hlld1d_f for two interfaces: fluxes of rho, E, the normal momentum without and the star total
// pressure pg, the transverse momenta
__device__ __forceinline__ void hlld1d_2(const State2 &l, const State2 &q, V2 a, float gamma, float entho, V2 f[5], V2 &pg) {
    const float half = 0.5f;
    const V2 aa = a * a, one = s2(1.0f);
    const V2 sg = p2(copysignf(1.0f, a.x), copysignf(1.0f, a.y));
    auto side = [&](const State2 &s, V2 &et, V2 &pt, V2 &vb) {
        const V2 b2 = fma2(s.b, s.b, fma2(s.c, s.c, aa)), em = half * b2;
        const V2 ke = fma2(s.u, s.u, dot2(s.v, s.v, s.w, s.w));
        et = fma2(s.p, s2(entho), fma2(half * ke, s.r, em));
        pt = s.p + em;
        vb = fma2(s.u, a, dot2(s.v, s.b, s.w, s.c));
        const V2 ir = rcp2(s.r), c2 = gamma * s.p * ir, d2 = half * fma2(b2, ir, c2);
        const V2 disc = fma2(neg2(c2 * aa), ir, d2 * d2);
        return d2 + root2(max2(disc, s2(0.0f)));
    };
    V2 el, er, tl, tr, xl, xr;
    const V2 fl = side(l, el, tl, xl), fr = side(q, er, tr, xr);
    const V2 cf = root2(max2(fl, fr));
    const V2 sl = min2(l.u, q.u) - cf, sr = max2(l.u, q.u) + cf;
    const V2 dl = sl - l.u, dr = sr - q.u;         // s - u of either side
    const V2 ml = l.r * dl, mr = q.r * dr;         // rho (s - u)
    const V2 irc = rcp2(mr - ml);
    const V2 us = (dot2(mr, q.u, neg2(ml), l.u) + (tl - tr)) * irc;  // the pressures' difference first: it is small
    const V2 ts = fma2(mr, tl, neg2(ml * fma2(mr, l.u - q.u, tr))) * irc;
    auto star = [&](const State2 &s, V2 sd, V2 d, V2 m, V2 e, V2 t, V2 x, V2 &rs, V2 &vs, V2 &ws, V2 &bs, V2 &cs, V2 &xs,
                    V2 &es) {
        const V2 dus = sd - us, is = rcp2(dus);
        rs = m * is;
        const V2 es0 = fma2(m, dus, neg2(aa)), e0 = fma2(m, d, neg2(aa));
        const V2 ie = p2(es0.x != 0.0f ? 1.0f / es0.x : 0.0f, es0.y != 0.0f ? 1.0f / es0.y : 0.0f);
        const V2 g = a * (us - s.u) * ie;
        V2 h = e0 * ie;
        if (es0.x == 0.0f) h.x = 1.0f;  // g is zero there: the state's own v, w, b, c
        if (es0.y == 0.0f) h.y = 1.0f;
        vs = fma2(neg2(s.b), g, s.v);
        ws = fma2(neg2(s.c), g, s.w);
        bs = s.b * h;
        cs = s.c * h;
        xs = fma2(us, a, dot2(vs, bs, ws, cs));
        es = fma2(d, e, fma2(neg2(t), s.u, fma2(ts, us, a * (x - xs)))) * is;
    };
    V2 rsl, vsl, wsl, bsl, csl, xsl, esl, rsr, vsr, wsr, bsr, csr, xsr, esr;
    star(l, sl, dl, ml, el, tl, xl, rsl, vsl, wsl, bsl, csl, xsl, esl);
    star(q, sr, dr, mr, er, tr, xr, rsr, vsr, wsr, bsr, csr, xsr, esr);
    const V2 il = rsq2(rsl), ir = rsq2(rsr), ql = rsl * il, qr = rsr * ir;
    const V2 al = fma2(neg2(abs2(a)), il, us), ar = fma2(abs2(a), ir, us);
    const V2 is = rcp2(ql + qr), sq = sg * ql * qr;
    const V2 v2 = fma2(sg, bsr - bsl, dot2(ql, vsl, qr, vsr)) * is;
    const V2 w2 = fma2(sg, csr - csl, dot2(ql, wsl, qr, wsr)) * is;
    const V2 b2 = fma2(sq, vsr - vsl, dot2(ql, bsr, qr, bsl)) * is;
    const V2 c2 = fma2(sq, wsr - wsl, dot2(ql, csr, qr, csl)) * is;
    const V2 x2 = fma2(us, a, dot2(v2, b2, w2, c2));
    const V2 e2l = fma2(neg2(sg * ql), xsl - x2, esl), e2r = fma2(sg * qr, xsr - x2, esr);
    // sample at x/t = 0, each interface by itself
    V2 ro, uo, vo, wo, bo, co, to, eo, xo;
#define DG_SAMPLE(m)                                                                                            \
    if (sl.m > 0.0f) { ro.m = l.r.m; uo.m = l.u.m; vo.m = l.v.m; wo.m = l.w.m; bo.m = l.b.m; co.m = l.c.m; to.m = tl.m; eo.m = el.m; xo.m = xl.m; } \
    else if (al.m > 0.0f) { ro.m = rsl.m; uo.m = us.m; vo.m = vsl.m; wo.m = wsl.m; bo.m = bsl.m; co.m = csl.m; to.m = ts.m; eo.m = esl.m; xo.m = xsl.m; } \
    else if (us.m > 0.0f) { ro.m = rsl.m; uo.m = us.m; vo.m = v2.m; wo.m = w2.m; bo.m = b2.m; co.m = c2.m; to.m = ts.m; eo.m = e2l.m; xo.m = x2.m; } \
    else if (ar.m > 0.0f) { ro.m = rsr.m; uo.m = us.m; vo.m = v2.m; wo.m = w2.m; bo.m = b2.m; co.m = c2.m; to.m = ts.m; eo.m = e2r.m; xo.m = x2.m; } \
    else if (sr.m > 0.0f) { ro.m = rsr.m; uo.m = us.m; vo.m = vsr.m; wo.m = wsr.m; bo.m = bsr.m; co.m = csr.m; to.m = ts.m; eo.m = esr.m; xo.m = xsr.m; } \
    else { ro.m = q.r.m; uo.m = q.u.m; vo.m = q.v.m; wo.m = q.w.m; bo.m = q.b.m; co.m = q.c.m; to.m = tr.m; eo.m = er.m; xo.m = xr.m; }
    DG_SAMPLE(x)
    DG_SAMPLE(y)
#undef DG_SAMPLE
    const V2 m = ro * uo, na = neg2(a);
    f[0] = m;
    f[1] = fma2(eo + to, uo, na * xo);
    f[2] = fma2(m, uo, neg2(aa));
    f[3] = fma2(m, vo, na * bo);
    f[4] = fma2(m, wo, na * co);
    pg = to;
}

// two faces of direction d from the trace core of their minus-side (left) and plus-side (right)
// cells, into the records t of those with ok; i: their x index
template <int d, class Left, class Right>
__device__ __forceinline__ void face_pair_flux(const Geo &G, Left left, Right right, const bool ok[2], const int i[2],
                                               const long long t[2], float dt, float *__restrict__ out) {
    const float smallp = (float)G.smallp;
    V2 bl, br;
    State2 l = face_side<d, +1>(left, smallp, bl), r = face_side<d, -1>(right, smallp, br);
    const V2 a = 0.5f * (bl + br), pl = l.p, pr = r.p;
    if (G.iso) {
        const float c2 = (float)(G.ciso * G.ciso);
        l.p = c2 * l.r;
        r.p = c2 * r.r;
    }
    V2 f[5], pg;
    hlld1d_2(l, r, a, (float)G.gamma, (float)G.entho, f, pg);
    if ((G.omega0 > 0.0) && d == 1 && !G.fargo) {
        // shearing-box upwind terms (solver.f90:199-241), as flux_store adds them
#define DG_SHEAR(m, n)                                                                                     \
        {                                                                                                      \
            const float sh = (float)(-1.5 * G.omega0 * G.xc(i[n]));                                            \
            const State2 &s = sh > 0.0f ? l : r;                                                               \
            const float em = 0.5f * (a.m * a.m + s.b.m * s.b.m + s.c.m * s.c.m);                               \
            const float ek = 0.5f * (s.u.m * s.u.m + s.v.m * s.v.m + s.w.m * s.w.m);                           \
            const float et = ek + em + (sh > 0.0f ? pl.m : pr.m) / ((float)G.gamma - 1.0f);                                        \
            f[0].m += sh * s.r.m;                                                                              \
            f[1].m += sh * (et + em - a.m * a.m);                                                              \
            f[2].m += sh * s.r.m * s.u.m;                                                                      \
            f[3].m += sh * s.r.m * s.v.m;                                                                      \
            f[4].m += sh * s.r.m * s.w.m;                                                                      \
        }
        DG_SHEAR(x, 0)
        DG_SHEAR(y, 1)
#undef DG_SHEAR
    }
    const float ds = (float)(d == 0 ? G.dy * G.dz : d == 1 ? G.dx * G.dz : G.dx * G.dy);
    const V2 k = s2(ds * dt);
    constexpr int mn_ = 2 + d, m1 = d == 0 ? 3 : 2, m2 = d == 2 ? 3 : 4;  // record places of the momenta
    V2 o[6];
    o[0] = f[0] * k;
    o[1] = f[1] * k;
    o[mn_] = f[2] * k;
    o[m1] = f[3] * k;
    o[m2] = f[4] * k;
    o[5] = pg;
    const float x[6] = {o[0].x, o[1].x, o[2].x, o[3].x, o[4].x, o[5].x};
    const float y[6] = {o[0].y, o[1].y, o[2].y, o[3].y, o[4].y, o[5].y};
    if (ok[0]) store6(out + t[0] * kFluxRec3, x);
    if (ok[1]) store6(out + t[1] * kFluxRec3, y);
}

struct Corner2 {
    V2 r, p, u, v, A, B, C;
};

// corner state of edge direction e on the (sa, sb) side of a pair of cells (corner_state)
template <bool kShift, int e, int sa, int sb>
__device__ __forceinline__ Corner2 corner_pair(const Geo &G, const float *core, long long c, float smallp) {
    auto L = [&](int f) { return pair_at<kShift>(core, f, c); };
    constexpr int b1 = e == 0 ? C_DRY : C_DRX, b2 = e == 2 ? C_DRY : C_DRZ;
    auto comb = [&](int f0, int f1, int f2) {
        const V2 m = L(f0), d1 = L(f1), d2 = L(f2);
        const V2 n = sa > 0 ? m + d1 : m - d1;
        return sb > 0 ? n + d2 : n - d2;
    };
    auto prim = [&](int n) { return comb(C_R + n, b1 + n, b2 + n); };
    auto side = [&](int f, int df, int sg) { return sg > 0 ? L(f) + L(df) : L(f) - L(df); };
    Corner2 s;
    s.r = floor2((float)kSmallr, prim(0));
    if (G.iso) s.p = (float)(G.ciso * G.ciso) * s.r;
    else s.p = floor2(smallp, prim(4));
    if constexpr (e == 0) {
        s.u = prim(2);
        s.v = prim(3);
        s.C = comb(C_A, C_DAY, C_DAZ);
        s.A = side(sa > 0 ? C_BR : C_BL, sa > 0 ? C_DBRZ : C_DBLZ, sb);
        s.B = side(sb > 0 ? C_CR : C_CL, sb > 0 ? C_DCRY : C_DCLY, sa);
    } else if constexpr (e == 1) {
        s.u = prim(3);
        s.v = prim(1);
        s.C = comb(C_B, C_DBX, C_DBZ);
        s.B = side(sa > 0 ? C_AR : C_AL, sa > 0 ? C_DARZ : C_DALZ, sb);
        s.A = side(sb > 0 ? C_CR : C_CL, sb > 0 ? C_DCRX : C_DCLX, sa);
    } else {
        s.u = prim(1);
        s.v = prim(2);
        s.C = comb(C_C, C_DCX, C_DCY);
        s.A = side(sa > 0 ? C_AR : C_AL, sa > 0 ? C_DARY : C_DALY, sb);
        s.B = side(sb > 0 ? C_BR : C_BL, sb > 0 ? C_DBRX : C_DBLX, sa);
    }
    return s;
}

// hlld2d_f for two edges; the corners' A and B are the averages of solver_magnetic_utils
__device__ __forceinline__ V2 hlld2d_2(const Corner2 &LL, const Corner2 &LR, const Corner2 &RL, const Corner2 &RR, float gamma) {
    const float half = 0.5f, smallc = (float)kSmallc;
    auto fast = [&](const Corner2 &q, V2 &fx, V2 &fy, V2 &pt) {
        const V2 ir = rcp2(q.r), a2 = q.A * q.A, b2 = q.B * q.B, s = fma2(q.C, q.C, a2 + b2);
        const V2 c2 = gamma * q.p * ir, d2 = half * fma2(s, ir, c2), dd = d2 * d2, k = neg2(c2 * ir);
        fx = d2 + root2(max2(fma2(k, a2, dd), s2(0.0f)));
        fy = d2 + root2(max2(fma2(k, b2, dd), s2(0.0f)));
        pt = fma2(s, s2(half), q.p);
    };
    V2 x0, x1, x2, x3, y0, y1, y2, y3, pLL, pLR, pRL, pRR;
    fast(LL, x0, y0, pLL);
    fast(LR, x1, y1, pLR);
    fast(RL, x2, y2, pRL);
    fast(RR, x3, y3, pRR);
    auto mx4v = [](V2 a, V2 b, V2 c, V2 d) { return p2(mx4(a.x, b.x, c.x, d.x), mx4(a.y, b.y, c.y, d.y)); };
    auto mn4v = [](V2 a, V2 b, V2 c, V2 d) { return p2(mn4(a.x, b.x, c.x, d.x), mn4(a.y, b.y, c.y, d.y)); };
    const V2 cfx = root2(mx4v(x0, x1, x2, x3)), cfy = root2(mx4v(y0, y1, y2, y3));
    const V2 SL = mn4v(LL.u, LR.u, RL.u, RR.u) - cfx, SR = mx4v(LL.u, LR.u, RL.u, RR.u) + cfx;
    const V2 SB = mn4v(LL.v, LR.v, RL.v, RR.v) - cfy, ST = mx4v(LL.v, LR.v, RL.v, RR.v) + cfy;
    // S - u and S - v of the corners; rho (S - u)
    const V2 aLL = SL - LL.u, aLR = SL - LR.u, aRL = SR - RL.u, aRR = SR - RR.u;
    const V2 bLL = SB - LL.v, bLR = ST - LR.v, bRL = SB - RL.v, bRR = ST - RR.v;
    const V2 mLL = LL.r * aLL, mLR = LR.r * aLR, mRL = RL.r * aRL, mRR = RR.r * aRR;
    const V2 nLL = LL.r * bLL, nLR = LR.r * bLR, nRL = RL.r * bRL, nRR = RR.r * bRR;
    const V2 us = (dot2(mRL, RL.u, mRR, RR.u) - dot2(mLL, LL.u, mLR, LR.u) + ((pLL - pRL) + (pLR - pRR))) *
                  rcp2((mRL + mRR) - (mLL + mLR));
    const V2 vs = (dot2(nLR, LR.v, nRR, RR.v) - dot2(nLL, LL.v, nRL, RL.v) + ((pLL - pLR) + (pRL - pRR))) *
                  rcp2((nLR + nRR) - (nLL + nRL));
    const V2 iL = rcp2(SL - us), iR = rcp2(SR - us), iB = rcp2(SB - vs), iT = rcp2(ST - vs);
    const V2 fLLx = aLL * iL, fLRx = aLR * iL, fRLx = aRL * iR, fRRx = aRR * iR;
    const V2 fLLy = bLL * iB, fLRy = bLR * iT, fRLy = bRL * iB, fRRy = bRR * iT;
    const V2 BsLL = LL.B * fLLx, BsLR = LR.B * fLRx, BsRL = RL.B * fRLx, BsRR = RR.B * fRRx;
    const V2 AsLL = LL.A * fLLy, AsLR = LR.A * fLRy, AsRL = RL.A * fRLy, AsRR = RR.A * fRRy;
    // Alfven speeds: |A| / sqrt(rho_x), |A*| / sqrt(rho_xy) across x, and with B across y
    auto alfven = [&](const Corner2 &q, V2 fx, V2 fy, V2 As, V2 Bs, V2 &ax, V2 &ay) {
        const V2 rx = q.r * fx, ix = rsq2(rx), iy = rsq2(q.r * fy), ixy = rsq2(rx * fy);
        ax = max2(abs2(q.A) * ix, abs2(As) * ixy);
        ay = max2(abs2(q.B) * iy, abs2(Bs) * ixy);
    };
    V2 cL, cR, cB, cT, h0, h1, g0, g1;
    alfven(LL, fLLx, fLLy, AsLL, BsLL, cL, cB);
    alfven(LR, fLRx, fLRy, AsLR, BsLR, h0, cT);
    alfven(RL, fRLx, fRLy, AsRL, BsRL, cR, g0);
    alfven(RR, fRRx, fRRy, AsRR, BsRR, h1, g1);
    cL = max2(max2(cL, h0), s2(smallc));
    cR = max2(max2(cR, h1), s2(smallc));
    cB = max2(max2(cB, g0), s2(smallc));
    cT = max2(max2(cT, g1), s2(smallc));
    const V2 SAL = min2(us - cL, s2(0.0f)), SAR = max2(us + cR, s2(0.0f));
    const V2 SAB = min2(vs - cB, s2(0.0f)), SAT = max2(vs + cT, s2(0.0f));
    const V2 ix = rcp2(SAR - SAL), iy = rcp2(SAT - SAB);
    // the zone inside all four fast waves
    const V2 ELL = us * BsLL - vs * AsLL, ELR = us * BsLR - vs * AsLR;
    const V2 ERL = us * BsRL - vs * AsRL, ERR = us * BsRR - vs * AsRR;
    const V2 At = dot2(SAR, AsRR, neg2(SAL), AsLR), Ab = dot2(SAR, AsRL, neg2(SAL), AsLL);
    const V2 Br = dot2(SAT, BsRR, neg2(SAB), BsRL), Bl = dot2(SAT, BsLR, neg2(SAB), BsLL);
    const V2 ixy = ix * iy;
    const V2 lo = dot2(SAL, ERR, neg2(SAR), ELR), hi = dot2(SAR, ELL, neg2(SAL), ERL);
    V2 E = dot2(SAB, lo, SAT, hi) * ixy;
    E = fma2(neg2(SAT * SAB * ixy), At - Ab, E);
    E = fma2(SAR * SAL * ixy, Br - Bl, E);
    // the other zones, edge by edge (solver_magnetic.f90:520-547)
#define DG_ZONE(m)                                                                                             \
    {                                                                                                          \
        auto plain = [&](const Corner2 &q) { return q.u.m * q.B.m - q.v.m * q.A.m; };                          \
        auto across_x = [&](const Corner2 &l, const Corner2 &r, float Bsl, float Bsr) {                        \
            const float El = us.m * Bsl - l.v.m * l.A.m, Er = us.m * Bsr - r.v.m * r.A.m;                      \
            return (SAR.m * El - SAL.m * Er + SAR.m * SAL.m * (r.B.m - l.B.m)) * ix.m;                         \
        };                                                                                                     \
        auto across_y = [&](const Corner2 &b, const Corner2 &t, float Asb, float Ast) {                        \
            const float Eb = b.u.m * b.B.m - vs.m * Asb, Et = t.u.m * t.B.m - vs.m * Ast;                      \
            return (SAT.m * Eb - SAB.m * Et - SAT.m * SAB.m * (t.A.m - b.A.m)) * iy.m;                         \
        };                                                                                                     \
        if (SB.m > 0.0f) E.m = SL.m > 0.0f ? plain(LL) : SR.m < 0.0f ? plain(RL) : across_x(LL, RL, BsLL.m, BsRL.m);       \
        else if (ST.m < 0.0f) E.m = SL.m > 0.0f ? plain(LR) : SR.m < 0.0f ? plain(RR) : across_x(LR, RR, BsLR.m, BsRR.m);  \
        else if (SL.m > 0.0f) E.m = across_y(LL, LR, AsLL.m, AsLR.m);                                          \
        else if (SR.m < 0.0f) E.m = across_y(RL, RR, AsRL.m, AsRR.m);                                          \
    }
    DG_ZONE(x)
    DG_ZONE(y)
#undef DG_ZONE
    return E;
}

// the edges of direction e of cells c and c + 1
template <int e>
__device__ __forceinline__ void edge_pair_emf(const Geo &G, const float *core, long long c, long long py, long long pz,
                                              const bool ok[2], const int i[2], const long long t[2], float dt,
                                              float *__restrict__ out) {
    const float smallp = (float)G.smallp;
    Corner2 LL, LR, RL, RR;
    if constexpr (e == 0) {
        LL = corner_pair<false, 0, +1, +1>(G, core, c - py - pz, smallp);
        RL = corner_pair<false, 0, -1, +1>(G, core, c - pz, smallp);
        LR = corner_pair<false, 0, +1, -1>(G, core, c - py, smallp);
        RR = corner_pair<false, 0, -1, -1>(G, core, c, smallp);
    } else if constexpr (e == 1) {
        LL = corner_pair<true, 1, +1, +1>(G, core, c - pz, smallp);
        RL = corner_pair<true, 1, +1, -1>(G, core, c, smallp);
        LR = corner_pair<false, 1, -1, +1>(G, core, c - pz, smallp);
        RR = corner_pair<false, 1, -1, -1>(G, core, c, smallp);
    } else {
        LL = corner_pair<true, 2, +1, +1>(G, core, c - py, smallp);
        RL = corner_pair<false, 2, -1, +1>(G, core, c - py, smallp);
        LR = corner_pair<true, 2, +1, -1>(G, core, c, smallp);
        RR = corner_pair<false, 2, -1, -1>(G, core, c, smallp);
    }
    const float half = 0.5f;
    LL.A = RL.A = half * (LL.A + RL.A);
    LR.A = RR.A = half * (LR.A + RR.A);
    LL.B = LR.B = half * (LL.B + LR.B);
    RL.B = RR.B = half * (RL.B + RR.B);
    V2 E = dt * hlld2d_2(LL, LR, RL, RR, (float)G.gamma);
    if ((G.omega0 > 0.0) && !G.fargo && e != 1) {  // edge_shear
#define DG_SHEAR(m, n)                                                                                     \
        {                                                                                                      \
            const float sh = (float)(-1.5 * G.omega0 * (e == 0 ? G.xc(i[n]) : 0.5 * (G.xc(i[n]) + G.xc(i[n] - 1)))); \
            if (e == 0) E.m += sh * (sh > 0.0f ? LL.B.m : RR.B.m) * dt;                                        \
            else E.m -= sh * (sh > 0.0f ? LL.A.m : RR.A.m) * dt;                                               \
        }
        DG_SHEAR(x, 0)
        DG_SHEAR(y, 1)
#undef DG_SHEAR
    }
    if (ok[0]) out[t[0]] = E.x;
    if (ok[1]) out[t[1]] = E.y;
}

// All six solves of a pair in one thread; faces = 0: the edges alone (the faces come from the network).
// 128 registers, 4 blocks per SM: 1.79 ms at 256^3 against k_riemann3d's 1.94, 0.231 against 0.255 at 128^3 (3
// blocks 1.99, 5 blocks, with spills, 1.88; one kind of solve per block as in k_riemann64 2.13, 6 such
// blocks 2.47).  With rows of odd length a pair is two loads and the kernel is slower than one cell per
// thread (101 x 75 x 53: 61 against 58 us): it runs where nx is even (riemann_pairs).
inline bool riemann_pairs(const Geo &G) { return G.CX % 2 == 0; }
__global__ void __launch_bounds__(kThreads, 4)
k_riemann32(const __grid_constant__ Geo G, const float *__restrict__ core, float *__restrict__ fx, float *__restrict__ fy,
            float *__restrict__ fz, float *__restrict__ ex, float *__restrict__ ey, float *__restrict__ ez,
            const Scalars *S, int faces) {
    const long long py = G.CX, pz = (long long)G.CX * G.CY;  // core index steps
    // pairs from the first plane with faces (k = 1) on; a row starts at an even place, so a pair lies in one row
    const long long c = pz + 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x);
    if (c >= G.csz) return;
    int i[2], j, k;
    split3((unsigned)c, G.dCX, G.dCY, i[0], j, k);
    if (j < 1 || k < 1) return;
    i[1] = i[0] + 1;
    const bool in = i[0] >= 1;  // the first of the pair: cell 0 has no face of its own
    long long t[2];
    t[1] = (long long)(i[1] - 1) + (long long)G.FX * ((j - 1) + (long long)G.FY * (k - 1));
    t[0] = t[1] - 1;
    const float dt = (float)S->dt;
    const bool x1 = i[1] <= G.nx, y1 = j <= G.ny, z1 = k <= G.nz;  // i[0] <= nx always: it is even, nx + 1 odd
    const bool all[2] = {in, true}, inner[2] = {in, x1};
    if (faces) {
        auto own = [&](int f) { return pair_at<false>(core, f, c); };
        auto xm = [&](int f) { return pair_at<true>(core, f, c); };
        auto ym = [&](int f) { return pair_at<false>(core, f, c - py); };
        auto zm = [&](int f) { return pair_at<false>(core, f, c - pz); };
        if (y1 && z1) face_pair_flux<0>(G, xm, own, all, i, t, dt, fx);
        if (z1 && (in || x1)) face_pair_flux<1>(G, ym, own, inner, i, t, dt, fy);
        if (y1 && (in || x1)) face_pair_flux<2>(G, zm, own, inner, i, t, dt, fz);
    }
    if (z1) edge_pair_emf<2>(G, core, c, py, pz, all, i, t, dt, ez);
    if (y1) edge_pair_emf<1>(G, core, c, py, pz, all, i, t, dt, ey);
    if (in || x1) edge_pair_emf<0>(G, core, c, py, pz, inner, i, t, dt, ex);
}

// HLLD for the faces the network sent back, two list entries per thread with the arithmetic of
// k_riemann32 (a face's flux is the same bit for bit whichever kernel solves it): 0.130 ms at 128^3 with
// scattered faces against 0.118 one entry per thread, the edge solves gaining 0.013
template <int d>
__global__ void __launch_bounds__(kThreads) k_nn_fallback32(const __grid_constant__ Geo G, const float *__restrict__ core,
                                                            float *__restrict__ flux, const int *__restrict__ list,
                                                            const unsigned long long *cnt, const Scalars *S) {
    const long long n = (long long)cnt[3 + d];
    const float dt = (float)S->dt;
    const long long step = d == 0 ? 1 : d == 1 ? G.CX : (long long)G.CX * G.CY;
    for (long long q = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x); q < n;
         q += 2 * (long long)gridDim.x * blockDim.x) {
        const bool ok[2] = {true, q + 1 < n};
        long long t[2], l[2], r[2];  // record, and the two cells' places in the core
        int i[2];
#pragma unroll
        for (int m = 0; m < 2; m++) {
            int j, k;
            t[m] = list[ok[m] ? q + m : q];
            split3((unsigned)t[m], G.dFX, G.dFY, i[m], j, k);
            i[m]++;
            const long long c = G.cidx(i[m], j + 1, k + 1);
            l[m] = core_base(c - step, kCore3);
            r[m] = core_base(c, kCore3);
        }
        auto left = [&](int f) { return p2(ld(core + l[0] + f * kCoreLane), ld(core + l[1] + f * kCoreLane)); };
        auto right = [&](int f) { return p2(ld(core + r[0] + f * kCoreLane), ld(core + r[1] + f * kCoreLane)); };
        face_pair_flux<d>(G, left, right, ok, i, t, dt, flux);
    }
}

}  // namespace
}  // namespace f32
}  // namespace dg
