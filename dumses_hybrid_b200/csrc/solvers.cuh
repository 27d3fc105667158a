// Riemann solvers of the MHD step as device functions, templated on the
// arithmetic type T (double for the plain path, float for the mixed path).
//
// 1D interface solvers (face fluxes), src/modules/solvers/solver.f90:
//   llf :393-498, hll :504-612, hlld :618-836, upwind :842-935.
//   State order: 0 rho, 1 P, 2 u_n, 3 B_n, 4 v_t1, 5 B_t1, 6 v_t2, 7 B_t2.
//   HLLD returns the normal-momentum flux without total pressure and the star
//   total pressure p*_T separately (solver.f90:818-833); the other solvers put
//   the pressure in the flux and report p*_T = 0 (pgstar is zeroed, :94-99).
// 2D edge solvers (EMFs), src/modules/solvers/solver_magnetic.f90:
//   llf :241-356, hlld :362-548, upwind :554-600, hlla :688-727.
//   Corner order LL, LR, RL, RR as set by solver_magnetic_utils (:32-49).
#pragma once
#include "dg_common.cuh"
#include "round64.cuh"

namespace dg {

// the square of the fast magnetosonic speed; the solvers that only need the largest of several
// speeds take one square root of the largest square: sqrt is monotone and correctly rounded, so
// sqrt(max(x)) is max(sqrt(x)) bit for bit (and the ternary max picks the same element either way)
template <typename T>
__device__ __forceinline__ T cfast2(T gamma, T ploc, T rho, T a, T b, T c) {
    const T half = T(0.5);
    T c2 = gamma * ploc / rho;
    T b2 = a * a + b * b + c * c;
    T d2 = half * (c2 + b2 / rho);
    return d2 + sqr(d2 * d2 - c2 * a * a / rho);
}
template <typename T>
__device__ __forceinline__ T cfast(T gamma, T ploc, T rho, T a, T b, T c) {
    return sqr(cfast2(gamma, ploc, rho, a, b, c));
}
// left/right physical fluxes and conserved states shared by llf, hll, upwind
template <typename T>
__device__ __forceinline__ void lr_fluxes(const T *ql, const T *qr, T gamma, T ciso, int iso,
                                          T *fl, T *cl, T *fr, T *cr, T &ploc, T &proc, T &a) {
    const T one = T(1), half = T(0.5);
    const T rl = ql[0], ul = ql[2], vl = ql[4], bl = ql[5], wl = ql[6], clv = ql[7];
    const T rr = qr[0], ur = qr[2], vr = qr[4], br = qr[5], wr = qr[6], crv = qr[7];
    const T entho = one / (gamma - one);
    a = half * (ql[3] + qr[3]);
    const T al = a, ar = a;
    if (iso) { ploc = rl * (ciso * ciso); proc = rr * (ciso * ciso); }
    else { ploc = ql[1]; proc = qr[1]; }
    T ecin = half * (ul * ul + vl * vl + wl * wl) * rl;
    T emag = half * (a * a + bl * bl + clv * clv);
    T etot = ploc * entho + ecin + emag;
    T ptot = ploc + emag;
    fl[0] = rl * ul;
    fl[1] = (etot + ptot) * ul - al * (ul * al + vl * bl + wl * clv);
    fl[2] = rl * ul * ul + ptot - al * al;
    fl[3] = T(0);
    fl[4] = rl * ul * vl - al * bl;
    fl[5] = bl * ul - al * vl;
    fl[6] = rl * ul * wl - al * clv;
    fl[7] = clv * ul - al * wl;
    cl[0] = rl; cl[1] = etot; cl[2] = rl * ul; cl[3] = al; cl[4] = rl * vl; cl[5] = bl; cl[6] = rl * wl; cl[7] = clv;
    ecin = half * (ur * ur + vr * vr + wr * wr) * rr;
    emag = half * (a * a + br * br + crv * crv);
    etot = proc * entho + ecin + emag;
    ptot = proc + emag;
    fr[0] = rr * ur;
    fr[1] = (etot + ptot) * ur - ar * (ur * ar + vr * br + wr * crv);
    fr[2] = rr * ur * ur + ptot - ar * ar;
    fr[3] = T(0);
    fr[4] = rr * ur * vr - ar * br;
    fr[5] = br * ur - ar * vr;
    fr[6] = rr * ur * wr - ar * crv;
    fr[7] = crv * ur - ar * wr;
    cr[0] = rr; cr[1] = etot; cr[2] = rr * ur; cr[3] = ar; cr[4] = rr * vr; cr[5] = br; cr[6] = rr * wr; cr[7] = crv;
}

template <typename T>
__device__ void llf1d(const T *ql, const T *qr, T *f, T gamma, T ciso, int iso) {
    const T half = T(0.5);
    T fl[8], cl[8], fr[8], cr[8], ploc, proc, a;
    lr_fluxes(ql, qr, gamma, ciso, iso, fl, cl, fr, cr, ploc, proc, a);
    T vleft = cfast(gamma, ploc, ql[0], a, ql[5], ql[7]) + fab(ql[2]);
    T vright = cfast(gamma, proc, qr[0], a, qr[5], qr[7]) + fab(qr[2]);
    T vel_info = mx(vleft, vright);
#pragma unroll
    for (int n = 0; n < 8; n++) f[n] = half * (fl[n] + fr[n]) - vel_info * half * (cr[n] - cl[n]);
}

template <typename T>
__device__ void hll1d(const T *ql, const T *qr, T *f, T gamma, T ciso, int iso) {
    T fl[8], cl[8], fr[8], cr[8], ploc, proc, a;
    lr_fluxes(ql, qr, gamma, ciso, iso, fl, cl, fr, cr, ploc, proc, a);
    const T cfmax = sqr(mx(cfast2(gamma, ploc, ql[0], a, ql[5], ql[7]), cfast2(gamma, proc, qr[0], a, qr[5], qr[7])));
    T ul = ql[2], ur = qr[2];
    T sl = mn(mn(ul, ur) - cfmax, T(0));
    T sr = mx(mx(ul, ur) + cfmax, T(0));
    if constexpr (sizeof(T) == 4) {
        const T is = T(1) / (sr - sl);
#pragma unroll
        for (int n = 0; n < 8; n++) f[n] = (sr * fl[n] - sl * fr[n] + sr * sl * (cr[n] - cl[n])) * is;
        return;
    }
#pragma unroll
    for (int n = 0; n < 8; n++) f[n] = (sr * fl[n] - sl * fr[n] + sr * sl * (cr[n] - cl[n])) / (sr - sl);
}

template <typename T>
__device__ void upwind1d(const T *ql, const T *qr, T *f, T gamma, T ciso, int iso) {
    const T half = T(0.5);
    T fl[8], cl[8], fr[8], cr[8], ploc, proc, a;
    lr_fluxes(ql, qr, gamma, ciso, iso, fl, cl, fr, cr, ploc, proc, a);
    T vleft = half * (ql[2] + qr[2]);
#pragma unroll
    for (int n = 0; n < 8; n++) f[n] = half * (fl[n] + fr[n]) - fab(vleft) * half * (cr[n] - cl[n]);
}

// ---------------------------------------------------------------------------
// FP32 forms of the same solvers for the mixed path: identical formulas, with each
// repeated divisor turned into one reciprocal (or reciprocal square root) and the
// fast-speed discriminant clamped at zero against FP32 rounding.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float cfast2_r(float gamma, float p, float irho, float a, float b, float c) {
    const float c2 = gamma * p * irho;
    const float d2 = 0.5f * (c2 + (a * a + b * b + c * c) * irho);
    return d2 + sqrtf(fmaxf(d2 * d2 - c2 * a * a * irho, 0.0f));
}
__device__ __forceinline__ float cfast_r(float gamma, float p, float irho, float a, float b, float c) {
    return sqrtf(cfast2_r(gamma, p, irho, a, b, c));
}

// packed FP32 (sm_100 FADD2 / FMUL2 / FFMA2: two lanes per instruction) for the mirrored
// left / right arithmetic of the solvers: x = left, y = right
__device__ __forceinline__ float2 p2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 s2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

__device__ __forceinline__ void hlld1d_f(const float *ql, const float *qr, float *f, float &pg, float gamma,
                                         float ciso, int iso, float entho) {
    const float half = 0.5f, zero = 0.0f;
    const float2 r = p2(ql[0], qr[0]), u = p2(ql[2], qr[2]), v = p2(ql[4], qr[4]), b = p2(ql[5], qr[5]);
    const float2 w = p2(ql[6], qr[6]), c = p2(ql[7], qr[7]);
    const float a = half * (ql[3] + qr[3]);
    const float aa = a * a;
    const float sgnm = copysignf(1.0f, a);
    const float2 p = iso ? mul2(r, s2(ciso * ciso)) : p2(ql[1], qr[1]);
    const float2 bsum = fma2(b, b, fma2(c, c, s2(aa)));  // a^2 + b^2 + c^2
    const float2 emag = mul2(s2(half), bsum);
    const float2 ke = fma2(u, u, fma2(v, v, mul2(w, w)));
    const float2 etot = fma2(p, s2(entho), fma2(mul2(s2(half), ke), r, emag));
    const float2 ptot = add2(p, emag);
    const float2 vdotb = fma2(u, s2(a), fma2(v, b, mul2(w, c)));
    // fast speeds (cfast2_r of each side), one square root of the larger
    const float2 irho = p2(1.0f / r.x, 1.0f / r.y);
    const float2 c2 = mul2(mul2(s2(gamma), p), irho);
    const float2 d2 = mul2(s2(half), fma2(bsum, irho, c2));
    const float2 disc = fma2(neg2(mul2(c2, s2(aa))), irho, mul2(d2, d2));
    const float cf = sqrtf(fmaxf(d2.x + sqrtf(fmaxf(disc.x, 0.0f)), d2.y + sqrtf(fmaxf(disc.y, 0.0f))));
    const float sl = fminf(u.x, u.y) - cf;
    const float sr = fmaxf(u.x, u.y) + cf;
    const float2 S = p2(sl, sr);
    const float2 Su = sub2(S, u);                     // (sl - ul, sr - ur)
    const float2 rSu = mul2(r, Su);
    const float2 rc = mul2(rSu, p2(-1.0f, 1.0f));     // (rl (ul - sl), rr (sr - ur))
    const float irc = 1.0f / (rc.y + rc.x);
    const float ustar = (rc.y * u.y + rc.x * u.x + (ptot.x - ptot.y)) * irc;
    const float ptotstar = (rc.y * ptot.x + rc.x * ptot.y + rc.x * rc.y * (u.x - u.y)) * irc;
    // single-star regions, left (x) and right (y)
    const float2 Sus = sub2(S, s2(ustar));
    const float2 is = p2(1.0f / Sus.x, 1.0f / Sus.y);
    const float2 rstar = mul2(rSu, is);
    const float2 estar = fma2(rSu, Sus, s2(-aa));
    const float2 e = fma2(rSu, Su, s2(-aa));
    const float2 ie = p2(estar.x != zero ? 1.0f / estar.x : zero, estar.y != zero ? 1.0f / estar.y : zero);
    const float2 adu_ie = mul2(mul2(s2(a), sub2(s2(ustar), u)), ie);
    const float2 eie = mul2(e, ie);
    float2 vstar = sub2(v, mul2(b, adu_ie)), wstar = sub2(w, mul2(c, adu_ie));
    float2 bstar = mul2(b, eie), cstar = mul2(c, eie);
    if (estar.x == zero) { vstar.x = v.x; bstar.x = b.x; wstar.x = w.x; cstar.x = c.x; }
    if (estar.y == zero) { vstar.y = v.y; bstar.y = b.y; wstar.y = w.y; cstar.y = c.y; }
    const float2 vdotbstar = fma2(s2(ustar), s2(a), fma2(vstar, bstar, mul2(wstar, cstar)));
    const float2 etotstar = mul2(fma2(Su, etot, fma2(neg2(ptot), u, fma2(s2(ptotstar), s2(ustar),
                                                                            mul2(s2(a), sub2(vdotb, vdotbstar))))), is);
    const float2 rs = p2(rsqrtf(rstar.x), rsqrtf(rstar.y));
    const float2 sqrr = mul2(rstar, rs);
    const float sal = ustar - fabsf(a) * rs.x;
    const float sar = ustar + fabsf(a) * rs.y;
    // double star region
    const float isum = 1.0f / (sqrr.x + sqrr.y);
    const float vstarstar = (sqrr.x * vstar.x + sqrr.y * vstar.y + sgnm * (bstar.y - bstar.x)) * isum;
    const float wstarstar = (sqrr.x * wstar.x + sqrr.y * wstar.y + sgnm * (cstar.y - cstar.x)) * isum;
    const float bstarstar = (sqrr.x * bstar.y + sqrr.y * bstar.x + sgnm * sqrr.x * sqrr.y * (vstar.y - vstar.x)) * isum;
    const float cstarstar = (sqrr.x * cstar.y + sqrr.y * cstar.x + sgnm * sqrr.x * sqrr.y * (wstar.y - wstar.x)) * isum;
    const float vdotbstarstar = ustar * a + vstarstar * bstarstar + wstarstar * cstarstar;
    // sample at x/t = 0
    float ro, uo, vo, wo, bo, co, ptoto, etoto, vdotbo;
    if (sl > zero) {
        ro = r.x; uo = u.x; vo = v.x; wo = w.x; bo = b.x; co = c.x; ptoto = ptot.x; etoto = etot.x; vdotbo = vdotb.x;
    } else if (sal > zero) {
        ro = rstar.x; uo = ustar; vo = vstar.x; wo = wstar.x; bo = bstar.x; co = cstar.x;
        ptoto = ptotstar; etoto = etotstar.x; vdotbo = vdotbstar.x;
    } else if (ustar > zero) {
        ro = rstar.x; uo = ustar; vo = vstarstar; wo = wstarstar; bo = bstarstar; co = cstarstar;
        ptoto = ptotstar; etoto = etotstar.x - sgnm * sqrr.x * (vdotbstar.x - vdotbstarstar); vdotbo = vdotbstarstar;
    } else if (sar > zero) {
        ro = rstar.y; uo = ustar; vo = vstarstar; wo = wstarstar; bo = bstarstar; co = cstarstar;
        ptoto = ptotstar; etoto = etotstar.y + sgnm * sqrr.y * (vdotbstar.y - vdotbstarstar); vdotbo = vdotbstarstar;
    } else if (sr > zero) {
        ro = rstar.y; uo = ustar; vo = vstar.y; wo = wstar.y; bo = bstar.y; co = cstar.y;
        ptoto = ptotstar; etoto = etotstar.y; vdotbo = vdotbstar.y;
    } else {
        ro = r.y; uo = u.y; vo = v.y; wo = w.y; bo = b.y; co = c.y; ptoto = ptot.y; etoto = etot.y; vdotbo = vdotb.y;
    }
    f[0] = ro * uo;
    f[1] = (etoto + ptoto) * uo - a * vdotbo;
    f[2] = ro * uo * uo - a * a;
    f[3] = zero;
    f[4] = ro * uo * vo - a * bo;
    f[5] = bo * uo - a * vo;
    f[6] = ro * uo * wo - a * co;
    f[7] = co * uo - a * wo;
    pg = ptoto;
}

// HLLD in FP64; returns p*_T in pg.  entho = 1 / (gamma - 1), the same for every interface of a run
// (formed once per context by the caller).  M: IeeeMath, or FastMath whose caller tests m.bad().
// Quotients by the negative sl - ustar are taken as (-numerator) / (ustar - sl), the same number.
template <class M>
__device__ __forceinline__ void hlld1d64(const double *ql, const double *qr, double *f, double &pg, double gamma,
                                         double ciso, int iso, double entho, M &m) {
    using T = double;
    const T half = T(0.5), zero = T(0);
    const T rl = ql[0], ul = ql[2], vl = ql[4], bl = ql[5], wl = ql[6], cl = ql[7];
    const T rr = qr[0], ur = qr[2], vr = qr[4], br = qr[5], wr = qr[6], cr = qr[7];
    const T a = half * (ql[3] + qr[3]);
    const T sgnm = sgn1(a);
    T ploc, proc;
    if (iso) { ploc = rl * (ciso * ciso); proc = rr * (ciso * ciso); }
    else { ploc = ql[1]; proc = qr[1]; }
    const T ecinl = half * (ul * ul + vl * vl + wl * wl) * rl;
    const T bsql = a * a + bl * bl + cl * cl;
    const T emagl = half * bsql;
    const T etotl = ploc * entho + ecinl + emagl;
    const T ptotl = ploc + emagl;
    const T vdotbl = ul * a + vl * bl + wl * cl;
    const T ecinr = half * (ur * ur + vr * vr + wr * wr) * rr;
    const T bsqr = a * a + br * br + cr * cr;
    const T emagr = half * bsqr;
    const T etotr = proc * entho + ecinr + emagr;
    const T ptotr = proc + emagr;
    const T vdotbr = ur * a + vr * br + wr * cr;
    // the fast speeds (cfast2 of each side), one root of the larger
    const auto irl = m.rec(rl), irr = m.rec(rr);
    const T c2l = m.div(gamma * ploc, rl, irl), c2r = m.div(gamma * proc, rr, irr);
    const T d2l = half * (c2l + m.div(bsql, rl, irl)), d2r = half * (c2r + m.div(bsqr, rr, irr));
    const T f2l = d2l + m.root(d2l * d2l - m.div(c2l * a * a, rl, irl));
    const T f2r = d2r + m.root(d2r * d2r - m.div(c2r * a * a, rr, irr));
    const T cfmax = m.root(mx(f2l, f2r));
    const T sl = mn(ul, ur) - cfmax;
    const T sr = mx(ul, ur) + cfmax;
    const T rcl = rl * (ul - sl);
    const T rcr = rr * (sr - ur);
    const T rcs = rcr + rcl;
    const auto ircs = m.rec(rcs);
    const T ustar = m.div(rcr * ur + rcl * ul + (ptotl - ptotr), rcs, ircs);
    const T ptotstar = m.div(rcr * ptotl + rcl * ptotr + rcl * rcr * (ul - ur), rcs, ircs);
    // left star region
    const T usl = ustar - sl;
    const auto iusl = m.rec(usl);
    const T rstarl = m.div(-(rl * (sl - ul)), usl, iusl);
    const T estarl = rl * (sl - ul) * (sl - ustar) - a * a;
    const T el = rl * (sl - ul) * (sl - ul) - a * a;
    T vstarl, bstarl, wstarl, cstarl;
    if (M::kZeroTest && estarl == zero) { vstarl = vl; bstarl = bl; wstarl = wl; cstarl = cl; }
    else {
        const auto ie = m.rec(estarl);
        vstarl = vl - m.div(a * bl * (ustar - ul), estarl, ie);
        bstarl = m.div(bl * el, estarl, ie);
        wstarl = wl - m.div(a * cl * (ustar - ul), estarl, ie);
        cstarl = m.div(cl * el, estarl, ie);
    }
    const T vdotbstarl = ustar * a + vstarl * bstarl + wstarl * cstarl;
    const T etotstarl = m.div(-((sl - ul) * etotl - ptotl * ul + ptotstar * ustar + a * (vdotbl - vdotbstarl)), usl, iusl);
    typename M::Rec isql, isqr;
    const T sqrrstarl = m.root(rstarl, isql);
    const T calfvenl = m.div(fab(a), sqrrstarl, isql);
    const T sal = ustar - calfvenl;
    // right star region
    const T sru = sr - ustar;
    const auto isru = m.rec(sru);
    const T rstarr = m.div(rr * (sr - ur), sru, isru);
    const T estarr = rr * (sr - ur) * (sr - ustar) - a * a;
    const T er = rr * (sr - ur) * (sr - ur) - a * a;
    T vstarr, bstarr, wstarr, cstarr;
    if (M::kZeroTest && estarr == zero) { vstarr = vr; bstarr = br; wstarr = wr; cstarr = cr; }
    else {
        const auto ie = m.rec(estarr);
        vstarr = vr - m.div(a * br * (ustar - ur), estarr, ie);
        bstarr = m.div(br * er, estarr, ie);
        wstarr = wr - m.div(a * cr * (ustar - ur), estarr, ie);
        cstarr = m.div(cr * er, estarr, ie);
    }
    const T vdotbstarr = ustar * a + vstarr * bstarr + wstarr * cstarr;
    const T etotstarr = m.div((sr - ur) * etotr - ptotr * ur + ptotstar * ustar + a * (vdotbr - vdotbstarr), sru, isru);
    const T sqrrstarr = m.root(rstarr, isqr);
    const T calfvenr = m.div(fab(a), sqrrstarr, isqr);
    const T sar = ustar + calfvenr;
    // double star region
    const T sqs = sqrrstarl + sqrrstarr;
    const auto isqs = m.rec(sqs);
    const T vstarstar = m.div(sqrrstarl * vstarl + sqrrstarr * vstarr + sgnm * (bstarr - bstarl), sqs, isqs);
    const T wstarstar = m.div(sqrrstarl * wstarl + sqrrstarr * wstarr + sgnm * (cstarr - cstarl), sqs, isqs);
    const T bstarstar = m.div(sqrrstarl * bstarr + sqrrstarr * bstarl + sgnm * sqrrstarl * sqrrstarr * (vstarr - vstarl), sqs, isqs);
    const T cstarstar = m.div(sqrrstarl * cstarr + sqrrstarr * cstarl + sgnm * sqrrstarl * sqrrstarr * (wstarr - wstarl), sqs, isqs);
    const T vdotbstarstar = ustar * a + vstarstar * bstarstar + wstarstar * cstarstar;
    const T etotstarstarl = etotstarl - sgnm * sqrrstarl * (vdotbstarl - vdotbstarstar);
    const T etotstarstarr = etotstarr + sgnm * sqrrstarr * (vdotbstarr - vdotbstarstar);
    // sample at x/t = 0
    T ro, uo, vo, wo, bo, co, ptoto, etoto, vdotbo;
    if (sl > zero) {
        ro = rl; uo = ul; vo = vl; wo = wl; bo = bl; co = cl; ptoto = ptotl; etoto = etotl; vdotbo = vdotbl;
    } else if (sal > zero) {
        ro = rstarl; uo = ustar; vo = vstarl; wo = wstarl; bo = bstarl; co = cstarl;
        ptoto = ptotstar; etoto = etotstarl; vdotbo = vdotbstarl;
    } else if (ustar > zero) {
        ro = rstarl; uo = ustar; vo = vstarstar; wo = wstarstar; bo = bstarstar; co = cstarstar;
        ptoto = ptotstar; etoto = etotstarstarl; vdotbo = vdotbstarstar;
    } else if (sar > zero) {
        ro = rstarr; uo = ustar; vo = vstarstar; wo = wstarstar; bo = bstarstar; co = cstarstar;
        ptoto = ptotstar; etoto = etotstarstarr; vdotbo = vdotbstarstar;
    } else if (sr > zero) {
        ro = rstarr; uo = ustar; vo = vstarr; wo = wstarr; bo = bstarr; co = cstarr;
        ptoto = ptotstar; etoto = etotstarr; vdotbo = vdotbstarr;
    } else {
        ro = rr; uo = ur; vo = vr; wo = wr; bo = br; co = cr; ptoto = ptotr; etoto = etotr; vdotbo = vdotbr;
    }
    f[0] = ro * uo;
    f[1] = (etoto + ptoto) * uo - a * vdotbo;
    f[2] = ro * uo * uo - a * a;
    f[3] = zero;
    f[4] = ro * uo * vo - a * bo;
    f[5] = bo * uo - a * vo;
    f[6] = ro * uo * wo - a * co;
    f[7] = co * uo - a * wo;
    pg = ptoto;
}

// HLLD, either arithmetic
template <typename T>
__device__ void hlld1d(const T *ql, const T *qr, T *f, T &pg, T gamma, T ciso, int iso, T entho) {
    if constexpr (sizeof(T) == 4) {
        hlld1d_f(ql, qr, f, pg, gamma, ciso, iso, entho);
    } else {
        IeeeMath m;
        hlld1d64(ql, qr, f, pg, gamma, ciso, iso, entho, m);
    }
}

// the four corner states of an edge after solver_magnetic_utils
template <typename T>
struct Corners {
    T rLL, rLR, rRL, rRR, pLL, pLR, pRL, pRR, uLL, uLR, uRL, uRR;
    T vLL, vLR, vRL, vRR, ALL, ALR, ARL, ARR, BLL, BLR, BRL, BRR;
    T CLL, CLR, CRL, CRR, ELL, ELR, ERL, ERR;
};

template <typename T> __device__ __forceinline__ T mn4(T a, T b, T c, T d) { return mn(mn(mn(a, b), c), d); }
template <typename T> __device__ __forceinline__ T mx4(T a, T b, T c, T d) { return mx(mx(mx(a, b), c), d); }
__device__ __forceinline__ float mn4(float a, float b, float c, float d) { return mn_nan(mn_nan(mn_nan(a, b), c), d); }
__device__ __forceinline__ float mx4(float a, float b, float c, float d) { return mx_nan(mx_nan(mx_nan(a, b), c), d); }

template <typename T>
__device__ T llf2d(const Corners<T> &c, T dt, T gamma, T ciso, int iso) {
    const T half = T(0.5), forth = T(0.25);
    T E = forth * (c.ELL + c.ERL + c.ELR + c.ERR);
    T rl = half * (c.rLL + c.rLR), pl = half * (c.pLL + c.pLR), ul = half * (c.uLL + c.uLR);
    T al = half * (c.ALL + c.ALR), bl = half * (c.BLL + c.BLR), cl = half * (c.CLL + c.CLR);
    T rr = half * (c.rRR + c.rRL), pr = half * (c.pRR + c.pRL), ur = half * (c.uRR + c.uRL);
    T ar = half * (c.ARR + c.ARL), br = half * (c.BRR + c.BRL), cr = half * (c.CRR + c.CRL);
    T ploc, proc;
    if (iso) { ploc = rl * (ciso * ciso); proc = rr * (ciso * ciso); } else { ploc = pl; proc = pr; }
    al = half * (al + ar); ar = al;
    T vleft = cfast(gamma, ploc, rl, al, bl, cl) + fab(ul);
    T vright = cfast(gamma, proc, rr, ar, br, cr) + fab(ur);
    T vel_info = mx(vleft, vright);
    T flux_x = -vel_info * half * (br - bl);
    rl = half * (c.rLL + c.rRL); pl = half * (c.pLL + c.pRL); ul = half * (c.vLL + c.vRL);
    al = half * (c.BLL + c.BRL); bl = half * (c.ALL + c.ARL); cl = half * (c.CLL + c.CRL);
    rr = half * (c.rRR + c.rLR); pr = half * (c.pRR + c.pLR); ur = half * (c.vRR + c.vLR);
    ar = half * (c.BRR + c.BLR); br = half * (c.ARR + c.ALR); cr = half * (c.CRR + c.CLR);
    if (iso) { ploc = rl * (ciso * ciso); proc = rr * (ciso * ciso); } else { ploc = pl; proc = pr; }
    al = half * (al + ar); ar = al;
    vleft = cfast(gamma, ploc, rl, al, bl, cl) + fab(ul);
    vright = cfast(gamma, proc, rr, ar, br, cr) + fab(ur);
    vel_info = mx(vleft, vright);
    T flux_y = -vel_info * half * (br - bl);
    T emf = E + (flux_x - flux_y);
    return emf * dt;
}

// FP32 form of hlld2d: per corner one reciprocal density, one sum of squares and one half trace
// shared by the x and y fast speeds and the total pressure; reciprocal square roots of the star
// densities.  Its kernel is bound by issue slots, so shared terms and one-instruction maxima count:
// k_riemann3d at 256^3 2.02 -> 1.93 ms.
__device__ __forceinline__ float hlld2d_f(const Corners<float> &c, float dt, float gamma) {
    const float half = 0.5f, zero = 0.0f, smallc = (float)kSmallc;
    auto corner = [&](float r, float p, float a, float b, float cc, float &fx, float &fy, float &pt) {
        const float ir = 1.0f / r, a2 = a * a, b2 = b * b, s2 = a2 + b2 + cc * cc;
        const float c2 = gamma * p * ir, d2 = half * (c2 + s2 * ir), dd = d2 * d2, k = c2 * ir;
        fx = d2 + sqrtf(fmaxf(dd - k * a2, zero));
        fy = d2 + sqrtf(fmaxf(dd - k * b2, zero));
        pt = p + half * s2;
    };
    float xLL, xLR, xRL, xRR, yLL, yLR, yRL, yRR, PtotLL, PtotLR, PtotRL, PtotRR;
    corner(c.rLL, c.pLL, c.ALL, c.BLL, c.CLL, xLL, yLL, PtotLL);
    corner(c.rLR, c.pLR, c.ALR, c.BLR, c.CLR, xLR, yLR, PtotLR);
    corner(c.rRL, c.pRL, c.ARL, c.BRL, c.CRL, xRL, yRL, PtotRL);
    corner(c.rRR, c.pRR, c.ARR, c.BRR, c.CRR, xRR, yRR, PtotRR);
    const float cfx = sqrtf(mx4(xLL, xLR, xRL, xRR)), cfy = sqrtf(mx4(yLL, yLR, yRL, yRR));
    const float SL = mn4(c.uLL, c.uLR, c.uRL, c.uRR) - cfx;
    const float SR = mx4(c.uLL, c.uLR, c.uRL, c.uRR) + cfx;
    const float SB = mn4(c.vLL, c.vLR, c.vRL, c.vRR) - cfy;
    const float ST = mx4(c.vLL, c.vLR, c.vRL, c.vRR) + cfy;
    const float rcLLx = c.rLL * (c.uLL - SL), rcRLx = c.rRL * (SR - c.uRL);
    const float rcLRx = c.rLR * (c.uLR - SL), rcRRx = c.rRR * (SR - c.uRR);
    const float rcLLy = c.rLL * (c.vLL - SB), rcLRy = c.rLR * (ST - c.vLR);
    const float rcRLy = c.rRL * (c.vRL - SB), rcRRy = c.rRR * (ST - c.vRR);
    const float ustar = (rcLLx * c.uLL + rcLRx * c.uLR + rcRLx * c.uRL + rcRRx * c.uRR + (PtotLL - PtotRL + PtotLR - PtotRR))
                      / (rcLLx + rcLRx + rcRLx + rcRRx);
    const float vstar = (rcLLy * c.vLL + rcLRy * c.vLR + rcRLy * c.vRL + rcRRy * c.vRR + (PtotLL - PtotLR + PtotRL - PtotRR))
                      / (rcLLy + rcLRy + rcRLy + rcRRy);
    const float SLustar = 1.0f / (SL - ustar), SRustar = 1.0f / (SR - ustar);
    const float SBvstar = 1.0f / (SB - vstar), STvstar = 1.0f / (ST - vstar);
    const float fLLx = (SL - c.uLL) * SLustar, fLLy = (SB - c.vLL) * SBvstar;
    const float fLRx = (SL - c.uLR) * SLustar, fLRy = (ST - c.vLR) * STvstar;
    const float fRLx = (SR - c.uRL) * SRustar, fRLy = (SB - c.vRL) * SBvstar;
    const float fRRx = (SR - c.uRR) * SRustar, fRRy = (ST - c.vRR) * STvstar;
    const float BstarLL = c.BLL * fLLx, AstarLL = c.ALL * fLLy;
    const float BstarLR = c.BLR * fLRx, AstarLR = c.ALR * fLRy;
    const float BstarRL = c.BRL * fRLx, AstarRL = c.ARL * fRLy;
    const float BstarRR = c.BRR * fRRx, AstarRR = c.ARR * fRRy;
    const float EstarLLx = ustar * BstarLL - c.vLL * c.ALL, EstarLLy = c.uLL * c.BLL - vstar * AstarLL;
    const float EstarLRx = ustar * BstarLR - c.vLR * c.ALR, EstarLRy = c.uLR * c.BLR - vstar * AstarLR;
    const float EstarRLx = ustar * BstarRL - c.vRL * c.ARL, EstarRLy = c.uRL * c.BRL - vstar * AstarRL;
    const float EstarRRx = ustar * BstarRR - c.vRR * c.ARR, EstarRRy = c.uRR * c.BRR - vstar * AstarRR;
    const float EstarLL = ustar * BstarLL - vstar * AstarLL, EstarLR = ustar * BstarLR - vstar * AstarLR;
    const float EstarRL = ustar * BstarRL - vstar * AstarRL, EstarRR = ustar * BstarRR - vstar * AstarRR;
    // 1/sqrt of rstar, rstarx, rstary per corner (rstar = rho fx fy)
    const float qLL = rsqrtf(c.rLL * fLLx * fLLy), qLR = rsqrtf(c.rLR * fLRx * fLRy);
    const float qRL = rsqrtf(c.rRL * fRLx * fRLy), qRR = rsqrtf(c.rRR * fRRx * fRRy);
    const float calfvenL = fmaxf(fmaxf(fmaxf(fmaxf(fabsf(c.ALR) * rsqrtf(c.rLR * fLRx), fabsf(AstarLR) * qLR),
                                             fabsf(c.ALL) * rsqrtf(c.rLL * fLLx)), fabsf(AstarLL) * qLL), smallc);
    const float calfvenR = fmaxf(fmaxf(fmaxf(fmaxf(fabsf(c.ARR) * rsqrtf(c.rRR * fRRx), fabsf(AstarRR) * qRR),
                                             fabsf(c.ARL) * rsqrtf(c.rRL * fRLx)), fabsf(AstarRL) * qRL), smallc);
    const float calfvenB = fmaxf(fmaxf(fmaxf(fmaxf(fabsf(c.BLL) * rsqrtf(c.rLL * fLLy), fabsf(BstarLL) * qLL),
                                             fabsf(c.BRL) * rsqrtf(c.rRL * fRLy)), fabsf(BstarRL) * qRL), smallc);
    const float calfvenT = fmaxf(fmaxf(fmaxf(fmaxf(fabsf(c.BLR) * rsqrtf(c.rLR * fLRy), fabsf(BstarLR) * qLR),
                                             fabsf(c.BRR) * rsqrtf(c.rRR * fRRy)), fabsf(BstarRR) * qRR), smallc);
    const float SAL = fminf(ustar - calfvenL, zero), SAR = fmaxf(ustar + calfvenR, zero);
    const float SAB = fminf(vstar - calfvenB, zero), SAT = fmaxf(vstar + calfvenT, zero);
    const float SARSAL = 1.0f / (SAR - SAL);
    const float SATSAB = 1.0f / (SAT - SAB);
    float E;
    if (SB > zero) {
        if (SL > zero) E = c.ELL;
        else if (SR < zero) E = c.ERL;
        else E = (SAR * EstarLLx - SAL * EstarRLx + SAR * SAL * (c.BRL - c.BLL)) * SARSAL;
    } else if (ST < zero) {
        if (SL > zero) E = c.ELR;
        else if (SR < zero) E = c.ERR;
        else E = (SAR * EstarLRx - SAL * EstarRRx + SAR * SAL * (c.BRR - c.BLR)) * SARSAL;
    } else if (SL > zero) {
        E = (SAT * EstarLLy - SAB * EstarLRy - SAT * SAB * (c.ALR - c.ALL)) * SATSAB;
    } else if (SR < zero) {
        E = (SAT * EstarRLy - SAB * EstarRRy - SAT * SAB * (c.ARR - c.ARL)) * SATSAB;
    } else {
        const float AstarT = (SAR * AstarRR - SAL * AstarLR) * SARSAL;
        const float AstarB = (SAR * AstarRL - SAL * AstarLL) * SARSAL;
        const float BstarR = (SAT * BstarRR - SAB * BstarRL) * SATSAB;
        const float BstarL = (SAT * BstarLR - SAB * BstarLL) * SATSAB;
        E = (SAL * SAB * EstarRR - SAL * SAT * EstarRL - SAR * SAB * EstarLR + SAR * SAT * EstarLL) * SARSAL * SATSAB
          - SAT * SAB * SATSAB * (AstarT - AstarB) + SAR * SAL * SARSAL * (BstarR - BstarL);
    }
    return E * dt;
}

// 2D HLLD in FP64 (M as in hlld1d64); reciprocals of the negative SL - ustar and SB - vstar are
// taken as -1 / (ustar - SL) and -1 / (vstar - SB)
template <class M>
__device__ __forceinline__ double hlld2d64(const Corners<double> &c, double dt, double gamma, M &m) {
    using T = double;
    const T half = T(0.5), zero = T(0), smallc = T(kSmallc);
    const T b2LL = c.ALL * c.ALL + c.BLL * c.BLL + c.CLL * c.CLL, b2LR = c.ALR * c.ALR + c.BLR * c.BLR + c.CLR * c.CLR;
    const T b2RL = c.ARL * c.ARL + c.BRL * c.BRL + c.CRL * c.CRL, b2RR = c.ARR * c.ARR + c.BRR * c.BRR + c.CRR * c.CRR;
    // the squared fast speeds of a corner along x and y (cfast2): c2 = gamma p / rho, the sum of the
    // squares in either order is the same number, so one quotient by rho serves both
    auto fast = [&](T p, T r, T a, T b, T b2, T &fx, T &fy) {
        const auto ir = m.rec(r);
        const T c2 = m.div(gamma * p, r, ir);
        const T d2 = half * (c2 + m.div(b2, r, ir));
        fx = d2 + m.root(d2 * d2 - m.div(c2 * a * a, r, ir));
        fy = d2 + m.root(d2 * d2 - m.div(c2 * b * b, r, ir));
    };
    T xLL, yLL, xLR, yLR, xRL, yRL, xRR, yRR;
    fast(c.pLL, c.rLL, c.ALL, c.BLL, b2LL, xLL, yLL);
    fast(c.pLR, c.rLR, c.ALR, c.BLR, b2LR, xLR, yLR);
    fast(c.pRL, c.rRL, c.ARL, c.BRL, b2RL, xRL, yRL);
    fast(c.pRR, c.rRR, c.ARR, c.BRR, b2RR, xRR, yRR);
    const T cfx = m.root(mx4(xLL, xLR, xRL, xRR));
    const T cfy = m.root(mx4(yLL, yLR, yRL, yRR));
    const T SL = mn4(c.uLL, c.uLR, c.uRL, c.uRR) - cfx;
    const T SR = mx4(c.uLL, c.uLR, c.uRL, c.uRR) + cfx;
    const T SB = mn4(c.vLL, c.vLR, c.vRL, c.vRR) - cfy;
    const T ST = mx4(c.vLL, c.vLR, c.vRL, c.vRR) + cfy;
    const T PtotLL = c.pLL + half * b2LL, PtotLR = c.pLR + half * b2LR;
    const T PtotRL = c.pRL + half * b2RL, PtotRR = c.pRR + half * b2RR;
    const T rcLLx = c.rLL * (c.uLL - SL), rcRLx = c.rRL * (SR - c.uRL);
    const T rcLRx = c.rLR * (c.uLR - SL), rcRRx = c.rRR * (SR - c.uRR);
    const T rcLLy = c.rLL * (c.vLL - SB), rcLRy = c.rLR * (ST - c.vLR);
    const T rcRLy = c.rRL * (c.vRL - SB), rcRRy = c.rRR * (ST - c.vRR);
    const T rcx = rcLLx + rcLRx + rcRLx + rcRRx, rcy = rcLLy + rcLRy + rcRLy + rcRRy;
    const T ustar = m.div(rcLLx * c.uLL + rcLRx * c.uLR + rcRLx * c.uRL + rcRRx * c.uRR + (PtotLL - PtotRL + PtotLR - PtotRR),
                          rcx, m.rec(rcx));
    const T vstar = m.div(rcLLy * c.vLL + rcLRy * c.vLR + rcRLy * c.vRL + rcRRy * c.vRR + (PtotLL - PtotLR + PtotRL - PtotRR),
                          rcy, m.rec(rcy));
    const T SLustar = -m.inv(ustar - SL), SRustar = m.inv(SR - ustar);
    const T SBvstar = -m.inv(vstar - SB), STvstar = m.inv(ST - vstar);
    const T rstarLLx = c.rLL * (SL - c.uLL) * SLustar;
    const T BstarLL = c.BLL * (SL - c.uLL) * SLustar;
    const T rstarLLy = c.rLL * (SB - c.vLL) * SBvstar;
    const T AstarLL = c.ALL * (SB - c.vLL) * SBvstar;
    const T rstarLL = c.rLL * (SL - c.uLL) * SLustar * (SB - c.vLL) * SBvstar;
    const T EstarLLx = ustar * BstarLL - c.vLL * c.ALL;
    const T EstarLLy = c.uLL * c.BLL - vstar * AstarLL;
    const T EstarLL = ustar * BstarLL - vstar * AstarLL;
    const T rstarLRx = c.rLR * (SL - c.uLR) * SLustar;
    const T BstarLR = c.BLR * (SL - c.uLR) * SLustar;
    const T rstarLRy = c.rLR * (ST - c.vLR) * STvstar;
    const T AstarLR = c.ALR * (ST - c.vLR) * STvstar;
    const T rstarLR = c.rLR * (SL - c.uLR) * SLustar * (ST - c.vLR) * STvstar;
    const T EstarLRx = ustar * BstarLR - c.vLR * c.ALR;
    const T EstarLRy = c.uLR * c.BLR - vstar * AstarLR;
    const T EstarLR = ustar * BstarLR - vstar * AstarLR;
    const T rstarRLx = c.rRL * (SR - c.uRL) * SRustar;
    const T BstarRL = c.BRL * (SR - c.uRL) * SRustar;
    const T rstarRLy = c.rRL * (SB - c.vRL) * SBvstar;
    const T AstarRL = c.ARL * (SB - c.vRL) * SBvstar;
    const T rstarRL = c.rRL * (SR - c.uRL) * SRustar * (SB - c.vRL) * SBvstar;
    const T EstarRLx = ustar * BstarRL - c.vRL * c.ARL;
    const T EstarRLy = c.uRL * c.BRL - vstar * AstarRL;
    const T EstarRL = ustar * BstarRL - vstar * AstarRL;
    const T rstarRRx = c.rRR * (SR - c.uRR) * SRustar;
    const T BstarRR = c.BRR * (SR - c.uRR) * SRustar;
    const T rstarRRy = c.rRR * (ST - c.vRR) * STvstar;
    const T AstarRR = c.ARR * (ST - c.vRR) * STvstar;
    const T rstarRR = c.rRR * (SR - c.uRR) * SRustar * (ST - c.vRR) * STvstar;
    const T EstarRRx = ustar * BstarRR - c.vRR * c.ARR;
    const T EstarRRy = c.uRR * c.BRR - vstar * AstarRR;
    const T EstarRR = ustar * BstarRR - vstar * AstarRR;
    const T sqrtrstarLR = m.inv_root(rstarLR);
    const T sqrtrstarRL = m.inv_root(rstarRL);
    const T sqrtrstarRR = m.inv_root(rstarRR);
    const T sqrtrstarLL = m.inv_root(rstarLL);
    auto per_root = [&](T a, T r) {  // |a| / sqrt(r)
        typename M::Rec z;
        const T s = m.root(r, z);
        return m.div(fab(a), s, z);
    };
    const T calfvenL = mx(mx(mx(mx(per_root(c.ALR, rstarLRx), fab(AstarLR) * sqrtrstarLR),
                                per_root(c.ALL, rstarLLx)), fab(AstarLL) * sqrtrstarLL), smallc);
    const T calfvenR = mx(mx(mx(mx(per_root(c.ARR, rstarRRx), fab(AstarRR) * sqrtrstarRR),
                                per_root(c.ARL, rstarRLx)), fab(AstarRL) * sqrtrstarRL), smallc);
    const T calfvenB = mx(mx(mx(mx(per_root(c.BLL, rstarLLy), fab(BstarLL) * sqrtrstarLL),
                                per_root(c.BRL, rstarRLy)), fab(BstarRL) * sqrtrstarRL), smallc);
    const T calfvenT = mx(mx(mx(mx(per_root(c.BLR, rstarLRy), fab(BstarLR) * sqrtrstarLR),
                                per_root(c.BRR, rstarRRy)), fab(BstarRR) * sqrtrstarRR), smallc);
    const T SAL = mn(ustar - calfvenL, zero), SAR = mx(ustar + calfvenR, zero);
    const T SAB = mn(vstar - calfvenB, zero), SAT = mx(vstar + calfvenT, zero);
    const T SARSAL = m.inv(SAR - SAL);
    const T SATSAB = m.inv(SAT - SAB);
    const T AstarT = (SAR * AstarRR - SAL * AstarLR) * SARSAL;
    const T AstarB = (SAR * AstarRL - SAL * AstarLL) * SARSAL;
    const T BstarR = (SAT * BstarRR - SAB * BstarRL) * SATSAB;
    const T BstarL = (SAT * BstarLR - SAB * BstarLL) * SATSAB;
    T E;
    if (SB > zero) {
        if (SL > zero) E = c.ELL;
        else if (SR < zero) E = c.ERL;
        else E = (SAR * EstarLLx - SAL * EstarRLx + SAR * SAL * (c.BRL - c.BLL)) * SARSAL;
    } else if (ST < zero) {
        if (SL > zero) E = c.ELR;
        else if (SR < zero) E = c.ERR;
        else E = (SAR * EstarLRx - SAL * EstarRRx + SAR * SAL * (c.BRR - c.BLR)) * SARSAL;
    } else if (SL > zero) {
        E = (SAT * EstarLLy - SAB * EstarLRy - SAT * SAB * (c.ALR - c.ALL)) * SATSAB;
    } else if (SR < zero) {
        E = (SAT * EstarRLy - SAB * EstarRRy - SAT * SAB * (c.ARR - c.ARL)) * SATSAB;
    } else {
        E = (SAL * SAB * EstarRR - SAL * SAT * EstarRL - SAR * SAB * EstarLR + SAR * SAT * EstarLL) * SARSAL * SATSAB
          - SAT * SAB * SATSAB * (AstarT - AstarB) + SAR * SAL * SARSAL * (BstarR - BstarL);
    }
    return E * dt;
}

template <typename T>
__device__ T hlld2d(const Corners<T> &c, T dt, T gamma) {
    if constexpr (sizeof(T) == 4) {
        return hlld2d_f(c, dt, gamma);
    } else {
        IeeeMath m;
        return hlld2d64(c, dt, gamma, m);
    }
}

template <typename T>
__device__ T upwind2d(const Corners<T> &c, T dt) {
    const T half = T(0.5), forth = T(0.25);
    T E = forth * (c.ELL + c.ERL + c.ELR + c.ERR);
    T ul = half * (c.uLL + c.uLR), bl = half * (c.BLL + c.BLR);
    T ur = half * (c.uRR + c.uRL), br = half * (c.BRR + c.BRL);
    T vel_info = half * (ul + ur);
    T flux_x = -fab(vel_info) * half * (br - bl);
    ul = half * (c.vLL + c.vRL); bl = half * (c.ALL + c.ARL);
    ur = half * (c.vRR + c.vLR); br = half * (c.ARR + c.ALR);
    vel_info = half * (ul + ur);
    T flux_y = -fab(vel_info) * half * (br - bl);
    T emf = E + (flux_x - flux_y);
    return emf * dt;
}

template <typename T>
__device__ T hlla2d(const Corners<T> &c, T dt) {
    const T zero = T(0), smallc = T(kSmallc);
    const T cLLx = sqr(c.ALL * c.ALL / c.rLL), cLRx = sqr(c.ALR * c.ALR / c.rLR);
    const T cRLx = sqr(c.ARL * c.ARL / c.rRL), cRRx = sqr(c.ARR * c.ARR / c.rRR);
    const T cLLy = sqr(c.BLL * c.BLL / c.rLL), cLRy = sqr(c.BLR * c.BLR / c.rLR);
    const T cRLy = sqr(c.BRL * c.BRL / c.rRL), cRRy = sqr(c.BRR * c.BRR / c.rRR);
    const T SL = mn(mn4(c.uLL, c.uLR, c.uRL, c.uRR) - mx(mx4(cLLx, cLRx, cRLx, cRRx), smallc), zero);
    const T SR = mx(mx4(c.uLL, c.uLR, c.uRL, c.uRR) + mx(mx4(cLLx, cLRx, cRLx, cRRx), smallc), zero);
    const T SB = mn(mn4(c.vLL, c.vLR, c.vRL, c.vRR) - mx(mx4(cLLy, cLRy, cRLy, cRRy), smallc), zero);
    const T ST = mx(mx4(c.vLL, c.vLR, c.vRL, c.vRR) + mx(mx4(cLLy, cLRy, cRLy, cRRy), smallc), zero);
    T emf = (SL * SB * c.ERR - SL * ST * c.ERL - SR * SB * c.ELR + SR * ST * c.ELL) / (SR - SL) / (ST - SB)
          - ST * SB / (ST - SB) * (c.ARR - c.ALL) + SR * SL / (SR - SL) * (c.BRR - c.BLL);
    return emf * dt;
}

}  // namespace dg
