// rg_fast.cuh -- branch-free forms of the face step's arithmetic with the same bits.
//
// What bounds the face kernels in the plain forms is the latency of the FP64
// chains and the instructions around them, not the FP64 pipe (36 % busy in the
// brick face kernel at 16 warps per SM, 601 us at 128^3): every IEEE division
// and square root of the compiler carries a branch to its slow path, and every early return of a Riemann
// solver another, so nothing of a cell's two problems overlaps.  The forms
// here have no branch: quotients and roots come from a Newton iteration and a
// final correction that is correctly rounded for operands away from the ends
// of the exponent range, one reciprocal serves every quotient by the same
// divisor, selects replace the early returns, and what a form assumes about
// its operands is gathered in a Check that the caller looks at once per cell
// and direction; where it fails (ranges, floors, rare branches of the
// reference) the caller takes the plain form instead, so every result has the
// bits of the plain form.
//
// Division: y = RN(1/b) by Newton's iteration, q = RN(a y), r = RN(a - b q)
// (exact), q' = RN(q + r y) is RN(a/b) -- P. Markstein, IBM J. Res. Dev. 34
// (1990); with y known in advance: Brisebarre, Muller, Raina, IEEE Trans.
// Comput. 53 (2004).  Square root: Goldschmidt's iteration and the same kind
// of correction (Markstein; Cornea, Harrison, Tang, "Scientific Computing on
// Itanium-based Systems", ch. 7-8).  The seeds are the PTX approximations
// (2^-19.9 and 2^-19.0 relative, measured), so one cubic step reaches 2^-57.
// tests/test_gpu_fast_forms.py holds them to the IEEE operations on 2e9 random
// pairs and roots, numerators of 2^-600 .. 2^600 over divisors of 2^-130 ..
// 2^570, quotients, divisors and roots next to their hard cases among them.
// The results do not carry the sign of a negative zero numerator over a positive
// divisor; no numerator here can be one.
#pragma once

#include "rg_physics.cuh"

namespace rg {

// RN(1/b).  The last step rounds correctly from any value within an ulp of
// 1/b, but for a divisor whose significand is all ones only from above (from
// below it meets a tie: b = 1 - 2^-53 would give 1, and 1/b with it); so the
// cubic step adds 2^-55, more than its error and a quarter ulp at most.
__device__ __forceinline__ double rcp_fast(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    y = fma(y, fma(e, fma(-b, y, 2.0), 0x1p-55), y);
    return fma(y, fma(-b, y, 1.0), y);
}
// a / b with y = rcp_fast(b) (or the correctly rounded 1 / b)
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ double sqrt_fast(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    const double r = fma(-g, h, 0.5), t = fma(1.5 * r, r, r);
    g = fma(g, t, g);
    h = fma(h, t, h);
    return fma(fma(-g, g, x), h, g);
}

// Operand checks, gathered: magnitudes below 2^170 (finite with them) by the
// largest high word, numerators zero or above 2^-560 by the smallest (0 wraps
// to the top; a nonzero low word counts).  The divisors lie between 2^-67 (a
// pressure + 1e-20) and 2^410 (the HLLC's sum of density times wave speed, the
// density below 2^235 by gas()), or 2^600 in the exact solver, whose
// numerators there are above 2^-240; so no step of a quotient over- or
// underflows, and the remainder of the correction is exact.
//
// gas(): a pressure of at least 2^-64 times the density, from the difference
// of the high words (an exponent and the mantissa's leading bits: the ratio's
// logarithm within 0.1).  Then neither pressure floor (density times 1e-20 /
// gamma or 1e-20) nor the floor of the squared sound speed (1e-20) can act,
// gamma being above 1, and the forms leave the floors out; gas below that (a
// flow so fast that its thermal energy is lost in the rounding of the total,
// say) takes the forms with floors in the brick kernels, the plain ones
// elsewhere.  The bias keeps the difference positive for pressures below 2^170 over
// densities from 1e-10 on; a negative pressure's is far above the limit.
struct Check {
    static constexpr unsigned kTop = (1023u + 170u) << 20, kBottom = (1023u - 560u) << 20;
    static constexpr unsigned kBias = 204u << 20, kCold = kBias + (64u << 20);
    unsigned mx = 0, mn = 0xffffffffu, cold = 0;
    __device__ __forceinline__ void gas(double r, double p) {
        cold = max(cold, (unsigned)__double2hiint(r) - (unsigned)__double2hiint(p) + kBias);
        up(p);
    }
    __device__ __forceinline__ bool gas_ok() const { return cold < kCold; }
    __device__ __forceinline__ void up(double x) { mx = max(mx, (unsigned)__double2hiint(x) & 0x7fffffffu); }
    __device__ __forceinline__ void num(double a) {
        const unsigned h = ((unsigned)__double2hiint(a) & 0x7fffffffu) | min((unsigned)__double2loint(a), 1u);
        mn = min(mn, h - 1u);
    }
    __device__ __forceinline__ bool top_ok() const { return mx < kTop; }
    __device__ __forceinline__ bool num_ok() const { return mn >= kBottom; }
};

// Limited slope parameters: the slope types 1, 2, 3 and 8 (and those the
// reference treats as 1) are min(th min(|l|, |r|), cf |l + r|) with the sign of
// l where l r > 0, and so are the interpolation types 1..3 of the ghost
// branch: |l + r| >= max(|l|, |r|) there, so cf = 1 leaves a minmod as it is,
// and th = infinity the centred slope.
struct Limiter {
    double th, cf;
};
// CHK: the caller has not looked at the states, so the difference is checked
// (finite, not huge) here
template <bool CHK>
__device__ __forceinline__ double limited(double ql, double qc, double qr, const Limiter& L, Check& C) {
    const double l = qc - ql, r = qr - qc;
    const double c = L.cf * fabs(l + r);
    if (CHK) C.up(c);
    const double al = fabs(l), ar = fabs(r);
    double m = L.th * (ar < al ? ar : al);
    m = c < m ? c : m;
    m = copysign(m, l);
    return l * r > 0.0 ? m : 0.0;
}

// Cell sizes that keep the slopes' quotients in range.
__device__ __forceinline__ bool forms_take(double dx) { return dx > 0x1p-60 && dx < 0x1p60; }

// Values of a step the branch-free forms share (per cell size).
struct FastStep {
    double hdt, hdt0;       // dt / 2, and times zero: the tangential source term
    double dx, inv;         // cell size of the slope, its reciprocal
    double hdx;             // half the cell size
};
__device__ __forceinline__ FastStep fast_step(double dt, double dx, double inv) {
    return FastStep{0.5 * dt, 0.5 * dt * 0.0, dx, inv, 0.5 * dx};
}

// compute_slopes / ghost slopes and trace of a rotated state: the upper face
// state in qm, the lower in qp (either may be left out).  Primitive states:
// their density is at least 1e-10 (ctoprim).  The caller has checked the gas
// (gas_ok) and, without CHK, the states (top_ok); FLOOR: with the pressure
// floors, for gas that gas_ok refuses.
template <int NDIM, bool POW2, bool CHK, bool QM, bool QP, bool FLOOR = false>
__device__ __forceinline__ void trace_fast(const double* q, const double* ql, const double* qr, const Limiter& L,
                                           const FastStep& S, double gamma, double* qm, double* qp, Check& C) {
    constexpr int NV = Dims<NDIM>::NV, IP = Dims<NDIM>::IP;
    double dq[NV];
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        const double s = limited<CHK>(ql[iv], q[iv], qr[iv], L, C);
        if (POW2) {
            dq[iv] = s * S.inv;
        } else {
            C.num(s);
            dq[iv] = div_by(s, S.dx, S.inv);
        }
    }
    const double r = q[0], u = q[1], p = FLOOR ? smax(q[IP], r * 1e-20) : q[IP];
    const double y = rcp_fast(r);
    if (CHK) {
        if (FLOOR) {
            C.up(r);
            C.up(p);
        }
        C.up(dq[IP]);
    }
    C.num(dq[IP]);
    // (the floor of cs2, 1e-20, cannot act on a pressure of 1e-20 r or more: gamma - 1 is above 2^-20)
    const double cs2 = div_by(gamma * p, r, y);
    const double ru = dq[1] * r;
    const double b[3] = {S.hdt * (-u * dq[0] - ru), S.hdt * (-u * dq[1] - div_by(dq[IP], r, y)),
                         S.hdt * (-u * dq[IP] - ru * cs2)};
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        const double a = S.hdx * dq[iv];
        const double bb = iv == 0 ? b[0] : (iv == 1 ? b[1] : (iv == IP ? b[2] : S.hdt0));
        if (QP) qp[iv] = q[iv] - a + bb;
        if (QM) qm[iv] = q[iv] + a + bb;
    }
    if (QP && qp[0] < 1e-10) qp[0] = r;
    if (QM && qm[0] < 1e-10) qm[0] = r;
}

// The solvers' constants: gamma, gamma - 1 and its reciprocal, the pressure floor's factor.
struct FastGas {
    double gamma, gm1, rgm1, smallp;
    double g6, rg;  // (gamma + 1) / (2 gamma) and 1 / gamma: the exact solver's
    int fast;       // gamma - 1 in 2^-20 .. 2^20: quotients by it may use rgm1
};

// compute_flux and prim_to_cons of one state
template <int NDIM>
__device__ __forceinline__ void flux_cons(const double* q, const FastGas& G, double* f, double* u, Check& C) {
    constexpr int IP = Dims<NDIM>::IP;
    double v2 = q[1] * q[1];
#pragma unroll
    for (int i = 2; i <= NDIM; ++i) v2 = v2 + q[i] * q[i];
    const double E = 0.5 * q[0] * v2 + div_by(q[IP], G.gm1, G.rgm1);
    C.up(E);
    const double m = q[0] * q[1];
    f[0] = m;
    f[1] = m * q[1] + q[IP];
    u[0] = q[0];
    u[1] = m;
#pragma unroll
    for (int i = 2; i <= NDIM; ++i) {
        f[i] = m * q[i];
        u[i] = q[0] * q[i];
    }
    f[IP] = (E + q[IP]) * q[1];
    u[IP] = E;
}

template <int NDIM, bool FLOOR = false>
__device__ __forceinline__ double cs2_fast(const double* q, const FastGas& G, Check& C) {
    constexpr int IP = Dims<NDIM>::IP;
    if (!FLOOR) {
        C.up(q[1]);
        C.gas(q[0], q[IP]);
    }
    const double c2 = div_by(G.gamma * q[IP], q[0], rcp_fast(q[0]));
    return FLOOR ? smax(c2, 1e-20) : c2;
}
// Do the checks of a solver's states hold?  With floors the energies of both
// sides, which flux_cons checks, bound velocity and pressure; and a traced
// pressure is zero or above 2^-220, the state's being at least its floor.
template <bool FLOOR>
__device__ __forceinline__ bool states_ok(const Check& C) {
    return C.top_ok() && (FLOOR || C.gas_ok());
}

// The Riemann solvers on traced states (their density is at least 1e-10 by
// the trace's floor).  False: take the plain form.
template <int NDIM, bool FLOOR = false>
__device__ __forceinline__ bool hllc_fast(const double* ql, const double* qr, double* f, const FastGas& G) {
    constexpr int NV = Dims<NDIM>::NV, IP = Dims<NDIM>::IP;
    Check C;
    const double rl = ql[0], ul = ql[1], pl = FLOOR ? smax(ql[IP], rl * G.smallp) : ql[IP];
    const double rr = qr[0], ur = qr[1], pr = FLOOR ? smax(qr[IP], rr * G.smallp) : qr[IP];
    // the larger of two roots is the root of the larger: one root, same bits
    const double c2l = cs2_fast<NDIM, FLOOR>(ql, G, C), c2r = cs2_fast<NDIM, FLOOR>(qr, G, C);
    const double cmax = sqrt_fast(smax(c2l, c2r));
    const double sl = smin(ul, ur) - cmax, sr = smax(ul, ur) + cmax;
    const double rcl = rl * (ul - sl), rcr = rr * (sr - ur), div = rcr + rcl;
    const double nu = rcr * ur + rcl * ul + (pl - pr), np = rcr * pl + rcl * pr + rcl * rcr * (ul - ur);
    const double yd = rcp_fast(div);
    double ustar = div_by(nu, div, yd);  // (without floors its clamp to +-1e6 and that of den are checked below)
    if (FLOOR) ustar = smax(-1e6, smin(1e6, ustar));
    const double pstar = smax(div_by(np, div, yd), 0.0);
    const bool supl = sl > 0.0, supr = sr < 0.0, star = !(supl || supr);
    const bool left = supl || (!supr && ustar > 0.0);
    double q[NV], u0[NV];
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) q[iv] = left ? ql[iv] : qr[iv];
    flux_cons<NDIM>(q, G, f, u0, C);
    if (FLOOR) {
        C.up(rl);
        C.up(rr);
    }
    // nearly equal slow states (their density times wave speed below 1e-5): the mean of the two fluxes
    const bool mean = FLOOR && star && div < 1e-5;
    double fm[NV];
    if (FLOOR) {
        double qo[NV], uo[NV];
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) qo[iv] = left ? qr[iv] : ql[iv];
        flux_cons<NDIM>(qo, G, fm, uo, C);
#pragma unroll
        for (int iv = 0; iv < NV; ++iv) fm[iv] = 0.5 * (f[iv] + fm[iv]);
    }
    const bool base_ok = states_ok<FLOOR>(C);
    Check D;
    D.num(nu);
    D.num(np);
    const double so = left ? sl : sr;
    double den = so - ustar;
    if (FLOOR) den = left ? smin(den, -1e-10) : smax(den, 1e-10);
    const bool den_ok = FLOOR || (__double2hiint(den) ^ (left ? (int)0x80000000 : 0)) > __double2hiint(1e-10);
    const bool ustar_ok = FLOOR || (__double2hiint(ustar) & 0x7fffffff) < __double2hiint(1e6);
    const double yn = rcp_fast(den);
    const double w = so - q[1];
    const double rstar = div_by(q[0] * w, den, yn);
    const double ne = w * u0[IP] - (FLOOR ? (left ? pl : pr) : q[IP]) * q[1] + pstar * ustar;
    D.num(ne);
    double us[NV];
    us[0] = rstar;
    us[1] = rstar * ustar;
#pragma unroll
    for (int i = 2; i <= NDIM; ++i) us[i] = rstar * q[i];
    us[IP] = div_by(ne, den, yn);
#pragma unroll
    for (int iv = 0; iv < NV; ++iv) {
        const double fs = f[iv] + so * (us[iv] - u0[iv]);
        f[iv] = star ? fs : f[iv];
        if (FLOOR && mean) f[iv] = fm[iv];
    }
    return base_ok && (!star || mean || (D.num_ok() && den_ok && ustar_ok && !(div < 1e-5)));
}

template <int NDIM, bool FLOOR = false>
__device__ __forceinline__ bool llf_fast(const double* ql, const double* qr, double* f, const FastGas& G) {
    constexpr int NV = Dims<NDIM>::NV;
    Check C;
    double fl[NV], fr[NV], ul[NV], ur[NV];
    flux_cons<NDIM>(ql, G, fl, ul, C);
    flux_cons<NDIM>(qr, G, fr, ur, C);
    const double al = sqrt_fast(cs2_fast<NDIM, FLOOR>(ql, G, C)), ar = sqrt_fast(cs2_fast<NDIM, FLOOR>(qr, G, C));
    const double ha = 0.5 * smax(fabs(ql[1]) + al, fabs(qr[1]) + ar);
#pragma unroll
    for (int i = 0; i < NV; ++i) f[i] = 0.5 * (fl[i] + fr[i]) - ha * (ur[i] - ul[i]);
    return states_ok<FLOOR>(C);
}

template <int NDIM, bool FLOOR = false>
__device__ __forceinline__ bool hll_fast(const double* ql, const double* qr, double* f, const FastGas& G) {
    constexpr int NV = Dims<NDIM>::NV;
    Check C;
    double fl[NV], fr[NV], ul[NV], ur[NV];
    flux_cons<NDIM>(ql, G, fl, ul, C);
    flux_cons<NDIM>(qr, G, fr, ur, C);
    const double al = sqrt_fast(cs2_fast<NDIM, FLOOR>(ql, G, C)), ar = sqrt_fast(cs2_fast<NDIM, FLOOR>(qr, G, C));
    const double sl = smin(0.0, smin(ql[1] - al, qr[1] - ar)), sr = smax(0.0, smax(ql[1] + al, qr[1] + ar));
    const double w = sr - sl, inv = div_by(1.0, w, rcp_fast(w));
#pragma unroll
    for (int i = 0; i < NV; ++i) f[i] = (sr * fl[i] - sl * fr[i] + sr * sl * (ur[i] - ul[i])) * inv;
    return states_ok<FLOOR>(C) && !(w < 1e-20);
}

// One Newton update of the two-shock solver (RiemannSolver.cpp:221-233).
struct NewtonSide {
    double u, p, c, b, y;  // velocity, pressure, gamma p rho, p + 1e-20 and its reciprocal
};
__device__ __forceinline__ double newton_mass(const NewtonSide& s, double p, double g6) {
    return sqrt_fast(s.c * (1.0 + div_by(g6 * (p - s.p), s.b, s.y)));
}
__device__ __forceinline__ double newton_drop(const NewtonSide& s, double p, double w) {
    const double d = w + 1e-20;
    return div_by(p - s.p, d, rcp_fast(d));
}
__device__ __forceinline__ double newton_slope(const NewtonSide& s, double w) {
    const double w2 = w * w, d = w2 + s.c + 1e-20;
    return div_by(2.0 * (w2 * w), d, rcp_fast(d));
}
__device__ __forceinline__ double newton_update(const NewtonSide& l, const NewtonSide& r, double p, double g6, double* gap) {
    const double wl = newton_mass(l, p, g6), wr = newton_mass(r, p, g6);
    const double ql = newton_slope(l, wl), qr = newton_slope(r, wr);
    *gap = (l.u - newton_drop(l, p, wl)) - (r.u + newton_drop(r, p, wr));
    const double d = qr + ql + 1e-20;
    return smax(div_by(qr * ql, d, rcp_fast(d)) * *gap, -p);
}
// |d / p| < tol as the division gives it: the product decides unless it is
// within 2^-50 of the limit
__device__ __forceinline__ bool newton_done(double d, double p, double tol) {
    const double a = fabs(d), c = tol * p;
    if (fabs(a - c) <= c * 0x1p-50) return a / p < tol;
    return a < c;
}

// solve_exact_p (rg_physics.cuh) with the quotients and roots above, the same
// iteration, stop, polish and sampling.  gamma > 1; false: take the plain form.
template <int NDIM>
__device__ __forceinline__ bool exact_fast(const double* ql, const double* qr, double* flux, const FastGas& G, int niter,
                                           double tol, double p_guess, double* pstar_out, int* it_out) {
    constexpr int IP = Dims<NDIM>::IP;
    Check C;
    const double gamma = G.gamma, g6 = G.g6;
    const double rl = smax(ql[0], 1e-10), rr = smax(qr[0], 1e-10);
    NewtonSide L, R;
    L.u = ql[1];
    R.u = qr[1];
    L.p = smax(ql[IP], rl * G.smallp);
    R.p = smax(qr[IP], rr * G.smallp);
    L.c = gamma * L.p * rl;
    R.c = gamma * R.p * rr;
    L.b = L.p + 1e-20;
    R.b = R.p + 1e-20;
    L.y = rcp_fast(L.b);
    R.y = rcp_fast(R.b);
    C.up(rl);
    C.up(rr);
    C.up(L.u);
    C.up(R.u);
    C.up(L.p);
    C.up(R.p);
    const double wl = sqrt_fast(L.c), wr = sqrt_fast(R.c);
    const double ws = wl + wr + 1e-20, ns = wr * L.p + wl * R.p + wl * wr * (L.u - R.u);
    C.num(ns);
    double pstar = smax(div_by(ns, ws, rcp_fast(ws)), 0.0);
    if (p_guess > 0.0) pstar = p_guess;
    double pold = pstar;
    int it = 0;
    const bool safe = tol < 1e-6;
    double lo = 0.0, hi = CUDART_INF;
    for (int iter = 0; iter < niter; ++iter) {
        double gv;
        C.up(pold);
        const double delp = newton_update(L, R, pold, g6, &gv);
        ++it;
        if (safe) {
            if (gv > 0.0) lo = smax(lo, pold);
            else if (gv < 0.0) hi = smin(hi, pold);
            else break;
            double pn = pold + delp;
            if (newton_done(delp, pn + 1e-10, tol)) {
                pold = pn;
                break;
            }
            if (!((pn > lo || pn == 0.0) && pn < hi)) pn = hi < CUDART_INF ? 0.5 * (lo + hi) : 2.0 * lo + 1e-300;
            pold = pn;
            if (hi - lo <= tol * (lo + 1e-10)) break;
            continue;
        }
        pold = pold + delp;
        if (newton_done(delp, pold + 1e-10, tol)) break;
    }
    C.up(pold);
    if (safe) {
        pold = __longlong_as_double(__double_as_longlong(pold) & ~((1LL << 22) - 1));
        for (int k = 0; k < 2; ++k) {
            double gv;
            pold = pold + newton_update(L, R, pold, g6, &gv);
            C.up(pold);
        }
    }
    pstar = pold;
    if (pstar_out) *pstar_out = pstar;
    const double dl = newton_mass(L, pstar, g6) + 1e-20, dr = newton_mass(R, pstar, g6) + 1e-20;
    const double ustar = 0.5 * (L.u + div_by(L.p - pstar, dl, rcp_fast(dl)) + R.u - div_by(R.p - pstar, dr, rcp_fast(dr)));
    const bool left = ustar > 0;
    double ro = left ? rl : rr, po = left ? L.p : R.p;
    double rstar;
    C.num(pstar);
    if (pstar >= po) {
        const double d = G.gm1 * pstar + (gamma + 1.0) * po;
        rstar = div_by(ro * ((gamma + 1.0) * pstar + G.gm1 * po), d, rcp_fast(d));
    } else {
        rstar = ro * pow(div_by(pstar, left ? L.b : R.b, left ? L.y : R.y), G.rg);
    }
    rstar = smax(rstar, 1e-10);
    const double c2l = smax(div_by(gamma * L.p, rl, rcp_fast(rl)), 1e-20);
    const double c2r = smax(div_by(gamma * R.p, rr, rcp_fast(rr)), 1e-20);
    const double cm = sqrt_fast(smax(c2l, c2r));
    double uo;
    if (smin(L.u, R.u) - cm > 0.0) {
        ro = rl;
        uo = L.u;
        po = L.p;
    } else if (smax(L.u, R.u) + cm < 0.0) {
        ro = rr;
        uo = R.u;
        po = R.p;
    } else {
        ro = rstar;
        uo = ustar;
        po = pstar;
    }
    double e_kin = 0.5 * ro * uo * uo;
#pragma unroll
    for (int i = 2; i <= NDIM; ++i) {
        const double vt = left ? ql[i] : qr[i];
        e_kin = e_kin + 0.5 * ro * vt * vt;
    }
    const double E = div_by(po, G.gm1, G.rgm1) + e_kin;
    flux[0] = ro * uo;
    flux[1] = ro * uo * uo + po;
#pragma unroll
    for (int i = 2; i <= NDIM; ++i) flux[i] = flux[0] * (left ? ql[i] : qr[i]);
    flux[IP] = (E + po) * uo;
    *it_out = it;
    return C.top_ok() && C.num_ok();
}

}  // namespace rg
