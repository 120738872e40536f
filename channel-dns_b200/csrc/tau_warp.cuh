// The tau solve of one column by a warp: its recurrences as affine scans along the
// lanes of a parity (warp_columns.cuh).  It reassociates the sequential sums; the
// results agree with the sequential order to round-off.  Used where the order of
// operations is part of the result (solver_scan.cu, the flux column in solver.cu).
#pragma once

#include "warp_columns.cuh"

namespace cdns {

// Tau solve of (D^2 - k^2 - g) f = r with a f + b f' = (lower, upper) at
// y = (+1, -1), both parities at once (src/solver/eqsolve_pv.cpp:64-128).
// r must be zero beyond ny.  Returns false in a lane whose parity's pivot is
// zero or not finite.
template <int E>
__device__ bool tau_warp(int ny, double g, double a, double b, bool zero_col, double2 lower,
                         double2 upper, double w, const double2 (&r)[E], double2 (&out)[E],
                         const double (&ad)[E], const double *__restrict__ WL,
                         const double *__restrict__ WD, const double *__restrict__ WR) {
    const int L = lane_id(), p = L & 1;
    const bool normalize = g == 0.0 && a == 0.0 && zero_col;
    const int top = ((ny & 1) == p) ? ny : ny - 1;
    double2 rr[E];
#pragma unroll
    for (int e = 0; e < E; ++e) rr[e] = r[e];
    if (normalize) {
        // the even chain of the singular zero column is closed by the mean
        // (eqsolve_pv.cpp:71-79): r_0 <- sum_{y>=2 even} r_y/(y^2-1) + (lo+up)/(2b)
        double2 part = mk(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int y = ycoef<E>(e);
            if (p == 0 && y >= 2 && y <= ny) part = cadd(part, cdivr(r[e], (double)(y * y - 1)));
        }
        part = sum_parity(part);
        if (b != 0.0) part = cadd(part, cdivr(cadd(lower, upper), 2.0 * b));
        if (L == 0) rr[0] = part;
    }
    // three-term combination of the rhs
    double2 rm2_0 = shfl2_up(rr[E - 1], 2);
    double2 rp2_l = shfl2_down(rr[0], 2);
    if (L + 2 >= 32) rp2_l = mk(0.0, 0.0);
    double2 X[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        const double2 rm2 = e > 0 ? rr[(e + E - 1) % E] : rm2_0;
        const double2 rp2 = e + 1 < E ? rr[(e + 1) % E] : rp2_l;
        if (y > ny) X[e] = mk(0.0, 0.0);
        else if (y == p) X[e] = (p == 0) ? cdivr(cadd(lower, upper), 2.0) : cdivr(csub(lower, upper), 2.0);
        else if (y >= ny - 1) X[e] = cadd(cscale(WL[y], rm2), cscale(WD[y], rr[e]));
        else X[e] = cadd(cadd(cscale(WL[y], rm2), cscale(WD[y], rr[e])), cscale(WR[y], rp2));
    }
    // pivots one step up the chain, AD(y + 2)
    double adn_l = __shfl_down_sync(kFull, ad[0], 2);
    if (L + 2 >= 32) adn_l = 0.0;
    // backward sweep X_y -= (WR_y w AD_{y+2}) X_{y+2} for 2 <= y <= top - 2
    double A[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        const double adn = e + 1 < E ? ad[(e + 1) % E] : adn_l;
        A[e] = (y >= 2 && y <= top - 2) ? -((WR[y] * w) * adn) : 0.0;
    }
    affine_suffix<E>(A, X);
    // pivot chain ad01_j = tau(j) - (WL_{j+2} w ad01_{j+2}) AD_{j+2}, ad01_top = tau(top)
    double Aa[E], Ba[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        const double adn = e + 1 < E ? ad[(e + 1) % E] : adn_l;
        if (y > top) {
            Aa[e] = 0.0;
            Ba[e] = 0.0;
        } else if (y == top) {
            Aa[e] = 0.0;
            Ba[e] = tau_func(a, b, y);
        } else {
            Aa[e] = -((WL[y + 2] * w) * adn);
            Ba[e] = tau_func(a, b, y);
        }
    }
    affine_suffix<E>(Aa, Ba);
    // o0 = X_par - sum_{j = par+2..top} ad01_j AD_j X_j ; pivot ad01_par
    double2 s = mk(0.0, 0.0);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        if (y >= p + 2 && y <= top) s = cadd(s, cscale(Ba[e] * ad[e], X[e]));
    }
    s = sum_parity(s);
    double2 o0 = csub(shfl2(X[0], p), s);
    double piv = __shfl_sync(kFull, Ba[0], p);
    if (normalize && p == 0) {
        o0 = mk(0.0, 0.0);
        piv = 1.0;
    }
    const bool ok = isfinite(piv) && piv != 0.0;
    const double2 zpar = cdivr(o0, piv);
    // forward sweep Z_y = AD_y (X_y - WL_y w Z_{y-2})
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        if (y == p) {
            A[e] = 0.0;
            X[e] = zpar;
        } else if (y <= ny) {
            A[e] = -(ad[e] * (WL[y] * w));
            X[e] = cscale(ad[e], X[e]);
        } else {
            A[e] = 0.0;
            X[e] = mk(0.0, 0.0);
        }
    }
    affine_prefix<E>(A, X);
#pragma unroll
    for (int e = 0; e < E; ++e) out[e] = ycoef<E>(e) <= ny ? X[e] : mk(0.0, 0.0);
    return ok;
}

}  // namespace cdns
