// The column solve by warp scans (EqSolvePV, src/solver/eqsolve_pv.cpp): the form of
// the mixed-precision contexts.
//
// One warp owns one spectral column (kz, kx) and keeps all its y coefficients in
// registers; the tau recurrences (src/solver/eqsolve_pv.cpp:64-128) and Chebyshev
// derivatives (src/solver/vector_ops.cpp:17-25) are scans over the lanes of a parity
// (tau_warp.cuh).  A block of TC warps stages one tile of the state through swizzled
// shared memory; the influence-matrix and sigma corrections run over the block as one
// coalesced elementwise pass.
//
// Why mixed contexts do not take the sequential chains of solver.cu: the order of the
// operations is part of what they return.  The FP32 stages round every value that the
// FP64 solve leaves, so that a difference in its last bit becomes, here and there, one of
// 6e-8, and after some five steps the FP32 noise of two orders is unrelated.  The
// velocity shows that at 1e-8; dp/dx at a constant flow rate, a difference of fluxes that
// agree to 4e-6, at 1e-6; the pressure at 7e-7 (48 x 85 x 112, 8 steps).  Mixed results
// are held to 2e-7 of what this order gives.  The chains, with the curl inside, take 139
// us at 128 x 129 x 128, this kernel and k_curl 172 + 32 (201 with the curl inside and
// half of the influence fields, hence neither).  The Chebyshev transforms of FP32 stages
// keep their order, too (k_ydct_r), and no other form of them is taken (any_length.cu).
#include "cdns_kernels.cuh"
#include "tau_warp.cuh"

namespace cdns {

namespace {
constexpr int TC = kColsPerBlock;     // columns (warps) per block
constexpr int kThreads = 32 * TC;

template <int E>
__global__ void __launch_bounds__(kThreads, E <= 4 ? 2 : 1)
k_solve_scan(Dims d, Tables t, PhysParams pp, double g_v, SolverState st, StepArgs s) {
    chain_begin();
    extern __shared__ double2 tile[];   // [4][ncy][TC]
    __shared__ double2 s_c0[TC], s_c1[TC], s_sg[2][TC];   // per-column correction coefficients
    const int ncy = d.ncy, ny = d.NYS, nkx = d.nkx, ncol = d.ncol;
    const int S = ncy * TC;
    const int col0 = blockIdx.x * TC;
    const int tid = threadIdx.x;
    const int w = tid >> 5;
    const int L = tid & 31, p = L & 1;
    const int col = col0 + w;

    // ---- stage R = a0 u + a1 u_prev + b0 N + b1 N_prev and N_y -------------
#pragma unroll 2
    for (int i = tid; i < S; i += kThreads) {
        const int y = i / TC, l = i - (i / TC) * TC;
        const int c2 = col0 + l;
        if (c2 < ncol) {
            const int kzi = c2 / nkx, kx = c2 - (c2 / nkx) * nkx;
            const long long off = spectral_base(d, kzi, kx) + (long long)y * d.sy;
            const int sl = tile_slot<E>(y, l);
            double2 nv[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long o = c * d.Ns + off;
                nv[c] = s.N[o];
                // R (src/sim/simulation.cpp:151-158)
                tile[c * S + sl] = cadd(cadd(cadd(cscale(s.a0, s.u[o]), cscale(s.a1, s.u_prev[o])),
                                             cscale(s.b0, nv[c])),
                                        cscale(s.b1, s.N_prev[o]));
            }
            tile[3 * S + sl] = nv[1];
        }
    }
    __syncthreads();

    if (col < ncol) {
        const int kzi = col / nkx, kx = col - kzi * nkx;
        const double ax = t.wavx[kx], az = t.wavz[kzi];
        const bool zero_col = col == d.zc;
        const long long cm = (long long)col * ncy;   // column-major base
        bool pivot_fail = false;
        double2 pv[E], v0[E], v1[E], v2[E], dy[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int y = ycoef<E>(e);
            if (y <= ny) {
                const int sl = tile_slot<E>(y, w);
                v0[e] = tile[sl];
                v1[e] = tile[S + sl];
                v2[e] = tile[2 * S + sl];
                dy[e] = tile[3 * S + sl];
            } else {
                v0[e] = v1[e] = v2[e] = dy[e] = mk(0.0, 0.0);
            }
        }
        double2 lower, upper;
        if (s.bc_p) {
            lower = s.bc_p[col];
            upper = s.bc_p[ncol + col];
        } else {
            // pressure wall data (src/solver/eqsolve_pv.cpp:322-337)
            double2 st_ = mk(0, 0), sb_ = mk(0, 0);
#pragma unroll
            for (int e = 0; e < E; ++e) {
                st_ = cadd(st_, dy[e]);
                sb_ = p ? cadd(sb_, dy[e]) : csub(sb_, dy[e]);
            }
            st_ = sum_warp(st_);
            sb_ = sum_warp(sb_);
            const double2 bt = cadd(s.bw[col], st_);
            const double2 bb = cadd(s.bw[ncol + col], sb_);
            if (L == 0) {
                s.B_new[col] = bt;
                s.B_new[ncol + col] = bb;
            }
            // combined wall data b0 B + b1 B_prev (src/sim/simulation.cpp:146-150)
            lower = cadd(cscale(s.b0, bt), cscale(s.b1, s.B_prev[col]));
            upper = cadd(cscale(s.b0, bb), cscale(s.b1, s.B_prev[ncol + col]));
        }
        // divergence of R (src/solver/eqsolve_pv.cpp:340-357)
        deriv_warp<E>(ny, v1, dy);
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (ycoef<E>(e) <= ny) dy[e] = cadd(cadd(fderiv(ax, v0[e]), dy[e]), fderiv(az, v2[e]));
        // pressure
        double ad[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int y = ycoef<E>(e);
            ad[e] = y <= ny ? st.ad_p[cm + y] : 0.0;
        }
        pivot_fail |= !tau_warp<E>(ny, pp.G_pre, pp.a_pre0, pp.b_pre0, zero_col, lower, upper, st.wn_p[col], dy, pv,
                                   ad, t.WL, t.WD, t.WR);
        const double2 tail0 = elem<E>(v1, ny), tail1 = elem<E>(v1, ny - 1);
        // velocity: Re (grad P - R) (src/solver/eqsolve_pv.cpp:359-395)
        deriv_warp<E>(ny, pv, dy);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int y = ycoef<E>(e);
            ad[e] = y <= ny ? st.ad_v[cm + y] : 0.0;
        }
        const double wv = st.wn_v[col];
        auto velocity = [&](int c, double2(&vc)[E]) {
            double2 f[E];
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const double2 grad = (c == 0) ? fderiv(ax, pv[e]) : (c == 1) ? dy[e] : fderiv(az, pv[e]);
                f[e] = ycoef<E>(e) <= ny ? cscale(pp.Re, csub(grad, vc[e])) : mk(0.0, 0.0);
            }
            const double2 blo = s.bc_v[(2 * c) * ncol + col], bup = s.bc_v[(2 * c + 1) * ncol + col];
            pivot_fail |= !tau_warp<E>(ny, g_v, pp.a_V[c], pp.b_V[c], zero_col, blo, bup, wv, f, vc, ad,
                                       t.WL, t.WD, t.WR);
        };
        velocity(0, v0);
        velocity(1, v1);
        velocity(2, v2);
        // wall divergence by endpoint sums (src/solver/eqsolve_pv.cpp:397-406)
        double2 div0 = mk(0, 0), div1 = mk(0, 0);
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int y = ycoef<E>(e);
            const double2 tang = cadd(fderiv(ax, v0[e]), fderiv(az, v2[e]));
            const double2 nrm = cscale((double)(y * y), v1[e]);
            div0 = cadd(div0, cadd(tang, nrm));
            div1 = p ? cadd(div1, cadd(mk(-tang.x, -tang.y), nrm)) : cadd(div1, csub(tang, nrm));
        }
        div0 = sum_warp(div0);
        div1 = sum_warp(div1);
        // influence and sigma coefficients (src/solver/eqsolve_pv.cpp:408-429)
        const double2 i00 = st.inf_div[col], i01 = st.inf_div[ncol + col];
        const double2 i10 = st.inf_div[2 * ncol + col], i11 = st.inf_div[3 * ncol + col];
        const double2 c0 = csub(cmul(div1, i10), cmul(div0, i11));
        const double2 c1 = csub(cmul(div0, i01), cmul(div1, i00));
        const long long o_n = spectral_base(d, kzi, kx) + (long long)ny * d.sy, o_n1 = o_n - d.sy;
        const double2 ptop = cadd(elem<E>(pv, ny), cadd(inf_mul(c0, st.p_inf[o_n], false),
                                                        inf_mul(c1, st.p_inf[d.Ns + o_n], false)));
        const double2 vt0 = cadd(elem<E>(v1, ny), cadd(inf_mul(c0, st.v_inf[d.Ns + o_n], false),
                                                       inf_mul(c1, st.v_inf[4 * d.Ns + o_n], false)));
        const double2 vt1 = cadd(elem<E>(v1, ny - 1), cadd(inf_mul(c0, st.v_inf[d.Ns + o_n1], false),
                                                           inf_mul(c1, st.v_inf[4 * d.Ns + o_n1], false)));
        const double2 n0 = csub(cscale(-wv, vt0), cscale(pp.Re, tail0));
        const double2 n1 = cadd(cscale(-wv, vt1), cscale(pp.Re, csub(cscale(2.0 * ny, ptop), tail1)));
        if (L == 0) {
            s_c0[w] = c0;
            s_c1[w] = c1;
            s_sg[0][w] = cdiv(n0, st.sigma0[col]);
            s_sg[1][w] = cdiv(n1, st.sigma0[ncol + col]);
        }
        // uncorrected solution into the tile (each warp rewrites only its own column's slots)
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int y = ycoef<E>(e);
            if (y > ny) continue;
            const int sl = tile_slot<E>(y, w);
            tile[sl] = pv[e];
            tile[S + sl] = v0[e];
            tile[2 * S + sl] = v1[e];
            tile[3 * S + sl] = v2[e];
        }
        if (__any_sync(kFull, pivot_fail) && L == 0) atomicOr(s.err, ERR_PIVOT);
    }
    __syncthreads();

    // ---- influence and sigma corrections, coalesced over the block --------
    // odd-y coefficients take sigma_0 for p, u, w and sigma_1 for v; even-y the reverse
    const int zc = d.zc;   // the (kz, kx) = (0, 0) column (-1: not on this rank)
    const bool fix_zero = !s.solve_only && zc >= col0 && zc < col0 + TC;
    bool bad = false;
    for (int i = tid; i < S; i += kThreads) {
        const int y = i / TC, l = i - (i / TC) * TC;
        const int c2 = col0 + l;
        if (c2 >= ncol) continue;
        const int kzi = c2 / nkx, kx = c2 - (c2 / nkx) * nkx;
        const long long off = spectral_base(d, kzi, kx) + (long long)y * d.sy;
        const int sl = tile_slot<E>(y, l);
        const double2 c0 = s_c0[l], c1 = s_c1[l];
        const double2 sq = s_sg[(y + 1) & 1][l], sv = s_sg[y & 1][l];
        double2 pr = cadd(tile[sl], cadd(inf_mul(c0, st.p_inf[off], false), inf_mul(c1, st.p_inf[d.Ns + off], false)));
        pr = cadd(pr, inf_mul(sq, st.p_b[off], false));
        double2 v[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            v[c] = cadd(tile[(1 + c) * S + sl], cadd(inf_mul(c0, st.v_inf[c * d.Ns + off], inf_imag(c)),
                                                     inf_mul(c1, st.v_inf[(3 + c) * d.Ns + off], inf_imag(c))));
            v[c] = cadd(v[c], inf_mul(c == 1 ? sv : sq, st.v_b[c * d.Ns + off], inf_imag(c)));
        }
        if (fix_zero && c2 == zc) {
            tile[sl] = pr;
#pragma unroll
            for (int c = 0; c < 3; ++c) tile[(1 + c) * S + sl] = v[c];
            continue;
        }
        bad |= !(isfinite(pr.x) && isfinite(pr.y) && isfinite(v[0].x) && isfinite(v[0].y) && isfinite(v[1].x) &&
                 isfinite(v[1].y) && isfinite(v[2].x) && isfinite(v[2].y));
        s.p_out[off] = pr;
#pragma unroll
        for (int c = 0; c < 3; ++c) s.u_out[c * d.Ns + off] = v[c];
    }
    if (fix_zero) {
        __syncthreads();
        if (w == zc - col0) {
            double2 pz[E], u0[E], u1[E], u2[E];
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int y = ycoef<E>(e);
                const int sl = tile_slot<E>(y <= ny ? y : 0, w);
                pz[e] = tile[sl];
                u0[e] = tile[S + sl];
                u2[e] = tile[3 * S + sl];
            }
            // correct_zero_mode (src/solver/timestepper.cpp:60-68)
            const double2 v1w = cscale(0.5, cadd(s.bc_v[2 * ncol + zc], s.bc_v[3 * ncol + zc]));
#pragma unroll
            for (int e = 0; e < E; ++e) u1[e] = ycoef<E>(e) == 0 ? v1w : mk(0.0, 0.0);
            // correct_flow (src/sim/simulation.cpp:111-140), single-rank branch
            const double *uu = st.unit;
            double dpdx, dpdz;
            bool pfail = false;
            if (pp.grad_pre == 1) {
                dpdx = pp.gx;
                dpdz = pp.gz;
            } else {
                double qx = 0.0, qz = 0.0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int y = ycoef<E>(e);
                    if (p == 0 && y <= ny) {
                        qx += u0[e].x / (double)(y * y - 1);
                        qz += u2[e].x / (double)(y * y - 1);
                    }
                }
                qx = -sum_warp(qx);
                qz = -sum_warp(qz);
                const double qxu = uu[2 * ncy], qzu = uu[2 * ncy + 1];
                pfail = !isfinite(qxu) || qxu == 0.0 || !isfinite(qzu) || qzu == 0.0;
                dpdx = (pp.qxm - qx) / qxu;
                dpdz = (pp.qzm - qz) / qzu;
            }
            if (L == 0) {
                s.dpdx[0] = dpdx;
                s.dpdx[1] = dpdz;
                if (pfail) atomicOr(s.err, ERR_PIVOT);
            }
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int y = ycoef<E>(e);
                if (y > ny) continue;
                u0[e].x += dpdx * uu[y];
                u2[e].x += dpdz * uu[ncy + y];
                bad |= !(isfinite(pz[e].x) && isfinite(pz[e].y) && isfinite(u0[e].x) && isfinite(u0[e].y) &&
                         isfinite(u1[e].x) && isfinite(u1[e].y) && isfinite(u2[e].x) && isfinite(u2[e].y));
                const long long off = spectral_base(d, d.NZS, zc - d.NZS * nkx) + (long long)y * d.sy;
                s.p_out[off] = pz[e];
                s.u_out[off] = u0[e];
                s.u_out[d.Ns + off] = u1[e];
                s.u_out[2 * d.Ns + off] = u2[e];
            }
        }
    }
    if (__any_sync(kFull, bad) && L == 0) atomicOr(s.err, ERR_NONFINITE);
}

size_t scan_smem(const Dims &d) { return sizeof(double2) * 4 * (size_t)d.ncy * TC; }
}  // namespace

cudaError_t configure_scan_solve(const Dims &d) {
    cudaError_t e = cudaErrorInvalidValue;
    with_elems(d, [&](auto n) { e = raise_smem(k_solve_scan<decltype(n)::value>, scan_smem(d)); });
    return e;
}

void launch_scan_solve(const Dims &d, const Tables &t, const PhysParams &pp, double g_v, const SolverState &st,
                       const StepArgs &a, cudaStream_t s) {
    with_elems(d, [&](auto n) {
        launch_chained(k_solve_scan<decltype(n)::value>, (d.ncol + TC - 1) / TC, kThreads, scan_smem(d), s, d, t, pp,
                       g_v, st, a);
    });
}

}  // namespace cdns
