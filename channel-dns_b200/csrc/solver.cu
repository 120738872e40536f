// Per-(kz, kx) Chebyshev-tau pressure/velocity solve of the channel-dns step
// (EqSolvePV, src/solver/eqsolve_pv.cpp) for sm_100a.
//
// Every tau recurrence (src/solver/eqsolve_pv.cpp:64-128) and every Chebyshev
// derivative recurrence (src/solver/vector_ops.cpp:17-25) couples only
// coefficients of one parity of y, and its multipliers are real: a column is
// four independent scalar chains per field, (parity, re/im).  One thread runs
// one chain sequentially over columns staged in shared memory: a block holds TC
// consecutive columns, a warp the 4 TC chains of one field, so that a row of the
// tile is read by 16 lanes as 128 consecutive bytes.  The whole solve is two sweeps down and up the chain for the pressure
// (one warp) and two for the velocity (three warps, one per component); the
// right-hand sides (divergence of R, Re (grad P - R)) are formed inside the
// downward sweep and the wall sums inside the upward one.
//
// The influence-matrix and sigma corrections then run over the block as one
// coalesced elementwise pass over the influence and B-problem fields
// (solver_setup.cu).  Three symmetries cut what that pass reads from twelve
// real fields to six over the kz <= 0 half:
//   - the second influence response is the mirror image of the first under
//     y -> -y (the wall conditions are the same on both sides): its pressure, u
//     and w coefficients are (-1)^y times the first's, its v -(-1)^y times;
//   - u and w are i kx phi and i kz phi of one phi where u and w have the same
//     wall condition, so one of the two gives the other;
//   - column -kz has the same pressure, u, v and pivots and w negated.
// Two things keep the warp scans that this form replaced, because the order of the
// operations shows in what they give: the mixed form (solver_scan.cu) and the column
// that gives dp/dx and the mean wall shear (flux_column).
// The curl of the new velocity (vector_ops.cpp:112-151) and its wall sums are
// formed from the columns while they are in shared memory.
// What bounds it: the chains' latency at 12 warps per SM against the streams
// of the multistep state (317 MB of DRAM, 2.3 TB/s); blocks of kz and -kz run next
// to each other, so the half fields are read from HBM once.  At 128 x 129 x 128 138
// us; a warp per column with shuffle scans, twelve fields and a curl kernel of its
// own took 176 + 32 us.
#include "cdns_kernels.cuh"
#include "tau_warp.cuh"

namespace cdns {

namespace {
constexpr int TC = kColsPerBlock;     // columns per block
constexpr int kThreads = 128;         // warp 0: pressure; warps 0-2: velocity; all: staging
constexpr int kRowGroups = kThreads / TC;

// Loads with a prefetch of the 256-byte neighbourhood.  They read what the kernel before
// wrote: volatile and with a memory clobber, so that none moves above chain_begin's wait
// or across a barrier.
__device__ __forceinline__ double2 ld256(const double2 *p) {
    double2 v;
    asm volatile("ld.global.L2::256B.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double ld256(const double *p) {
    double v;
    asm volatile("ld.global.L2::256B.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}
struct SolveArgs {
    double p_a, p_b;           // pressure wall condition a P + b dP/dn
    double2 *p_out;            // [Ns]
    double2 *v_out;            // [3][Ns]
    StepArgs step;
};

// Row stride of the staged pivots [TC][ncy]: = 2 (mod 16) doubles, so that the
// chains of one warp (columns l, parities p: offset l stride + p) fall on
// distinct banks.
__host__ __device__ inline int pivot_stride(int ncy) { return ncy + ((2 - ncy % 16) + 16) % 16; }

// Rows of a chain that are worked on together.  One warp runs 32 chains, so a
// chain costs what its instructions cost in sequence: a row has two dependent
// operations of the recurrence (9 cycles each) and about 15 that do not depend
// on it and overlap with those of the other rows of a group.
constexpr int kRows = 4;

// One chain of the tau solve of (D^2 - k^2 - g) f = r with a f + b f' =
// (lower, upper) at y = (+1, -1): the coefficients of parity p of one scalar
// part (re or im) of one column, in f[y * 2 TC].
//   down  X_y = t_y - (WR w AD_{y+2}) X_{y+2},  t_y = WL r_{y-2} + WD r_y + WR r_{y+2},
//         o = X_p - sum ad01_y AD_y X_y, ad01_{y-2} = tau(y-2) - (WL_y w AD_y) ad01_y
//   up    Z_p = o / ad01_p,  Z_y = AD_y X_y - (WL_y w AD_y) Z_{y-2}
// carried as g_y = AD_y X_y, which is what f holds between the sweeps.  As WD =
// -(WL + WR) (half of WL at y = 2, where r_0 counts twice), t_y = WL D_y - WR
// D_{y+2} with the differences D_y = r_{y-2} - r_y, D_2 = r_0 - r_2 / 2: a y
// derivative in r then is a local term, 2 (y - 1) f_{y-1}, and needs no recurrence
// of its own.  The two top rows, where the tau truncation drops terms, are written
// out.  rhs.start(top) returns r_top; rhs.load(i, y) fetches the operands of row y
// into slot i, rhs.diff(i, yd) returns D_y (yd = y, rows descending), rhs.diff2(i) D_2.
// W[y] = (WL, WR).  acc(yd, Z_y) sees the solution.  Returns false if the pivot is
// zero or not finite.
template <class Rhs, class Acc>
__device__ __forceinline__ bool tau_chain(int ny, int p, double a, double b, bool normalize, double lower,
                                          double upper, double w, const double2 *W,
                                          const double *__restrict__ WD, const double *ad, double *f, Rhs &rhs,
                                          Acc &&acc) {
    const int top = ((ny & 1) == p) ? ny : ny - 1;
    // diagonal of the boundary row, tau(y) = ta + tb y^2 (eqsolve_pv.cpp:64-70)
    const bool dir = a == 0.0 && b == 0.0;
    const double ta = dir ? (double)p : a, tb = dir ? (double)(1 - p) : b;
    const double x0 = p ? (lower - upper) / 2.0 : (lower + upper) / 2.0;
    const bool even_zero = normalize && p == 0;
    double d2 = 0.0;
    if (even_zero) {
        // the even chain of the singular zero column is closed by the mean
        // (eqsolve_pv.cpp:71-79): r_0 <- sum_{y>=2 even} r_y/(y^2-1) + (lo+up)/(2b)
        Rhs pre = rhs;
        double r = pre.start(top), corr = 0.0;
        for (int y = top; y >= 2; y -= 2) {
            const double yq = (double)y;
            corr += r / (yq * yq - 1.0);
            if (y == 2) break;
            pre.load(0, y);
            r += pre.diff(0, yq);
        }
        if (b != 0.0) corr += (lower + upper) / (2.0 * b);
        d2 = corr - 0.5 * r;
    }
    double yd = (double)top, ad01 = ta + tb * (yd * yd), g = 0.0, o = 0.0, dup = 0.0;   // dup = D_{y+2}
    // one row: g_y from t_y; the boundary sum and its next multiplier
    auto row = [&](int y, double t, double av, double2 wy) {
        const double wa = w * av;
        g = av * t - (wa * wy.y) * g;
        o += ad01 * g;
        yd -= 2.0;
        ad01 = (ta + tb * (yd * yd)) - (wa * wy.x) * ad01;
        f[y * (2 * TC)] = g;
    };
    int y = top;
    {
        const double r0 = rhs.start(top);
        rhs.load(0, y);
        const double dt = rhs.diff(0, yd), r1 = dt + r0;   // r_{top-2}
        row(y, W[y].x * r1, ad[y], W[y]);
        y -= 2;
        if (y >= 2) {
            rhs.load(0, y);
            dup = y > 2 ? rhs.diff(0, yd) : even_zero ? d2 : rhs.diff2(0);
            row(y, W[y].x * (dup + (y > 2 ? r1 : 0.5 * r1)) + WD[y] * r1, ad[y], W[y]);
            y -= 2;
        }
    }
    for (; y - 2 * (kRows - 1) >= 3; y -= 2 * kRows) {
        double av[kRows], t[kRows];
        double2 wy[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            rhs.load(i, y - 2 * i);
            wy[i] = W[y - 2 * i];
            av[i] = ad[y - 2 * i];
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const double dq = rhs.diff(i, yd - (double)(2 * i));
            t[i] = wy[i].x * dq - wy[i].y * dup;
            dup = dq;
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) row(y - 2 * i, t[i], av[i], wy[i]);
    }
    for (; y >= 2; y -= 2) {
        rhs.load(0, y);
        const double2 wy = W[y];
        const double dq = y > 2 ? rhs.diff(0, yd) : even_zero ? d2 : rhs.diff2(0);
        row(y, wy.x * dq - wy.y * dup, ad[y], wy);
        dup = dq;
    }
    double z = x0 - o;
    if (even_zero) {
        z = 0.0;
        ad01 = 1.0;
    }
    const bool ok = isfinite(ad01) && ad01 != 0.0;
    z /= ad01;
    f[p * (2 * TC)] = z;
    yd = (double)p;
    acc(yd, z);
    y = p + 2;
    for (; y + 2 * (kRows - 1) <= ny; y += 2 * kRows) {
        double gv[kRows], n[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            gv[i] = f[(y + 2 * i) * (2 * TC)];
            n[i] = W[y + 2 * i].x * (w * ad[y + 2 * i]);
        }
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            z = gv[i] - n[i] * z;
            f[(y + 2 * i) * (2 * TC)] = z;
            yd += 2.0;
            acc(yd, z);
        }
    }
    for (; y <= ny; y += 2) {
        z = f[y * (2 * TC)] - (W[y].x * (w * ad[y])) * z;
        f[y * (2 * TC)] = z;
        yd += 2.0;
        acc(yd, z);
    }
    return ok;
}

// Right-hand side of the pressure: the divergence of R, q + dR_1/dy with q =
// i kx R_0 + i kz R_2 (src/solver/eqsolve_pv.cpp:340-357).  own / other: this
// thread's part of the column and the other one (i k swaps re and im; sx, sz
// carry the sign).
struct DivergenceRhs {
    const double *r0_other, *r1_own, *r2_other;
    double sx, sz;
    int ny;
    double q = 0.0, a0[kRows], a1[kRows], a2[kRows];
    __device__ __forceinline__ double start(int top) {
        q = sx * r0_other[top * (2 * TC)] + sz * r2_other[top * (2 * TC)];
        return top < ny ? q + (2.0 * ny) * r1_own[ny * (2 * TC)] : q;
    }
    __device__ __forceinline__ void load(int i, int y) {
        a0[i] = r0_other[(y - 2) * (2 * TC)];
        a2[i] = r2_other[(y - 2) * (2 * TC)];
        a1[i] = r1_own[(y - 1) * (2 * TC)];
    }
    __device__ __forceinline__ double diff(int i, double yd) {
        const double qn = sx * a0[i] + sz * a2[i], d = (qn - q) + (2.0 * yd - 2.0) * a1[i];
        q = qn;
        return d;
    }
    __device__ __forceinline__ double diff2(int i) { return (sx * a0[i] + sz * a2[i] - 0.5 * q) + a1[i]; }
};

// Right-hand side of velocity component C: Re (grad P - R_C)
// (src/solver/eqsolve_pv.cpp:359-395); pp: P's own part for C = 1, else the other one.
template <int C> struct VelocityRhs {
    const double *pp, *r_own;
    double s_i, re;
    int ny;
    double q = 0.0, a[kRows], r[kRows];   // q: C = 1: -Re R_1, else the whole r_y
    __device__ __forceinline__ double start(int top) {
        if (C == 1) {
            q = -re * r_own[top * (2 * TC)];
            return top < ny ? q + re * ((2.0 * ny) * pp[ny * (2 * TC)]) : q;
        }
        q = re * (s_i * pp[top * (2 * TC)] - r_own[top * (2 * TC)]);
        return q;
    }
    __device__ __forceinline__ void load(int i, int y) {
        r[i] = r_own[(y - 2) * (2 * TC)];
        a[i] = pp[(C == 1 ? y - 1 : y - 2) * (2 * TC)];
    }
    __device__ __forceinline__ double diff(int i, double yd) {
        double d;
        if (C == 1) {
            const double qn = -re * r[i];
            d = (qn - q) + (re * (2.0 * yd - 2.0)) * a[i];
            q = qn;
        } else {
            const double qn = re * (s_i * a[i] - r[i]);
            d = qn - q;
            q = qn;
        }
        return d;
    }
    __device__ __forceinline__ double diff2(int i) {
        if (C == 1) return (-re * r[i] - 0.5 * q) + re * a[i];
        return re * (s_i * a[i] - r[i]) - 0.5 * q;
    }
};

// The real parts of u and w of the (kz, kx) = (0, 0) column before their pressure
// gradient, by warp scans and from the multistep state: the column that gives dp/dx and
// dp/dz where the flow rate is fixed, and the mean wall shear.  dp/dx = (Q - q) / q_unit,
// with Q - q some 4e-6 of Q, shows each last bit of it as 5e-11, and the shear weights
// coefficient k by k^2, so that the order of its operations is part of the result: by
// the chains, dp/dx of a 32 x 49 x 32 channel is 5e-11 to 1e-10 off after six steps, the
// mean shear of a 50 x 27 x 40 one 7e-12 after twelve.  No pressure enters (kx = kz = 0),
// nor do the corrections.  Warp 3 of one block does it beside the pressure chains.  That
// block is the first to start: with it among the last, its 4 to 7 us more were the
// kernel's (144 us instead of 138 at 128 x 129 x 128, 547 instead of 528 at 256 x 193 x
// 192).  (u, w) are one double2 column where their wall conditions are the same (c = 0,
// both), else one after the other.
template <int E>
__device__ __forceinline__ void flux_column(const Dims &d, const Tables &t, const PhysParams &pp, double g,
                                         const SolverState &st, const StepArgs &s, double2 *v_out, int c, bool both) {
    const int ny = d.NYS, zc = d.zc;
    const long long base = spectral_base(d, d.NZS, zc - d.NZS * d.nkx), cu = c * d.Ns, cw = both ? 2 * d.Ns : cu;
    const double *adv = st.ad_v + (long long)zc * d.ncy;
    double2 f[E], z[E];
    double ad[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        f[e] = mk(0.0, 0.0);
        ad[e] = 0.0;
        if (y > ny) continue;
        const long long o = base + (long long)y * d.sy;
        auto pair = [&](const double2 *q) { return mk(q[cu + o].x, q[cw + o].x); };
        const double2 r = cadd(cadd(cadd(cscale(s.a0, pair(s.u)), cscale(s.a1, pair(s.u_prev))),
                                    cscale(s.b0, pair(s.N))),
                               cscale(s.b1, pair(s.N_prev)));
        f[e] = cscale(pp.Re, mk(-r.x, -r.y));
        ad[e] = adv[y];
    }
    auto wall = [&](int side) {
        return mk(s.bc_v[(2 * c + side) * d.ncol + zc].x, s.bc_v[(2 * (both ? 2 : c) + side) * d.ncol + zc].x);
    };
    tau_warp<E>(ny, g, pp.a_V[c], pp.b_V[c], true, wall(0), wall(1), st.wn_v[zc], f, z, ad, t.WL, t.WD, t.WR);
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int y = ycoef<E>(e);
        if (y > ny) continue;
        const long long o = base + (long long)y * d.sy;   // (v_out may be u_prev: read above)
        v_out[cu + o].x = z[e].x;
        if (both) v_out[cw + o].x = z[e].y;
    }
}
template <int E>
__global__ void __launch_bounds__(kThreads, 3)
k_solve(const __grid_constant__ Dims d, const __grid_constant__ Tables t, const __grid_constant__ PhysParams pp,
        double g_v, const __grid_constant__ SolverState st, const __grid_constant__ SolveArgs A) {
    chain_begin();
    extern __shared__ double2 tile[];   // [4][ncy][TC]: R_0, R_1, R_2, P; then (WL, WR) and the pivots
    __shared__ double s_wall[3][2][2 * TC];
    __shared__ double2 s_cs[TC], s_cd[TC], s_sg[2][TC];   // c0 + c1, c0 - c1, sigma
    const int ncy = d.ncy, ny = d.NYS, nkx = d.nkx, ncol = d.ncol;
    const int S = ncy * TC;
    const int AS = pivot_stride(ncy);
    double2 *s_w = tile + 3 * S + max(ncy, kRowGroups) * TC;         // [ncy] (WL, WR)
    double *s_ad = reinterpret_cast<double *>(s_w + ncy);             // [TC][AS]
    // blocks of kz and -kz next to each other: from the middle outwards, so that the block
    // with flux_column's work starts first
    const int bi = (int)gridDim.x - 1 - (int)blockIdx.x;
    const int blk = (bi & 1) ? (int)gridDim.x - 1 - (bi >> 1) : (bi >> 1);
    const int col0 = blk * TC;
    const int tid = threadIdx.x;
    const int w = tid >> 5, lane = tid & 31;
    const StepArgs &s = A.step;

    // this thread's column in the row-wise passes: l = tid mod TC, rows g, g + 16, ...
    const int l = tid & (TC - 1), g = tid / TC;
    const int c2 = col0 + l;
    const bool ok = c2 < ncol;
    const int kzi = ok ? c2 / nkx : 0, kx = ok ? c2 - kzi * nkx : 0;
    const int kzn = kzi <= d.NZS ? kzi : 2 * d.NZS - kzi;   // the kz <= 0 column of this |kz|

    // ---- pivots of the kz <= 0 columns (column-major) and the row weights ---
    auto pivot_base = [&](int q) {
        const int c = min(col0 + q, ncol - 1), kq = c / nkx;
        return (long long)(min(kq, 2 * d.NZS - kq) * nkx + (c - kq * nkx)) * ncy;
    };
    for (int q = w; q < TC; q += kThreads / 32) {
        const double *src = st.ad_p + pivot_base(q);
        for (int y = lane; y < ncy; y += 32) cp_async8(s_ad + q * AS + y, src + y, 8);
    }
    for (int y = tid; y < ncy; y += kThreads) {
        cp_async8(&s_w[y].x, t.WL + y, 8);
        cp_async8(&s_w[y].y, t.WR + y, 8);
    }
    cp_async_commit();

    // lane = 16 p + 2 cl + r: parity p, column cl of the block, part r (re, im)
    const int p = lane >> 4, cl = (lane >> 1) & (TC - 1), r = lane & 1;
    const int own = 2 * cl + r, oth = own ^ 1;
    const int col = col0 + cl;
    const bool live = col < ncol;
    const int ccol = live ? col : ncol - 1;
    const double ax = t.wavx[ccol % nkx], az = t.wavz[ccol / nkx];
    const double sx = r ? ax : -ax, sz = r ? az : -az;
    const bool zero_col = col == d.zc;
    double *T = reinterpret_cast<double *>(tile);
    const double *ad = s_ad + cl * AS;
    bool pivot_fail = false;
    // warps 1-3 hold the velocity pivots in registers while warp 0 solves the pressure
    constexpr int kHoldCols = (TC + 2) / 3, kHoldRows = 8;   // NYS + 1 <= 256
    double hold[kHoldCols][kHoldRows];
    // warp 0's lanes fetch their column's influence data before the chains run:
    // lane p uses sigma_0's entry p, and v of the first response at y = ny - p
    const int coln = min(ccol / nkx, 2 * d.NZS - ccol / nkx) * nkx + ccol % nkx;   // the kz <= 0 column
    double i00 = 0.0, i01 = 0.0, i10 = 0.0, i11 = 0.0, sg = 1.0, pn = 0.0, vn = 0.0, tail = 0.0;
    double wt = 0.0, wb = 0.0, pt = 0.0, pb = 0.0, wp = 0.0;   // wall data of the pressure, its w
    if (w == 0) {
        const long long o_n = spectral_base(d, coln / nkx, coln % nkx) + (long long)ny * d.sy;
        i00 = st.inf_div[coln].x;
        i01 = st.inf_div[ncol + coln].x;
        i10 = st.inf_div[2 * ncol + coln].x;
        i11 = st.inf_div[3 * ncol + coln].x;
        sg = st.sigma0[p * ncol + coln].x;
        pn = st.p_inf[o_n];
        vn = st.v_inf[d.Ns + o_n - p * d.sy];
        wp = st.wn_p[ccol];
        if (s.bc_p) {
            wt = reinterpret_cast<const double *>(s.bc_p + ccol)[r];
            wb = reinterpret_cast<const double *>(s.bc_p + ncol + ccol)[r];
        } else {
            wt = reinterpret_cast<const double *>(s.bw + ccol)[r];
            wb = reinterpret_cast<const double *>(s.bw + ncol + ccol)[r];
            pt = reinterpret_cast<const double *>(s.B_prev + ccol)[r];
            pb = reinterpret_cast<const double *>(s.B_prev + ncol + ccol)[r];
        }
    }
    // ---- stage R = a0 u + a1 u_prev + b0 N + b1 N_prev; sums of N_y --------
    // (the loads of two rows are issued before the first use)
    {
        constexpr int kBatch = 2;
        double2 sy = mk(0.0, 0.0);   // N_y over this thread's rows (all of parity g & 1)
        const long long base = spectral_base(d, kzi, kx);
        for (int y0 = g; ok && y0 < ncy; y0 += kBatch * kRowGroups) {
            double2 u[kBatch][3], up[kBatch][3], nv[kBatch][3], np[kBatch][3];
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                const int y = min(y0 + b * kRowGroups, ny);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const long long o = c * d.Ns + base + (long long)y * d.sy;
                    u[b][c] = ld256(s.u + o);
                    up[b][c] = ld256(s.u_prev + o);
                    nv[b][c] = ld256(s.N + o);
                    np[b][c] = ld256(s.N_prev + o);
                }
            }
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                const int y = y0 + b * kRowGroups;
                if (y >= ncy) break;
#pragma unroll
                for (int c = 0; c < 3; ++c)   // R (src/sim/simulation.cpp:151-158)
                    tile[c * S + y * TC + l] =
                        cadd(cadd(cadd(cscale(s.a0, u[b][c]), cscale(s.a1, up[b][c])), cscale(s.b0, nv[b][c])),
                             cscale(s.b1, np[b][c]));
                sy = cadd(sy, nv[b][1]);
            }
        }
        tile[3 * S + g * TC + l] = sy;   // [16][TC], in P's tile until its first sweep
    }
    cp_async_wait<0>();
    __syncthreads();

    // the (kz, kx) = (0, 0) column (-1: not on this rank); its block
    const int zc = d.zc;
    const bool fix_zero = !s.solve_only && zc >= col0 && zc < col0 + TC;
    // ---- chains ------------------------------------------------------------
    if (w == 3 && fix_zero) {
        const bool both = pp.a_V[0] == pp.a_V[2] && pp.b_V[0] == pp.b_V[2];
#pragma unroll 1
        for (int c = 0; c < (both ? 1 : 3); c += 2) flux_column<E>(d, t, pp, g_v, st, s, A.v_out, c, both);
    }
    if (w == 0) {
        const double *sum = T + 6 * S;
        double lower, upper;
        // sums of N_y over this parity's rows, then over both
        double mine = 0.0;
#pragma unroll
        for (int q = 0; q < kRowGroups / 2; ++q) mine += sum[(2 * q + p) * (2 * TC) + own];
        const double other = __shfl_xor_sync(kFull, mine, 16);
        const double even = p ? other : mine, odd = p ? mine : other;
        if (s.bc_p) {
            lower = wt;
            upper = wb;
        } else {
            // pressure wall data (src/solver/eqsolve_pv.cpp:322-337) and its
            // combination b0 B + b1 B_prev (src/sim/simulation.cpp:146-150)
            const double bt = wt + (even + odd);
            const double bb = wb + (odd - even);
            lower = s.b0 * bt + s.b1 * pt;
            upper = s.b0 * bb + s.b1 * pb;
            if (live) reinterpret_cast<double *>(s.B_new + p * ncol + col)[r] = p ? bb : bt;
        }
        tail = T[(2 * S) + (ny - p) * (2 * TC) + own];   // R_1 at ny, ny - 1
        __syncwarp();   // the sums were read by every lane before P's sweep overwrites them
        DivergenceRhs rhs{T + oth, T + 2 * S + own, T + 4 * S + oth, sx, sz, ny};
        pivot_fail |= !tau_chain(ny, p, A.p_a, A.p_b, pp.G_pre == 0.0 && A.p_a == 0.0 && zero_col, lower, upper,
                                 wp, s_w, t.WD, ad, T + 6 * S + own, rhs, [](double, double) {});
    } else {
#pragma unroll
        for (int i = 0; i < kHoldCols; ++i) {
            const int q = w - 1 + 3 * i;
            const double *src = st.ad_v + pivot_base(min(q, TC - 1));
#pragma unroll
            for (int k = 0; k < kHoldRows; ++k) {
                const int y = lane + 32 * k;
                if (q < TC && y < ncy) hold[i][k] = src[y];
            }
        }
    }
    __syncthreads();
    if (w > 0) {
#pragma unroll
        for (int i = 0; i < kHoldCols; ++i) {
            const int q = w - 1 + 3 * i;
#pragma unroll
            for (int k = 0; k < kHoldRows; ++k) {
                const int y = lane + 32 * k;
                if (q < TC && y < ncy) s_ad[q * AS + y] = hold[i][k];
            }
        }
    }
    __syncthreads();
    const double wv = st.wn_v[ccol];
    if (w < 3) {
        const double lower = reinterpret_cast<const double *>(s.bc_v + (2 * w) * ncol + ccol)[r];
        const double upper = reinterpret_cast<const double *>(s.bc_v + (2 * w + 1) * ncol + ccol)[r];
        const double a = w == 0 ? pp.a_V[0] : w == 1 ? pp.a_V[1] : pp.a_V[2];
        const double b = w == 0 ? pp.b_V[0] : w == 1 ? pp.b_V[1] : pp.b_V[2];
        const bool nrm = g_v == 0.0 && a == 0.0 && zero_col;
        double *f = T + w * 2 * S + own;
        double sum = 0.0;   // wall sums of this chain (src/solver/eqsolve_pv.cpp:397-406)
        if (w == 1) {
            VelocityRhs<1> rhs{T + 6 * S + own, f, 0.0, pp.Re, ny};
            pivot_fail |= !tau_chain(ny, p, a, b, nrm, lower, upper, wv, s_w, t.WD, ad, f, rhs,
                                     [&](double yd, double z) { sum += (yd * yd) * z; });
        } else {
            VelocityRhs<0> rhs{T + 6 * S + oth, f, w == 0 ? sx : sz, pp.Re, ny};
            pivot_fail |= !tau_chain(ny, p, a, b, nrm, lower, upper, wv, s_w, t.WD, ad, f, rhs,
                                     [&](double, double z) { sum += z; });
        }
        s_wall[w][p][own] = sum;
    }
    if (pivot_fail && live) atomicOr(s.err, ERR_PIVOT);
    __syncthreads();

    // ---- influence and sigma coefficients (src/solver/eqsolve_pv.cpp:397-429) ----
    // The influence divergences and sigma_0 are real (real wall data, fields real
    // or imaginary): part r of a column's coefficients needs only scalars.  Lane
    // 16 q + 2 cl + r also divides by sigma_0's entry q.
    if (w == 0 && live) {
        // sums over parity q of i kx u + i kz w (this part) and of y^2 v
        const double te = sx * s_wall[0][0][oth] + sz * s_wall[2][0][oth], ne = s_wall[1][0][own];
        const double to = sx * s_wall[0][1][oth] + sz * s_wall[2][1][oth], no = s_wall[1][1][own];
        const double div0 = (te + ne) + (to + no), div1 = (te - ne) + (no - to);
        const double c0 = div1 * i10 - div0 * i11, c1 = div0 * i01 - div1 * i00;
        const double cs = c0 + c1, cdf = c0 - c1;
        const bool ev = (ny & 1) == 0;   // parity of ny
        const double vt = T[2 * S + (ny - p) * (2 * TC) + own] + vn * (ev == (p == 0) ? cdf : cs);
        double num;
        if (p == 0) {
            num = -wv * vt - pp.Re * tail;
        } else {
            const double ptop = T[6 * S + ny * (2 * TC) + own] + pn * (ev ? cs : cdf);
            num = -wv * vt + pp.Re * (2.0 * ny * ptop - tail);
        }
        reinterpret_cast<double *>(s_sg[p])[own] = num / sg;
        if (p == 0) {
            reinterpret_cast<double *>(s_cs)[own] = cs;
            reinterpret_cast<double *>(s_cd)[own] = cdf;
        }
    }
    __syncthreads();

    // ---- influence and sigma corrections, coalesced over the block --------
    // rows g, g + 16, ... all have the parity of g.  Odd-y coefficients take
    // sigma_0 for p, u, w and sigma_1 for v, even-y the reverse; the second
    // response's sign makes c0 + c1 the even p, u, w and odd v coefficient.
    bool bad = false;
    if (ok) {
        const bool odd = g & 1;
        const double2 cq = odd ? s_cd[l] : s_cs[l], cv = odd ? s_cs[l] : s_cd[l];
        const double2 sq = s_sg[odd ? 0 : 1][l], sv = s_sg[odd ? 1 : 0][l];
        const double axl = t.wavx[kx], azl = t.wavz[kzi];
        const bool same_uw = pp.a_V[0] == pp.a_V[2] && pp.b_V[0] == pp.b_V[2];
        // q = the stored field that gives both u and w: u (w = az/ax u) where kx > 0, w where kx = 0
        const double sgn = kzi > d.NZS ? -1.0 : 1.0;   // w of the kz <= 0 column, negated
        const double fu = axl != 0.0 ? 1.0 : 0.0;
        const double fw = same_uw && axl != 0.0 ? azl / axl : sgn;
        const long long comp = axl != 0.0 ? 0 : 2 * d.Ns;
        const long long in0 = spectral_base(d, kzn, kx), out0 = spectral_base(d, kzi, kx);
        constexpr int kBatch = 4;
        for (int y0 = g; y0 < ncy; y0 += kBatch * kRowGroups) {
            double pi[kBatch], qi[kBatch], vi[kBatch], wi[kBatch], pb[kBatch], qb[kBatch], vb[kBatch], wb[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const long long o = in0 + (long long)min(y0 + k * kRowGroups, ny) * d.sy;
                pi[k] = ld256(st.p_inf + o);
                vi[k] = ld256(st.v_inf + d.Ns + o);
                pb[k] = ld256(st.p_b + o);
                vb[k] = ld256(st.v_b + d.Ns + o);
                qi[k] = ld256(st.v_inf + comp + o);
                qb[k] = ld256(st.v_b + comp + o);
                wi[k] = qi[k];
                wb[k] = qb[k];
                if (!same_uw && comp == 0) {
                    wi[k] = st.v_inf[2 * d.Ns + o];
                    wb[k] = st.v_b[2 * d.Ns + o];
                }
            }
#pragma unroll
            for (int k = 0; k < kBatch; ++k) {
                const int y = y0 + k * kRowGroups;
                if (y >= ncy) break;
                const int sl = y * TC + l;
                const double2 pr = cadd(cadd(tile[3 * S + sl], cscale(pi[k], cq)), cscale(pb[k], sq));
                double2 v[3];
                v[0] = cadd(cadd(tile[sl], fderiv(fu * qi[k], cq)), fderiv(fu * qb[k], sq));
                v[1] = cadd(cadd(tile[S + sl], cscale(vi[k], cv)), cscale(vb[k], sv));
                v[2] = cadd(cadd(tile[2 * S + sl], fderiv(fw * wi[k], cq)), fderiv(fw * wb[k], sq));
                if (fix_zero && c2 == zc) {
                    tile[3 * S + sl] = pr;
#pragma unroll
                    for (int c = 0; c < 3; ++c) tile[c * S + sl] = v[c];
                    continue;
                }
                bad |= !(isfinite(pr.x) && isfinite(pr.y) && isfinite(v[0].x) && isfinite(v[0].y) &&
                         isfinite(v[1].x) && isfinite(v[1].y) && isfinite(v[2].x) && isfinite(v[2].y));
                const long long o = out0 + (long long)y * d.sy;
                A.p_out[o] = pr;
#pragma unroll
                for (int c = 0; c < 3; ++c) A.v_out[c * d.Ns + o] = v[c];
                if (s.om) {
                    s.om[d.Ns + o] = csub(fderiv(azl, v[0]), fderiv(axl, v[2]));
#pragma unroll
                    for (int c = 0; c < 3; ++c) tile[c * S + sl] = v[c];
                }
            }
        }
    }
    if (fix_zero) {
        __syncthreads();
        if (w == 0) {
            const int lz = zc - col0;
            // correct_zero_mode (src/solver/timestepper.cpp:60-68)
            const double2 v1w = cscale(0.5, cadd(s.bc_v[2 * ncol + zc], s.bc_v[3 * ncol + zc]));
            // correct_flow (src/sim/simulation.cpp:111-140), single-rank branch
            const double *uu = st.unit;
            double dpdx, dpdz;
            bool pfail = false;
            if (pp.grad_pre == 1) {
                dpdx = pp.gx;
                dpdz = pp.gz;
            } else {
                double qx = 0.0, qz = 0.0;
                // summed as flux_column holds the column (the order matters there)
                const double2 *f = A.v_out + spectral_base(d, d.NZS, zc - d.NZS * nkx);
                for (int e = 0; e < E && !(lane & 1); ++e) {
                    const int y = 2 * (E * (lane >> 1) + e);
                    if (y > ny) break;
                    qx += f[(long long)y * d.sy].x / (double)(y * y - 1);
                    qz += f[2 * d.Ns + (long long)y * d.sy].x / (double)(y * y - 1);
                }
                qx = -sum_warp(qx);
                qz = -sum_warp(qz);
                const double qxu = uu[2 * ncy], qzu = uu[2 * ncy + 1];
                pfail = !isfinite(qxu) || qxu == 0.0 || !isfinite(qzu) || qzu == 0.0;
                dpdx = (pp.qxm - qx) / qxu;
                dpdz = (pp.qzm - qz) / qzu;
            }
            if (lane == 0) {
                s.dpdx[0] = dpdx;
                s.dpdx[1] = dpdz;
                if (pfail) atomicOr(s.err, ERR_PIVOT);
            }
            for (int y = lane; y <= ny; y += 32) {
                const double2 pz = tile[3 * S + y * TC + lz];
                const long long off = spectral_base(d, d.NZS, zc - d.NZS * nkx) + (long long)y * d.sy;
                double2 u0 = tile[y * TC + lz], u2 = tile[2 * S + y * TC + lz];
                u0.x = A.v_out[off].x;
                u2.x = A.v_out[2 * d.Ns + off].x;
                const double2 u1 = y == 0 ? v1w : mk(0.0, 0.0);
                u0.x += dpdx * uu[y];
                u2.x += dpdz * uu[ncy + y];
                bad |= !(isfinite(pz.x) && isfinite(pz.y) && isfinite(u0.x) && isfinite(u0.y) && isfinite(u1.x) &&
                         isfinite(u1.y) && isfinite(u2.x) && isfinite(u2.y));
                A.p_out[off] = pz;
                A.v_out[off] = u0;
                A.v_out[d.Ns + off] = u1;
                A.v_out[2 * d.Ns + off] = u2;
                if (s.om) {
                    s.om[d.Ns + off] = mk(0.0, 0.0);
                    tile[y * TC + lz] = u0;
                    tile[S + y * TC + lz] = u1;
                    tile[2 * S + y * TC + lz] = u2;
                }
            }
        }
    }
    if (__any_sync(kFull, bad) && lane == 0) atomicOr(s.err, ERR_NONFINITE);
    if (!s.om) return;

    // ---- curl of the new velocity (src/solver/vector_ops.cpp:112-151), for the
    // next step: om_x = dw/dy - i kz v, om_z = i kx v - du/dy (om_y is written
    // above), and its pressure-wall sums.  Warps 0 and 1 differentiate u and w in
    // place, warp 2 sums v: from the tile, this saves a kernel of its own that
    // read the velocity back.
    __syncthreads();
    if (w < 3) {
        double *f = T + (w == 0 ? 0 : w == 1 ? 4 * S : 2 * S) + own;
        double sum = 0.0;
        if (w < 2) {
            // d_y = sum of 2 j f_j over j = y + 1, y + 3, ..., halved at y = 0, left
            // in row y + 1, whose operand its thread has just read (d_NYS = 0)
            double acc = 0.0;
            int q = ((ny & 1) == p) ? ny - 1 : ny;   // rows of the other parity, descending
            double qd = 2.0 * (double)q;
            for (; q - 2 * (kRows - 1) >= 2; q -= 2 * kRows) {
                double v[kRows];
#pragma unroll
                for (int i = 0; i < kRows; ++i) v[i] = (qd - (double)(4 * i)) * f[(q - 2 * i) * (2 * TC)];
                qd -= (double)(4 * kRows);
#pragma unroll
                for (int i = 0; i < kRows; ++i) {
                    acc += v[i];
                    f[(q - 2 * i) * (2 * TC)] = acc;
                    sum += acc;
                }
            }
            for (; q >= 1; q -= 2, qd -= 4.0) {
                acc += qd * f[q * (2 * TC)];
                const double dv = q == 1 ? 0.5 * acc : acc;
                f[q * (2 * TC)] = dv;
                sum += dv;
            }
        } else {
            for (int y = p; y <= ny; y += 2) sum += f[y * (2 * TC)];
        }
        s_wall[w][p][own] = sum;
    }
    __syncthreads();
    if (ok) {
        const double axl = t.wavx[kx], azl = t.wavz[kzi];
        const long long out0 = spectral_base(d, kzi, kx);
#pragma unroll 4
        for (int y = g; y < ncy; y += kRowGroups) {
            const int sl = y * TC + l;
            const long long o = out0 + (long long)y * d.sy;
            const double2 v = tile[S + sl];
            const double2 du = y < ny ? tile[sl + TC] : mk(0.0, 0.0);
            const double2 dw = y < ny ? tile[2 * S + sl + TC] : mk(0.0, 0.0);
            s.om[o] = csub(dw, fderiv(azl, v));
            s.om[2 * d.Ns + o] = csub(fderiv(axl, v), du);
        }
        if (tid < TC) {
            // sums over y of i kx/Re om_z - i kz/Re om_x, signs (+1, (-1)^(y+1))
            // (src/solver/timestepper.cpp:26-43)
            double2 part[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const double2 du = mk(s_wall[0][q][2 * l], s_wall[0][q][2 * l + 1]);
                const double2 dw = mk(s_wall[1][q][2 * l], s_wall[1][q][2 * l + 1]);
                const double2 sv = mk(s_wall[2][q][2 * l], s_wall[2][q][2 * l + 1]);
                part[q] = csub(fderiv(axl / pp.Re, csub(fderiv(axl, sv), du)),
                               fderiv(azl / pp.Re, csub(dw, fderiv(azl, sv))));
            }
            s.bw_out[c2] = cadd(part[0], part[1]);
            s.bw_out[ncol + c2] = csub(part[1], part[0]);
        }
    }
}

// the four tiles (P's holds the [16][TC] sums of N_y first, also where NYS + 1 < 16),
// the row weights and the pivots
size_t solve_smem(const Dims &d) {
    const size_t tiles = 3 * (size_t)d.ncy * TC + (size_t)(d.ncy > kRowGroups ? d.ncy : kRowGroups) * TC;
    return sizeof(double2) * (tiles + d.ncy) + sizeof(double) * TC * (size_t)pivot_stride(d.ncy);
}

__global__ void k_pressure_bc(Dims d, const double2 *N, const double2 *bw, double2 *B) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const int kzi = col / d.nkx, kx = col - (col / d.nkx) * d.nkx;
    const double2 *Ny = N + d.Ns + spectral_base(d, kzi, kx);
    double2 st_ = mk(0, 0), sb_ = mk(0, 0);
    for (int y = 0; y <= d.NYS; ++y) {
        const double2 n1 = Ny[(long long)y * d.sy];
        st_ = cadd(st_, n1);
        sb_ = (y & 1) ? cadd(sb_, n1) : csub(sb_, n1);
    }
    B[col] = cadd(bw[col], st_);
    B[d.ncol + col] = cadd(bw[d.ncol + col], sb_);
}

}  // namespace

void launch_pressure_bc(const Dims &d, const double2 *N, const double2 *bw, double2 *B,
                        cudaStream_t s) {
    k_pressure_bc<<<(d.ncol + 127) / 128, 128, 0, s>>>(d, N, bw, B);
}

cudaError_t configure_solver_kernels(const Dims &d) {
    cudaError_t e = configure_setup_kernels(d);
    if (e != cudaSuccess) return e;
    e = configure_scan_solve(d);   // (refuses more than 256 Chebyshev coefficients)
    if (e != cudaSuccess) return e;
    with_elems(d, [&](auto n) { e = raise_smem(k_solve<decltype(n)::value>, solve_smem(d)); });
    return e;
}

void launch_step_solve(const Dims &d, const Tables &t, const PhysParams &pp, double g_v,
                       const SolverState &st, const StepArgs &a, cudaStream_t s) {
    if (a.scan) return launch_scan_solve(d, t, pp, g_v, st, a, s);
    SolveArgs A{};
    A.p_a = pp.a_pre0;
    A.p_b = pp.b_pre0;
    A.p_out = a.p_out;
    A.v_out = a.u_out;
    A.step = a;
    const int blocks = (d.ncol + TC - 1) / TC;
    with_elems(d, [&](auto n) {
        launch_chained(k_solve<decltype(n)::value>, blocks, kThreads, solve_smem(d), s, d, t, pp, g_v, st, A);
    });
}

}  // namespace cdns
