// Precomputation of the column solver (EqSolvePV::setup,
// src/solver/eqsolve_pv.cpp:148-168, 266-303, 452-493) for sm_100a.
//
// The setup problems run in the reference's sequential operation order, a
// thread per chain (column, y parity, velocity component) over shared-memory columns.  Their
// results enter the step through differences that cancel: the second sigma
// denominator Re + w v_b(n-1) - 2 n Re p_b(n) of the lowest wavenumbers is
// about 1e-6 of its terms, so round-off of the B-problem differs from the
// reference's by 1e-9 relative after that cancellation unless the B-problem is
// computed in the same order.  Setup runs at steps 1 and 2 only.
//
// Outputs: the pivots ad_p, ad_v are stored column-major ([col][y]), read by
// the step solve's chains; the influence / B-problem fields are in the tiled
// layout, read by its coalesced correction pass.
#include "cdns_kernels.cuh"

namespace cdns {

namespace {
constexpr int TC = 4;          // spectral columns per block
constexpr int kThreads = 64;
static_assert(3 * TC * 2 <= 32, "the velocity chains of a block in one warp");

enum SetupMode { MODE_BASE = 1, MODE_COUPLED = 2 };

struct SetupArgs {
    double bcp_top, bcp_bot;   // constant pressure wall data
    double *p_out;             // [Ns], real
    double *v_out;             // [3][Ns], parts as inf_imag(c)
    double2 *divb_out;         // [2][ncol] raw wall divergence (MODE_BASE)
};

__device__ inline double tau_func(double a, double b, int y) {
    const int q = y & 1;
    if (a == 0.0 && b == 0.0) return (double)((1 - q) * y * y + q);
    return a + b * y * y;
}

// The setup fields are real or purely imaginary (real wall data, real operators;
// i kx and i kz enter only through the pressure gradient), so every chain runs on
// the one nonzero part: the products with the exact zeros of the other part drop
// out and leave the same bits.

// Chebyshev derivative coefficients of parity `par` (src/solver/vector_ops.cpp:17-25):
// d_k = d_{k+2} + 2(k+1) f_{k+1}, d_NYS = 0, d_0 halved.
__device__ void deriv_chain(int par, int ny, const double *f, double *dout, int st) {
    int k = ((ny & 1) == par) ? ny : ny - 1;
    double dd = 0.0;
    if (k == ny) {
        dout[(long long)ny * st] = dd;
        k -= 2;
    }
    for (; k >= 0; k -= 2) {
        dd = dd + (double)(2 * (k + 1)) * f[(long long)(k + 1) * st];
        if (k == 0) dd = 0.5 * dd;
        dout[(long long)k * st] = dd;
    }
}

// One parity of the column tau solve of (D^2 - k^2 - g) f = r with
// a f + b f' = (lower, upper) at y = (+1, -1)  (src/solver/eqsolve_pv.cpp:64-128),
// with r_y = scale * rhs[y] (rhs null: zero).  The right-hand side combination,
// the backward sweep and the pivot sum share one descending loop; every operation
// and its order are the reference's.  Returns false if a pivot is zero or not finite.
__device__ __forceinline__ bool tau_chain(int par, int ny, double g, double a, double b, bool zero_col, double lower,
                          double upper, double w, double scale, double mult, const double *rhs, double *out,
                          const double *ad, int st, const double *WL, const double *WD, const double *WR) {
    const bool normalize = g == 0.0 && a == 0.0 && zero_col;
    auto r = [&](int y) { return rhs ? scale * (mult * rhs[(long long)y * st]) : 0.0; };
    double r0 = r(0);
    if (normalize && par == 0) {
        double corr = 0.0;
        for (int y = 2; y <= ny; y += 2) corr = corr + r(y) / (double)(y * y - 1);
        if (b != 0.0) corr = corr + (lower + upper) / (2.0 * b);
        r0 = corr;
    }
#define OUT(yy) out[(long long)(yy) * st]
#define AD(yy) ad[(long long)(yy) * st]
    const int top = ((ny & 1) == par) ? ny : ny - 1;
    double o0 = par == 0 ? (lower + upper) / 2.0 : (lower - upper) / 2.0;
    double ad01 = tau_func(a, b, top);
    double rr2 = 0.0, rr = r(top), xup = 0.0;
    for (int y = top; y >= 2; y -= 2) {
        const double rm = y == 2 ? r0 : r(y - 2);
        double x;
        if (y >= ny - 1) x = WL[y] * rm + WD[y] * rr;
        else x = (WL[y] * rm + WD[y] * rr) + WR[y] * rr2;
        if (y <= ny - 2) x = x - ((WR[y] * w) * AD(y + 2)) * xup;
        const double ady = AD(y);
        OUT(y) = x;
        o0 = o0 - (ad01 * ady) * x;
        ad01 = tau_func(a, b, y - 2) - ((WL[y] * w) * ad01) * ady;
        rr2 = rr;
        rr = rm;
        xup = x;
    }
    if (normalize && par == 0) {
        o0 = 0.0;
        ad01 = 1.0;
    }
    const bool ok = isfinite(ad01) && ad01 != 0.0;
    double z = o0 / ad01;
    OUT(par) = z;
    for (int y = 2 + par; y <= ny; y += 2) {
        z = AD(y) * (OUT(y) - (WL[y] * w) * z);
        OUT(y) = z;
    }
#undef OUT
#undef AD
    return ok;
}

// Unit pressure-gradient responses of the zero mode (src/solver/eqsolve_pv.cpp:479-493):
// lanes (component, parity) of one warp, one column.  work: 4 ncy + 2 ncy doubles.
__device__ void unit_responses(const Dims &d, const Tables &t, const PhysParams &pp, double g_v,
                               const double *ad_v, double *unit, double *work) {
    const int ncy = d.ncy, ny = d.NYS;
    double *WL = work, *WD = WL + ncy, *WR = WD + ncy, *ad = WR + ncy, *rhs = ad + ncy, *o = rhs + ncy;   // o [2][ncy]
    const long long zc = (long long)d.zc * ncy;
    for (int y = threadIdx.x; y < ncy; y += blockDim.x) {
        rhs[y] = y == 0 ? pp.Re : 0.0;
        ad[y] = ad_v[zc + y];
        WL[y] = t.WL[y];
        WD[y] = t.WD[y];
        WR[y] = t.WR[y];
    }
    __syncthreads();
    const double w = -((0.0 + 0.0) + g_v);
    if (threadIdx.x < 4) {
        const int pass = threadIdx.x >> 1, par = threadIdx.x & 1, c = pass == 0 ? 0 : 2;
        double *op = o + pass * ncy;
        tau_chain(par, ny, g_v, pp.a_V[c], pp.b_V[c], true, 0.0, 0.0, w, 1.0, 1.0, rhs, op, ad, 1, WL, WD, WR);
        __syncwarp(0xfu);
        if (par == 0) {
            double q = 0.0;
            for (int y = 0; y <= ny; y += 2) q -= op[y] / (double)(y * y - 1);
            unit[2 * ncy + pass] = q;
        }
    }
    __syncthreads();
    for (int y = threadIdx.x; y < 2 * ncy; y += blockDim.x) unit[y] = o[y];
}

// Setup column solve: pressure tau with constant wall data (MODE_BASE) or the
// B-problem right-hand side (MODE_COUPLED), velocity taus of Re grad P, wall
// divergence, and for MODE_COUPLED the influence correction
// (src/solver/eqsolve_pv.cpp:241-264, 311-450 without sigma).
//
// Only the columns kz <= 0 are solved.  Column -kz has the same k^2, so the
// same pivots and pressure; its right-hand sides differ only by the sign of
// the kz derivative, and every operation is linear with the rounding of a
// negated operand negated, so its solution is this column's with w negated,
// bit for bit, and its wall divergences are equal.  Both columns are written.
//
// A column's chains are sequential, so what counts is how many run at once: the
// two parities of the pressure, then those of all three velocity components
// (lanes 3 x TC x 2 of one warp, the same instructions with the component's
// source and multiplier selected).  MODE_COUPLED's last block solves the unit
// responses of the zero mode, which need nothing of the others.
template <int MODE>
__global__ void __launch_bounds__(kThreads)
k_setup_solve(Dims d, Tables t, PhysParams pp, double g_v, SolverState st, SetupArgs A) {
    extern __shared__ double sm[];
    const int ncy = d.ncy, ny = d.NYS, nkx = d.nkx;
    const int nhalf = (d.NZS + 1) * nkx;   // columns kz <= 0 (kz index 0 .. NZS)
    if (MODE == MODE_COUPLED && (int)blockIdx.x * TC >= nhalf) {
        unit_responses(d, t, pp, g_v, st.ad_v, st.unit, sm);
        return;
    }
    if (MODE == MODE_BASE && blockIdx.y == 1) {
        // the second influence response: pressure data (0, 1), its own outputs
        A.bcp_top = 0.0;
        A.bcp_bot = 1.0;
        A.p_out += d.Ns;
        A.v_out += 3 * d.Ns;
        A.divb_out += 2 * d.ncol;
    }
    const int S = ncy * TC;
    double *rv = sm;              // [3][ncy][TC] velocity: u, w imaginary, v real parts
    double *pc = rv + 3 * S;      // [ncy][TC] pressure
    double *dyb = pc + S;         // pressure right-hand side, then dP/dy
    double *adp = dyb + S;
    double *adv = adp + S;
    double *sWL = adv + S;
    double *sWD = sWL + ncy;
    double *sWR = sWD + ncy;
    __shared__ double s_c0[TC], s_c1[TC];

    const int col0 = blockIdx.x * TC;
    const int tid = threadIdx.x;
    for (int i = tid; i < ncy; i += blockDim.x) {
        sWL[i] = t.WL[i];
        sWD[i] = t.WD[i];
        sWR[i] = t.WR[i];
    }
    for (int i = tid; i < S; i += blockDim.x) {
        const int l = i / ncy, y = i - (i / ncy) * ncy;   // column-major, as the pivots are stored
        const int col = col0 + l, k = y * TC + l;
        double rp = 0.0;
        if (col < nhalf) {
            const long long cm = (long long)col * ncy + y;
            adp[k] = st.ad_p[cm];
            adv[k] = st.ad_v[cm];
            if (MODE == MODE_COUPLED) {
                // B-problem pressure RHS (src/solver/eqsolve_pv.cpp:452-461)
                if (y == 0) rp = (double)(ny - 1);
                else if (y < ny) rp = (double)(2 * (ny - ((y + 1) % 2)));
            }
        } else {
            adp[k] = 1.0;
            adv[k] = 1.0;
        }
        dyb[k] = rp;
    }
    __syncthreads();

    if (tid < 32) {
        // lane = 8 c + 2 l + par (c < 3): component c, column l, parity par
        const int c = tid >> 3, l = (tid >> 1) & (TC - 1), par = tid & 1;
        const int col = col0 + l;
        const bool active = c < 3 && col < nhalf;
        const int kzi = active ? col / nkx : 0;
        const int kx = active ? col - kzi * nkx : 0;
        const double ax = t.wavx[kx], az = t.wavz[kzi];
        const bool zero_col = active && col == d.zc;
        if (active && c == 0)
            tau_chain(par, ny, pp.G_pre, 1.0, 0.0, zero_col, A.bcp_top, A.bcp_bot, st.wn_p[col], 1.0, 1.0,
                      MODE == MODE_COUPLED ? dyb + l : nullptr, pc + l, adp + l, TC, sWL, sWD, sWR);
        __syncwarp();
        if (active && c == 0) deriv_chain(par, ny, pc + l, dyb + l, TC);
        __syncwarp();
        if (active) {
            // Re grad P: i kx P, dP/dy, i kz P
            const double mult = c == 0 ? ax : c == 1 ? 1.0 : az;
            tau_chain(par, ny, g_v, pp.a_V[c], pp.b_V[c], zero_col, 0.0, 0.0, st.wn_v[col], pp.Re, mult,
                      (c == 1 ? dyb : pc) + l, rv + c * S + l, adv + l, TC, sWL, sWD, sWR);
        }
        __syncwarp();
        if (active && par == 0 && c == 0) {
            // wall divergence by endpoint sums (src/solver/eqsolve_pv.cpp:397-406)
            double div0 = 0.0, div1 = 0.0;
            for (int y = 0; y <= ny; ++y) {
                const int k = y * TC + l;
                const double tang = -ax * rv[k] + -az * rv[2 * S + k];
                const double nrm = (double)(y * y) * rv[S + k];
                div0 = div0 + (tang + nrm);
                div1 = (y & 1) ? div1 + (-tang + nrm) : div1 + (tang - nrm);
            }
            if (MODE == MODE_BASE) {
                const int mir = (2 * d.NZS - kzi) * nkx + kx;   // column -kz
                A.divb_out[col] = mk(div0, 0.0);
                A.divb_out[d.ncol + col] = mk(div1, 0.0);
                A.divb_out[mir] = mk(div0, 0.0);
                A.divb_out[d.ncol + mir] = mk(div1, 0.0);
            } else {
                const double i00 = st.inf_div[col].x, i01 = st.inf_div[d.ncol + col].x;
                const double i10 = st.inf_div[2 * d.ncol + col].x, i11 = st.inf_div[3 * d.ncol + col].x;
                s_c0[l] = div1 * i10 - div0 * i11;
                s_c1[l] = div0 * i01 - div1 * i00;
            }
        }
    }
    __syncthreads();

    for (int i = tid; i < S; i += blockDim.x) {
        const int y = i / TC, l = i - (i / TC) * TC;
        const int col = col0 + l;
        if (col >= nhalf) continue;
        const int kzi = col / nkx, kx = col - (col / nkx) * nkx;
        const long long cm = spectral_base(d, kzi, kx) + (long long)y * d.sy;
        double p = pc[i];
        double v[3] = {rv[i], rv[S + i], rv[2 * S + i]};
        if (MODE == MODE_COUPLED) {
            const double c0 = s_c0[l], c1 = s_c1[l];
            p = p + (c0 * st.p_inf[cm] + c1 * st.p_inf[d.Ns + cm]);
            for (int c = 0; c < 3; ++c) v[c] = v[c] + (c0 * st.v_inf[c * d.Ns + cm] + c1 * st.v_inf[(3 + c) * d.Ns + cm]);
        }
        A.p_out[cm] = p;
        for (int c = 0; c < 3; ++c) A.v_out[c * d.Ns + cm] = v[c];
        const int kzm = 2 * d.NZS - kzi;
        if (kzm != kzi) {
            const long long mm = spectral_base(d, kzm, kx) + (long long)y * d.sy;
            A.p_out[mm] = p;
            A.v_out[mm] = v[0];
            A.v_out[d.Ns + mm] = v[1];
            A.v_out[2 * d.Ns + mm] = -v[2];
        }
    }
}

size_t setup_smem(const Dims &d) {
    // the columns' arrays and row weights, or the unit responses' seven rows
    return sizeof(double) * (7 * (size_t)d.ncy * TC + 3 * (size_t)d.ncy);
}

// EqSolvePV::build_wn_ad (src/solver/eqsolve_pv.cpp:148-168), one thread per column
// kz <= 0 and parity of y (the recurrence steps by 2), column -kz the same;
// blockIdx.y = 0: the pressure operator (g = G_pre), 1: the velocity operator (g_v).
__global__ void k_wn_ad(Dims d, Tables t, double g_p, double g_v, double *wn_p, double *ad_p, double *wn_v,
                        double *ad_v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = i >> 1, par = i & 1;
    if (col >= (d.NZS + 1) * d.nkx) return;
    const bool vel = blockIdx.y == 1;
    const double g = vel ? g_v : g_p;
    double *wn = vel ? wn_v : wn_p, *ad = vel ? ad_v : ad_p;
    const int kzi = col / d.nkx, kx = col - (col / d.nkx) * d.nkx;
    const int mir = (2 * d.NZS - kzi) * d.nkx + kx;
    const double ax = t.wavx[kx], az = t.wavz[kzi];
    const double w = -((ax * ax + az * az) + g);
    if (par == 0) {
        wn[col] = w;
        wn[mir] = w;
    }
    const int n = d.NYS;
    double *A = ad + (long long)col * d.ncy, *M = ad + (long long)mir * d.ncy;
    const int top = ((n & 1) == par) ? n : n - 1;
    double up = 1.0 / (1.0 + t.WD[top] * w);
    A[top] = M[top] = up;
    for (int y = top - 2; y >= 2; y -= 2) {
        const double fc = t.WR[y] * t.WL[y + 2];
        const double den = 1.0 + (t.WD[y] - (fc * w) * up) * w;
        up = 1.0 / den;
        A[y] = M[y] = up;
    }
    A[par] = M[par] = 0.0;
}

// Influence normalisation (src/solver/eqsolve_pv.cpp:282-302).
__global__ void k_inf_normalize(Dims d, double a_v1, double2 *inf_div) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    double2 *I = inf_div;
    const int nc = d.ncol;
    const double2 i00 = I[col], i01 = I[nc + col], i10 = I[2 * nc + col], i11 = I[3 * nc + col];
    double2 den = csub(cmul(i00, i11), cmul(i01, i10));
    const bool root = (col == d.zc);
    if (root) den = (a_v1 == 0.0) ? mk(1.0, 0.0) : cdiv(mk(0.25, 0.0), i00);
    if (root) {
        I[col] = den;
        I[nc + col] = mk(0, 0);
        I[2 * nc + col] = den;
        I[3 * nc + col] = mk(0, 0);
    } else {
        I[col] = cdiv(i00, den);
        I[nc + col] = cdiv(i01, den);
        I[2 * nc + col] = cdiv(i10, den);
        I[3 * nc + col] = cdiv(i11, den);
    }
}

// sigma0 denominators (src/solver/eqsolve_pv.cpp:466-476).
__global__ void k_sigma0(Dims d, double re, const double *wn_v, const double *p_b,
                         const double *v_b, double2 *sigma0) {
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= d.ncol) return;
    const int kzi = col / d.nkx, kx = col - (col / d.nkx) * d.nkx;
    const int n = d.NYS;
    const long long on = spectral_base(d, kzi, kx) + (long long)n * d.sy;
    const double w = wn_v[col];
    const double2 vbn = inf_value(v_b[d.Ns + on], false);
    const double2 vbn1 = inf_value(v_b[d.Ns + on - d.sy], false);
    const double2 pbn = inf_value(p_b[on], false);
    sigma0[col] = mk(re + w * vbn.x, w * vbn.y);
    double2 s1 = csub(mk(re + w * vbn1.x, w * vbn1.y), cscale(re * (2.0 * n), pbn));
    if (col == d.zc) s1 = mk(1.0, 0.0);
    sigma0[d.ncol + col] = s1;
}

}  // namespace

cudaError_t configure_setup_kernels(const Dims &d) {
    const int sm = (int)setup_smem(d);
    cudaError_t e = raise_smem(k_setup_solve<MODE_BASE>, sm);
    if (e != cudaSuccess) return e;
    return raise_smem(k_setup_solve<MODE_COUPLED>, sm);
}

void setup_solver(const Dims &d, const Tables &t, const PhysParams &pp, double g_v, SolverState &st,
                  double2 *, cudaStream_t s) {
    const int nb = (d.ncol + 127) / 128;
    k_wn_ad<<<dim3(((d.NZS + 1) * d.nkx * 2 + 127) / 128, 2), 128, 0, s>>>(d, t, pp.G_pre, g_v, st.wn_p, st.ad_p, st.wn_v,
                                                                           st.ad_v);
    const int blocks = ((d.NZS + 1) * d.nkx + TC - 1) / TC;   // columns kz <= 0
    const size_t sm = setup_smem(d);
    // influence responses: pressure Dirichlet data (1,0) and (0,1), in one launch
    // (blockIdx.y = the response)
    {
        SetupArgs A{};
        A.bcp_top = 1.0;
        A.bcp_bot = 0.0;
        A.p_out = st.p_inf;
        A.v_out = st.v_inf;
        A.divb_out = st.inf_div;
        k_setup_solve<MODE_BASE><<<dim3(blocks, 2), kThreads, sm, s>>>(d, t, pp, g_v, st, A);
    }
    k_inf_normalize<<<nb, 128, 0, s>>>(d, pp.a_V[1], st.inf_div);
    {
        SetupArgs A{};
        A.p_out = st.p_b;
        A.v_out = st.v_b;
        // one block more where the zero mode is held: its unit responses (correct_flow)
        k_setup_solve<MODE_COUPLED><<<blocks + (d.zc >= 0), kThreads, sm, s>>>(d, t, pp, g_v, st, A);
    }
    k_sigma0<<<nb, 128, 0, s>>>(d, pp.Re, st.wn_v, st.p_b, st.v_b, st.sigma0);
}

}  // namespace cdns
