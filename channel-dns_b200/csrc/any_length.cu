// Register-form transforms of the product lengths without a compiled split of
// their own (z and x stages and Chebyshev DCT, FP64): n = N1 x N2 with both factors
// among the in-register DFT lengths (reg_fft.cuh), chosen on the host and
// switched over inside the kernels, so that one kernel serves every such length.
//
// They replace the Stockham passes of fft_lines.cuh there: those make a trip
// through shared memory with integer divisions per radix (5 passes at 288 and
// 384), these one exchange per transform with the radix code straight-line.
// The lengths that the switch does not cover (a prime factor above 7, or no
// split into two factors of at most 25) keep the Stockham form.  A step of 60 x 51 x
// 66 takes 67 us instead of 150, one of 256 x 193 x 192 2.9 ms instead of 7.1 (x
// stage of 384 points 1.12 instead of 2.94, z of 288 0.53 instead of 1.24, y of 288
// 0.75 instead of 1.56 as matrix products).  Bound by latency at the warps that the
// registers leave, and by the shared-memory pipe.  FP32 stages take none of these
// (their x and z lengths all have compiled splits; why not y: solver_scan.cu).
//
// Three instances of each kernel, by the largest factor (16, 20 or 25): a DFT of
// 20 needs some 20 registers more than one of 16, one of 24 another 30, and the
// registers are those of the largest radix in the instance.
#include <algorithm>

#include "cdns_kernels.cuh"
#include "fast_div.cuh"
#include "reg_fft.cuh"
#include "transform_ops.cuh"

namespace cdns {

namespace {

template <int V> struct Radix { static constexpr int value = V; };

// fn(Radix<r>) for the in-register length r; MAXR bounds the instances.
template <int MAXR, class Fn> __device__ __forceinline__ void with_radix(int r, const Fn &fn) {
    switch (r) {
    case 3: fn(Radix<3>{}); return;
    case 4: fn(Radix<4>{}); return;
    case 5: fn(Radix<5>{}); return;
    case 6: fn(Radix<6>{}); return;
    case 7: fn(Radix<7>{}); return;
    case 8: fn(Radix<8>{}); return;
    case 9: fn(Radix<9>{}); return;
    case 10: fn(Radix<10>{}); return;
    case 12: fn(Radix<12>{}); return;
    case 14: fn(Radix<14>{}); return;
    case 15: fn(Radix<15>{}); return;
    case 16: fn(Radix<16>{}); return;
    default: break;
    }
    if constexpr (MAXR > 16) {
        switch (r) {
        case 18: fn(Radix<18>{}); return;
        case 20: fn(Radix<20>{}); return;
        default: break;
        }
    }
    if constexpr (MAXR > 20) {
        switch (r) {
        case 21: fn(Radix<21>{}); return;
        case 24: fn(Radix<24>{}); return;
        case 25: fn(Radix<25>{}); return;
        default: break;
        }
    }
}
constexpr int kRadices[] = {3, 4, 5, 6, 7, 8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25};

// fft2_lines (transforms.cu) with run-time factors: TL lines, one exchange
// through S[k1][n2][l] (row stride fft2_kstride), at least max(N1, N2) TL threads.
template <int MAXR, int SIGN, class Src, class Dst>
__device__ __forceinline__ void fft2_any(int N1, int N2, int TL, const Twiddles<double2> &tw, double2 *S,
                                         const Src &src, const Dst &dst) {
    const int KS = fft2_kstride(N2, TL);
    const int t = threadIdx.x;
    const int q = t / TL, l = t - q * TL;
    with_radix<MAXR>(N1, [&](auto r) {
        constexpr int R = decltype(r)::value;
        double2 v[R];
        const bool act = q < N2;
        if (act) {
#pragma unroll
            for (int n1 = 0; n1 < R; ++n1) v[n1] = src(q + N2 * n1, l);
        }
        __syncthreads();   // twiddles complete; src's shared operands read
        if (act) {
            dft_reg<R, SIGN>(v, tw, 0);
            S[t] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < R; ++k1) S[k1 * KS + t] = tw.template mul<SIGN>(v[k1], q * k1);
        }
    });
    __syncthreads();
    with_radix<MAXR>(N2, [&](auto r) {
        constexpr int R = decltype(r)::value;
        if (q < N1) {
            double2 v[R];
#pragma unroll
            for (int m = 0; m < R; ++m) v[m] = S[q * KS + m * TL + l];
            dft_reg<R, SIGN>(v, tw, 0);
#pragma unroll
            for (int k2 = 0; k2 < R; ++k2) dst(q + N1 * k2, l, v[k2]);
        }
    });
}

// threads per block; 18 warps per SM of at most 96 registers in every instance (with
// the 160 that the larger ones take when left free, 12 warps: 162 lines-and-rows 97
// and 63 us instead of 78 and 52, 288 424 and 222 instead of 338 and 191, although
// the 25 instance spills a kilobyte)
__host__ __device__ constexpr int z_threads(int maxr) { return maxr > 16 ? 192 : 272; }
__host__ __device__ constexpr int z_blocks(int maxr) { return maxr > 16 ? 3 : 2; }
template <int MAXR>
__global__ void __launch_bounds__(z_threads(MAXR), z_blocks(MAXR))
k_z_backward_any(Dims d, int N1, int N2, const double2 *__restrict__ roots, const double2 *__restrict__ F,
                 double2 *__restrict__ G, int TL, bool coarse) {
    chain_begin();
    extern __shared__ double2 sm_d[];
    const int n = N1 * N2;
    const int f = blockIdx.z, j = blockIdx.y, kx0 = blockIdx.x * TL;
    const Twiddles<double2> tw = load_twiddles<double2>(sm_d, roots, n);
    const ZExpandSrc<double2> src{F + ((long long)f * d.ny2 + j) * d.fcol, d.nkx, kx0, d.NZS, n, coarse};
    const RowDst<double2> dst{G + ((long long)f * d.ny2 + j) * (long long)n * d.nkx, d.nkx, kx0};
    fft2_any<MAXR, +1>(N1, N2, TL, tw, sm_d + n, src, dst);
}
template <int MAXR>
__global__ void __launch_bounds__(z_threads(MAXR), z_blocks(MAXR))
k_z_forward_any(Dims d, int N1, int N2, const double2 *__restrict__ roots, const double2 *__restrict__ H,
                double2 *__restrict__ F, int TL, bool coarse) {
    chain_begin();
    extern __shared__ double2 sm_d[];
    const int n = N1 * N2;
    const int f = blockIdx.z, j = blockIdx.y, kx0 = blockIdx.x * TL;
    const Twiddles<double2> tw = load_twiddles<double2>(sm_d, roots, n);
    const RowSrc<double2> src{H + ((long long)f * d.ny2 + j) * (long long)n * d.nkx, d.nkx, kx0};
    const ZTruncDst<double2> dst{F + ((long long)f * d.ny2 + j) * d.fcol, d.nkx, kx0, d.NZS, n, 1.0 / (double)n,
                                 coarse};
    fft2_any<MAXR, -1>(N1, N2, TL, tw, sm_d + n, src, dst);
}

// ---------------------------------------------------------------------------
// x stage: inverse transforms of u and omega, N = u x omega, forward transforms.
// Two rows z, z + 1 of one field make a line (a + i b), so that the products
// are formed part by part: N_c = u_a om_b - u_b om_a needs four lines, each out
// line three such operands fewer than a packing of two fields would.  A block
// holds NP row pairs, 6 NP inverse lines [line][N1][SP], SP = N2 | 1, T =
// max(N1, N2) threads per line:
//   1  thread n2: spectrum slots n2 + N2 n1 from HBM, N1-point DFT, twiddle
//      -> rows k1
//   2  thread k1: N2-point DFT of row k1 in place: x = k1 + N1 k2 at [k1][k2]
//   3  thread k1 (out lines): products of row k1, N2-point DFT over k2
//      (frequency q2), twiddle -> row k1
//   4  thread q2: N1-point DFT of column q2 in place: q = q2 + N2 q1 at [q1][q2]
//   5  Hermitian unpack of q and n - q, modes q <= NXS -> HBM, along kx.
// Rows are written where they were read in 2 and 4, so those need no barrier
// between; SP odd keeps rows and columns free of bank conflicts.
// ---------------------------------------------------------------------------
// 18 to 20 warps per SM of at most 96 registers (176 and 380 bytes spilled), 15 of
// 128 in the 25 instance (484): warps count for more than spills here.  With 15 of
// 128 the smaller instances took 271 instead of 251 us at 240 points and 216 instead
// of 196 at 200; with 10 of 168 the 25 instance took 1.39 ms at 384 instead of 1.12.
__host__ __device__ constexpr int x_threads(int maxr) { return maxr > 20 ? 160 : 128; }
template <int MAXR>
__global__ void __launch_bounds__(x_threads(MAXR), MAXR > 20 ? 3 : 5)
k_x_cross_any(Dims d, int N1, int N2, int NP, const double2 *__restrict__ roots, const double2 *__restrict__ G,
              double2 *__restrict__ H) {
    chain_begin();
    extern __shared__ double2 sm_d[];
    const int n = N1 * N2, SP = N2 | 1, LS = N1 * SP;
    const int T = N1 > N2 ? N1 : N2;
    double2 *tab = sm_d;             // W_n^(n2 k1) at [k1][n2], row stride SP
    double2 *buf = sm_d + N1 * SP;   // [6 NP][LS]
    const int nkx = d.nkx, nxs = d.NXS;
    const int j = blockIdx.y, z0 = blockIdx.x * 2 * NP;
    const long long fstride = (long long)d.ny2 * d.NZ2 * nkx;
    const double2 *Gj = G + (long long)j * d.NZ2 * nkx;
    const FastDiv byN2(N2);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int k1 = byN2(i), n2 = i - k1 * N2;
        tab[k1 * SP + n2] = roots[k1 * n2];
    }
    const Twiddles<double2> none{nullptr, nullptr};
    const int line = threadIdx.x / T, sub = threadIdx.x - line * T;
    const int L = 6 * NP, L2 = 3 * NP;
    const int nyq = (n % 2 == 0) ? n / 2 : -1;
    // ---- 1 ----
    with_radix<MAXR>(N1, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        double2 v[R];
        const bool act = line < L && sub < N2;
        if (act) {
            const int pr = line / 6, f = line - (line / 6) * 6;
            const int z = z0 + 2 * pr;
            const bool hasA = z < d.NZ2, hasB = z + 1 < d.NZ2;
            const double2 *rowA = Gj + f * fstride + (long long)z * nkx;
            const double2 *rowB = rowA + nkx;
#pragma unroll
            for (int n1 = 0; n1 < R; ++n1) {
                const int m = sub + N2 * n1;
                const bool lo = m <= nxs, in = lo || (m >= n - nxs && m != nyq);
                const int mm = lo ? m : n - m;
                double2 A = mk(0.0, 0.0), B = mk(0.0, 0.0);
                if (in && hasA) A = rowA[mm];
                if (in && hasB) B = rowB[mm];
                if (mm == 0 || mm == nyq) {
                    A.y = 0.0;
                    B.y = 0.0;
                }
                v[n1] = lo ? mk(A.x - B.y, A.y + B.x) : mk(A.x + B.y, B.x - A.y);
            }
        }
        __syncthreads();   // table complete
        if (act) {
            dft_reg<R, +1>(v, none, 0);
            double2 *o = buf + line * LS + sub;
            o[0] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < R; ++k1) o[k1 * SP] = cmul(v[k1], cconj(tab[k1 * SP + sub]));
        }
    });
    __syncthreads();
    // ---- 2 ----
    with_radix<MAXR>(N2, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        if (line < L && sub < N1) {
            double2 v[R];
            double2 *o = buf + line * LS + sub * SP;
#pragma unroll
            for (int m = 0; m < R; ++m) v[m] = o[m];
            dft_reg<R, +1>(v, none, 0);
#pragma unroll
            for (int m = 0; m < R; ++m) o[m] = v[m];
        }
    });
    __syncthreads();
    // ---- 3 ----
    with_radix<MAXR>(N2, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        double2 v[R];
        const bool act = line < L2 && sub < N1;
        if (act) {
            const int pr = line / 3, c = line - (line / 3) * 3;
            const int ca = c == 2 ? 0 : c + 1, cb = c == 0 ? 2 : c - 1;
            const double2 *base = buf + pr * 6 * LS + sub * SP;
            const double2 *ua = base + ca * LS, *ub = base + cb * LS;
            const double2 *oa = base + (3 + ca) * LS, *ob = base + (3 + cb) * LS;
#pragma unroll
            for (int m = 0; m < R; ++m) {
                const double2 a = ua[m], b = ub[m], x = oa[m], y = ob[m];
                v[m] = mk(a.x * y.x - b.x * x.x, a.y * y.y - b.y * x.y);
            }
        }
        __syncthreads();
        if (act) {
            dft_reg<R, -1>(v, none, 0);
            double2 *o = buf + line * LS + sub * SP;
            const double2 *w = tab + sub * SP;
            o[0] = v[0];
#pragma unroll
            for (int m = 1; m < R; ++m) o[m] = cmul(v[m], w[m]);
        }
    });
    __syncthreads();
    // ---- 4 ----
    with_radix<MAXR>(N1, [&](auto rr) {
        constexpr int R = decltype(rr)::value;
        if (line < L2 && sub < N2) {
            double2 v[R];
            double2 *o = buf + line * LS + sub;
#pragma unroll
            for (int m = 0; m < R; ++m) v[m] = o[m * SP];
            dft_reg<R, -1>(v, none, 0);
#pragma unroll
            for (int m = 0; m < R; ++m) o[m * SP] = v[m];
        }
    });
    __syncthreads();
    // ---- 5 ----
    const double invn = 1.0 / (double)n;
    const FastDiv byK(nkx);
    for (int i = threadIdx.x; i < L2 * nkx; i += blockDim.x) {
        const int ol = byK(i), k = i - ol * nkx;
        const int pr = ol / 3, c = ol - (ol / 3) * 3;
        const int km = k == 0 ? 0 : n - k;
        const int k1 = byN2(k), m1 = byN2(km);
        const double2 *o = buf + ol * LS;
        const double2 p0 = o[k1 * SP + (k - k1 * N2)], pm = o[m1 * SP + (km - m1 * N2)];
        const int z = z0 + 2 * pr;
        double2 *h = H + c * fstride + ((long long)j * d.NZ2 + z) * nkx + k;
        if (z < d.NZ2) h[0] = cscale(invn, mk(0.5 * (p0.x + pm.x), 0.5 * (p0.y - pm.y)));
        if (z + 1 < d.NZ2) h[nkx] = cscale(invn, mk(0.5 * (p0.y + pm.y), -0.5 * (p0.x - pm.x)));
    }
}

// ---------------------------------------------------------------------------
// Chebyshev DCT-I of N + 1 points, N = NY2 = N1 x N2 even: k_ydct_r's algebra and
// phases (transforms.cu) with run-time factors and line width.  R = max(16, N1,
// N2) row groups of TL lines; thread t owns line t mod TL and row group t / TL.
// ---------------------------------------------------------------------------
constexpr int kYThreads = 256;
// blocks of kYThreads per SM that the registers are held to: 24 warps of 80 with
// factors up to 16 (181 points: 138 us a synthesis, 148 with 16 warps), else 16 of 128
__host__ __device__ constexpr int y_blocks(int maxr) { return maxr > 16 ? 2 : 3; }
constexpr int kYPairs = 4;     // pairs of rows of a thread in flight
constexpr int kYChunk = 13;    // (N/2 + 1) / R, rounded up, is at most this for N1, N2 <= 25
template <int MAXR, bool ANA>
__global__ void __launch_bounds__(kYThreads, y_blocks(MAXR))
k_ydct_any(Dims d, int N1, int N2, int TL, int R, const double2 *__restrict__ roots,
           const double *__restrict__ cosy, YdctArgs<double2> A) {
    chain_begin();
    const int N = N1 * N2;
    const int KS = fft2_kstride(N2, TL);
    const int M = N / 2 - 1;               // odd outputs beyond Y_1: k = 1..M
    const int CH = (N / 2 + R) / R;        // k = 0..N/2 in R chunks of CH
    extern __shared__ double2 sm_d[];
    double2 *Y = sm_d + N;
    double2 *P = Y + N1 * KS;
    double2 *Y1 = P + R * TL;
    const int f = blockIdx.z, kzi = blockIdx.y, kx0 = blockIdx.x * TL;
    const int t = threadIdx.x;
    const int r = t / TL, l = t - r * TL;
    const int nkx = d.nkx, ncy = d.ncy, kx = kx0 + l;
    const bool lok = kx < nkx;
    const Twiddles<double2> tw = load_twiddles<double2>(sm_d, roots, N);
    const FastDiv byN2(N2), byN1(N1);
    auto row = [&](int n) {
        const int q = byN2(n);
        return q * KS + (n - q * N2) * TL + l;
    };
    double2 y1 = mk(0.0, 0.0);
    {
        const double2 *S = nullptr;
        const double2 *F = nullptr;
        if (!ANA) S = (f < A.nsplit ? A.spec0 + (long long)f * d.Ns : A.spec1 + (long long)(f - A.nsplit) * d.Ns) +
                      spectral_base(d, kzi, kx);
        else F = A.Fin + (long long)f * d.ny2 * d.fcol + (long long)kzi * nkx + kx;
        for (int n0 = r; n0 <= N / 2; n0 += kYPairs * R) {
            double2 xa[kYPairs], xb[kYPairs];
#pragma unroll
            for (int i = 0; i < kYPairs; ++i) {
                const int n = n0 + R * i, m = N - n;
                const bool in = n <= N / 2 && lok;
                if (!ANA) {
                    xa[i] = (in && n < ncy) ? S[(long long)n * d.sy] : mk(0.0, 0.0);
                    xb[i] = (in && m < ncy) ? S[(long long)m * d.sy] : mk(0.0, 0.0);
                } else {
                    xa[i] = in ? F[(long long)n * d.fcol] : mk(0.0, 0.0);
                    xb[i] = in ? F[(long long)m * d.fcol] : mk(0.0, 0.0);
                }
            }
#pragma unroll
            for (int i = 0; i < kYPairs; ++i) {
                const int n = n0 + R * i;
                if (n > N / 2) break;
                const double w0 = !ANA ? (n == 0 ? 2.0 * A.in0 : A.in1) : (n == 0 ? A.inE : A.inI);
                const double w1 = !ANA ? A.in1 : (n == 0 ? A.inE : A.inI);
                const double2 a = cscale(w0, xa[i]), b = cscale(w1, xb[i]);
                const double2 h = cscale(0.5, cadd(a, b)), df = csub(a, b);
                const double sn = cosy[n < N / 2 ? n + N + N / 2 : 0];   // sin(pi n / N)
                y1 = cadd(y1, cscale(n == 0 ? 0.5 : cosy[n], df));
                Y[row(n)] = csub(h, cscale(sn, df));
                if (n > 0 && n < N / 2) Y[row(N - n)] = cadd(h, cscale(sn, df));
            }
        }
    }
    P[r * TL + l] = y1;
    __syncthreads();
    if (r == 0) {
        double2 acc = P[l];
        for (int q = 1; q < R; ++q) acc = cadd(acc, P[q * TL + l]);
        Y1[l] = acc;
    }
    // Z = DFT_N(y), in place
    with_radix<MAXR>(N1, [&](auto rr) {
        constexpr int Q = decltype(rr)::value;
        if (r < N2) {
            double2 v[Q];
            double2 *q = Y + r * TL + l;
#pragma unroll
            for (int n1 = 0; n1 < Q; ++n1) v[n1] = q[n1 * KS];
            dft_reg<Q, -1>(v, tw, 0);
            q[0] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < Q; ++k1) q[k1 * KS] = tw.template mul<-1>(v[k1], r * k1);
        }
    });
    __syncthreads();
    with_radix<MAXR>(N2, [&](auto rr) {
        constexpr int Q = decltype(rr)::value;
        if (r < N1) {
            double2 v[Q];
            double2 *q = Y + r * KS + l;
#pragma unroll
            for (int m = 0; m < Q; ++m) v[m] = q[m * TL];
            dft_reg<Q, -1>(v, tw, 0);
#pragma unroll
            for (int k2 = 0; k2 < Q; ++k2) q[k2 * TL] = v[k2];
        }
    });
    __syncthreads();
    auto Z = [&](int k) {
        const int q = byN1(k);
        return Y[(k - q * N1) * KS + q * TL + l];
    };
    double2 *Fo = nullptr;
    double2 *So = nullptr;
    if (!ANA) Fo = A.Fout + (long long)f * d.ny2 * d.fcol + (long long)kzi * nkx + kx;
    else So = A.S + (long long)f * d.Ns + spectral_base(d, kzi, kx);
    auto out = [&](int j, double2 v) {
        if (!lok) return;
        if (!ANA) {
            Fo[(long long)j * d.fcol] = cscale(j == 0 || j == N ? A.outE : A.outI, v);
        } else if (j < ncy) {
            So[(long long)j * d.sy] = cscale(j == 0 ? A.s0 : A.sk, v);
        }
    };
    double2 part[kYChunk];
    double2 run = mk(0.0, 0.0);
#pragma unroll
    for (int c = 0; c < kYChunk; ++c) {
        const int k = r * CH + c;
        if (c < CH && k <= N / 2) {
            const double2 zk = Z(k), zm = Z(k == 0 ? 0 : N - k);
            out(2 * k, cscale(0.5, cadd(zk, zm)));
            if (k >= 1 && k <= M) {
                const double2 dz = csub(zk, zm);
                run = cadd(run, mk(-0.5 * dz.y, 0.5 * dz.x));
            }
        }
        part[c] = run;
    }
    P[r * TL + l] = run;
    __syncthreads();
    double2 carry = mk(0.0, 0.0);
    for (int q = 0; q < r; ++q) carry = cadd(carry, P[q * TL + l]);
    const double2 y = Y1[l];
    if (r == 0) out(1, y);
#pragma unroll
    for (int c = 0; c < kYChunk; ++c) {
        const int k = r * CH + c;
        if (c < CH && k >= 1 && k <= M) out(2 * k + 1, cadd(y, cadd(carry, part[c])));
    }
}

// Most balanced split n = n1 x n2 into in-register lengths; false if none.
bool any_split(int n, int &n1, int &n2) {
    int best = 1 << 30;
    for (int a : kRadices) {
        if (n % a) continue;
        const int b = n / a;
        bool ok = false;
        for (int q : kRadices) ok = ok || q == b;
        if (ok && std::max(a, b) < best) {
            best = std::max(a, b);
            n1 = a;
            n2 = b;
        }
    }
    return best < (1 << 30);
}

// instance of a split: its largest factor's class; fn(Radix<16 | 20 | 25>)
template <class Fn> void with_instance(int n1, int n2, Fn &&fn) {
    const int t = std::max(n1, n2);
    if (t <= 16) fn(Radix<16>{});
    else if (t <= 20) fn(Radix<20>{});
    else fn(Radix<25>{});
}
int instance(int n1, int n2) {
    int m = 0;
    with_instance(n1, n2, [&](auto r) { m = decltype(r)::value; });
    return m;
}

size_t smem_z(int n1, int n2, int tl) {
    return sizeof(double2) * ((size_t)n1 * n2 + (size_t)n1 * fft2_kstride(n2, tl));
}
int z_width(int n1, int n2) { return z_threads(instance(n1, n2)) / std::max(n1, n2); }   // lines at most
// row pairs per block of the x stage: the most that stay within the thread bound
int x_pairs(int n1, int n2) { return std::max(1, x_threads(instance(n1, n2)) / (6 * std::max(n1, n2))); }
size_t smem_x(int n1, int n2) { return sizeof(double2) * (size_t)n1 * (n2 | 1) * (1 + 6 * x_pairs(n1, n2)); }
int y_rows(int n1, int n2) { return std::max(16, std::max(n1, n2)); }
size_t smem_y(int n1, int n2, int tl) {
    return sizeof(double2) *
           ((size_t)n1 * n2 + (size_t)n1 * fft2_kstride(n2, tl) + (size_t)(y_rows(n1, n2) + 1) * tl);
}
// kx lines per block of the DCT: as ydct_lines (transforms.cu), the width that
// keeps the most threads per SM on real lines
int y_lines(const Dims &d, int n1, int n2) {
    const int R = y_rows(n1, n2);
    int best = 8;
    double best_useful = -1.0;
    for (int tl : {16, 13, 11, 8}) {
        if (R * tl > kYThreads) continue;
        const int blocks = (int)std::min<size_t>((228u * 1024u) / (smem_y(n1, n2, tl) + 1024),
                                                 y_blocks(instance(n1, n2)) * kYThreads / (R * tl));
        const int padded = ((d.nkx + tl - 1) / tl) * tl;
        const double useful = (double)blocks * R * tl * d.nkx / padded;
        if (useful > best_useful) {
            best_useful = useful;
            best = tl;
        }
    }
    return best;
}
}  // namespace

bool any_length(int n) {
    int a, b;
    return any_split(n, a, b);
}

cudaError_t configure_any_kernels(const Dims &d) {
    int a, b;
    cudaError_t e = cudaSuccess;
    auto up = [&](auto *k, size_t sm) {
        if (e == cudaSuccess) e = raise_smem(k, sm);
    };
    if (any_split(d.NZ2, a, b)) {
        const size_t sm = smem_z(a, b, z_width(a, b));
        with_instance(a, b, [&](auto r) {
            constexpr int M = decltype(r)::value;
            up(k_z_backward_any<M>, sm);
            up(k_z_forward_any<M>, sm);
        });
    }
    if (any_split(d.NX2, a, b))
        with_instance(a, b, [&](auto r) { up(k_x_cross_any<decltype(r)::value>, smem_x(a, b)); });
    if (d.NY2 % 2 == 0 && any_split(d.NY2, a, b)) {
        const size_t sm = smem_y(a, b, y_lines(d, a, b));
        with_instance(a, b, [&](auto r) {
            constexpr int M = decltype(r)::value;
            up(k_ydct_any<M, false>, sm);
            up(k_ydct_any<M, true>, sm);
        });
    }
    return e;
}

bool launch_z_any(const Dims &d, const double2 *roots, const double2 *in, double2 *out, int nf, bool backward,
                  int lines, bool coarse, cudaStream_t s) {
    int a, b;
    if (!any_split(d.NZ2, a, b)) return false;
    const int t = std::max(a, b), tl = std::min(lines, z_width(a, b));
    dim3 grid((d.nkx + tl - 1) / tl, d.ny2, nf);
    const size_t sm = smem_z(a, b, tl);
    with_instance(a, b, [&](auto r) {
        constexpr int M = decltype(r)::value;
        if (backward) launch_chained(k_z_backward_any<M>, grid, t * tl, sm, s, d, a, b, roots, in, out, tl, coarse);
        else launch_chained(k_z_forward_any<M>, grid, t * tl, sm, s, d, a, b, roots, in, out, tl, coarse);
    });
    return true;
}

bool launch_x_cross_any(const Dims &d, const double2 *roots, const double2 *G, double2 *H, cudaStream_t s) {
    int a, b;
    if (!any_split(d.NX2, a, b)) return false;
    const int t = std::max(a, b), np = x_pairs(a, b);
    dim3 grid((d.NZ2 + 2 * np - 1) / (2 * np), d.ny2);
    with_instance(a, b, [&](auto r) {
        launch_chained(k_x_cross_any<decltype(r)::value>, grid, 6 * np * t, smem_x(a, b), s, d, a, b, np, roots, G, H);
    });
    return true;
}

bool launch_ydct_any(const Dims &d, const Tables &t, int nf, bool ana, const YdctArgs<double2> &A, cudaStream_t s) {
    int a, b;
    if (d.NY2 % 2 || !any_split(d.NY2, a, b)) return false;
    const int R = y_rows(a, b), tl = y_lines(d, a, b);
    dim3 grid((d.nkx + tl - 1) / tl, d.nkz, nf);
    const size_t sm = smem_y(a, b, tl);
    with_instance(a, b, [&](auto r) {
        constexpr int M = decltype(r)::value;
        if (ana) launch_chained(k_ydct_any<M, true>, grid, R * tl, sm, s, d, a, b, tl, R, t.root_y, t.cosy, A);
        else launch_chained(k_ydct_any<M, false>, grid, R * tl, sm, s, d, a, b, tl, R, t.root_y, t.cosy, A);
    });
    return true;
}

}  // namespace cdns
