// Pieces shared by the transform kernels: the row functors of the z stage,
// the twiddle table and exchange stride of the register transforms, and the
// operands of the DCT kernels.
#pragma once

#include "cdns_kernels.cuh"
#include "fft_lines.cuh"

namespace cdns {

// The coarse-grid transform (coarse = true, src/fft/transforms.cpp:560-572)
// instead sums the two Nyquist coefficients into the shared slot.
template <class C> struct ZExpandSrc {
    const C *Fp;   // one (field, y point) plane [kz][kx]
    int nkx, kx0, NZS, n;
    bool coarse;
    __device__ __forceinline__ C operator()(int z, int line) const {
        const int kx = kx0 + line;
        if (kx >= nkx) return mkc<C>(0, 0);
        int kz;
        if (z <= NZS) {
            if (z == n - NZS) {
                if (coarse) return cadd(Fp[(2 * NZS) * nkx + kx], Fp[kx]);
                kz = -NZS;
            } else {
                kz = z;
            }
        } else if (z >= n - NZS) {
            kz = z - n;
        } else {
            return mkc<C>(0, 0);
        }
        return Fp[(kz + NZS) * nkx + kx];
    }
};
template <class C> struct RowDst {
    C *p;   // [pos][kx]
    int nkx, kx0;
    __device__ __forceinline__ void operator()(int pos, int line, C v) const {
        const int kx = kx0 + line;
        if (kx < nkx) p[(long long)pos * nkx + kx] = v;
    }
};
template <class C> struct RowSrc {
    const C *p;
    int nkx, kx0;
    __device__ __forceinline__ C operator()(int pos, int line) const {
        const int kx = kx0 + line;
        return kx < nkx ? p[(long long)pos * nkx + kx] : mkc<C>(0, 0);
    }
};
// Forward z: keep kz in [-NZS, NZS] scaled by 1/NZ2 (src/fft/transforms.cpp:658-665);
// at a full z spectrum slot NZS feeds both kz = +NZS and kz = -NZS, halved on
// the coarse grid (coarse = true, src/fft/transforms.cpp:506-511).
template <class C> struct ZTruncDst {
    C *Fp;
    int nkx, kx0, NZS, n;
    typename CReal<C>::T invn;
    bool coarse;
    __device__ __forceinline__ void operator()(int z, int line, C v) const {
        const int kx = kx0 + line;
        if (kx >= nkx) return;
        C s = cscale(invn, v);
        if (coarse && z <= NZS && z >= n - NZS) s = cscale((typename CReal<C>::T)0.5, s);
        if (z <= NZS) Fp[(z + NZS) * nkx + kx] = s;
        if (z >= n - NZS) Fp[(z - n + NZS) * nkx + kx] = s;
    }
};

// Row stride of fft2_lines' exchange between k1 groups: N2 TL padded to = TL
// (mod 8), so that a quarter-warp whose threads span two k1 groups touches 8
// distinct 16-byte bank groups (unpadded, N2 TL = 0 mod 8 for the even N2 used).
__host__ __device__ constexpr int fft2_kstride(int n2, int tl) { return n2 * tl + (((tl - n2 * tl) % 8) + 8) % 8; }

// Shared twiddle table of the register forms: n double2 slots, holding the
// FP64 roots, or the FP32 roots and their rounding residues.
template <class C> __device__ __forceinline__ Twiddles<C> load_twiddles(double2 *sm_d, const double2 *roots, int n) {
    C *hi = reinterpret_cast<C *>(sm_d);
    C *lo = sizeof(C) == 8 ? hi + n : hi;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double2 r = roots[i];
        hi[i] = cto<C>(r);
        if (sizeof(C) == 8) lo[i] = mkc<C>(r.x - (double)hi[i].x, r.y - (double)hi[i].y);
    }
    return Twiddles<C>{hi, lo};
}
// Operands of the DCT kernels; CT is the stage buffer's complex type (double2,
// or float2 for the mixed form's FP32 stages).  Synthesis: spectral
// spec0 / spec1 (fields f < nsplit / the rest), coefficient k weighted by
// in0 (k = 0) or in1, -> F, row j weighted by outE (j = 0, N) or outI; with
// `mean` (FP32 stages) the (kz, kx) = (0, 0) column goes to mean[f][j] in FP64
// and zeros to F.  Analysis: F, row j weighted by inE (j = 0, N) or inI, ->
// spectral S, coefficient k scaled by s0 (k = 0) or sk.  The forward
// transforms take unit weights and s0 = 1/N, sk = 2/N (times 1 / (NX2 NZ2) for
// FP32 stages, whose z and x analyses leave it out); the discrete adjoint's
// transposed stages take other weights (launch_ydct_adjoint_*).
template <class CT> struct YdctArgs {
    const double2 *spec0 = nullptr, *spec1 = nullptr;
    int nsplit = 0;
    const CT *Fin = nullptr;
    CT *Fout = nullptr;
    double2 *S = nullptr;
    double *mean = nullptr;
    double in0 = 1.0, in1 = 1.0, outE = 1.0, outI = 1.0;   // synthesis weights
    double inE = 1.0, inI = 1.0, s0 = 0.0, sk = 0.0;       // analysis weights and scales
};

// ---- any_length.cu: lengths n = N1 x N2 by factors switched at run time ----
bool any_length(int n);
cudaError_t configure_any_kernels(const Dims &d);
// false (nothing launched) where the length has no such split
bool launch_z_any(const Dims &d, const double2 *roots, const double2 *in, double2 *out, int nf, bool backward,
                  int lines, bool coarse, cudaStream_t s);
bool launch_x_cross_any(const Dims &d, const double2 *roots, const double2 *G, double2 *H, cudaStream_t s);
bool launch_ydct_any(const Dims &d, const Tables &t, int nf, bool ana, const YdctArgs<double2> &A, cudaStream_t s);

}  // namespace cdns
