// Layout conversion between the reference's interleaved-component arrays
// ([kz][y][kx][c], src/core/array4d.hpp:62-67) and the component-planar tiled
// device layout (cdns_common.cuh).
#include "cdns_kernels.cuh"

namespace cdns {

// i: element of a component in the reference's order [kz][y][kx]
__device__ __forceinline__ long long tiled_index(const Dims &d, long long i) {
    const int kx = (int)(i % d.nkx);
    const long long q = i / d.nkx;
    const int y = (int)(q % d.ncy), kzi = (int)(q / d.ncy);
    return spectral_base(d, kzi, kx) + (long long)y * d.sy;
}

__global__ void k_deinterleave(const double2 *__restrict__ src, double2 *__restrict__ dst, Dims d, int nc) {
    const long long total = d.Nl * nc;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long e = i / nc;
        const int c = (int)(i - e * nc);
        dst[c * d.Ns + tiled_index(d, e)] = src[i];
    }
}

__global__ void k_interleave(const double2 *__restrict__ src, double2 *__restrict__ dst, Dims d, int nc) {
    const long long total = d.Nl * nc;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long e = i / nc;
        const int c = (int)(i - e * nc);
        dst[i] = src[c * d.Ns + tiled_index(d, e)];
    }
}

static int grid_for(long long total) {
    long long b = (total + 255) / 256;
    if (b > 148 * 32) b = 148 * 32;
    return (int)(b < 1 ? 1 : b);
}

void launch_deinterleave(const Dims &d, const double2 *src, double2 *dst, int nc, cudaStream_t s) {
    k_deinterleave<<<grid_for(d.Nl * nc), 256, 0, s>>>(src, dst, d, nc);
}

void launch_interleave(const Dims &d, const double2 *src, double2 *dst, int nc, cudaStream_t s) {
    k_interleave<<<grid_for(d.Nl * nc), 256, 0, s>>>(src, dst, d, nc);
}

}  // namespace cdns
