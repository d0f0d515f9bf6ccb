// The angular scattering kernel of a context, built on the device
// (bfpm_solver.cu:1723-1790; tables.cpp: angular_kernel is the host's form, kept
// for table downloads): for each source group with mu1, mu2 != 0,
//   theta(in, out)^(mu1-1) exp(-theta/mu2) (1+|w_in|^2)^-1.5
// normalised over the input directions, entries below 1e-3 dropped; theta the
// angle between two directions in degrees.  All in double and in the host's
// order of operations (no contraction), each column's sum over increasing
// inputs, so the entries are the host's up to the last bits of acos, pow and exp.
//
// Why here: Ng NA^2 power and exponential evaluations (15M for a 16 x 16 x 222
// beam), the table's upload and the scan for its non-zero blocks were most of
// the time to load a beam's tables (28 ms of the 45 ms before a served beam's
// first step).  A thread takes one output direction of a group and walks the
// inputs twice -- the sum, then the entries -- which costs less than keeping the
// values.
#include "common.cuh"

#include <algorithm>
#include <type_traits>

namespace bfpn {

namespace {

// cos of the angle between directions, as the host evaluates it.
__device__ __forceinline__ double direction_norm2(double y, double z) {
    return __dadd_rn(__dadd_rn(1.0, __dmul_rn(y, y)), __dmul_rn(z, z));
}

template <typename T>
__global__ void __launch_bounds__(256) angular_kernel_kernel(const double* __restrict__ omega, const double* __restrict__ mu,
                                                             int NA, int Ng, T* __restrict__ ker_v) {
    extern __shared__ double dir[];  // [NA] y, z, norm and Jacobian of the input directions
    const int ek = blockIdx.y;
    T* K = ker_v + static_cast<size_t>(ek) * NA * NA;
    const double m1 = mu[ek * 3], m2 = mu[ek * 3 + 1];
    const int out = blockIdx.x * blockDim.x + threadIdx.x;
    if (ek == Ng - 1 || m1 == 0.0 || m2 == 0.0) {
        for (int in = 0; in < NA && out < NA; ++in) K[static_cast<size_t>(in) * NA + out] = T(0);
        return;
    }
    for (int in = threadIdx.x; in < NA; in += blockDim.x) {
        const double y = omega[2 * in], z = omega[2 * in + 1], n2 = direction_norm2(y, z);
        dir[4 * in] = y;
        dir[4 * in + 1] = z;
        dir[4 * in + 2] = __dsqrt_rn(n2);
        dir[4 * in + 3] = pow(n2, -1.5);
    }
    __syncthreads();
    if (out >= NA) return;
    const double oy = dir[4 * out], oz = dir[4 * out + 1], on = dir[4 * out + 2];
    auto value = [&](int in) {
        const double iy = dir[4 * in], iz = dir[4 * in + 1];
        const double dot = __dadd_rn(__dadd_rn(1.0, __dmul_rn(iy, oy)), __dmul_rn(iz, oz));
        double c = __ddiv_rn(dot, fmax(__dmul_rn(dir[4 * in + 2], on), kEpsilon));
        c = fmax(-1.0, fmin(1.0, c));
        const double theta = fabs(__ddiv_rn(__dmul_rn(acos(c), 180.0), 3.14159265358979323846));
        const double v = __dmul_rn(__dmul_rn(pow(theta, m1 - 1.0), exp(__ddiv_rn(-theta, m2))), dir[4 * in + 3]);
        return isfinite(v) ? v : 0.0;
    };
    double sum = 0.0;
    for (int in = 0; in < NA; ++in) sum = __dadd_rn(sum, value(in));
    for (int in = 0; in < NA; ++in) {
        double v = value(in);
        if (sum > kEpsilon) {
            v = __ddiv_rn(v, sum);
            if (v < 1e-3) v = 0.0;
        }
        K[static_cast<size_t>(in) * NA + out] = static_cast<T>(v);
    }
}

// First and one past the last non-zero column (within the tile) of each BK-row
// chunk of each NT-column tile of the listed groups' kernels; a warp per chunk.
__global__ void __launch_bounds__(256) angular_ranges_kernel(const float* __restrict__ ker_v, const int* __restrict__ groups,
                                                             int NA, int NT, int BK, int nk, int2* __restrict__ ranges) {
    const int nt = blockIdx.x, gz = blockIdx.y, lane = threadIdx.x & 31;
    const float* K = ker_v + static_cast<size_t>(groups[gz]) * NA * NA;
    const int n0 = nt * NT, n1 = min(NA, n0 + NT);
    for (int kc = threadIdx.x >> 5; kc < nk; kc += blockDim.x >> 5) {
        int lo = NT, hi = 0;
        for (int in = kc * BK; in < min(NA, (kc + 1) * BK); ++in)
            for (int o = n0 + lane; o < n1; o += 32)
                if (K[static_cast<size_t>(in) * NA + o] != 0.0f) {
                    lo = min(lo, o - n0);
                    hi = max(hi, o - n0 + 1);
                }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) ranges[(static_cast<size_t>(gz) * gridDim.x + nt) * nk + kc] = make_int2(lo, hi);
    }
}

}  // namespace

template <typename T>
cudaError_t launch_angular_kernel(const double* omega, const double* mu, int NA, int Ng, T* ker_v, cudaStream_t s) {
    const int block = std::min(256, (NA + 31) / 32 * 32);
    const size_t smem = static_cast<size_t>(NA) * 4 * sizeof(double);
    auto kern = angular_kernel_kernel<T>;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    if (e != cudaSuccess) return e;
    kern<<<dim3((NA + block - 1) / block, Ng), block, smem, s>>>(omega, mu, NA, Ng, ker_v);
    return cudaGetLastError();
}
template cudaError_t launch_angular_kernel<float>(const double*, const double*, int, int, float*, cudaStream_t);
template cudaError_t launch_angular_kernel<double>(const double*, const double*, int, int, double*, cudaStream_t);

cudaError_t launch_angular_ranges(const float* ker_v, const int* groups, int n_groups, int NA, int NT, int BK, int n_ntiles,
                                  int2* ranges, cudaStream_t s) {
    if (n_groups <= 0) return cudaSuccess;
    angular_ranges_kernel<<<dim3(n_ntiles, n_groups), 256, 0, s>>>(ker_v, groups, NA, NT, BK, (NA + BK - 1) / BK, ranges);
    return cudaGetLastError();
}

}  // namespace bfpn
