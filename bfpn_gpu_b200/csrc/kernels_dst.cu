// Angular diffusion, Eq. (19) (angle_diffusion.cu:7-34, 254-362, 420-483), on any
// angular grid up to 32 x 32: rows and columns of different lengths, or of a
// length without a kernel of its own (kernels_step.cu has the square grids).
//
// One block holds a tile of consecutive slices in shared memory and runs the
// forward u, forward v * factor * inverse v and inverse u passes there, a thread
// carrying a whole line in registers -- two lines on fp32x2 arithmetic for float
// state -- so a line's products take no shared-memory traffic (the
// run-time-length kernel reads two operands per product: 15 x 12 angles took
// 1.36 ms for 62M float cells, 0.29 here).  The transforms are compiled per length and
// picked by a block-uniform switch; a kernel is compiled for lengths up to 8,
// 16, 24 and 32, since the longest sets its registers.  What bounds it: latency -- a
// whole line per thread takes 148 registers at 15 x 12 angles, so 18 % of the
// warps are there to cover a line's chains and the block's barriers (issue 44 %, fma
// pipe 41 % busy).
#include "common.cuh"
#include "dst.cuh"

#include <algorithm>
#include <type_traits>

namespace bfpn {

namespace {

constexpr int kRectThreads = 128;

// Lines a thread carries: two floats on fp32x2, or one double.
template <typename T> struct RectLine;
template <> struct RectLine<float> {
    using V = float2;
    static constexpr int W = 2;
};
template <> struct RectLine<double> {
    using V = double;
    static constexpr int W = 1;
};
// Float: the N x N products in order, the run-time-length kernel's sums bit for bit
// (folding the line first would halve them, but round differently).
template <int N>
__device__ __forceinline__ void rect_dst(const float (&c)[(N + 1) / 2], const float2 (&x)[N], float2 (&y)[N]) {
#pragma unroll
    for (int m = 0; m < N; ++m) {
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int k = sine_k(N, m, i);
            if (k == 0) continue;
            const float cc = sine_neg(N, m, i) ? -c[k - 1] : c[k - 1];
            acc = __ffma2_rn(make_float2(cc, cc), x[i], acc);
        }
        y[m] = acc;
    }
}
template <int N>
__device__ __forceinline__ void rect_dst(const double (&c)[(N + 1) / 2], const double (&x)[N], double (&y)[N]) { dst1<N, double>(c, x, y); }

template <int N, typename T>
__device__ __forceinline__ void load_sines(const T* __restrict__ s, T (&c)[(N + 1) / 2]) {
#pragma unroll
    for (int k = 0; k < (N + 1) / 2; ++k) c[k] = __ldg(s + k);  // row 0 of the sine table
}

// Rows of N values at stride rs: in-place DST-I.  A float thread takes rows i
// and i + half (an odd last one is its own partner).
template <int N, typename T>
__device__ __noinline__ void rect_rows(T* X, int rs, int rows, const T* sines) {
    using V = typename RectLine<T>::V;
    constexpr int W = RectLine<T>::W;
    T c[(N + 1) / 2];
    load_sines<N, T>(sines, c);
    const int half = (rows + W - 1) / W;
    for (int i = threadIdx.x; i < half; i += kRectThreads) {
        T* a = X + i * rs;
        V x[N], y[N];
        if constexpr (W == 2) {
            T* b = X + (i + half < rows ? i + half : i) * rs;
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = make_float2(a[k], b[k]);
            rect_dst<N>(c, x, y);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                a[k] = y[k].x;
                b[k] = y[k].y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = a[k];
            rect_dst<N>(c, x, y);
#pragma unroll
            for (int k = 0; k < N; ++k) a[k] = y[k];
        }
    }
}

// Columns of N values (Nom per slice): DST-I, times the slice's factors, DST-I.
template <int N, typename T>
__device__ __noinline__ void rect_cols(T* X, int rs, int Nom, int slices, const T* __restrict__ fac0, int first, int nyz,
                                       const T* sines) {
    using V = typename RectLine<T>::V;
    constexpr int W = RectLine<T>::W;
    T c[(N + 1) / 2];
    load_sines<N, T>(sines, c);
    const int cols = slices * Nom, half = (cols + W - 1) / W, NA = N * Nom;
    for (int i = threadIdx.x; i < half; i += kRectThreads) {
        const int sa = i / Nom, ma = i - sa * Nom;
        T* a = X + sa * N * rs + ma;
        const T* fa = fac0 + static_cast<size_t>((first + sa) / nyz) * NA + ma;
        V x[N], y[N];
        if constexpr (W == 2) {
            const int q = i + half < cols ? i + half : i, sb = q / Nom, mb = q - sb * Nom;
            T* b = X + sb * N * rs + mb;
            const T* fb = fac0 + static_cast<size_t>((first + sb) / nyz) * NA + mb;
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = make_float2(a[k * rs], b[k * rs]);
            rect_dst<N>(c, x, y);
#pragma unroll
            for (int k = 0; k < N; ++k) y[k] = __fmul2_rn(y[k], make_float2(__ldg(fa + k * Nom), __ldg(fb + k * Nom)));
            rect_dst<N>(c, y, x);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                a[k * rs] = x[k].x;
                b[k * rs] = x[k].y;
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k) x[k] = a[k * rs];
            rect_dst<N>(c, x, y);
#pragma unroll
            for (int k = 0; k < N; ++k) y[k] = mul_rn(y[k], __ldg(fa + k * Nom));
            rect_dst<N>(c, y, x);
#pragma unroll
            for (int k = 0; k < N; ++k) a[k * rs] = x[k];
        }
    }
}

// Calls f with the run-time length n (1 .. NMAX) as a compile-time constant.
template <int NMAX, typename F>
__device__ __forceinline__ void with_length(int n, const F& f) {
    switch (n) {
#define BFPN_LEN(k)                                                          \
    case k:                                                                  \
        if constexpr (k <= NMAX) f(std::integral_constant<int, k>());        \
        break;
        BFPN_LEN(1) BFPN_LEN(2) BFPN_LEN(3) BFPN_LEN(4) BFPN_LEN(5) BFPN_LEN(6) BFPN_LEN(7) BFPN_LEN(8)
        BFPN_LEN(9) BFPN_LEN(10) BFPN_LEN(11) BFPN_LEN(12) BFPN_LEN(13) BFPN_LEN(14) BFPN_LEN(15) BFPN_LEN(16)
        BFPN_LEN(17) BFPN_LEN(18) BFPN_LEN(19) BFPN_LEN(20) BFPN_LEN(21) BFPN_LEN(22) BFPN_LEN(23) BFPN_LEN(24)
        BFPN_LEN(25) BFPN_LEN(26) BFPN_LEN(27) BFPN_LEN(28) BFPN_LEN(29) BFPN_LEN(30) BFPN_LEN(31) BFPN_LEN(32)
#undef BFPN_LEN
        default: break;
    }
}

// magic: e / Nom = e * magic >> 20 for the elements of a tile (e Nom < 2^20).
template <int NMAX, typename T>
__global__ void __launch_bounds__(kRectThreads) angle_rect_kernel(AngleArgs<T> a, unsigned magic) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* const X = reinterpret_cast<T*>(smem_raw);
    const int Nom = a.Nom, Nmu = a.Nmu, NA = Nom * Nmu, SL = a.slices_per_block, rs = Nom | 1;  // odd stride: no bank conflicts
    const long long s0 = static_cast<long long>(blockIdx.x) * SL, total = static_cast<long long>(a.Ng) * a.nyz;
    const int ns = static_cast<int>(min(static_cast<long long>(SL), total - s0)), n = ns * NA;
    T* __restrict__ F = a.F + s0 * NA;
    // element e of the tile's contiguous run lies at row e / Nom of the padded layout
    for (int e = threadIdx.x; e < n; e += kRectThreads) {
        const unsigned row = (static_cast<unsigned>(e) * magic) >> 20;
        X[e + row * (rs - Nom)] = F[e];
    }
    __syncthreads();
    const long long ek0 = s0 / a.nyz;
    const int first = static_cast<int>(s0 - ek0 * a.nyz);  // the tile's first slice within group ek0
    with_length<NMAX>(Nom, [&](auto N) { rect_rows<decltype(N)::value, T>(X, rs, ns * Nmu, a.sine_u); });
    __syncthreads();
    with_length<NMAX>(Nmu, [&](auto N) {
        rect_cols<decltype(N)::value, T>(X, rs, Nom, ns, a.fac + ek0 * NA, first, a.nyz, a.sine_v);
    });
    __syncthreads();
    with_length<NMAX>(Nom, [&](auto N) { rect_rows<decltype(N)::value, T>(X, rs, ns * Nmu, a.sine_u); });
    __syncthreads();
    for (int e = threadIdx.x; e < n; e += kRectThreads) {
        const unsigned row = (static_cast<unsigned>(e) * magic) >> 20;
        F[e] = X[e + row * (rs - Nom)];
    }
}

}  // namespace

// Slices per block: as many as give every thread a line (two for float) in each
// pass.
template <typename T>
cudaError_t launch_angle_rect(const AngleArgs<T>& a, cudaStream_t s) {
    const int longest = std::max(a.Nom, a.Nmu);
    if (longest > 32) return cudaErrorNotSupported;
    AngleArgs<T> b = a;
    b.slices_per_block = std::max(1, RectLine<T>::W * kRectThreads / longest);
    const size_t smem = static_cast<size_t>(b.slices_per_block) * a.Nmu * (a.Nom | 1) * sizeof(T);
    const long long total = static_cast<long long>(a.Ng) * a.nyz;
    const long long blocks = (total + b.slices_per_block - 1) / b.slices_per_block;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    const unsigned magic = (1u << 20) / a.Nom + 1;
    auto go = [&](auto kern) {
        cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        kern<<<static_cast<unsigned>(blocks), kRectThreads, smem, s>>>(b, magic);
        return cudaGetLastError();
    };
    if (longest <= 8) return go(angle_rect_kernel<8, T>);
    if (longest <= 16) return go(angle_rect_kernel<16, T>);
    if (longest <= 24) return go(angle_rect_kernel<24, T>);
    return go(angle_rect_kernel<32, T>);
}
template cudaError_t launch_angle_rect<float>(const AngleArgs<float>&, cudaStream_t);
template cudaError_t launch_angle_rect<double>(const AngleArgs<double>&, cudaStream_t);

}  // namespace bfpn
