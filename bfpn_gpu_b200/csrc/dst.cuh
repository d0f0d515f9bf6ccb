// The discrete sine transform DST-I of one line of N values held in a thread's
// registers, for the angular-diffusion kernels.
#pragma once

#include <cuda_runtime.h>

namespace bfpn {

// One thread owns a whole row (or column) of a slice in registers.  The DST-I matrix is symmetric and
// S[m][N-1-i] = (-1)^m S[m][i], so y = S x needs only the first ceil(N/2)
// columns applied to x[i] +- x[N-1-i]: N*ceil(N/2) FMAs per row instead of N^2.
// Every entry sin(pi (m+1)(i+1) / (N+1)) is +- sin(pi k / (N+1)) for one
// k in 1..(N+1)/2, so the whole table is (N+1)/2 values held in registers;
// which value and which sign each FMA takes is fixed at compile time.
template <int N, typename T>
struct SineTable {
    T c[(N + 1) / 2];  // c[k-1] = sin(pi k / (N+1))
};

// Entry (m, i) of the DST-I matrix as (k, sign): the argument (m+1)(i+1) is
// reduced modulo 2(N+1); sin is 0 at 0 and N+1, negative on (N+1, 2(N+1)),
// and sin(pi b/(N+1)) = sin(pi (N+1-b)/(N+1)).
__host__ __device__ constexpr int sine_arg(int N, int m, int i) { return ((m + 1) * (i + 1)) % (2 * (N + 1)); }
__host__ __device__ constexpr int sine_k(int N, int m, int i) {
    const int a = sine_arg(N, m, i), b = a > N + 1 ? a - (N + 1) : a;
    return b < N + 1 - b ? b : N + 1 - b;
}
__host__ __device__ constexpr bool sine_neg(int N, int m, int i) { return sine_arg(N, m, i) > N + 1; }

// A product rounded on its own (never fused into a following add), so that
// every DST variant rounds the CN factor step the same way.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

template <int N, typename T>
__device__ __forceinline__ void dst1(const T (&c)[(N + 1) / 2], const T (&x)[N], T (&y)[N]) {
    constexpr int H = N / 2, HC = (N + 1) / 2;
    T p[HC], q[H > 0 ? H : 1];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        p[i] = x[i] + x[N - 1 - i];
        q[i] = x[i] - x[N - 1 - i];
    }
    if (N & 1) p[H] = x[H];
#pragma unroll
    for (int m = 0; m < N; ++m) {
        T acc = T(0);
        const int n_terms = (m & 1) ? H : HC;
#pragma unroll
        for (int i = 0; i < n_terms; ++i) {
            const int k = sine_k(N, m, i);
            if (k == 0) continue;  // sin(pi) = 0: (m+1)(i+1) a multiple of N+1
            const T v = (m & 1) ? q[i] : p[i];
            acc = sine_neg(N, m, i) ? fma(-c[k - 1], v, acc) : fma(c[k - 1], v, acc);
        }
        y[m] = acc;
    }
}

// DST-I of two lines at once (fp32x2): the scalar dst1's operations, pairwise.
template <int N>
__device__ __forceinline__ void dst1_pair(const float (&c)[(N + 1) / 2], const float2 (&x)[N], float2 (&y)[N]) {
    constexpr int H = N / 2, HC = (N + 1) / 2;
    float2 p[HC], q[H > 0 ? H : 1];
#pragma unroll
    for (int i = 0; i < H; ++i) {
        p[i] = __fadd2_rn(x[i], x[N - 1 - i]);
        q[i] = __ffma2_rn(x[N - 1 - i], make_float2(-1.f, -1.f), x[i]);
    }
    if (N & 1) p[H] = x[H];
#pragma unroll
    for (int m = 0; m < N; ++m) {
        float2 acc = make_float2(0.f, 0.f);
        const int n_terms = (m & 1) ? H : HC;
#pragma unroll
        for (int i = 0; i < n_terms; ++i) {
            const int k = sine_k(N, m, i);
            if (k == 0) continue;
            const float cc = sine_neg(N, m, i) ? -c[k - 1] : c[k - 1];
            acc = __ffma2_rn(make_float2(cc, cc), (m & 1) ? q[i] : p[i], acc);
        }
        y[m] = acc;
    }
}

}  // namespace bfpn
