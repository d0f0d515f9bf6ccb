// Catastrophic secondary source (secondarySourceFromPrimaryKernel,
// energy_solver.cu:287-333):
//
//   S[e, pos, out] = dg * sum_{s in band(e)} sum_in ker_v[s, in, out]
//                      * (e1[e, s] * max(P1[s, pos, in], 0) + e2[e, s] * P2[s, pos, in] / 3)
//
// factorised into two contractions that each read their operands once:
//   A1[s, pos, out] = sum_in max(P1[s, pos, in], 0) * ker_v[s, in, out]   (angular GEMM per source group)
//   A2[s, pos, out] = sum_in P2[s, pos, in] * ker_v[s, in, out]
//   S[e, l]         = dg * (sum_s e1[e, s] A1[s, l] + (sum_s e2[e, s] A2[s, l]) / 3)   (banded energy GEMM)
// The reference re-reads the primary band*NA times per output cell.

#include "common.cuh"
#include "async_copy.cuh"

#include <algorithm>

namespace bfpn {

// Angular stage: per source group g, C[pos][out] = X[pos][in] * K[in][out]
// for X = max(P1, 0) and X = P2 at once (they share the K tiles).
// 64 x 64 output tile per block, 16 x 16 threads, 4 x 4 outputs per thread
// per operand, K staged through shared memory 16 deep.
template <typename T>
__global__ void __launch_bounds__(256) source_angular_kernel(SourceArgs<T> a) {
    constexpr int BM = 64, BN = 64, BK = 16;
    __shared__ T X1s[BK][BM + 1];
    __shared__ T X2s[BK][BM + 1];
    __shared__ T Ks[BK][BN];
    const int g = a.groups[blockIdx.z];
    const int NA = a.NA, nyz = a.nyz;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const T* __restrict__ P1 = a.P1 + static_cast<size_t>(g) * nyz * NA;
    const T* __restrict__ P2 = a.P2 + static_cast<size_t>(g) * nyz * NA;
    const T* __restrict__ K = a.ker_v + static_cast<size_t>(g) * NA * NA;
    T acc1[4][4], acc2[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) { acc1[i][j] = T(0); acc2[i][j] = T(0); }

    for (int k0 = 0; k0 < NA; k0 += BK) {
        for (int e = threadIdx.x; e < BM * BK; e += 256) {
            const int k = e % BK, m = e / BK;
            const int gm = m0 + m, gk = k0 + k;
            T x1 = T(0), x2 = T(0);
            if (gm < nyz && gk < NA) {
                x1 = P1[static_cast<size_t>(gm) * NA + gk];
                x2 = P2[static_cast<size_t>(gm) * NA + gk];
            }
            X1s[k][m] = max(x1, T(0));
            X2s[k][m] = x2;
        }
        for (int e = threadIdx.x; e < BK * BN; e += 256) {
            const int n = e % BN, k = e / BN;
            const int gn = n0 + n, gk = k0 + k;
            Ks[k][n] = (gn < NA && gk < NA) ? K[static_cast<size_t>(gk) * NA + gn] : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            T x1[4], x2[4], kv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { x1[i] = X1s[k][ty + 16 * i]; x2[i] = X2s[k][ty + 16 * i]; }
#pragma unroll
            for (int j = 0; j < 4; ++j) kv[j] = Ks[k][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc1[i][j] += x1[i] * kv[j];
                    acc2[i][j] += x2[i] * kv[j];
                }
        }
        __syncthreads();
    }
    T* __restrict__ A1 = a.A1 + static_cast<size_t>(g) * nyz * NA;
    T* __restrict__ A2 = a.A2 + static_cast<size_t>(g) * nyz * NA;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty + 16 * i;
        if (gm >= nyz) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx + 16 * j;
            if (gn < NA) {
                A1[static_cast<size_t>(gm) * NA + gn] = acc1[i][j];
                A2[static_cast<size_t>(gm) * NA + gn] = acc2[i][j];
            }
        }
    }
}

template <typename T>
cudaError_t launch_source_angular(const SourceArgs<T>& a, cudaStream_t s) {
    if (a.n_groups <= 0) return cudaSuccess;
    dim3 grid((a.NA + 63) / 64, (a.nyz + 63) / 64, a.n_groups);
    source_angular_kernel<T><<<grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// FP64 angular stage on the double tensor instruction, block-sparse.  The
// kernel drops entries below 1e-3, so most of its (8 rows x 32 columns) blocks
// are zero (63 % on water's 20 x 20 angles); block_mask_kernel marks the others
// once per table load and a block multiplies only those.  A block computes 64
// positions x 32 outputs of both operands: a warp 16 positions, per k = 4 step
// 16 m8n8k4 products from 8 operand loads (the SIMT tile above loads 12 values
// per 32 multiply-adds and covers every block).  441 positions, 400 angles, 385
// groups: 9.16 -> 1.50 ms (35 TFLOP/s of the multiplied blocks); 121 positions,
// 121 angles: 0.297 -> 0.162 ms.  Chunks of 8 rows
// come in through three cp.async stages; the pitches (12 and 36 doubles) keep
// the fragment loads off each other's banks.  The sums are IEEE fma chains in
// the chunks' order.
// ---------------------------------------------------------------------------
constexpr int kMaskRows = 8, kMaskCols = 32;

__global__ void __launch_bounds__(256) block_mask_kernel(const double* __restrict__ ker_v, const int* __restrict__ groups,
                                                         int NA, int words, uint32_t* __restrict__ mask) {
    const int gz = blockIdx.y, tile = blockIdx.x, lane = threadIdx.x & 31;
    const double* K = ker_v + static_cast<size_t>(groups[gz]) * NA * NA;
    uint32_t* out = mask + (static_cast<size_t>(gz) * gridDim.x + tile) * words;
    const int n = tile * kMaskCols + lane, chunks = (NA + kMaskRows - 1) / kMaskRows;
    for (int w = threadIdx.x >> 5; w < words; w += 8) {  // a warp per word
        uint32_t bits = 0;
        for (int b = 0; b < 32 && w * 32 + b < chunks; ++b) {
            bool any = false;
            for (int r = 0; r < kMaskRows; ++r) {
                const int k = (w * 32 + b) * kMaskRows + r;
                if (k < NA && n < NA) any |= K[static_cast<size_t>(k) * NA + n] != 0.0;
            }
            if (__any_sync(0xffffffffu, any)) bits |= 1u << b;
        }
        if (lane == 0) out[w] = bits;
    }
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(128) source_angular_f64_kernel(SourceArgs<double> a, const uint32_t* __restrict__ mask,
                                                                 int words) {
    constexpr int BM = 64, BN = kMaskCols, BK = kMaskRows, AP = 12, BP = 36, NST = 3;
    __shared__ __align__(16) double As[NST][2][BM][AP];
    __shared__ __align__(16) double Bs[NST][BK][BP];
    __shared__ unsigned short list[4096 / BK];
    __shared__ int count;
    const int gz = blockIdx.z, g = a.groups[gz], NA = a.NA, nyz = a.nyz, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    if (warp == 0) {  // the chunks to multiply
        const uint32_t* w = mask + (static_cast<size_t>(gz) * gridDim.x + blockIdx.x) * words;
        int n = 0;
        for (int i = 0; i < words; ++i) {
            const uint32_t bits = __ldg(w + i);
            if ((bits >> lane) & 1) list[n + __popc(bits & ((1u << lane) - 1))] = static_cast<unsigned short>(i * 32 + lane);
            n += __popc(bits);
        }
        if (lane == 0) count = n;
    }
    __syncthreads();
    const int n = count;
    const double* __restrict__ K = a.ker_v + static_cast<size_t>(g) * NA * NA;
    const bool vec = NA % 2 == 0;  // rows on 16-byte boundaries
    auto fill = [&](int i) {       // chunk list[i] into stage i % NST, one commit group
        if (i < n) {
            const int k0 = list[i] * BK, st = i % NST;
            const int per = vec ? BK / 2 : BK;  // pieces per row of 8
            for (int v = tid; v < 2 * BM * per; v += 128) {
                const int c = v % per, m = (v / per) % BM, op = v / (per * BM), k = k0 + c * (vec ? 2 : 1);
                const bool in = m0 + m < nyz && k < NA;
                const double* P = (op ? a.P2 : a.P1) + static_cast<size_t>(g) * nyz * NA;
                const double* src = in ? P + static_cast<size_t>(m0 + m) * NA + k : P;
                if (vec) cp_async16(&As[st][op][m][c * 2], src, in);
                else cp_async8(&As[st][op][m][c], src, in);
            }
            const int pern = vec ? BN / 2 : BN;
            for (int v = tid; v < BK * pern; v += 128) {
                const int c = v % pern, k = k0 + v / pern, col = n0 + c * (vec ? 2 : 1);
                const bool in = k < NA && col < NA;
                const double* src = in ? K + static_cast<size_t>(k) * NA + col : K;
                if (vec) cp_async16(&Bs[st][v / pern][c * 2], src, in);
                else cp_async8(&Bs[st][v / pern][c], src, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[2][2][BN / 8][2];
#pragma unroll
    for (int op = 0; op < 2; ++op)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int nt = 0; nt < BN / 8; ++nt) acc[op][mt][nt][0] = acc[op][mt][nt][1] = 0.0;
    for (int i = 0; i < NST - 1; ++i) fill(i);
    const int r = lane >> 2, q = lane & 3;
    for (int i = 0; i < n; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
        __syncthreads();  // chunk i has landed for every thread; chunk i - 1's stage is free
        fill(i + NST - 1);
        const int st = i % NST;
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            double av[2][2], bv[BN / 8];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                av[0][mt] = fmax(As[st][0][warp * 16 + mt * 8 + r][k4 + q], 0.0);
                av[1][mt] = As[st][1][warp * 16 + mt * 8 + r][k4 + q];
            }
#pragma unroll
            for (int nt = 0; nt < BN / 8; ++nt) bv[nt] = Bs[st][k4 + q][nt * 8 + r];
#pragma unroll
            for (int op = 0; op < 2; ++op)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int nt = 0; nt < BN / 8; ++nt) dmma(acc[op][mt][nt], av[op][mt], bv[nt]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int op = 0; op < 2; ++op) {
        double* __restrict__ A = (op ? a.A2 : a.A1) + static_cast<size_t>(g) * nyz * NA;
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const int m = m0 + warp * 16 + mt * 8 + r;
            if (m >= nyz) continue;
#pragma unroll
            for (int nt = 0; nt < BN / 8; ++nt) {
                const int col = n0 + nt * 8 + 2 * q;
                double* o = A + static_cast<size_t>(m) * NA + col;
                if (vec && col < NA) {
                    *reinterpret_cast<double2*>(o) = make_double2(acc[op][mt][nt][0], acc[op][mt][nt][1]);
                } else {
                    if (col < NA) o[0] = acc[op][mt][nt][0];
                    if (col + 1 < NA) o[1] = acc[op][mt][nt][1];
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 energy stage on the double tensor instruction.  A block computes 32 output
// groups x 64 lanes, a warp 8 of the groups: per k = 4 step 16 m8n8k4 products
// for both operands.  The source groups of the 32 outputs' union band stream
// through three cp.async stages, 8 at a time; a warp multiplies only the chunks
// its own 8 outputs' band meets (band8).  Coefficients and values are read once
// per block from L2, blocks of one lane range next to each other.  Against 16
// output groups per SIMT thread, whose every multiply-add loaded its coefficient
// from shared memory: 441 positions x 400 angles x 500 groups 1.75 -> 1.06 ms,
// 121 x 121 x 500 0.168 -> 0.128 ms, 289 x 64 x 200 0.073 -> 0.050 ms.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) source_energy_f64_kernel(SourceArgs<double> a, const int2* __restrict__ band8) {
    constexpr int BE = 32, BN = 64, BK = 8, EP = 12, VP = 68, NST = 3;
    __shared__ __align__(16) double Es[NST][2][BE][EP];
    __shared__ __align__(16) double Vs[NST][2][BK][VP];
    const int Ng = a.Ng, n_et = (Ng + BE - 1) / BE, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int e0 = static_cast<int>(blockIdx.x % n_et) * BE;
    const long long per_e = static_cast<long long>(a.nyz) * a.NA, l0 = static_cast<long long>(blockIdx.x / n_et) * BN;
    int lo = Ng, hi = 0;
    int2 own = make_int2(0, 0);
    for (int w = 0; w < BE / 8; ++w) {
        if (e0 + 8 * w >= Ng) break;
        const int2 b = __ldg(band8 + e0 / 8 + w);
        if (w == warp) own = b;
        if (b.x < b.y) {
            lo = min(lo, b.x);
            hi = max(hi, b.y);
        }
    }
    const int n = hi > lo ? (hi - lo + BK - 1) / BK : 0;
    const bool vec = per_e % 2 == 0;  // rows on 16-byte boundaries
    auto fill = [&](int i) {          // source groups lo + 8 i .. of the band into stage i % NST
        if (i < n) {
            const int s0 = lo + i * BK, st = i % NST;
            for (int v = tid; v < 2 * BE * BK; v += 128) {
                const int k = v % BK, e = (v / BK) % BE, op = v / (BK * BE), s = s0 + k;
                const bool in = s < hi && e0 + e < Ng;
                const double* E = op ? a.e2 : a.e1;
                cp_async8(&Es[st][op][e][k], in ? E + static_cast<size_t>(e0 + e) * Ng + s : E, in);
            }
            const int per = vec ? BN / 2 : BN, step = vec ? 2 : 1;
            for (int v = tid; v < 2 * BK * per; v += 128) {
                const int c = (v % per) * step, k = (v / per) % BK, op = v / (per * BK), s = s0 + k;
                const bool in = s < hi && l0 + c < per_e;
                const double* A = op ? a.A2 : a.A1;
                const double* src = in ? A + s * per_e + l0 + c : A;
                if (vec) cp_async16(&Vs[st][op][k][c], src, in);
                else cp_async8(&Vs[st][op][k][c], src, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[2][BN / 8][2];
#pragma unroll
    for (int op = 0; op < 2; ++op)
#pragma unroll
        for (int nt = 0; nt < BN / 8; ++nt) acc[op][nt][0] = acc[op][nt][1] = 0.0;
    for (int i = 0; i < NST - 1; ++i) fill(i);
    const int r = lane >> 2, q = lane & 3;
    for (int i = 0; i < n; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
        __syncthreads();  // chunk i has landed for every thread; chunk i - 1's stage is free
        fill(i + NST - 1);
        const int st = i % NST, s0 = lo + i * BK;
        if (s0 >= own.y || s0 + BK <= own.x) continue;  // zero coefficients for this warp's outputs
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
#pragma unroll
            for (int op = 0; op < 2; ++op) {
                const double ev = Es[st][op][warp * 8 + r][k4 + q];
                double bv[BN / 8];
#pragma unroll
                for (int nt = 0; nt < BN / 8; ++nt) bv[nt] = Vs[st][op][k4 + q][nt * 8 + r];
#pragma unroll
                for (int nt = 0; nt < BN / 8; ++nt) dmma(acc[op][nt], ev, bv[nt]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const int e = e0 + warp * 8 + r;
    if (e >= Ng) return;
    const double dg = a.dg, third = 1.0 / 3.0;
#pragma unroll
    for (int nt = 0; nt < BN / 8; ++nt) {
        const long long l = l0 + nt * 8 + 2 * q;
        const double v0 = dg * (acc[0][nt][0] + acc[1][nt][0] * third), v1 = dg * (acc[0][nt][1] + acc[1][nt][1] * third);
        double* o = a.S + e * per_e + l;
        if (vec && l < per_e) {
            *reinterpret_cast<double2*>(o) = make_double2(v0, v1);
        } else {
            if (l < per_e) o[0] = v0;
            if (l + 1 < per_e) o[1] = v1;
        }
    }
}

cudaError_t launch_source_energy_f64(const SourceArgs<double>& a, const int2* band8, cudaStream_t s) {
    const long long per_e = static_cast<long long>(a.nyz) * a.NA, blocks = (per_e + 63) / 64 * ((a.Ng + 31) / 32);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    source_energy_f64_kernel<<<static_cast<unsigned>(blocks), 128, 0, s>>>(a, band8);
    return cudaGetLastError();
}

int source_mask_words(int NA) { return ((NA + kMaskRows - 1) / kMaskRows + 31) / 32; }
size_t source_mask_bytes(int n_groups, int NA) {
    return static_cast<size_t>(n_groups) * ((NA + kMaskCols - 1) / kMaskCols) * source_mask_words(NA) * sizeof(uint32_t);
}
cudaError_t launch_source_mask(const double* ker_v, const int* groups, int n_groups, int NA, uint32_t* mask, cudaStream_t s) {
    if (n_groups <= 0) return cudaSuccess;
    const dim3 grid((NA + kMaskCols - 1) / kMaskCols, n_groups);
    block_mask_kernel<<<grid, 256, 0, s>>>(ker_v, groups, NA, source_mask_words(NA), mask);
    return cudaGetLastError();
}
cudaError_t launch_source_angular_f64(const SourceArgs<double>& a, const uint32_t* mask, cudaStream_t s) {
    if (a.n_groups <= 0) return cudaSuccess;
    if (a.NA > 4096) return cudaErrorNotSupported;
    const dim3 grid((a.NA + kMaskCols - 1) / kMaskCols, (a.nyz + 63) / 64, a.n_groups);
    source_angular_f64_kernel<<<grid, 128, 0, s>>>(a, mask, source_mask_words(a.NA));
    return cudaGetLastError();
}

// Float state: the same contraction on packed fp32x2 FMAs.  Accumulators
// pair neighbouring output groups of one lane, so one instruction applies the
// coefficients of outputs (2t, 2t+1) -- one 8-byte piece of a shared-memory
// row -- to the lane's value held twice.  Products and sums are the scalar
// kernel's, output by output.
template <int TE, int LN>
__global__ void __launch_bounds__(128) source_energy_f2_kernel(SourceArgs<float> a) {
    constexpr int SC = 32, TP = TE / 2;
    __shared__ __align__(16) float E1[SC][TE];
    __shared__ __align__(16) float E2[SC][TE];
    const int tile = blockIdx.x;
    const long long per_e = static_cast<long long>(a.nyz) * a.NA;
    const long long l0 = static_cast<long long>(blockIdx.y) * blockDim.x * LN + threadIdx.x;
    const int Ng = a.Ng, e0 = tile * TE;
    const int lo = a.tile_lo[tile], hi = a.tile_hi[tile];
    float2 q1[TP][LN], q2[TP][LN];
#pragma unroll
    for (int t = 0; t < TP; ++t)
#pragma unroll
        for (int j = 0; j < LN; ++j) q1[t][j] = q2[t][j] = make_float2(0.f, 0.f);
    long long lj[LN];
    bool ok[LN];
#pragma unroll
    for (int j = 0; j < LN; ++j) {
        lj[j] = l0 + static_cast<long long>(j) * blockDim.x;
        ok[j] = lj[j] < per_e;
    }
    for (int s0 = lo; s0 < hi; s0 += SC) {
        const int n = min(SC, hi - s0);
        __syncthreads();
        for (int k = threadIdx.x; k < SC * TE; k += blockDim.x) {
            const int ss = k / TE, t = k - ss * TE, e = e0 + t;
            const bool in = ss < n && e < Ng;
            E1[ss][t] = in ? static_cast<float>(a.e1[static_cast<size_t>(e) * Ng + s0 + ss]) : 0.f;
            E2[ss][t] = in ? static_cast<float>(a.e2[static_cast<size_t>(e) * Ng + s0 + ss]) : 0.f;
        }
        __syncthreads();
#pragma unroll 2
        for (int ss = 0; ss < n; ++ss) {
            const long long row = static_cast<long long>(s0 + ss) * per_e;
            float2 x1[LN], x2[LN];
#pragma unroll
            for (int j = 0; j < LN; ++j) {
                const float v1 = ok[j] ? a.A1[row + lj[j]] : 0.f, v2 = ok[j] ? a.A2[row + lj[j]] : 0.f;
                x1[j] = make_float2(v1, v1);
                x2[j] = make_float2(v2, v2);
            }
            const float2* c1 = reinterpret_cast<const float2*>(E1[ss]);
            const float2* c2 = reinterpret_cast<const float2*>(E2[ss]);
#pragma unroll
            for (int t = 0; t < TP; ++t) {
                const float2 a1 = c1[t], a2 = c2[t];
#pragma unroll
                for (int j = 0; j < LN; ++j) {
                    q1[t][j] = __ffma2_rn(a1, x1[j], q1[t][j]);
                    q2[t][j] = __ffma2_rn(a2, x2[j], q2[t][j]);
                }
            }
        }
    }
    const float dg = static_cast<float>(a.dg), third = 1.f / 3.f;
#pragma unroll
    for (int t = 0; t < TP; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = e0 + 2 * t + h;
            if (e >= Ng) continue;
#pragma unroll
            for (int j = 0; j < LN; ++j)
                if (ok[j]) {
                    const float s1 = h ? q1[t][j].y : q1[t][j].x, s2 = h ? q2[t][j].y : q2[t][j].x;
                    a.S[e * per_e + lj[j]] = dg * (s1 + s2 * third);
                }
        }
}

cudaError_t launch_source_energy(const SourceArgs<float>& a, int tile_e, cudaStream_t s) {
    constexpr int LN = 2;
    const long long per_e = static_cast<long long>(a.nyz) * a.NA;
    const int tiles = (a.Ng + tile_e - 1) / tile_e;
    const long long ly = (per_e + 128 * LN - 1) / (128 * LN);
    if (ly > 65535) return cudaErrorInvalidConfiguration;
    dim3 grid(tiles, static_cast<unsigned>(ly));
    switch (tile_e) {
        case 8: source_energy_f2_kernel<8, LN><<<grid, 128, 0, s>>>(a); break;
        case 16: source_energy_f2_kernel<16, LN><<<grid, 128, 0, s>>>(a); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template cudaError_t launch_source_angular<float>(const SourceArgs<float>&, cudaStream_t);

}  // namespace bfpn
