// Energy half-steps: the eq15 DG / Crank-Nicolson sweep and the legacy upwind
// sweep over the energy groups (energyDgCnKernel, energy_solver.cu:41-161),
// with the depth dose fused in, for one beam, the slots of a bundle, and the
// primary's closing and opening half-steps in one pass.
//
// A lane is one (position, angle); its groups are swept from Ng-1 down to 0 in
// place, the recursion in double for both state types.  The update of group g
// is linear in the group's old values (F, f), the difference u of the group
// above's old values, the source s and the difference d of the group above's
// new values (straggling adds the old F above and below):
//   F' = aF F + af f + au u + as s (+ ah F_above + al F_below) + ad d
//   f' = bF F + bf f + bu u + bs s (+ bh F_above + bl F_below) + bd d
// with the 8 to 14 constants of a group formed once on the host in double
// (tables.cpp: energy_coefficients).  Everything but the d terms is known
// before the sweep reaches the group, so the serial chain of a group is one
// fma and one subtraction; written operator by operator it was five double
// operations long and took 17 instead of 10 of them.
//
// What bounds it: on large planes HBM (and the 4-5 float/double conversions of
// a cell); on small planes (fewer lanes than the GPU has threads) the time of
// one group's chain, since the groups are serial.  So the values of the next
// groups are always in flight: each thread keeps a ring of its own lanes' old
// values in shared memory, filled by cp.async (no registers held by the
// prefetch, no barrier: a thread only reads what it copied), takes U groups
// per trip so their loads and their independent parts overlap, and the group
// constants sit in shared memory (read from L2 by every warp they cost a small
// plane about 1 us per group).  Measured per pass on a B200, before (a register
// ring, constants from L2, the update operator by operator) and now:
//   FP64  17 x 17 x 64 lanes, 200 groups    0.193 -> 0.038 ms
//   FP64  11 x 11 x 121 lanes, 500 groups   0.518 -> 0.090 ms
//   FP64  21 x 21 x 400 lanes, 500 groups   1.15  -> 0.553 ms (5.1 TB/s)
//   float 21 x 21 x 400 lanes, 500 groups   0.395 -> 0.321 ms (5.0 TB/s)
//   float 81 x 81 x 400 lanes, 500 groups   4.71  -> 4.39 ms  (5.7 TB/s)
//   fused 21 x 21 x 400 / 81 x 81 x 400     0.704 -> 0.510 / 8.76 -> 6.84 ms
#include "common.cuh"
#include "async_copy.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

namespace bfpn {

namespace {

// LPT consecutive lanes of T moved as one vector.
template <typename T, int LPT> struct LaneVec;
template <> struct LaneVec<float, 1> { using type = float; };
template <> struct LaneVec<float, 4> { using type = float4; };
template <> struct LaneVec<double, 1> { using type = double; };
template <> struct LaneVec<double, 2> { using type = double2; };

__device__ __forceinline__ void unpack(float v, float (&x)[1]) { x[0] = v; }
__device__ __forceinline__ void unpack(float4 v, float (&x)[4]) {
    x[0] = v.x;
    x[1] = v.y;
    x[2] = v.z;
    x[3] = v.w;
}
__device__ __forceinline__ void unpack(double v, double (&x)[1]) { x[0] = v; }
__device__ __forceinline__ void unpack(double2 v, double (&x)[2]) {
    x[0] = v.x;
    x[1] = v.y;
}
__device__ __forceinline__ void store_lanes(float* p, const float (&x)[1]) { *p = x[0]; }
__device__ __forceinline__ void store_lanes(float* p, const float (&x)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}
__device__ __forceinline__ void store_lanes(double* p, const double (&x)[1]) { *p = x[0]; }
__device__ __forceinline__ void store_lanes(double* p, const double (&x)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(x[0], x[1]);
}

// Ring depth (groups) and groups per trip.  One lane per thread: 16 groups
// deep, 4 per trip -- the few lanes of a small plane must cover the latency
// alone.  Vectors: 6 deep, 2 per trip -- more blocks fit beside the constants.
constexpr int ring_depth(int lpt) { return lpt == 1 ? 16 : 6; }
template <int LPT> struct RingShape { static constexpr int D = ring_depth(LPT), U = LPT == 1 ? 4 : 2; };

// Constants of a group kept in shared memory (double2 each: psi^1 row, psi^2 row).
template <int MODE, bool SRC>
constexpr int coef_count() {
    return MODE == EMODE_LEGACY ? 2 : 4 + (SRC ? 1 : 0) + (MODE == EMODE_EQ15_STRAG ? 2 : 0);
}
// Place in the global table of the j-th kept constant.
template <int MODE, bool SRC>
__device__ __forceinline__ int coef_place(int j) {
    return (!SRC && MODE == EMODE_EQ15_STRAG && j >= 4) ? j + 1 : j;
}

template <int MODE>
struct GroupCoef {
    double2 F, f, u, d, s, hi, lo;  // legacy: F = (1/dt, hi), f = (1/denominator, laplacian)
};

template <int MODE, bool SRC>
__device__ __forceinline__ GroupCoef<MODE> group_coef(const double2* k) {
    GroupCoef<MODE> c;
    c.F = k[0];
    c.f = k[1];
    if (MODE != EMODE_LEGACY) {
        c.u = k[2];
        c.d = k[3];
        if (SRC) c.s = k[4];
        if (MODE == EMODE_EQ15_STRAG) {
            c.hi = k[SRC ? 5 : 4];
            c.lo = k[SRC ? 6 : 5];
        }
    }
    return c;
}

// What a lane carries from group to group.
struct Carry {
    double Fo = 0.0, uo = 0.0;  // old F, and F - f, of the group above
    double F = 0.0, f = 0.0;    // eq15: F = F' - f' of the group above; legacy: its new F, f
};

// One group of one lane: old values Fg, fg, source sg, Flo the old F below
// (0 below group 0).  Advances the carry.
template <int MODE, bool SRC>
__device__ __forceinline__ void group_update(const GroupCoef<MODE>& c, Carry& y, double Fg, double fg, double sg,
                                             double Flo, double& Fv, double& fv) {
    if (MODE == EMODE_LEGACY) {
        double x = fma(c.F.y, y.F, fmax(Fg, 0.0) * c.F.x);
        if (SRC) x += sg;
        Fv = x * c.f.x;
        fv = fma(c.F.y, y.f, fg * c.F.x) * c.f.x;
        if (c.f.y > 0.0) Fv += c.f.y * (fmax(y.Fo, 0.0) - 2.0 * fmax(Fg, 0.0) + fmax(Flo, 0.0));
        Fv = fmax(Fv, 0.0);
        fv = fmax(fv, 0.0);
        y.Fo = Fg;
        y.F = Fv;
        y.f = fv;
    } else {
        double eF = c.u.x * y.uo, ef = c.u.y * y.uo;
        eF = fma(c.F.x, Fg, eF);
        ef = fma(c.F.y, Fg, ef);
        eF = fma(c.f.x, fg, eF);
        ef = fma(c.f.y, fg, ef);
        if (SRC) {
            eF = fma(c.s.x, sg, eF);
            ef = fma(c.s.y, sg, ef);
        }
        if (MODE == EMODE_EQ15_STRAG) {
            eF = fma(c.hi.x, y.Fo, eF);
            ef = fma(c.hi.y, y.Fo, ef);
            eF = fma(c.lo.x, Flo, eF);
            ef = fma(c.lo.y, Flo, ef);
        }
        Fv = fma(c.d.x, y.F, eF);
        fv = fma(c.d.y, y.F, ef);
        y.Fo = Fg;
        y.uo = Fg - fg;
        y.F = Fv - fv;
    }
}

// Sum of (acc, accp) over the block into the block's partial pair.
__device__ __forceinline__ void block_partials(double acc, double accp, double* out) {
    __shared__ double red[2][32];
    for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_down_sync(0xffffffffu, acc, o);
        accp += __shfl_down_sync(0xffffffffu, accp, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 0) {
        red[0][w] = acc;
        red[1][w] = accp;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s0 = 0.0, s1 = 0.0;
        for (int k = 0; k < static_cast<int>(blockDim.x >> 5); ++k) {
            s0 += red[0][k];
            s1 += red[1][k];
        }
        out[0] = s0;
        out[1] = s1;
    }
}

// A thread's lanes.  Consecutive ones, except in the float passes that write
// or stand in for the source operand's pass (tile): there a warp takes 8
// positions x 16 angles (four per thread) or 4 x 8 (one), so that what it
// stores in the operand -- 16 bytes for 8 angles of a position, 8 positions
// one line -- fills whole lines or sectors.  Half sectors from warps that
// drift apart cost the fused pass a factor of three (80x80: 21.0 ms with
// consecutive lanes, 7.8 ms with 4 x 32 tiles, 6.8 ms with 8 x 16); a pass
// without the operand is 3-10 % faster on consecutive lanes.
struct LaneSpan {
    long long lane0;
    int pos, ang;
    bool ok;
};
template <typename T, int LPT>
__device__ __forceinline__ LaneSpan lane_span(const EnergyArgs<T>& a, long long bid, bool tile) {
    LaneSpan s;
    const long long id = bid * blockDim.x + threadIdx.x;
    if (sizeof(T) == 4 && tile) {
        constexpr int TA = LPT == 4 ? 4 : 8, TP = 32 / TA;  // threads along the angles, positions
        const int l = threadIdx.x & 31, n_ang = (a.NA + TA * LPT - 1) / (TA * LPT);
        const long long warp = id >> 5, pg = warp / n_ang, pos = pg * TP + l / TA;
        s.ang = (static_cast<int>(warp - pg * n_ang) * TA + l % TA) * LPT;
        s.lane0 = pos * a.NA + s.ang;
        s.ok = s.ang < a.NA && s.lane0 < a.lanes;  // NA is a multiple of LPT, lanes of NA
        s.pos = static_cast<int>(pos);
    } else {
        s.lane0 = id * LPT;
        s.ok = s.lane0 < a.lanes;
        s.pos = s.ang = 0;
    }
    return s;
}

// Trapezoidal weight of a lane (1 elsewhere).
template <typename T>
__device__ __forceinline__ double lane_weight(const EnergyArgs<T>& a, long long lane) {
    double w = 1.0;
    if (a.partials && a.trapezoidal && lane < a.lanes) {
        const int pos = static_cast<int>((lane + a.lane0) / a.NA);
        const int iy = pos % (a.Ny + 1), iz = pos / (a.Ny + 1);
        if (iy == 0 || iy == a.Ny) w *= 0.5;
        if (iz == 0 || iz == a.Nz) w *= 0.5;
    }
    return w;
}

// Copies the group constants (and the dose weights, when the pass sums the
// dose) to shared memory; CS = false leaves them in global memory (tables too
// long for it).  Returns the ring's place behind them.
template <int MODE, bool SRC, bool CS, typename T>
__device__ __forceinline__ unsigned char* stage_coef(const EnergyArgs<T>& a, unsigned char* smem) {
    if (!CS) return smem;
    constexpr int NC = coef_count<MODE, SRC>();
    double2* tab = reinterpret_cast<double2*>(smem);
    const double2* g = reinterpret_cast<const double2*>(a.coef);
    for (int e = threadIdx.x; e < a.Ng * NC; e += blockDim.x) {
        const int ek = e / NC, j = e - ek * NC;
        tab[e] = __ldg(g + ek * (kEnergyCoef / 2) + coef_place<MODE, SRC>(j));
    }
    tab += a.Ng * NC;
    if (a.partials) {
        const double2* d = reinterpret_cast<const double2*>(a.dose_coef);
        for (int ek = threadIdx.x; ek < a.Ng; ek += blockDim.x) tab[ek] = __ldg(d + ek);
        tab += a.Ng;
    }
    __syncthreads();
    return reinterpret_cast<unsigned char*>(tab);
}

template <int MODE, bool SRC, bool CS, typename T>
__device__ __forceinline__ GroupCoef<MODE> coef_of(const EnergyArgs<T>& a, const unsigned char* smem, int ek) {
    constexpr int NC = coef_count<MODE, SRC>();
    if (CS) return group_coef<MODE, SRC>(reinterpret_cast<const double2*>(smem) + ek * NC);
    double2 k[NC];
    const double2* g = reinterpret_cast<const double2*>(a.coef) + static_cast<size_t>(ek) * (kEnergyCoef / 2);
#pragma unroll
    for (int j = 0; j < NC; ++j) k[j] = __ldg(g + coef_place<MODE, SRC>(j));
    return group_coef<MODE, SRC>(k);
}

template <int MODE, bool SRC, bool CS, typename T>
__device__ __forceinline__ double2 dose_of(const EnergyArgs<T>& a, const unsigned char* smem, int ek) {
    if (CS) return reinterpret_cast<const double2*>(smem)[a.Ng * coef_count<MODE, SRC>() + ek];
    return __ldg(reinterpret_cast<const double2*>(a.dose_coef) + ek);
}

// A thread's ring of the next groups' old values: NARR arrays of LPT lanes.
// Slot i % D holds group Ng-1-i; the slots a trip consumed are refilled in the
// next trip, one commit group per trip.
template <typename T, int LPT, int NARR>
struct Ring {
    static constexpr int D = RingShape<LPT>::D, U = RingShape<LPT>::U, DB = D / U;
    using V = typename LaneVec<T, LPT>::type;
    V* base;
    const T* src[NARR];
    long long L;
    int Ng;
    bool ok;

    __device__ __forceinline__ V* slot(int k, int arr) const {
        return base + (k * NARR + arr) * static_cast<int>(blockDim.x) + static_cast<int>(threadIdx.x);
    }
    __device__ __forceinline__ void fill(int trip) const {
        const int k0 = (trip % DB) * U;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = Ng - 1 - (trip * U + u);
            if (ok && e >= 0) {
                const size_t off = static_cast<size_t>(e) * L;
#pragma unroll
                for (int arr = 0; arr < NARR; ++arr) cp_async_ca<sizeof(V)>(slot(k0 + u, arr), src[arr] + off);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    __device__ __forceinline__ void start() const {
        for (int t = 0; t < DB; ++t) fill(t);
    }
    // The slots of `trip` (and, NEXT, the first one after it) have landed.
    template <bool NEXT>
    __device__ __forceinline__ void wait(int trip) const {
        if (trip > 0) fill(trip - 1 + DB);
        asm volatile("cp.async.wait_group %0;" ::"n"(NEXT ? DB - 2 : DB - 1) : "memory");
    }
};

// ---------------------------------------------------------------------------
// One half-step over one species' lanes [bid * blockDim.x * LPT, ...).
// ---------------------------------------------------------------------------
template <int MODE, bool SRC, bool CS, typename T, int LPT>
__device__ __forceinline__ void energy_body(const EnergyArgs<T>& a, long long bid) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int U = RingShape<LPT>::U, DB = RingShape<LPT>::D / U, NARR = SRC ? 3 : 2;
    constexpr bool kLow = MODE != EMODE_EQ15;  // needs the old F of the group below
    using R = Ring<T, LPT, NARR>;
    const int Ng = a.Ng;
    const LaneSpan span = lane_span<T, LPT>(a, bid, energy_tiled(SRC, a.partials != nullptr));
    const long long L = a.lanes, lane0 = span.lane0;
    const bool ok = span.ok;  // the lanes of a thread are all in or all out
    R ring;
    ring.L = L;
    ring.Ng = Ng;
    ring.ok = ok;
    ring.src[0] = a.F + lane0;
    ring.src[1] = a.f + lane0;
    if (SRC) ring.src[NARR - 1] = a.src + lane0;
    ring.base = reinterpret_cast<typename R::V*>(smem_raw + energy_table_bytes(Ng, coef_count<MODE, SRC>(), a.partials != nullptr, CS));
    ring.start();
    stage_coef<MODE, SRC, CS>(a, smem_raw);
    Carry y[LPT];
    double w[LPT], acc = 0.0, accp = 0.0;
#pragma unroll
    for (int j = 0; j < LPT; ++j) w[j] = lane_weight(a, lane0 + j);
    const bool dose = a.partials != nullptr;
    auto trip_of = [&](auto FULLc, int t) {
        constexpr bool full = decltype(FULLc)::value;
        ring.template wait<kLow>(t);
        const int k0 = (t % DB) * U, e0 = Ng - 1 - t * U;
        T F[U][LPT], f[U][LPT], s[U][LPT], Fn[LPT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            unpack(*ring.slot(k0 + u, 0), F[u]);
            unpack(*ring.slot(k0 + u, 1), f[u]);
            if (SRC) unpack(*ring.slot(k0 + u, NARR - 1), s[u]);
        }
        if (kLow) unpack(*ring.slot(((t + 1) % DB) * U, 0), Fn);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int ek = e0 - u;
            if (!full && ek < 0) break;
            const GroupCoef<MODE> c = coef_of<MODE, SRC, CS>(a, smem_raw, ek);
            const double2 dc = dose ? dose_of<MODE, SRC, CS>(a, smem_raw, ek) : make_double2(0.0, 0.0);
            T Fs[LPT], fs[LPT];
#pragma unroll
            for (int j = 0; j < LPT; ++j) {
                const double Flo = (kLow && ek > 0) ? static_cast<double>(u + 1 < U ? F[u + 1 < U ? u + 1 : u][j] : Fn[j]) : 0.0;
                double Fv, fv;
                group_update<MODE, SRC>(c, y[j], static_cast<double>(F[u][j]), static_cast<double>(f[u][j]),
                                        SRC ? static_cast<double>(s[u][j]) : 0.0, Flo, Fv, fv);
                Fs[j] = static_cast<T>(Fv);
                fs[j] = static_cast<T>(fv);
                if (dose && ok) {
                    acc = fma(w[j], fma(dc.x, static_cast<double>(Fs[j]), dc.y * static_cast<double>(fs[j])), acc);
                    accp += static_cast<double>(fs[j]);
                }
            }
            if (ok) {
                const size_t off = static_cast<size_t>(ek) * L + lane0;
                store_lanes(a.F + off, Fs);
                store_lanes(a.f + off, fs);
            }
        }
    };
    const int full_trips = Ng / U;
#pragma unroll 1
    for (int t = 0; t < full_trips; ++t) trip_of(std::true_type(), t);
    if (Ng % U) trip_of(std::false_type(), full_trips);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (dose) block_partials(acc, accp, a.partials + 2 * bid);
}

// One register budget per form: the vector forms run at least two blocks of up to
// 160 threads (320 double) beside each other, all but the fused pass with
// straggling, whose 220 registers leave one; the scalar ones one block of up to
// 640 threads, or what its ring leaves of that (block_threads).
template <int MODE, bool SRC, bool CS, typename T, int LPT>
__global__ void __launch_bounds__(kEnergyMaxLanes / LPT) energy_kernel(EnergyArgs<T> a) {
    energy_body<MODE, SRC, CS, T, LPT>(a, blockIdx.x);
}

template <int MODE, bool SRC, bool CS, int LPT>
__global__ void __launch_bounds__(kEnergyMaxLanes / LPT) energy_slots_kernel(const EnergyArgs<float>* __restrict__ args,
                                                                             const int* __restrict__ begin, int nslots) {
    const int s = find_slot(begin, nslots, blockIdx.x);
    const EnergyArgs<float> a = args[s];
    energy_body<MODE, SRC, CS, float, LPT>(a, blockIdx.x - __ldg(begin + s));
}

// ---------------------------------------------------------------------------
// Fused primary energy half-steps: the closing E1/2 of step n and the opening
// E1/2 of step n+1 in one sweep.  Without straggling the opening update of a
// group needs only the group's own midpoint and the opening results above it,
// so both updates of a group run together on one set of constants; straggling
// also needs the midpoint of the group below, so there the opening sweep runs
// one group behind.  The midpoint is rounded to float as the separate passes
// store it, so the states equal theirs.  The closing pass's IDD partials are
// those of energy_kernel.  At the midpoint the source groups' values go to the
// angular contraction's operand (split bf16), which removes that operand's own
// pass over the primary.
// ---------------------------------------------------------------------------
// LPT angles of one operand row, split into bf16 hi and lo.
constexpr size_t kOperandPart = 128 * 16 * 2;  // one (hi or lo) 128 x 16 bf16 tile
__device__ __forceinline__ void put_operand(uint8_t* p, const float (&x)[4]) {
    const __nv_bfloat162 h01 = __floats2bfloat162_rn(x[0], x[1]), h23 = __floats2bfloat162_rn(x[2], x[3]);
    const __nv_bfloat162 l01 = __floats2bfloat162_rn(x[0] - __low2float(h01), x[1] - __high2float(h01));
    const __nv_bfloat162 l23 = __floats2bfloat162_rn(x[2] - __low2float(h23), x[3] - __high2float(h23));
    uint2 hv, lv;
    hv.x = *reinterpret_cast<const uint32_t*>(&h01);
    hv.y = *reinterpret_cast<const uint32_t*>(&h23);
    lv.x = *reinterpret_cast<const uint32_t*>(&l01);
    lv.y = *reinterpret_cast<const uint32_t*>(&l23);
    *reinterpret_cast<uint2*>(p) = hv;
    *reinterpret_cast<uint2*>(p + kOperandPart) = lv;
}
__device__ __forceinline__ void put_operand(uint8_t* p, const float (&x)[1]) {
    const __nv_bfloat16 h = __float2bfloat16_rn(x[0]);
    *reinterpret_cast<__nv_bfloat16*>(p) = h;
    *reinterpret_cast<__nv_bfloat16*>(p + kOperandPart) = __float2bfloat16_rn(x[0] - __bfloat162float(h));
}

template <int MODE, bool CS, int LPT>
__global__ void __launch_bounds__(kEnergyMaxLanes / LPT) energy_fused_kernel(EnergyFusedArgs A) {
    const EnergyArgs<float>& a = A.e;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int U = RingShape<LPT>::U, DB = RingShape<LPT>::D / U;
    constexpr bool kStrag = MODE == EMODE_EQ15_STRAG;
    using R = Ring<float, LPT, 2>;
    const int Ng = a.Ng;
    const long long bid = blockIdx.x, L = a.lanes;
    const LaneSpan span = lane_span<float, LPT>(a, bid, true);
    const long long lane0 = span.lane0;
    const bool ok = span.ok;
    R ring;
    ring.L = L;
    ring.Ng = Ng;
    ring.ok = ok;
    ring.src[0] = a.F + lane0;
    ring.src[1] = a.f + lane0;
    ring.base = reinterpret_cast<typename R::V*>(smem_raw + energy_table_bytes(Ng, coef_count<MODE, false>(), a.partials != nullptr, CS));
    ring.start();
    stage_coef<MODE, false, CS>(a, smem_raw);
    Carry yc[LPT], yo[LPT];                 // closing and opening sweeps
    double pF[LPT], pf[LPT];                // straggling: midpoint of the group above
    double w[LPT], acc = 0.0, accp = 0.0;
#pragma unroll
    for (int j = 0; j < LPT; ++j) {
        w[j] = lane_weight(a, lane0 + j);
        pF[j] = pf[j] = 0.0;
    }
    // this thread's place in the source operand: position p, angles k0 .. of chunk k0 / 16
    const int p = ok ? span.pos : 0, k0 = ok ? span.ang : 0;
    uint8_t* op = A.ablob + (static_cast<size_t>(p >> 6) * A.nk + (k0 >> 4)) * 2 * kOperandPart;
    const size_t a_off1 = umma_kmajor_offset(p & 63, k0 & 15, 128), a_off2 = umma_kmajor_offset(64 + (p & 63), k0 & 15, 128);
    const size_t a_group = static_cast<size_t>(A.n_mt) * A.nk * 2 * kOperandPart;
    const bool dose = a.partials != nullptr, operand = A.ablob != nullptr && ok;
    // opening update of group eo from its midpoint mF, mf, Flo the midpoint below (straggling)
    auto open = [&](const GroupCoef<MODE>& c, int eo, const double (&mF)[LPT], const double (&mf)[LPT],
                    const double (&Flo)[LPT]) {
        float Fs[LPT], fs[LPT];
#pragma unroll
        for (int j = 0; j < LPT; ++j) {
            double Fv, fv;
            group_update<MODE, false>(c, yo[j], mF[j], mf[j], 0.0, Flo[j], Fv, fv);
            Fs[j] = static_cast<float>(Fv);
            fs[j] = static_cast<float>(fv);
        }
        if (ok) {
            const size_t off = static_cast<size_t>(eo) * L + lane0;
            store_lanes(a.F + off, Fs);
            store_lanes(a.f + off, fs);
        }
    };
    auto trip_of = [&](auto FULLc, int t) {
        constexpr bool full = decltype(FULLc)::value;
        ring.template wait<kStrag>(t);
        const int s0 = (t % DB) * U, e0 = Ng - 1 - t * U;
        float F[U][LPT], f[U][LPT], Fn[LPT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            unpack(*ring.slot(s0 + u, 0), F[u]);
            unpack(*ring.slot(s0 + u, 1), f[u]);
        }
        if (kStrag) unpack(*ring.slot(((t + 1) % DB) * U, 0), Fn);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int ek = e0 - u;
            if (!full && ek < 0) break;
            const GroupCoef<MODE> c = coef_of<MODE, false, CS>(a, smem_raw, ek);
            const double2 dc = dose ? dose_of<MODE, false, CS>(a, smem_raw, ek) : make_double2(0.0, 0.0);
            const int gz = operand ? __ldg(A.gmap + ek) : -1;
            float nF[LPT], nf[LPT];
            double mF[LPT], mf[LPT];
#pragma unroll
            for (int j = 0; j < LPT; ++j) {
                const double Flo = (kStrag && ek > 0) ? static_cast<double>(u + 1 < U ? F[u + 1 < U ? u + 1 : u][j] : Fn[j]) : 0.0;
                double Fv, fv;
                group_update<MODE, false>(c, yc[j], static_cast<double>(F[u][j]), static_cast<double>(f[u][j]), 0.0, Flo,
                                          Fv, fv);
                nF[j] = static_cast<float>(Fv);
                nf[j] = static_cast<float>(fv);
                mF[j] = static_cast<double>(nF[j]);
                mf[j] = static_cast<double>(nf[j]);
                if (dose && ok) {
                    acc = fma(w[j], fma(dc.x, mF[j], dc.y * mf[j]), acc);
                    accp += mf[j];
                }
            }
            if (gz >= 0) {
                uint8_t* o = op + static_cast<size_t>(gz) * a_group;
                float pos[LPT];
#pragma unroll
                for (int j = 0; j < LPT; ++j) pos[j] = fmaxf(nF[j], 0.f);
                put_operand(o + a_off1, pos);
                put_operand(o + a_off2, nf);
            }
            if (kStrag) {
                if (ek + 1 < Ng) open(coef_of<MODE, false, CS>(a, smem_raw, ek + 1), ek + 1, pF, pf, mF);
#pragma unroll
                for (int j = 0; j < LPT; ++j) {
                    pF[j] = mF[j];
                    pf[j] = mf[j];
                }
            } else {
                open(c, ek, mF, mf, mF);
            }
        }
    };
    const int full_trips = Ng / U;
#pragma unroll 1
    for (int t = 0; t < full_trips; ++t) trip_of(std::true_type(), t);
    if (Ng % U) trip_of(std::false_type(), full_trips);
    if (kStrag) {
        const double none[LPT] = {};
        open(coef_of<MODE, false, CS>(a, smem_raw, 0), 0, pF, pf, none);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (dose) block_partials(acc, accp, a.partials + 2 * bid);
}

// ---------------------------------------------------------------------------
// Lite-memory primary step (litePrimaryEnergyStepKernel, bfpm_solver.cu:593-620):
// psi^1 only, first-order upwind in energy with catastrophic attenuation,
// groups swept from Ng-1 down, in place:
//   F_g <- max((max(F_g,0)/dt + S_hi/dg * F_{g+1}) / max(denom, eps), 0)
// as max(k max(F_g, 0) + h F_{g+1}, 0) with the constants (k, h) of a group
// formed once on the host: the two FP64 divisions of a group were the serial
// chain (21 x 21 x 400 lanes, 500 groups, float: 0.88 ms a step against 0.11 ms
// of HBM traffic).  The IDD of the new state (Eq. 24 with psi^2 = 0,
// integratedDepthDoseLiteKernel, bfpm_solver.cu:523-591) is accumulated on the
// way as per-block partials; the psi^2 column is 0.
// ---------------------------------------------------------------------------
template <typename T, int LPT, bool CS>
__global__ void __launch_bounds__(kEnergyMaxLanes / LPT) lite_energy_kernel(EnergyArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int U = RingShape<LPT>::U, DB = RingShape<LPT>::D / U;
    using R = Ring<T, LPT, 1>;
    const int Ng = a.Ng;
    const LaneSpan span = lane_span<T, LPT>(a, blockIdx.x, false);
    const long long L = a.lanes, lane0 = span.lane0;
    const bool ok = span.ok;
    R ring;
    ring.L = L;
    ring.Ng = Ng;
    ring.ok = ok;
    ring.src[0] = a.F + lane0;
    ring.base = reinterpret_cast<typename R::V*>(smem_raw + energy_table_bytes(Ng, 1, true, CS));
    ring.start();
    double2* tab = reinterpret_cast<double2*>(smem_raw);  // [Ng] (k, h), then [Ng] dose weights
    const double2* gk = reinterpret_cast<const double2*>(a.coef);
    const double2* gd = reinterpret_cast<const double2*>(a.dose_coef);
    if (CS) {
        for (int e = threadIdx.x; e < Ng; e += blockDim.x) {
            tab[e] = __ldg(gk + e);
            tab[Ng + e] = __ldg(gd + e);
        }
        __syncthreads();
    }
    double w[LPT], next[LPT], acc = 0.0;
#pragma unroll
    for (int j = 0; j < LPT; ++j) {
        w[j] = lane_weight(a, lane0 + j);
        next[j] = 0.0;
    }
    auto trip_of = [&](auto FULLc, int t) {
        constexpr bool full = decltype(FULLc)::value;
        ring.template wait<false>(t);
        const int k0 = (t % DB) * U, e0 = Ng - 1 - t * U;
        T F[U][LPT];
#pragma unroll
        for (int u = 0; u < U; ++u) unpack(*ring.slot(k0 + u, 0), F[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int ek = e0 - u;
            if (!full && ek < 0) break;
            const double2 c = CS ? tab[ek] : __ldg(gk + ek);
            const double dose = CS ? tab[Ng + ek].x : __ldg(gd + ek).x;
            T Fs[LPT];
#pragma unroll
            for (int j = 0; j < LPT; ++j) {
                Fs[j] = static_cast<T>(fmax(fma(c.y, next[j], c.x * fmax(static_cast<double>(F[u][j]), 0.0)), 0.0));
                next[j] = static_cast<double>(Fs[j]);
                if (ok) acc = fma(w[j] * dose, next[j], acc);
            }
            if (ok) store_lanes(a.F + static_cast<size_t>(ek) * L + lane0, Fs);
        }
    };
    const int full_trips = Ng / U;
#pragma unroll 1
    for (int t = 0; t < full_trips; ++t) trip_of(std::true_type(), t);
    if (Ng % U) trip_of(std::false_type(), full_trips);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    block_partials(acc, 0.0, a.partials + 2 * static_cast<long long>(blockIdx.x));
}

// ---- launch shapes ----------------------------------------------------------
// Lanes per thread: vectors once they leave four warps for each SM; a vector
// never straddles two positions.
constexpr int kEnergySMs = 148;
int vector_lanes(size_t elem, long long lanes, int NA) {
    const int v = elem == 4 ? 4 : 2;
    return (NA % v == 0 && lanes >= static_cast<long long>(kEnergySMs) * 128 * v) ? v : 1;
}

// Threads of a pass (tile: whole warp tiles of lane_span).
long long pass_threads(size_t elem, long long lanes, int NA, int lpt, bool tile) {
    if (elem != 4 || !tile) return (lanes + lpt - 1) / lpt;
    const int ta = lpt == 4 ? 4 : 8, tp = 32 / ta;
    return 32 * ((lanes / NA + tp - 1) / tp) * ((NA + ta * lpt - 1) / (ta * lpt));
}

// Shared memory a block's ring may take: what a block may have less the partial
// sums' static array.
constexpr size_t kEnergyRingLimit = 227 * 1024 - 512;

// Blocks of at most kEnergyMaxLanes lanes and no more than have their ring of
// `arrays` values in shared memory (576 threads for FP64 single lanes with a
// source, at 384 bytes each; every other form's 640 lanes fit), as many for each
// SM (rounds), so the last round is as full as the others; at least 128 lanes, so
// a block's warps cover a copy's latency.
int block_threads(long long threads, size_t elem, int lpt, int arrays) {
    const size_t per_thread = static_cast<size_t>(ring_depth(lpt)) * arrays * lpt * elem;
    const long long most = std::min<long long>(kEnergyMaxLanes / lpt, kEnergyRingLimit / per_thread / 32 * 32),
                    rounds = std::max<long long>(1, (threads + kEnergySMs * most - 1) / (kEnergySMs * most));
    const long long per = (threads + kEnergySMs * rounds - 1) / (kEnergySMs * rounds);
    return static_cast<int>(std::max<long long>(128 / lpt, std::min<long long>(most, (per + 31) / 32 * 32)));
}

// arrays: what the pass's ring holds for a lane (psi^1, psi^2, the source).
struct PassShape { int lpt, threads; unsigned grid; };
PassShape pass_shape(size_t elem, long long lanes, int NA, int lpt, int arrays, bool tile) {
    const long long n = pass_threads(elem, lanes, NA, lpt, tile);
    const int b = block_threads(n, elem, lpt, arrays);
    return {lpt, b, static_cast<unsigned>((n + b - 1) / b)};
}

// Constants in shared memory while they leave room for the ring.
constexpr size_t kEnergySmemLimit = 200 * 1024;
template <int LPT, typename T>
size_t ring_bytes(int threads, int narr) {
    return static_cast<size_t>(RingShape<LPT>::D) * narr * threads * LPT * sizeof(T);
}

// Launches KERN<..., CS> with its shared memory.  CS only while the table fits.
template <int MODE, bool SRC, int LPT, typename T, typename FS, typename FG>
cudaError_t launch_staged(int Ng, bool dose, int threads, const FS& in_smem, const FG& in_global) {
    const size_t ring = ring_bytes<LPT, T>(threads, SRC ? 3 : 2);
    const size_t tab = energy_table_bytes(Ng, coef_count<MODE, SRC>(), dose, true);
    return tab + ring <= kEnergySmemLimit ? in_smem(tab + ring) : in_global(ring);
}

template <int MODE, bool SRC, typename T, int LPT>
cudaError_t launch_one(const EnergyArgs<T>& a, cudaStream_t s) {
    const PassShape sh = pass_shape(sizeof(T), a.lanes, a.NA, LPT, SRC ? 3 : 2, energy_tiled(SRC, a.partials != nullptr));
    auto go = [&](auto kern, size_t smem) {
        cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        kern<<<sh.grid, sh.threads, smem, s>>>(a);
        return cudaGetLastError();
    };
    return launch_staged<MODE, SRC, LPT, T>(
        a.Ng, a.partials != nullptr, sh.threads, [&](size_t b) { return go(energy_kernel<MODE, SRC, true, T, LPT>, b); },
        [&](size_t b) { return go(energy_kernel<MODE, SRC, false, T, LPT>, b); });
}

template <int MODE, bool SRC, int LPT>
cudaError_t launch_slots(const EnergyArgs<float>* args, const int* begin, int nslots, int blocks, int max_ng,
                         long long lanes, int NA, bool dose, cudaStream_t s) {
    const int threads = pass_shape(4, lanes, NA, LPT, SRC ? 3 : 2, energy_tiled(SRC, dose)).threads;
    auto go = [&](auto kern, size_t smem) {
        cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        kern<<<blocks, threads, smem, s>>>(args, begin, nslots);
        return cudaGetLastError();
    };
    return launch_staged<MODE, SRC, LPT, float>(
        max_ng, dose, threads, [&](size_t b) { return go(energy_slots_kernel<MODE, SRC, true, LPT>, b); },
        [&](size_t b) { return go(energy_slots_kernel<MODE, SRC, false, LPT>, b); });
}

template <int MODE, int LPT>
cudaError_t launch_fused(const EnergyFusedArgs& A, cudaStream_t s) {
    const PassShape sh = pass_shape(4, A.e.lanes, A.e.NA, LPT, 2, true);
    auto go = [&](auto kern, size_t smem) {
        cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        kern<<<sh.grid, sh.threads, smem, s>>>(A);
        return cudaGetLastError();
    };
    return launch_staged<MODE, false, LPT, float>(
        A.e.Ng, A.e.partials != nullptr, sh.threads, [&](size_t b) { return go(energy_fused_kernel<MODE, true, LPT>, b); },
        [&](size_t b) { return go(energy_fused_kernel<MODE, false, LPT>, b); });
}

template <typename T, int LPT>
cudaError_t launch_lite(const EnergyArgs<T>& a, cudaStream_t s) {
    const PassShape sh = pass_shape(sizeof(T), a.lanes, a.NA, LPT, 1, false);
    const size_t ring = ring_bytes<LPT, T>(sh.threads, 1), tab = energy_table_bytes(a.Ng, 1, true, true);
    const bool cs = tab + ring <= kEnergySmemLimit;
    auto kern = cs ? lite_energy_kernel<T, LPT, true> : lite_energy_kernel<T, LPT, false>;
    const size_t smem = cs ? tab + ring : ring;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
    if (e != cudaSuccess) return e;
    kern<<<sh.grid, sh.threads, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

int energy_grid(size_t elem, long long lanes, int NA, bool src, bool dose, int lanes_per_thread) {
    const int lpt = lanes_per_thread ? lanes_per_thread : vector_lanes(elem, lanes, NA);
    return static_cast<int>(pass_shape(elem, lanes, NA, lpt, src ? 3 : 2, energy_tiled(src, dose)).grid);
}

int lite_energy_grid(size_t elem, long long lanes, int NA) {
    return static_cast<int>(pass_shape(elem, lanes, NA, vector_lanes(elem, lanes, NA), 1, false).grid);
}

int energy_grid_most(size_t elem, long long lanes, int NA) {
    int most = lite_energy_grid(elem, lanes, NA);
    for (int lpt : {1, elem == 4 ? 4 : 2})
        for (bool src : {false, true}) most = std::max(most, energy_grid(elem, lanes, NA, src, true, lpt));
    return most;
}

template <typename T>
cudaError_t launch_energy(const EnergyArgs<T>& a, cudaStream_t s) {
    constexpr int V = sizeof(T) == 4 ? 4 : 2;
    const bool vec = vector_lanes(sizeof(T), a.lanes, a.NA) == V;
#define BFPN_ENERGY(mode, src) \
    return vec ? launch_one<mode, src, T, V>(a, s) : launch_one<mode, src, T, 1>(a, s)
    switch (a.mode) {
        case EMODE_EQ15:
            if (a.src) BFPN_ENERGY(EMODE_EQ15, true);
            BFPN_ENERGY(EMODE_EQ15, false);
        case EMODE_EQ15_STRAG:
            if (a.src) BFPN_ENERGY(EMODE_EQ15_STRAG, true);
            BFPN_ENERGY(EMODE_EQ15_STRAG, false);
        default:
            if (a.src) BFPN_ENERGY(EMODE_LEGACY, true);
            BFPN_ENERGY(EMODE_LEGACY, false);
    }
#undef BFPN_ENERGY
}
template cudaError_t launch_energy<float>(const EnergyArgs<float>&, cudaStream_t);
template cudaError_t launch_energy<double>(const EnergyArgs<double>&, cudaStream_t);

template <typename T>
cudaError_t launch_lite_energy(const EnergyArgs<T>& a, cudaStream_t s) {
    constexpr int V = sizeof(T) == 4 ? 4 : 2;
    return vector_lanes(sizeof(T), a.lanes, a.NA) == V ? launch_lite<T, V>(a, s) : launch_lite<T, 1>(a, s);
}
template cudaError_t launch_lite_energy<float>(const EnergyArgs<float>&, cudaStream_t);
template cudaError_t launch_lite_energy<double>(const EnergyArgs<double>&, cudaStream_t);

cudaError_t launch_energy_slots(const EnergyArgs<float>* args, const int* begin, int nslots, int blocks, int mode,
                                bool vec, bool src, bool dose, int max_ng, long long lanes, int NA, cudaStream_t s) {
    if (nslots <= 0 || blocks <= 0) return cudaSuccess;
    if (mode == EMODE_LEGACY || (vec && NA % 4 != 0)) return cudaErrorNotSupported;
#define BFPN_SLOTS(m, src_)                                                                                     \
    return vec ? launch_slots<m, src_, 4>(args, begin, nslots, blocks, max_ng, lanes, NA, dose, s)                  \
               : launch_slots<m, src_, 1>(args, begin, nslots, blocks, max_ng, lanes, NA, dose, s)
    if (mode == EMODE_EQ15) {
        if (src) BFPN_SLOTS(EMODE_EQ15, true);
        BFPN_SLOTS(EMODE_EQ15, false);
    }
    if (src) BFPN_SLOTS(EMODE_EQ15_STRAG, true);
    BFPN_SLOTS(EMODE_EQ15_STRAG, false);
#undef BFPN_SLOTS
}

bool energy_fused_supported(int mode) { return mode != EMODE_LEGACY; }

cudaError_t launch_energy_fused(const EnergyFusedArgs& A, cudaStream_t s) {
    const EnergyArgs<float>& a = A.e;
    if (!energy_fused_supported(a.mode) || a.src || a.lane0 != 0) return cudaErrorNotSupported;
    const bool vec = vector_lanes(4, a.lanes, a.NA) == 4;
    if (a.mode == EMODE_EQ15) return vec ? launch_fused<EMODE_EQ15, 4>(A, s) : launch_fused<EMODE_EQ15, 1>(A, s);
    return vec ? launch_fused<EMODE_EQ15_STRAG, 4>(A, s) : launch_fused<EMODE_EQ15_STRAG, 1>(A, s);
}

}  // namespace bfpn
