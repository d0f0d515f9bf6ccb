// Lateral transport, Eq. (18) (spatial_transport.cu:23-161, 202-262), any plane
// up to 128 points wide, in place: the MUSCL predictor-corrector as a march
// over the z rows with whole y lines in the lanes of a warp.
//
// A block serves one (group, chunk) plane: a chunk is the 32 bytes of
// consecutive angles (8 float, 4 double) that one memory sector holds at each
// position.  Its angles form lines -- two float angles whose direction cosines
// share their signs run as one line on fp32x2 arithmetic; an angle without such
// a partner, or a double one, is a line of its own.  LW lanes carry a line's
// positions, YT consecutive ones each; 32 / LW lines share a warp.  A thread
// marches over the z rows with its cells' z-stencils in registers and takes
// the values beyond its own cells from the neighbouring lanes by shuffles.  So
// a cell's neighbours cost 12 / YT shuffles over both stages and no shared
// memory; rows of F come in through a shared ring by cp.async (32 bytes per
// position, whole sectors) and rows of the result leave through a shared
// buffer, so that global memory sees 16-byte pieces although the lanes run
// along y.  One block barrier per row publishes both.
//
// A line with omega_y < 0 is laid out from the far end, so that the upwind
// neighbour is always the previous position; the limiter's epsilon stays on
// the difference towards higher y, as in the reference.  Positions before the
// plane's first repeat its value, which makes their slopes and fluxes zero, so
// a line is padded at its upwind end and needs no boundary code but two masks.
//
// What bounds it: the limiter's minimum / compare instructions (10 per angle
// pair and face at half rate, 40 of them per pair and cell) and the issue slots
// around them.  Lanes without a position are lost, so the host takes the
// (LW, YT) with the fewest of them (plane of 81: 27 of 32 lanes, 3 positions
// each).  Measured per launch on a B200 (float; before: the row-streaming kernel
// with its y-stencil in shared memory, or, for directions that do not pair and
// for FP64, 27 x 27 tiles with halos and one angle per thread):
//   81 x 81 x 400 angles x 500 groups     5.72  -> 4.00 ms (issue 70 % busy)
//   49 x 49 x 256 x 400                   1.17  -> 0.96 ms
//   38 x 30 x (15 x 12) x 301, unpaired   1.38  -> 0.42 ms
//   62 x 62 x (7 x 15) x 94, unpaired     0.86  -> 0.32 ms
//   FP64 31 x 47 x (14 x 16) x 42         0.747 -> 0.158 ms
#include "common.cuh"
#include "async_copy.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace bfpn {

namespace {

constexpr int kMarchRing = 8;     // rows of F in shared memory; kMarchRing - 1 are copied ahead
constexpr int kMarchPitch = 48;   // bytes per position in shared memory: the chunk's 32, spread over the banks
constexpr int kMarchChunk = 32;   // bytes of consecutive angles per block

// ---- arithmetic of one line value: a pair of float angles, or one double ----
__device__ __forceinline__ float2 vneg(float2 x) { return make_float2(-x.x, -x.y); }  // (a modifier of the operand)
__device__ __forceinline__ float2 vsub(float2 x, float2 y) { return __fadd2_rn(x, vneg(y)); }
__device__ __forceinline__ float2 vadd(float2 x, float2 y) { return __fadd2_rn(x, y); }
__device__ __forceinline__ float2 vmul(float2 x, float2 y) { return __fmul2_rn(x, y); }
__device__ __forceinline__ float2 vfma(float2 x, float2 y, float2 z) { return __ffma2_rn(x, y, z); }
__device__ __forceinline__ float2 vmax(float2 x, float lo) { return make_float2(fmaxf(x.x, lo), fmaxf(x.y, lo)); }
__device__ __forceinline__ double vsub(double x, double y) { return x - y; }
__device__ __forceinline__ double vadd(double x, double y) { return x + y; }
__device__ __forceinline__ double vmul(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ double vfma(double x, double y, double z) { return fma(x, y, z); }
__device__ __forceinline__ double vmax(double x, double lo) { return fmax(x, lo); }
__device__ __forceinline__ float2 vselect(bool p, float2 x, float2 y) { return make_float2(p ? x.x : y.x, p ? x.y : y.y); }
__device__ __forceinline__ double vselect(bool p, double x, double y) { return p ? x : y; }

template <typename T> struct LineOf;
template <> struct LineOf<float> {
    using V = float2;
    static constexpr int W = 2;  // angles per line
    __device__ static V both(float x) { return make_float2(x, x); }
};
template <> struct LineOf<double> {
    using V = double;
    static constexpr int W = 1;
    __device__ static V both(double x) { return x; }
};

__device__ __forceinline__ float2 lane_up(float2 v, int w) {
    return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1, w), __shfl_up_sync(0xffffffffu, v.y, 1, w));
}
__device__ __forceinline__ float2 lane_down(float2 v, int w) {
    return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1, w), __shfl_down_sync(0xffffffffu, v.y, 1, w));
}
// Shared-memory stores under a predicate (no branch).
__device__ __forceinline__ void store_if(float2* p, float2 v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p st.shared.v2.f32 [%0], {%1, %2};\n\t}" ::"r"(smem_u32(p)),
                 "f"(v.x), "f"(v.y), "r"(static_cast<int>(on))
                 : "memory");
}
__device__ __forceinline__ void store_if(float* p, float v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(smem_u32(p)), "f"(v),
                 "r"(static_cast<int>(on))
                 : "memory");
}
__device__ __forceinline__ void store_if(double* p, double v, bool on) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.f64 [%0], %1;\n\t}" ::"r"(smem_u32(p)), "d"(v),
                 "r"(static_cast<int>(on))
                 : "memory");
}
__device__ __forceinline__ double lane_up(double v, int w) { return __shfl_up_sync(0xffffffffu, v, 1, w); }
__device__ __forceinline__ double lane_down(double v, int w) { return __shfl_down_sync(0xffffffffu, v, 1, w); }

// The limited slope (muscl_paper_slope, spatial_transport.cu:23-29) of the two
// differences around a cell is fwd max(0, max(min(2 theta, 1), min(theta, 2))),
// 0 where |fwd| < eps.  march_limit is it without the epsilon and the division:
// sgn(fwd) max(0, min(2b, |fwd|), min(b, 2|fwd|)) with b = sgn(fwd) back.
// march_keep is 1 where the difference towards higher indices (cut) is at
// least eps, else 0.  Float: min.xorsign.abs gives the smaller magnitude,
// negative where the signs differ; the compare is one saturating fma, exact
// because 2^57 eps is an integer below 2^24 (compares and selects run at half
// rate, on this kernel's scarce pipe).
__device__ __forceinline__ float march_limit1(float back, float back2, float fwd, float fwd2) {
    float a, b, m;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(a) : "f"(back2), "f"(fwd));
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(b) : "f"(back), "f"(fwd2));
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(0.f), "f"(a), "f"(b));
    return __int_as_float(__float_as_int(m) | (__float_as_int(fwd) & static_cast<int>(0x80000000u)));
}
__device__ __forceinline__ float march_keep1(float cut) {
    constexpr float scale = 144115188075855872.f;  // 2^57: eps = 1e-10 lies in [2^-34, 2^-33)
    constexpr float shift = 1.f - static_cast<float>(kEpsilon) * scale;
    static_assert(static_cast<float>(kEpsilon) * scale < 16777216.f && static_cast<float>(kEpsilon) * scale >= 8388608.f,
                  "2^57 eps is an integer of 24 bits");
    float k;
    asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(k) : "f"(fabsf(cut)), "f"(scale), "f"(shift));
    return k;
}
__device__ __forceinline__ float2 march_limit(float2 back, float2 back2, float2 fwd, float2 fwd2) {
    return make_float2(march_limit1(back.x, back2.x, fwd.x, fwd2.x), march_limit1(back.y, back2.y, fwd.y, fwd2.y));
}
__device__ __forceinline__ float2 march_keep(float2 cut) { return make_float2(march_keep1(cut.x), march_keep1(cut.y)); }
__device__ __forceinline__ double flip(double x, double s) {
    return __longlong_as_double(__double_as_longlong(x) ^
                                (__double_as_longlong(s) & static_cast<long long>(0x8000000000000000ull)));
}
// Same signs: min(max(|back|, |fwd|), 2 min(|back|, |fwd|)).
__device__ __forceinline__ double march_limit(double back, double, double fwd, double) {
    const double ab = fabs(back), af = fabs(fwd);
    const bool less = ab < af;
    const double lo = less ? ab : af, hi = less ? af : ab, lo2 = lo + lo;
    const double m = hi < lo2 ? hi : lo2;
    return (__double2hiint(back) ^ __double2hiint(fwd)) >= 0 ? flip(m, fwd) : 0.0;
}
__device__ __forceinline__ double march_keep(double cut) { return fabs(cut) >= kEpsilon ? 1.0 : 0.0; }

// Copies of one row between global memory and its shared slot, in the largest
// pieces (16, 8 or 4 bytes) the angle count allows.
struct RowCopy {
    int lg;      // log2 of the pieces per position
    int bytes;   // of a piece
    int n;       // pieces of a row
    int valid;   // bytes of the chunk inside the angle grid
};

// ---------------------------------------------------------------------------
// Row r of F arrives in iteration r.  Its differences complete the z face of
// row r-1.  Upwind from below (omega_z >= 0, lag 1) that closes the
// z-divergence of row i = r-1, from above (lag 2) that of row i = r-2; with the
// y-divergence of row i this gives the predictor P(i) and the half-updated row;
// P's own y-divergence follows at once (shuffles), and the z face of P the new
// row completes closes the corrector of row j = i - lag.  Rows beyond the plane
// repeat the edge row, as the reference's clamped indices do.  A warp whose
// lines share the sign of omega_z runs that sign's march (DNZ 0 or 1: 7 or 9
// values per cell live from row to row); a mixed one selects (DNZ 2, lag 2).
// Row j leaves the shared buffer in iteration j + 5, when every warp has it.
// ---------------------------------------------------------------------------
constexpr int kMarchOut = 4;  // output rows in shared memory

template <typename T, int LW, int YT, bool LONE>
__device__ __forceinline__ void march_body(const TransportArgs<T>& a, int n_chunks, int bid) {
    using V = typename LineOf<T>::V;
    constexpr int W = LineOf<T>::W, AC = kMarchChunk / static_cast<int>(sizeof(T)), PT = kMarchPitch / static_cast<int>(sizeof(T));
    constexpr int RF = kMarchRing;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int Ny = a.Ny, Nz = a.Nz, Ny1 = Ny + 1, NA = a.NA, RS = Ny1 * PT;
    T* const ring = reinterpret_cast<T*>(smem_raw);  // [RF][Ny1][PT]
    T* const outb = ring + RF * RS;                  // [kMarchOut][Ny1][PT]
    const int chunk = bid % n_chunks, ek = bid / n_chunks, a0 = chunk * AC, tid = threadIdx.x;
    const size_t zs = static_cast<size_t>(Ny1) * NA;
    const size_t base = static_cast<size_t>(ek) * (Nz + 1) * zs + a0;

    // ---- row copies ----
    RowCopy rc;
    const int abytes = NA * static_cast<int>(sizeof(T));
    rc.lg = abytes % 16 == 0 ? 1 : abytes % 8 == 0 ? 2 : 3;
    rc.bytes = kMarchChunk >> rc.lg;
    rc.n = Ny1 << rc.lg;
    rc.valid = min(kMarchChunk, (NA - a0) * static_cast<int>(sizeof(T)));
    const char* const gin = reinterpret_cast<const char*>(a.in + base);
    char* const gout = reinterpret_cast<char*>(a.out + base);
    // 16-byte pieces (the usual case): two per thread at most, their places fixed
    constexpr int NP = 2;
    const bool vec = rc.lg == 1;
    int so[NP];        // shared-memory byte offset in a row
    unsigned go[NP];   // global byte offset in a row
    bool in[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        const int v = tid + k * static_cast<int>(blockDim.x), q = v >> 1, o = (v & 1) * 16;
        in[k] = v < 2 * Ny1 && o < rc.valid;
        so[k] = q * kMarchPitch + o;
        go[k] = static_cast<unsigned>(q * abytes + o);
    }
    auto fill = [&](int r) {  // row r into slot r % RF; one commit group per call
        if (r <= Nz) {
            char* d = reinterpret_cast<char*>(ring + (r % RF) * RS);
            const char* s = gin + static_cast<size_t>(r) * zs * sizeof(T);
            if (vec) {
#pragma unroll
                for (int k = 0; k < NP; ++k)
                    cp_async16_if(d + so[k], s + go[k], in[k]);
            } else {
                for (int v = tid; v < rc.n; v += blockDim.x) {
                    const int q = v >> rc.lg, o = (v & ((1 << rc.lg) - 1)) * rc.bytes;
                    if (o >= rc.valid) continue;
                    if (rc.lg == 2) cp_async_ca<8>(d + q * kMarchPitch + o, s + static_cast<size_t>(q) * abytes + o);
                    else cp_async_ca<4>(d + q * kMarchPitch + o, s + static_cast<size_t>(q) * abytes + o);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto drain = [&](int j) {  // output row j from its buffer
        const char* s = reinterpret_cast<const char*>(outb + (j % kMarchOut) * RS);
        char* d = gout + static_cast<size_t>(j) * zs * sizeof(T);
        if (vec) {
#pragma unroll
            for (int k = 0; k < NP; ++k)
                if (in[k]) *reinterpret_cast<float4*>(d + go[k]) = *reinterpret_cast<const float4*>(s + so[k]);
        } else {
            for (int v = tid; v < rc.n; v += blockDim.x) {
                const int q = v >> rc.lg, o = (v & ((1 << rc.lg) - 1)) * rc.bytes;
                if (o >= rc.valid) continue;
                const char* sp = s + q * kMarchPitch + o;
                char* dp = d + static_cast<size_t>(q) * abytes + o;
                if (rc.lg == 2) *reinterpret_cast<float2*>(dp) = *reinterpret_cast<const float2*>(sp);
                else *reinterpret_cast<float*>(dp) = *reinterpret_cast<const float*>(sp);
            }
        }
    };
    for (int r = 0; r < RF - 1; ++r) fill(r);

    // ---- this thread's line: angles e0, e1 of the chunk ----
    const int sl = tid % LW, line = tid / LW;
    auto omega = [&](int e, int axis) { return a.omega[2 * min(a0 + e, NA - 1) + axis]; };
    int e0 = 0, e1 = 0, found = 0;
    bool live = false;
    for (int e = 0; e < AC; e += W) {
        const bool second = W == 2 && a0 + e + 1 < NA;
        const bool paired = second && (omega(e, 0) < T(0)) == (omega(e + 1, 0) < T(0)) &&
                            (omega(e, 1) < T(0)) == (omega(e + 1, 1) < T(0));
        if (a0 + e < NA) {
            if (found++ == line) { e0 = e; e1 = paired ? e + 1 : e; live = true; }
            if (second && !paired && found++ == line) { e0 = e1 = e + 1; live = true; }
        }
    }
    // a float angle on its own still moves as the pair it belongs to; its half alone is stored
    const bool lone = LONE && e1 == e0;
    const int at0 = e0 & ~(W - 1);
    const bool dny = omega(e0, 0) < T(0), dnz = omega(e0, 1) < T(0);
    // Where registers are scarcest, z fluxes are kept doubled: the slope's half and sign
    // then need none (81 x 81 3.22 -> 3.15 ms per 400 groups, 62 x 62 unpaired 0.348 ->
    // 0.318; paired lines of two cells lose, 49 x 49 0.941 -> 0.982, and so does FP64,
    // 81 x 81 0.993 -> 1.010).
    constexpr bool kDouble = W == 2 && (YT >= 3 || LONE);
    V wy, wz;  // |omega_y| / dy (the line runs downwind), omega_z / dz (half of it for doubled fluxes)
    const T zs1 = kDouble ? T(0.5) : T(1);
    if constexpr (W == 2) {
        wy = make_float2(fabsf(omega(at0, 0) / a.dy), fabsf(omega(at0 + 1, 0) / a.dy));
        wz = make_float2(zs1 * (omega(at0, 1) / a.dz), zs1 * (omega(at0 + 1, 1) / a.dz));
    } else {
        wy = fabs(omega(e0, 0) / a.dy);
        wz = zs1 * (omega(e0, 1) / a.dz);
    }
    const V hz = LineOf<T>::both((dnz ? T(-1) : T(1)) * (kDouble ? T(1) : T(0.5)));
    // half the slope, kept where the difference towards higher y is at least eps
    const V hl = LineOf<T>::both(dny ? T(0.5) : T(0)), hr = LineOf<T>::both(dny ? T(0) : T(0.5));
    const V ndt = LineOf<T>::both(-a.dt), nhdt = LineOf<T>::both(T(-0.5) * a.dt);
    const T lo = a.preserve_sign ? -INFINITY : T(0);

    // ---- this thread's cells: positions YT sl + c - pad along the line ----
    const int nl = (Ny1 + YT - 1) / YT, pad = nl * YT - Ny1;
    const V mL = LineOf<T>::both(sl == 0 ? T(0) : T(1)), mR = LineOf<T>::both(sl == nl - 1 ? T(0) : T(1));
    int at[YT];  // shared-memory place of each cell's line value
    bool own[YT];  // its value is this thread's to store
#pragma unroll
    for (int c = 0; c < YT; ++c) {
        const int yl = YT * sl + c - pad, yc = min(max(yl, 0), Ny);
        own[c] = live && yl >= 0 && yl <= Ny;
        at[c] = (dny ? Ny - yc : yc) * PT + at0;
    }
    auto load = [&](const T* row, int c) -> V { return *reinterpret_cast<const V*>(row + at[c]); };

    // y-divergence (times |w| / dy) of the row x held by the line's lanes
    auto y_div = [&](const V (&x)[YT], V (&dy)[YT]) {
        V d[YT + 1], d2[YT + 1], k[YT + 1], g[YT];
        d[0] = vmul(vsub(x[0], lane_up(x[YT - 1], LW)), mL);
#pragma unroll
        for (int c = 1; c < YT; ++c) d[c] = vsub(x[c], x[c - 1]);
        d[YT] = vmul(vsub(lane_down(x[0], LW), x[YT - 1]), mR);
#pragma unroll
        for (int c = 0; c <= YT; ++c) {
            d2[c] = vadd(d[c], d[c]);
            k[c] = march_keep(d[c]);
        }
#pragma unroll
        for (int c = 0; c < YT; ++c)
            g[c] = vfma(march_limit(d[c], d2[c], d[c + 1], d2[c + 1]), vfma(k[c], hl, vmul(k[c + 1], hr)), x[c]);
        dy[0] = vmul(wy, vmul(vsub(g[0], lane_up(g[YT - 1], LW)), mL));
#pragma unroll
        for (int c = 1; c < YT; ++c) dy[c] = vmul(wy, vsub(g[c], g[c - 1]));
    };
    // z face of the cell with value x between the differences back and fwd
    auto z_face = [&](auto DNZc, V back, V fwd, V x) {
        if constexpr (kDouble) {
            constexpr int DNZ = decltype(DNZc)::value;
            const V k = march_keep(fwd), m = march_limit(back, vadd(back, back), fwd, vadd(fwd, fwd));
            return vfma(m, DNZ == 0 ? k : DNZ == 1 ? vneg(k) : vmul(k, hz), vadd(x, x));
        } else {
            return vfma(march_limit(back, vadd(back, back), fwd, vadd(fwd, fwd)), vmul(march_keep(fwd), hz), x);
        }
    };
    auto z_flat = [&](V x) { return kDouble ? vadd(x, x) : x; };  // the face of a cell without slope

    // Row r has landed, the rows of iteration r-1 are written and may leave.
    auto meet = [&](int r) {
        asm volatile("cp.async.wait_group %0;" ::"n"(RF - 2) : "memory");
        asm volatile("bar.sync 0;" ::: "memory");  // reached from each sign's march
        fill(r + RF - 1);
        if (r > 4) drain(r - 5);
    };
    auto march = [&](auto DNZc) {
        constexpr int DNZ = decltype(DNZc)::value, LAG = DNZ == 0 ? 1 : 2;
        V f1[YT], f2[YT], zd[YT], g1[YT], ez[YT];  // F(r-1), F(r-2); F(r-1) - F(r-2); G(r-2); G(r-2) - G(r-3)
        V p1[YT], pd[YT], gp[YT], ep[YT];          // P(i-1); P(i-1) - P(i-2); G'(i-2); G'(i-2) - G'(i-3)
        V t1[YT], t2[YT];                          // F - dt/2 (div F + y-part of div P) of rows i-1, i-2
        const V zero = LineOf<T>::both(T(0));
        meet(0);
#pragma unroll
        for (int c = 0; c < YT; ++c) {
            f1[c] = f2[c] = p1[c] = load(ring, c);
            g1[c] = gp[c] = z_flat(f1[c]);
            zd[c] = ez[c] = pd[c] = ep[c] = t1[c] = t2[c] = zero;
        }
        // one copy of the body for every row: the march is long straight-line code
#pragma unroll 1
        for (int r = 1; r <= Nz + 5; ++r) {
            meet(r);
            const int i = r - LAG, j = i - LAG;
            if (j > Nz) continue;  // the other sign's last rows
            V p[YT], t[YT];
            if (i <= Nz) {
                const T* row = ring + (min(r, Nz) % RF) * RS;  // the last row stays in its slot
                V dz[YT], x[YT], dy[YT];
#pragma unroll
                for (int c = 0; c < YT; ++c) {
                    x[c] = load(row, c);
                    const V d = vsub(x[c], f1[c]);
                    const V g = z_face(DNZc, zd[c], d, f1[c]);
                    const V e = vsub(g, g1[c]);
                    dz[c] = DNZ == 2 ? vselect(dnz, e, ez[c]) : e;
                    if (DNZ == 2) ez[c] = e;
                    g1[c] = g;
                    zd[c] = d;
                }
                V(&fi)[YT] = LAG == 1 ? f1 : f2;
                y_div(fi, dy);
#pragma unroll
                for (int c = 0; c < YT; ++c) {
                    // (rounded as in the kernels of these planes' other options, so the values
                    // are theirs: the tiled kernel's sum is one fma, the paired kernels' two
                    // operations; one scaled sum for p and t saved 2 % and differed by up to
                    // 4e-5 in a sum of signed values)
                    const V d = LONE || W == 1 ? vfma(wz, dz[c], dy[c]) : vadd(dy[c], vmul(wz, dz[c]));
                    p[c] = vmax(vfma(ndt, d, fi[c]), lo);
                    t[c] = vfma(nhdt, d, fi[c]);
                }
                y_div(p, dy);
#pragma unroll
                for (int c = 0; c < YT; ++c) {
                    t[c] = vfma(nhdt, dy[c], t[c]);
                    if (LAG == 2) f2[c] = f1[c];
                    f1[c] = x[c];
                }
            } else {  // the predictor repeats its last row
#pragma unroll
                for (int c = 0; c < YT; ++c) {
                    p[c] = p1[c];
                    t[c] = zero;
                }
            }
            if (i <= 0) {  // before and at the first predictor row: P(-1) = P(0)
#pragma unroll
                for (int c = 0; c < YT; ++c) {
                    pd[c] = ep[c] = zero;
                    p1[c] = p[c];
                    gp[c] = z_flat(p[c]);
                    if (LAG == 2) t2[c] = t1[c];
                    t1[c] = t[c];
                }
                continue;
            }
            T* out = outb + (j & (kMarchOut - 1)) * RS;
#pragma unroll
            for (int c = 0; c < YT; ++c) {
                const V d = vsub(p[c], p1[c]);
                const V g = z_face(DNZc, pd[c], d, p1[c]);
                const V e = vsub(g, gp[c]);
                const V dz = DNZ == 2 ? vselect(dnz, e, ep[c]) : e;
                const V v = vmax(vfma(nhdt, vmul(wz, dz), LAG == 1 ? t1[c] : t2[c]), lo);
                // (a row before the first lands in a slot that a later row takes)
                if constexpr (!LONE) {
                    store_if(reinterpret_cast<V*>(out + at[c]), v, own[c]);
                } else {
                    store_if(reinterpret_cast<V*>(out + at[c]), v, own[c] && !lone);
                    store_if(reinterpret_cast<T*>(out + at[c]) + (e0 & 1), (e0 & 1) ? v.y : v.x, own[c] && lone);
                }
                if (DNZ == 2) ep[c] = e;
                gp[c] = g;
                pd[c] = d;
                if (LAG == 2) t2[c] = t1[c];
                t1[c] = t[c];
                p1[c] = p[c];
            }
        }
    };
    const bool up = __all_sync(0xffffffffu, !dnz), down = __all_sync(0xffffffffu, dnz);
    if (up) march(std::integral_constant<int, 0>());
    else if (down) march(std::integral_constant<int, 1>());
    else march(std::integral_constant<int, 2>());
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Registers per thread: two, three or four cells' rows (the cap leaves five,
// four or three blocks of four warps per SM).
constexpr int march_regs(int yt) { return yt == 2 ? 96 : yt == 3 ? 128 : 168; }

template <typename T, int LW, int YT, bool LONE>
__global__ void __maxnreg__(march_regs(YT)) transport_march_kernel(TransportArgs<T> a, int n_chunks) {
    march_body<T, LW, YT, LONE>(a, n_chunks, blockIdx.x);
}

template <int LW, int YT>
__global__ void __maxnreg__(march_regs(YT)) transport_march_slots_kernel(const TransportArgs<float>* __restrict__ args,
                                                                       const int* __restrict__ begin, int nslots,
                                                                       int n_chunks) {
    const int s = find_slot(begin, nslots, blockIdx.x);
    const TransportArgs<float> a = args[s];
    march_body<float, LW, YT, false>(a, n_chunks, blockIdx.x - __ldg(begin + s));
}

// The (LW, YT) that leaves the fewest lanes without a position, of two or three
// positions per lane (three where both waste the same: fewer shuffles); four,
// with their registers, only for planes wider than 96.
struct MarchShape { int lw = 0, yt = 0; };
MarchShape march_shape(int Ny1) {
    MarchShape best{32, 4};
    int least = 1 << 30;
    for (int yt : {3, 2})
        for (int lw : {4, 8, 16, 32})
            if (lw * yt >= Ny1 && lw * yt < least) {
                least = lw * yt;
                best = {lw, yt};
            }
    return best;
}

size_t march_smem(int Ny1) { return static_cast<size_t>(kMarchRing + kMarchOut) * Ny1 * kMarchPitch; }
// (four lines at least: a row is two 16-byte pieces per thread then)
int march_threads(const MarchShape& m, int lines) { return (std::max(lines, 4) * m.lw + 31) / 32 * 32; }

template <typename F>
cudaError_t with_shape(const MarchShape& m, const F& f) {
#define BFPN_MARCH(l, y) \
    if (m.lw == l && m.yt == y) return f(std::integral_constant<int, l>(), std::integral_constant<int, y>())
    BFPN_MARCH(4, 2);
    BFPN_MARCH(8, 2);
    BFPN_MARCH(16, 2);
    BFPN_MARCH(32, 2);
    BFPN_MARCH(4, 3);
    BFPN_MARCH(8, 3);
    BFPN_MARCH(16, 3);
    BFPN_MARCH(32, 3);
    BFPN_MARCH(32, 4);
#undef BFPN_MARCH
    return cudaErrorNotSupported;
}

}  // namespace

// (a row's byte offsets stay within 32 bits)
bool transport_march_supported(int Ny, int NA) { return Ny >= 1 && Ny + 1 <= 128 && NA <= 1 << 20; }

int transport_march_chunks(int NA, size_t elem) {
    const int ac = kMarchChunk / static_cast<int>(elem);
    return (NA + ac - 1) / ac;
}

// Most lines any chunk holds (float: pairs of angles (2i, 2i+1) that share their signs count once).
int transport_march_lines(const double* omega, int NA, size_t elem) {
    const int ac = kMarchChunk / static_cast<int>(elem);
    int most = 0;
    for (int a0 = 0; a0 < NA; a0 += ac) {
        int n = 0;
        for (int g = a0; g < std::min(NA, a0 + ac); ++n) {
            const bool pair = elem == 4 && (g - a0) % 2 == 0 && g + 1 < std::min(NA, a0 + ac) &&
                              (omega[2 * g] < 0) == (omega[2 * g + 2] < 0) && (omega[2 * g + 1] < 0) == (omega[2 * g + 3] < 0);
            g += pair ? 2 : 1;
        }
        most = std::max(most, n);
    }
    return most;
}

template <typename T>
cudaError_t launch_transport_march(const TransportArgs<T>& a, int lines, cudaStream_t s) {
    if (!transport_march_supported(a.Ny, a.NA) || lines <= 0) return cudaErrorNotSupported;
    const MarchShape m = march_shape(a.Ny + 1);
    const int n_chunks = transport_march_chunks(a.NA, sizeof(T));
    const long long blocks = static_cast<long long>(a.Ng) * n_chunks;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    return with_shape(m, [&](auto lw, auto yt) {
        constexpr int L = decltype(lw)::value, Y = decltype(yt)::value;
        auto kern = transport_march_kernel<T, L, Y, false>;
        if constexpr (sizeof(T) == 4)  // some pair (2i, 2i+1) differs in its signs or lacks its second angle
            if (!a.pairs) kern = transport_march_kernel<T, L, Y, true>;
        const size_t smem = march_smem(a.Ny + 1);
        cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        kern<<<static_cast<unsigned>(blocks), march_threads(m, lines), smem, s>>>(a, n_chunks);
        return cudaGetLastError();
    });
}
template cudaError_t launch_transport_march<float>(const TransportArgs<float>&, int, cudaStream_t);
template cudaError_t launch_transport_march<double>(const TransportArgs<double>&, int, cudaStream_t);

cudaError_t launch_transport_march_slots(const TransportArgs<float>* args, const int* begin, int nslots, int blocks,
                                         int Ny, int NA, int lines, cudaStream_t s) {
    if (nslots <= 0 || blocks <= 0) return cudaSuccess;
    if (!transport_march_supported(Ny, NA) || lines <= 0) return cudaErrorNotSupported;
    const MarchShape m = march_shape(Ny + 1);
    const int n_chunks = transport_march_chunks(NA, 4);
    return with_shape(m, [&](auto lw, auto yt) {
        auto kern = transport_march_slots_kernel<decltype(lw)::value, decltype(yt)::value>;
        const size_t smem = march_smem(Ny + 1);
        cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(kern), smem);
        if (e != cudaSuccess) return e;
        kern<<<blocks, march_threads(m, lines), smem, s>>>(args, begin, nslots, n_chunks);
        return cudaGetLastError();
    });
}

}  // namespace bfpn
