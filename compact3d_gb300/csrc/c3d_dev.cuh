// c3d_dev.cuh -- device-side layout and line-solver primitives of the GB300 channel step.
//
// Layout in HBM.  Every 3-D field is plane-major: element (i, j, k) of a field lives at
//   ((j * N3M) + k) * N1M + i,   i in [0,N1M), k in [0,N3M), j in [0, N2]
// with i = I-1, k = K-1 and j = J of the reference's Fortran indices.  One x-z plane
// (N1M*N3M values) is contiguous, rows along x are contiguous, and the wall planes
// j = 0 and j = N2 are stored like interior planes.  The periodic x and z directions
// carry no halo: the kernels wrap indices.
//
// Compact (Pade) operators.  The reference solves constant-coefficient cyclic systems
//   a x_{i-1} + b x_i + a x_{i+1} = d_i                 (CTDMA11/33, CTDMA1J/3I)
// by bordered LU.  With beta = b/a and r the root of r^2 + beta r + 1 = 0 with |r| < 1,
//   tridiag(a, b, a) = (-a/r) (1 - r S)(1 - r S^-1)      (S = cyclic shift)
// so x = s * B(F(d)) with s = -r/a, F: y_i = d_i + r y_{i-1} and B: z_i = y_i + r z_{i+1},
// both cyclic.  The kernels evaluate these two first-order recurrences:
//   * along x (contiguous rows): one warp per row (or, for short rows, a segment of 8 or 16
//     lanes per row), every lane owns C consecutive points, and the cyclic carries between
//     lanes come from shuffle scans of affine maps (FP32 and double-float: xsolve_full,
//     xsolve_general) or from doubling round the ring of lanes until the next power of r^C
//     is below rounding (FP64: xsolve_ring);
//   * along z (strided columns): one thread per (column, segment of L points).  FP32 and
//     double-float start each recurrence M points early (zsweep), M chosen so |r|^M is below
//     the working precision's rounding unit; FP64, and FP32 where the schedule says so, joins
//     the segments of a line through shared memory (zjoin), which reach as far.
// The result equals the reference's bordered-LU solution to rounding.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

namespace c3d {

constexpr unsigned FULL = 0xffffffffu;

// Coefficients of one constant-coefficient cyclic operator in a given precision.
template <typename R>
struct Cyc {
    R r;      // root of r^2 + (b/a) r + 1 = 0, |r| < 1
    R s;      // output scale -r/a
    int m;    // warm-up length for segment solves
};

// Geometry and constants handed to every kernel by value.
struct Geo {
    int n1m, n2m, n3m, n2;   // cells; n2 = N2 = n2m + 1
    int np;                  // n1m * n3m (plane)
    long long nf;            // (n2 + 1) * np (field)
    int n1h;                 // n1m/2 + 1 (half spectrum along x)
    double dx1, dx3, dx1q, dx3q, re, alx, aly, alz, vol;
    // y metrics indexed by Fortran J (arrays of n2+1 values, entry 0 = DY(0) etc.);
    // hz = HP+HM-HC and dyz = DYP+DYM-DYC are zero up to rounding (used by the mixed form)
    const double *dy, *h, *hp, *hc, *hm, *dyp, *dyc, *dym, *hz, *dyz;
};

__host__ __device__ inline long long fidx(const Geo &g, int i, int j, int k) {
    return ((long long)j * g.n3m + k) * g.n1m + i;
}

// ---------------------------------------------------------------------------------
// x direction: warp per row, lane chunks of C points, P = N1M / C active lanes (the
// lane_* helpers; the kernels' segmented forms use sprev/snext/xsolve with a width).
// ---------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T lane_prev(T last, int lane, int P) {
    int src = (lane == 0) ? P - 1 : lane - 1;
    return __shfl_sync(FULL, last, src);
}
template <typename T>
__device__ __forceinline__ T lane_next(T first, int lane, int P) {
    int src = (lane + 1 >= P) ? 0 : lane + 1;
    return __shfl_sync(FULL, first, src);
}

// Double-float value hi + lo (about 48 significant bits) made of FP32 operations: error-
// free two-sum (Knuth) and FMA-based two-product.  The line solvers are templates on the
// value type, so the same recurrences run in double-float where a result must be
// accurate well below FP32 rounding (the residual of the pressure refinement).
struct dfl {
    float h, l;
    __host__ __device__ dfl() : h(0.f), l(0.f) {}
    __host__ __device__ dfl(float x) : h(x), l(0.f) {}
    __host__ __device__ dfl(float a, float b) : h(a), l(b) {}
    static __host__ dfl from(double x) {
        float a = (float)x;
        return dfl(a, (float)(x - (double)a));
    }
};
__device__ __forceinline__ dfl dfl_norm(float s, float e) {
    float h = s + e;
    return dfl(h, e - (h - s));
}
__device__ __forceinline__ dfl operator+(dfl a, dfl b) {
    float s = a.h + b.h, v = s - a.h;
    float e = (a.h - (s - v)) + (b.h - v);
    return dfl_norm(s, e + (a.l + b.l));
}
__device__ __forceinline__ dfl operator-(dfl a, dfl b) { return a + dfl(-b.h, -b.l); }
__device__ __forceinline__ dfl operator*(dfl a, dfl b) {
    float p = a.h * b.h;
    float e = fmaf(a.h, b.h, -p);
    e = fmaf(a.h, b.l, e);
    e = fmaf(a.l, b.h, e);
    return dfl_norm(p, e);
}
__device__ __forceinline__ dfl operator/(dfl a, dfl b) {
    float q1 = a.h / b.h;
    dfl r = a - dfl(q1) * b;
    float q2 = r.h / b.h;
    dfl q = dfl_norm(q1, q2);
    r = a - q * b;
    return q + dfl(r.h / b.h);
}
__device__ __forceinline__ dfl &operator+=(dfl &a, dfl b) { return a = a + b; }
__device__ __forceinline__ dfl &operator*=(dfl &a, dfl b) { return a = a * b; }

// Warp shuffles for every value type of the line solvers.
// Shuffles within segments of w lanes (w = 32: the whole warp); lane indexes and
// offsets are relative to the segment.
__device__ __forceinline__ double shfl_up(double v, int d, int w = 32) { return __shfl_up_sync(FULL, v, d, w); }
__device__ __forceinline__ float shfl_up(float v, int d, int w = 32) { return __shfl_up_sync(FULL, v, d, w); }
__device__ __forceinline__ dfl shfl_up(dfl v, int d, int w = 32) {
    return dfl(__shfl_up_sync(FULL, v.h, d, w), __shfl_up_sync(FULL, v.l, d, w));
}
__device__ __forceinline__ double shfl_down(double v, int d, int w = 32) { return __shfl_down_sync(FULL, v, d, w); }
__device__ __forceinline__ float shfl_down(float v, int d, int w = 32) { return __shfl_down_sync(FULL, v, d, w); }
__device__ __forceinline__ dfl shfl_down(dfl v, int d, int w = 32) {
    return dfl(__shfl_down_sync(FULL, v.h, d, w), __shfl_down_sync(FULL, v.l, d, w));
}
__device__ __forceinline__ double shfl_idx(double v, int s, int w = 32) { return __shfl_sync(FULL, v, s, w); }
__device__ __forceinline__ float shfl_idx(float v, int s, int w = 32) { return __shfl_sync(FULL, v, s, w); }
__device__ __forceinline__ dfl shfl_idx(dfl v, int s, int w = 32) {
    return dfl(__shfl_sync(FULL, v.h, s, w), __shfl_sync(FULL, v.l, s, w));
}

// 1 - x rounds to 1 (so that y / (1 - x) is y exactly) for |x| below half an ulp of 1.
__device__ __forceinline__ bool below_half_ulp(float x) { return fabsf(x) < 0x1p-25f; }
template <typename R>
__device__ __forceinline__ bool below_half_ulp(R) { return false; }

// x^L for a compile-time L by repeated squaring.
template <int L, typename R>
__device__ __forceinline__ R rpow(R x) {
    if constexpr (L == 1) return x;
    else if constexpr (L % 2 == 0) return rpow<L / 2>(x * x);
    else return x * rpow<L / 2>(x * x);
}

// xsolve for a row whose every lane holds a chunk (P = W): every lane's chunk multiplier is
// r^C, so the scans combine with the constant powers r^(C 2^b) (one shuffle and one
// multiply-add per level), the chunk sweeps carry no multiplier, and the cyclic closure
// y / (1 - r^(C W)) needs no division once r^(C W) is below half an ulp.  The powers are
// formed with the same products, in the same order, as the general form forms its
// multipliers at each level.
template <int W, typename R, int C>
__device__ __forceinline__ void xsolve_full(R (&x)[C], int lane, const Cyc<R> &c) {
    constexpr int LW = W == 32 ? 5 : W == 16 ? 4 : W == 8 ? 3 : 2;
    const R r = c.r;
    R pw[LW + 1];
    {
        R m = R(1);
#pragma unroll
        for (int t = 0; t < C; ++t) m *= r;
        pw[0] = m;
#pragma unroll
        for (int b = 0; b < LW; ++b) pw[b + 1] = pw[b] * pw[b];
    }
    R ml = R(1), mr = R(1);   // r^(C lane) and r^(C (W - 1 - lane))
#pragma unroll
    for (int b = 0; b < LW; ++b) {
        if ((lane >> b) & 1) ml = ml * pw[b];
        if (((W - 1 - lane) >> b) & 1) mr = mr * pw[b];
    }
    const bool exact1 = below_half_ulp(pw[LW]);
    R y = R(0);
#pragma unroll
    for (int t = 0; t < C; ++t) y = x[t] + r * y;
    R e = y;
#pragma unroll
    for (int b = 0; b < LW; ++b) {
        const int off = 1 << b;
        const R ep = shfl_up(e, off, W);
        if (lane >= off) e = e + pw[b] * ep;
    }
    {
        const R et = shfl_idx(e, W - 1, W);
        const R y0 = exact1 ? et : et / (R(1) - pw[LW]);
        const R ex = shfl_up(e, 1, W);
        y = (lane == 0) ? y0 : ex + ml * y0;
    }
#pragma unroll
    for (int t = 0; t < C; ++t) {
        y = x[t] + r * y;
        x[t] = y;
    }
    R z = R(0);
#pragma unroll
    for (int t = C - 1; t >= 0; --t) z = x[t] + r * z;
    e = z;
#pragma unroll
    for (int b = 0; b < LW; ++b) {
        const int off = 1 << b;
        const R en = shfl_down(e, off, W);
        if (lane + off < W) e = e + pw[b] * en;
    }
    {
        const R e0 = shfl_idx(e, 0, W);
        const R z0 = exact1 ? e0 : e0 / (R(1) - pw[LW]);
        const R en1 = shfl_down(e, 1, W);
        z = (lane == W - 1) ? z0 : en1 + mr * z0;
    }
    const R s = c.s;
#pragma unroll
    for (int t = C - 1; t >= 0; --t) {
        z = x[t] + r * z;
        x[t] = s * z;
    }
}

// |x| < 2^-56 by its exponent (an integer test: FP64 instructions are what bounds the FP64 form).
__device__ __forceinline__ bool negligible(double x) { return (__double2hiint(x) & 0x7ff00000) < (1023 - 56) << 20; }

// Decaying roots r of 1 + OP r + r^2 for the compact operators (1, OP, 1), known at compile
// time, so that the FP64 solves' powers of r are constants.  OP = 0: the root is the caller's
// (the Crank-Nicolson factors').
template <int OP> struct Root { static constexpr double r = 0.0; };
template <> struct Root<6> { static constexpr double r = -0.171572875253809902396622551580603842860; };    // -3 + sqrt(8)
template <> struct Root<10> { static constexpr double r = -0.101020514433643803605431850588217216068; };   // -5 + sqrt(24)
template <> struct Root<22> { static constexpr double r = -0.04554884989667773086060434398395732094; };    // -11 + sqrt(120)
__host__ __device__ constexpr double cpow(double x, int n) {
    double p = 1.0;
    for (int i = 0; i < n; ++i) p *= x;
    return p;
}
__host__ __device__ constexpr bool cnegligible(double x) { return (x < 0 ? -x : x) < 1.0 / 72057594037927936.0; }   // 2^-56
// Points after which r^n is negligible, at most C.
template <int OP, int C>
__host__ __device__ constexpr int croot_len() {
    if (OP == 0) return C;
    int n = 1;
    while (n < C && !cnegligible(cpow(Root<OP>::r, n))) ++n;
    return n;
}
// The root of a z solve's operator: the constant in FP64, the argument in FP32.
template <int OP> __device__ __forceinline__ double zroot(double) { return Root<OP>::r; }
template <int OP> __device__ __forceinline__ float zroot(float r) { return r; }

// What enters each lane's chunk in the FP64 recurrences of one direction: e = the chunk's own
// sum, m = r^C.  The sums of the lanes before it (DIR -1) or after it (DIR +1) are added over
// a ring of P lanes by doubling, each level covering twice the lanes, and the levels stop
// where the next factor r^(C 2^b) is below the rounding unit: for the compact operators after
// three at most with chunks of 4 points or more (r^16 is 2^-41 for (1,6,1), 2^-53 for (1,10,1),
// 2^-71 for (1,22,1)), two with chunks of 8 (a scan over 32 lanes has five).  A level
// that runs round the ring adds the next period of the periodic sum, so there is no closure.
// LV levels at most: 12 reach 4096 chunks; more, or a bound that a launch could change, cost
// xB 4% (192 x 128 x 144 points, 291 -> 304 us), so CN roots past that take their own instance.
template <int W, int DIR, int LV>
__device__ __forceinline__ double ring_carry(double e, double m, int lane, int P) {
    int off = 1;
    for (int b = 0; b < LV && !negligible(m); ++b) {
        int src = DIR < 0 ? lane - off : lane + off;
        if (DIR < 0 && src < 0) src += P;
        if (DIR > 0 && src >= P) src -= P;
        e = e + m * shfl_idx(e, src, W);
        m *= m;
        off *= 2;
        if (off >= P) off -= P;
    }
    return shfl_idx(e, DIR < 0 ? (lane == 0 ? P - 1 : lane - 1) : (lane + 1 >= P ? 0 : lane + 1), W);
}

// The same with a compile-time root: the levels and their factors are constants.
template <int W, int DIR, int OP, int C, int B = 0>
__device__ __forceinline__ double ring_carry_op(double e, int lane, int P, int off = 1) {
    constexpr double m = cpow(Root<OP>::r, C << B);
    if constexpr (!cnegligible(m) && B < 6) {
        int src = DIR < 0 ? lane - off : lane + off;
        if (DIR < 0 && src < 0) src += P;
        if (DIR > 0 && src >= P) src -= P;
        e = e + m * shfl_idx(e, src, W);
        off *= 2;
        if (off >= P) off -= P;
        return ring_carry_op<W, DIR, OP, C, B + 1>(e, lane, P, off);
    } else {
        return shfl_idx(e, DIR < 0 ? (lane == 0 ? P - 1 : lane - 1) : (lane + 1 >= P ? 0 : lane + 1), W);
    }
}

// FP64 solve on lane chunks without the scale s (B(F(d)); callers fold s into their
// constants): two sweeps of C multiply-adds each way and the ring carries.  Against scans
// over all lanes with per-lane multipliers and a closure it executes about half the FP64
// instructions, and the FP64 pipe bounds the FP64 x passes (192 x 128 x 144 points: xA's
// pieces 409, 312, 222 -> 264, 240, 152 us, xB 529 -> 353, xC 337 -> 303, xD 279 -> 244).
// With a compile-time root a chunk's sum takes only its last points that reach the next chunk.
template <int W, int OP, int LV = 12, int C>
__device__ __forceinline__ void xsolve_ring(double (&x)[C], int lane, int P, const Cyc<double> &c) {
    constexpr int T = croot_len<OP, C>();
    const double r = OP ? Root<OP>::r : c.r, m = OP ? 0.0 : rpow<C>(r);
    double y = x[C - T];
#pragma unroll
    for (int t = C - T + 1; t < C; ++t) y = x[t] + r * y;
    if constexpr (OP != 0) y = ring_carry_op<W, -1, OP, C>(y, lane, P);
    else y = ring_carry<W, -1, LV>(y, m, lane, P);
#pragma unroll
    for (int t = 0; t < C; ++t) {
        y = x[t] + r * y;
        x[t] = y;
    }
    double z = x[T - 1];
#pragma unroll
    for (int t = T - 2; t >= 0; --t) z = x[t] + r * z;
    if constexpr (OP != 0) z = ring_carry_op<W, +1, OP, C>(z, lane, P);
    else z = ring_carry<W, +1, LV>(z, m, lane, P);
#pragma unroll
    for (int t = C - 1; t >= 0; --t) {
        z = x[t] + r * z;
        x[t] = z;
    }
}

// The general form of a segment with idle lanes (P < W).
template <int W, typename R, int C>
__device__ __forceinline__ void xsolve_general(R (&x)[C], int lane, int P, const Cyc<R> &c) {
    const bool act = lane < P;
    const R r = c.r;
    R y = R(0), m = R(1);
#pragma unroll
    for (int t = 0; t < C; ++t) {
        y = x[t] + r * y;
        m *= r;
    }
    R e = act ? y : R(0);
    if (!act) m = R(1);
#pragma unroll
    for (int off = 1; off < W; off <<= 1) {
        R ep = shfl_up(e, off, W), mp = shfl_up(m, off, W);
        if (lane >= off) {
            e = e + m * ep;
            m = m * mp;
        }
    }
    {
        R et = shfl_idx(e, W - 1, W), mt = shfl_idx(m, W - 1, W);
        R y0 = et / (R(1) - mt);
        R ex = shfl_up(e, 1, W), mx = shfl_up(m, 1, W);
        y = (lane == 0) ? y0 : ex + mx * y0;
    }
#pragma unroll
    for (int t = 0; t < C; ++t) {
        y = x[t] + r * y;
        x[t] = y;
    }
    R z = R(0);
    m = R(1);
#pragma unroll
    for (int t = C - 1; t >= 0; --t) {
        z = x[t] + r * z;
        m *= r;
    }
    e = act ? z : R(0);
    if (!act) m = R(1);
#pragma unroll
    for (int off = 1; off < W; off <<= 1) {
        R en = shfl_down(e, off, W), mn = shfl_down(m, off, W);
        if (lane + off < W) {
            e = e + m * en;
            m = m * mn;
        }
    }
    {
        R e0 = shfl_idx(e, 0, W), m0 = shfl_idx(m, 0, W);
        R z0 = e0 / (R(1) - m0);
        R en1 = shfl_down(e, 1, W), mn1 = shfl_down(m, 1, W);
        z = (lane == W - 1) ? z0 : en1 + mn1 * z0;
    }
    const R s = c.s;
#pragma unroll
    for (int t = C - 1; t >= 0; --t) {
        z = x[t] + r * z;
        x[t] = s * z;
    }
}

// Cyclic solve on a row held as lane chunks x[0..C) by a segment of W lanes (lane =
// the lane within the segment; W = 32: one row per warp, W < 32: 32/W rows per warp,
// every segment of the warp calling together); in place, returns s*B(F(x)).  FP64 takes the
// ring form; otherwise P = W takes the constant-multiplier form above and P < W (idle lanes)
// the general one.
template <int W = 32, int OP = 0, typename R, int C>
__device__ __forceinline__ void xsolve(R (&x)[C], int lane, int P, const Cyc<R> &c) {
    static_assert(W == 4 || W == 8 || W == 16 || W == 32, "row segments of 4, 8, 16 or 32 lanes");
    if constexpr (std::is_same<R, double>::value) {
        xsolve_ring<W, OP>(x, lane, P, c);
#pragma unroll
        for (int t = 0; t < C; ++t) x[t] *= c.s;
        return;
    } else if (P == W) {
        xsolve_full<W>(x, lane, c);
        return;
    }
    if constexpr (!std::is_same<R, double>::value) xsolve_general<W>(x, lane, P, c);
}

// The same with the FP64 scale left to the caller: xfold(f, c) is the factor f of a
// right-hand side with the operator's scale folded in (FP64) or f itself.
template <int W = 32, int OP = 0, int LV = 12, typename R, int C>
__device__ __forceinline__ void xsolve_f(R (&x)[C], int lane, int P, const Cyc<R> &c) {
    if constexpr (std::is_same<R, double>::value) xsolve_ring<W, OP, LV>(x, lane, P, c);
    else xsolve<W>(x, lane, P, c);
}
__device__ __forceinline__ double xfold(double f, const Cyc<double> &c) { return f * c.s; }
__device__ __forceinline__ float xfold(float f, const Cyc<float> &) { return f; }

// Lane-chunk load/store of one row (row pointer + lane*C).  Inactive lanes are skipped.
template <int C>
__device__ __forceinline__ void row_load(double (&v)[C], const double *__restrict__ row, int lane, int P) {
    if (lane < P) {
        const double *p = row + lane * C;
        if constexpr (C % 2 == 0) {
#pragma unroll
            for (int t = 0; t < C; t += 2) {
                double2 q = __ldg(reinterpret_cast<const double2 *>(p + t));
                v[t] = q.x;
                v[t + 1] = q.y;
            }
        } else {
#pragma unroll
            for (int t = 0; t < C; ++t) v[t] = __ldg(p + t);
        }
    } else {
#pragma unroll
        for (int t = 0; t < C; ++t) v[t] = 0.0;
    }
}
template <int C>
__device__ __forceinline__ void row_load(float (&v)[C], const float *__restrict__ row, int lane, int P) {
    if (lane < P) {
        const float *p = row + lane * C;
        if constexpr (C % 4 == 0) {
#pragma unroll
            for (int t = 0; t < C; t += 4) {
                float4 q = __ldg(reinterpret_cast<const float4 *>(p + t));
                v[t] = q.x; v[t + 1] = q.y; v[t + 2] = q.z; v[t + 3] = q.w;
            }
        } else if constexpr (C % 2 == 0) {
#pragma unroll
            for (int t = 0; t < C; t += 2) {
                float2 q = __ldg(reinterpret_cast<const float2 *>(p + t));
                v[t] = q.x; v[t + 1] = q.y;
            }
        } else {
#pragma unroll
            for (int t = 0; t < C; ++t) v[t] = __ldg(p + t);
        }
    } else {
#pragma unroll
        for (int t = 0; t < C; ++t) v[t] = 0.f;
    }
}
template <typename T, int C>
__device__ __forceinline__ void row_store(T *__restrict__ row, const T (&v)[C], int lane, int P) {
    if (lane < P) {
        T *p = row + lane * C;
#pragma unroll
        for (int t = 0; t < C; ++t) p[t] = v[t];
    }
}

// ---------------------------------------------------------------------------------
// z direction: thread per (column, segment of L points) with warm-up M.
// D(k) is a functor returning the right-hand side at wrapped index k in [0,n).
// ---------------------------------------------------------------------------------
__device__ __forceinline__ int wrapi(int q, int n) {
    while (q < 0) q += n;
    while (q >= n) q -= n;
    return q;
}

template <typename R, int L, typename F>
__device__ __forceinline__ void zseg(R (&out)[L], int k0, int n, const Cyc<R> &c, F D) {
    const R r = c.r;
    R y = R(0);
    int kk = wrapi(k0 - c.m, n);
    for (int q = 0; q < c.m; ++q) {
        y = D(kk) + r * y;
        kk = (kk + 1 == n) ? 0 : kk + 1;
    }
    R ys[L];
#pragma unroll
    for (int t = 0; t < L; ++t) {
        y = D(kk) + r * y;
        ys[t] = y;
        kk = (kk + 1 == n) ? 0 : kk + 1;
    }
    R acc = R(0), pw = R(1);
    for (int q = 0; q < c.m; ++q) {
        y = D(kk) + r * y;
        acc = acc + pw * y;
        pw *= r;
        kk = (kk + 1 == n) ? 0 : kk + 1;
    }
    R z = acc;
    const R s = c.s;
#pragma unroll
    for (int t = L - 1; t >= 0; --t) {
        z = ys[t] + r * z;
        out[t] = s * z;
    }
}

// Several cyclic solves along one column in a single sweep.  The functor f walks the
// column once, in order, from position k0 - M (wrapped): f.start(k) positions it and
// f.next(d) returns the NR right-hand sides at the current position and advances, so it
// can keep a sliding window of the stencil inputs in registers and load one new value per
// position.  Recurrence q uses root r[q] and scale s[q]; M is the largest warm-up needed.
template <typename R, int L, int M, int NR, typename F>
__device__ __forceinline__ void zsweep(R (&out)[NR][L], int k0, int n, const R (&r)[NR], const R (&s)[NR], F &f) {
    f.start(wrapi(k0 - M, n));
    R y[NR], d[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) y[q] = R(0);
#pragma unroll
    for (int t = 0; t < M; ++t) {
        f.next(d);
#pragma unroll
        for (int q = 0; q < NR; ++q) y[q] = d[q] + r[q] * y[q];
    }
    R ys[NR][L];
#pragma unroll
    for (int t = 0; t < L; ++t) {
        f.next(d);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            y[q] = d[q] + r[q] * y[q];
            ys[q][t] = y[q];
        }
    }
    R acc[NR], pw[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) { acc[q] = R(0); pw[q] = R(1); }
#pragma unroll
    for (int t = 0; t < M; ++t) {
        f.next(d);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            y[q] = d[q] + r[q] * y[q];
            acc[q] = acc[q] + pw[q] * y[q];
            pw[q] *= r[q];
        }
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        R z = acc[q];
#pragma unroll
        for (int t = L - 1; t >= 0; --t) {
            z = ys[q][t] + r[q] * z;
            out[q][t] = s[q] * z;
        }
    }
}

// Thread layout of a joined z pass (zjoin): the block's threads are `cols` columns
// (consecutive threads) times the nseg = N3M / L segments of a line.
struct ZJ {
    int cols, lx, seg, nseg;
};

// Cyclic solve of NR recurrences on z lines whose segments of L points are all in one
// block: each thread reads its own segment's right-hand sides once (f.next), the state
// entering a segment is joined from the segments before it (after it, backward) through
// shared memory, and the sweeps run with it, so a solve costs 2 L multiply-adds each way
// and no warm-up (a warm-up of M points reads M + L + M points and evaluates their
// right-hand sides for L results).  A segment multiplies what enters it by r^L, so only
// the K = ceil(M / L) nearest segments reach it above the precision's rounding unit
// (|r|^M below it, as for the warm-ups).  No scale: out is B(F(d)); the caller folds s
// into its constants.  sh holds 2 NH blockDim.x values, NH >= NR; every thread of the
// block calls it (it synchronises the block twice; calls with the same NH may follow each
// other directly, because a call's two exchanges use different halves of sh).
template <typename R, int L, int M, int NR, int NH, typename F>
__device__ __forceinline__ void zjoin(R (&out)[NR][L], int k0, const R (&r)[NR], F &f, const ZJ &z, R *sh) {
    constexpr int K = (M + L - 1) / L;
    const int nt = z.cols * z.nseg;
    f.start(k0);
    R y[NR], d[NR], rl[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        y[q] = R(0);
        rl[q] = rpow<L>(r[q]);
    }
#pragma unroll
    for (int t = 0; t < L; ++t) {
        f.next(d);
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            out[q][t] = d[q];
            y[q] = d[q] + r[q] * y[q];
        }
    }
#pragma unroll
    for (int q = 0; q < NR; ++q) sh[q * nt + z.seg * z.cols + z.lx] = y[q];
    __syncthreads();
    int p[K];
    p[0] = z.seg == 0 ? z.nseg - 1 : z.seg - 1;
#pragma unroll
    for (int k = 1; k < K; ++k) p[k] = p[k - 1] == 0 ? z.nseg - 1 : p[k - 1] - 1;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const R *v = sh + q * nt + z.lx;
        R c = v[p[K - 1] * z.cols];
#pragma unroll
        for (int k = K - 2; k >= 0; --k) c = v[p[k] * z.cols] + rl[q] * c;
#pragma unroll
        for (int t = 0; t < L; ++t) {
            c = out[q][t] + r[q] * c;
            out[q][t] = c;
        }
        R b = R(0);
#pragma unroll
        for (int t = L - 1; t >= 0; --t) b = out[q][t] + r[q] * b;
        y[q] = b;
    }
    sh += NH * nt;
#pragma unroll
    for (int q = 0; q < NR; ++q) sh[q * nt + z.seg * z.cols + z.lx] = y[q];
    __syncthreads();
    p[0] = z.seg + 1 == z.nseg ? 0 : z.seg + 1;
#pragma unroll
    for (int k = 1; k < K; ++k) p[k] = p[k - 1] + 1 == z.nseg ? 0 : p[k - 1] + 1;
#pragma unroll
    for (int q = 0; q < NR; ++q) {
        const R *v = sh + q * nt + z.lx;
        R c = v[p[K - 1] * z.cols];
#pragma unroll
        for (int k = K - 2; k >= 0; --k) c = v[p[k] * z.cols] + rl[q] * c;
#pragma unroll
        for (int t = L - 1; t >= 0; --t) {
            c = out[q][t] + r[q] * c;
            out[q][t] = c;
        }
    }
}

// Warm-up lengths M = ceil(log(tol)/log|r|) of the Pade operators (1,6,1), (1,10,1),
// (1,22,1) and the Crank-Nicolson operators (b/a > 10 while DT DX^2 / (2 RE) < 1/12, so MCN is
// the length of (1,10,1)): tol = 1e-17 in FP64, 3e-8 in FP32.
template <typename R> struct WM;
template <> struct WM<double> { static constexpr int M6 = 23, M22 = 13, MCN = 18; };
template <> struct WM<float> { static constexpr int M6 = 10, M22 = 6, MCN = 8; };

}  // namespace c3d
