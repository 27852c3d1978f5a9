// c3d_zcols.cuh -- what the z-column passes share: thread coordinates, the two forms of the
// line solve, batched column loads, and the launch shape of the joined form.
#pragma once
#include "c3d_kern.cuh"

namespace c3d {

__device__ __forceinline__ int znext(int k, int n) { return (k + 1 == n) ? 0 : k + 1; }
__device__ __forceinline__ int zprev(int k, int n) { return (k == 0) ? n - 1 : k - 1; }

// Most threads of a joined block (128 or 170 registers each).
template <typename R, int L>
__host__ __device__ constexpr int zjt() {
    return sizeof(R) == 8 && L > 8 ? 384 : 512;
}

// Thread coordinates and the line solve of the two z-pass forms.  MODE 0: one thread per
// (i, segment of L points, plane) with warm-up recurrences (zsweep).  MODE 1: a block holds
// whole lines of consecutive columns (i fastest, then the plane), one thread per segment,
// and joins the segments through shared memory (zjoin); threads past the last column
// compute the last one again and store nothing (zc.act).
struct ZCo {
    int i, j, k0;
    bool act;
    ZJ z;
};
template <int L, int MODE>
__device__ __forceinline__ bool zcoords(const Blk blk, const Geo &g, int jlo, ZCo &c) {
    if constexpr (MODE == 1) {
        c.z.nseg = g.n3m / L;
        c.z.cols = (int)blockDim.x / c.z.nseg;
        const int sh = 31 - __clz(c.z.cols);   // cols is a power of 2
        c.z.seg = (int)threadIdx.x >> sh;
        c.z.lx = (int)threadIdx.x & (c.z.cols - 1);
        const unsigned n1 = (unsigned)g.n1m, tot = (unsigned)(g.n2m - jlo + 1) * n1;
        unsigned q = blk.x * (unsigned)c.z.cols + (unsigned)c.z.lx;
        c.act = q < tot;
        if (!c.act) q = tot - 1;
        const unsigned jq = q / n1;
        c.i = (int)(q - jq * n1);
        c.j = jlo + (int)jq;
        c.k0 = c.z.seg * L;
        return true;
    } else {
        c.act = zcoord<L>(blk, g, jlo, c.i, c.j, c.k0);
        return c.act;
    }
}
// MODE 0: out = s B(F(d)) as the reference's solve; MODE 1: out = B(F(d)), the caller's
// constants carry s and the right-hand side's factor (zfold).
template <typename R, int L, int M, int NR, int MODE, int NH = NR, typename F>
__device__ __forceinline__ void zsolve(R (&out)[NR][L], const ZCo &c, int n, const R (&r)[NR], const R (&s)[NR], F &f) {
    if constexpr (MODE == 1) {
        extern __shared__ __align__(16) unsigned char zsh_raw[];
        zjoin<R, L, M, NR, NH>(out, c.k0, r, f, c.z, reinterpret_cast<R *>(zsh_raw));
    } else {
        zsweep<R, L, M, NR>(out, c.k0, n, r, s, f);
    }
}
// The factor of a walker's right-hand side (1 in MODE 1) and of a solve's result (f s in MODE 1).
template <int MODE, typename R>
__device__ __forceinline__ R zrhs(R f) { return MODE == 1 ? R(1) : f; }
template <int MODE, typename R>
__device__ __forceinline__ R zfold(R f, R s) { return MODE == 1 ? f * s : R(1); }

// What a pass reads and updates beside its solve is loaded ZTB positions at a time before
// the first of them is stored: the compiler may not move a load above a store that could
// alias it, and one position at a time is a chain of L memory latencies per thread.
// 384 x 256 x 384 points, mixed form: zA_u 194 -> 132 us, zA_wp 214 -> 184, zA_v 220 -> 165,
// zB 234 -> 191, zE 510 -> 430 (6.9 TB/s of algorithmic bytes).
template <int L> constexpr int ztb() { return L < 8 ? L : L % 8 == 0 ? 8 : 6; }
template <int B, typename T>
__device__ __forceinline__ void zload(T (&v)[B], const T *col, int k, int s) {
#pragma unroll
    for (int t = 0; t < B; ++t) v[t] = col[(k + t) * s];
}

// Columns per block of a joined pass over ncol columns with segments of L points, or 0 when a
// line has too many segments for a block.  FP64: the fewest of 8, 16, 32 that give 96 threads
// (small blocks overlap one block's loads with another's FP64 arithmetic: 192 x 128 x 144
// points, L = 12, the seven z sweeps 0.84 ms at 8 columns, 0.89 at 16, 0.98 at 32), and 8 while
// the blocks are fewer than two per SM (32 x 24 x 48 points have 24 blocks at 32 columns: every
// warp instruction holds its SM's FP64 pipe for 16 cycles, so idle SMs cost most).  FP32: the
// most up to 32 that a block holds (whole sectors of 4-byte rows).
template <typename R, int L>
inline int zjoin_cols(int n3m, long long ncol) {
    const int nseg = n3m / L, most = zjt<R, L>();
    if (n3m % L != 0 || 8 * nseg > most) return 0;
    int cols = 8;
    if (sizeof(R) == 8) while (cols < 32 && cols * nseg < 96 && ncol >= 304LL * 2 * cols) cols *= 2;
    else while (cols < 32 && 2 * cols * nseg <= most) cols *= 2;
    return cols;
}

// The segment length of a joined pass over N3M points, 0 when no length fits (the warm-up
// form runs).  FP64, whatever the schedule: 12 where it divides N3M, else 8, else 16 (long
// lines).  Against 12 at N3M = 144, 8 and 16 cost 12% and 9% more over the seven z sweeps;
// at N3M = 64, 16 costs 9% more than 8.  FP32 (schedule 0): 8, 12 or 16, at most 32 segments.
template <typename R>
inline int zjoin_len(int n3m) {
    if constexpr (sizeof(R) == 8) {
        if (zjoin_cols<R, 12>(n3m, 0)) return 12;
        if (zjoin_cols<R, 8>(n3m, 0)) return 8;
        return zjoin_cols<R, 16>(n3m, 0) ? 16 : 0;
    } else {
        if (n3m % 8 == 0 && n3m / 8 <= 32) return 8;
        if (n3m % 12 == 0 && n3m / 12 <= 32) return 12;
        return n3m % 16 == 0 && n3m / 16 <= 32 ? 16 : 0;
    }
}

}  // namespace c3d
