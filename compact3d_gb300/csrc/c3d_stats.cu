// c3d_stats.cu -- ENERGY's plane statistics (compact3d.f:10003-10232) on the device, FP64:
// per plane J the cell-centre means, second moments, vorticity statistics, the two third
// moments ENERGY keeps, the third and fourth central moments and the mean wall-normal
// gradients (29 values; the column order is that of c3d_plane_stats in include/c3d.h).
//
// Every kernel here is bound by the FP64 pipe (2 lanes per clock and SM), so the sums are
// arranged for few FP64 instructions: a thread marches along z and keeps the values that the
// next points share, the x neighbours come by shuffles, cell-centre values are kept doubled
// (a sum of two, the powers of two leave in the last step), divisions by plane constants are
// products, and the mixed state converts in integer arithmetic (f2d).  192 x 128 x 192
// points, mixed state: plane statistics 2.95 -> 1.07 ms, spectra and correlations 8.5 -> 2.2.
#include "c3d_kern.cuh"

namespace c3d {

constexpr int SB = 8;        // blocks per plane of the quadrant sums
constexpr int STB = 128;     // threads per block
constexpr int NS1 = 23;      // first-pass sums: 20 moments + 3 gradients
constexpr int NS2 = 6;       // third and fourth central moments / means and squares

template <typename R>
__device__ __forceinline__ double sv(const typename SType<R>::S *a, const Geo &g, int i, int j, int k) {
    return St<R>::dbl(a[fidx(g, i, j, k)]);
}

// The marching sums: a warp takes MI = 30 columns i of plane J (lanes 1..30; lanes 0 and 31
// hold the neighbours) and a chunk of k.
constexpr int MI = 30, MW = STB / 32;
struct March {
    int nib, nkc, kc;   // column groups, chunks of k, points per chunk
    __host__ __device__ int nw() const { return nib * nkc; }
};
// Chunks of k: enough warps to fill the device 16 per SM, at least 8 points each.
__host__ __device__ inline March march_of(const Geo &g) {
    March m;
    m.nib = (g.n1m + MI - 1) / MI;
    int want = (152 * 16 + m.nib * g.n2m - 1) / (m.nib * g.n2m);
    if (want > g.n3m / 8) want = g.n3m / 8;
    if (want < 1) want = 1;
    m.kc = (g.n3m + want - 1) / want;
    m.nkc = (g.n3m + m.kc - 1) / m.kc;
    return m;
}
struct MPos {
    int j, w, k0, k1, i;   // plane, the warp's slot in it, its k range, the lane's column
    bool act;
};
__device__ __forceinline__ bool march_pos(const Geo &g, const March &m, MPos &p) {
    const int wid = blockIdx.x * MW + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (wid >= m.nw() * g.n2m) return false;
    p.j = 1 + wid / m.nw();
    p.w = wid % m.nw();
    const int ib = p.w % m.nib, c = p.w / m.nib;
    p.k0 = c * m.kc;
    p.k1 = min(g.n3m, p.k0 + m.kc);
    const int q = ib * MI + lane - 1;
    p.act = lane >= 1 && lane <= MI && q < g.n1m;
    p.i = q < 0 ? g.n1m - 1 : q % g.n1m;
    return true;
}
// The warp's sums in a fixed order to part[(J - 1) nw + w][NQ].
template <int NQ>
__device__ __forceinline__ void march_store(const double (&acc)[NQ], bool act, const March &m, const MPos &p, double *part) {
    double *o = part + ((size_t)(p.j - 1) * m.nw() + p.w) * NQ;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        double v = act ? acc[q] : 0.0;
        for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(FULL, v, off);
        if ((threadIdx.x & 31) == 0) o[q] = v;
    }
}

// pass 1.  Doubled cell-centre values U, V, W (2u at the cell), face values E at the cell's
// lower and upper face, vorticities W1..W3 in the units of the doubled values times one half.
template <typename R>
__global__ void __launch_bounds__(STB) k_stats1(StepArgs<R> a, March m, double *part) {
    typedef St<R> ST;
    const Geo &g = a.g;
    MPos p;
    if (!march_pos(g, m, p)) return;
    const int j = p.j, n = g.n3m, s = g.n1m;
    const double *DY = g.dy, *H = g.h;
    // face interpolation from the cells below and above; the wall values themselves on the walls
    double lo0 = 1.0, lo1 = 0.0, up0 = 0.0, up1 = 1.0;
    if (j > 1) { lo0 = 0.5 * DY[j] / H[j]; lo1 = 0.5 * DY[j - 1] / H[j]; }
    if (j < g.n2m) { up0 = 0.5 * DY[j + 1] / H[j + 1]; up1 = 0.5 * DY[j] / H[j + 1]; }
    const double hy = 1.0 / DY[j], qx = 0.5 * g.dx1, qz = 0.5 * g.dx3;   // of the doubled values
    const long long o = fidx(g, p.i, j, 0), om = o - g.np, op = o + g.np;
    auto at = [&](const typename SType<R>::S *f, long long b, int k) { return ST::dbl(f[b + (long long)k * s]); };
    auto pair = [&](double x) { return x + __shfl_down_sync(FULL, x, 1); };   // u(i) + u(i+1)
    const int km = p.k0 == 0 ? n - 1 : p.k0 - 1;
    double Um = pair(at(a.u, o, km)), U = pair(at(a.u, o, p.k0));
    double Vm = at(a.v, o, km) + at(a.v, op, km), v0 = at(a.v, o, p.k0), v1 = at(a.v, op, p.k0);
    double w = at(a.w, o, p.k0), wd = at(a.w, om, p.k0), wu = at(a.w, op, p.k0);
    double acc[NS1];
#pragma unroll
    for (int q = 0; q < NS1; ++q) acc[q] = 0.0;
    for (int k = p.k0; k < p.k1; ++k) {
        const int kp = k + 1 == n ? 0 : k + 1;
        const double Up = pair(at(a.u, o, kp)), Ud = pair(at(a.u, om, k)), Uu = pair(at(a.u, op, k));
        const double V = v0 + v1, vn0 = at(a.v, o, kp), vn1 = at(a.v, op, kp);
        const double wn = at(a.w, o, kp), wdn = at(a.w, om, kp), wun = at(a.w, op, kp);
        const double W = w + wn, Wd = wd + wdn, Wu = wu + wun, pp = at(a.p, o, k);
        const double dV = __shfl_down_sync(FULL, V, 1) - __shfl_up_sync(FULL, V, 1);
        const double dW = __shfl_down_sync(FULL, W, 1) - __shfl_up_sync(FULL, W, 1);
        const double gu = (up0 * U + up1 * Uu) - (lo0 * Ud + lo1 * U);
        const double gw = (up0 * W + up1 * Wu) - (lo0 * Wd + lo1 * W);
        const double o1 = hy * gw - qz * ((vn0 + vn1) - Vm), o2 = qz * (Up - Um) - qx * dW, o3 = qx * dV - hy * gu;
        const double uv = U * V, vw = V * W;
        acc[0] += U; acc[1] += V; acc[2] += W; acc[3] += pp;
        acc[4] += o1; acc[5] += o2; acc[6] += o3;
        acc[7] += U * U; acc[8] += V * V; acc[9] += W * W;
        acc[10] += uv; acc[11] += U * W; acc[12] += vw;
        acc[13] += pp * pp; acc[14] += pp * V;
        acc[15] += o1 * o1; acc[16] += o2 * o2; acc[17] += o3 * o3;
        acc[18] += U * uv; acc[19] += vw * W;
        acc[20] += gu; acc[21] += v1 - v0; acc[22] += gw;
        Um = U; U = Up; Vm = V; v0 = vn0; v1 = vn1; w = wn; wd = wdn; wu = wun;
    }
    march_store<NS1>(acc, p.act, m, p, part);
}

// The plane's sums over its warps' partial sums, in a fixed order (lane q adds q, q + 32, ...).
__device__ __forceinline__ double plane_sum(const double *part, int j0, int nw, int nq, int q) {
    double s = 0.0;
    for (int w = threadIdx.x & 31; w < nw; w += 32) s += part[((size_t)j0 * nw + w) * nq + q];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(FULL, s, off);
    return s;
}

// pass 1's plane means: out[J][0..19], [26..28].  A warp per sum; the doubled values leave
// their powers of two here.
__global__ void k_stats1_fin(Geo g, int nw, const double *part, double *out) {
    const int j = blockIdx.x, q = threadIdx.x >> 5;
    const double s = plane_sum(part, j, nw, NS1, q) / ((double)g.n1m * (double)g.n3m);
    if ((threadIdx.x & 31) != 0) return;
    double f = 1.0;
    if (q < 3 || q == 14) f = 0.5;
    else if (q >= 4 && q <= 6) f = 0.5;
    else if ((q >= 7 && q <= 12) || (q >= 15 && q <= 17)) f = 0.25;
    else if (q == 18 || q == 19) f = 0.125;
    else if (q >= 20) f = (q == 21 ? 1.0 : 0.5) / g.dy[j + 1];
    out[(size_t)j * 29 + (q < 20 ? q : q + 6)] = f * s;
}

// The marching loop over the cell-centre velocities alone: f(2u, 2v, 2w) at every point.
template <typename R, typename F>
__device__ __forceinline__ void march_cells(const StepArgs<R> &a, const MPos &p, F f) {
    typedef St<R> ST;
    const Geo &g = a.g;
    const long long s = g.n1m, o = fidx(g, p.i, p.j, 0), op = o + g.np;
    double w = ST::dbl(a.w[o + p.k0 * s]);
    for (int k = p.k0; k < p.k1; ++k) {
        const double u = ST::dbl(a.u[o + k * s]);
        const double wn = ST::dbl(a.w[o + (k + 1 == g.n3m ? 0 : k + 1) * s]);
        f(u + __shfl_down_sync(FULL, u, 1), ST::dbl(a.v[o + k * s]) + ST::dbl(a.v[op + k * s]), w + wn);
        w = wn;
    }
}

// pass 2: third and fourth central moments of the cell-centre velocities
template <typename R>
__global__ void __launch_bounds__(STB) k_stats2(StepArgs<R> a, March m, const double *out, double *part) {
    MPos p;
    if (!march_pos(a.g, m, p)) return;
    const double *mo = out + (size_t)(p.j - 1) * 29;
    const double m0 = 2.0 * mo[0], m1 = 2.0 * mo[1], m2 = 2.0 * mo[2];
    double acc[NS2] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    march_cells<R>(a, p, [&](double u, double v, double w) {
        const double x = u - m0, y = v - m1, z = w - m2, xx = x * x, yy = y * y, zz = z * z;
        acc[0] += xx * x; acc[1] += yy * y; acc[2] += zz * z;
        acc[3] += xx * xx; acc[4] += yy * yy; acc[5] += zz * zz;
    });
    march_store<NS2>(acc, p.act, m, p, part);
}

__global__ void k_stats2_fin(Geo g, int nw, const double *part, double *out) {
    const int j = blockIdx.x, q = threadIdx.x >> 5;
    const double s = plane_sum(part, j, nw, NS2, q) / ((double)g.n1m * (double)g.n3m);
    if ((threadIdx.x & 31) == 0) out[(size_t)j * 29 + 20 + q] = s * (q < 3 ? 0.125 : 0.0625);
}

// The means and mean squares of the cell-centre velocities alone (columns 0-2 and 7-9 of the
// table), for the spectra and correlations.
template <typename R>
__global__ void __launch_bounds__(STB) k_means(StepArgs<R> a, March m, double *part) {
    MPos p;
    if (!march_pos(a.g, m, p)) return;
    double acc[NS2] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    march_cells<R>(a, p, [&](double u, double v, double w) {
        acc[0] += u; acc[1] += v; acc[2] += w;
        acc[3] += u * u; acc[4] += v * v; acc[5] += w * w;
    });
    march_store<NS2>(acc, p.act, m, p, part);
}

__global__ void k_means_fin(Geo g, int nw, const double *part, double *out) {
    const int j = blockIdx.x, q = threadIdx.x >> 5;
    const double s = plane_sum(part, j, nw, NS2, q) / ((double)g.n1m * (double)g.n3m);
    if ((threadIdx.x & 31) == 0) out[(size_t)j * 29 + (q < 3 ? q : q + 4)] = s * (q < 3 ? 0.5 : 0.25);
}

static int march_blocks(const Geo &g, const March &m) { return nblk((long long)m.nw() * g.n2m, MW); }

template <typename R>
int launch_stats_t(c3d_channel *ch, StepArgs<R> &a, double *out, double *part, int means) {
    const Geo &g = ch->g;
    const March m = march_of(g);
    const int nb = march_blocks(g, m);
    if (means) {
        k_means<R><<<nb, STB, 0, ch->stream>>>(a, m, part);
        k_means_fin<<<g.n2m, 32 * NS2, 0, ch->stream>>>(g, m.nw(), part, out);
    } else {
        k_stats1<R><<<nb, STB, 0, ch->stream>>>(a, m, part);
        k_stats1_fin<<<g.n2m, 32 * NS1, 0, ch->stream>>>(g, m.nw(), part, out);
        k_stats2<R><<<nb, STB, 0, ch->stream>>>(a, m, out, part);
        k_stats2_fin<<<g.n2m, 32 * NS2, 0, ch->stream>>>(g, m.nw(), part, out);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : C3D_ECUDA;
}

template int launch_stats_t<double>(c3d_channel *, StepArgs<double> &, double *, double *, int);
template int launch_stats_t<float>(c3d_channel *, StepArgs<float> &, double *, double *, int);

// ---------------------------------------------------------------------------------
// ENERGY's 1-D spectra and two-point correlations (compact3d.f:10243-10515), FP64.
// Spectra: one block of SPW warps per (plane, component), Stockham FFTs with the channel's
// plans and double twiddles.  x: an x line of N1M reals as N1M/2 complex pairs and the
// real-input split, both modes of a split pair at once.  z: two lines as one complex line;
// the sum over lines of |X_k|^2 needs no split, because |X1_k|^2 + |X2_k|^2 =
// (|Z_k|^2 + |Z_-k|^2) / 2.  Constant factors are applied once to the sums.  The warps' sums
// are added in a fixed order.  Correlations: one block per (plane, component) walks the plane
// in tiles of CT rows k held in shared memory: RXX and RXY with a thread per x point summing
// over K in order, RZZ with a warp per tile row.
// ---------------------------------------------------------------------------------
constexpr int SPW = 4;

// cell-centre velocity of component L (0..2) at (i, j, k), v between j and jv
template <typename R>
__device__ __forceinline__ double vcell(const StepArgs<R> &a, int L, int i, int j, int k, int jv) {
    const Geo &g = a.g;
    if (L == 0) return (sv<R>(a.u, g, i, j, k) + sv<R>(a.u, g, i + 1 == g.n1m ? 0 : i + 1, j, k)) * 0.5;
    if (L == 1) return (sv<R>(a.v, g, i, j, k) + sv<R>(a.v, g, i, jv, k)) * 0.5;
    return (sv<R>(a.w, g, i, j, k) + sv<R>(a.w, g, i, j, k + 1 == g.n3m ? 0 : k + 1)) * 0.5;
}
// twice that, less m2
template <typename R>
__device__ __forceinline__ double vcell2(const StepArgs<R> &a, int L, int i, int j, int k, int jv, double m2) {
    const Geo &g = a.g;
    if (L == 0) return (sv<R>(a.u, g, i, j, k) + sv<R>(a.u, g, i + 1 == g.n1m ? 0 : i + 1, j, k)) - m2;
    if (L == 1) return (sv<R>(a.v, g, i, j, k) + sv<R>(a.v, g, i, jv, k)) - m2;
    return (sv<R>(a.w, g, i, j, k) + sv<R>(a.w, g, i, j, k + 1 == g.n3m ? 0 : k + 1)) - m2;
}

// x spectra: dynamic shared memory SPW x (2 (N1M/2) double2 + (N1M/2 + 1) doubles)
template <typename R>
__global__ void __launch_bounds__(32 * SPW) k_spec_x(StepArgs<R> a, const double *vmo, const double2 *twp,
                                                     double *xs) {
    const Geo g = a.g;
    const int j = 1 + blockIdx.x, L = blockIdx.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = g.n1m, M = N / 2;
    extern __shared__ double2 smx[];
    double2 *bufa = smx + (size_t)w * (2 * M), *bufb = bufa + M;
    double *acc = reinterpret_cast<double *>(smx + (size_t)SPW * 2 * M) + (size_t)w * (M + 1);
    const double m2 = 2.0 * vmo[L * g.n2m + (j - 1)];
    for (int q = lane; q <= M; q += 32) acc[q] = 0.0;
    for (int k = w; k < g.n3m; k += SPW) {
        for (int q = lane; q < M; q += 32)
            bufa[q] = make_double2(vcell2(a, L, 2 * q, j, k, j + 1, m2), vcell2(a, L, 2 * q + 1, j, k, j + 1, m2));
        __syncwarp();
        double2 *Z = fft_smem<double2, false>(bufa, bufb, a.fx, 0, 1, 0, -1, lane, 32);
        // modes q and M - q: 2E = Z_q + conj Z_(M-q), 2O = -i (Z_q - conj Z_(M-q)), T = exp(..) 2O:
        // 2 X_q = 2E + T, 2 conj X_(M-q) = 2E - T
        for (int q = lane; 2 * q <= M; q += 32) {
            const double2 zk = Z[q], zm = Z[q == 0 ? 0 : M - q], t = twp[q];
            const double Ex = zk.x + zm.x, Ey = zk.y - zm.y, Ox = zk.y + zm.y, Oy = zm.x - zk.x;
            const double Tx = t.x * Ox - t.y * Oy, Ty = t.x * Oy + t.y * Ox;
            const double ax = Ex + Tx, ay = Ey + Ty, bx = Ex - Tx, by = Ey - Ty;
            acc[q] += ax * ax + ay * ay;
            if (2 * q < M) acc[M - q] += bx * bx + by * by;
        }
        __syncwarp();
    }
    __syncthreads();
    double *out = xs + (size_t)N * ((j - 1) + (size_t)g.n2m * L);
    const double f = 0.0625 / N / (3.141592653589793 * g.dx1) / (double)g.n3m;   // 1/2 of the values, 1/2 of the split
    for (int q = threadIdx.x; q < N; q += blockDim.x) {
        const int kk = q <= M ? q : N - q;
        double s = 0.0;
        for (int ww = 0; ww < SPW; ++ww)
            s += reinterpret_cast<double *>(smx + (size_t)SPW * 2 * M)[(size_t)ww * (M + 1) + kk];
        out[q] = s * f;
    }
}

// z spectra: dynamic shared memory SPW x (2 N3M double2 + N3M doubles); lines i and i + 1
// (N1M is even) as one complex line
template <typename R>
__global__ void __launch_bounds__(32 * SPW) k_spec_z(StepArgs<R> a, const double *vmo, double *zs) {
    const Geo g = a.g;
    const int j = 1 + blockIdx.x, L = blockIdx.y, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int N = g.n3m;
    extern __shared__ double2 smz[];
    double2 *bufa = smz + (size_t)w * (2 * N), *bufb = bufa + N;
    double *accs = reinterpret_cast<double *>(smz + (size_t)SPW * 2 * N), *acc = accs + (size_t)w * N;
    const double m2 = 2.0 * vmo[L * g.n2m + (j - 1)];
    for (int q = lane; q < N; q += 32) acc[q] = 0.0;
    for (int i = 2 * w; i < g.n1m; i += 2 * SPW) {
        for (int q = lane; q < N; q += 32)
            bufa[q] = make_double2(vcell2(a, L, i, j, q, j + 1, m2), vcell2(a, L, i + 1, j, q, j + 1, m2));
        __syncwarp();
        const double2 *Z = fft_smem<double2, false>(bufa, bufb, a.fz, 0, 1, 0, -1, lane, 32);
        for (int q = lane; q < N; q += 32) acc[q] += Z[q].x * Z[q].x + Z[q].y * Z[q].y;
        __syncwarp();
    }
    __syncthreads();
    double *out = zs + (size_t)N * ((j - 1) + (size_t)g.n2m * L);
    const double f = 0.125 / N / (3.141592653589793 * g.dx3) / (double)g.n1m;   // 1/4 of the values, 1/2 of the pair
    for (int q = threadIdx.x; q < N; q += blockDim.x) {
        double s = 0.0;
        for (int ww = 0; ww < SPW; ++ww) s += accs[(size_t)ww * N + q] + accs[(size_t)ww * N + (q == 0 ? 0 : N - q)];
        out[q] = s * f;
    }
}

// correlations; st = the plane statistics table (VM in columns 0..2, VRMS in 7..9).  Dynamic
// shared memory: the two reference lines (N3M each), the reference row and CT rows of N1M + 1.
constexpr int CT = 8, CTB = 256;
template <typename R>
__global__ void __launch_bounds__(CTB) k_corr(StepArgs<R> a, const double *st, double *rxx, double *rzz,
                                             double *rxy) {
    const Geo g = a.g;
    const int j = 1 + blockIdx.x, L = blockIdx.y, N = g.n1m;
    const int n1h = g.n1m / 2, n3h = g.n3m / 2;   // N1H - 1, N3H - 1 (0-based)
    const double vm = st[(size_t)(j - 1) * 29 + L], var = st[(size_t)(j - 1) * 29 + 7 + L] - vm * vm;
    const double vm1 = st[L], var1 = st[7 + L] - vm1 * vm1;
    const int jv = j == g.n2m ? g.n2m : j + 1, jv1 = g.n2m == 1 ? 1 : 2;   // JPA(J), JPA(1)
    extern __shared__ double smc[];
    double *r0 = smc, *r1 = r0 + g.n3m, *rz = r1 + g.n3m, *T = rz + N;
    for (int k = threadIdx.x; k < g.n3m; k += CTB) {
        r0[k] = vcell(a, L, n1h, j, k, jv) - vm;
        r1[k] = vcell(a, L, n1h, 1, k, jv1) - vm1;
    }
    for (int i = threadIdx.x; i < N; i += CTB) rz[i] = vcell(a, L, i, j, n3h, jv) - vm;
    const size_t o = (size_t)g.n2m * L + (j - 1);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double rx[2] = {0.0, 0.0}, ry[2] = {0.0, 0.0};   // columns threadIdx.x and + CTB (N1M <= 384)
    for (int k0 = 0; k0 < g.n3m; k0 += CT) {         // N3M is a multiple of 16
        __syncthreads();
        for (int e = threadIdx.x; e < CT * N; e += CTB) {
            const int r = e / N, i = e - r * N;
            T[r * (N + 1) + i] = vcell(a, L, i, j, k0 + r, jv) - vm;
        }
        __syncthreads();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = threadIdx.x + h * CTB;
            if (i < N)
                for (int r = 0; r < CT; ++r) {
                    const double p = T[r * (N + 1) + i];
                    rx[h] = rx[h] + r0[k0 + r] * p;
                    ry[h] = ry[h] + r1[k0 + r] * p;
                }
        }
        if (rzz && w < CT) {
            double s = 0.0;
            for (int i = lane; i < N; i += 32) s += rz[i] * T[w * (N + 1) + i];
            for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(FULL, s, off);
            if (lane == 0) rzz[o * g.n3m + k0 + w] = s / (double)g.n1m / var;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = threadIdx.x + h * CTB;
        if (i >= N) continue;
        if (rxx) rxx[o * N + i] = rx[h] / (double)g.n3m / var;
        if (rxy) rxy[o * N + i] = ry[h] / (double)g.n3m / sqrt(var) / sqrt(var1);
    }
}

// ENERGY's quadrant analysis (compact3d.f:10560-10604): per plane the sums of
// u'v' = (u - VMP)(v - VMP) over the points of each sign quadrant of (u', v') and the
// points' counts; cell-centre u and v (V between J and J+1); vmp = VMP(J,1..2) (the
// reference's VMP is a local never assigned: zero-valued in practice).
__device__ __forceinline__ void block_sums(double *acc, int n, double *sh, double *outp) {
    for (int q = 0; q < n; ++q) sh[q * STB + threadIdx.x] = acc[q];
    __syncthreads();
    for (int s = STB / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
            for (int q = 0; q < n; ++q) sh[q * STB + threadIdx.x] += sh[q * STB + threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int q = 0; q < n; ++q) outp[q] = sh[q * STB];
}

template <typename R>
__global__ void __launch_bounds__(STB) k_quad(StepArgs<R> a, const double *vmp, double *part) {
    __shared__ double sh[8 * STB];
    const Geo &g = a.g;
    const int j = 1 + blockIdx.y;
    const int chunk = (g.np + SB - 1) / SB, e0 = blockIdx.x * chunk, e1 = min(g.np, e0 + chunk);
    const double m1 = vmp ? 2.0 * vmp[j - 1] : 0.0, m2 = vmp ? 2.0 * vmp[g.n2m + j - 1] : 0.0;
    double acc[8];
    int cnt[4] = {0, 0, 0, 0};
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.0;
    for (int e = e0 + threadIdx.x; e < e1; e += STB) {
        const int i = e % g.n1m, k = e / g.n1m;
        // doubled u', v': their quadrant by sign bits (zeros lie in none), the count as an integer
        const double V1P = vcell2(a, 0, i, j, k, j + 1, m1), V2P = vcell2(a, 1, i, j, k, j + 1, m2);
        const double uv = V1P * V2P;
        const unsigned long long b1 = (unsigned long long)__double_as_longlong(V1P), b2 = (unsigned long long)__double_as_longlong(V2P);
        const bool in = (b1 << 1) != 0 && (b2 << 1) != 0 && abs_bits(V1P) <= INF_BITS && abs_bits(V2P) <= INF_BITS;
        const bool n1 = (b1 >> 63) != 0, n2 = (b2 >> 63) != 0;
        const int q = n1 ? (n2 ? 2 : 1) : (n2 ? 3 : 0);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (in && q == c) { acc[c] += uv; ++cnt[c]; }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) { acc[c] *= 0.25; acc[4 + c] = (double)cnt[c]; }
    block_sums(acc, 8, sh, part + ((size_t)blockIdx.y * SB + blockIdx.x) * 8);
}

// Q(J,1..4) = -sum / (N1M N3M), QP(J,1..4) = count / (N1M N3M): out[(J-1) 8 + q]
__global__ void k_quad_fin(Geo g, const double *part, double *out) {
    const int j = blockIdx.x, q = threadIdx.x;
    if (q >= 8) return;
    double s = 0.0;
    for (int b = 0; b < SB; ++b) s += part[((size_t)j * SB + b) * 8 + q];
    const double NXZ = 1.0 / (double)(g.n1m * g.n3m);
    out[(size_t)j * 8 + q] = q < 4 ? -s * NXZ : s * NXZ;
}

template <typename R>
int launch_quadrants_t(c3d_channel *ch, StepArgs<R> &a, const double *vmp, double *out, double *part) {
    const Geo &g = ch->g;
    k_quad<R><<<dim3(SB, g.n2m), STB, 0, ch->stream>>>(a, vmp, part);
    k_quad_fin<<<g.n2m, 32, 0, ch->stream>>>(g, part, out);
    return cudaGetLastError() == cudaSuccess ? 0 : C3D_ECUDA;
}

template int launch_quadrants_t<double>(c3d_channel *, StepArgs<double> &, const double *, double *, double *);
template int launch_quadrants_t<float>(c3d_channel *, StepArgs<float> &, const double *, double *, double *);

// ENERGY's wall-stress spectrum (compact3d.f:10394-10416): the 2-D DFT of the bottom
// wall's TAUW - UTAU^2.  k_wspec_x: a warp per z row, the x transform of N1M reals as
// N1M/2 complex pairs and the real-input split, C1(kx, k) for kx = 0..N1M/2 into c1;
// k_wspec_z: a warp per kx, the z transform and |C|^2 / N1M / N3M / (PI DX3) / (PI DX1)
// at (kx, kz) and, by the conjugate symmetry of real data, at (N1M - kx, -kz).
__global__ void __launch_bounds__(32 * SPW) k_wspec_x(Geo g, FftPlan fx, const double *tauw, double utau,
                                                      const double2 *twp, double2 *c1) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, M = g.n1m / 2;
    const int k = blockIdx.x * SPW + w;
    extern __shared__ double2 smw[];
    double2 *bufa = smw + (size_t)w * (2 * M), *bufb = bufa + M;
    if (k >= g.n3m) return;
    const double t2 = utau * utau;
    const double *row = tauw + (size_t)k * g.n1m;
    for (int q = lane; q < M; q += 32) bufa[q] = make_double2(row[2 * q] - t2, row[2 * q + 1] - t2);
    __syncwarp();
    const double2 *Z = fft_smem<double2, false>(bufa, bufb, fx, 0, 1, 0, -1, lane, 32);
    for (int q = lane; q <= M; q += 32) {
        const double2 zk = Z[q == M ? 0 : q], zc = Z[q == 0 ? 0 : M - q];
        const double2 zm = make_double2(zc.x, -zc.y);
        const double Ex = 0.5 * (zk.x + zm.x), Ey = 0.5 * (zk.y + zm.y);
        const double Ox = 0.5 * (zk.y - zm.y), Oy = -0.5 * (zk.x - zm.x);
        const double2 t = twp[q];
        c1[(size_t)q * g.n3m + k] = make_double2(Ex + (t.x * Ox - t.y * Oy), Ey + (t.x * Oy + t.y * Ox));
    }
}

__global__ void __launch_bounds__(32 * SPW) k_wspec_z(Geo g, FftPlan fz, const double2 *c1, double *out) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, M = g.n1m / 2, N = g.n3m;
    const int kx = blockIdx.x * SPW + w;
    extern __shared__ double2 smw[];
    double2 *bufa = smw + (size_t)w * (2 * N), *bufb = bufa + N;
    if (kx > M) return;
    for (int q = lane; q < N; q += 32) bufa[q] = c1[(size_t)kx * N + q];
    __syncwarp();
    const double2 *Z = fft_smem<double2, false>(bufa, bufb, fz, 0, 1, 0, -1, lane, 32);
    const double s = 1.0 / g.n1m / N / (3.141592653589793 * g.dx3) / (3.141592653589793 * g.dx1);
    for (int q = lane; q < N; q += 32) {
        const double p = (Z[q].x * Z[q].x + Z[q].y * Z[q].y);
        out[(size_t)q * g.n1m + kx] = p * s;
        if (kx > 0 && kx < M) out[(size_t)((N - q) % N) * g.n1m + (g.n1m - kx)] = p * s;
    }
}

// ENERGY's 3-D two-point correlation (compact3d.f:10524-10556), a thread per point:
// RXYZ(I,J,K,L) = VP(N1H,N2H,N3H,L) VP(I,J,K,L) / rms(J) / rms(N2H), Fortran (N1M,N2M,N3M,3)
template <typename R>
__global__ void __launch_bounds__(256) k_corr3d(StepArgs<R> a, const double *st, double *out) {
    const Geo g = a.g;
    const long long n = (long long)g.n1m * g.n2m * g.n3m;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * n) return;
    const int L = (int)(t / n);
    long long r = t - L * n;
    const int i = (int)(r % g.n1m);
    r /= g.n1m;
    const int j = 1 + (int)(r % g.n2m), k = (int)(r / g.n2m);
    const int jh = g.aly == 1.0 ? g.n2m / 2 + 1 : g.n2m / 4 + 1, ih = g.n1m / 2, kh = g.n3m / 2;
    auto vm = [&](int jj) { return st[(size_t)(jj - 1) * 29 + L]; };
    auto rms = [&](int jj) { return sqrt(st[(size_t)(jj - 1) * 29 + 7 + L] - vm(jj) * vm(jj)); };
    auto jpa = [&](int jj) { return jj == g.n2m ? g.n2m : jj + 1; };
    const double ref = vcell(a, L, ih, jh, kh, jpa(jh)) - vm(jh);
    const double vp = vcell(a, L, i, j, k, jpa(j)) - vm(j);
    out[t] = ref * vp / rms(j) / rms(jh);
}

template <typename R>
int launch_corr3d_t(c3d_channel *ch, StepArgs<R> &a, const double *st, double *out) {
    const long long n = 3LL * ch->g.n1m * ch->g.n2m * ch->g.n3m;
    k_corr3d<R><<<(unsigned)((n + 255) / 256), 256, 0, ch->stream>>>(a, st, out);
    return cudaGetLastError() == cudaSuccess ? 0 : C3D_ECUDA;
}
template int launch_corr3d_t<double>(c3d_channel *, StepArgs<double> &, const double *, double *);
template int launch_corr3d_t<float>(c3d_channel *, StepArgs<float> &, const double *, double *);

int launch_wall_spectrum(c3d_channel *ch, double utau, double2 *c1, double *out) {
    const Geo &g = ch->g;
    const int M = g.n1m / 2;
    const size_t smx = (size_t)SPW * 2 * M * sizeof(double2), smz = (size_t)SPW * 2 * g.n3m * sizeof(double2);
    if (cudaFuncSetAttribute(k_wspec_x, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smx) != cudaSuccess ||
        cudaFuncSetAttribute(k_wspec_z, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smz) != cudaSuccess)
        return C3D_ECUDA;
    const double2 *twp = ch->tw64 + g.n1m / 2 + g.n3m;
    k_wspec_x<<<(g.n3m + SPW - 1) / SPW, 32 * SPW, smx, ch->stream>>>(g, ch->fx, ch->tauw, utau, twp, c1);
    k_wspec_z<<<(M + 1 + SPW - 1) / SPW, 32 * SPW, smz, ch->stream>>>(g, ch->fz, c1, out);
    return cudaGetLastError() == cudaSuccess ? 0 : C3D_ECUDA;
}

template <typename R>
int launch_spectra_t(c3d_channel *ch, StepArgs<R> &a, const double *vmo, const double *st, double *xs, double *zs,
                     double *rxx, double *rzz, double *rxy) {
    const Geo &g = ch->g;
    const dim3 grid(g.n2m, 3);
    if (xs) {
        const int M = g.n1m / 2;
        const size_t sm = (size_t)SPW * (2 * M * sizeof(double2) + (M + 1) * sizeof(double));
        if (cudaFuncSetAttribute(k_spec_x<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
            return C3D_ECUDA;
        const double2 *twp = ch->tw64 + g.n1m / 2 + g.n3m;   // exp(-2 pi i q / N1M), q = 0..N1M/2
        k_spec_x<R><<<grid, 32 * SPW, sm, ch->stream>>>(a, vmo, twp, xs);
    }
    if (zs) {
        const size_t sm = (size_t)SPW * (2 * g.n3m * sizeof(double2) + g.n3m * sizeof(double));
        if (cudaFuncSetAttribute(k_spec_z<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
            return C3D_ECUDA;
        k_spec_z<R><<<grid, 32 * SPW, sm, ch->stream>>>(a, vmo, zs);
    }
    if (rxx || rzz || rxy) {
        const size_t sm = (2 * (size_t)g.n3m + g.n1m + (size_t)CT * (g.n1m + 1)) * sizeof(double);
        if (cudaFuncSetAttribute(k_corr<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
            return C3D_ECUDA;
        k_corr<R><<<grid, CTB, sm, ch->stream>>>(a, st, rxx, rzz, rxy);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : C3D_ECUDA;
}

template int launch_spectra_t<double>(c3d_channel *, StepArgs<double> &, const double *, const double *, double *,
                                      double *, double *, double *, double *);
template int launch_spectra_t<float>(c3d_channel *, StepArgs<float> &, const double *, const double *, double *,
                                     double *, double *, double *, double *);

// Scratch the statistics need on the device: the output table and the partial sums.
size_t stats_scratch_doubles(const Geo &g) {
    const size_t part = (size_t)march_of(g).nw() * NS1, quad = (size_t)SB * 8;
    return (size_t)g.n2m * (29 + (part > quad ? part : quad));
}

}  // namespace c3d
