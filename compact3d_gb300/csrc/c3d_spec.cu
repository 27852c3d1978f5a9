// c3d_spec.cu -- the spectral part of GETDP (compact3d.f:9271-9441): complex FFT of the
// half spectrum along z, and one wall-normal Thomas solve (TDMAP, 9444-9459) per (kx, kz).
#include "c3d_kern.cuh"

namespace c3d {

// Complex FFT along kz of a tile of `tw` kx columns of one plane, in shared memory.
template <typename R>
__device__ __forceinline__ void b_fftz(const StepArgs<R> &a, int sign, int tw, const Blk blk) {
    typedef typename Cx<R>::T C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Geo g = a.g;
    const int n = g.n3m;
    C2 *A = reinterpret_cast<C2 *>(smem_raw), *B = A + n * tw;
    const int ntile = (g.n1h + tw - 1) / tw;
    const int plane = blk.x / ntile, tile = blk.x % ntile;
    const int kx0 = tile * tw;
    const int w = min(tw, g.n1h - kx0);
    C2 *S = reinterpret_cast<C2 *>(a.spec) + (long long)plane * n * g.n1h + kx0;
    const int lsh = __ffs(tw) - 1, lm = tw - 1;   // tw is a power of 2
    // asynchronous copies, all in flight at once (a load and a shared store per element waits
    // for each load: 256 x 192 x 256 points, FP32, 127 us a transform)
    for (int e = threadIdx.x; e < n * tw; e += blockDim.x) {
        const int q = e >> lsh, l = e & lm;
        if (l < w) cp_async_c2(&A[e], &S[q * g.n1h + l]);
        else { A[e].x = 0; A[e].y = 0; }
    }
    cp_async_wait_all();
    __syncthreads();
    C2 *Z = fft_smem<C2, true>(A, B, a.fz, lsh, tw, 1, sign, threadIdx.x, blockDim.x);
    for (int e = threadIdx.x; e < n * tw; e += blockDim.x) {
        const int q = e >> lsh, l = e & lm;
        if (l < w) S[q * g.n1h + l] = Z[e];
    }
}
template <typename R>
__global__ void __launch_bounds__(TPB) k_fftz(StepArgs<R> a, int sign, int tw) {
    pdl_enter();
    b_fftz<R>(a, sign, tw, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// Complex FFT along kz, one warp per kx column, for N3M = 32 N1 (four-step form).  The
// block stages a tile of TWW kx columns of one plane in shared memory (coalesced rows,
// padded pitch); a warp holds its column as x[n1] = X(32 n1 + lane), takes the N1-point
// DFT over n1 in registers, multiplies by exp(sign 2 pi i lane k1 / N3M), and finishes
// with a 32-point DFT across the lanes (five decimation-in-frequency shuffle stages),
// after which lane l holds the outputs k1 + N1 bitrev5(l).  Twiddles come from the z
// plan's table exp(-2 pi i j / N3M).
constexpr int TWW = 16;    // kx columns per block
constexpr int FZW = 8;     // warps per block
template <typename R, int N1, int SIGN>
__device__ __forceinline__ void b_fftz4(const StepArgs<R> &a, const Blk blk) {
    typedef typename Cx<R>::T C2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C2 *T = reinterpret_cast<C2 *>(smem_raw);
    const Geo g = a.g;
    constexpr int n = 32 * N1, pitch = TWW + 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int ntile = (g.n1h + TWW - 1) / TWW;
    const int plane = blk.x / ntile, kx0 = (blk.x % ntile) * TWW;
    const int w = min(TWW, g.n1h - kx0);
    C2 *S = reinterpret_cast<C2 *>(a.spec) + (long long)plane * n * g.n1h + kx0;
    const C2 *tw = twsel<C2>(a.fz);
    auto twd = [&](int j) {   // exp(SIGN 2 pi i j / n)
        C2 t = __ldg(&tw[j]);
        if constexpr (SIGN > 0) t.y = -t.y;
        return t;
    };
    // the tile arrives by asynchronous copies (no register staging), all in flight at once
    for (int e = threadIdx.x; e < n * TWW; e += FZW * 32) {
        const int q = e >> 4, l = e & (TWW - 1);
        if (l < w) cp_async_c2(&T[q * pitch + l], &S[q * g.n1h + l]);
    }
    cp_async_wait_all();
    C2 wn1[N1], tl[N1], ts[5];
#pragma unroll
    for (int j = 0; j < N1; ++j) { wn1[j] = twd(32 * j); tl[j] = twd(lane * j); }
#pragma unroll
    for (int st = 0; st < 5; ++st) {   // stage with half-distance h = 16 >> st: exp(SIGN 2 pi i (lane mod h) / 2h)
        const int h = 16 >> st;
        ts[st] = twd((lane & (h - 1)) * (n / (2 * h)));
    }
    __syncthreads();
    for (int c = wid; c < w; c += FZW) {
        C2 x[N1];
#pragma unroll
        for (int m = 0; m < N1; ++m) x[m] = T[(32 * m + lane) * pitch + c];
        rdft<N1, SIGN, N1>(x, wn1);
#pragma unroll
        for (int k = 1; k < N1; ++k) x[k] = cmul(x[k], tl[k]);
#pragma unroll
        for (int st = 0; st < 5; ++st) {
            const int h = 16 >> st;
            const bool hi = (lane & h) != 0;
#pragma unroll
            for (int k = 0; k < N1; ++k) {
                C2 o;
                o.x = __shfl_xor_sync(0xffffffffu, x[k].x, h);
                o.y = __shfl_xor_sync(0xffffffffu, x[k].y, h);
                x[k] = hi ? cmul(csub(o, x[k]), ts[st]) : cadd(x[k], o);
            }
        }
        __syncwarp();
        // x[k] is frequency k + N1 * bitrev5(lane); it goes to tile row lane + 32 k, so that
        // the 16 lanes of a half-warp write 16 distinct bank pairs (row k + N1 bitrev5(lane)
        // puts them on 2 when N1 = 12), and the copy-out below reads each frequency's row.
#pragma unroll
        for (int k = 0; k < N1; ++k) T[(lane + 32 * k) * pitch + c] = x[k];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * TWW; e += FZW * 32) {
        const int q = e >> 4, l = e & (TWW - 1);
        const int lq = q / N1, kq = q - lq * N1;
        const int row = (int)(__brev((unsigned)lq) >> 27) + 32 * kq;
        if (l < w) S[q * g.n1h + l] = T[row * pitch + l];
    }
}
template <typename R, int N1, int SIGN>
__global__ void __launch_bounds__(FZW * 32) k_fftz4(StepArgs<R> a) {
    pdl_enter();
    b_fftz4<R, N1, SIGN>(a, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// One Thomas solve per mode (kx, kz) with A_J = PMJ, B_J = PCJ - AK3 - AK1, C_J = PPJ,
// factors tabulated by k_ptables; the (0,0) mode has row 1 = (0, 1, 0 | 0) and the
// imaginary parts of the self-conjugate modes are zero (compact3d.f:9363-9397).
// FP64 form: FP64 arithmetic.  Mixed form: the same recurrences in double-float
// arithmetic (FP32 instructions), with double-float factor tables: on stretched grids the
// low-wavenumber systems are near-singular and an FP32 recurrence loses accuracy.  The
// forward values are stored at the spectrum's precision between the two sweeps.
// A mode is one sequential chain over the planes and there are few modes per SM, so a warp's own
// instructions bound it.  The real and the imaginary part of a mode are two threads; each sweep
// runs in batches of UJ planes without guards, two sets of registers take turns (one is loaded
// while the other computes), positions are 32-bit, and the tables' planes up to UPF further on
// are requested from DRAM into L2.  Against a thread per mode with guarded batches (55 to 78
// instructions a plane): 64^3 points, FP64, 31 -> 18 us, 192 x 128 x 144 67 -> 37, mixed
// 128 x 96 x 128 27 -> 23, 256 x 192 x 256 111 -> 109; 384 x 256 x 384 points, with modes
// enough for every SM, is slower: 132 -> 151.
constexpr int UJ = 8, UPF = 32;

// The warp's 16 modes of a table's rows (`row` points at the calling thread's own value) at UJ
// planes p, p + DIR, ..., requested from DRAM into L2: a line of 128 bytes a plane.
template <int DIR, typename T>
__device__ __forceinline__ void pf_modes(const T *row, unsigned s, int p, int N) {
    const int lane = threadIdx.x & 31, pl = p + DIR * lane;
    if (lane < UJ && pl >= 0 && pl < N) pf_l2(row + (unsigned)pl * s - (lane >> 1));
}

// What the sweeps of both forms are made of: V one component of a mode's spectrum value, F a
// factor.
template <typename V, typename F>
struct PzBatch {
    V q[UJ];
    F f[UJ];
    // planes p, p + d, ... of the spectrum S and the table T (one plane further on for OFF = 1)
    template <int OFF>
    __device__ __forceinline__ void load(const V *S, const F *T, int p, unsigned s, int d) {
#pragma unroll
        for (int u = 0; u < UJ; ++u) {
            q[u] = S[(unsigned)(p + d * u) * 2u * s];
            f[u] = T[(unsigned)(p + d * u + OFF) * s];
        }
    }
    __device__ __forceinline__ void store(V *S, int p, unsigned s, int d) const {
#pragma unroll
        for (int u = 0; u < UJ; ++u) S[(unsigned)(p + d * u) * 2u * s] = q[u];
    }
};
// Both sweeps of one component of one mode.  `fwd(q, f, am)` and `bwd(q, f)` advance the
// recurrence by one plane and return what the plane takes (the last plane `last()`); the first plane's
// recurrence starts from zero, and `zero` clears its right-hand side.
template <typename V, typename F, typename FW, typename BW, typename LA>
__device__ __forceinline__ void pz_sweeps(V *S, const F *RB, const F *GM, const F *PM, int N, unsigned s, bool zero,
                                          FW fwd, BW bwd, LA last) {
    PzBatch<V, F> A, B;
    const int nb = N / UJ;   // full batches
    auto run = [&](PzBatch<V, F> &b, int p) {
        pf_modes<1>(RB, s, p + UPF, N);
        if (p == 0 && zero) b.q[0] = V(0);
#pragma unroll
        for (int u = 0; u < UJ; ++u) b.q[u] = fwd(b.q[u], b.f[u], PM[p + u + 1]);
        b.store(S, p, s, 1);
    };
    for (int p = UJ; p < UPF; p += UJ) pf_modes<1>(RB, s, p, N);
    if (nb > 0) A.template load<0>(S, RB, 0, s, 1);
    for (int b = 0; b < nb; b += 2) {
        if (b + 1 < nb) B.template load<0>(S, RB, (b + 1) * UJ, s, 1);
        run(A, b * UJ);
        if (b + 1 >= nb) break;
        if (b + 2 < nb) A.template load<0>(S, RB, (b + 2) * UJ, s, 1);
        run(B, (b + 1) * UJ);
    }
    for (int p = nb * UJ; p < N; ++p) S[(unsigned)p * 2u * s] = fwd(p == 0 && zero ? V(0) : S[(unsigned)p * 2u * s], RB[(unsigned)p * s], PM[p + 1]);
    S[(unsigned)(N - 1) * 2u * s] = last();
    // the planes N-2 .. 0, of which the first batch reads values this thread stored above
    const int mb = (N - 1) / UJ, top = N - 2;
    auto runb = [&](PzBatch<V, F> &b, int p) {
        pf_modes<-1>(GM, s, p - UPF + 1, N);
#pragma unroll
        for (int u = 0; u < UJ; ++u) b.q[u] = bwd(b.q[u], b.f[u]);
        b.store(S, p, s, -1);
    };
    for (int p = UJ; p < UPF; p += UJ) pf_modes<-1>(GM, s, top - p + 1, N);
    if (mb > 0) A.template load<1>(S, GM, top, s, -1);
    for (int b = 0; b < mb; b += 2) {
        if (b + 1 < mb) B.template load<1>(S, GM, top - (b + 1) * UJ, s, -1);
        runb(A, top - b * UJ);
        if (b + 1 >= mb) break;
        if (b + 2 < mb) A.template load<1>(S, GM, top - (b + 2) * UJ, s, -1);
        runb(B, top - (b + 1) * UJ);
    }
    for (int p = top - mb * UJ; p >= 0; --p) S[(unsigned)p * 2u * s] = bwd(S[(unsigned)p * 2u * s], GM[(unsigned)(p + 1) * s]);
}
// The thread's mode and component (0 real, 1 imaginary); true for a self-conjugate mode.
__device__ __forceinline__ bool pz_mode(const Geo &g, const Blk blk, int &mode, int &comp) {
    const int t = blk.x * blockDim.x + threadIdx.x;
    mode = t >> 1;
    comp = t & 1;
    const int kx = mode % g.n1h, kz = mode / g.n1h;
    return (kx == 0 || kx == g.n1m / 2) && (kz == 0 || kz == g.n3m / 2);
}

__device__ __forceinline__ void b_poisson64(const StepArgs<double> &a, const Blk blk) {
    const Geo g = a.g;
    const int nm = g.n1h * g.n3m;
    int mode, comp;
    const bool selfc = pz_mode(g, blk, mode, comp) && comp;
    if (mode >= nm) return;
    double x = 0.0;
    pz_sweeps(
        reinterpret_cast<double *>(a.spec) + 2 * mode + comp, a.prb + mode, a.pgam + mode, a.pmj, g.n2m, nm,
        mode == 0 && comp == 0,      // row 1 of the (1,1) mode: x_1 = 0
        [&](double q, double rb, double am) { return x = (q - am * x) * rb; },
        [&](double q, double gm) {
            x = q - gm * x;
            return selfc ? 0.0 : x;
        },
        [&]() { return selfc ? 0.0 : x; });
}
__global__ void __launch_bounds__(TPB) k_poisson64(StepArgs<double> a) {
    pdl_enter();
    b_poisson64(a, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

__device__ __forceinline__ void b_poisson32(const StepArgs<float> &a, const Blk blk) {
    const Geo g = a.g;
    const int nm = g.n1h * g.n3m;
    int mode, comp;
    const bool selfc = pz_mode(g, blk, mode, comp) && comp;
    if (mode >= nm) return;
    float2 x = make_float2(0.f, 0.f);
    pz_sweeps(
        reinterpret_cast<float *>(a.spec) + 2 * mode + comp, a.prbdf + mode, a.pgamdf + mode, a.pmjdf, g.n2m, nm,
        mode == 0 && comp == 0,      // row 1 of the (1,1) mode: x_1 = 0
        [&](float q, float2 rb, float2 am) {
            x = df_mul(df_fsub(q, df_mul(am, x)), rb);
            return x.x;
        },
        [&](float q, float2 gm) {
            x = df_fsub(q, df_mul(gm, x));
            return selfc ? 0.f : x.x;
        },
        [&]() { return selfc ? 0.f : x.x; });
}
__global__ void __launch_bounds__(TPB) k_poisson32(StepArgs<float> a) {
    pdl_enter();
    b_poisson32(a, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// Factor tables of TDMAP's recurrence for every mode (FP64; double-float copies when rb32 != 0).
__global__ void k_ptables(Geo g, const double *ak1, const double *ak3, const double *pmj, const double *pcj,
                          const double *ppj, double *rb, double *gam, float2 *rb32, float2 *gam32) {
    const int nm = g.n1h * g.n3m;
    const int mode = blockIdx.x * blockDim.x + threadIdx.x;
    if (mode >= nm) return;
    const int kx = mode % g.n1h, kz = mode / g.n1h;
    const int kzs = kz <= g.n3m / 2 ? kz : g.n3m - kz;
    const double lam3 = ak3[kzs], lam1 = ak1[kx];
    double B1 = pcj[1] - lam3 - lam1, C1 = ppj[1];
    if (mode == 0) { B1 = 1.0; C1 = 0.0; }
    double bet = B1;
    rb[mode] = 1.0 / bet;
    gam[mode] = 0.0;
    if (rb32) { rb32[mode] = St<float>::from_double(1.0 / bet); gam32[mode] = make_float2(0.f, 0.f); }
    double cprev = C1;
    for (int J = 2; J <= g.n2m; ++J) {
        double gm = cprev / bet;
        bet = (pcj[J] - lam3 - lam1) - pmj[J] * gm;
        const long long q = (long long)(J - 1) * nm + mode;
        gam[q] = gm;
        rb[q] = 1.0 / bet;
        if (rb32) { gam32[q] = St<float>::from_double(gm); rb32[q] = St<float>::from_double(1.0 / bet); }
        cprev = ppj[J];
    }
}

constexpr int TWZ_MAX = 16;   // widest z-FFT tile the autotuner tries

constexpr size_t SMEM_MAX = 227 * 1024;

// The widest z-FFT tile, from `want` kx columns down, whose two buffers fit in shared memory
// (N3M lines of C2 values: FP64 lines of more than 900 points narrow a tile of 8, FP32 of 1800).
template <typename C2>
static int fftz_tile(int n3m, int want) {
    int tw = want;
    while (tw > 1 && 2 * (size_t)n3m * tw * sizeof(C2) > SMEM_MAX) tw /= 2;
    return tw;
}

template <typename R>
void set_spec_smem(c3d_channel *ch) {
    typedef typename Cx<R>::T C2;
    const size_t smz = 2 * (size_t)ch->g.n3m * TWZ_MAX * sizeof(C2);
    cudaFuncSetAttribute(k_fftz<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smz < SMEM_MAX ? smz : SMEM_MAX));
}

// The four-step z FFT for N3M = 32 N1; false when N3M is not of that form.
template <typename R, int SIGN>
static bool launch_fftz4(c3d_channel *ch, StepArgs<R> &a) {
    typedef typename Cx<R>::T C2;
    const Geo &g = ch->g;
    if (g.n3m % 32 != 0) return false;
    const int ntile = (g.n1h + TWW - 1) / TWW;
    const size_t sm = (size_t)g.n3m * (TWW + 1) * sizeof(C2);
    const dim3 grid(g.n2m * ntile), blk(FZW * 32);
    void (*fn)(StepArgs<R>) = nullptr;
    switch (g.n3m / 32) {
        case 2: fn = k_fftz4<R, 2, SIGN>; break;
        case 3: fn = k_fftz4<R, 3, SIGN>; break;
        case 4: fn = k_fftz4<R, 4, SIGN>; break;
        case 6: fn = k_fftz4<R, 6, SIGN>; break;
        case 8: fn = k_fftz4<R, 8, SIGN>; break;
        case 12: fn = k_fftz4<R, 12, SIGN>; break;
        case 16: fn = k_fftz4<R, 16, SIGN>; break;
        default: return false;
    }
    if (sm > 227 * 1024) return false;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    klaunch(ch, ch->stream, fn, grid, blk, sm, a);
    return true;
}

// ---------------------------------------------------------------------------------
// Batch form: the z FFTs of the channels with the same N3M in one launch (the four-step
// warp form when N3M = 32 N1, tiles of 8 kx columns in shared memory otherwise, of fewer where
// a long line's would not fit) and the Poisson solves of every channel in one launch.
// ---------------------------------------------------------------------------------
constexpr int TW_BATCH = 8;

template <typename R, int N1, int SIGN>
__global__ void __launch_bounds__(FZW * 32) kb_fftz4(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    b_fftz4<R, N1, SIGN>(A[m.ch], Blk{m.x, m.y, m.gx});
}
template <typename R, int SIGN, int TW>
__global__ void __launch_bounds__(TPB) kb_fftz(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    b_fftz<R>(A[m.ch], SIGN, TW, Blk{m.x, m.y, m.gx});
}
__global__ void __launch_bounds__(TPB) kb_poisson64(const StepArgs<double> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    b_poisson64(A[m.ch], Blk{m.x, m.y, m.gx});
}
__global__ void __launch_bounds__(TPB) kb_poisson32(const StepArgs<float> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    b_poisson32(A[m.ch], Blk{m.x, m.y, m.gx});
}

template <typename R, int SIGN>
static const void *fftz4_batch_fn(int n1) {
    switch (n1) {
        case 2: return (const void *)kb_fftz4<R, 2, SIGN>;
        case 3: return (const void *)kb_fftz4<R, 3, SIGN>;
        case 4: return (const void *)kb_fftz4<R, 4, SIGN>;
        case 6: return (const void *)kb_fftz4<R, 6, SIGN>;
        case 8: return (const void *)kb_fftz4<R, 8, SIGN>;
        case 12: return (const void *)kb_fftz4<R, 12, SIGN>;
        case 16: return (const void *)kb_fftz4<R, 16, SIGN>;
        default: return nullptr;
    }
}

template <typename R, int SIGN>
static const void *fftz_batch_fn(int tw) {
    switch (tw) {
        case 1: return (const void *)kb_fftz<R, SIGN, 1>;
        case 2: return (const void *)kb_fftz<R, SIGN, 2>;
        case 4: return (const void *)kb_fftz<R, SIGN, 4>;
        default: return (const void *)kb_fftz<R, SIGN, TW_BATCH>;
    }
}

template <typename R>
int spec_bkern(const c3d_channel *ch, int which, std::vector<BKern> &out) {
    typedef typename Cx<R>::T C2;
    const Geo &g = ch->g;
    if (which == 1) {
        const void *fn = sizeof(R) == 8 ? (const void *)kb_poisson64 : (const void *)kb_poisson32;
        out.push_back({fn, TPB, 0, (unsigned)nblk(2LL * g.n1h * g.n3m)});
        return 0;
    }
    if (which != 0 && which != 2) return C3D_EINVAL;
    const void *f4 = nullptr;
    if (g.n3m % 32 == 0) f4 = which == 0 ? fftz4_batch_fn<R, -1>(g.n3m / 32) : fftz4_batch_fn<R, +1>(g.n3m / 32);
    const size_t sm4 = (size_t)g.n3m * (TWW + 1) * sizeof(C2);
    if (f4 && sm4 <= 227 * 1024) {
        out.push_back({f4, FZW * 32, sm4, (unsigned)(g.n2m * ((g.n1h + TWW - 1) / TWW))});
        return 0;
    }
    const int tw = fftz_tile<C2>(g.n3m, TW_BATCH);
    const size_t smz = 2 * (size_t)g.n3m * tw * sizeof(C2);
    const void *fn = which == 0 ? fftz_batch_fn<R, -1>(tw) : fftz_batch_fn<R, +1>(tw);
    out.push_back({fn, TPB, smz, (unsigned)(g.n2m * ((g.n1h + tw - 1) / tw))});
    return 0;
}
template int spec_bkern<double>(const c3d_channel *, int, std::vector<BKern> &);
template int spec_bkern<float>(const c3d_channel *, int, std::vector<BKern> &);

template <typename R>
int launch_spec(c3d_channel *ch, StepArgs<R> &a, int which, int *nl) {
    typedef typename Cx<R>::T C2;
    cudaStream_t st = ch->stream;
    const double N = (double)ch->g.n1m * ch->g.n2m * ch->g.n3m, Rb = sizeof(R);
    if (ch->tune.twz == 0 && (which == 0 || which == 2)) {   // four-step form when N3M allows
        if (which == 0 ? launch_fftz4<R, -1>(ch, a) : launch_fftz4<R, +1>(ch, a)) {
            mark(ch, nl, which == 0 ? "fftz_fwd" : "fftz_inv", N * 2 * Rb);
            return 0;
        }
    }
    const int tw = fftz_tile<C2>(ch->g.n3m, ch->tune.twz == 0 ? 8 : ch->tune.twz);
    const int ntile = (ch->g.n1h + tw - 1) / tw;
    const size_t smz = 2 * (size_t)ch->g.n3m * tw * sizeof(C2);
    switch (which) {
        case 0: klaunch(ch, st, k_fftz<R>, ch->g.n2m * ntile, TPB, smz, a, -1, tw); mark(ch, nl, "fftz_fwd", N * 2 * Rb); break;
        case 1: {
            // blocks of 64: the few modes of a small grid reach every SM
            const int nb = nblk(2LL * ch->g.n1h * ch->g.n3m, 64);
            if constexpr (sizeof(R) == 8) klaunch(ch, st, k_poisson64, nb, 64, 0, a);
            else klaunch(ch, st, k_poisson32, nb, 64, 0, a);
            mark(ch, nl, "poisson", N * 2 * Rb + N * 8);
            break;
        }
        case 2: klaunch(ch, st, k_fftz<R>, ch->g.n2m * ntile, TPB, smz, a, +1, tw); mark(ch, nl, "fftz_inv", N * 2 * Rb); break;
        default: return C3D_EINVAL;
    }
    return 0;
}

int launch_ptables(c3d_channel *ch, const double *ak1, const double *ak3, const double *pm, const double *pc,
                   const double *pp) {
    const int nm = ch->g.n1h * ch->g.n3m;
    k_ptables<<<nblk(nm), TPB, 0, ch->stream>>>(ch->g, ak1, ak3, pm, pc, pp, ch->prb, ch->pgam, ch->prbdf,
                                                ch->pgamdf);
    return 0;
}

template void set_spec_smem<double>(c3d_channel *);
template void set_spec_smem<float>(c3d_channel *);
template int launch_spec<double>(c3d_channel *, StepArgs<double> &, int, int *);
template int launch_spec<float>(c3d_channel *, StepArgs<float> &, int, int *);

}  // namespace c3d
