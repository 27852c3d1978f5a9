// c3d_zpass.cu -- z-column passes of the step: one thread per (i, segment of L points,
// plane j); consecutive threads take consecutive i, so every access is coalesced.  The
// cyclic compact solves run with warm-ups (zsweep: FP32) or with the segments of a line
// joined in the block (zjoin: FP64, and FP32 under schedule 0).
//   zA  RHS1/2/3 pieces along z (compact3d.f:6160-6185, 6337-6433, 6957-7060, 7474-7705)
//   zB  d(uw)/dz, d(vw)/dz, d(ww)/dz (1,22,1)
//   zC  z factor of Crank-Nicolson (CTDMA3I in GETUH1-3)
//   zD  RHSDP along z (8187-8210)
//   zE  UPCALC along z and the velocity / pressure update (1052-1238)
//   diag_z  DIVCHECK z part and max|div| (9099-9128)
// Compiled once per precision (C3D_BITS).
#include "c3d_zcols.cuh"

namespace c3d {

// ---------------------------------------------------------------------------------
// Column walkers for zsweep: each keeps a sliding window of its stencil inputs in
// registers and loads one new value per position.
// ---------------------------------------------------------------------------------
// Prefetch ring of a column: the values at the D positions after the walker's current
// one, loaded D steps before they are used so the loads of consecutive steps overlap.
constexpr int ZPF = 4;
template <typename T>
struct ZRing {
    T v[ZPF];
    int kf;   // position of v[ZPF-1]
    __device__ void fill(const T *col, int k, int n, int s) {
        kf = k;
#pragma unroll
        for (int d = 0; d < ZPF; ++d) {
            kf = znext(kf, n);
            v[d] = col[kf * s];
        }
    }
    // value at the next position; the ring advances by one
    __device__ T pop(const T *col, int n, int s) {
        const T r = v[0];
#pragma unroll
        for (int d = 0; d < ZPF - 1; ++d) v[d] = v[d + 1];
        kf = znext(kf, n);
        v[ZPF - 1] = col[kf * s];
        return r;
    }
};

// state column: (1,10,1) RHS f12*(u- - 2u + u+) and (1,6,1) RHS 4*(u- + u) (face k)
template <typename R>
struct WalkVisBack {
    typedef typename SType<R>::S S;
    const S *col; int n, s; R f12, four; S um, uc; ZRing<S> ru;
    __device__ void start(int k) { um = col[zprev(k, n) * s]; uc = col[k * s]; ru.fill(col, k, n, s); }
    __device__ void next(R (&d)[2]) {
        S up = ru.pop(col, n, s);
        d[0] = f12 * St<R>::d2(um, uc, up);
        d[1] = four * (St<R>::hi(um) + St<R>::hi(uc));
        um = uc; uc = up;
    }
};

// W and P columns: f12*(w- - 2w + w+), 4*(w + w+) (centre k) and f24*(p - p-) (face k)
template <typename R>
struct WalkWP {
    typedef typename SType<R>::S S;
    const S *W, *P; int n, s; R f12, four, f24; S wm, wc, pm, pc; ZRing<S> rw, rp;
    __device__ void start(int k) {
        wm = W[zprev(k, n) * s]; wc = W[k * s]; pm = P[zprev(k, n) * s]; pc = P[k * s];
        rw.fill(W, k, n, s);
        rp.fill(P, k, n, s);
    }
    __device__ void next(R (&d)[3]) {
        S wp = rw.pop(W, n, s);
        d[0] = f12 * St<R>::d2(wm, wc, wp);
        d[1] = four * (St<R>::hi(wc) + St<R>::hi(wp));
        d[2] = f24 * St<R>::d(pc, pm);
        wm = wc; wc = wp; pm = pc; pc = rp.pop(P, n, s);
    }
};

// zB: f*(Exz+ - Exz), f*(Q - Q-), f*(Eyz+ - Eyz)
template <typename R>
struct WalkZB {
    const R *E1, *Q, *E2; int n, s; R f; R e1, qm, e2; int kn, kc; bool v;
    __device__ void start(int k) {
        e1 = E1[k * s]; qm = Q[zprev(k, n) * s]; e2 = v ? E2[k * s] : R(0); kc = k; kn = znext(k, n);
    }
    __device__ void next(R (&d)[3]) {
        R e1p = E1[kn * s], qc = Q[kc * s], e2p = v ? E2[kn * s] : R(0);
        d[0] = f * (e1p - e1);
        d[1] = f * (qc - qm);
        d[2] = f * (e2p - e2);
        e1 = e1p; qm = qc; e2 = e2p; kc = kn; kn = znext(kn, n);
    }
};

// zC: (x- + 10x) + x+ for the three components
template <typename R>
struct WalkCN {
    const R *X[3]; int n, s; R xm[3], xc[3]; ZRing<R> rx[3];
    __device__ void start(int k) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            xm[c] = X[c][zprev(k, n) * s]; xc[c] = X[c][k * s];
            rx[c].fill(X[c], k, n, s);
        }
    }
    __device__ void next(R (&d)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            R xp = rx[c].pop(X[c], n, s);
            d[c] = (xm[c] + (R)10.0 * xc[c]) + xp;
            xm[c] = xc[c]; xc[c] = xp;
        }
    }
};

// zC by partial fractions (FP64): x itself
template <typename R>
struct WalkX3 {
    const R *X[3]; int n, s; int k;
    __device__ void start(int k0) { k = k0; }
    __device__ void next(R (&d)[3]) {
#pragma unroll
        for (int c = 0; c < 3; ++c) d[c] = X[c][k * s];
        ++k;
    }
};

// zD: f24*((W+ + D+) - (W + D))
template <typename R>
struct WalkDivZ {
    typedef typename SType<R>::S S;
    const S *W; const R *D; int n, s; R f24; S wc; R dc; ZRing<S> rw; ZRing<R> rd;
    __device__ void start(int k) { wc = W[k * s]; dc = D[k * s]; rw.fill(W, k, n, s); rd.fill(D, k, n, s); }
    __device__ void next(R (&d)[1]) {
        S wp = rw.pop(W, n, s); R dp = rd.pop(D, n, s);
        d[0] = f24 * Sten<R>::dd(wp, dp, wc, dc);
        wc = wp; dc = dp;
    }
};

// zE: f24*(DP - DP-)
template <typename R>
struct WalkGradZ {
    const R *DP; int n, s; R f24; R pm; ZRing<R> rp;
    __device__ void start(int k) { pm = DP[zprev(k, n) * s]; rp.fill(DP, zprev(k, n), n, s); }
    __device__ void next(R (&d)[1]) {
        R pc = rp.pop(DP, n, s);
        d[0] = f24 * (pc - pm);
        pm = pc;
    }
};

// PART 0 runs the three sweeps in one kernel; PART 1, 2, 3 run only the u, the (w, P) or
// the v sweep (the split form has fewer registers per thread and moves the same bytes).
template <typename R, int L, int PART, int MODE>
__device__ __forceinline__ void b_zA(const StepArgs<R> &a, const Blk blk) {
    typedef typename SType<R>::S S;
    typedef St<R> ST;
    const Geo g = a.g;
    ZCo c;
    // the v sweep has no face at J = 1: joined lines start at J = 2, so that a block's
    // threads all take part in the solve
    if (!zcoords<L, MODE>(blk, g, MODE == 1 && PART == 3 ? 2 : 1, c)) return;
    const int i = c.i, j = c.j, k0 = c.k0;
    const int n = g.n3m, s = g.n1m;
    const R RE1 = a.re1;
    const long long o = fidx(g, i, j, 0);
    constexpr int M6 = WM<R>::M6, B = ztb<L>();
    constexpr int NH = PART == 0 ? 3 : 2;   // the fused form's three solves share the exchange area
    if (MODE == 0 && (g.n1m & 31) == 0) {   // the warp's column windows (32 consecutive i), requested at once
        const int lane = threadIdx.x & 31;
        const long long o0 = fidx(g, i - lane, j, 0), sb = (long long)g.n1m;
        const int ss = 32 * (int)sizeof(S), sr = 32 * (int)sizeof(R);
        if (PART <= 1) {
            pf_cols(a.u + o0, sb * sizeof(S), ss, k0, M6 + 1, L, n, lane);
            pf_cols(a.ww1 + o0, sb * sizeof(R), sr, k0, 0, L, n, lane);
            pf_cols(a.r[0] + o0, sb * sizeof(R), sr, k0, 0, L, n, lane);
        }
        if (PART == 0 || PART == 2) {
            pf_cols(a.w + o0, sb * sizeof(S), ss, k0, M6 + 1, L, n, lane);
            pf_cols(a.p + o0, sb * sizeof(S), ss, k0, M6 + 1, L, n, lane);
            pf_cols(a.r[2] + o0, sb * sizeof(R), sr, k0, 0, L, n, lane);
        }
        if ((PART == 0 || PART == 3) && j >= 2) {
            pf_cols(a.v + o0, sb * sizeof(S), ss, k0, M6 + 1, L, n, lane);
            pf_cols(a.r[1] + o0, sb * sizeof(R), sr, k0, 0, L, n, lane);
            // w at the y face: planes J and J-1 of the segment, read after the solve
            if (PART == 3) pf_cols(a.w + o0, sb * sizeof(S), ss, k0, 0, L, n, lane);
            pf_cols(a.w + fidx(g, i - lane, j - 1, 0), sb * sizeof(S), ss, k0, 0, L, n, lane);
        }
    }
    const R f12 = zrhs<MODE>(a.f12z), four = zrhs<MODE>((R)4.0), f24 = zrhs<MODE>(a.f24z);
    const R kv = RE1 * zfold<MODE>(a.f12z, a.c10z.s), ki = zfold<MODE>((R)4.0, a.c6z.s), kp = zfold<MODE>(a.f24z, a.c22z.s);
    if (PART == 0 || PART == 1) {   // u: R1 += (1/RE) d2u/dz2 ; E_xz = UU3 * WW1
        R out[2][L];
        const R rr[2] = {zroot<10>(a.c10z.r), zroot<6>(a.c6z.r)}, ss[2] = {a.c10z.s, a.c6z.s};
        WalkVisBack<R> f{a.u + o, n, s, f12, four};
        zsolve<R, L, M6, 2, MODE, NH>(out, c, n, rr, ss, f);
        R *Rp = a.r[0] + o, *E = a.exz + o;
        const R *Wx = a.ww1 + o;
        const R kw = ki * ((R)4.0 * a.c6x.s);   // FP64: WW1 comes without its factor
        if (c.act) {
#pragma unroll
            for (int b = 0; b < L; b += B) {
                R rv[B], wv[B];
                zload(rv, Rp, k0 + b, s);
                zload(wv, Wx, k0 + b, s);
#pragma unroll
                for (int t = 0; t < B; ++t) {
                    const int kk = (k0 + b + t) * s;
                    Rp[kk] = rv[t] + kv * out[0][b + t];
                    E[kk] = sizeof(R) == 8 ? out[1][b + t] * (kw * wv[t])
                            : MODE == 1    ? out[1][b + t] * (ki * wv[t]) : out[1][b + t] * wv[t];
                }
            }
        }
    }
    if (PART == 0 || PART == 2) {   // w, P: R3 += (1/RE) d2w/dz2 - dP/dz - PRESG3 ; WW3^2
        R out[3][L];
        const R rr[3] = {zroot<10>(a.c10z.r), zroot<6>(a.c6z.r), zroot<22>(a.c22z.r)}, ss[3] = {a.c10z.s, a.c6z.s, a.c22z.s};
        WalkWP<R> f{a.w + o, a.p + o, n, s, f12, four, f24};
        zsolve<R, L, M6, 3, MODE>(out, c, n, rr, ss, f);
        const R presg3 = sizeof(R) == 8 ? R(0) : (R)a.scal[SCAL_PRESG3];   // FP64: in xA's sum
        R *Rp = a.r[2] + o, *Q = a.wsq + o;
        if (c.act) {
#pragma unroll
            for (int b = 0; b < L; b += B) {
                R rv[B];
                zload(rv, Rp, k0 + b, s);
#pragma unroll
                for (int t = 0; t < B; ++t) {
                    const int kk = (k0 + b + t) * s;
                    if constexpr (MODE == 1) {
                        const R rn = rv[t] + kv * out[0][b + t] - kp * out[2][b + t];
                        Rp[kk] = sizeof(R) == 8 ? rn : rn - presg3;
                        const R ww3 = ki * out[1][b + t];
                        Q[kk] = ww3 * ww3;
                    } else {
                        Rp[kk] = rv[t] + RE1 * out[0][b + t] - out[2][b + t] - presg3;
                        Q[kk] = out[1][b + t] * out[1][b + t];
                    }
                }
            }
        }
    }
    if (PART == 0 || PART == 3) {   // v: R2 += (1/RE) d2v/dz2 ; E_yz = VV3 * (w at y face J)
        if (MODE == 0 && j < 2) return;
        R out[2][L];
        const R rr[2] = {zroot<10>(a.c10z.r), zroot<6>(a.c6z.r)}, ss[2] = {a.c10z.s, a.c6z.s};
        WalkVisBack<R> f{a.v + o, n, s, f12, four};
        zsolve<R, L, M6, 2, MODE, NH>(out, c, n, rr, ss, f);
        const R Hj1 = a.m.rh[j], a1 = a.m.hdy[j], a2 = a.m.hdy[j - 1];
        const S *W = a.w + o, *Wm = a.w + fidx(g, i, j - 1, 0);
        R *Rp = a.r[1] + o, *E = a.eyz + o;
        if (c.act && j >= 2) {
            const R b1 = ki * Hj1 * a1, b2 = ki * Hj1 * a2;
#pragma unroll
            for (int b = 0; b < L; b += B) {
                R rv[B];
                S wm[B], wc[B];
                zload(rv, Rp, k0 + b, s);
                zload(wm, Wm, k0 + b, s);
                zload(wc, W, k0 + b, s);
#pragma unroll
                for (int t = 0; t < B; ++t) {
                    const int kk = (k0 + b + t) * s;
                    Rp[kk] = rv[t] + kv * out[0][b + t];
                    R wy = MODE == 1 ? b1 * ST::hi(wm[t]) + b2 * ST::hi(wc[t])
                                     : Hj1 * (a1 * ST::hi(wm[t]) + a2 * ST::hi(wc[t]));
                    E[kk] = out[1][b + t] * wy;
                }
            }
        }
    }
}
template <typename R, int L, int PART, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) k_zA(StepArgs<R> a) {
    pdl_enter();
    b_zA<R, L, PART, MODE>(a, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// H += k z with one rounding at every position, written out: left to the compiler, which
// multiply-adds it fuses differs between the instances, and with it the bits of a channel alone
// and in an ensemble.
template <typename R, int L, int MODE>
__device__ __forceinline__ void b_zB(const StepArgs<R> &a, const Blk blk) {
    const Geo g = a.g;
    ZCo c;
    if (!zcoords<L, MODE>(blk, g, 1, c)) return;
    const int i = c.i, j = c.j, k0 = c.k0;
    const int n = g.n3m, s = g.n1m;
    const long long o = fidx(g, i, j, 0);
    if (MODE == 0 && (g.n1m & 31) == 0) {
        const int lane = threadIdx.x & 31;
        const long long o0 = fidx(g, i - lane, j, 0), sb = (long long)g.n1m;
        pf_cols(a.exz + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::M22 + 1, L, n, lane);
        pf_cols(a.wsq + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::M22 + 1, L, n, lane);
        pf_cols(a.eyz + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::M22 + 1, L, n, lane);
        pf_cols(a.hh[0] + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, 0, L, n, lane);
        pf_cols(a.hh[1] + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, 0, L, n, lane);
    }
    R out[3][L];
    const R r22 = zroot<22>(a.c22z.r), rr[3] = {r22, r22, r22}, ss[3] = {R(1), R(1), R(1)};
    WalkZB<R> f{a.exz + o, a.wsq + o, a.eyz + o, n, s, zrhs<MODE>(a.f24z)};
    f.v = (j >= 2);
    zsolve<R, L, WM<R>::M22, 3, MODE>(out, c, n, rr, ss, f);
    R *H1 = a.hh[0] + o, *H2 = a.hh[1] + o, *H3 = a.hh[2] + o;
    const R ks = MODE == 1 ? zfold<MODE>(a.f24z, a.c22z.s) : a.c22z.s;
    if (!c.act) return;
    constexpr int B = ztb<L>();
#pragma unroll
    for (int b = 0; b < L; b += B) {
        R h1[B], h2[B];
        zload(h1, H1, k0 + b, s);
        if (j >= 2) zload(h2, H2, k0 + b, s);
#pragma unroll
        for (int t = 0; t < B; ++t) {
            const int kk = (k0 + b + t) * s;
            H1[kk] = fma(ks, out[0][b + t], h1[t]);               // d(uw)/dz
            H3[kk] = ks * out[1][b + t];                          // d(ww)/dz
            if (j >= 2) H2[kk] = fma(ks, out[2][b + t], h2[t]);   // d(vw)/dz
        }
    }
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) k_zB(StepArgs<R> a) {
    pdl_enter();
    b_zB<R, L, MODE>(a, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// z factor of Crank-Nicolson: r[c] -> d[c] for the three components (the v component at
// J=1 is computed from zeros and never read)
template <typename R, int L, int MODE>
__device__ __forceinline__ void b_zC(const StepArgs<R> &a, R *d0, R *d1, R *d2, const Blk blk) {
    const Geo g = a.g;
    ZCo c;
    if (!zcoords<L, MODE>(blk, g, 1, c)) return;
    const int i = c.i, j = c.j, k0 = c.k0;
    const int n = g.n3m, s = g.n1m;
    const long long o = fidx(g, i, j, 0);
    if (MODE == 0 && (g.n1m & 31) == 0) {
        const int lane = threadIdx.x & 31;
        const long long o0 = fidx(g, i - lane, j, 0), sb = (long long)g.n1m;
        pf_cols(a.r[0] + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::MCN + 1, L, n, lane);
        pf_cols(a.r[1] + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::MCN + 1, L, n, lane);
        pf_cols(a.r[2] + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::MCN + 1, L, n, lane);
    }
    R out[3][L];
    const R rr[3] = {a.cnz.r, a.cnz.r, a.cnz.r}, ss[3] = {a.cnz.s, a.cnz.s, a.cnz.s};
    R *D0 = d0 + o, *D1 = d1 + o, *D2 = d2 + o;
    const R ks = zfold<MODE>(R(1), a.cnz.s);
    if constexpr (sizeof(R) == 8 && MODE == 1) {
        if (a.kz[0] != R(0)) {   // partial fractions, as in xB (which applied their common factor)
            WalkX3<R> f{{a.r[0] + o, a.r[1] + o, a.r[2] + o}, n, s, 0};
            zsolve<R, L, WM<R>::MCN, 3, MODE>(out, c, n, rr, ss, f);
            if (!c.act) return;
            constexpr int B = ztb<L>() / 2;
            const R kz = a.kz[1];
#pragma unroll
            for (int b = 0; b < L; b += B) {
                R x0[B], x1[B], x2[B];
                zload(x0, f.X[0], k0 + b, s);
                zload(x1, f.X[1], k0 + b, s);
                zload(x2, f.X[2], k0 + b, s);
#pragma unroll
                for (int t = 0; t < B; ++t) {
                    const int kk = (k0 + b + t) * s;
                    D0[kk] = x0[t] + kz * out[0][b + t];
                    D1[kk] = x1[t] + kz * out[1][b + t];
                    D2[kk] = x2[t] + kz * out[2][b + t];
                }
            }
            return;
        }
    }
    WalkCN<R> f;
    f.X[0] = a.r[0] + o; f.X[1] = a.r[1] + o; f.X[2] = a.r[2] + o;
    f.n = n; f.s = s;
    zsolve<R, L, WM<R>::MCN, 3, MODE>(out, c, n, rr, ss, f);
    if (!c.act) return;
#pragma unroll
    for (int t = 0; t < L; ++t) {
        const int kk = (k0 + t) * s;
        D0[kk] = ks * out[0][t];
        D1[kk] = ks * out[1][t];
        D2[kk] = ks * out[2][t];
    }
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) k_zC(StepArgs<R> a, R *d0, R *d1, R *d2) {
    pdl_enter();
    b_zC<R, L, MODE>(a, d0, d1, d2, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// zC where the root reaches past the warm-ups (a.zfar.m > 0: q = DT DX3^2 / (2 RE) above about
// 1/5; the channels' own DT keep it some 1e-3): s B(F(d)) as s/(1 - r^2) times the sum of r^|m|
// over both sides, each side from up to a whole line of points before the segment, closed over
// the line by 1/(1 - r^N).  In FP64 whatever the form: the gain 1/(1 - r)^2 grows with q.
template <typename R>
__device__ __forceinline__ void b_zCfar(const StepArgs<R> &a, R *d0, R *d1, R *d2, const Blk blk) {
    constexpr int L = ZL;
    const Geo g = a.g;
    ZCo c;
    if (!zcoords<L, 0>(blk, g, 1, c)) return;
    const CnFar f = a.zfar;
    const int n = g.n3m, s = g.n1m;
    const long long o = fidx(g, c.i, c.j, 0);
#pragma unroll 1
    for (int q = 0; q < 3; ++q) {
        const R *X = (q == 0 ? a.r[0] : q == 1 ? a.r[1] : a.r[2]) + o;
        R *D = (q == 0 ? d0 : q == 1 ? d1 : d2) + o;
        // right-hand sides from position k on, upwards (DIR 1) or downwards: xa, xb the values at
        // the position before and at k
        int k = wrapi(c.k0 - f.m, n);
        double xa = X[zprev(k, n) * s], xb = X[k * s];
        auto up = [&]() {
            k = znext(k, n);
            const double xc = X[k * s], d = (xa + 10.0 * xb) + xc;
            xa = xb;
            xb = xc;
            return d;
        };
        auto down = [&]() {
            k = zprev(k, n);
            const double xc = X[k * s], d = (xa + 10.0 * xb) + xc;
            xa = xb;
            xb = xc;
            return d;
        };
        double y = 0.0, out[L];
        for (int t = 0; t < f.m; ++t) y = up() + f.r * y;
        y *= f.y0;
#pragma unroll
        for (int t = 0; t < L; ++t) {
            y = up() + f.r * y;
            out[t] = y;
        }
        k = wrapi(c.k0 + L - 1 + f.m, n);
        xa = X[znext(k, n) * s];
        xb = X[k * s];
        y = 0.0;
        for (int t = 0; t < f.m; ++t) y = down() + f.r * y;
        y *= f.y0;
#pragma unroll
        for (int t = L - 1; t >= 0; --t) {
            D[(c.k0 + t) * s] = (R)(f.c * (out[t] + f.r * y));
            y = down() + f.r * y;
        }
    }
}
template <typename R>
__global__ void __launch_bounds__(TPB) k_zCfar(StepArgs<R> a, R *d0, R *d1, R *d2) {
    pdl_enter();
    b_zCfar<R>(a, d0, d1, d2, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// z part of RHSDP: rdpz = compact d(UH3)/dz / DT with UH3 = W + delta3
template <typename R, int L, int MODE>
__device__ __forceinline__ void b_zD(const StepArgs<R> &a, const R *d2, const Blk blk) {
    const Geo g = a.g;
    ZCo c;
    if (!zcoords<L, MODE>(blk, g, 1, c)) return;
    const int i = c.i, j = c.j, k0 = c.k0;
    const int n = g.n3m, s = g.n1m;
    const long long o = fidx(g, i, j, 0);
    if (MODE == 0 && (g.n1m & 31) == 0) {
        const int lane = threadIdx.x & 31;
        const long long o0 = fidx(g, i - lane, j, 0), sb = (long long)g.n1m;
        pf_cols(a.w + o0, sb * sizeof(typename SType<R>::S), 32 * (int)sizeof(typename SType<R>::S), k0, WM<R>::M22 + 1, L, n, lane);
        pf_cols(d2 + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::M22 + 1, L, n, lane);
    }
    R out[1][L];
    const R rr[1] = {zroot<22>(a.c22z.r)}, ss[1] = {a.c22z.s};
    WalkDivZ<R> f{a.w + o, d2 + o, n, s, zrhs<MODE>(a.f24z)};
    zsolve<R, L, WM<R>::M22, 1, MODE>(out, c, n, rr, ss, f);
    const R rdt = a.rdt * zfold<MODE>(a.f24z, a.c22z.s);
    R *Q = a.rdpz + o;
    if (!c.act) return;
#pragma unroll
    for (int t = 0; t < L; ++t) Q[(k0 + t) * s] = out[0][t] * rdt;
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) k_zD(StepArgs<R> a, const R *d2) {
    pdl_enter();
    b_zD<R, L, MODE>(a, d2, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// UPCALC along z and the state update
template <typename R, int L, int MODE>
__device__ __forceinline__ void b_zE(const StepArgs<R> &a, const R *d0, const R *d1, const R *d2, int updp, const Blk blk) {
    typedef typename SType<R>::S S;
    typedef St<R> ST;
    const Geo g = a.g;
    ZCo c;
    if (!zcoords<L, MODE>(blk, g, 1, c)) return;
    const int i = c.i, j = c.j, k0 = c.k0;
    const int n = g.n3m, s = g.n1m;
    const long long o = fidx(g, i, j, 0);
    const R dt = (R)a.dt;
    const R dtdm = dt * (R)a.scal[SCAL_DMPRESG], dtdm3 = dt * (R)a.scal[SCAL_DMPRESG3];
    const R *DP = a.dp + o;
    if (MODE == 0 && (g.n1m & 31) == 0) {
        const int lane = threadIdx.x & 31;
        const long long o0 = fidx(g, i - lane, j, 0), sb = (long long)g.n1m;
        pf_cols(a.dp + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, WM<R>::M22 + 1, L, n, lane);
        pf_cols(a.u + o0, sb * sizeof(S), 32 * (int)sizeof(S), k0, 0, L, n, lane);
        pf_cols(a.v + o0, sb * sizeof(S), 32 * (int)sizeof(S), k0, 0, L, n, lane);
        pf_cols(a.w + o0, sb * sizeof(S), 32 * (int)sizeof(S), k0, 0, L, n, lane);
        pf_cols(a.p + o0, sb * sizeof(S), 32 * (int)sizeof(S), k0, 0, L, n, lane);
        if (sizeof(R) == 8) pf_cols(d0 + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, 0, L, n, lane);
        pf_cols(d1 + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, 0, L, n, lane);
        pf_cols(d2 + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, 0, L, n, lane);
        pf_cols(a.g1 + o0, sb * sizeof(R), 32 * (int)sizeof(R), k0, 0, L, n, lane);
    }
    R out[1][L];
    const R rr[1] = {zroot<22>(a.c22z.r)}, ss[1] = {a.c22z.s};
    WalkGradZ<R> f{DP, n, s, zrhs<MODE>(a.f24z)};
    zsolve<R, L, WM<R>::M22, 1, MODE>(out, c, n, rr, ss, f);
    S *W = a.w + o, *U = a.u + o, *V = a.v + o, *Pp = a.p + o;
    const R *D0 = d0 + o, *D1 = d1 + o, *D2 = d2 + o, *G1 = a.g1 + o;
    const R *DPm = a.dp + fidx(g, i, j - 1, 0);
    const R rHj = a.m.rh[j], dtg = dt * zfold<MODE>(a.f24z, a.c22z.s), dth = dt * rHj;
    const R dtx = dt * xfold(a.f24x, a.c22x);   // FP64: g1 without its factor (xD)
    if (!c.act) return;
    constexpr int B = ztb<L>() / 2;   // nine fields are live
#pragma unroll
    for (int b = 0; b < L; b += B) {
        S uv[B], vv[B], wv[B], pv[B];
        R d0v[B], d1v[B], d2v[B], gv[B], pc[B], pm[B];
        zload(wv, W, k0 + b, s);
        zload(d2v, D2, k0 + b, s);
        zload(uv, U, k0 + b, s);
        zload(gv, G1, k0 + b, s);
        if (sizeof(R) == 8) zload(d0v, D0, k0 + b, s);
        zload(pc, DP, k0 + b, s);
        if (j >= 2) {
            zload(vv, V, k0 + b, s);
            zload(d1v, D1, k0 + b, s);
            zload(pm, DPm, k0 + b, s);
        }
        if (updp) zload(pv, Pp, k0 + b, s);
#pragma unroll
        for (int t = 0; t < B; ++t) {
            const int kk = (k0 + b + t) * s;
            W[kk] = Sten<R>::upd(wv[t], d2v[t], dtg * out[0][b + t], dtdm3);
            if constexpr (sizeof(R) == 4) U[kk] = ST::add(uv[t], gv[t] - dtdm);   // G1: delta1 - DT dDP/dx (xD)
            else U[kk] = Sten<R>::upd(uv[t], d0v[t], dtx * gv[t], dtdm);
            if (j >= 2) {
                const R dpy = MODE == 1 ? dth * (pc[t] - pm[t]) : dt * (pc[t] - pm[t]) * rHj;
                V[kk] = Sten<R>::upd(vv[t], d1v[t], dpy, R(0));
            }
            if (updp) Pp[kk] = ST::add(pv[t], pc[t]);
        }
    }
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) k_zE(StepArgs<R> a, const R *d0, const R *d1, const R *d2, int updp) {
    pdl_enter();
    b_zE<R, L, MODE>(a, d0, d1, d2, updp, Blk{blockIdx.x, blockIdx.y, gridDim.x});
}

// DIVCHECK z part and max |div| (FP64): joined segments, or warm-ups (L = ZL) on lines too
// long for a block.
template <typename R>
struct WalkDiagZ {
    typedef typename SType<R>::S S;
    const S *W; int n, s; double wc; int kn;
    __device__ void start(int k) { wc = St<R>::dbl(W[k * s]); kn = znext(k, n); }
    __device__ void next(double (&d)[1]) {
        const double wp = St<R>::dbl(W[kn * s]);
        d[0] = wp - wc;
        wc = wp;
        kn = znext(kn, n);
    }
};
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<double, L>() : TPB) k_diag_z(StepArgs<R> a, const double *divx,
                                                                               Cyc<double> c22) {
    pdl_enter();
    const Geo g = a.g;
    ZCo c;
    unsigned long long m = 0;
    bool bad = false;
    if (zcoords<L, MODE>(Blk{blockIdx.x, blockIdx.y, gridDim.x}, g, 1, c)) {
        const int n = g.n3m, s = g.n1m;
        const long long o = fidx(g, c.i, c.j, 0);
        const double *DX = divx + o;
        double out[1][L], dx[L];
        const double rr[1] = {c22.r}, ss[1] = {1.0}, f = 24.0 * g.dx3 * c22.s;
        WalkDiagZ<R> w{a.w + o, n, s};
        zsolve<double, L, WM<double>::M22, 1, MODE>(out, c, n, rr, ss, w);
        zload(dx, DX, c.k0, s);
#pragma unroll
        for (int t = 0; t < L; ++t) {
            const unsigned long long dv = abs_bits(dx[t] + f * out[0][t]);
            bad |= c.act && dv >= INF_BITS;
            if (c.act && dv <= INF_BITS && dv > m) m = dv;
        }
    }
    warp_max_to(&a.scal[SCAL_DIVMAX], m, bad, &a.scal[SCAL_NONFIN]);
}

template <typename R, int L, int MODE>
static int launch_zpass_l(c3d_channel *ch, StepArgs<R> &a, int which, R *d0, R *d1, R *d2, int flag, int *nl);

// ---------------------------------------------------------------------------------
// Batch form: one launch per pass covers every channel (segment form, segments of ZL
// points, which divides every supported N3M); zA as its three sweeps; the work arrays
// are the channel's exz / eyz / wsq as in the step, and zE adds DP to P.
// ---------------------------------------------------------------------------------
template <typename R, int PART, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) kb_zA(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    b_zA<R, L, PART, MODE>(A[m.ch], Blk{m.x, m.y, m.gx});
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) kb_zB(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    b_zB<R, L, MODE>(A[m.ch], Blk{m.x, m.y, m.gx});
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) kb_zC(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    const StepArgs<R> &a = A[m.ch];
    b_zC<R, L, MODE>(a, a.exz, a.eyz, a.wsq, Blk{m.x, m.y, m.gx});
}
template <typename R>
__global__ void __launch_bounds__(TPB) kb_zCfar(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    const StepArgs<R> &a = A[m.ch];
    b_zCfar<R>(a, a.exz, a.eyz, a.wsq, Blk{m.x, m.y, m.gx});
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) kb_zD(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    const StepArgs<R> &a = A[m.ch];
    b_zD<R, L, MODE>(a, a.wsq, Blk{m.x, m.y, m.gx});
}
template <typename R, int L, int MODE>
__global__ void __launch_bounds__(MODE == 1 ? zjt<R, L>() : TPB) kb_zE(const StepArgs<R> *__restrict__ A, const BMap *__restrict__ map) {
    pdl_enter();
    const BMap m = map[blockIdx.x];
    const StepArgs<R> &a = A[m.ch];
    b_zE<R, L, MODE>(a, a.exz, a.eyz, a.wsq, 1, Blk{m.x, m.y, m.gx});
}

template <typename R, int L, int MODE>
static int zbk(const c3d_channel *ch, int which, std::vector<BKern> &out) {
    const Geo &g = ch->g;
    const unsigned nb = (unsigned)nblk((long long)g.n2m * (g.n3m / L) * g.n1m);
    auto put = [&](auto *fn, int njoin, int jn, int run, int piece) {
        if (MODE == 0) {
            out.push_back({(const void *)fn, TPB, 0, nb, run, piece});
            return;
        }
        const long long ncol = (long long)jn * g.n1m;
        const int cols = zjoin_cols<R, L>(g.n3m, ncol);
        const unsigned nt = (unsigned)(cols * (g.n3m / L));
        out.push_back({(const void *)fn, nt, 2 * (size_t)njoin * nt * sizeof(R), (unsigned)nblk(ncol, cols), run, piece});
    };
    switch (which) {
        case 0:
            put(kb_zA<R, 1, L, MODE>, 2, g.n2m, 2, 0);
            put(kb_zA<R, 2, L, MODE>, 3, g.n2m, 2, 1);
            put(kb_zA<R, 3, L, MODE>, 2, g.n2m - 1, 2, 2);
            return 0;
        case 1: put(kb_zB<R, L, MODE>, 3, g.n2m, 0, 0); return 0;
        case 2: put(kb_zC<R, L, MODE>, 3, g.n2m, 0, 0); return 0;
        case 3: put(kb_zD<R, L, MODE>, 1, g.n2m, 0, 0); return 0;
        case 4: put(kb_zE<R, L, MODE>, 1, g.n2m, 0, 0); return 0;
        default: return C3D_EINVAL;
    }
}

// z pass `which` of a batch channel in segments of L points (8, 16 or 32; 16 where N3M
// is not a multiple of L).
template <typename R>
int zpass_bkern(const c3d_channel *ch, int which, int L, std::vector<BKern> &out) {
    if (ch->g.n3m % ZL != 0) return C3D_EINVAL;
    if (L != 8 && L != 32) L = 16;
    if (ch->g.n3m % L != 0) L = 16;
    if (which == 2 && cn_far(ch, ch->dt_cached).m > 0) {   // DT of the step that is captured
        out.push_back({(const void *)kb_zCfar<R>, TPB, 0, (unsigned)nblk((long long)ch->g.n2m * (ch->g.n3m / ZL) * ch->g.n1m)});
        return 0;
    }
    if constexpr (sizeof(R) == 8) {   // joined segments, as for one channel
        switch (zjoin_len<R>(ch->g.n3m)) {
            case 8: return zbk<R, 8, 1>(ch, which, out);
            case 12: return zbk<R, 12, 1>(ch, which, out);
            case 16: return zbk<R, 16, 1>(ch, which, out);
            default: return zbk<R, 16, 0>(ch, which, out);
        }
    } else {
        if (L == 8) return zbk<R, 8, 0>(ch, which, out);
        if (L == 32) return zbk<R, 32, 0>(ch, which, out);
        return zbk<R, 16, 0>(ch, which, out);
    }
}
#if C3D_BITS == 64
template int zpass_bkern<double>(const c3d_channel *, int, int, std::vector<BKern> &);
#else
template int zpass_bkern<float>(const c3d_channel *, int, int, std::vector<BKern> &);
#endif

template <typename R>
static int launch_diag_z(c3d_channel *ch, StepArgs<R> &a, const double *divx, int *nl) {
    const Geo &g = ch->g;
    const double b = 22.0, r = -2.0 / (b + sqrt(b * b - 4.0));
    const Cyc<double> c22 = {r, -r, WM<double>::M22};
    const long long ncol = (long long)g.n2m * g.n1m;
    auto go = [&](auto *fn, int L, int cols) {
        const int nt = cols * (g.n3m / L);
        klaunch(ch, ch->stream, fn, nblk(ncol, cols), nt, 2 * (size_t)nt * sizeof(double), a, divx, c22);
    };
    switch (zjoin_len<double>(g.n3m)) {
        case 8: go(k_diag_z<R, 8, 1>, 8, zjoin_cols<double, 8>(g.n3m, ncol)); break;
        case 12: go(k_diag_z<R, 12, 1>, 12, zjoin_cols<double, 12>(g.n3m, ncol)); break;
        case 16: go(k_diag_z<R, 16, 1>, 16, zjoin_cols<double, 16>(g.n3m, ncol)); break;
        default: klaunch(ch, ch->stream, k_diag_z<R, ZL, 0>, nblk(ncol * (g.n3m / ZL)), TPB, 0, a, divx, c22);
    }
    mark(ch, nl, "diag_z", (double)ncol * g.n3m * 16);
    return 0;
}

template <typename R>
int launch_zpass(c3d_channel *ch, StepArgs<R> &a, int which, R *d0, R *d1, R *d2, int flag, int *nl) {
    if (which == 5) return launch_diag_z<R>(ch, a, (const double *)d0, nl);
    if (which == 2 && a.zfar.m > 0) {
        const Geo &g = ch->g;
        klaunch(ch, ch->stream, k_zCfar<R>, nblk((long long)g.n2m * (g.n3m / ZL) * g.n1m), TPB, 0, a, d0, d1, d2);
        mark(ch, nl, "zC", (double)g.n1m * g.n2m * g.n3m * 6 * sizeof(R));
        return 0;
    }
    const int zl = ch->tune.zl[which];
    // FP64 always joins its segments: the FP64 pipe (2 lanes per clock and SM) bounds these
    // passes, and with M = 23 warm-up points a segment of 16 evaluates 62 right-hand sides
    // for 16 results.  FP32 joins them where the schedule says 0; its short warm-ups (6 to
    // 10 points) cost less than the two block synchronisations on most shapes.
    if (sizeof(R) == 8 || zl == 0) {
        switch (zjoin_len<R>(ch->g.n3m)) {
            case 8: return launch_zpass_l<R, 8, 1>(ch, a, which, d0, d1, d2, flag, nl);
            case 12: return launch_zpass_l<R, 12, 1>(ch, a, which, d0, d1, d2, flag, nl);
            case 16: return launch_zpass_l<R, 16, 1>(ch, a, which, d0, d1, d2, flag, nl);
            default: return launch_zpass_l<R, 16, 0>(ch, a, which, d0, d1, d2, flag, nl);
        }
    }
    if constexpr (sizeof(R) == 4) {
        switch (zl) {
            case 8: return launch_zpass_l<R, 8, 0>(ch, a, which, d0, d1, d2, flag, nl);
            case 32: return launch_zpass_l<R, 32, 0>(ch, a, which, d0, d1, d2, flag, nl);
            default: break;
        }
    }
    return launch_zpass_l<R, 16, 0>(ch, a, which, d0, d1, d2, flag, nl);
}

template <typename R, int L, int MODE>
static int launch_zpass_l(c3d_channel *ch, StepArgs<R> &a, int which, R *d0, R *d1, R *d2, int flag, int *nl) {
    const Geo &g = ch->g;
    const long long nt = (long long)g.n2m * (g.n3m / L) * g.n1m, ncol = (long long)g.n2m * g.n1m;
    // MODE 0: TPB-thread blocks over all threads; MODE 1: blocks of `cols` whole lines
    const int cols = MODE == 1 ? zjoin_cols<R, L>(g.n3m, ncol) : 0;
    const dim3 nb = MODE == 1 ? dim3(nblk(ncol, cols)) : dim3(nblk(nt));
    const dim3 TB = MODE == 1 ? dim3(cols * (g.n3m / L)) : dim3(TPB);
    const dim3 nbv = MODE == 1 ? dim3(nblk(ncol - g.n1m, cols)) : nb;   // zA's v piece: J >= 2
    const size_t zs1 = MODE == 1 ? 2 * (size_t)TB.x * sizeof(R) : 0, zs2 = 2 * zs1, zsm = 3 * zs1;
    cudaStream_t st = ch->stream;
    const double N = (double)ch->g.n1m * ch->g.n2m * ch->g.n3m, Rb = sizeof(R);
    switch (which) {
        case 0:
            if (ch->tune.zsplit) {   // u, (w, P), v sweeps as three kernels
                // as concurrent branches with knob 15: each writes its own R component and
                // product, and they share only inputs that none of them writes
                const bool cc = par_on(ch);
                int rc;
                if (cc && (rc = par_fork(ch))) return rc;
                klaunch(ch, cc ? ch->par[0] : st, k_zA<R, L, 1, MODE>, nb, TB, zs2, a);
                mark(ch, nl, "zA_u", N * (8 + 4 * Rb));    // u; WW1, R1 -> R1, E_xz
                klaunch(ch, cc ? ch->par[1] : st, k_zA<R, L, 2, MODE>, nb, TB, zsm, a);
                mark(ch, nl, "zA_wp", N * (16 + 3 * Rb));  // w, P; R3 -> R3, WW3^2
                klaunch(ch, st, k_zA<R, L, 3, MODE>, nbv, TB, zs2, a);
                mark(ch, nl, "zA_v", N * (16 + 3 * Rb));   // v, w; R2 -> R2, E_yz
                if (cc && (rc = par_join(ch))) return rc;
            } else {
                klaunch(ch, st, k_zA<R, L, 0, MODE>, nb, TB, zsm, a);
                mark(ch, nl, "zA", N * (32 + 10 * Rb));
            }
            break;
        case 1: klaunch(ch, st, k_zB<R, L, MODE>, nb, TB, zsm, a); mark(ch, nl, "zB", N * 8 * Rb); break;
        case 2: klaunch(ch, st, k_zC<R, L, MODE>, nb, TB, zsm, a, d0, d1, d2); mark(ch, nl, "zC", N * 6 * Rb); break;
        case 3: klaunch(ch, st, k_zD<R, L, MODE>, nb, TB, zs1, a, d2); mark(ch, nl, "zD", N * (8 + 2 * Rb)); break;
        case 4:   // the mixed form reads delta1 - DT dDP/dx from one field (xD), FP64 both
            klaunch(ch, st, k_zE<R, L, MODE>, nb, TB, zs1, a, d0, d1, d2, flag);
            mark(ch, nl, "zE", N * (64 + (sizeof(R) == 4 ? 4 : 5) * Rb));
            break;
        default: return C3D_EINVAL;
    }
    return 0;
}

#if C3D_BITS == 64
template int launch_zpass<double>(c3d_channel *, StepArgs<double> &, int, double *, double *, double *, int, int *);
#else
template int launch_zpass<float>(c3d_channel *, StepArgs<float> &, int, float *, float *, float *, int, int *);
#endif

}  // namespace c3d
