// c3d_x64.cuh -- xA's pieces in FP64.  The FP64 pipe bounds them (two lanes per clock and SM:
// it is 84% busy and DRAM 7% at 192 x 128 x 144 points), so every constant factor is folded:
// the solves run without their scales on plain differences and sums, 1/RE and the operators'
// factors enter one multiply-add per point with the term's sum, PRESG, PRESG3 start the sums,
// and WW1 leaves without its factor 4 s (zA's u sweep applies it).
#pragma once
#include "c3d_kern.cuh"

namespace c3d {

// One row (j, k), held by W lanes with C points each, of the u (PART 1), v (PART 2, faces
// J >= 2) or w (PART 3) piece; rows as in xa_piece.
template <int C, int PART, int W = 32>
__device__ __forceinline__ void xa64(const StepArgs<double> &a, int j, long long o, long long om, long long op,
                                     int lane, int P) {
    typedef double D;
    const D RE1 = a.re1, k10 = RE1 * a.f12x * a.c10x.s;
    auto row = [&](D (&v)[C], int r) {
        drow_load(v, xa_src<false, PART>(a, r, o, om, op, (const D *)nullptr, 0), lane, P);
    };
    if constexpr (PART == 2) {
        if (j < 2) return;
        const D rh = a.m.rh[j], hp = RE1 * a.m.dyp[j], hc = -RE1 * a.m.dyc[j], hm = RE1 * a.m.dym[j], rq = 0.25 * rh;
        D acc[C], vc[C], d[C];
        row(vc, XA_VC);
        {
            D vm[C], vp[C], hh[C];
            row(vm, XA_VM);
            row(vp, XA_VP);
#pragma unroll
            for (int t = 0; t < C; ++t) {
                acc[t] = hp * vp[t] + (hc * vc[t] + hm * vm[t]);
                const D v2 = vp[t] + vc[t], v1 = vc[t] + vm[t];
                hh[t] = rq * (v2 * v2 - v1 * v1);
            }
            drow_store(a.hh[1] + o, hh, lane, P);
        }
        {
            D pc[C], pm[C];
            row(pc, XA_PC);
            row(pm, XA_PM);
#pragma unroll
            for (int t = 0; t < C; ++t) acc[t] = acc[t] - rh * (pc[t] - pm[t]);
        }
        const D pv = sprev<W>(vc[C - 1], lane, P), nx = snext<W>(vc[0], lane, P);
#pragma unroll
        for (int t = 0; t < C; ++t) {
            const D l = t == 0 ? pv : vc[t - 1], r = t == C - 1 ? nx : vc[t + 1];
            d[t] = (l - 2.0 * vc[t]) + r;
        }
        xsolve_ring<W, 10>(d, lane, P, a.c10x);
#pragma unroll
        for (int t = 0; t < C; ++t) acc[t] = acc[t] + k10 * d[t];
        drow_store(a.r[1] + o, acc, lane, P);
#pragma unroll
        for (int t = 0; t < C; ++t) d[t] = (t == 0 ? pv : vc[t - 1]) + vc[t];
        xsolve_ring<W, 6>(d, lane, P, a.c6x);
        {   // u at the y faces
            D uc[C], um[C];
            row(uc, XA_UC);
            row(um, XA_UM);
            const D k6 = 4.0 * a.c6x.s * rh, a1 = k6 * a.m.hdy[j], a2 = k6 * a.m.hdy[j - 1];
#pragma unroll
            for (int t = 0; t < C; ++t) d[t] = d[t] * (a1 * um[t] + a2 * uc[t]);
        }
        drow_store(a.exy + o, d, lane, P);
    } else {
        // u: the y stencil, the x terms (HH1 stored), -dP/dx; w: the y stencil, the x terms
        constexpr int XC = PART == 1 ? XA_UC : XA_WC, XM = PART == 1 ? XA_UM : XA_WM, XP = PART == 1 ? XA_UP : XA_WP;
        const D hp = RE1 * a.m.hp[j], hc = -RE1 * a.m.hc[j], hm = RE1 * a.m.hm[j];
        const D pg = a.scal[PART == 1 ? SCAL_PRESG : SCAL_PRESG3];
        D acc[C], xc[C], d[C];
        row(xc, XC);
        {
            D xm[C], xp[C];
            row(xm, XM);
            row(xp, XP);
#pragma unroll
            for (int t = 0; t < C; ++t) acc[t] = hp * xp[t] + (hc * xc[t] + (hm * xm[t] - pg));
        }
        const D pv = sprev<W>(xc[C - 1], lane, P), nx = snext<W>(xc[0], lane, P);
#pragma unroll
        for (int t = 0; t < C; ++t) {
            const D l = t == 0 ? pv : xc[t - 1], r = t == C - 1 ? nx : xc[t + 1];
            d[t] = (l - 2.0 * xc[t]) + r;
        }
        xsolve_ring<W, 10>(d, lane, P, a.c10x);
#pragma unroll
        for (int t = 0; t < C; ++t) acc[t] = acc[t] + k10 * d[t];
        if constexpr (PART == 3) {
            drow_store(a.r[2] + o, acc, lane, P);
#pragma unroll
            for (int t = 0; t < C; ++t) d[t] = (t == 0 ? pv : xc[t - 1]) + xc[t];
            xsolve_ring<W, 6>(d, lane, P, a.c6x);
            drow_store(a.ww1 + o, d, lane, P);
        } else {
            const D kp = a.f24x * a.c22x.s, k6 = 4.0 * a.c6x.s, kq = kp * k6 * k6;
#pragma unroll
            for (int t = 0; t < C; ++t) d[t] = xc[t] + (t == C - 1 ? nx : xc[t + 1]);
            xsolve_ring<W, 6>(d, lane, P, a.c6x);
#pragma unroll
            for (int t = 0; t < C; ++t) xc[t] = d[t] * d[t];
            const D ps = sprev<W>(xc[C - 1], lane, P);
#pragma unroll
            for (int t = 0; t < C; ++t) d[t] = xc[t] - (t == 0 ? ps : xc[t - 1]);
            xsolve_ring<W, 22>(d, lane, P, a.c22x);
#pragma unroll
            for (int t = 0; t < C; ++t) d[t] = kq * d[t];
            drow_store(a.hh[0] + o, d, lane, P);
            row(xc, XA_PC);
            const D pp = sprev<W>(xc[C - 1], lane, P);
#pragma unroll
            for (int t = 0; t < C; ++t) d[t] = xc[t] - (t == 0 ? pp : xc[t - 1]);
            xsolve_ring<W, 22>(d, lane, P, a.c22x);
#pragma unroll
            for (int t = 0; t < C; ++t) acc[t] = acc[t] - kp * d[t];
            drow_store(a.r[0] + o, acc, lane, P);
        }
    }
}

}  // namespace c3d
