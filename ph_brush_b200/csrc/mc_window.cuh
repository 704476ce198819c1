// The reciprocal-space interaction of a trial's stencils with other stencils: sums over windows of
// the influence kernel, read from its unfolded, blocked table (RepDesc::gx_*).
#pragma once
#include "common.cuh"

// Geometry of the window of G that a stencil pair reads: x in NCH chunks of four values (one
// 16-byte load), RW rows, RW planes; the two stencils of a displaced charge, whose bases differ
// by at most one point per axis, share a window one point wider.
template <int P>
struct Win {
    static constexpr int W = 2 * P - 1, RW = W + 1;
    // chunks of a row at any alignment (order 5: three, which leaves out one alignment of the wider
    // window, so that a plane's 3 x 10 chunks are one load per lane)
    static constexpr int NCH = P == 5 ? 3 : (RW + 3 + 3) / 4;
    static constexpr int RWP = (RW + 3) / 4 * 4;
    static constexpr int TAB = 4 * NCH + 2 * RWP;      // floats of one stencil's 1-D tables: x, y, z
    static constexpr int ITEMS = NCH * RW, EL = (ITEMS + 31) / 32;
};

// A charge's stencil with its weights padded by P zeros on either side, so that a shifted product
// of two stencils needs no bounds test.
template <int P>
struct PadSt {
    int base[3];
    float coef;
    int m[3][P];          // wrapped mesh coordinates
    float wp[3][3 * P];
};

template <int P>
__device__ __forceinline__ void pad_stencil_axis(PadSt<P>& s, const RepDesc& D, float4 p, int k) {
    const float pk = (k == 0) ? p.x : (k == 1 ? p.y : p.z);
    const float g = pk / D.L[k] * (float)D.mesh[k];
    const float fl = floorf(g);
    float w[P];
    bspline_weights<P>(g - fl, w);
    const int base = (int)fl + P / 2 - P + 1;
    s.base[k] = base;
#pragma unroll
    for (int j = 0; j < P; ++j) {  // base + j lies in [-P, n + P): one correction wraps it
        int m = base + j;
        m += (m < 0) ? D.mesh[k] : 0;
        m -= (m >= D.mesh[k]) ? D.mesh[k] : 0;
        s.m[k][j] = m;
        s.wp[k][j] = 0.0f; s.wp[k][P + j] = w[j]; s.wp[k][2 * P + j] = 0.0f;
    }
}

// What a lane holds of a trial's one or two stencils while its warp goes through the earlier ones:
// its axis and place in the 1-D tables, that axis's weights and bases.
template <int P>
struct LaneSt {
    int k, u, at, n;      // axis, table entry, its place in the table, mesh size
    int base0, dl;        // first stencil's base; the second's against it (minimum image)
    float w0[P], w1[P], coef0, coef1;
    bool near;            // the two bases within one point on every axis
};

// The lane's entry of the window tables: x chunks, y rows, z planes.
template <int P>
__device__ __forceinline__ void lane_place(LaneSt<P>& L, const RepDesc& D, int lane) {
    using Q = Win<P>;
    L.k = lane < 4 * Q::NCH ? 0 : (lane < 4 * Q::NCH + Q::RW ? 1 : 2);
    L.u = lane - (L.k == 0 ? 0 : (L.k == 1 ? 4 * Q::NCH : 4 * Q::NCH + Q::RW));
    L.at = L.k < 2 ? lane : lane - Q::RW + Q::RWP;
    L.n = max(1, D.mesh[L.k]);
}

template <int P>
__device__ __forceinline__ void lane_stencils(LaneSt<P>& L, const RepDesc& D, const PadSt<P>* st, int nst) {
    const PadSt<P>&a0 = st[0], &a1 = st[nst - 1];
    L.base0 = a0.base[L.k];
    int dl = a1.base[L.k] - L.base0;
    dl += (2 * dl < -L.n) ? L.n : 0;
    dl -= (2 * dl > L.n) ? L.n : 0;
    L.dl = dl;
    L.near = __all_sync(0xffffffffu, dl >= -1 && dl <= 1) && nst == 2;
    L.coef0 = a0.coef;
    L.coef1 = a1.coef;
#pragma unroll
    for (int i = 0; i < P; ++i) { L.w0[i] = a0.wp[L.k][P + i]; L.w1[i] = a1.wp[L.k][P + i]; }
}

// Sum over a window of the influence kernel G of the product of the 1-D cross-correlations of the
// trial's stencils with stencil b, times c0 (first) and c1 (second): returned per lane.
// which: 0 the first stencil, 1 the second, 2 both in one window (false if they do not share one).
// A lane takes EL 16-byte chunks of the window's (y, x) plane, the loads of all planes in flight
// (four planes at a time at order 6); FP32 over a chunk and the two stencils, FP64 over planes and
// lanes.  The two stencils' terms nearly cancel for a displaced charge, so one fma of both loses less
// than rounding each and adding them in FP64 would (error of the two terms against 64 bits at order 5 and
// displacements up to 0.3: 1.5e-7 of their sum, 2.0e-7 the other way).  What bounds it: instruction issue (~280 a window) and the loads' line lookups; the
// unfolded, blocked table puts a plane into ~6 lines of 128 bytes (12 to 24 of a folded octant).
template <int P>
__device__ __forceinline__ bool window_sum(const RepDesc& D, const float* __restrict__ G, const LaneSt<P>& L,
                                           const PadSt<P>& b, int which, float c0, float c1, float* tab, int lane, double& acc) {
    using Q = Win<P>;
    constexpr int RW = Q::RW, NCH = Q::NCH, EL = Q::EL, NTAB = 4 * NCH + 2 * RW;
    static_assert(4 * NCH + RW < 32, "each axis's first table entry in the first round");
    int lo = 0;
    const bool both = which == 2;
    __syncwarp();
#pragma unroll
    for (int e0 = 0; e0 < NTAB; e0 += 32) {
        // (order 6 has more entries than lanes: the second round's are on the last axis)
        const int k = e0 == 0 ? L.k : 2, n = e0 == 0 ? L.n : D.mesh[2];
        int u = e0 == 0 ? L.u : 32 - (4 * NCH + RW) + lane;
        const int base0 = e0 == 0 ? L.base0 : __shfl_sync(0xffffffffu, L.base0, 31);
        const int dl = e0 == 0 ? L.dl : __shfl_sync(0xffffffffu, L.dl, 31);
        // fold the bases' difference to [0, n/2], mirroring the offsets where it was negative
        int m = base0 + (which == 1 ? dl : 0) - b.base[k];
        m += (m < 0) ? n : 0;
        m += (m < 0) ? n : 0;
        m -= (m >= n) ? n : 0;
        m -= (m >= n) ? n : 0;
        const bool flip = 2 * m > n;
        const int dm = both ? min(0, flip ? -dl : dl) : 0;
        const int low = (flip ? n - m : m) + dm + 1;  // table index of the window's first point
        if (e0 == 0) lo = low;
        u -= (k == 0) ? (low & 3) : 0;
        const int o = u + dm - (P - 1);  // offset from the centre, folded frame
        const int d0 = flip ? -o : o;
        const float* wb0 = b.wp[k] + P - max(-P, min(P, d0));
        const float* wb1 = b.wp[k] + P - max(-P, min(P, d0 - dl));
        float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            float w0 = L.w0[i], w1 = L.w1[i];
            if (e0 > 0) { w0 = __shfl_sync(0xffffffffu, w0, 31); w1 = __shfl_sync(0xffffffffu, w1, 31); }
            s0 += (which == 1 ? w1 : w0) * wb0[i];
            if (both) s1 += w1 * wb1[i];
        }
        if (k == 2) { s0 *= which == 1 ? c1 : c0; s1 *= c1; }
        const int at = e0 == 0 ? L.at : 4 * NCH + Q::RWP + u;
        if (e0 + lane < NTAB) { tab[at] = s0; tab[Q::TAB + at] = s1; }
    }
    const int xl = __shfl_sync(0xffffffffu, lo, 0), yl = __shfl_sync(0xffffffffu, lo, 4 * NCH),
              zl = __shfl_sync(0xffffffffu, lo, 4 * NCH + RW);
    // (a window one wider in x may not fit the chunks at every alignment)
    if (both && (xl & 3) + Q::W + (__shfl_sync(0xffffffffu, L.dl, 0) != 0) > 4 * NCH) return false;
    __syncwarp();
    const int plane = D.gx_xb * D.gx_yb * 32;
    const float* Gw = G + (size_t)zl * plane;
    int off[EL];
    float4 wa[EL], wb[EL];
#pragma unroll
    for (int k = 0; k < EL; ++k) {
        const int it = lane + 32 * k;
        const bool in = it < Q::ITEMS;
        const int c = in ? it / RW : 0, r = in ? it - c * RW : 0;
        const int y = yl + r;
        off[k] = ((y >> 3) * D.gx_xb + (xl >> 2) + c) * 32 + (y & 7) * 4;
        const float4 x0 = *reinterpret_cast<const float4*>(tab + 4 * c);
        const float4 x1 = *reinterpret_cast<const float4*>(tab + Q::TAB + 4 * c);
        const float y0 = in ? tab[4 * NCH + r] : 0.0f, y1 = in ? tab[Q::TAB + 4 * NCH + r] : 0.0f;
        wa[k] = make_float4(x0.x * y0, x0.y * y0, x0.z * y0, x0.w * y0);
        wb[k] = make_float4(x1.x * y1, x1.y * y1, x1.z * y1, x1.w * y1);
    }
    const float* z0 = tab + 4 * NCH + Q::RWP;
    constexpr int PC = EL > 1 ? 4 : RW;  // planes in flight
#pragma unroll
    for (int d0 = 0; d0 < RW; d0 += PC) {
        float4 g[PC][EL];
#pragma unroll
        for (int dz = 0; dz < PC; ++dz)
#pragma unroll
            for (int k = 0; k < EL; ++k) g[dz][k] = __ldg(reinterpret_cast<const float4*>(Gw + (d0 + dz) * plane + off[k]));
#pragma unroll
        for (int dz = 0; dz < PC; ++dz) {
            float t = 0.0f, v = 0.0f;
#pragma unroll
            for (int k = 0; k < EL; ++k) {
                t = fmaf(wa[k].w, g[dz][k].w, fmaf(wa[k].z, g[dz][k].z, fmaf(wa[k].y, g[dz][k].y, fmaf(wa[k].x, g[dz][k].x, t))));
                v = fmaf(wb[k].w, g[dz][k].w, fmaf(wb[k].z, g[dz][k].z, fmaf(wb[k].y, g[dz][k].y, fmaf(wb[k].x, g[dz][k].x, v))));
            }
            acc += (double)fmaf(z0[d0 + dz], t, z0[Q::TAB + d0 + dz] * v);
        }
    }
    return true;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
