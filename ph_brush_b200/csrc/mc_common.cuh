// Pieces shared by the Monte Carlo kernels (k_mc.cu, k_mc_run.cu): the trial's random
// words, B-spline stencils, index- and cell-list updates, the charge-mesh update.
#pragma once
#include "common.cuh"
#include "engine.h"

__device__ __forceinline__ float4 rand_pos(const RepDesc& D, uint32_t a, uint32_t b, uint32_t c) {
    float4 p;
    p.x = __fmul_rn(D.L[0], u24(a));
    p.y = __fmul_rn(D.L[1], u24(b));
    p.z = D.walls ? __fadd_rn(D.wall_lo, __fmul_rn(__fsub_rn(D.wall_hi, D.wall_lo), u24(c))) : __fmul_rn(D.L[2], u24(c));
    p.w = 0.0f;
    return p;
}

// The 16 Philox words of trial t: A = ctr (t, 0), B = ctr (t, 1), C = ctr (t, 2),
// and ctr (t, 3), whose first two words are the delayed-acceptance first-stage uniform.
__device__ __forceinline__ void trial_words(const RepDesc& D, long long t, uint32_t* w) {
    const uint32_t lo = (uint32_t)t, hi = (uint32_t)((unsigned long long)t >> 32);
    philox4x32_10(D.key[0], D.key[1], lo, hi, 0u, 0u, w);
    philox4x32_10(D.key[0], D.key[1], lo, hi, 1u, 0u, w + 4);
    philox4x32_10(D.key[0], D.key[1], lo, hi, 2u, 0u, w + 8);
    philox4x32_10(D.key[0], D.key[1], lo, hi, 3u, 0u, w + 12);
}

__device__ __forceinline__ int move_of(const RepDesc& D, uint32_t a0) {
    const float um = u24(a0);
    if (um < D.p_disp) return PHMC_MOVE_DISP;
    if (um < D.p_disp + D.p_titr) return PHMC_MOVE_TITR;
    if (um < D.p_disp + D.p_titr + D.p_swap) return PHMC_MOVE_SWAP;
    return PHMC_MOVE_NONE;
}

__device__ __forceinline__ int wrap1(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }
// i mod n for |i| within a few periods (descriptor cell offsets)
__device__ __forceinline__ int wrap_small(int i, int n) {
    while (i < 0) i += n;
    while (i >= n) i -= n;
    return i;
}

__device__ __forceinline__ void list_remove(int* list, int* pos, int& n, int so, int i) {
    const int k = pos[so + i];
    const int last = list[so + n - 1];
    list[so + k] = last; pos[so + last] = k;
    --n;
    pos[so + i] = -1;
}
__device__ __forceinline__ void list_append(int* list, int* pos, int& n, int so, int i) {
    list[so + n] = i; pos[so + i] = n; ++n;
}

__device__ __forceinline__ bool cell_remove(const DevPtrs& d, const RepDesc& D, int i) {
    const int gi = D.slot_off + i;
    const int c = d.cell_of[gi], k = d.cell_pos[gi];
    int* cnt = d.cell_count + D.cell_off + c;
    int* l = d.cell_list + ((size_t)D.cell_off + c) * D.cell_cap;
    const int n = *cnt;
    const int last = l[n - 1];
    l[k] = last; d.cell_pos[D.slot_off + last] = k;
    *cnt = n - 1;
    d.cell_of[gi] = -1; d.cell_pos[gi] = -1;
    return true;
}
__device__ __forceinline__ bool cell_insert(const DevPtrs& d, const RepDesc& D, int i, int c) {
    const int gi = D.slot_off + i;
    int* cnt = d.cell_count + D.cell_off + c;
    const int n = *cnt;
    if (n >= D.cell_cap) return false;
    d.cell_list[((size_t)D.cell_off + c) * D.cell_cap + n] = i;
    *cnt = n + 1;
    d.cell_of[gi] = c; d.cell_pos[gi] = n;
    return true;
}

__device__ __forceinline__ double slab_energy(const RepDesc& D, double Q, double Mz, double S2) {
    if (!D.slab) return 0.0;
    double e = D.slab_coef * Mz * Mz;
    if (fabs(Q) > 1e-4) e -= D.slab_coef * Q * (S2 + Q * D.Lz2_12);
    return e;
}

// (an atomic add whose result is unused does not wait for the line: the commit thread goes on)
__device__ __forceinline__ void cls_add(const DevPtrs& d, const RepDesc& D, int cell, int cls, int delta) {
    if (cls >= 0 && cell >= 0) atomicAdd(reinterpret_cast<int*>(d.cell_cls + D.cell_off + cell) + cls, delta);
}

// One warp: the charge pq added to (neg: taken out of) the band's fixed-point charge mesh,
// integer adds of the very values a full spread computes, so the mesh stays equal to a
// spread of the current configuration.
template <int P>
__device__ __forceinline__ void qmesh_update(const RepDesc& D, const DevPtrs& d, float4 pq, bool neg, int lane) {
    float w[3][P];
    int base[3];
    qmesh_stencil<P>(D, pq, w, base);
    const int nx = D.mesh[0], ny = D.mesh[1], nz = D.mesh[2];
    unsigned long long* qb = d.qband + D.qb_off;
    const int bb = lane % P, c = lane / P;  // lane (bb, c) < P^2 writes the row of P points
    int zr = base[2] + c - D.zb_lo;
    zr %= nz;
    zr += (zr < 0) ? nz : 0;
    if (lane < P * P && zr < D.zb_n) {
        float wy = 0.0f, wz = 0.0f;  // selects keep the weights in registers
#pragma unroll
        for (int j = 0; j < P; ++j) { wy = (j == bb) ? w[1][j] : wy; wz = (j == c) ? w[2][j] : wz; }
        int yb = base[1] + bb;
        yb += (yb < 0) ? ny : 0;
        yb -= (yb >= ny) ? ny : 0;
        unsigned long long* row = qb + ((size_t)zr * ny + yb) * nx;
#pragma unroll
        for (int a = 0; a < P; ++a) {
            int xa = base[0] + a;
            xa += (xa < 0) ? nx : 0;
            xa -= (xa >= nx) ? nx : 0;
            const long long v = qmesh_value(pq.w, w[0][a], wy, wz);
            atomicAdd(&row[xa], (unsigned long long)(neg ? -v : v));
        }
    }
}
