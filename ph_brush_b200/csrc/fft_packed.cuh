// Register-resident DFTs on packed pairs (sm_100a): the steps of rfft::rdft, same operations and
// roundings, with a complex value in one 64-bit register pair and its additions as one packed
// instruction (add/fma.f32x2) instead of two.  The packed instructions run at the rate of the
// scalar ones per operation, so this pays where instruction issue is the bound.  Inputs that are known to be
// zero leave out their butterflies: bit k of MASK says that element k may differ from zero (others
// are not read); outputs that the caller does not use are dropped by the compiler.
#pragma once
#include <cuda_runtime.h>
#include <type_traits>
#include "fft_reg.cuh"

namespace pfft {

typedef unsigned long long c2;  // (re, im)

__device__ __forceinline__ c2 pk(float x, float y) {
    c2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 up(c2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ c2 add(c2 a, c2 b) {
    c2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ c2 fma(c2 a, c2 b, c2 c) {
    c2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ c2 mul(c2 a, c2 b) {
    c2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ c2 sub(c2 a, c2 b) { return fma(b, pk(-1.0f, -1.0f), a); }  // (exact product)

// a * (c + i s), rounded as the compiler rounds cmul
__device__ __forceinline__ c2 cmulr(c2 a, float c, float s) {
    const float2 v = up(a);
    return pk(__fmaf_rn(v.x, c, -__fmul_rn(v.y, s)), __fmaf_rn(v.y, c, __fmul_rn(v.x, s)));
}
// the same of a constant of rdft<N, S>, as it rounds rfft::cmulc: of an odd multiple of an eighth
// turn the two products are shared, and others of them are fused
template <int S>
__device__ __forceinline__ c2 cmulc(c2 a, float c, float s) {
    const float2 v = up(a);
    if (c == s || c == -s) {
        const bool other = c < 0.0f && (S < 0) == (s < 0.0f);
        const float x = other && S < 0 ? __fmaf_rn(-v.y, s, __fmul_rn(v.x, c)) : __fmaf_rn(v.x, c, -__fmul_rn(v.y, s));
        const float y = other ? __fmaf_rn(v.y, c, __fmul_rn(v.x, s)) : __fmaf_rn(v.x, s, __fmul_rn(v.y, c));
        return pk(x, y);
    }
    return cmulr(a, c, s);
}

template <bool ZA, bool ZB>
__device__ __forceinline__ c2 addz(c2 a, c2 b) {
    if constexpr (ZA) return b;
    else if constexpr (ZB) return a;
    else return add(a, b);
}
// (a - b).yx
template <bool ZA, bool ZB>
__device__ __forceinline__ c2 subz_swapped(c2 a, c2 b) {
    const float2 u = up(a), v = up(b);
    if constexpr (ZA) return pk(-v.y, -v.x);
    else if constexpr (ZB) return pk(u.y, u.x);
    else return pk(__fsub_rn(u.y, v.y), __fsub_rn(u.x, v.x));
}

constexpr unsigned long long every(int n, int r, int step, unsigned long long mask) {  // bits r, r + step, ... of mask, packed
    unsigned long long m = 0;
    for (int k = r, i = 0; k < n; k += step, ++i) m |= ((mask >> k) & 1ull) << i;
    return m;
}
constexpr unsigned long long all(int n) { return n >= 64 ? ~0ull : (1ull << n) - 1ull; }

template <int N, int S, unsigned long long MASK = all(N)>
__device__ __forceinline__ void dft(c2 (&v)[N]) {
    static_assert(S == 1 || S == -1, "sign");
    static_assert((MASK & all(N)) != 0, "no input");
    constexpr float sg = (float)S;
    constexpr bool Z0 = !(MASK & 1), Z1 = !(MASK & 2), Z2 = !(MASK & 4), Z3 = !(MASK & 8);
    if constexpr (N == 1) {
    } else if constexpr ((MASK & all(N)) == 1) {
#pragma unroll
        for (int k = 1; k < N; ++k) v[k] = v[0];
    } else if constexpr (N == 2) {
        const c2 a = v[0], b = v[1];
        v[0] = addz<Z0, Z1>(a, b);
        v[1] = Z0 ? mul(b, pk(-1.0f, -1.0f)) : sub(a, b);
    } else if constexpr (N == 3) {
        const float s3 = sg * 0.86602540378443864676f;
        const c2 s = addz<Z1, Z2>(v[1], v[2]), d = subz_swapped<Z1, Z2>(v[1], v[2]);
        const c2 h = pk(-0.5f, -0.5f), m = Z0 ? mul(s, h) : fma(s, h, v[0]);
        v[0] = addz<Z0, false>(v[0], s);
        v[1] = fma(d, pk(-s3, s3), m);
        v[2] = fma(d, pk(s3, -s3), m);
    } else if constexpr (N == 4) {
        static_assert(!Z0, "first element");
        const c2 a = addz<false, Z2>(v[0], v[2]), b = Z2 ? v[0] : sub(v[0], v[2]);
        if constexpr (Z1 && Z3) {
            v[0] = a; v[2] = a; v[1] = b; v[3] = b;
        } else {
            const c2 c = addz<Z1, Z3>(v[1], v[3]), d = subz_swapped<Z1, Z3>(v[1], v[3]);
            v[0] = add(a, c); v[2] = sub(a, c);
            v[1] = fma(d, pk(-sg, sg), b);
            v[3] = fma(d, pk(sg, -sg), b);
        }
    } else {
        constexpr int R = (N % 4 == 0) ? 4 : (N % 2 == 0) ? 2 : 3;
        constexpr int M = N / R;
        static_assert(R * M == N, "length must be 2^a 3^b");
        constexpr rfft::Tw<N> T{};
        constexpr unsigned long long any = (every(N, 0, R, MASK) != 0 ? 1 : 0) | (every(N, 1, R, MASK) != 0 ? 2 : 0) |
                                           (R > 2 && every(N, 2, R, MASK) != 0 ? 4 : 0) |
                                           (R > 3 && every(N, 3, R, MASK) != 0 ? 8 : 0);  // sequences with an input
        c2 s[R][M];
        auto part = [&](auto rc) {
            constexpr int r = decltype(rc)::value;
#pragma unroll
            for (int m = 0; m < M; ++m)
                if (MASK >> (R * m + r) & 1) s[r][m] = v[R * m + r];
            if constexpr (every(N, r, R, MASK) != 0) dft<M, S, every(N, r, R, MASK)>(s[r]);
        };
        part(std::integral_constant<int, 0>{});
        part(std::integral_constant<int, 1>{});
        if constexpr (R > 2) part(std::integral_constant<int, 2>{});
        if constexpr (R > 3) part(std::integral_constant<int, 3>{});
#pragma unroll
        for (int k = 0; k < M; ++k) {
            c2 t[R];
            t[0] = s[0][k];
#pragma unroll
            for (int r = 1; r < R; ++r)
                if (any >> r & 1) t[r] = k == 0 ? s[r][k] : cmulc<S>(s[r][k], T.c[r * k], sg * T.s[r * k]);
            dft<R, S, any>(t);
#pragma unroll
            for (int q = 0; q < R; ++q) v[k + M * q] = t[q];
        }
    }
}

}  // namespace pfft
