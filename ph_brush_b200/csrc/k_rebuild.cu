// Potential-mesh rebuild for meshes with even nx: three passes over the
// half-spectrum mesh of each replica's fixed-point charge mesh.
//
//  The charge mesh Q (2^40 fixed point, 64-bit integers: deterministic, order-
//  independent sums) covers the planes of each replica's wall band.  It is kept
//  current incrementally: the MC kernel adds the stencil values of every accepted
//  change (old charges out, new charges in) with integer atomics, computed with the
//  same exactly-rounded weights as the full spread (k_band_spread, run at every full
//  recompute), so Q always equals a fresh spread of the current configuration.
//
//  k_band_spread (replica, z): gather the charges whose order-P stencils reach plane
//            z from the cell list, accumulate them in a shared-memory fixed-point
//            plane, store it to Q.
//  k_rb_fwd  (replica, z): Q plane -> float, real-to-complex FFT along x (length
//            nx/2 complex FFT of packed pairs + split) and complex FFT along y;
//            writes (nx/2+1) x ny complex values.
//  k_rb_zpass / k_rb_zreg / k_rb_zband (column tiles): FFT along z, E += w theta |F|^2,
//            F *= theta, inverse FFT along z.
//  k_rb_inv  (replica, z): inverse FFT along y, complex-to-real along x; writes
//            the real potential plane.
// With hard walls the charges stay in a band of planes (RepDesc::zb_lo, zb_n) and the
// MC kernel reads the potential only there: the first and last passes run on the
// band's planes, the z pass loads and stores only those (the rest of the input is
// zero).  The unit-charge rebuild of the influence kernel computes every plane.
// Replaces the memset + k_spread_cubic + cuFFT R2C + influence kernel chain of
// the reference (MC/src/pme.cu:140-249,362,384-422).
#include <algorithm>
#include "common.cuh"
#include "engine.h"
#include "fft.cuh"
#include "fft_reg.cuh"
#include "fft_packed.cuh"

// sum of |q| up to which a block of the spread adds in 32-bit halves
constexpr float spread_qmax(int order) { return order == 4 ? 6900.0f : 9000.0f; }

// One block per (replica, ZP consecutive band planes): the charges whose order-P stencils reach
// them, from the cell list, added into fixed-point planes in shared memory.  A value (2^-40 units, 41 bits) is
// added as two 32-bit halves, its low 20 bits and the rest, since 64-bit adds in shared memory are
// compare-and-swap loops.  The low halves hold the sums of 4095 charges; the upper ones hold |q| w^3 2^20
// below 2^31 at a point, w the largest 1-D weight (2/3, 115/192, 11/20 at order 4, 5, 6): 6912, 9531,
// 12309 units in all.  Planes that more reach (spread_qmax: a little less, for the roundings down
// and the FP32 sum of |q|) are done over with 64-bit adds.  A warp takes 32 cells at a time, one per
// lane for the counts, then one lane per member; those that reach the plane (~40 %) queue up and
// are added 32 at a time: issue and the adds' bank conflicts bound it (half of either's peak).  Measured on 64 replicas of 8.7k particles: 300 us
// with 64-bit adds, 262 us as global integer adds, 197 us in 32-bit halves, 182 us two planes at a
// time; of 5k: 143 us, 111 us three planes at a time; one replica of 11.7k: 40 -> 24 us.
template <int P, int ZP, int NT>
__global__ void __launch_bounds__(NT) k_band_spread(DevPtrs d, const int2* __restrict__ jobs) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    constexpr int NW = NT / 32;
    __shared__ float4 s_queue[NW][64];
    __shared__ int s_n;
    __shared__ float s_qsum;
    const int2 job = jobs[blockIdx.x];
    const int r = job.x;
    const RepDesc& D = d.desc[r];
    const int nx = D.mesh[0], ny = D.mesh[1], nz = D.mesh[2], np = nx * ny;
    const int planes = ZP > 1 ? min(ZP, D.zb_n - job.y) : 1;  // band planes job.y .. job.y + planes - 1
    const int z = D.zb_lo + job.y - (D.zb_lo + job.y >= nz ? nz : 0);
    const int all = planes * np;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4* queue = s_queue[warp];
    unsigned* s_lo = reinterpret_cast<unsigned*>(sm_raw);
    int* s_hi = reinterpret_cast<int*>(sm_raw) + all;
    unsigned long long* s_64 = reinterpret_cast<unsigned long long*>(sm_raw);
    // floor(g_z) of a contributing charge lies in [z - P/2, z + planes - 1 - P/2 + P - 1] (mod nz)
    const float hz = D.L[2] / (float)nz;
    const float zlo = (float)(z - P / 2) * hz, zhi = (float)(z + planes - 1 - P / 2 + P) * hz;
    const int ncz = D.ncell[2], ncxy = D.ncell[0] * D.ncell[1];
    // the cell layers of [zlo, zhi), widened by a rounding margin (the exact test is per charge)
    int c_lo = (int)floorf((zlo - 1e-3f * hz) * D.cell_scale[2]), c_hi = (int)floorf((zhi + 1e-3f * hz) * D.cell_scale[2]);
    int nlay = c_hi - c_lo + 1;
    if (nlay > ncz) { nlay = ncz; c_lo = 0; }
    c_lo %= ncz;
    c_lo += (c_lo < 0) ? ncz : 0;
    const int ncell = nlay * ncxy;
    for (int wide = 0; wide < 2; ++wide) {
        for (int i = tid; i < all; i += NT) s_64[i] = 0ull;
        if (tid == 0) { s_n = 0; s_qsum = 0.0f; }
        __syncthreads();
        int n_in = 0, nh = 0;
        float q_in = 0.0f;
        auto add = [&](float4 pq) {
            float w[3][P];
            int base[3];
            qmesh_stencil<P>(D, pq, w, base);
            int ci = z - base[2];
            ci %= nz;
            ci += (ci < 0) ? nz : 0;
            ++n_in;
            q_in += fabsf(pq.w);
            int xa[P];
#pragma unroll
            for (int aa = 0; aa < P; ++aa) {
                xa[aa] = base[0] + aa;
                xa[aa] += (xa[aa] < 0) ? nx : 0;
                xa[aa] -= (xa[aa] >= nx) ? nx : 0;
            }
            for (int q = 0; q < planes; ++q) {  // (one plane: no loop)
                int cq = ci + q;
                cq -= (cq >= nz) ? nz : 0;
                if (ZP > 1 && cq >= P) continue;
                float wz = 0.0f;  // select: w[2][cq] without a dynamic index
#pragma unroll
                for (int j = 0; j < P; ++j) wz = (j == cq) ? w[2][j] : wz;
#pragma unroll
                for (int bb = 0; bb < P; ++bb) {
                    int yb = base[1] + bb;
                    yb += (yb < 0) ? ny : 0;
                    yb -= (yb >= ny) ? ny : 0;
                    yb = q * np + yb * nx;
#pragma unroll
                    for (int aa = 0; aa < P; ++aa) {
                        const long long v = qmesh_value(pq.w, w[0][aa], w[1][bb], wz);
                        if (wide) atomicAdd(&s_64[yb + xa[aa]], (unsigned long long)v);
                        else {
                            atomicAdd(&s_lo[yb + xa[aa]], (unsigned)(v & 0xfffff));
                            atomicAdd(&s_hi[yb + xa[aa]], (int)(v >> 20));
                        }
                    }
                }
            }
        };
        for (int g = warp * 32; g < ncell; g += NW * 32) {
            const int cc = g + lane;
            int cell = 0, cnt = 0;
            if (cc < ncell) {  // layer c_lo + cc / ncxy (wrapped), in-layer index cc % ncxy: consecutive cells
                cell = c_lo * ncxy + cc;
                cell -= (cell >= ncz * ncxy) ? ncz * ncxy : 0;
                cnt = min(d.cell_count[D.cell_off + cell], D.cell_cap);
            }
            int ofs = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, ofs, o);
                if (lane >= o) ofs += y;
            }
            const int m = __shfl_sync(0xffffffffu, ofs, 31);
            ofs -= cnt;
            for (int i0 = 0; i0 < m; i0 += 32) {
                const int i = i0 + lane;
                int h = 0;  // last cell of the 32 whose offset is <= i
#pragma unroll
                for (int st = 16; st > 0; st >>= 1)
                    if (__shfl_sync(0xffffffffu, ofs, h + st) <= i) h += st;
                const int hc = __shfl_sync(0xffffffffu, cell, h), ho = __shfl_sync(0xffffffffu, ofs, h);
                bool hit = false;
                float4 pq = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < m) {
                    pq = d.posq[D.slot_off + d.cell_list[((size_t)D.cell_off + hc) * D.cell_cap + i - ho]];
                    if (pq.w != 0.0f) {  // the stencil's first plane, as qmesh_axis has it
                        int ci = z - ((int)floorf(__fmul_rn(__fdiv_rn(pq.z, D.L[2]), (float)nz)) + P / 2 - P + 1);
                        ci %= nz;
                        ci += (ci < 0) ? nz : 0;
                        hit = ci < P || ci + planes > nz;
                    }
                }
                const unsigned hm = __ballot_sync(0xffffffffu, hit);
                if (hit) queue[nh + __popc(hm & ((1u << lane) - 1u))] = pq;
                nh += __popc(hm);
                if (nh >= 32) {
                    __syncwarp();
                    add(queue[lane]);
                    const float4 rest = queue[32 + lane];
                    __syncwarp();
                    if (lane < nh - 32) queue[lane] = rest;
                    nh -= 32;
                }
            }
        }
        __syncwarp();
        if (lane < nh) add(queue[lane]);
        if (n_in) { atomicAdd(&s_n, n_in); atomicAdd(&s_qsum, q_in); }
        __syncthreads();
        unsigned long long* q = d.qband + D.qb_off + (size_t)job.y * np;
        const bool fits = s_n <= 4095 && s_qsum <= spread_qmax(P);
        if (wide || fits) {
            for (int i = tid; i < all; i += NT)
                q[i] = wide ? s_64[i] : (unsigned long long)(((long long)s_hi[i] << 20) + (long long)s_lo[i]);
            return;
        }
        __syncthreads();
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) k_rb_fwd(DevPtrs d, const int2* __restrict__ jobs, int unit_charge,
                                               const int* __restrict__ dirty) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    const int2 job = jobs[blockIdx.x];
    const int r = job.x, z = job.y;
    if (dirty && !dirty[r]) return;
    const RepDesc& D = d.desc[r];
    const int nx = D.mesh[0], ny = D.mesh[1], nz = D.mesh[2];
    const int M = nx / 2, nxh = M + 1;
    // two complex buffers of nxh x ny; the real plane Q[y][x] (row length nx) is loaded as
    // the packed pairs a[y*M + j] = (Q[y][2j], Q[y][2j+1])
    float2* a = reinterpret_cast<float2*>(sm_raw);
    float2* b = a + nxh * ny;
    const int tid = threadIdx.x;
    if (unit_charge) {  // a unit charge on mesh point 0 (the influence kernel's source)
        for (int i = tid; i < M * ny; i += NT) a[i] = make_float2((z == 0 && i == 0) ? 1.0f : 0.0f, 0.0f);
    } else {
        int zrel = z - D.zb_lo;
        zrel += (zrel < 0) ? nz : 0;
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(d.qband + D.qb_off + (size_t)zrel * nx * ny);
        for (int i = tid; i < M * ny; i += NT) {
            const ulonglong2 v = q[i];
            a[i] = make_float2((float)((double)(long long)v.x * PHMC_FIX_INV), (float)((double)(long long)v.y * PHMC_FIX_INV));
        }
    }
    __syncthreads();
    float2* zr = fft_lines<NT>(a, b, M, ny, M, 1, d.twiddle + D.tw_off_h, -1.0f, false);
    float2* xo = (zr == a) ? b : a;
    const float2* twn = d.twiddle + D.tw_off[0];  // exp(-2 pi i k / nx)
    // split: X_k = 1/2 (Z_k + conj Z_{M-k}) - i/2 W^k (Z_k - conj Z_{M-k}), k = 0..M
    for (int i = tid; i < nxh * ny; i += NT) {
        const int y = i / nxh, k = i - y * nxh;
        const float2 zk = zr[y * M + (k == M ? 0 : k)];
        float2 zc = zr[y * M + (k == 0 ? 0 : M - k)];
        zc.y = -zc.y;
        const float2 w = twn[k];
        const float2 s = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
        const float2 df = make_float2(0.5f * (zk.x - zc.x), 0.5f * (zk.y - zc.y));
        const float2 wd = cmul(w, df);  // W * (Z_k - conj Z_{M-k}) / 2
        xo[y * nxh + k] = make_float2(s.x + wd.y, s.y - wd.x);  // s - i * wd
    }
    __syncthreads();
    float2* res = fft_lines<NT>(xo, zr, ny, nxh, 1, nxh, d.twiddle + D.tw_off[1], -1.0f, true);
    float2* c = d.cmesh + D.meshh_off + (size_t)z * ny * nxh;
    for (int i = tid; i < nxh * ny; i += NT) c[i] = res[i];
}

// The z pass of any nz = 2^a 3^b 5^c: TX consecutive columns of the flattened half-spectrum plane,
// job = (replica, first column, columns, 0), Stockham stages of fft_lines' radices, operations and
// roundings.  A thread stays on one column; the first stage takes its inputs from global memory (without its
// twiddles, which are one), the last forward stage leaves its outputs times theta, the last
// inverse stage stores the band's planes: for s stages 2 s - 1 round trips through shared memory
// instead of 2 s + 3.  Bound by instruction issue and those round trips: 24 uneven replicas (18k
// columns of 192 to 288 planes) 69 -> 29 us, one without walls (1.9k columns, fewer blocks than SMs) 43 -> 32 us.
template <int R, bool FIRST, int NT, int TX, class Load, class Store>
__device__ __forceinline__ void zstage(int n, int Ns, const float2* __restrict__ tw, float sign, Load ld, Store st) {
    const int nb = n / R, ts = n / (Ns * R);
    const FastDiv dns(Ns);
    for (int j = threadIdx.x / TX; j < nb; j += NT / TX) {
        int k = 0, jq = j;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ld(j + r * nb);
        if constexpr (!FIRST) {
            jq = dns.div(j, k);
#pragma unroll
            for (int r = 1; r < R; ++r) {
                float2 w = __ldg(&tw[r * k * ts]);
                if (sign > 0.0f) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        dft_radix(v, R, sign);
        const int idx = jq * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) st(idx + r * Ns, v[r]);
    }
    __syncthreads();
}

template <int NT, int TX>
__global__ void __launch_bounds__(NT) k_rb_zpass(DevPtrs d, const int4* __restrict__ jobs, double* __restrict__ epart,
                                                 const int* __restrict__ dirty, int full) {
    static_assert(NT % TX == 0, "a thread stays on one column");
    extern __shared__ float2 sm[];
    __shared__ double red[40];
    const int4 job = jobs[blockIdx.x];
    const int r = job.x, c0 = job.y, ncol = job.z;
    if (dirty && !dirty[r]) { if (threadIdx.x == 0) epart[blockIdx.x] = 0.0; return; }
    const RepDesc& D = d.desc[r];
    const int nxh = D.mesh[0] / 2 + 1, nz = D.mesh[2], plane = D.mesh[1] * nxh;
    const int col = threadIdx.x % TX;
    const bool valid = col < ncol;
    float2* a = sm + col;
    float2* b = a + TX * nz;
    float2* c = d.cmesh + D.meshh_off + c0 + col;
    const float2* tw = d.twiddle + D.tw_off[2];
    const float2* thz = d.thtab + D.th_off[2];
    // planes outside the wall band hold no charge (zero input) and are not read back
    const int zlo = full ? 0 : D.zb_lo, zbn = full ? nz : D.zb_n;
    auto in_band = [&](int z) { int t = z - zlo; t += (t < 0) ? nz : 0; return valid && t < zbn; };
    const int idx = c0 + col, y = idx / nxh, kx = idx - y * nxh;
    const float2 fx = valid ? d.thtab[D.th_off[0] + kx] : make_float2(0.0f, 1.0f);
    const float2 fy = valid ? d.thtab[D.th_off[1] + y] : make_float2(0.0f, 1.0f);
    const float cxy = D.th_c * fx.x * fy.x, kxy2 = fx.y + fy.y;
    const float wgt = (kx == 0 || kx == nxh - 1) ? 1.0f : 2.0f;  // half spectrum, Hermitian partners counted
    double e_loc = 0.0;
    auto global = [&](int z) { return in_band(z) ? c[(size_t)z * plane] : make_float2(0.f, 0.f); };
    auto shared = [&](int z) { return a[z * TX]; };
    auto keep = [&](int z, float2 v) { b[z * TX] = v; };
    auto scale = [&](int kz, float2 F) {  // theta = th_c tx ty tz / |k|^2 from the per-axis factor tables
        const float2 fz = __ldg(&thz[kz]);
        float th = __fdividef(cxy * fz.x, kxy2 + fz.y);
        if (kz == 0 && idx == 0) th = 0.0f;
        e_loc += (double)(wgt * th) * ((double)F.x * F.x + (double)F.y * F.y);
        b[kz * TX] = make_float2(__fmul_rn(F.x, th), __fmul_rn(F.y, th));
    };
    auto store = [&](int z, float2 v) { if (in_band(z)) c[(size_t)z * plane] = v; };
    auto stages = [&](float sign, auto first, auto last) {
        auto one = [&](auto rc, int Ns, int m) {
            constexpr int R = decltype(rc)::value;
            if (Ns == 1) {
                if (m == R) zstage<R, true, NT, TX>(nz, Ns, tw, sign, first, last);
                else zstage<R, true, NT, TX>(nz, Ns, tw, sign, first, keep);
            } else if (m == R) zstage<R, false, NT, TX>(nz, Ns, tw, sign, shared, last);
            else zstage<R, false, NT, TX>(nz, Ns, tw, sign, shared, keep);
            float2* t = a; a = b; b = t;
        };
        for (int Ns = 1, m = nz; m > 1;) {
            const int R = m % 4 == 0 ? 4 : (m % 2 == 0 ? 2 : (m % 3 == 0 ? 3 : 5));
            if (R == 4) one(std::integral_constant<int, 4>{}, Ns, m);
            else if (R == 2) one(std::integral_constant<int, 2>{}, Ns, m);
            else if (R == 3) one(std::integral_constant<int, 3>{}, Ns, m);
            else one(std::integral_constant<int, 5>{}, Ns, m);
            Ns *= R;
            m /= R;
        }
    };
    stages(-1.0f, global, scale);
    stages(1.0f, shared, store);
    const double s = block_sum<NT>(e_loc, red);
    if (threadIdx.x == 0) epart[blockIdx.x] = 0.5 * s;
}

// z pencils with register-resident DFTs, nz = N1 * N2: TX consecutive columns of the
// flattened half-spectrum plane (ny x (nx/2+1)); job = (replica, first column, columns, 0).
//   stage A: per (n2, column) the length-N1 DFT over x[N2 n1 + n2] straight from global
//            memory, times W_nz^(n2 k1), into shared memory at [k1][n2];
//   stage B: per (k1, column) the length-N2 DFT over n2 gives F(kz = k1 + N1 k2);
//            E += w theta |F|^2, F *= theta; the inverse length-N2 DFT and W_nz^(-n2 k1)
//            go back to the same shared-memory row;
//   stage A': per (n2, column) the inverse length-N1 DFT over k1, stored to global memory.
// Shared memory is touched twice per direction instead of once per radix stage.
template <int N1, int N2, int NT, int TX>
__global__ void __launch_bounds__(NT) k_rb_zreg(DevPtrs d, const int4* __restrict__ jobs, double* __restrict__ epart,
                                                const int* __restrict__ dirty, int full) {
    constexpr int N = N1 * N2;
    static_assert((TX & (TX - 1)) == 0, "TX must be a power of two");
    extern __shared__ float2 sm[];
    __shared__ double red[40];
    const int4 job = jobs[blockIdx.x];
    const int r = job.x, c0 = job.y, ncol = job.z;
    if (dirty && !dirty[r]) { if (threadIdx.x == 0) epart[blockIdx.x] = 0.0; return; }
    const RepDesc& D = d.desc[r];
    const int nx = D.mesh[0], ny = D.mesh[1];
    const int M = nx / 2, nxh = M + 1;
    const size_t plane = (size_t)ny * nxh;
    float2* s = sm;            // [k1][n2][column]
    float2* tw = sm + N * TX;  // exp(-2 pi i j / nz)
    float2* thz = tw + N;      // z influence factor and k_z^2 per kz
    float2* c = d.cmesh + D.meshh_off + c0;
    // planes outside the wall band hold no charge (zero input) and are not read back
    const int zlo = full ? 0 : D.zb_lo, zbn = full ? N : D.zb_n;
    auto in_band = [&](int z) { int t = z - zlo; t += (t < 0) ? N : 0; return t < zbn; };
    for (int i = threadIdx.x; i < N; i += NT) { tw[i] = d.twiddle[D.tw_off[2] + i]; thz[i] = d.thtab[D.th_off[2] + i]; }
    // stage A: the loads of the first round go out before the barrier that publishes tw
    for (int base = 0; base < N2 * TX; base += NT) {
        const int it = base + threadIdx.x;
        const int n2 = it / TX, col = it & (TX - 1);
        const bool act = it < N2 * TX;
        float2 v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1)
            v[n1] = (act && col < ncol && in_band(N2 * n1 + n2)) ? c[(size_t)(N2 * n1 + n2) * plane + col]
                                                                 : make_float2(0.f, 0.f);
        if (base == 0) __syncthreads();
        if (act) {
            rfft::rdft<N1, -1>(v);
            s[n2 * TX + col] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) s[(k1 * N2 + n2) * TX + col] = cmul(v[k1], tw[n2 * k1]);
        }
    }
    __syncthreads();
    double e_loc = 0.0;
    for (int it = threadIdx.x; it < N1 * TX; it += NT) {
        const int k1 = it / TX, col = it & (TX - 1);
        float2 u[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) u[n2] = s[(k1 * N2 + n2) * TX + col];
        rfft::rdft<N2, -1>(u);
        const int idx = c0 + col;
        const int y = idx / nxh, kx = idx - y * nxh;
        const bool valid = col < ncol;
        // theta = th_c tx ty tz / |k|^2 from the per-axis factor tables (column part once)
        const float2 fx = valid ? d.thtab[D.th_off[0] + kx] : make_float2(0.0f, 1.0f);
        const float2 fy = valid ? d.thtab[D.th_off[1] + y] : make_float2(0.0f, 1.0f);
        const float cxy = D.th_c * fx.x * fy.x, kxy2 = fx.y + fy.y;
        const float wgt = (kx == 0 || kx == M) ? 1.0f : 2.0f;  // half spectrum, Hermitian partners counted
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
            const int kz = k1 + N1 * k2;
            const float2 F = u[k2];
            float th = 0.0f;
            if (valid && !(kx == 0 && y == 0 && kz == 0)) {
                const float2 fz = thz[kz];
                th = __fdividef(cxy * fz.x, kxy2 + fz.y);
                e_loc += (double)(wgt * th) * ((double)F.x * F.x + (double)F.y * F.y);
            }
            u[k2] = make_float2(F.x * th, F.y * th);
        }
        rfft::rdft<N2, 1>(u);
        s[k1 * N2 * TX + col] = u[0];
#pragma unroll
        for (int n2 = 1; n2 < N2; ++n2) {
            float2 w = tw[n2 * k1];
            w.y = -w.y;
            s[(k1 * N2 + n2) * TX + col] = cmul(u[n2], w);
        }
    }
    __syncthreads();
    for (int it = threadIdx.x; it < N2 * TX; it += NT) {
        const int n2 = it / TX, col = it & (TX - 1);
        float2 v[N1];
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) v[k1] = s[(k1 * N2 + n2) * TX + col];
        rfft::rdft<N1, 1>(v);
        if (col < ncol) {
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1)
                if (in_band(N2 * n1 + n2)) c[(size_t)(N2 * n1 + n2) * plane + col] = v[n1];
        }
    }
    const double es = block_sum<NT>(e_loc, red);
    if (threadIdx.x == 0) epart[blockIdx.x] = 0.5 * es;
}

// The register z pass of a band that lies in the first third of the planes and wraps by less than
// N2 of them (walls at the bottom of a padded box): of the N1 decimated inputs n1 only the first
// H1 and the last can hold charge, and only those outputs are read, so the first level of the
// forward and the last of the inverse transform mostly fall away.  Same operations otherwise, bit
// for bit; values packed in pairs, the column's factors once per thread, twiddles at [k1][n2] so
// that both stages read them at constant offsets.  Instruction issue bounds both passes: 63 -> 41
// million warp instructions and 82 -> 57 us for 64 replicas (61k columns of 243 planes).  Taken
// wherever every replica's band fits it; a band elsewhere, no walls and the influence kernel's unit
// charge take k_rb_zreg.
constexpr int zband_lead(int n1) { return (n1 + 2) / 3 + 1; }

// blocks per SM asked of the compiler: 64 registers a thread hold transforms of up to 18 values, 80 longer ones
constexpr int zband_blocks(int n1, int n2, int nt) { return 65536 / ((n1 > 18 || n2 > 18 ? 80 : 64) * nt); }

template <int N1, int N2, int NT, int TX>
__global__ void __launch_bounds__(NT, zband_blocks(N1, N2, NT)) k_rb_zband(DevPtrs d, const int4* __restrict__ jobs, double* __restrict__ epart,
                                                 const int* __restrict__ dirty) {
    constexpr int N = N1 * N2, H1 = zband_lead(N1);
    constexpr unsigned long long MASK = pfft::all(H1) | 1ull << (N1 - 1);
    static_assert((TX & (TX - 1)) == 0 && NT % TX == 0, "a thread stays on one column");
    extern __shared__ float2 sm[];
    __shared__ double red[40];
    using pfft::c2;
    const int4 job = jobs[blockIdx.x];
    const int r = job.x, c0 = job.y, ncol = job.z;
    if (dirty && !dirty[r]) { if (threadIdx.x == 0) epart[blockIdx.x] = 0.0; return; }
    const RepDesc& D = d.desc[r];
    const int nxh = D.mesh[0] / 2 + 1, plane = D.mesh[1] * nxh;
    c2* s = reinterpret_cast<c2*>(sm);  // [k1][n2][column]
    float2* tw = sm + N * TX;           // exp(-2 pi i n2 k1 / nz) at [k1][n2]
    float2* thz = tw + N;               // z influence factor and k_z^2 per kz
    const int col = threadIdx.x & (TX - 1);
    const bool valid = col < ncol;
    c2* c = reinterpret_cast<c2*>(d.cmesh + D.meshh_off + c0) + col;
    // the band: planes [za, zb) and, where it wraps, [zc, N)
    const bool wraps = D.zb_lo + D.zb_n > N;
    const int za = wraps ? 0 : D.zb_lo, zb = D.zb_lo + D.zb_n - (wraps ? N : 0), zc = wraps ? D.zb_lo : N;
    for (int i = threadIdx.x; i < N; i += NT) {
        const int k1 = i / N2;
        tw[i] = d.twiddle[D.tw_off[2] + k1 * (i - k1 * N2)];
        thz[i] = d.thtab[D.th_off[2] + i];
    }
    const int idx = c0 + col, y = idx / nxh, kx = idx - y * nxh;
    const float2 fx = valid ? d.thtab[D.th_off[0] + kx] : make_float2(0.0f, 1.0f);
    const float2 fy = valid ? d.thtab[D.th_off[1] + y] : make_float2(0.0f, 1.0f);
    const float cxy = D.th_c * fx.x * fy.x, kxy2 = fx.y + fy.y;
    const float wgt = (kx == 0 || kx == nxh - 1) ? 1.0f : 2.0f;  // half spectrum, Hermitian partners counted
    auto in = [&](int n1, int z) { return n1 < H1 ? (unsigned)(z - za) < (unsigned)(zb - za) : z >= zc; };
    // stage A: the loads of the first round go out before the barrier that publishes tw
    for (int base = 0; base < N2 * TX; base += NT) {
        const int n2 = (base + (int)threadIdx.x) / TX;
        const bool act = n2 < N2;
        c2 v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1)
            if (MASK >> n1 & 1) {
                v[n1] = 0ull;
                if (act && valid && in(n1, N2 * n1 + n2)) v[n1] = c[(size_t)(N2 * n1 + n2) * plane];
            }
        if (base == 0) __syncthreads();
        if (act) {
            pfft::dft<N1, -1, MASK>(v);
            s[n2 * TX + col] = v[0];
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1) {
                const float2 w = tw[k1 * N2 + n2];
                s[(k1 * N2 + n2) * TX + col] = pfft::cmulr(v[k1], w.x, w.y);
            }
        }
    }
    __syncthreads();
    double e_loc = 0.0;
    for (int k1 = threadIdx.x / TX; k1 < N1; k1 += NT / TX) {
        c2 u[N2];
        c2* sk = s + k1 * N2 * TX + col;
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) u[n2] = sk[n2 * TX];
        pfft::dft<N2, -1>(u);
        float2 f[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) {
            const float2 F = pfft::up(u[k2]), fz = thz[k1 + N1 * k2];
            // theta = th_c tx ty tz / |k|^2 from the per-axis factor tables
            float th = __fdividef(cxy * fz.x, kxy2 + fz.y);
            if (k2 == 0 && k1 == 0 && idx == 0) th = 0.0f;
            e_loc += (double)(wgt * th) * ((double)F.x * F.x + (double)F.y * F.y);
            f[k2] = k2 < N2 - 1 ? make_float2(__fmul_rn(F.x, th), __fmul_rn(F.y, th)) : make_float2(F.x * th, F.y * th);
        }
        rfft::rdft<N2, 1>(f);  // (scalar: k_rb_zreg's roundings, which fuse the last product into its addition)
        sk[0] = pfft::pk(f[0].x, f[0].y);
#pragma unroll
        for (int n2 = 1; n2 < N2; ++n2) {
            float2 w = tw[k1 * N2 + n2];
            w.y = -w.y;
            const float2 t = cmul(f[n2], w);
            sk[n2 * TX] = pfft::pk(t.x, t.y);
        }
    }
    __syncthreads();
    for (int n2 = threadIdx.x / TX; n2 < N2; n2 += NT / TX) {
        c2 v[N1];
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) v[k1] = s[(k1 * N2 + n2) * TX + col];
        pfft::dft<N1, 1>(v);
        if (valid) {
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1)
                if (MASK >> n1 & 1)
                    if (in(n1, N2 * n1 + n2)) c[(size_t)(N2 * n1 + n2) * plane] = v[n1];
        }
    }
    const double es = block_sum<NT>(e_loc, red);
    if (threadIdx.x == 0) epart[blockIdx.x] = 0.5 * es;
}

// (id, nz, N1, N2) of the register z passes; id 0 = shared-memory z pass.  The first entry
// of an nz is its default; the others are the splits the autotuner also tries.
#define ZREG_LIST(X) X(1, 48, 8, 6) X(2, 128, 16, 8) X(3, 162, 18, 9) X(4, 192, 16, 12) X(5, 216, 24, 9) \
                     X(6, 243, 27, 9) X(7, 256, 16, 16) X(8, 288, 32, 9) X(9, 384, 32, 12)            \
                     X(10, 48, 6, 8) X(11, 128, 8, 16) X(12, 162, 9, 18) X(13, 192, 12, 16)           \
                     X(14, 216, 9, 24) X(15, 243, 9, 27) X(16, 288, 9, 32) X(17, 384, 24, 16)         \
                     X(18, 384, 12, 32)
constexpr int ZREG_NT(int n2) { return (n2 * ZREG_TX + 31) / 32 * 32 > 256 ? 256 : (n2 * ZREG_TX + 31) / 32 * 32; }

int zreg_variant(int nz) {
#define ZREG_CASE(id, n, a, b) if (nz == n) return id;
    ZREG_LIST(ZREG_CASE)
#undef ZREG_CASE
    return 0;
}
int zreg_variants(int nz, int* ids, int max_ids) {
    int n = 0;
#define ZREG_ALL(id, nn, a, b) if (nz == nn && n < max_ids) ids[n++] = id;
    ZREG_LIST(ZREG_ALL)
#undef ZREG_ALL
    return n;
}
void zreg_split(int id, int* n1, int* n2) {
    *n1 = 0; *n2 = 0;
#define ZREG_SPLIT(i, nn, a, b) if (id == i) { *n1 = a; *n2 = b; }
    ZREG_LIST(ZREG_SPLIT)
#undef ZREG_SPLIT
}
bool zband_fits(int id, int nz, int zb_lo, int zb_n) {
    int n1 = 0, n2 = 0;
    zreg_split(id, &n1, &n2);
    const bool wraps = zb_lo + zb_n > nz;
    const int end = zb_lo + zb_n - (wraps ? nz : 0);
    return n2 > 0 && end <= zband_lead(n1) * n2 && zband_lead(n1) < n1 && (!wraps || zb_lo >= nz - n2);
}
size_t zreg_smem(int nz) { return (size_t)(ZREG_TX + 2) * nz * sizeof(float2); }

template <int NT>
__global__ void __launch_bounds__(NT) k_rb_inv(DevPtrs d, const int2* __restrict__ jobs, const int* __restrict__ dirty) {
    extern __shared__ float2 sm[];
    const int2 job = jobs[blockIdx.x];
    const int r = job.x, z = job.y;
    if (dirty && !dirty[r]) return;
    const RepDesc& D = d.desc[r];
    const int nx = D.mesh[0], ny = D.mesh[1];
    const int M = nx / 2, nxh = M + 1;
    float2* a = sm;
    float2* b = sm + nxh * ny;
    const float2* c = d.cmesh + D.meshh_off + (size_t)z * ny * nxh;
    for (int i = threadIdx.x; i < nxh * ny; i += NT) a[i] = c[i];
    __syncthreads();
    float2* xr = fft_lines<NT>(a, b, ny, nxh, 1, nxh, d.twiddle + D.tw_off[1], 1.0f, true);
    float2* zo = (xr == a) ? b : a;
    const float2* twn = d.twiddle + D.tw_off[0];
    // merge: Z'_k = (X_k + conj X_{M-k}) + i W^{-k} (X_k - conj X_{M-k}), k = 0..M-1
    for (int i = threadIdx.x; i < M * ny; i += NT) {
        const int y = i / M, k = i - y * M;
        const float2 A = xr[y * nxh + k];
        float2 B = xr[y * nxh + (M - k)];
        B.y = -B.y;
        float2 w = twn[k];
        w.y = -w.y;  // W^{-k}
        const float2 s = make_float2(A.x + B.x, A.y + B.y);
        const float2 wd = cmul(w, make_float2(A.x - B.x, A.y - B.y));
        zo[y * M + k] = make_float2(s.x - wd.y, s.y + wd.x);  // s + i * wd
    }
    __syncthreads();
    float2* zz = fft_lines<NT>(zo, xr, M, ny, M, 1, d.twiddle + D.tw_off_h, 1.0f, false);
    float* phi = d.phi + D.mesh_off + (size_t)z * ny * nx;
    for (int i = threadIdx.x; i < M * ny; i += NT) {
        const int y = i / M, j = i - y * M;
        phi[y * nx + 2 * j] = zz[i].x;
        phi[y * nx + 2 * j + 1] = zz[i].y;
    }
}

// ---------------------------------------------------------------------------
// ---------------------------------------------------------------------------
// First and last passes with register-resident DFTs, for square lateral meshes
// n = nx = ny in the PLANE_LIST set (one block per (replica, z) plane, the
// replica's n picked at run time).  x: one thread per row, the row's n/2 packed
// complex values in registers (a row stride of odd length in float2 keeps the
// rows' shared-memory accesses free of bank conflicts); y: n = N1 * N2 in two
// register stages over the n/2 + 1 columns.  Shared memory is passed once per
// stage instead of once per radix stage.
// ---------------------------------------------------------------------------
#define PLANE_LIST(X) X(16, 4, 4) X(32, 8, 4) X(36, 6, 6) X(48, 8, 6) X(54, 9, 6) X(64, 8, 8)
constexpr int plane_ms(int m) { return (m % 2 == 0) ? m + 1 : m + 2; }  // odd row stride (float2)
constexpr int PLANE_NT = 128;
constexpr int PLANE_STAGE_BYTES = 64 * 64 * 8;  // one staged plane of the largest listed lateral mesh

// qs: the plane's fixed-point charges already staged in shared memory (the pipelined
// pass), or null to read them from global memory.
template <int N, int N1, int N2, int NT>
__device__ void plane_fwd(const DevPtrs& d, const RepDesc& D, int z, int unit_charge, float2* sa, float2* sb,
                          const ulonglong2* qs = nullptr) {
    constexpr int M = N / 2, NXH = M + 1, MS = plane_ms(M);
    static_assert(N1 * N2 == N, "y split");
    const int tid = threadIdx.x;
    float2* xa = sa;  // [y][j] packed real pairs, row stride MS; later the y stage-A output [k1 N2 + n2][k]
    float2* xb = sb;  // [y][k] after the split, row stride NXH
    if (unit_charge) {  // a unit charge on mesh point 0 (the influence kernel's source)
        for (int i = tid; i < N * M; i += NT) {
            const int y = i / M, j = i - y * M;
            xa[y * MS + j] = make_float2((z == 0 && i == 0) ? 1.0f : 0.0f, 0.0f);
        }
    } else {
        int zrel = z - D.zb_lo;
        zrel += (zrel < 0) ? D.mesh[2] : 0;
        const ulonglong2* q = qs ? qs : reinterpret_cast<const ulonglong2*>(d.qband + D.qb_off + (size_t)zrel * N * N);
        // batches of LB loads issued back to back before their shared-memory stores (the stores
        // could alias the loads as far as the compiler knows, so it would not hoist them)
        constexpr int LB = 8;
        for (int i0 = tid; i0 < N * M; i0 += LB * NT) {
            ulonglong2 v[LB];
#pragma unroll
            for (int u = 0; u < LB; ++u) {
                const int i = i0 + u * NT;
                if (i < N * M) v[u] = q[i];
            }
#pragma unroll
            for (int u = 0; u < LB; ++u) {
                const int i = i0 + u * NT;
                if (i >= N * M) break;
                const int y = i / M, j = i - y * M;
                xa[y * MS + j] = make_float2((float)((double)(long long)v[u].x * PHMC_FIX_INV),
                                             (float)((double)(long long)v[u].y * PHMC_FIX_INV));
            }
        }
    }
    __syncthreads();
    for (int y = tid; y < N; y += NT) {  // x: length-M DFT of the packed pairs of row y
        float2 v[M];
#pragma unroll
        for (int j = 0; j < M; ++j) v[j] = xa[y * MS + j];
        rfft::rdft<M, -1>(v);
#pragma unroll
        for (int j = 0; j < M; ++j) xa[y * MS + j] = v[j];
    }
    __syncthreads();
    const float2* twn = d.twiddle + D.tw_off[0];  // exp(-2 pi i k / nx)
    // split: X_k = 1/2 (Z_k + conj Z_{M-k}) - i/2 W^k (Z_k - conj Z_{M-k}), k = 0..M
    for (int i = tid; i < N * NXH; i += NT) {
        const int y = i / NXH, k = i - y * NXH;
        const float2 zk = xa[y * MS + (k == M ? 0 : k)];
        float2 zc = xa[y * MS + (k == 0 ? 0 : M - k)];
        zc.y = -zc.y;
        const float2 w = twn[k];
        const float2 s = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
        const float2 df = make_float2(0.5f * (zk.x - zc.x), 0.5f * (zk.y - zc.y));
        const float2 wd = cmul(w, df);
        xb[y * NXH + k] = make_float2(s.x + wd.y, s.y - wd.x);
    }
    __syncthreads();
    const float2* twy = d.twiddle + D.tw_off[1];  // exp(-2 pi i j / ny)
    for (int it = tid; it < N2 * NXH; it += NT) {  // y stage A: DFT over n1 of rows N2 n1 + n2, times W^(n2 k1)
        const int n2 = it / NXH, k = it - n2 * NXH;
        float2 v[N1];
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) v[n1] = xb[(N2 * n1 + n2) * NXH + k];
        rfft::rdft<N1, -1>(v);
        xa[n2 * NXH + k] = v[0];
#pragma unroll
        for (int k1 = 1; k1 < N1; ++k1) xa[(k1 * N2 + n2) * NXH + k] = cmul(v[k1], twy[n2 * k1]);
    }
    __syncthreads();
    float2* c = d.cmesh + D.meshh_off + (size_t)z * N * NXH;
    for (int it = tid; it < N1 * NXH; it += NT) {  // y stage B: DFT over n2 gives row ky = k1 + N1 k2
        const int k1 = it / NXH, k = it - k1 * NXH;
        float2 u[N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) u[n2] = xa[(k1 * N2 + n2) * NXH + k];
        rfft::rdft<N2, -1>(u);
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) c[(k1 + N1 * k2) * NXH + k] = u[k2];
    }
}

template <int N, int N1, int N2, int NT>
__device__ void plane_inv(const DevPtrs& d, const RepDesc& D, int z, float2* sa, float2* sb) {
    constexpr int M = N / 2, NXH = M + 1, MS = plane_ms(M);
    const int tid = threadIdx.x;
    float2* xa = sa;
    float2* xb = sb;
    const float2* c = d.cmesh + D.meshh_off + (size_t)z * N * NXH;
    const float2* twy = d.twiddle + D.tw_off[1];
    for (int it = tid; it < N1 * NXH; it += NT) {  // inverse y stage B: over k2, then W^(-n2 k1)
        const int k1 = it / NXH, k = it - k1 * NXH;
        float2 u[N2];
#pragma unroll
        for (int k2 = 0; k2 < N2; ++k2) u[k2] = c[(k1 + N1 * k2) * NXH + k];
        rfft::rdft<N2, 1>(u);
        xa[k1 * N2 * NXH + k] = u[0];
#pragma unroll
        for (int n2 = 1; n2 < N2; ++n2) {
            float2 w = twy[n2 * k1];
            w.y = -w.y;
            xa[(k1 * N2 + n2) * NXH + k] = cmul(u[n2], w);
        }
    }
    __syncthreads();
    for (int it = tid; it < N2 * NXH; it += NT) {  // inverse y stage A: over k1 gives row N2 n1 + n2
        const int n2 = it / NXH, k = it - n2 * NXH;
        float2 v[N1];
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) v[k1] = xa[(k1 * N2 + n2) * NXH + k];
        rfft::rdft<N1, 1>(v);
#pragma unroll
        for (int n1 = 0; n1 < N1; ++n1) xb[(N2 * n1 + n2) * NXH + k] = v[n1];
    }
    __syncthreads();
    const float2* twn = d.twiddle + D.tw_off[0];
    // merge: Z'_k = (X_k + conj X_{M-k}) + i W^{-k} (X_k - conj X_{M-k}), k = 0..M-1
    for (int i = tid; i < N * M; i += NT) {
        const int y = i / M, k = i - y * M;
        const float2 A = xb[y * NXH + k];
        float2 B = xb[y * NXH + (M - k)];
        B.y = -B.y;
        float2 w = twn[k];
        w.y = -w.y;
        const float2 s = make_float2(A.x + B.x, A.y + B.y);
        const float2 wd = cmul(w, make_float2(A.x - B.x, A.y - B.y));
        xa[y * MS + k] = make_float2(s.x - wd.y, s.y + wd.x);
    }
    __syncthreads();
    for (int y = tid; y < N; y += NT) {  // inverse x: length-M DFT of row y's packed pairs
        float2 v[M];
#pragma unroll
        for (int j = 0; j < M; ++j) v[j] = xa[y * MS + j];
        rfft::rdft<M, 1>(v);
#pragma unroll
        for (int j = 0; j < M; ++j) xa[y * MS + j] = v[j];
    }
    __syncthreads();
    float2* phi = reinterpret_cast<float2*>(d.phi + D.mesh_off + (size_t)z * N * N);
    for (int i = tid; i < N * M; i += NT) {  // the real plane: row y, points 2j and 2j + 1
        const int y = i / M, j = i - y * M;
        phi[i] = xa[y * MS + j];
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) k_rb_fwd_reg(DevPtrs d, const int2* __restrict__ jobs, int unit_charge,
                                                   const int* __restrict__ dirty) {
    extern __shared__ __align__(16) float2 psm[];
    const int2 job = jobs[blockIdx.x];
    const int r = job.x, z = job.y;
    if (dirty && !dirty[r]) return;
    const RepDesc& D = d.desc[r];
    const int n = D.mesh[0];
    float2* sa = psm;
    float2* sb = psm + n * plane_ms(n / 2);
    switch (n) {
#define PLANE_FWD(nn, a, b) case nn: plane_fwd<nn, a, b, NT>(d, D, z, unit_charge, sa, sb); break;
        PLANE_LIST(PLANE_FWD)
#undef PLANE_FWD
        default: break;
    }
}

// Pipelined first pass: persistent blocks walk the band-plane jobs with a stride of the
// grid; while a block transforms one plane, the next plane's fixed-point charges (N^2
// 8-byte values, contiguous) arrive in the other half of a two-stage shared-memory
// buffer by a bulk asynchronous copy (this GPU's own memory, no multicast), so the
// loads of the planes overlap the FFT work instead of opening every block.  Waits are
// bounded: a copy that does not arrive records PHMC_ERR_BUDGET in the replica's state
// and the block stops (the rebuild is then reported as failed).
template <int NT>
__global__ void __launch_bounds__(NT) k_rb_fwd_pipe(DevPtrs d, const int2* __restrict__ jobs, int njobs,
                                                    const int* __restrict__ dirty, int stage_off) {
    extern __shared__ __align__(16) float2 psm[];
    __shared__ __align__(8) uint64_t s_bar[2];
    __shared__ int s_fail;
    unsigned char* stage[2] = {reinterpret_cast<unsigned char*>(psm) + stage_off,
                               reinterpret_cast<unsigned char*>(psm) + stage_off + PLANE_STAGE_BYTES};
    if (threadIdx.x == 0) { sur_mbar_init(&s_bar[0]); sur_mbar_init(&s_bar[1]); s_fail = 0; }
    __syncthreads();
    auto wanted = [&](int j) { return j < njobs && (!dirty || dirty[jobs[j].x]); };
    auto issue = [&](int j, int s) {  // thread 0: the plane of job j into stage s
        const int2 job = jobs[j];
        const RepDesc& D = d.desc[job.x];
        const int n = D.mesh[0];
        int zrel = job.y - D.zb_lo;
        zrel += (zrel < 0) ? D.mesh[2] : 0;
        sur_bulk_load(stage[s], d.qband + D.qb_off + (size_t)zrel * n * n, (uint32_t)(n * n * 8), &s_bar[s]);
    };
    int uses[2] = {0, 0};  // copies issued into each stage (every thread counts alike)
    int j = blockIdx.x, it = 0;
    if (wanted(j)) { if (threadIdx.x == 0) issue(j, 0); uses[0]++; }
    for (; j < njobs; j += gridDim.x, ++it) {
        const int s = it & 1, jn = j + gridDim.x;
        if (wanted(jn)) { if (threadIdx.x == 0) issue(jn, s ^ 1); uses[s ^ 1]++; }  // its stage was read last step
        if (!wanted(j)) continue;
        if (threadIdx.x == 0 && !sur_mbar_wait(&s_bar[s], (uint32_t)((uses[s] - 1) & 1))) s_fail = 1;
        __syncthreads();
        if (s_fail) {
            if (threadIdx.x == 0) {
                atomicExch(&d.state[jobs[j].x].error, PHMC_ERR_BUDGET);
                sur_mbar_wait(&s_bar[s ^ 1], (uint32_t)((uses[s ^ 1] - 1) & 1));  // the copy in flight, bounded
            }
            return;
        }
        const int2 job = jobs[j];
        const RepDesc& D = d.desc[job.x];
        const int n = D.mesh[0];
        float2* sa = psm;
        float2* sb = psm + n * plane_ms(n / 2);
        const ulonglong2* qs = reinterpret_cast<const ulonglong2*>(stage[s]);
        switch (n) {
#define PLANE_FWD(nn, a, b) case nn: plane_fwd<nn, a, b, NT>(d, D, job.y, 0, sa, sb, qs); break;
            PLANE_LIST(PLANE_FWD)
#undef PLANE_FWD
            default: break;
        }
        __syncthreads();  // every thread is done with stage s and the plane buffers
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) k_rb_inv_reg(DevPtrs d, const int2* __restrict__ jobs, const int* __restrict__ dirty) {
    extern __shared__ __align__(16) float2 psm[];
    const int2 job = jobs[blockIdx.x];
    const int r = job.x, z = job.y;
    if (dirty && !dirty[r]) return;
    const RepDesc& D = d.desc[r];
    const int n = D.mesh[0];
    float2* sa = psm;
    float2* sb = psm + n * plane_ms(n / 2);
    switch (n) {
#define PLANE_INV(nn, a, b) case nn: plane_inv<nn, a, b, NT>(d, D, z, sa, sb); break;
        PLANE_LIST(PLANE_INV)
#undef PLANE_INV
        default: break;
    }
}

bool plane_reg_supported(int nx, int ny) {
    if (nx != ny) return false;
#define PLANE_OK(nn, a, b) if (nx == nn) return true;
    PLANE_LIST(PLANE_OK)
#undef PLANE_OK
    return false;
}
size_t plane_reg_smem(int n) { return ((size_t)n * plane_ms(n / 2) + (size_t)n * (n / 2 + 1)) * sizeof(float2); }

// The unit-charge rebuild (influence kernel) computes every plane; a rebuild of the
// particles' mesh only the planes of each replica's wall band.
void launch_rebuild_r2c(Engine& E, const int* dirty, int unit_charge, cudaStream_t st) {
    const int2* pj = unit_charge ? E.d_plane_jobs : E.d_band_jobs;
    const int npj = unit_charge ? E.n_plane_jobs : E.n_band_jobs;
    if (E.plane_reg && E.fwd_pipe && !unit_charge && E.nsm > 0) {
        const int off = (int)((E.rb_fwd_smem + 127) / 128 * 128);
        const int grid = std::min(npj, 2 * E.nsm);
        k_rb_fwd_pipe<PLANE_NT><<<grid, PLANE_NT, off + 2 * PLANE_STAGE_BYTES, st>>>(E.d, pj, npj, dirty, off);
    } else if (E.plane_reg) k_rb_fwd_reg<PLANE_NT><<<npj, PLANE_NT, E.rb_fwd_smem, st>>>(E.d, pj, unit_charge, dirty);
    else k_rb_fwd<256><<<npj, 256, E.rb_fwd_smem, st>>>(E.d, pj, unit_charge, dirty);
    switch (E.zreg) {
#define ZREG_LAUNCH(id, n, a, b) \
        case id: \
            if (E.zband && !unit_charge) k_rb_zband<a, b, ZREG_NT(b), ZREG_TX><<<E.n_zjobs, ZREG_NT(b), E.zpass_smem, st>>>(E.d, E.d_zjobs, E.d_epart, dirty); \
            else k_rb_zreg<a, b, ZREG_NT(b), ZREG_TX><<<E.n_zjobs, ZREG_NT(b), E.zpass_smem, st>>>(E.d, E.d_zjobs, E.d_epart, dirty, unit_charge); \
            break;
        ZREG_LIST(ZREG_LAUNCH)
#undef ZREG_LAUNCH
        default: k_rb_zpass<256, ZPASS_TX><<<E.n_zjobs, 256, E.zpass_smem, st>>>(E.d, E.d_zjobs, E.d_epart, dirty, unit_charge);
    }
    if (E.plane_reg) k_rb_inv_reg<PLANE_NT><<<npj, PLANE_NT, E.rb_inv_smem, st>>>(E.d, pj, dirty);
    else k_rb_inv<256><<<npj, 256, E.rb_inv_smem, st>>>(E.d, pj, dirty);
}

// Planes per block of the spread: a charge is found and its weights are made once per block that it
// reaches, (ZP + P - 1) / ZP times per plane, so as many as leave three blocks to an SM (the block's
// queues take 8 KB more; four planes of 48 x 48 leave two and take 119 us where three take 111); one
// where the band's planes would not fill the device with four blocks to an SM.
int spread_planes(int n_planes, int np_max, int nsm) {
    int zp = 1;
    while (zp < 4 && (size_t)(zp + 1) * np_max * 8 <= 64 * 1024 && n_planes >= 4 * nsm * (zp + 1)) ++zp;
    return zp;
}

template <class F>
static void spread_dispatch(const Engine& E, F&& f) {
    auto planes = [&](auto p) {
        switch (E.spread_zp) {
            case 1: f(p, std::integral_constant<int, 1>{}); break;
            case 2: f(p, std::integral_constant<int, 2>{}); break;
            case 3: f(p, std::integral_constant<int, 3>{}); break;
            default: f(p, std::integral_constant<int, 4>{}); break;
        }
    };
    if (E.order == 4) planes(std::integral_constant<int, 4>{});
    else if (E.order == 5) planes(std::integral_constant<int, 5>{});
    else planes(std::integral_constant<int, 6>{});
}

// Charge mesh of every replica's wall band from scratch (full recompute).
void launch_band_spread(Engine& E, cudaStream_t st) {
    spread_dispatch(E, [&](auto p, auto zp) {
        k_band_spread<decltype(p)::value, decltype(zp)::value, 256>
            <<<E.n_spread_jobs, 256, E.spread_zp * E.band_spread_smem, st>>>(E.d, E.d_spread_jobs);
    });
}

template <typename K>
static cudaError_t raise_cap(K kernel, int device, size_t need) {
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    const int cap = optin - (int)fa.sharedSizeBytes;
    if (cap < (int)need) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
}

cudaError_t rebuild_set_smem_limits(Engine& E) {
    cudaError_t e = cudaSuccess;
    spread_dispatch(E, [&](auto p, auto zp) {
        e = raise_cap(k_band_spread<decltype(p)::value, decltype(zp)::value, 256>, E.device, E.spread_zp * E.band_spread_smem);
    });
    if (e != cudaSuccess) return e;
    e = E.plane_reg ? raise_cap(k_rb_fwd_reg<PLANE_NT>, E.device, E.rb_fwd_smem) : raise_cap(k_rb_fwd<256>, E.device, E.rb_fwd_smem);
    if (e != cudaSuccess) return e;
    if (E.nsm == 0) {
        e = cudaDeviceGetAttribute(&E.nsm, cudaDevAttrMultiProcessorCount, E.device);
        if (e != cudaSuccess) return e;
    }
    if (E.plane_reg) e = raise_cap(k_rb_fwd_pipe<PLANE_NT>, E.device, (E.rb_fwd_smem + 127) / 128 * 128 + 2 * PLANE_STAGE_BYTES);
    if (e != cudaSuccess) return e;
    switch (E.zreg) {
#define ZREG_CAP(id, n, a, b) \
        case id: \
            e = raise_cap(k_rb_zreg<a, b, ZREG_NT(b), ZREG_TX>, E.device, E.zpass_smem); \
            if (e == cudaSuccess) e = raise_cap(k_rb_zband<a, b, ZREG_NT(b), ZREG_TX>, E.device, E.zpass_smem); \
            break;
        ZREG_LIST(ZREG_CAP)
#undef ZREG_CAP
        default: e = raise_cap(k_rb_zpass<256, ZPASS_TX>, E.device, E.zpass_smem);
    }
    if (e != cudaSuccess) return e;
    return E.plane_reg ? raise_cap(k_rb_inv_reg<PLANE_NT>, E.device, E.rb_inv_smem) : raise_cap(k_rb_inv<256>, E.device, E.rb_inv_smem);
}
