// Cell list (counting sort into padded per-cell slots) and the full-energy
// kernels: LJ/WCA + real-space Coulomb over the 27 neighbour cells, FENE
// bonds, walls and charge moments, all reduced in FP64 in a fixed order.
// Replaces build_half_neighbors_gpu (O(N^2), MC/src/neighbor.cu:21-125) and
// k_lj_energy / k_coul_energy / k_real_ewald_energy plus the Thrust
// reductions of pmeEnergy (MC/src/energy_gpu.cu:14-135, MC/src/pme.cu:252-288,425-447).
#include <algorithm>
#include "common.cuh"
#include "engine.h"
#include "fft.cuh"

__global__ void k_cell_assign(DevPtrs d, const int* __restrict__ rep_of, int total) {
    const int gs = blockIdx.x * blockDim.x + threadIdx.x;
    if (gs >= total) return;
    const int r = rep_of[gs];
    const RepDesc& D = d.desc[r];
    if (d.flags[gs] & PHMC_F_GHOST) { d.cell_of[gs] = -1; d.cell_pos[gs] = -1; return; }
    const float4 p = d.posq[gs];
    const int c = cell_index(D, p.x, p.y, p.z);
    const int k = atomicAdd(&d.cell_count[D.cell_off + c], 1);
    if (k < D.cell_cap) d.cell_list[((size_t)D.cell_off + c) * D.cell_cap + k] = gs - D.slot_off;
    else atomicExch(&d.state[r].error, PHMC_ERR_CAPACITY);
    d.cell_of[gs] = c;
}

// Sort every cell's members by slot index (deterministic order) and record
// each member's position inside its cell.
__global__ void k_cell_sort(DevPtrs d, const int* __restrict__ cell_rep, int total_cells) {
    const int gc = blockIdx.x * blockDim.x + threadIdx.x;
    if (gc >= total_cells) return;
    const RepDesc& D = d.desc[cell_rep[gc]];
    const int n = min(d.cell_count[gc], D.cell_cap);
    int* l = d.cell_list + (size_t)gc * D.cell_cap;
    for (int a = 1; a < n; ++a) {
        int v = l[a], b = a - 1;
        while (b >= 0 && l[b] > v) { l[b + 1] = l[b]; --b; }
        l[b + 1] = v;
    }
    int4 cc = make_int4(0, 0, 0, 0);
    for (int a = 0; a < n; ++a) {
        const int gi = D.slot_off + l[a];
        d.cell_pos[gi] = a;
        const int c = desc_class(d.flags[gi], d.posq[gi].w);
        cc.x += (c == 0); cc.y += (c == 1); cc.z += (c == 2); cc.w += (c == 3);
    }
    d.cell_cls[gc] = cc;
}

void launch_cell_build(Engine& E, cudaStream_t st) {
    cudaMemsetAsync(E.d.cell_count, 0, sizeof(int) * (size_t)E.total_cells, st);
    k_cell_assign<<<(E.total_slots + 255) / 256, 256, 0, st>>>(E.d, E.d_rep_of, E.total_slots);
    k_cell_sort<<<(E.total_cells + 127) / 128, 128, 0, st>>>(E.d, E.d_cell_rep, E.total_cells);
}

#define NCOMP 7
#define FE_CAND 128  // candidates of a warp at a time
#define FE_OWN 32    // particles of a cell at a time

// Sums of all pair, bond and charge-moment terms, one warp per cell (cells strided over the
// grid's warps): the cell's own particles against those of the own cell and of the 13 neighbour
// cells in the forward half shell, each unordered pair once (with at least 3 cells per axis the 13
// are distinct).  The warp lists its candidates (one lane per cell for the counts, then one lane
// per candidate for list entry and particle: two dependent loads in all, where a thread per
// particle walked 14 cells one after the other) and its lanes take the (own, candidate) pairs.
// Bound by instruction issue (46 % of the slots: list search, culling, erfc of the ~30 pairs within
// the cutoff) and those loads' latency.  Measured: 11.7k particles 153 -> 14 us, 64 replicas of 5k
// 286 -> 191 us, of 8.7k 516 -> 308 us; more warps per SM (fewer registers) were slower.
template <int NT>
__global__ void __launch_bounds__(NT) k_full_energy(DevPtrs d, int bpr) {
    constexpr int NW = NT / 32;
    __shared__ float4 s_p[NW][FE_CAND], s_o[NW][FE_OWN];
    __shared__ int s_j[NW][FE_CAND], s_t[NW][FE_CAND], s_ot[NW][FE_OWN];
    __shared__ int4 s_ob[NW][FE_OWN];
    __shared__ int s_off[NW][16], s_cell[NW][16];
    __shared__ int s_hit[NW][64];
    __shared__ double s_red[NW][NCOMP];
    const int r = blockIdx.y, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // the descriptor in shared memory: an evaluation reads a dozen of its fields
    __shared__ __align__(16) RepDesc sD;
    for (int k = threadIdx.x; k < (int)(sizeof(RepDesc) / sizeof(int)); k += NT)
        reinterpret_cast<int*>(&sD)[k] = reinterpret_cast<const int*>(d.desc + r)[k];
    __syncthreads();
    const RepDesc& D = sD;
    const int nc0 = D.ncell[0], nc1 = D.ncell[1], nc2 = D.ncell[2], cap = D.cell_cap, so = D.slot_off;
    const int ncells = nc0 * nc1 * nc2;
    double acc[NCOMP] = {0, 0, 0, 0, 0, 0, 0};  // lj, coul, fene(+walls), Q, Q2, Mz, S2
    const float Lx = D.L[0], Ly = D.L[1], Lz = D.L[2], iLx = 1.0f / Lx, iLy = 1.0f / Ly, iLz = 1.0f / Lz;
    // beyond this squared distance two particles have no pair term
    float rc2 = D.coulomb != PHMC_COUL_NONE ? D.rc_coul2 : 0.0f;
    for (int k = lane; k < D.T * D.T; k += 32)
        if (D.lj_eps[k] > 0.0f) rc2 = fmaxf(rc2, D.lj_rc2[k]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rc2 = fmaxf(rc2, __shfl_xor_sync(0xffffffffu, rc2, o));
    rc2 *= 1.0001f;
    int nh = 0;
    const unsigned below = (1u << lane) - 1u;
    auto evaluate = [&](int n) {  // the first n (<= 32) queued pairs, one per lane
        if (lane < n) {
            const int i = s_hit[w][lane] >> 16, k = s_hit[w][lane] & 0xffff;
            const float4 pi = s_o[w][i], pj = s_p[w][k];
            float elj, ec;
            pair_energy(D, near_image(pi.x - pj.x, Lx, iLx), near_image(pi.y - pj.y, Ly, iLy), near_image(pi.z - pj.z, Lz, iLz), s_ot[w][i], s_t[w][k], pi.w, pj.w, in_bonds(s_ob[w][i], s_j[w][k]), elj, ec);
            acc[0] += elj; acc[1] += ec;
        }
    };
    auto own_terms = [&](float4 p) {  // single-particle terms
        acc[3] += p.w; acc[4] += (double)p.w * p.w;
        acc[5] += (double)p.w * p.z; acc[6] += (double)p.w * p.z * p.z;
        if (D.walls && (p.z < D.wall_lo || p.z >= D.wall_hi)) acc[2] = __longlong_as_double(0x7ff0000000000000ll);
    };
    auto load_partners = [&](int i, float4 p, int4 b, float4 (&pj)[4]) {
        const int bl[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) pj[k] = bl[k] > i ? d.posq[so + bl[k]] : p;
    };
    auto bond_terms = [&](int i, float4 p, int4 b, const float4 (&pj)[4]) {
        const int bl[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (bl[k] <= i) continue;
            const float dx = min_image(p.x - pj[k].x, Lx), dy = min_image(p.y - pj[k].y, Ly), dz = min_image(p.z - pj[k].z, Lz);
            acc[2] += fene_energy(D, dx * dx + dy * dy + dz * dz);
        }
    };
    // pairs within the largest cutoff (~15 %) queue up and are evaluated 32 at a time
    auto near = [&](float4 a, float4 b) {
        const float dx = near_image(a.x - b.x, Lx, iLx), dy = near_image(a.y - b.y, Ly, iLy), dz = near_image(a.z - b.z, Lz, iLz);
        return dx * dx + dy * dy + dz * dz <= rc2;
    };
    auto push = [&](bool hit, int i, int k) {
        const unsigned hm = __ballot_sync(0xffffffffu, hit);
        if (hit) s_hit[w][nh + __popc(hm & below)] = (i << 16) | k;
        nh += __popc(hm);
        if (nh >= 32) {
            __syncwarp();
            evaluate(32);
            const int rest = s_hit[w][32 + lane];
            __syncwarp();
            s_hit[w][lane] = rest;
            nh -= 32;
        }
    };
    auto finish = [&]() {  // (the candidates the queue refers to are about to be replaced)
        __syncwarp();
        evaluate(nh);
        nh = 0;
    };
    // the 14 cells of c (own cell first), one per lane, and their counts
    const int hz = lane < 5 ? 0 : 1;
    const int hy = lane < 2 ? 0 : (lane < 5 ? 1 : (lane - 5) / 3 - 1);
    const int hx = lane == 0 ? 0 : (lane == 1 ? 1 : (lane < 5 ? lane - 3 : (lane - 5) % 3 - 1));
    const FastDiv by_x(nc0), by_y(nc1);
    auto neighbours = [&](int c, int& nc, int& cnt) {
        nc = 0; cnt = 0;
        if (lane < 14) {
            int row, x, y;
            int z;
            if (ncells < (1 << 22)) {  // (products of floats are exact enough up to there)
                row = by_x.div(c, x);
                z = by_y.div(row, y);
            } else {
                row = c / nc0; x = c - row * nc0;
                z = row / nc1; y = row - z * nc1;
            }
            x += hx; y += hy; z += hz;
            x += (x < 0) ? nc0 : (x >= nc0 ? -nc0 : 0);
            y += (y < 0) ? nc1 : (y >= nc1 ? -nc1 : 0);
            z -= (z >= nc2) ? nc2 : 0;
            nc = (z * nc1 + y) * nc0 + x;
            cnt = min(d.cell_count[D.cell_off + nc], cap);
        }
    };
    const int step = bpr * NW;
    for (int c0 = blockIdx.x * NW + w; c0 < ncells; c0 += 32 * step) {
        // the warp's next 32 cells at once: most cells of a padded slab are empty
        const int cl = c0 + lane * step;
        unsigned todo = __ballot_sync(0xffffffffu, cl < ncells && d.cell_count[D.cell_off + cl] > 0);
        int nc = 0, cnt = 0;
        if (todo) neighbours(c0 + (__ffs(todo) - 1) * step, nc, cnt);
        while (todo) {
            const int c = c0 + (__ffs(todo) - 1) * step;
            todo &= todo - 1;
            const int n = __shfl_sync(0xffffffffu, cnt, 0);
            int ofs = cnt;
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, ofs, o);
                if (lane >= o) ofs += y;
            }
            const int m = __shfl_sync(0xffffffffu, ofs, 13);
            __syncwarp();
            if (lane < 16) { s_off[w][lane] = lane < 14 ? ofs - cnt : 0x7fffffff; s_cell[w][lane] = nc; }
            __syncwarp();
            if (todo) neighbours(c0 + (__ffs(todo) - 1) * step, nc, cnt);  // the next cell's, in flight meanwhile
            auto cell_of = [&](int x) {  // last cell whose offset is <= x
                int h = 0;
#pragma unroll
                for (int st = 8; st > 0; st >>= 1)
                    if (s_off[w][h + st] <= x) h += st;
                return h;
            };
            if (n <= FE_OWN && m <= FE_CAND) {
                // usual case: list entries of all candidates, then all particles, each in one round trip;
                // the own particles are the first n of them
                int j[FE_CAND / 32];
                float4 p[FE_CAND / 32];
                int ty[FE_CAND / 32];
#pragma unroll
                for (int u = 0; u < FE_CAND / 32; ++u) {
                    const int x = lane + 32 * u;
                    if (x < m) {
                        const int h = cell_of(x);
                        j[u] = d.cell_list[((size_t)D.cell_off + s_cell[w][h]) * cap + x - s_off[w][h]];
                    }
                }
#pragma unroll
                for (int u = 0; u < FE_CAND / 32; ++u)
                    if (lane + 32 * u < m) { p[u] = d.posq[so + j[u]]; ty[u] = d.type[so + j[u]]; }
                int4 b = make_int4(-1, -1, -1, -1);
                if (lane < n) b = d.bonds[so + j[0]];
#pragma unroll
                for (int u = 0; u < FE_CAND / 32; ++u)
                    if (lane + 32 * u < m) { s_j[w][lane + 32 * u] = j[u]; s_p[w][lane + 32 * u] = p[u]; s_t[w][lane + 32 * u] = ty[u]; }
                float4 pj[4];
                const bool fene = lane < n && D.fene_k > 0.0f;
                if (lane < n) {
                    s_ot[w][lane] = ty[0]; s_o[w][lane] = p[0]; s_ob[w][lane] = b;
                    if (fene) load_partners(j[0], p[0], b, pj);
                }
                __syncwarp();
                const int mu = (m + 31) / 32;
                for (int i = 0; i < n; ++i) {
                    const float4 pi = s_o[w][i];
#pragma unroll
                    for (int u = 0; u < FE_CAND / 32; ++u) {
                        if (u >= mu) break;
                        const int k = lane + 32 * u;
                        push(k > i && k < m && near(pi, p[u]), i, k);  // (own cell: later members only)
                    }
                }
                finish();
                if (lane < n) own_terms(p[0]);
                if (fene) bond_terms(j[0], p[0], b, pj);
                __syncwarp();
                continue;
            }
            for (int i0 = 0; i0 < n; i0 += FE_OWN) {
                const int no = min(n - i0, FE_OWN);
                if (lane < no) {
                    const int i = d.cell_list[((size_t)D.cell_off + c) * cap + i0 + lane];
                    const float4 p = d.posq[so + i];
                    const int4 b = d.bonds[so + i];
                    s_ot[w][lane] = d.type[so + i]; s_o[w][lane] = p; s_ob[w][lane] = b;
                    own_terms(p);
                    if (D.fene_k > 0.0f) {
                        float4 pj[4];
                        load_partners(i, p, b, pj);
                        bond_terms(i, p, b, pj);
                    }
                }
                for (int base = 0; base < m; base += FE_CAND) {
                    const int mc = min(m - base, FE_CAND);
                    __syncwarp();
                    for (int k = lane; k < mc; k += 32) {
                        const int x = base + k, h = cell_of(x);
                        const int j = d.cell_list[((size_t)D.cell_off + s_cell[w][h]) * cap + x - s_off[w][h]];
                        s_j[w][k] = j; s_p[w][k] = d.posq[so + j]; s_t[w][k] = d.type[so + j];
                    }
                    __syncwarp();
                    for (int i = 0; i < no; ++i)
                        for (int k0 = 0; k0 < mc; k0 += 32) {
                            const int k = k0 + lane;
                            push(k < mc && base + k > i0 + i && near(s_o[w][i], s_p[w][k < mc ? k : 0]), i, k);
                        }
                    finish();
                }
                __syncwarp();
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NCOMP; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if (lane == 0) s_red[w][k] = acc[k];
    }
    __syncthreads();
    if (threadIdx.x < NCOMP) {
        double t = 0.0;
        for (int k = 0; k < NW; ++k) t += s_red[k][threadIdx.x];
        d.partials[((size_t)r * bpr + blockIdx.x) * 8 + threadIdx.x] = t;
    }
}

// One block per replica: threads over the blocks' partial sums, then over threads, in a fixed order.
template <int NT>
__global__ void __launch_bounds__(NT) k_full_reduce(DevPtrs d, int bpr) {
    __shared__ double s_red[NT / 32][NCOMP];
    const int r = blockIdx.x, lane = threadIdx.x & 31;
    double a[NCOMP] = {0, 0, 0, 0, 0, 0, 0};
    for (int b = threadIdx.x; b < bpr; b += NT)
#pragma unroll
        for (int k = 0; k < NCOMP; ++k) a[k] += d.partials[((size_t)r * bpr + b) * 8 + k];
#pragma unroll
    for (int k = 0; k < NCOMP; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
        if (lane == 0) s_red[threadIdx.x >> 5][k] = a[k];
    }
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < NT / 32; ++w)
        for (int k = 0; k < NCOMP; ++k) a[k] += s_red[w][k];
    const RepDesc& D = d.desc[r];
    RepState& S = d.state[r];
    S.E_pair_lj = a[0]; S.E_pair_c = a[1]; S.E_fene = a[2];
    S.Q = a[3]; S.Q2 = a[4]; S.Mz = a[5]; S.S2 = a[6];
    if (D.coulomb == PHMC_COUL_EWALD) {
        S.E_self = D.self_coef * S.Q2;
        S.E_qcorr = D.qcorr_coef * S.Q * S.Q;
        double es = 0.0;
        if (D.slab) {
            es = D.slab_coef * S.Mz * S.Mz;
            if (fabs(S.Q) > 1e-4) es -= D.slab_coef * S.Q * (S.S2 + S.Q * D.Lz2_12);
        }
        S.E_slab = es;
    } else {
        S.E_self = S.E_qcorr = S.E_slab = 0.0;
        S.E_rec = 0.0;
    }
    S.E = S.E_pair_lj + S.E_pair_c + S.E_fene + S.E_rec + S.E_self + S.E_qcorr + S.E_slab;
}

// Blocks per replica at nt threads each: one cell per warp, while all replicas' blocks stay within
// about four waves of the chip (the rest of the cells in turn), at most PHMC_FULL_MAX_BPR.
static int full_energy_bpr(const Engine& E, int nt) {
    const int want = (E.max_cells + nt / 32 - 1) / (nt / 32), room = std::max(8, 4 * E.nsm * 4 * 256 / nt / E.R);
    return std::max(1, std::min({PHMC_FULL_MAX_BPR, want, room}));
}

size_t full_energy_partials(const Engine& E) {
    const int bpr = std::max({full_energy_bpr(E, 64), full_energy_bpr(E, 128), full_energy_bpr(E, 256)});
    return (size_t)E.R * bpr * 8;
}

// E.energy_block (64, 128, 256 threads; 0: 256) is a tuning parameter.
void launch_full_energy(Engine& E, cudaStream_t st) {
    const int nt = E.energy_block ? E.energy_block : 256;
    const int bpr = full_energy_bpr(E, nt);
    dim3 grid(bpr, E.R);
    if (nt == 64) k_full_energy<64><<<grid, 64, 0, st>>>(E.d, bpr);
    else if (nt == 256) k_full_energy<256><<<grid, 256, 0, st>>>(E.d, bpr);
    else k_full_energy<128><<<grid, 128, 0, st>>>(E.d, bpr);
    k_full_reduce<128><<<E.R, 128, 0, st>>>(E.d, bpr);
}
