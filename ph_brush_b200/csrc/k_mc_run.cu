// Plain Monte Carlo (no surrogate first stage, no external trials): one thread block per
// replica evaluates a batch of up to RUN_BATCH consecutive trials against one state and
// then decides them in order.
//
// A trial evaluated alone is a chain of dependent loads and block barriers (17k-25k cycles
// on a B200, 25 % of the issue slots used): proposal, cell lists, particles, mesh windows,
// decision.  The proposals of consecutive trials come from a counter-based stream and
// almost never touch one another, so a batch pays each of those latencies once:
//  * proposal: lane b of warp 0 draws trial t0 + b;
//  * pair terms: one warp per probe (old or new state), a lane per neighbour cell;
//  * mesh terms: one warp per (trial, earlier stencil), the earlier stencils being the
//    pending ones and those of the batch's earlier trials;
//  * decision: lane b holds trial b's dE; the first accepting lane is found by a ballot,
//    its stencils' terms are added to the later lanes, and so on.
// Measured on a B200 (250-400 trials of a run, wall time of the whole call): one replica of 484
// particles 2120 -> 810 us, one of 11.7k particles 5170 -> 1570 us, 24 uneven replicas 4250 ->
// 2100 us; 256 replicas, two blocks to an SM, 16.1 -> 15.4 ms (half of it mesh rebuilds).
// (Titration-only runs, and how long batches are: run_length.)
// A batch ends early (and the next one starts there) where an accepted trial could have
// changed a later one: an inserted or removed particle changes the index lists that
// proposals draw from; a changed particle within the largest cutoff of a later trial's
// probe, or bonded to its particle, changes that trial's pair terms; and a moved particle
// that a later trial displaces again, also one that the walls refused from the old place,
// changes that trial.  What remains is
// exactly the sequence of one-at-a-time trials, and because every sum is formed per probe
// and per stencil pair in a fixed order, its energies are bit for bit independent of the
// batch's size and of the block's number of warps.
#include <algorithm>
#include <type_traits>
#include "common.cuh"
#include "engine.h"
#include "mc_common.cuh"
#include "mc_window.cuh"
#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define RUN_BATCH 16        // trials per batch at most (lanes of the deciding warp)
#define RUN_TST (2 * RUN_BATCH)    // stencils of a batch: at most two per trial (a displaced
                                   // charge's old and new place; a site's change and its ion)
#define RUN_PROBES (4 * RUN_BATCH)
#define RUN_LIST 256   // candidates of a probe listed at a time
#define RUN_HIT 64
#define RUN_TAB(p) (2 * Win<p>::TAB)  // floats of a warp's window tables

// One trial of a batch: its changes, bonds, stencils and probes, and the terms that need no other particle.
struct RunTrial {
    int move, skip, nch, nst, st0, np, p0, lists;
    int idx[2], pres_old[2], pres_new[2], to[2], tn[2], fo[2];
    uint32_t ua, ub;
    double logf;
    float4 po[2], pn[2];
    int4 bonds[2];
    double direct_lj, direct_c;
    double dQ, dQ2, dMz, dS2;
};

// Trials of a batch: a batch of n costs the latency of one and n trials' work, of which the trials after a
// cut are lost.  With cuts at a rate of h a trial the best n is near sqrt(worth / h), worth being twice
// the latency in units of a trial's work.  (Titrations and ion swaps change the lists that proposals draw
// from, so an accepted one always cuts: a run of titrations alone decided 2 of the 16 trials of a batch.
// 300 such trials, long batches always -> this rule (one trial at a time before batches): 12k particles 7.4 ->
// 5.5 ms (5.5), 96 uneven replicas 31 -> 12.7 (16.1), 256 replicas 30.4 -> 20.5 (24.2), 75 of 40 particles
// 15.2 -> 4.2 (4.2); with 90 % displacements 1.35 -> 1.35 (4.0), 7.6 -> 5.3 (9.7), 9.8 -> 9.2 (13.4), 3.6 -> 2.0
// (3.0).  Left behind: titrations alone on more small replicas than SMs, 15 % slower than one at a time,
// 23 % at order 6, whose windows take twice the instructions.)
__device__ __forceinline__ int run_length(float2 rate, float worth, int batch) {
    const float a = worth * rate.y;
    return rate.x > 0.0f ? max(1, (int)fminf(a * rsqrtf(a * rate.x) + 0.5f, (float)batch)) : batch;
}

// Proposal of trial t (the rules of the oracle's Monte Carlo, as in k_mc).
__device__ __forceinline__ void run_propose(RunTrial& T, long long t, const RepDesc& D, const RepState& S, const DevPtrs& d) {
    uint32_t A[4], B[4];
    const uint32_t lo = (uint32_t)t, hi = (uint32_t)((unsigned long long)t >> 32);
    philox4x32_10(D.key[0], D.key[1], lo, hi, 0u, 0u, A);
    philox4x32_10(D.key[0], D.key[1], lo, hi, 1u, 0u, B);
    const int move = move_of(D, A[0]);
    T.move = move; T.skip = 0; T.nch = 0; T.lists = 0; T.logf = 0.0;
    T.ua = B[2]; T.ub = B[3];
    const int so = D.slot_off;
    int i0 = -1, i1 = -1;
    // the changed particles' slots first, then all of their data in one round trip
    int kind = 0;  // 1 displacement, 2 titration, 3 pair insertion, 4 pair deletion
    if (move == PHMC_MOVE_DISP) {
        if (S.n_mobile > 0) { i0 = d.mobile[so + pick_index(A[1], S.n_mobile)]; kind = 1; }
    } else if (move == PHMC_MOVE_TITR) {
        if (D.n_titr > 0) { i0 = d.titr[so + pick_index(A[1], D.n_titr)]; kind = 2; }
    } else if (move == PHMC_MOVE_SWAP) {
        if (u24(A[1]) < 0.5f) {
            if (S.n_free >= 2) { i0 = d.freel[so + S.n_free - 1]; i1 = d.freel[so + S.n_free - 2]; kind = 3; }
        } else if (S.n_cation > 0 && S.n_anion > 0) {
            uint32_t C[4];
            philox4x32_10(D.key[0], D.key[1], lo, hi, 2u, 0u, C);
            i0 = d.cations[so + pick_index(B[1], S.n_cation)];
            i1 = d.anions[so + pick_index(C[3], S.n_anion)];
            kind = 4;
        }
    } else {
        T.skip = 3;  // no-op draw
        return;
    }
    if (!kind) { T.skip = 1; return; }
    auto load_old = [&](int k, int i) {
        const int fl = d.flags[so + i];
        const float4 p = d.posq[so + i];
        const int ty = d.type[so + i];
        const int4 b = d.bonds[so + i];
        T.idx[k] = i; T.fo[k] = fl; T.pres_old[k] = !(fl & PHMC_F_GHOST);
        T.po[k] = p; T.to[k] = ty; T.bonds[k] = b;
        return p;
    };
    const float4 po = load_old(0, i0);
    if (kind == 1) {
        const float dm = D.disp_max;
        const float dx = __fmul_rn(dm, __fsub_rn(__fmul_rn(2.0f, u24(A[2])), 1.0f));
        const float dy = __fmul_rn(dm, __fsub_rn(__fmul_rn(2.0f, u24(A[3])), 1.0f));
        const float dz = __fmul_rn(dm, __fsub_rn(__fmul_rn(2.0f, u24(B[0])), 1.0f));
        const float Lx = D.L[0], Ly = D.L[1], Lz = D.L[2];
        float nx = __fadd_rn(po.x, dx), ny = __fadd_rn(po.y, dy), nz = __fadd_rn(po.z, dz);
        if (nx < 0.0f) nx = __fadd_rn(nx, Lx); else if (nx >= Lx) nx = __fsub_rn(nx, Lx);
        if (ny < 0.0f) ny = __fadd_rn(ny, Ly); else if (ny >= Ly) ny = __fsub_rn(ny, Ly);
        const int walls = D.walls;
        if (!walls) { if (nz < 0.0f) nz = __fadd_rn(nz, Lz); else if (nz >= Lz) nz = __fsub_rn(nz, Lz); }
        T.pres_new[0] = 1; T.pn[0] = make_float4(nx, ny, nz, po.w); T.tn[0] = T.to[0];
        T.nch = 1;
        if (walls && (nz < D.wall_lo || nz >= D.wall_hi)) T.skip = 2;  // hard wall: infinite energy
    } else if (kind == 2) {
        T.pres_new[0] = 1;
        if (po.w == 0.0f) {
            if (S.n_free == 0) { T.skip = 1; return; }
            load_old(1, d.freel[so + S.n_free - 1]);
            T.pn[0] = make_float4(po.x, po.y, po.z, D.q_site_charged); T.tn[0] = D.type_site_charged;
            float4 pg = rand_pos(D, A[2], A[3], B[0]); pg.w = D.q_counterion;
            T.pres_new[1] = 1; T.pn[1] = pg; T.tn[1] = D.type_counterion;
            T.logf = D.titr_log;
        } else {
            if (S.n_anion == 0) { T.skip = 1; return; }
            const float4 p1 = load_old(1, d.anions[so + pick_index(B[1], S.n_anion)]);
            T.pn[0] = make_float4(po.x, po.y, po.z, 0.0f); T.tn[0] = D.type_site_neutral;
            T.pres_new[1] = 0; T.pn[1] = p1; T.tn[1] = T.to[1];
            T.logf = -D.titr_log;
        }
        T.nch = 2;
    } else if (kind == 3) {
        load_old(1, i1);
        uint32_t C[4];
        philox4x32_10(D.key[0], D.key[1], lo, hi, 2u, 0u, C);
        float4 p1 = rand_pos(D, A[2], A[3], B[0]); p1.w = D.q_cation;
        float4 p2 = rand_pos(D, C[0], C[1], C[2]); p2.w = D.q_counterion;
        T.pres_new[0] = 1; T.pn[0] = p1; T.tn[0] = D.type_cation;
        T.pres_new[1] = 1; T.pn[1] = p2; T.tn[1] = D.type_counterion;
        T.logf = log(D.salt_c2V2 / ((double)(S.n_cation + 1) * (double)(S.n_anion + 1)));
        T.nch = 2;
    } else {
        const float4 p1 = load_old(1, i1);
        T.pres_new[0] = 0; T.pn[0] = po; T.tn[0] = T.to[0];
        T.pres_new[1] = 0; T.pn[1] = p1; T.tn[1] = T.to[1];
        T.logf = log((double)S.n_cation * (double)S.n_anion / D.salt_c2V2);
        T.nch = 2;
    }
    for (int k = 0; k < T.nch; ++k) T.lists |= T.pres_old[k] != T.pres_new[k];
}

__host__ __device__ constexpr int run_unit_stride(int pend_max) { return (pend_max + RUN_TST + 2) | 1; }
template <int P>
__host__ __device__ constexpr size_t run_stencil_bytes(int pend_max) {
    return (sizeof(PadSt<P>) * (pend_max + RUN_TST) + 15) / 16 * 16;
}

// A block's probe tables, trials and counters of one batch (one object, so that the other blocks of a
// cluster can copy it).
struct __align__(16) RunShared {
    RunTrial T[RUN_BATCH];
    float4 pp[RUN_PROBES];                  // probes: position, type, sign, trial, which change
    float psg[RUN_PROBES];
    int pt[RUN_PROBES], pb[RUN_PROBES], pk[RUN_PROBES];
    int task[RUN_BATCH + 4];                // first mesh work item of each trial
    int npend, nb, ns, npr, ntask, stop, pad[2];
};

// CL: the replica's block is the first of a cluster whose other blocks share the pair and mesh
// work of each batch; they copy the batch's tables from the first block's shared memory and store
// their results into it.
template <int P, int NT, bool CL>
__global__ void __launch_bounds__(NT, 512 / NT) k_mc_run(DevPtrs d, int pend_max, int batch, float worth) {
    constexpr int P3 = P * P * P;
    constexpr int NW = NT / 32;
    extern __shared__ __align__(16) unsigned char dsm[];
    // stencils: pending [0, npend), then the batch's [npend, npend + ns)
    PadSt<P>* s_st = reinterpret_cast<PadSt<P>*>(dsm);
    const int us = run_unit_stride(pend_max);
    double* s_unit = reinterpret_cast<double*>(dsm + run_stencil_bytes<P>(pend_max));
    float* s_tab = reinterpret_cast<float*>(s_unit + (size_t)RUN_BATCH * us);  // a warp's window tables
    int* s_list = reinterpret_cast<int*>(s_tab + NW * RUN_TAB(P));             // a warp's candidates and
    int* s_hit = s_list + NW * RUN_LIST;                                       // those within the cutoff
    __shared__ RunShared B;
    __shared__ __align__(16) RepDesc sD;
    __shared__ RepState S;
    __shared__ float4 s_stp[RUN_TST];
    __shared__ float s_stc[RUN_TST];
    __shared__ double s_plj[RUN_PROBES], s_pc[RUN_PROBES], s_phi[RUN_BATCH], s_fene[RUN_BATCH][4];
    __shared__ int s_pn[RUN_PROBES];
    __shared__ unsigned s_conf[RUN_BATCH];
    __shared__ float4 s_qjob[4 * RUN_BATCH];
    __shared__ int s_qsgn[4 * RUN_BATCH], s_nq;
    __shared__ int s_qin;
    __shared__ volatile int s_qstop;
    __shared__ float s_rc2, s_iL[3];
    // accepted changes of the last batch whose bookkeeping is done beside the next proposals
    __shared__ double s_ev[RUN_BATCH][8];   // energy changes, in RepState's order from E on
    __shared__ int s_cp[RUN_TST][2], s_mv[2 * RUN_BATCH][3];  // stencil moves; cell moves (slot, from, to)
    __shared__ int s_nev, s_ncp, s_nmv;
    // recent batches: those that an accepted trial cut short, trials decided; the last batch's; trials of
    // the next one at most (made beside the pair terms, off the deciding lane's chain, so one batch late)
    __shared__ float2 s_rate;
    __shared__ int s_cut, s_decided, s_len;
    __shared__ unsigned int s_zh[3 * PHMC_ZHIST_MAX_BINS];

    unsigned rank = 0, csize = 1;
    if constexpr (CL) {
        rank = cg::this_cluster().block_rank();
        csize = cg::this_cluster().num_blocks();
    }
    const int r = blockIdx.x / csize;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const int* src = reinterpret_cast<const int*>(d.desc + r);
        int* dst = reinterpret_cast<int*>(&sD);
        for (int k = tid; k < (int)(sizeof(RepDesc) / sizeof(int)); k += NT) dst[k] = src[k];
    }
    const RepDesc& D = sD;
    if (tid == 0) {
        S = d.state[r];
        B.npend = 0; s_nq = 0; B.stop = 0; s_qstop = 0; s_qin = 0;
        s_nev = 0; s_ncp = 0; s_nmv = 0;
        if (rank == 0 && d.quorum < 1.0f && S.trial < S.target) { atomicAdd(&d.quorum_ctl[0], 1); s_qin = 1; }
    }
    if (tid == 32) {
        s_rate = d.run_rate[r];
        s_len = run_length(s_rate, worth, batch);
        s_cut = 0; s_decided = 0;
    }
    unsigned long long t_start = 0;
    if (tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
    long long clk_last = clock64();
    auto mark = [&](int ph) {  // phase clocks (thread 0, after the barrier that ends the phase)
        if (tid == 0 && d.phase_clk) {
            const long long now = clock64();
            S.clk[ph] += now - clk_last;
            clk_last = now;
        }
    };
    __syncthreads();
    if (tid == 0) {  // beyond this squared distance two particles have no pair term
        float m = D.coulomb != PHMC_COUL_NONE ? D.rc_coul2 : 0.0f;
        for (int k = 0; k < D.T * D.T; ++k)
            if (D.lj_eps[k] > 0.0f) m = fmaxf(m, D.lj_rc2[k]);
        s_rc2 = m * 1.0001f;
        for (int k = 0; k < 3; ++k) s_iL[k] = 1.0f / D.L[k];
    }
    const bool ewald = D.coulomb == PHMC_COUL_EWALD;
    const int so = D.slot_off;
    // where results go (the first block's shared memory), and loads of what the first block changes
    // during the launch (past the other blocks' L1)
    double *r_plj = s_plj, *r_pc = s_pc, *r_phi = s_phi, *r_unit = s_unit;
    int* r_pn = s_pn;
    if constexpr (CL) {
        auto c = cg::this_cluster();
        r_plj = c.map_shared_rank(s_plj, 0); r_pc = c.map_shared_rank(s_pc, 0); r_phi = c.map_shared_rank(s_phi, 0);
        r_unit = c.map_shared_rank(s_unit, 0); r_pn = c.map_shared_rank(s_pn, 0);
    }
    auto ld = [](auto* p) { if constexpr (CL) return __ldcg(p); else return *p; };
    LaneSt<P> L;
    lane_place<P>(L, D, lane);

    for (;;) {
        bool halt = false;
        if (rank == 0) {
        // ---------------- proposals ----------------
        if (warp == 0) {
            int stop = 0, nb = 0;
            if (S.error) stop = 1;
            else if (S.trial >= S.target) { stop = 1; if (lane == 0) S.stop_reason = 0; }
            else if (B.npend + 2 > pend_max) {
                stop = 1;
                if (lane == 0) { S.stop_reason = 1; if (s_qin) atomicAdd(&d.quorum_ctl[1], 1); }
            } else if (s_qstop) { stop = 1; if (lane == 0) S.stop_reason = 2; }
            if (!stop) {
                long long n = S.target - S.trial;
                if (d.zh_bins > 0) n = min(n, d.zh_every - S.trial % d.zh_every);  // a sample ends a batch
                nb = (int)min((long long)s_len, n);
                int np = 0, ns = 0;
                // a probe per old and per new state; a stencil per charge that appears, leaves or changes
                auto states = [&](auto&& probe, auto&& stencil) {
                    const RunTrial& t = B.T[lane];
                    if (t.skip) return;
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        if (k >= t.nch) break;
                        const bool pold = t.pres_old[k], pnew = t.pres_new[k];
                        const float4 o = t.po[k], n4 = t.pn[k];
                        if (pold) probe(o, t.to[k], -1.0f, k);
                        if (pnew) probe(n4, t.tn[k], 1.0f, k);
                        if (!ewald) continue;
                        if (pold && pnew && o.x == n4.x && o.y == n4.y && o.z == n4.z) {
                            if (n4.w - o.w != 0.0f) stencil(n4, n4.w - o.w);
                        } else {
                            if (pold && o.w != 0.0f) stencil(o, -o.w);
                            if (pnew && n4.w != 0.0f) stencil(n4, n4.w);
                        }
                    }
                };
                if (lane < nb) {
                    run_propose(B.T[lane], S.trial + lane, D, S, d);
                    states([&](float4, int, float, int) { ++np; }, [&](float4, float) { ++ns; });
                }
                int ps = np, ss = ns;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int a = __shfl_up_sync(0xffffffffu, ps, o), b = __shfl_up_sync(0xffffffffu, ss, o);
                    if (lane >= o) { ps += a; ss += b; }
                }
                const int p0 = ps - np, s0 = ss - ns;
                // mesh work items of the trial: every earlier stencil, then its own
                const int nt = ns ? B.npend + s0 + ns : 0;
                int ts = nt;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int a = __shfl_up_sync(0xffffffffu, ts, o);
                    if (lane >= o) ts += a;
                }
                if (lane < nb) {
                    B.T[lane].np = np; B.T[lane].p0 = p0; B.T[lane].nst = ns; B.T[lane].st0 = s0;
                    int p = p0, x = s0;
                    states([&](float4 q, int ty, float sg, int k) { B.pp[p] = q; B.pt[p] = ty; B.psg[p] = sg; B.pk[p] = k; B.pb[p] = lane; ++p; },
                           [&](float4 q, float c) { s_stp[x] = q; s_stc[x] = c; ++x; });
                    B.task[lane] = ts - nt;
                    s_conf[lane] = 0u;
                }
                if (lane == 31) { B.npr = ps; B.ns = ss; B.ntask = ts; }
            }
            if (lane == 0) { B.stop = stop; B.nb = nb; B.task[nb] = 0x7fffffff; if (stop) B.ns = 0; }
        } else if (warp == 1) {
            // the last batch's accepted changes, in trial order: stencils move down to the pending
            // list, energies, cell lists
            const int ncp = s_ncp, nev = s_nev, nmv = s_nmv;
            for (int k = 0; k < ncp; ++k) {
                const int* src = reinterpret_cast<const int*>(&s_st[s_cp[k][0]]);
                int* dst = reinterpret_cast<int*>(&s_st[s_cp[k][1]]);
                for (int w = lane; w < (int)(sizeof(PadSt<P>) / 4); w += 32) dst[w] = src[w];
                __syncwarp();
            }
            if (lane < 8) {
                double* e = &S.E + lane;
                double v = *e;
                for (int k = 0; k < nev; ++k) v += s_ev[k][lane];
                *e = v;
            }
            if (lane == 0 && !S.error) {
                for (int k = 0; k < nmv; ++k) {
                    if (s_mv[k][1] >= 0) cell_remove(d, D, s_mv[k][0]);
                    if (s_mv[k][2] >= 0 && !cell_insert(d, D, s_mv[k][0], s_mv[k][2])) { S.error = PHMC_ERR_CAPACITY; break; }
                }
            }
        } else {
            // ... and into the fixed-point charge mesh
            for (int j = warp - 2; j < s_nq; j += NW - 2) qmesh_update<P>(D, d, s_qjob[j], s_qsgn[j] < 0, lane);
        }
        __syncthreads();
        mark(0);
        mark(1);
        // the last batch's moves overflowed a cell while this one was drawn: it is dropped
        halt = B.stop || S.error;
        if (tid == 0 && halt) { B.stop = 1; B.ns = 0; }
        if (!halt) {
        const int nb = B.nb, npend = B.npend, ns = B.ns;
        // ---------------- stencils, direct and bonded terms, conflicts ----------------
        if (tid == 0) s_nq = 0;
        constexpr int Q_ST = 0, Q_FE = Q_ST + 3 * RUN_TST, Q_DI = Q_FE + 4 * RUN_BATCH, Q_CF = Q_DI + 32,
                      Q_END = Q_CF + RUN_BATCH * RUN_BATCH;
        for (int it = tid; it < Q_END; it += NT) {
            if (it < Q_FE) {
                const int x = it / 3, ax = it - 3 * x;
                if (x < ns) {
                    pad_stencil_axis<P>(s_st[npend + x], D, s_stp[x], ax);
                    if (ax == 0) s_st[npend + x].coef = s_stc[x];
                }
            } else if (it < Q_DI) {  // FENE: one thread per (trial, bond slot), over the changed particles
                const int b = (it - Q_FE) >> 2, sl = (it - Q_FE) & 3;
                double df = 0.0;
                if (b < nb && B.T[b].skip == 0 && D.fene_k > 0.0f) {
                    const RunTrial& t = B.T[b];
                    int jb[2];
                    float4 pjs[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const bool on = k < t.nch && t.pres_old[k] && t.pres_new[k];
                        const int4 bk = t.bonds[k];
                        const int j = (sl == 0) ? bk.x : (sl == 1 ? bk.y : (sl == 2 ? bk.z : bk.w));
                        jb[k] = on ? j : -1;
                        pjs[k] = (jb[k] >= 0) ? d.posq[so + jb[k]] : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const int j = jb[k];
                        if (j < 0 || (t.nch == 2 && (j == t.idx[0] || j == t.idx[1]))) continue;
                        const float4 pj = pjs[k], pn = t.pn[k], po = t.po[k];
                        float dx = min_image(pn.x - pj.x, D.L[0]), dy = min_image(pn.y - pj.y, D.L[1]),
                              dz = min_image(pn.z - pj.z, D.L[2]);
                        const float en = fene_energy(D, dx * dx + dy * dy + dz * dz);
                        dx = min_image(po.x - pj.x, D.L[0]); dy = min_image(po.y - pj.y, D.L[1]);
                        dz = min_image(po.z - pj.z, D.L[2]);
                        const float eo = fene_energy(D, dx * dx + dy * dy + dz * dz);
                        df += (double)en - (double)eo;
                    }
                }
                if (b < nb) s_fene[b][sl] = df;
            } else if (it < Q_CF) {  // direct terms between two changed particles, charge moments
                const int b = it - Q_DI;
                if (b < nb && B.T[b].skip == 0) {
                    RunTrial& t = B.T[b];
                    double dl = 0.0, dc = 0.0, dQ = 0, dQ2 = 0, dMz = 0, dS2 = 0;
                    if (t.nch == 2) {
                        const bool bonded = in_bonds(t.bonds[0], t.idx[1]);
                        float elj, ec;
                        if (t.pres_new[0] && t.pres_new[1]) {
                            pair_energy(D, min_image(t.pn[0].x - t.pn[1].x, D.L[0]), min_image(t.pn[0].y - t.pn[1].y, D.L[1]),
                                        min_image(t.pn[0].z - t.pn[1].z, D.L[2]), t.tn[0], t.tn[1], t.pn[0].w, t.pn[1].w, bonded, elj, ec);
                            dl += elj; dc += ec;
                        }
                        if (t.pres_old[0] && t.pres_old[1]) {
                            pair_energy(D, min_image(t.po[0].x - t.po[1].x, D.L[0]), min_image(t.po[0].y - t.po[1].y, D.L[1]),
                                        min_image(t.po[0].z - t.po[1].z, D.L[2]), t.to[0], t.to[1], t.po[0].w, t.po[1].w, bonded, elj, ec);
                            dl -= elj; dc -= ec;
                        }
                    }
                    for (int k = 0; k < t.nch; ++k) {
                        if (t.pres_new[k]) {
                            const double q = t.pn[k].w, z = t.pn[k].z;
                            dQ += q; dQ2 += q * q; dMz += q * z; dS2 += q * z * z;
                        }
                        if (t.pres_old[k]) {
                            const double q = t.po[k].w, z = t.po[k].z;
                            dQ -= q; dQ2 -= q * q; dMz -= q * z; dS2 -= q * z * z;
                        }
                    }
                    t.direct_lj = dl; t.direct_c = dc;
                    t.dQ = dQ; t.dQ2 = dQ2; t.dMz = dMz; t.dS2 = dS2;
                }
            } else {  // would trial i, accepted, change trial j's pair or bond terms, or its wall verdict?
                // (a refused trial j has no probes: only the particles are compared)
                const int i = (it - Q_CF) / RUN_BATCH, j = (it - Q_CF) % RUN_BATCH;
                if (i < j && j < nb && B.T[i].skip == 0 && (B.T[j].skip == 0 || B.T[j].skip == 2)) {
                    const RunTrial &a = B.T[i], &b = B.T[j];
                    bool hit = false;
                    for (int p = a.p0; p < a.p0 + a.np && !hit; ++p)
                        for (int q = b.p0; q < b.p0 + b.np; ++q) {
                            const float4 u = B.pp[p], v = B.pp[q];
                            const float dx = near_image(u.x - v.x, D.L[0], s_iL[0]), dy = near_image(u.y - v.y, D.L[1], s_iL[1]),
                                        dz = near_image(u.z - v.z, D.L[2], s_iL[2]);
                            if (dx * dx + dy * dy + dz * dz <= s_rc2) { hit = true; break; }
                        }
                    for (int k = 0; k < a.nch; ++k)
                        for (int l = 0; l < b.nch; ++l)
                            hit = hit || a.idx[k] == b.idx[l] || (b.skip == 0 && in_bonds(b.bonds[l], a.idx[k]));
                    if (hit) atomicOr(&s_conf[i], 1u << j);
                }
            }
        }
        }
        }
        if constexpr (CL) {
            cg::this_cluster().sync();
            if (rank != 0) {  // the batch's tables, and every stencil, from the first block
                const RunShared* B0 = cg::this_cluster().map_shared_rank(&B, 0);
                const int n0 = *(volatile const int*)&B0->npend, n1 = *(volatile const int*)&B0->ns;
                const uint4* src = reinterpret_cast<const uint4*>(B0);
                uint4* dst = reinterpret_cast<uint4*>(&B);
                for (int k = tid; k < (int)(sizeof(RunShared) / 16); k += NT) dst[k] = src[k];
                const uint4* ss = reinterpret_cast<const uint4*>(cg::this_cluster().map_shared_rank(dsm, 0));
                uint4* sd = reinterpret_cast<uint4*>(dsm);
                const int nv = (int)((sizeof(PadSt<P>) * (n0 + n1) + 15) / 16);
                for (int k = tid; k < nv; k += NT) sd[k] = ss[k];
                __syncthreads();
                halt = B.stop;
            }
            if (halt) break;
        } else {
            if (halt) break;
            __syncthreads();
        }
        mark(2);
        const int nb = B.nb, npend = B.npend, ns = B.ns, npr = B.npr;
        // quorum of the launch: read here, compared after the pair work
        const bool q_chk = tid == 32 && s_qin;
        int q_started = 0, q_blocked = 0;
        if (q_chk) { q_started = *(volatile int*)&d.quorum_ctl[0]; q_blocked = *(volatile int*)&d.quorum_ctl[1]; }
        if (d.phase_clk) { __syncthreads(); mark(3); }
        // ---------------- pair terms: one warp per probe ----------------
        // lanes read the 27 cells' lists into the warp's list, then test 32 candidates at a time;
        // those within the largest cutoff (~15 %) queue up and are evaluated 32 at a time
        for (int p = warp * csize + rank; p < npr; p += NW * csize) {
            const RunTrial& t = B.T[B.pb[p]];
            const float4 pp = B.pp[p];
            const int pt = B.pt[p];
            const float sg = B.psg[p];
            const int4 bo = t.bonds[B.pk[p]];
            const int e0 = t.idx[0], e1 = t.nch == 2 ? t.idx[1] : -1;
            const int cap = D.cell_cap;
            int* list = s_list + warp * RUN_LIST;
            int* hitq = s_hit + warp * RUN_HIT;
            const int* row = nullptr;
            int cnt = 0;
            const bool wide = (cap & 3) == 0 && cap >= 8;
            int4 l0 = make_int4(-1, -1, -1, -1), l1 = l0;
            if (lane < 27) {
                const int cx = min(D.ncell[0] - 1, max(0, (int)(pp.x * D.cell_scale[0])));
                const int cy = min(D.ncell[1] - 1, max(0, (int)(pp.y * D.cell_scale[1])));
                const int cz = min(D.ncell[2] - 1, max(0, (int)(pp.z * D.cell_scale[2])));
                const int nc = (wrap1(cz + lane / 9 - 1, D.ncell[2]) * D.ncell[1] + wrap1(cy + (lane / 3) % 3 - 1, D.ncell[1])) *
                                   D.ncell[0] + wrap1(cx + lane % 3 - 1, D.ncell[0]);
                row = d.cell_list + ((size_t)D.cell_off + nc) * cap;
                if (wide) {  // the leading list entries in the count's round trip (those past it are not used)
                    l0 = ld(reinterpret_cast<const int4*>(row));
                    l1 = ld(reinterpret_cast<const int4*>(row) + 1);
                }
                cnt = min(ld(d.cell_count + D.cell_off + nc), cap);
            }
            int ofs = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, ofs, o);
                if (lane >= o) ofs += y;
            }
            const int total = __shfl_sync(0xffffffffu, ofs, 31);
            ofs -= cnt;
            double alj = 0.0, ac = 0.0;
            int nh = 0;
            auto evaluate = [&](int n) {  // the first n (<= 32) queued candidates, one per lane
                if (lane < n) {
                    const int j = hitq[lane];
                    const float4 pj = ld(d.posq + so + j);
                    float elj, ec;
                    pair_energy(D, near_image(pp.x - pj.x, D.L[0], s_iL[0]), near_image(pp.y - pj.y, D.L[1], s_iL[1]),
                                near_image(pp.z - pj.z, D.L[2], s_iL[2]), pt, ld(d.type + so + j), pp.w, pj.w, in_bonds(bo, j), elj, ec);
                    alj += (double)(sg * elj);
                    ac += (double)(sg * ec);
                }
            };
            for (int base = 0; base < total; base += RUN_LIST) {
                __syncwarp();
                const int lead[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int at = ofs + k - base;
                    if (k < cnt && at >= 0 && at < RUN_LIST) list[at] = wide ? lead[k] : ld(row + k);
                }
                for (int k = 8; k < cnt; ++k) {
                    const int at = ofs + k - base;
                    if (at >= 0 && at < RUN_LIST) list[at] = ld(row + k);
                }
                __syncwarp();
                const int m = min(total - base, RUN_LIST);
                for (int i0 = 0; i0 < m; i0 += 64) {  // two candidates per lane and step
                    int j_u[2];
                    float4 q_u[2];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int i = i0 + 32 * u + lane;
                        j_u[u] = i < m ? list[i] : -1;
                        if (j_u[u] == e0 || j_u[u] == e1) j_u[u] = -1;
                        if (j_u[u] >= 0) q_u[u] = ld(d.posq + so + j_u[u]);
                    }
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        bool hit = false;
                        if (j_u[u] >= 0) {
                            const float dx = near_image(pp.x - q_u[u].x, D.L[0], s_iL[0]),
                                        dy = near_image(pp.y - q_u[u].y, D.L[1], s_iL[1]),
                                        dz = near_image(pp.z - q_u[u].z, D.L[2], s_iL[2]);
                            hit = dx * dx + dy * dy + dz * dz <= s_rc2;
                        }
                        const unsigned hm = __ballot_sync(0xffffffffu, hit);
                        if (hit) hitq[nh + __popc(hm & ((1u << lane) - 1u))] = j_u[u];
                        nh += __popc(hm);
                        if (nh >= 32) {
                            __syncwarp();
                            evaluate(32);
                            const int rest = lane < nh - 32 ? hitq[32 + lane] : 0;
                            __syncwarp();
                            if (lane < nh - 32) hitq[lane] = rest;
                            nh -= 32;
                        }
                    }
                }
            }
            __syncwarp();
            evaluate(nh);
            __syncwarp();
            alj = warp_sum(alj);
            ac = warp_sum(ac);
            if (lane == 0) { r_plj[p] = alj; r_pc[p] = ac; r_pn[p] = total; }
        }
        if (rank == 0 && tid == NT - 1) {
            const float2 q = make_float2(0.9f * s_rate.x + (float)s_cut, 0.9f * s_rate.y + (float)s_decided);
            s_rate = q;
            s_len = run_length(q, worth, batch);
        }
        if (d.phase_clk) { __syncthreads(); mark(4); }
        // ---------------- mesh terms ----------------
        if (ns > 0) {
            const float* G = d.gext + D.gx_off;
            float* tab = s_tab + warp * RUN_TAB(P);
            const int nwarp = NW * (int)csize, gw = warp * (int)csize + (int)rank;
            // W . phi of trial b (one warp per trial, from the last warp down)
            for (int b = nwarp - 1 - gw; b < nb; b += nwarp) {
                const int nst = B.T[b].nst;
                if (nst == 0) continue;
                const PadSt<P>* st = s_st + npend + B.T[b].st0;
                const float* phi = d.phi + D.mesh_off;
                const int nx = D.mesh[0], ny = D.mesh[1];
                double acc = 0.0;
#pragma unroll 4
                for (int it = lane; it < nst * P3; it += 32) {
                    const int k = it / P3, rem = it - k * P3;
                    const int c = rem / (P * P), rb = rem - c * (P * P);
                    const int bb = rb / P, a = rb - bb * P;
                    const PadSt<P>& q = st[k];
                    const float v = phi[((size_t)q.m[2][c] * ny + q.m[1][bb]) * nx + q.m[0][a]];
                    acc += (double)(q.coef * q.wp[0][P + a] * q.wp[1][P + bb] * q.wp[2][P + c] * v);
                }
                acc = warp_sum(acc);
                if (lane == 0) r_phi[b] = acc;
            }
            // trial b's stencils with every earlier one, then its own pairs: half of (0, 0), all of
            // (0, 1), half of (1, 1).  A warp takes consecutive items, so that it loads a trial's
            // weights once
            const int per = (B.ntask + nwarp - 1) / nwarp;
            const int u0 = gw * per, u1 = min(B.ntask, u0 + per);
            int b = 0;
            bool fresh = true;
            for (int u = u0; u < u1; ++u) {
                while (u >= B.task[b + 1]) { ++b; fresh = true; }
                const int e = u - B.task[b];
                const int nst = B.T[b].nst, x0 = npend + B.T[b].st0;
                if (fresh) { lane_stencils<P>(L, D, s_st + x0, nst); fresh = false; }
                const PadSt<P>& sb = s_st[e];
                const float c0 = (e == x0 ? 0.5f : 1.0f) * L.coef0 * sb.coef, c1 = (e == x0 + 1 ? 0.5f : 1.0f) * L.coef1 * sb.coef;
                double acc = 0.0;
                int w = L.near && e <= x0 ? 2 : (e == x0 + 1 ? 1 : 0);
                for (;;) {  // both at once, or one after the other
                    const bool done = window_sum<P>(D, G, L, sb, w, c0, c1, tab, lane, acc);
                    if (!done) { w = 0; continue; }
                    if (w == 0 && nst == 2) { w = 1; continue; }
                    break;
                }
                acc = warp_sum(acc);
                if (lane == 0) r_unit[(size_t)b * us + e] = acc;
            }
        }
        if (q_chk && q_blocked > 0 && (float)q_blocked >= d.quorum * (float)q_started) s_qstop = 1;
        if constexpr (CL) cg::this_cluster().sync();
        else __syncthreads();
        mark(5);
        if (rank != 0) continue;
        // ---------------- decisions, in trial order ----------------
        if (warp == 0) {
            const bool have = lane < nb;
            const RunTrial& t = B.T[have ? lane : 0];
            const int skip = have ? t.skip : 1;
            const bool live = have && skip == 0;
            const int nst = live ? t.nst : 0;
            double dlj = 0.0, dc = 0.0, df = 0.0, own = 0.0, a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
            int ncand = 0;
            if (live) {
                for (int p = t.p0; p < t.p0 + t.np; ++p) { dlj += s_plj[p]; dc += s_pc[p]; ncand += s_pn[p]; }
                dlj += t.direct_lj; dc += t.direct_c;
                df = ((s_fene[lane][0] + s_fene[lane][1]) + s_fene[lane][2]) + s_fene[lane][3];
                if (nst) {
                    const double* un = s_unit + (size_t)lane * us;
                    const int x0 = npend + t.st0;
                    own = s_phi[lane] + un[x0];
                    if (nst == 2) own += un[x0 + 1];
                    // pending stencil e adds to accumulator e mod 4, whatever batch it came from
                    int e = 0;
                    for (; e + 4 <= npend; e += 4) { a0 += un[e]; a1 += un[e + 1]; a2 += un[e + 2]; a3 += un[e + 3]; }
                    if (e < npend) a0 += un[e];
                    if (e + 1 < npend) a1 += un[e + 1];
                    if (e + 2 < npend) a2 += un[e + 2];
                }
            }
            const double u01 = live ? u53(t.ua, t.ub) : 0.0;
            const double logf = live ? t.logf : 0.0;
            const long long t0 = S.trial;
            const long long li = t0 + lane - S.run_start;
            const bool logged = r == 0 && d.log_move;
            int cur = 0, n_end = nb, np = npend;
            int my_np = 0;             // pending stencils when this lane's trial was decided
            unsigned taken = 0u;       // accepted trials
            double dE = 0.0, rec = 0.0, dself = 0.0, dqc = 0.0, dslab = 0.0;
            double Qs = S.Q, Ms = S.Mz, S2s = S.S2;
            if (live && ewald) dself = D.self_coef * t.dQ2;
            const bool replayed = r == 0 && d.replay && li < d.replay_n;
            const int told = live && replayed ? d.replay[li] : 0;
            while (cur < n_end) {
                const bool in = live && lane >= cur && lane < n_end;
                int acc = 0;
                if (in) {
                    rec = own + ((a0 + a1) + (a2 + a3));
                    if (ewald) {
                        const double Qn = Qs + t.dQ;
                        dqc = D.qcorr_coef * (Qn * Qn - Qs * Qs);
                        dslab = slab_energy(D, Qn, Ms + t.dMz, S2s + t.dS2) - slab_energy(D, Qs, Ms, S2s);
                    }
                    dE = dlj + dc + df + rec + dself + dqc + dslab;
                    const double expo = -D.beta * dE + logf;
                    if (replayed) acc = told;
                    else if (expo >= 0.0) acc = 1;
                    else {
                        // the FP64 exp only when the uniform lies within 1e-3 (relative) of a float
                        // estimate, whose error is below 1e-4 for every expo < 0
                        const double ef = (double)__expf((float)expo);
                        if (u01 < ef * (1.0 - 1e-3)) acc = 1;
                        else if (u01 > ef * (1.0 + 1e-3)) acc = 0;
                        else acc = u01 < exp(expo);
                    }
                }
                const unsigned am = __ballot_sync(0xffffffffu, acc != 0);
                const int a = am ? __ffs(am) - 1 : n_end - 1;  // the first trial to accept, or the last one
                if (lane >= cur && lane <= a) my_np = np;      // trials cur .. a are decided now
                cur = a + 1;
                if (!am) break;
                taken |= 1u << a;
                const RunTrial& ta = B.T[a];
                Qs += ta.dQ; Ms += ta.dMz; S2s += ta.dS2;
                // its stencils become pending: their terms go to the later trials, at the accumulator of
                // their place in the pending list
                const int na = ta.nst, xa = npend + ta.st0;
                if (live && lane > a && nst) {
                    const double* un = s_unit + (size_t)lane * us;
                    for (int k = 0; k < na; ++k) {
                        const double v = un[xa + k];
                        const int m = (np + k) & 3;
                        if (m == 0) a0 += v; else if (m == 1) a1 += v; else if (m == 2) a2 += v; else a3 += v;
                    }
                }
                np += na;
                // later trials that this change could have altered start the next batch
                const unsigned cm = s_conf[a] & ~((2u << a) - 1u);
                if (cm) n_end = min(n_end, __ffs(cm) - 1);
                if (ta.lists || np + 2 > pend_max) n_end = cur;
            }
            // ---- bookkeeping of the decided trials 0 .. cur - 1, lane by lane ----
            const bool fin = have && lane < cur, mine = (taken >> lane) & 1u;
            if (fin && logged && li < d.log_cap) {
                d.log_move[li] = t.move;
                d.log_dE[li] = live ? dE : (skip == 2 ? __longlong_as_double(0x7ff0000000000000ll)
                                                      : __longlong_as_double(0x7ff8000000000000ll));
                d.log_acc[li] = mine ? 1 : 0;
                if (d.log_stage) { d.log_stage[li] = 0; d.log_dEs[li] = 0.0; }
            }
            const int mv = fin ? t.move : 3;
            // algorithmic bytes: float4 + type of every candidate, the moved particle, the phi
            // stencils and the pending-correction reads (whole numbers: exact in FP64)
            const int by = fin ? (live ? 20 * ncand + 16 + 4 * P3 * nst + 16 * P3 * my_np + (mine ? 32 : 0) : 16) : 0;
            const int bs = __reduce_add_sync(0xffffffffu, by);
            int n_att = 0, n_acc = 0;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const unsigned m = __ballot_sync(0xffffffffu, mv == k);
                if (lane == k) { n_att = __popc(m); n_acc = __popc(m & taken); }
            }
            if (lane < 3) { S.att[lane] += n_att; S.acc[lane] += n_acc; }
            // what the accepted ones change
            int n_mv = 0, mvs[2][3];
            if (mine) {
                const int k0 = __popc(taken & ((1u << lane) - 1u));
                const double ev[8] = {dE, dlj, dc, df, rec, dself, dqc, dslab};
#pragma unroll
                for (int k = 0; k < 8; ++k) s_ev[k0][k] = ev[k];
                for (int k = 0; k < t.nch; ++k) {
                    const int i = t.idx[k], gi = so + i;
                    const float4 o = t.po[k], nw = t.pn[k];
                    const bool pold = t.pres_old[k], pnew = t.pres_new[k];
                    const int c_old = pold ? cell_index(D, o.x, o.y, o.z) : -1;
                    const int c_new = pnew ? cell_index(D, nw.x, nw.y, nw.z) : -1;
                    {  // descriptor class table: leave the old (cell, class), enter the new one
                        const int k_old = pold ? desc_class(t.fo[k], o.w) : -1;
                        int fl_new = t.fo[k];
                        if (!pold && pnew)
                            fl_new = PHMC_F_MOBILE | (nw.w > 0.0f ? PHMC_F_CATION : (nw.w < 0.0f ? PHMC_F_ANION : 0));
                        const int k_new = pnew ? desc_class(fl_new, nw.w) : -1;
                        if (c_old != c_new || k_old != k_new) {
                            cls_add(d, D, c_old, k_old, -1);
                            cls_add(d, D, c_new, k_new, 1);
                        }
                    }
                    if (d.qband && !(pold && pnew && o.x == nw.x && o.y == nw.y && o.z == nw.z && o.w == nw.w)) {
                        if (pold && o.w != 0.0f) { const int j = atomicAdd(&s_nq, 1); s_qjob[j] = o; s_qsgn[j] = -1; }
                        if (pnew && nw.w != 0.0f) { const int j = atomicAdd(&s_nq, 1); s_qjob[j] = nw; s_qsgn[j] = 1; }
                    }
                    if (pnew) { d.posq[gi] = nw; d.type[gi] = t.tn[k]; }
                    if (c_old != c_new) { mvs[n_mv][0] = i; mvs[n_mv][1] = c_old; mvs[n_mv][2] = c_new; ++n_mv; }
                    if (!pold && pnew) {  // insertion into a free slot
                        int fk = -1;
                        for (int f = S.n_free - 1; f >= 0; --f) if (d.freel[so + f] == i) { fk = f; break; }
                        if (fk >= 0) { d.freel[so + fk] = d.freel[so + S.n_free - 1]; S.n_free--; }
                        int fl = PHMC_F_MOBILE;
                        list_append(d.mobile, d.mobile_pos, S.n_mobile, so, i);
                        if (nw.w > 0.0f) { fl |= PHMC_F_CATION; list_append(d.cations, d.cation_pos, S.n_cation, so, i); }
                        else if (nw.w < 0.0f) { fl |= PHMC_F_ANION; list_append(d.anions, d.anion_pos, S.n_anion, so, i); }
                        d.flags[gi] = fl;
                    } else if (pold && !pnew) {  // deletion
                        const int fl = d.flags[gi];
                        if (fl & PHMC_F_CATION) list_remove(d.cations, d.cation_pos, S.n_cation, so, i);
                        if (fl & PHMC_F_ANION) list_remove(d.anions, d.anion_pos, S.n_anion, so, i);
                        if (fl & PHMC_F_MOBILE) list_remove(d.mobile, d.mobile_pos, S.n_mobile, so, i);
                        d.flags[gi] = PHMC_F_GHOST;
                        d.freel[so + S.n_free] = i; S.n_free++;
                    }
                }
            }
            // places in the deferred lists, in trial order
            const int n_cp = mine ? nst : 0;
            int sc = n_cp | (n_mv << 16);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, sc, o);
                if (lane >= o) sc += y;
            }
            const int c0 = (sc & 0xffff) - n_cp, m0 = (sc >> 16) - n_mv;
            for (int k = 0; k < n_cp; ++k) { s_cp[c0 + k][0] = npend + t.st0 + k; s_cp[c0 + k][1] = npend + c0 + k; }
            for (int k = 0; k < n_mv; ++k)
                for (int q = 0; q < 3; ++q) s_mv[m0 + k][q] = mvs[k][q];
            if (lane == 31) {
                s_ncp = sc & 0xffff; s_nmv = sc >> 16; s_nev = __popc(taken);
                S.trials_run += cur; S.alg_bytes += (double)bs;
                S.Q = Qs; S.Mz = Ms; S.S2 = S2s;
                S.trial = t0 + cur; B.npend = np;
                s_cut = np + 2 <= pend_max && (cur < nb || (((taken >> (cur - 1)) & 1u) && B.T[cur - 1].lists));
                s_decided = cur;
            }
            if (taken && lane == 30) {
                double q2 = S.Q2;
                for (unsigned m = taken; m; m &= m - 1) q2 += B.T[__ffs(m) - 1].dQ2;
                S.Q2 = q2;
            }
        }
        __syncthreads();
        // z-density sample after every zh_every trials of the run
        if (d.zh_bins > 0 && S.trial % d.zh_every == 0) {
            const int nbn = d.zh_bins;
            for (int k = tid; k < 3 * nbn; k += NT) s_zh[k] = 0u;
            __syncthreads();
            const float z0 = D.walls ? D.wall_lo : 0.0f;
            const float inv = (float)nbn / (D.walls ? (D.wall_hi - D.wall_lo) : D.L[2]);
            for (int i = tid; i < D.cap; i += NT) {
                const int fl = d.flags[so + i];
                if (fl & PHMC_F_GHOST) continue;
                const float4 pq = d.posq[so + i];
                int cls = -1;
                if (fl & PHMC_F_TITRATABLE) cls = pq.w != 0.0f ? 0 : -1;
                else if (fl & PHMC_F_ANION) cls = 1;
                else if (fl & PHMC_F_CATION) cls = 2;
                if (cls < 0) continue;
                const int b = min(max((int)((pq.z - z0) * inv), 0), nbn - 1);
                atomicAdd(&s_zh[cls * nbn + b], 1u);
            }
            __syncthreads();
            unsigned long long* h = d.zhist + (size_t)r * 3 * nbn;  // this replica's row: one block, no race
            for (int k = tid; k < 3 * nbn; k += NT) h[k] += s_zh[k];
            if (tid == 0) d.zh_samples[r] += 1;
            __syncthreads();
        }
        mark(6);
    }
    if constexpr (CL) cg::this_cluster().sync();  // the first block's shared memory stays until all have left the loop
    if (tid == 0 && rank == 0) {
        unsigned long long t_end;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
        S.busy_ns += (long long)(t_end - t_start);
        d.state[r] = S;
        d.run_rate[r] = s_rate;
        if (B.npend > 0) d.dirty[r] = 1;  // potential mesh is stale: rebuild before the next MC launch
    }
}

size_t run_smem_bytes(int order, int nt, int pend_max) {
    const size_t st = order == 4 ? run_stencil_bytes<4>(pend_max) : (order == 5 ? run_stencil_bytes<5>(pend_max) : run_stencil_bytes<6>(pend_max));
    const int tab = order == 4 ? RUN_TAB(4) : (order == 5 ? RUN_TAB(5) : RUN_TAB(6));
    return st + sizeof(double) * RUN_BATCH * run_unit_stride(pend_max) + sizeof(float) * (nt / 32) * (tab + RUN_LIST + RUN_HIT);
}

// Launch shape: with more replicas than SMs a block of the tuning's size per replica, two of
// them to an SM; otherwise a replica takes blocks of 512 threads, the largest cluster (8, 4, 2, 1)
// with which all replicas are resident at once.
template <int P, int NT, bool CL>
static cudaError_t launch_run_t(Engine& E, int csize, int batch, float worth, cudaStream_t st) {
    DevPtrs dd = E.d;
    auto kern = k_mc_run<P, NT, CL>;
    const size_t smem = run_smem_bytes(P, NT, E.pend_max);
    // launch quorum only when every replica's block is resident from the start (otherwise
    // late blocks would count against a quorum the early ones already reached)
    dd.quorum = 1.0f;
    if (E.quorum < 1.0f) {
        bool resident = CL;
        if (!CL) {
            int per_sm = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem);
            resident = (long long)per_sm * E.nsm >= E.R;
        }
        if (resident) {
            dd.quorum = E.quorum;
            cudaError_t e = cudaMemsetAsync(E.d.quorum_ctl, 0, 2 * sizeof(int), st);
            if (e != cudaSuccess) return e;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(E.R * csize);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = csize; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CL ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, dd, E.pend_max, batch, worth);
}

template <int P, int NT, bool CL>
static cudaError_t prepare_run_t(Engine& E) {
    int optin = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, E.device);
    if (e != cudaSuccess) return e;
    cudaFuncAttributes fa;
    e = cudaFuncGetAttributes(&fa, k_mc_run<P, NT, CL>);
    if (e != cudaSuccess) return e;
    const int cap = optin - (int)fa.sharedSizeBytes;
    if ((size_t)cap < run_smem_bytes(P, NT, E.pend_max)) return cudaErrorInvalidValue;
    return cudaFuncSetAttribute(k_mc_run<P, NT, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, cap);
}

// Picks the launch shape and raises that kernel's shared-memory limit.
template <int P>
static cudaError_t prepare_run_p(Engine& E) {
    E.run_cluster = 1;
    if (E.R > E.nsm) return E.threads == 256 ? prepare_run_t<P, 256, false>(E) : prepare_run_t<P, 128, false>(E);
    for (int cs = 8; cs > 1; cs /= 2) {
        if (E.R * cs > E.nsm) continue;
        cudaError_t e = prepare_run_t<P, 512, true>(E);
        if (e != cudaSuccess) return e;
        if (E.R <= 4) { E.run_cluster = cs; return cudaSuccess; }  // (every GPC holds at least one)
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(E.R * cs);
        cfg.blockDim = dim3(512);
        cfg.dynamicSmemBytes = run_smem_bytes(P, 512, E.pend_max);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;  // clusters resident at once
        if (cudaOccupancyMaxActiveClusters(&n, k_mc_run<P, 512, true>, &cfg) != cudaSuccess) { cudaGetLastError(); n = 0; }
        if (n >= E.R) { E.run_cluster = cs; return cudaSuccess; }
    }
    return prepare_run_t<P, 512, false>(E);
}

// The longest batch: on one block 16 trials' work takes longer than what they save (300 trials of 96
// uneven replicas 7.5 ms with 16, 5.6 with 8).  worth (run_length) by trial: 1 to 16 trials always,
// one to 149 replicas of 40 and 300 particles, titrations, swaps or displacements; within 5 % of the best.
template <int P>
static cudaError_t launch_run_p(Engine& E, cudaStream_t st) {
    if (E.run_cluster > 1) return launch_run_t<P, 512, true>(E, E.run_cluster, RUN_BATCH, E.run_cluster == 8 ? 28.0f : 2.5f * E.run_cluster, st);
    if (E.R <= E.nsm) return launch_run_t<P, 512, false>(E, 1, RUN_BATCH / 2, 2.2f, st);
    if (E.threads == 256) return launch_run_t<P, 256, false>(E, 1, RUN_BATCH / 2, 1.5f, st);
    return launch_run_t<P, 128, false>(E, 1, RUN_BATCH / 2, 1.2f, st);
}

cudaError_t prepare_mc_run(Engine& E) {
    if (E.nsm == 0) {
        cudaError_t e = cudaDeviceGetAttribute(&E.nsm, cudaDevAttrMultiProcessorCount, E.device);
        if (e != cudaSuccess) return e;
    }
    switch (E.order) {
        case 4: return prepare_run_p<4>(E);
        case 5: return prepare_run_p<5>(E);
        default: return prepare_run_p<6>(E);
    }
}

cudaError_t launch_mc_run(Engine& E, cudaStream_t st) {
    switch (E.order) {
        case 4: return launch_run_p<4>(E, st);
        case 5: return launch_run_p<5>(E, st);
        default: return launch_run_p<6>(E, st);
    }
}
