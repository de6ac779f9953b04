// Cholesky QR of unfoldings with at most 32 columns by one thread-block
// cluster (included by ptt_round.cu inside its anonymous namespace, after the
// warp-level TSQR).
//
// The Householder TSQR is a chain of c x (tree depth + 1) dependent reflector
// steps; here the only sequential work is a c-step Cholesky of a c x c Gram
// matrix per stage, in 8 x 8 blocks.  The rules of the stages are those of
// ptt_gramstage.cuh.
//
// CTA b of the cluster keeps rows [b h, (b+1) h) (h = ceil(m / CS)) in shared
// memory for all stages and writes the partial Gram matrix of its rows into its
// shared memory; after a cluster barrier CTA b sums slice b of the entries over
// all partials (distributed shared memory, CTA order 0..CS-1) and stores it
// into every CTA's Gram matrix, and after another one every CTA takes the same
// decision and factor from it -- identical data and arithmetic, so nothing
// else is broadcast.  (Every CTA summing all partials moves 15 times the
// matrix out of each SM: 2k cycles a stage at 16 columns, 5k at 32, against
// ~1.5k with the second barrier.)  Within a CTA every warp takes the decision
// by itself (lane = column) and warp 0 forms the factor.
//
// Bound by the latency of a stage (row solve, products, two barriers, remote
// sum, decision, factor: ~8k cycles at 16 columns, ~15k at 32).  With one lane
// per column in the Cholesky (~400 cycles a column, plain and shifted factors
// in two warps), the decision's column loops in sequence, the row solve's
// factor entries broadcast from shared memory one by one and 3.8 stages a
// bond instead of 2.7, a factorisation of a time step took 29 us at 16 columns
// and 123 us at 32; now 17 and 54.
//
// On success Q is written once: LEFT -> alt[k] (m x c, column-major), RIGHT_T
// -> core[k] in place (row-major rows of c; k_cq_write forms Q V_r from it
// after the bond's SVD).  A bond that does not converge within MAXST stages,
// has more columns than rows or meets a NaN or a zero matrix is left untouched
// and falls back to the Householder TSQR: k_wfactor / k_wapply skip the bonds
// finished here and k_cq_write skips the others.
#pragma once

namespace cq {

namespace cg = cooperative_groups;
using namespace gst;

constexpr int NT = 256;       // threads per CTA
constexpr int MAXST = 7;      // Gram stages per factorisation
constexpr int CSMAX = 16;     // CTAs per cluster (non-portable size)
constexpr double TAUC = 1e-15;  // as gst::TAU: a cluster's first-order finish costs one more row solve (~1 us), so
                                // it is taken down to the rounding of G itself
constexpr int RTARGET = 64;   // rows per CTA the cluster size aims at: every part but the two barriers shrinks
                              // with the rows (m = 1280, c = 20: 31 us with 4 CTAs, 27 with 16)
static_assert(DONE == wt::CQ_DONE, "state code shared with the TSQR kernels");

// Per-bond record at wsb + o_cq (REGION doubles).
struct State {
    int state;   // RUN, DONE or FALLBACK
    int nst;     // factors applied to Q
    int m, c;    // size of the factored unfolding
    int ndrop;   // columns dropped (diagnostic)
    int pad[3];
};
constexpr long long REGION = 32;

template <int CB>
struct Cfg {
    static constexpr int XP = CB + 4;  // shared row pitch: 4 mod 8 doubles, for the fragment loads
    static constexpr int NB = CB / 8, NTL = NB * (NB + 1) / 2, UP = NTL * 64;  // upper 8 x 8 tiles
};

// shared memory (doubles): 4 warp-pair partials (the factor in the first of
// them), the folded partial, the Gram matrix, two accumulated R, column
// scalars, then the CTA's rows
template <int CB>
__host__ __device__ constexpr long long fixed_smem() {
    return 8LL * Cfg<CB>::UP + 6 * 32;
}
template <int CB>
__host__ __device__ constexpr size_t smem(int rpb) {
    return sizeof(double) * (size_t)(fixed_smem<CB>() + (long long)((rpb + 15) & ~15) * Cfg<CB>::XP);
}
constexpr size_t SMEM_MAX = 226 * 1024;  // dynamic; leaves room for the static variables
template <int CB>
__host__ __device__ constexpr int rpb_max() {
    return (int)(((long long)(SMEM_MAX / sizeof(double)) - fixed_smem<CB>()) / Cfg<CB>::XP) & ~15;
}

// Cholesky factor of the equilibrated Gram matrix in the tiles at sF (nbc
// column blocks), in place, by one warp (see gst::chol8); `live`: bits of the
// columns kept; rinv[j] = 1 / R[j][j].
template <int CB>
__device__ __forceinline__ void warp_chol(double* sF, int nbc, unsigned live, double* rinv) {
    const int lane = threadIdx.x & 31, li = lane >> 2, lk = lane & 3;
    for (int J = 0; J < nbc; J++) {
        double r[8][8], inv[8];
        const int col = 8 * J + 8 + lane;  // this lane's column of the block row
        const unsigned weak = chol8(sF + tnum(J, J) * 64, (live >> (8 * J)) & 0xffu, r, inv);
        __syncwarp();
        if (col < 8 * nbc) solve8(sF + tnum(J, col >> 3) * 64, col & 7, r, inv, weak);
        if (lane == 31) {
            double* G = sF + tnum(J, J) * 64;
#pragma unroll
            for (int i = 0; i < 8; i++) {
#pragma unroll
                for (int j = 0; j < 8; j++) G[tix(i, j)] = j >= i ? r[i][j] : 0.0;
                rinv[8 * J + i] = inv[i];
            }
        }
        __syncwarp();
        for (int K = J + 1; K < nbc; K++)
            for (int I = J + 1; I <= K; I++) trail8(sF, J, I, K, li, lk);
        __syncwarp();
    }
}

// Factor core k's unfolding (mode) by the Cholesky sequence above.  Launched
// as one cluster of CS CTAs with room for rpb rows each (m <= CS rpb, else
// fallback); CTA b takes rows [b ceil(m / CS), ...).
template <int CB>
__global__ void __launch_bounds__(NT, 1) k_cq_factor(const DevDesc* D, int k, int mode, Plan pl, wt::WP wp,
                                                  double* wsb, int rpb, long long* qstat) {
    PTT_PDL_ENTRY();
    using C = Cfg<CB>;
    constexpr int XP = C::XP, NB = C::NB, NTL = C::NTL, UP = C::UP;
    constexpr unsigned FULL = 0xffffffffu;
    cg::cluster_group cl = cg::this_cluster();
    const int CS = (int)cl.num_blocks();
    const int crank = (int)cl.block_rank();
    extern __shared__ __align__(16) double csm[];
    double* sScr = csm;             // 4 warp-pair partials
    double* sF = csm;               // the factor of the stage, once the partials are folded
    double* sP = sScr + 4 * UP;     // folded partial, read by the other CTAs
    double* sG = sP + UP;           // Gram matrix of the whole unfolding, written by all CTAs
    double* sT = sG + UP;           // accumulated R = R_s ... R_1
    double* sTn = sT + UP;          // the other buffer of it
    double* s_rinv = sTn + UP;      // inverse pivots of sF
    double* s_an = s_rinv + 32;     // 1 / |a_j|
    double* s_d = s_an + 32;        // D of the columns kept, its inverse
    double* s_di = s_d + 32;
    unsigned long long* s_tm = (unsigned long long*)(s_di + 32);  // max_j |T_ij| / |a_j|, two buffers
    double* Xs = s_di + 96;         // rpb x XP rows of this CTA
    State* st = (State*)(wsb + wp.o_cq);
    const View A = make_view(D, k, mode, false);
    const int m = A.m, c = A.c;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, li = lane >> 2, lk = lane & 3;
    if (c > CB || c < 1 || m < c || (long long)m > (long long)rpb * CS) {  // uniform: Householder TSQR
        if (crank == 0 && tid == 0) {
            st->state = FALLBACK;
            st->nst = 0;
            if (qstat) atomicAdd((unsigned long long*)(qstat + 1), 1ull);
        }
        return;
    }
    if (pl.work && crank == 0 && tid == 0) atomicAdd(pl.work, 16.0 * (double)m * (double)c);
    // the actual rows spread evenly: the host sized rpb (and the shared
    // memory) from a bound on m, which the truncation sweep's shrinking
    // ranks leave well above the rows a bond has
    const int rpbd = (m + CS - 1) / CS;  // <= rpb
    const int r0 = crank * rpbd;
    const int h = (m - r0) < rpbd ? ((m - r0) > 0 ? (m - r0) : 0) : rpbd;
    const int nbc = (c + 7) >> 3, nt = nbc * (nbc + 1) / 2;
    // this CTA's rows, every element in flight by cp.async; zeros beyond c
    {
        const unsigned xs0 = (unsigned)__cvta_generic_to_shared(Xs);
        if (mode == LEFT) {  // column-major: a warp copies a column's contiguous rows
            for (int col = warp; col < c; col += NT / 32) {
                const double* g = A.p + (long long)r0 + (long long)col * m;
                for (int row = lane; row < h; row += 32)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(xs0 + 8u * (unsigned)(row * XP + col)),
                                 "l"(g + row)
                                 : "memory");
            }
        } else {  // RIGHT_T: this CTA's rows are one contiguous range, stepped without divisions
            const int dq = NT / c, dr = NT - dq * c, tot = h * c;
            int row = tid / c, col = tid - row * c;
            const double* g = A.p + (long long)r0 * c;
            for (int f = tid; f < tot; f += NT) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(xs0 + 8u * (unsigned)(row * XP + col)),
                             "l"(g + f)
                             : "memory");
                row += dq;
                col += dr;
                if (col >= c) {
                    col -= c;
                    row++;
                }
            }
        }
        const int cz = CB - c, h16 = (h + 15) & ~15;
        for (int col = warp; col < cz; col += NT / 32)
            for (int row = lane; row < h; row += 32) Xs[row * XP + c + col] = 0.0;
        for (int e = tid; e < (h16 - h) * XP; e += NT) Xs[h * XP + e] = 0.0;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    __syncthreads();
    // Gram warps: rows [4 ks0, 4 ks1) of this CTA, every 8 x 8 tile of the
    // column blocks (mma.m8n8k4: four rows a step, a block's fragment serves
    // as A and as B)
    const int nks = (h + 3) / 4;
    const int ks0 = (nks * warp) / (NT / 32), ks1 = (nks * (warp + 1)) / (NT / 32);
    const double dropc = DROP * sqrt((double)c);
    int dec = RUN, nst = 0, stage = 0, ndrop = 0;
    unsigned live = 0;
    for (stage = 0; stage < MAXST; stage++) {
        if (stage > 0) {  // Q_stage = Q_{stage-1} R_stage^{-1}
            tile_solve<XP, NT / 32>(Xs, h, sF, s_rinv, nbc);
            __syncthreads();
        }
        // partial Gram of this CTA's rows on the FP64 tensor cores: each warp
        // its rows, all tiles; warps w and w + 4 are added in shared memory,
        // then the four sums in warp order
        {
            double c0[NTL], c1[NTL];
#pragma unroll
            for (int t = 0; t < NTL; t++) c0[t] = c1[t] = 0.0;
            for (int ks = ks0; ks < ks1; ks++) {
                const double* xr = Xs + (4 * ks + lk) * XP + li;
                double f[NB];
#pragma unroll
                for (int bb = 0; bb < NB; bb++) f[bb] = xr[8 * bb];
                int t = 0;
#pragma unroll
                for (int J = 0; J < NB; J++)
#pragma unroll
                    for (int I = 0; I <= J; I++, t++) mma884(c0[t], c1[t], f[I], f[J]);
            }
            double* slot = sScr + (warp & 3) * UP + tix(li, 2 * lk);
            if (warp < 4) {
#pragma unroll
                for (int t = 0; t < NTL; t++) *(double2*)(slot + t * 64) = make_double2(c0[t], c1[t]);
            }
            __syncthreads();
            if (warp >= 4) {
#pragma unroll
                for (int t = 0; t < NTL; t++) {
                    const double2 v = *(const double2*)(slot + t * 64);
                    *(double2*)(slot + t * 64) = make_double2(v.x + c0[t], v.y + c1[t]);
                }
            }
            __syncthreads();
        }
        for (int u = tid; u < nt * 64; u += NT)
            sP[u] = ((sScr[u] + sScr[UP + u]) + sScr[2 * UP + u]) + sScr[3 * UP + u];
        cl.sync();  // every CTA's partial is complete and visible
        // this CTA's slice of the entries, summed in CTA order (every load
        // issued before the sums), into every CTA's Gram matrix
        {
            const int per = (nt * 64 + CS - 1) / CS, u0 = crank * per;
            for (int e = tid; e < per; e += NT) {
                const int u = u0 + e;
                if (u < nt * 64) {
                    double v[CSMAX];
#pragma unroll
                    for (int b = 0; b < CSMAX; b++) v[b] = b < CS ? cl.map_shared_rank(sP, b)[u] : 0.0;
                    double s2 = 0.0;
#pragma unroll
                    for (int b = 0; b < CSMAX; b++) s2 += v[b];  // zeros beyond CS leave the sum unchanged
#pragma unroll
                    for (int b = 0; b < CSMAX; b++)
                        if (b < CS) cl.map_shared_rank(sG, b)[u] = s2;
                }
            }
        }
        cl.sync();  // the Gram matrix is complete in every CTA
        // the decision, by every warp from the same data: lane = column
        double dj;
        float emaxf = 0.f;
        {
            const double gjj = lane < c ? sG[telem(lane, lane)] : 0.0;
            dj = gjj > 0.0 ? sqrt(gjj) : 0.0;
            bool on = gjj > 0.0;
            if (stage > 0)
                on = on && dj * __longlong_as_double((long long)s_tm[32 * (stage & 1) + lane]) > dropc;
            bool bad = lane < c && (!(gjj >= 0.0 && gjj < LARGE) || (gjj != 0.0 && gjj < SMALL));
            live = __ballot_sync(FULL, on);
            const unsigned l0 = live >> li, l1 = live >> (2 * lk);
#pragma unroll
            for (int J = 0; J < NB; J++) {
                if (8 * J < c) {  // uniform
#pragma unroll
                    for (int I = 0; I <= J; I++) {  // two entries a lane of every tile
                        const double2 v = *(const double2*)(sG + tnum(I, J) * 64 + tix(li, 2 * lk));
                        const bool d0 = I == J && li == 2 * lk, d1 = I == J && li == 2 * lk + 1;
                        bad = bad || !(v.x - v.x == 0.0) || !(v.y - v.y == 0.0);
                        const float e0 = fabsf((float)(v.x - (d0 ? 1.0 : 0.0))), e1 = fabsf((float)(v.y - (d1 ? 1.0 : 0.0)));
                        const bool oi = (l0 >> (8 * I)) & 1u;
                        if (oi && ((l1 >> (8 * J)) & 1u)) emaxf = fmaxf(emaxf, e0);
                        if (oi && ((l1 >> (8 * J + 1)) & 1u)) emaxf = fmaxf(emaxf, e1);
                    }
                }
            }
            // non-negative values order as their bits; the thresholds lie decades
            // apart, so single precision decides
            emaxf = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(emaxf)));
            if (__any_sync(FULL, bad)) live = 0u;
        }
        const double emax = (double)emaxf;
        ndrop = c - __popc(live);
        if (live == 0u) {
            dec = FALLBACK;
        } else if (stage >= 1 && emax <= TAUC) {
            dec = DONE;
        } else if (stage == MAXST - 1) {
            dec = FALLBACK;
        } else if (stage >= 1 && emax <= FIRST) {
            dec = emax <= FIRST_DONE ? FINISH : RUN;
        } else {
            dec = RUN;
        }
        if (dec == DONE || dec == FALLBACK) break;
        const bool first = stage >= 1 && emax <= FIRST;
        nst = stage + 1;
        // H (or the first-order factor) into sF by all warps; the column
        // scalars by each warp (the same values)
        {
            const bool on = (live >> lane) & 1u;
            double p2, ip2;
            pow2_above(dj, &p2, &ip2);
            s_d[lane] = on ? p2 : 0.0;
            s_di[lane] = on ? ip2 : 0.0;
            if (stage == 0) s_an[lane] = on ? 1.0 / dj : 0.0;
            if (warp == 0) s_tm[32 * ((stage + 1) & 1) + lane] = 0ull;
            __syncwarp();
        }
        for (int t = warp; t < nt; t += NT / 32) {
            int I, J;
            tile_of(t, &I, &J);
            const int at = t * 64 + tix(li, 2 * lk);
            const double2 v = *(const double2*)(sG + at);
            const int i = 8 * I + li, j = 8 * J + 2 * lk;
            double2 w;
            if (first) {
                const bool oi = (live >> i) & 1u, o0 = (live >> j) & 1u, o1 = (live >> (j + 1)) & 1u;
                w.x = !(oi && o0) || j < i ? 0.0 : (i == j ? 1.0 + 0.5 * (v.x - 1.0) : v.x);
                w.y = !(oi && o1) || j + 1 < i ? 0.0 : (i == j + 1 ? 1.0 + 0.5 * (v.y - 1.0) : v.y);
                if (i == j) s_rinv[i] = w.x != 0.0 ? 1.0 / w.x : 0.0;
                if (i == j + 1) s_rinv[i] = w.y != 0.0 ? 1.0 / w.y : 0.0;
            } else {
                w.x = v.x * s_di[i] * s_di[j];
                w.y = v.y * s_di[i] * s_di[j + 1];
            }
            *(double2*)(sF + at) = w;
        }
        __syncthreads();
        if (!first) {
            if (warp == 0) {
                warp_chol<CB>(sF, nbc, live, s_rinv);
                if (lane < 8 * nbc) s_rinv[lane] *= s_di[lane];
            }
            __syncthreads();
            for (int t = warp; t < nt; t += NT / 32) {  // R = chol(H) D
                int I, J;
                tile_of(t, &I, &J);
                double2* pv = (double2*)(sF + t * 64 + tix(li, 2 * lk));
                const double2 v = *pv;
                *pv = make_double2(v.x * s_d[8 * J + 2 * lk], v.y * s_d[8 * J + 2 * lk + 1]);
            }
            __syncthreads();
        }
        // R <- R_{stage+1} R into the other buffer, and max_j |R_ij| / |a_j|
        for (int t = warp; t < nt; t += NT / 32) {
            int I, J;
            tile_of(t, &I, &J);
            const int at = t * 64 + tix(li, 2 * lk);
            const double2 v = stage == 0 ? *(const double2*)(sF + at) : tile_product(sF, sT, I, J, li, lk);
            *(double2*)(sTn + at) = v;
            const int j = 8 * J + 2 * lk;
            const double w = fmax(fabs(v.x) * s_an[j], fabs(v.y) * s_an[j + 1]);
            atomicMax(&s_tm[32 * ((stage + 1) & 1) + 8 * I + li], (unsigned long long)__double_as_longlong(w));
        }
        {
            double* t2 = sT;
            sT = sTn;
            sTn = t2;
        }
        if (dec == FINISH) {  // apply the first-order factor; Q is final
            tile_solve<XP, NT / 32>(Xs, h, sF, s_rinv, nbc);
            __syncthreads();
            dec = DONE;
            live = FULL;  // R carries the dropped columns' zero rows
            break;
        }
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while another may still read its partials
    if (dec == DONE) {
        // a column dropped by the deciding stage is still in Xs: zero in Q, as its row of R
        if (mode == LEFT) {
            double* out = D->alt[k];
            for (int col = warp; col < c; col += NT / 32) {
                double* g = out + (long long)r0 + (long long)col * m;
                const bool on = (live >> col) & 1u;
                for (int row = lane; row < h; row += 32) g[row] = on ? Xs[row * XP + col] : 0.0;
            }
        } else {
            double* out = A.p + (long long)r0 * c;  // in place over A: this CTA's rows only
            const int dq = NT / c, dr = NT - dq * c, tot = h * c;
            int row = tid / c, col = tid - row * c;
            for (int f = tid; f < tot; f += NT) {
                out[f] = (live >> col) & 1u ? Xs[row * XP + col] : 0.0;
                row += dq;
                col += dr;
                if (col >= c) {
                    col -= c;
                    row++;
                }
            }
        }
        if (crank == 0) {
            double* Rs = wsb + wp.o_R;  // root slot, row-major 32 x 32
            for (int e = tid; e < 1024; e += NT) {
                const int i = e >> 5, j = e & 31;
                Rs[e] = (i < c && j < c && j >= i && ((live >> i) & 1u)) ? sT[telem(i, j)] : 0.0;
            }
            if (tid == 0) {
                Info* info = (Info*)(wsb + pl.o_info_d);
                info->m = m;
                info->c = c;
                info->q = c;
                info->rank = 0;
                info->status = 0;
                if (qstat) {
                    atomicAdd((unsigned long long*)qstat, 1ull);
                    atomicAdd((unsigned long long*)(qstat + 2), (unsigned long long)(stage + 1));
                }
            }
        }
    }
    if (crank == 0 && tid == 0) {
        st->state = dec;
        st->nst = nst;
        st->m = m;
        st->c = c;
        st->ndrop = ndrop;
        if (dec == FALLBACK && qstat) atomicAdd((unsigned long long*)(qstat + 1), 1ull);
    }
}

// alt[k][row * rank + col] = (Q V_r)(row, col) for the RIGHT_T bonds k0 ..
// k0 + gridDim.y - 1 that the Cholesky sequence finished: Q is in core[k]
// (row-major rows of c), V_r in Bn (row-major 32 x KC).
template <int CB>
__global__ void __launch_bounds__(NT) k_cq_write(const DevDesc* D, int k0, Plan pl, wt::WP wp, double* ws) {
    PTT_PDL_ENTRY();
    __shared__ double sB[32 * 33];
    const int k = k0 + blockIdx.y;
    double* wsb = ws + (long long)k * wp.stride;
    const State* st = (const State*)(wsb + wp.o_cq);
    if (st->state != DONE) return;
    const Info* info = (const Info*)(wsb + pl.o_info_d);
    if (info->status) return;
    const int m = info->m, c = info->c, qB = info->rank;
    const int tid = threadIdx.x;
    const double* Bn = wsb + pl.o_Bn;
    for (int e = tid; e < 1024; e += NT) {
        const int t = e >> 5, l = e & 31;
        sB[t * 33 + l] = (t < c && l < qB) ? Bn[(long long)t * pl.KC + l] : 0.0;
    }
    __syncthreads();
    const double* Q = D->core[k];
    double* out = D->alt[k];
    for (int row = blockIdx.x * NT + tid; row < m; row += gridDim.x * NT) {
        double x[CB];
#pragma unroll
        for (int t = 0; t < CB; t++) x[t] = t < c ? Q[(long long)row * c + t] : 0.0;
        for (int l = 0; l < qB; l++) {
            double y = 0.0;
#pragma unroll
            for (int t = 0; t < CB; t++) y = fma(x[t], sB[t * 33 + l], y);
            out[(long long)row * qB + l] = y;
        }
    }
}

}  // namespace cq
