// Cholesky QR of unfoldings with 33 to 128 columns by the whole GPU (included
// by ptt_round.cu inside its anonymous namespace, after ptt_cholqr.cuh).
//
// At 64 columns a bond's unfolding (16384 x 64 doubles at d = 40, n = 256,
// rank 64: 8.4 MB) does not fit one cluster's shared memory, and the
// Householder TSQR costs one block barrier per reflector and tree level.
// Here the rows are spread over all SMs and A = Q R is a sequence of Gram
// stages, two launches each:
//
//   k_gq_rows    CTA b loads its rows of Q_{s-1} (A for s <= 1), applies the
//                factor of the previous stage by a row-wise triangular solve
//                (s >= 1: Q_s = Q_{s-1} R_s^{-1}, written back) and forms the
//                partial Gram matrix of its rows of Q_s;
//   k_gq_decide  CTA t sums upper 8 x 8 tile t over all partials in a fixed
//                order; the last CTA to finish (atomic ticket, no waiting)
//                takes the decision of the stage from the whole Gram matrix.
//
// The sum is a launch of its own because one SM reading all partials took
// longer than everything else it had to do (the partials are 18 KB each at 64
// columns and 70 KB at 128; a single SM reads them at ~64 bytes a cycle).
//
// The rules of a stage are those of ptt_gramstage.cuh.
// The host launches MAXST stages; a launch finds the state left by the
// previous one and returns at once when the factorisation is finished.
//
// Q is written to Qbuf: LEFT -> alt[k] (m x c, column-major, its final place);
// RIGHT_T -> a scratch region (row-major rows of c), from which k_gq_write
// forms Q V_r after the bond's SVD.  A never changes, so a bond that falls
// back (NaN, zero matrix, more columns than rows, no convergence in MAXST
// stages) is factored by the Householder TSQR from the same input; those
// kernels skip the bonds finished here (Plan::gqstate).
#pragma once

namespace gq {

using namespace gst;

constexpr int NT = 256;
constexpr int RPB_MIN = 16;
constexpr int MAXST = 6;               // Gram stages per factorisation
constexpr int GROUP = 8;               // k_gram: CTAs summed by the first level
template <int CB>
struct Cfg {
    static constexpr int NB = CB / 8;
    static constexpr int NTI = NB * (NB + 1) / 2;
    static constexpr int UP = NTI * 64;          // doubles of the upper tiles
    static constexpr int XP = CB + 4;            // pitch of the rows in shared memory: 4 mod 16 doubles, so the
                                                 // 4 x 4 elements of a half-warp's fragment load fall in different
                                                 // banks (a pitch of 8 mod 16 cost two wavefronts more per load)
    static constexpr int RPB_MAX = CB <= 64 ? 112 : 128;  // rows per CTA: 16 for each of eight warps
    static constexpr int FL = UP + CB;           // a factor and its inverse pivots
    static constexpr size_t SM_ROWS = sizeof(double) * ((size_t)RPB_MAX * XP + FL);
    static constexpr size_t SM_DEC = sizeof(double) * (2 * (size_t)UP);
    // record (doubles): State, factor + inverse pivots, accumulated R, 1 / |a_j|, max_j |T_ij| / |a_j|, Gram sums
    static constexpr long long O_FAC = 8, O_T = O_FAC + FL, O_AN = O_T + UP, O_TM = O_AN + CB, O_G = O_TM + CB;
    static constexpr long long REC = O_G + UP;
};
// the Ozaki Gram (ptt_ozaki.cuh): the digit slices take the factor's region
// and beyond once the rows are solved; its 64 x 65 sum buffer the rows' region
constexpr size_t SM_ROWS_OZ = sizeof(double) * (size_t)Cfg<64>::RPB_MAX * Cfg<64>::XP + oz::SMEM;
static_assert(Cfg<64>::RPB_MAX == oz::KMAX, "one CTA's rows are one exact FP32 accumulation");
static_assert(SM_ROWS_OZ >= Cfg<64>::SM_ROWS && Cfg<64>::RPB_MAX * Cfg<64>::XP >= 64 * 65, "Ozaki buffers");
static_assert(Cfg<128>::SM_ROWS <= 227 * 1024 && Cfg<128>::SM_DEC <= 227 * 1024, "shared memory");

__host__ __device__ __forceinline__ bool finished(int s) { return s == DONE || s == FINISH; }

// Record of the factorisation in flight (rec[0..)):
struct State {
    int state;   // RUN, DONE, FALLBACK, FINISH
    int fin;     // FINISH: the stage launch that applies the last factor
    int nst;     // factors applied
    int ndrop;   // columns dropped (diagnostic)
    int m, c;
    int pad[2];
};

struct GQ {
    double* rec;         // State, then the arrays of Cfg
    double* part;        // per-CTA partial Gram matrices (UP each)
    double* qscr;        // Q rows of a RIGHT_T factorisation (row-major, pitch c)
    int* cnt;            // ticket, zero between launches
    int rpb;             // rows a CTA has room for
    int nb;              // CTAs of the row launches
};

// rows per CTA and CTAs for an unfolding of at most mcap rows
__host__ __forceinline__ int rows_per_cta(long long mcap, int nsm, int rmax) {
    long long r = (mcap + nsm - 1) / nsm;
    if (r < RPB_MIN) r = RPB_MIN;
    if (r > rmax) r = rmax;
    return (int)r;
}
__host__ __forceinline__ int ctas(long long mcap, int rpb) {
    long long b = (mcap + rpb - 1) / rpb;
    return (int)(b < 1 ? 1 : b);
}
// the rows a CTA takes: the actual ones spread evenly over the launched CTAs
// (the launch is sized from a bound on m)
__device__ __forceinline__ int rows_taken(int m, int nb) {
    const int r = (m + nb - 1) / nb;
    return r < RPB_MIN ? RPB_MIN : r;
}
__device__ __forceinline__ bool shape_ok(int m, int c, int cb, const GQ& g) {
    return c <= cb && c >= 1 && m >= c && (long long)m <= (long long)g.rpb * g.nb;
}

// Partial Gram matrix of the CTA's rows on the FP64 tensor cores
// (mma.m8n8k4, four rows a step; a block's fragment serves as A and as B):
// four sets of tiles x two halves of the rows for the eight warps, so a
// fragment loaded once serves every tile of its set.
template <int CB>
__host__ __device__ constexpr bool in_set(int s, int I, int J) {
    constexpr int HB = CB / 16, QB = CB / 32;  // half and quarter of the column blocks
    return I <= J && (s == 0 ? J < HB : s == 1 ? I >= HB : s == 2 ? (I < QB && J >= HB) : (I >= QB && I < HB && J >= HB));
}
template <int CB>
__host__ __device__ constexpr int set_max() {
    int mx = 0;
    for (int s = 0; s < 4; s++) {
        int n = 0;
        for (int J = 0; J < CB / 8; J++)
            for (int I = 0; I <= J; I++) n += in_set<CB>(s, I, J) ? 1 : 0;
        mx = n > mx ? n : mx;
    }
    return mx;
}
template <int CB, int S>
__device__ __forceinline__ void gram_set(const double* Xs, int ks0, int ks1, int nbc, double (&d0)[set_max<CB>()],
                                         double (&d1)[set_max<CB>()]) {
    constexpr int XP = Cfg<CB>::XP, NB = CB / 8;
    const int lane = threadIdx.x & 31, li = lane >> 2, lk = lane & 3;
    for (int ks = ks0; ks < ks1; ks++) {
        const double* xr = Xs + (4 * ks + lk) * XP + li;
        double f[NB];
#pragma unroll
        for (int b = 0; b < NB; b++) f[b] = b < nbc ? xr[8 * b] : 0.0;  // the blocks no tile of the set uses fold away
        int t = 0;
#pragma unroll
        for (int J = 0; J < NB; J++) {
#pragma unroll
            for (int I = 0; I <= J; I++) {
                if (in_set<CB>(S, I, J)) {
                    if (J < nbc) mma884(d0[t], d1[t], f[I], f[J]);
                    t++;
                }
            }
        }
    }
}
// store (how 0), or add what is stored at `red` and write to P (how 1)
template <int CB, int S>
__device__ __forceinline__ void gram_out(int nbc, const double (&d0)[set_max<CB>()], const double (&d1)[set_max<CB>()],
                                         double* red, double* P, bool first) {
    constexpr int NB = CB / 8;
    const int lane = threadIdx.x & 31, li = lane >> 2, lk = lane & 3;
    const int o = tix(li, 2 * lk);
    int t = 0;
#pragma unroll
    for (int J = 0; J < NB; J++) {
#pragma unroll
        for (int I = 0; I <= J; I++) {
            if (in_set<CB>(S, I, J)) {
                if (J < nbc) {
                    const int at = tnum(I, J) * 64 + o;
                    if (first) {
                        *(double2*)(red + at) = make_double2(d0[t], d1[t]);
                    } else {
                        const double2 v = *(const double2*)(red + at);
                        *(double2*)(P + at) = make_double2(d0[t] + v.x, d1[t] + v.y);
                    }
                }
                t++;
            }
        }
    }
}
// Xs: h rows, zero rows up to a multiple of 4; red: UP doubles of shared memory
template <int CB>
__device__ __forceinline__ void gram_fp64(const double* Xs, int h, int nbc, double* red, double* P) {
    const int warp = threadIdx.x >> 5, set = warp & 3, half = warp >> 2;
    const int nks = (h + 3) >> 2, mid = (nks + 1) >> 1;
    const int ks0 = half ? mid : 0, ks1 = half ? nks : mid;
    double d0[set_max<CB>()], d1[set_max<CB>()];
#pragma unroll
    for (int t = 0; t < set_max<CB>(); t++) d0[t] = d1[t] = 0.0;
    switch (set) {
        case 0: gram_set<CB, 0>(Xs, ks0, ks1, nbc, d0, d1); break;
        case 1: gram_set<CB, 1>(Xs, ks0, ks1, nbc, d0, d1); break;
        case 2: gram_set<CB, 2>(Xs, ks0, ks1, nbc, d0, d1); break;
        default: gram_set<CB, 3>(Xs, ks0, ks1, nbc, d0, d1);
    }
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
        if ((half == 1) == (pass == 0)) {
            switch (set) {
                case 0: gram_out<CB, 0>(nbc, d0, d1, red, P, pass == 0); break;
                case 1: gram_out<CB, 1>(nbc, d0, d1, red, P, pass == 0); break;
                case 2: gram_out<CB, 2>(nbc, d0, d1, red, P, pass == 0); break;
                default: gram_out<CB, 3>(nbc, d0, d1, red, P, pass == 0);
            }
        }
        if (pass == 0) __syncthreads();
    }
}

// The rows of one stage of the factorisation of core k's unfolding (mode);
// g.nb CTAs with room for g.rpb rows each.  OZ: the Gram partials by the
// Ozaki split on the fifth-generation tensor cores (ptt_ozaki.cuh) instead
// of FP64 mma (64 columns only).
// Bound by latency: at 111 rows x 64 columns the loads, the solve's chain of
// 8 blocks and 126 products a warp.  One stage takes 10 us at 16384 x 64 (23 at
// 9696 x 95) beside 23 (38) of k_gq_decide; a factorisation is two stages there
// and took 187 us with 3.6 stages whose last CTA summed and factored alone
// (2600 with the Householder tree at 95 columns).
template <int CB, bool OZ>
__global__ void __launch_bounds__(NT, 1) k_gq_rows(const DevDesc* D, int k, int mode, Plan pl, GQ g, int stage) {
    PTT_PDL_ENTRY();
    using C = Cfg<CB>;
    constexpr int XP = C::XP;
    extern __shared__ __align__(128) double gsm[];
    double* Xs = gsm;                       // RPB_MAX x XP rows
    double* sF = Xs + C::RPB_MAX * XP;      // factor tiles, inverse pivots; then the Gram halves
    __shared__ int s_go, s_fin;
    const State* st = (const State*)g.rec;
    const View A = make_view(D, k, mode, false);
    const int m = A.m, c = A.c;
    const int tid = threadIdx.x, b = (int)blockIdx.x;
    if (!shape_ok(m, c, CB, g)) return;  // uniform; k_gq_decide records the fallback
    const int rt = rows_taken(m, g.nb), r0 = b * rt;
    if (r0 >= m) return;
    if (stage > 0) {
        if (tid == 0) {
            const int s = ldcg(&st->state);
            s_fin = s == FINISH;
            s_go = s == RUN || (s == FINISH && ldcg(&st->fin) == stage);
        }
        __syncthreads();
        if (!s_go) return;
    }
    const int h = (m - r0) < rt ? (m - r0) : rt;
    const int h16 = (h + 15) & ~15, nbc = (c + 7) >> 3;
    // Qbuf: where the Q_s rows live
    View Qv;
    if (mode == LEFT) {
        Qv.p = D->alt[k];
        Qv.rs = 1;
        Qv.cs = m;
    } else {
        Qv.p = g.qscr;
        Qv.rs = c;
        Qv.cs = 1;
    }
    const View& src = (stage <= 1) ? A : Qv;
    const unsigned xs0 = (unsigned)__cvta_generic_to_shared(Xs);
    if (stage > 0) {  // the factor of the previous stage, 16 bytes at a time (UP and CB are even)
        const unsigned f0 = (unsigned)__cvta_generic_to_shared(sF);
        const double* F = g.rec + C::O_FAC;
        const int used = nbc * (nbc + 1) * 32;
        for (int e = 2 * tid; e < used; e += 2 * NT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(f0 + 8u * e), "l"(F + e) : "memory");
        for (int e = 2 * tid; e < CB; e += 2 * NT)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(f0 + 8u * (C::UP + e)), "l"(F + C::UP + e)
                         : "memory");
    }
    // this CTA's rows, every element in flight by cp.async; zeros beyond c up
    // to the block and beyond h up to 16 rows
    if (src.rs == 1) {
        // column-major: a warp copies 4 rows x 8 columns at a time (32
        // contiguous bytes of each column)
        const int nrb = (h + 3) / 4, ncb = (c + 7) / 8;
        const int lr = (tid & 31) & 3, lc = (tid & 31) >> 2;
        for (int t = tid >> 5; t < nrb * ncb; t += NT / 32) {
            const int cb = t / nrb, rb = t - cb * nrb;
            const int row = rb * 4 + lr, col = cb * 8 + lc;
            if (row < h && col < c) {
                const double* gp = src.p + (long long)(r0 + row) + (long long)col * src.cs;
                const unsigned sa = xs0 + 8u * (unsigned)(row * XP + col);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gp) : "memory");
            }
        }
    } else if ((c & 1) == 0) {  // row-major rows of an even c: pairs (every row starts on 16 bytes)
        const int c2 = c >> 1, dq = NT / c2, dr = NT - dq * c2;
        int row = tid / c2, col = tid - row * c2;
        const double* base = src.p + (long long)r0 * c;
        for (; row < h;) {
            const unsigned sa = xs0 + 8u * (unsigned)(row * XP + 2 * col);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(base + (long long)row * c + 2 * col)
                         : "memory");
            row += dq;
            col += dr;
            if (col >= c2) {
                col -= c2;
                row++;
            }
        }
    } else {
        const int dq = NT / c, dr = NT - dq * c;
        int row = tid / c, col = tid - row * c;
        const double* base = src.p + (long long)r0 * c;
        for (; row < h;) {
            const unsigned sa = xs0 + 8u * (unsigned)(row * XP + col);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(base + (long long)row * c + col)
                         : "memory");
            row += dq;
            col += dr;
            if (col >= c) {
                col -= c;
                row++;
            }
        }
    }
    const int cz = (OZ ? CB : 8 * nbc) - c;
    for (int e = tid; e < h * cz; e += NT) Xs[(e / cz) * XP + c + e % cz] = 0.0;
    for (int e = tid; e < (h16 - h) * XP; e += NT) Xs[h * XP + e] = 0.0;
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    if (stage > 0) {
        tile_solve<XP, NT / 32>(Xs, h, sF, sF + C::UP, nbc);
        __syncthreads();
        if (Qv.rs == 1) {  // column-major, in the load's 4 x 8 warp tiles
            const int nrb = (h + 3) / 4, ncb = (c + 7) / 8;
            const int lr = (tid & 31) & 3, lc = (tid & 31) >> 2;
            for (int t = tid >> 5; t < nrb * ncb; t += NT / 32) {
                const int cb = t / nrb, rb = t - cb * nrb;
                const int row = rb * 4 + lr, col = cb * 8 + lc;
                if (row < h && col < c) Qv.p[(long long)(r0 + row) + (long long)col * Qv.cs] = Xs[row * XP + col];
            }
        } else {
            const int dq = NT / c, dr = NT - dq * c;
            int row = tid / c, col = tid - row * c;
            for (; row < h;) {
                Qv.p[(long long)(r0 + row) * c + col] = Xs[row * XP + col];
                row += dq;
                col += dr;
                if (col >= c) {
                    col -= c;
                    row++;
                }
            }
        }
        if (s_fin) return;  // the last factor is applied: Q is final
    }
    double* P = g.part + (long long)b * C::UP;
    if constexpr (OZ)
        oz::gram_partial<NT>(Xs, XP, h, c, (unsigned char*)sF, Xs, P);
    else
        gram_fp64<CB>(Xs, h, nbc, sF, P);
}

// Cholesky factor of H in the tiles at sG (nbc column blocks), in place, by
// the whole CTA: per block column, every panel thread factors the 8 x 8
// diagonal block in its own registers (the same 8 steps in every thread, so
// nothing is broadcast), solves one column of the block row against it, and
// after a barrier all warps update the trailing tiles on the FP64 tensor
// cores.  A pivot not above PIV is set to PIV and its row to zero; a column
// outside `alive` (one byte of bits per block) gets a zero row.  rinv[j] =
// 1 / R[j][j] (zero where not alive).
// 64 columns: 8 x ~1.7k cycles where one warp with lane = column took ~45k
// (540 a column: a shuffle, the reciprocal square root and a shared-memory
// broadcast on the chain of every column).
template <int CB>
__device__ void chol_tiles(double* sG, int nbc, int c, const unsigned char* alive, double* rinv) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, li = lane >> 2, lk = lane & 3;
    for (int J = 0; J < nbc; J++) {
        double r[8][8], inv[8];
        const int col = 8 * J + 8 + tid;  // this thread's column of the block row
        if (tid < CB) {
            const unsigned weak = chol8(sG + tnum(J, J) * 64, alive[J], r, inv);
            if (col < 8 * nbc) solve8(sG + tnum(J, col >> 3) * 64, col & 7, r, inv, weak);
        }
        __syncthreads();
        if (tid == 0) {  // the diagonal block, read by every panel thread until the barrier
            double* G = sG + tnum(J, J) * 64;
#pragma unroll
            for (int i = 0; i < 8; i++) {
#pragma unroll
                for (int j = 0; j < 8; j++) G[tix(i, j)] = j >= i ? r[i][j] : 0.0;
                rinv[8 * J + i] = inv[i];
            }
        }
        const int n = nbc - J - 1;
        for (int t = warp; t < n * (n + 1) / 2; t += NT / 32) {
            int I, K;
            tile_of(t, &I, &K);
            trail8(sG, J, I + J + 1, K + J + 1, li, lk);
        }
        __syncthreads();
    }
}

// Sum of the partial Gram matrices (CTA t: tile t) and, in the last CTA to
// finish, the decision of the stage.  What counts is that CTA's chain after the
// sums: the norms and tests, the c-step Cholesky (a warp's 8 x 8 tile, then all
// warps' solves and updates, one barrier each) and the accumulated R.
template <int CB>
__global__ void __launch_bounds__(NT, 1) k_gq_decide(const DevDesc* D, int k, int mode, Plan pl, GQ g, double* ws,
                                                     int stage, long long* qstat) {
    PTT_PDL_ENTRY();
    using C = Cfg<CB>;
    extern __shared__ __align__(128) double gsm[];
    __shared__ int s_state, s_ticket, s_flags, s_nd;
    __shared__ double s_red[NT];
    __shared__ double s_d[CB], s_di[CB], s_an[CB], s_rinv[CB];
    __shared__ unsigned long long s_tm[CB];
    __shared__ unsigned char s_alive[CB / 8];
    State* st = (State*)g.rec;
    const View A = make_view(D, k, mode, false);
    const int m = A.m, c = A.c;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, li = lane >> 2, lk = lane & 3;
    if (stage == 0) {
        if (!shape_ok(m, c, CB, g)) {  // uniform
            if (blockIdx.x == 0 && tid == 0) {
                st->state = FALLBACK;
                st->nst = 0;
                st->m = m;
                st->c = c;
                if (qstat) atomicAdd((unsigned long long*)(qstat + 1), 1ull);
            }
            return;
        }
        if (pl.work && blockIdx.x == 0 && tid == 0) atomicAdd(pl.work, 16.0 * (double)m * (double)c);
    } else {
        if (tid == 0) s_state = ldcg(&st->state);
        __syncthreads();
        if (s_state != RUN) return;
    }
    const int nbc = (c + 7) >> 3, nt = nbc * (nbc + 1) / 2;
    if ((int)blockIdx.x >= nt) return;
    {
        // tile blockIdx.x: four quarters of the partials, each in CTA order
        // (eight loads in flight), the quarters in order
        const int rt = rows_taken(m, g.nb), np = (m + rt - 1) / rt;
        const int q = tid >> 6, p0 = np * q / 4, p1 = np * (q + 1) / 4;
        const double* P = g.part + (long long)blockIdx.x * 64 + (tid & 63);
        double a = 0.0;
        int p = p0;
        for (; p + 8 <= p1; p += 8) {
            double v[8];
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = ldcg(P + (long long)(p + t) * C::UP);
#pragma unroll
            for (int t = 0; t < 8; t++) a += v[t];
        }
        for (; p < p1; p++) a += ldcg(P + (long long)p * C::UP);
        s_red[tid] = a;
        __syncthreads();
        if (tid < 64)
            g.rec[C::O_G + blockIdx.x * 64 + tid] = ((s_red[tid] + s_red[64 + tid]) + s_red[128 + tid]) + s_red[192 + tid];
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_ticket = atomicAdd(g.cnt, 1);
    __syncthreads();
    if (s_ticket != nt - 1) return;
    // ---- the deciding CTA ----------------------------------------------------
    if (tid == 0) {
        *g.cnt = 0;
        s_flags = 0;
        s_nd = 0;
    }
    __threadfence();
    double* sG = gsm;            // Gram matrix, then the factor
    double* sT = gsm + C::UP;    // accumulated R of the factors applied so far
    {
        const unsigned g0 = (unsigned)__cvta_generic_to_shared(sG);
        const double* G = g.rec + C::O_G;
        const double* T = g.rec + C::O_T;
        for (int e = 2 * tid; e < nt * 64; e += 2 * NT) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(g0 + 8u * e), "l"(G + e) : "memory");
            if (stage > 0)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(g0 + 8u * (C::UP + e)), "l"(T + e)
                             : "memory");
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    __syncthreads();
    if (tid < CB) {
        const int j = tid;
        const double gjj = j < c ? sG[tnum(j >> 3, j >> 3) * 64 + tix(j & 7, j & 7)] : 0.0;
        const double dj = gjj > 0.0 ? sqrt(gjj) : 0.0;
        bool on = gjj > 0.0;
        if (stage > 0) {
            on = on && dj * ldcg(g.rec + C::O_TM + j) > DROP * sqrt((double)c);
            s_an[j] = ldcg(g.rec + C::O_AN + j);
        } else {
            s_an[j] = on ? 1.0 / dj : 0.0;
            g.rec[C::O_AN + j] = s_an[j];
        }
        double p2, ip2;
        pow2_above(dj, &p2, &ip2);
        s_d[j] = on ? p2 : 0.0;
        s_di[j] = on ? ip2 : 0.0;
        s_tm[j] = 0ull;
        if (j < c && !(gjj >= 0.0 && gjj < LARGE)) atomicOr(&s_flags, 1);      // NaN, Inf or near overflow
        if (j < c && gjj != 0.0 && gjj < SMALL) atomicOr(&s_flags, 1);
        if (gjj > 0.0 && !on) atomicOr(&s_flags, 2);  // dropped by this stage: q_j is still in Q_s
        const unsigned bits = __ballot_sync(0xffffffffu, on);
        if ((lane & 7) == 0) s_alive[j >> 3] = (unsigned char)((bits >> lane) & 0xffu);
        if (lane == 0 && j < c) atomicAdd(&s_nd, __popc(bits));
    }
    __syncthreads();
    const int nlive = s_nd;
    double emax = 0.0;
    for (int t = warp; t < nt; t += NT / 32) {
        int I, J;
        tile_of(t, &I, &J);
        const double2 v = *(const double2*)(sG + t * 64 + tix(li, 2 * lk));
        const int i = 8 * I + li, j = 8 * J + 2 * lk;
        const bool oi = (s_alive[I] >> li) & 1, o0 = (s_alive[J] >> (2 * lk)) & 1, o1 = (s_alive[J] >> (2 * lk + 1)) & 1;
        const double e0 = (oi && o0) ? fabs(v.x - (i == j ? 1.0 : 0.0)) : 0.0;
        const double e1 = (oi && o1) ? fabs(v.y - (i == j + 1 ? 1.0 : 0.0)) : 0.0;
        if (!(v.x - v.x == 0.0) || !(v.y - v.y == 0.0)) atomicOr(&s_flags, 1);
        emax = fmax(emax, fmax(e0, e1));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    if (lane == 0) s_red[warp] = emax;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < NT / 32; w++) emax = fmax(emax, s_red[w]);
    int nst = (stage == 0) ? 0 : ldcg(&st->nst);
    int dec;
    if ((s_flags & 1) || nlive == 0) {
        dec = FALLBACK;
    } else if (stage >= 1 && emax <= TAU && !(s_flags & 2)) {
        dec = DONE;
    } else if (stage == MAXST - 1) {
        dec = FALLBACK;  // no launch left to apply another factor
    } else if (stage >= 1 && emax <= FIRST) {
        dec = emax <= FIRST_DONE ? FINISH : RUN;
        for (int t = warp; t < nt; t += NT / 32) {
            int I, J;
            tile_of(t, &I, &J);
            double2* pv = (double2*)(sG + t * 64 + tix(li, 2 * lk));
            const double2 v = *pv;
            const int i = 8 * I + li, j = 8 * J + 2 * lk;
            const bool oi = (s_alive[I] >> li) & 1, o0 = (s_alive[J] >> (2 * lk)) & 1,
                       o1 = (s_alive[J] >> (2 * lk + 1)) & 1;
            double2 w;
            w.x = !(oi && o0) || j < i ? 0.0 : (i == j ? 1.0 + 0.5 * (v.x - 1.0) : v.x);
            w.y = !(oi && o1) || j + 1 < i ? 0.0 : (i == j + 1 ? 1.0 + 0.5 * (v.y - 1.0) : v.y);
            *pv = w;
            if (i == j) s_rinv[i] = w.x != 0.0 ? 1.0 / w.x : 0.0;
            if (i == j + 1) s_rinv[i] = w.y != 0.0 ? 1.0 / w.y : 0.0;
        }
    } else {
        dec = RUN;
        for (int t = warp; t < nt; t += NT / 32) {  // H = D^-1 G D^-1, zero for the dropped columns
            int I, J;
            tile_of(t, &I, &J);
            double2* pv = (double2*)(sG + t * 64 + tix(li, 2 * lk));
            const double di = s_di[8 * I + li];
            pv->x = pv->x * di * s_di[8 * J + 2 * lk];
            pv->y = pv->y * di * s_di[8 * J + 2 * lk + 1];
        }
        __syncthreads();
        chol_tiles<CB>(sG, nbc, c, s_alive, s_rinv);
        for (int t = warp; t < nt; t += NT / 32) {  // R = chol(H) D
            int I, J;
            tile_of(t, &I, &J);
            double2* pv = (double2*)(sG + t * 64 + tix(li, 2 * lk));
            pv->x *= s_d[8 * J + 2 * lk];
            pv->y *= s_d[8 * J + 2 * lk + 1];
        }
        if (tid < 8 * nbc) s_rinv[tid] *= s_di[tid];
    }
    __syncthreads();
    if (dec == RUN || dec == FINISH) {
        // the factor for the next launch, and the accumulated R = F T in tiles
        double* F = g.rec + C::O_FAC;
        for (int e = tid; e < nt * 32; e += NT) ((double2*)F)[e] = ((const double2*)sG)[e];
        if (tid < CB) F[C::UP + tid] = tid < 8 * nbc ? s_rinv[tid] : 0.0;
        double* T = g.rec + C::O_T;
        double* Rs = ws + pl.o_Rn;  // root slot (row-major CT x CT)
        for (int t = warp; t < nt; t += NT / 32) {
            int I, J;
            tile_of(t, &I, &J);
            double2 v;
            if (stage == 0) {
                v = *(const double2*)(sG + t * 64 + tix(li, 2 * lk));
            } else {
                v = tile_product(sG, sT, I, J, li, lk);
            }
            *(double2*)(T + t * 64 + tix(li, 2 * lk)) = v;
            const int i = 8 * I + li, j = 8 * J + 2 * lk;
            if (dec == FINISH) {
                Rs[(long long)i * CB + j] = j >= i ? v.x : 0.0;
                Rs[(long long)i * CB + j + 1] = j + 1 >= i ? v.y : 0.0;
            }
            const double w = fmax(fabs(v.x) * s_an[j], fabs(v.y) * s_an[j + 1]);
            atomicMax(&s_tm[i], (unsigned long long)__double_as_longlong(w));
        }
        __syncthreads();
        if (tid < CB) g.rec[C::O_TM + tid] = __longlong_as_double((long long)s_tm[tid]);
        nst++;
    } else if (dec == DONE) {
        double* Rs = ws + pl.o_Rn;
        for (int t = warp; t < nt; t += NT / 32) {
            int I, J;
            tile_of(t, &I, &J);
            const double2 v = *(const double2*)(sT + t * 64 + tix(li, 2 * lk));
            const int i = 8 * I + li, j = 8 * J + 2 * lk;
            const bool oi = (s_alive[I] >> li) & 1;  // a zero q_j needs no row of R
            Rs[(long long)i * CB + j] = oi && j >= i ? v.x : 0.0;
            Rs[(long long)i * CB + j + 1] = oi && j + 1 >= i ? v.y : 0.0;
        }
    }
    if (finished(dec)) {
        double* Rs = ws + pl.o_Rn;  // zeros: the tiles below the diagonal and the columns beyond the blocks
        for (int e = tid; e < CB * CB; e += NT) {
            const int i = e / CB, j = e - (e / CB) * CB;
            if ((j >> 3) < (i >> 3) || j >= 8 * nbc || i >= 8 * nbc) Rs[e] = 0.0;
        }
        if (tid == 0) {
            Info* info = pl.info;
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
    if (tid == 0) {
        if (dec == FALLBACK && qstat) atomicAdd((unsigned long long*)(qstat + 1), 1ull);
        st->fin = stage + 1;
        st->nst = nst;
        st->ndrop = c - nlive;
        st->m = m;
        st->c = c;
        __threadfence();
        st->state = dec;
    }
}

// alt[k] = Q V_r (m x rank, row-major) for a RIGHT_T bond this path finished:
// Q rows in g.qscr (row-major, pitch c), V_r at the root B slot (row-major CT
// x KC).  With a ticket the last block swaps the core, also for a bond the
// Householder tree wrote.
template <int CB>
__global__ void __launch_bounds__(256, Slab<CB>::PER_SM) k_gq_write(DevDesc* D, int k, Plan pl, GQ g, double* ws,
                                                                    Fin fin) {
    PTT_PDL_ENTRY();
    extern __shared__ __align__(128) double gsm[];
    const Info* info = pl.info;
    if (finished(ldcg((const int*)g.rec)) && info->status == 0) {
        const int m = info->m, c = info->c, rank = info->rank;
        slab_mul<CB>(ws + pl.o_Bn, 1, pl.KC, rank, c, g.qscr, 1, c, m, D->alt[k], 1, rank, blockIdx.x, gridDim.x, gsm);
    }
    fin_last_block(D, fin, info);
}

// G = A^T A of a column-major m x c matrix (c <= 64, leading dimension lda),
// the Gram matrix of an unfolding on its own (ptt_gram): CTA b forms the
// partial of rows [b RPB_MAX, (b + 1) RPB_MAX) -- on the FP64 tensor cores,
// or by the Ozaki split on tcgen05 when OZ -- the last-arriving CTA of each
// group of GROUP sums the group's partials in CTA order, the last-arriving
// group sums the groups in order and writes G (c x c, column-major, both
// triangles).  Deterministic; no CTA waits for another.
constexpr size_t SM_GRAM = sizeof(double) * ((size_t)Cfg<64>::RPB_MAX * Cfg<64>::XP + Cfg<64>::UP);
template <bool OZ>
__global__ void __launch_bounds__(NT, 1) k_gram(const double* A, long long m, int c, long long lda, double* part,
                                                double* gpart, int* cnt, double* G) {
    using C = Cfg<64>;
    constexpr int UP = C::UP, XP = C::XP, RPB_MAX = C::RPB_MAX;
    extern __shared__ __align__(128) double gsm[];
    double* Xs = gsm;
    __shared__ int s_ticket;
    const int tid = threadIdx.x, b = (int)blockIdx.x, nb = (int)gridDim.x;
    const long long r0 = (long long)b * RPB_MAX;
    const int h = (m - r0) < RPB_MAX ? (int)(m - r0) : RPB_MAX;
    for (int e = tid; e < RPB_MAX * XP; e += NT) Xs[e] = 0.0;
    __syncthreads();
    for (int e = tid; e < h * c; e += NT) {
        const int col = e / h, row = e - col * h;
        Xs[row * XP + col] = A[r0 + row + (long long)col * lda];
    }
    __syncthreads();
    if constexpr (OZ)
        oz::gram_partial<NT>(Xs, XP, h, c, (unsigned char*)(Xs + RPB_MAX * XP), Xs, part + (long long)b * UP);
    else
        gram_fp64<64>(Xs, h, 8, Xs + RPB_MAX * XP, part + (long long)b * UP);
    const int ngroups = (nb + GROUP - 1) / GROUP, grp = b / GROUP;
    const int gsize = (nb - grp * GROUP) < GROUP ? (nb - grp * GROUP) : GROUP;
    __threadfence();
    __syncthreads();
    if (tid == 0) s_ticket = atomicAdd(&cnt[grp], 1);
    __syncthreads();
    if (s_ticket != gsize - 1) return;
    if (tid == 0) cnt[grp] = 0;
    __threadfence();
    for (int u = tid; u < UP; u += NT) {
        double a = 0.0;
        for (int t = 0; t < gsize; t++) a += ldcg(part + (long long)(grp * GROUP + t) * UP + u);
        gpart[(long long)grp * UP + u] = a;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_ticket = atomicAdd(&cnt[ngroups], 1);
    __syncthreads();
    if (s_ticket != ngroups - 1) return;
    if (tid == 0) cnt[ngroups] = 0;
    __threadfence();
    for (int e = tid; e < UP; e += NT) {
        int ti, tj;
        tile_of(e >> 6, &ti, &tj);
        const int i = ti * 8 + ((e >> 3) & 7), j = tj * 8 + (e & 7);
        if (i < c && j < c && i <= j) {
            const int u = (e & ~63) + tix((e >> 3) & 7, e & 7);
            double a = 0.0;
            for (int t = 0; t < ngroups; t++) a += ldcg(gpart + (long long)t * UP + u);
            G[i + (long long)j * c] = a;
            G[j + (long long)i * c] = a;
        }
    }
}

}  // namespace gq
