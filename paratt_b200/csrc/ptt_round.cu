// TT rounding on the device, FP64: paratt_truncate (paratt.c:316-342) ->
// pattacTruncate (pattac.c:590-675) with ortho 'R':
//
//   left-to-right:  for i = 0..d-2   QR of the left unfolding of core i
//                   (pattacLOrthogonalization, pattac.c:244-294), R pushed into
//                   core i+1 (trapezoid_mult, utilities.c:233-308), Q kept.
//   right-to-left:  for i = d-1..1   LQ of the right unfolding (as QR of its
//                   transpose), SVD of L, tail-sum rank rule, core i <- V_r^T Q,
//                   core i-1 <- core i-1 * U_r S_r (pattacLTruncate,
//                   pattac.c:297-522).
//
// The grid normalisation of pattac.c:608-616/665-673 (divide every core by
// sqrt(n_k), multiply back afterwards) scales every bond's singular values by
// 1/sqrt(prod n_k); it is folded into the threshold instead of two passes
// over the cores: drop while sqrt(tail) < tol/sqrt(d-1) * sqrt(prod n_k).
//
// Every stage reads sizes from device memory (descriptor + Info record), so
// a rounding is a fixed launch sequence with no host synchronisation.
#include "ptt_tsqr.cuh"

#include <cooperative_groups.h>
#include <stdio.h>
#include <string.h>

#include <type_traits>

using namespace tsqr;

namespace {

__device__ __forceinline__ unsigned group_mask8(int tid) { return 0xFFu << ((tid & 31) & ~7); }

__device__ __forceinline__ double gsum8(double v, unsigned mask) {
    v += __shfl_xor_sync(mask, v, 4);
    v += __shfl_xor_sync(mask, v, 2);
    v += __shfl_xor_sync(mask, v, 1);
    return v;
}

#include "ptt_factor.cuh"

// ---------------------------------------------------------------------------
// Q application: out = Q * B, B = Bn[root] (q x k), k read from device.
// ---------------------------------------------------------------------------
template <int CT>
__device__ void replay_tsqrt(double* Rp, const double* Vs, const double* taus, int c, double* out, int col, int part) {
    constexpr int S = CT + 1;
    constexpr int NV = H / 8;
    const unsigned gm = 0xffffffffu;
    for (int j = c - 1; j >= 0; j--) {
        const double tau = taus[j];
        if (tau == 0.0) continue;
        double pr = 0.0;
#pragma unroll
        for (int v = 0; v < NV; v++) pr += Vs[(part + 8 * v) * S + j] * out[v];
        const double rj = Rp[j * KG + col];
        pr = gsum8(pr, gm);
        const double tw = tau * (rj + pr);
        if (part == 0) Rp[j * KG + col] = rj - tw;
#pragma unroll
        for (int v = 0; v < NV; v++) out[v] -= tw * Vs[(part + 8 * v) * S + j];
        __syncwarp();
    }
}

template <int CT>
__device__ void replay_geqrt(double* Rp, const double* Vb, const double* taus, int c, int col, int part) {
    constexpr int S = CT + 1;
    constexpr int NV = CT / 8;
    for (int j = c - 1; j >= 0; j--) {
        const double tau = taus[j];
        if (tau == 0.0) continue;
        double pr = 0.0;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const int t = part + 8 * v;
            if (t >= j) pr += (t == j ? 1.0 : Vb[t * S + j]) * Rp[t * KG + col];
        }
        pr = gsum8(pr, 0xffffffffu);
        const double tw = tau * pr;
#pragma unroll
        for (int v = 0; v < NV; v++) {
            const int t = part + 8 * v;
            if (t >= j) Rp[t * KG + col] -= tw * (t == j ? 1.0 : Vb[t * S + j]);
        }
        __syncwarp();
    }
}

// out = Q B for the Householder tree, a launch per range of its levels: block
// (p, y) takes node p of level l1 (the leaves are level log2 P) and 32 columns of
// B and walks down to it from its ancestor on level l0, replaying the reflectors
// of each node on its own copy of the node's rows in shared memory (the left
// child takes the triangle's rows, the right child the eliminated ones).  At a
// leaf it replays the leaf's reflectors too and writes Q B; above, it replays its
// own node and leaves both children's rows at their slots of Bn for the next
// launch.  B is V_r at the root slot (RIGHT_T) or the identity (LEFT).
//   Up to APPLY_LEAVES leaves one launch does it all: the chain is as deep as
// with a launch per level, and the upper nodes, replayed once per leaf below
// them, run on SMs that were idle.  Behind the grid Cholesky QR, which plans no
// more leaves than that, the launch is nearly always skipped and is all the tree
// costs (at 16384 x 64 seven launches of 1.0 us before, each 2 to 5 us of a
// lane's time in a batch: 12 trains of ranks to 96 took 64.1 ms, then 58.1).
//   With more leaves every SM is busy and the repeated replays cost time (1024
// modes of ranks 128, Householder only, 512 leaves: a rounding took 59 ms with a
// launch per level, 83 in one), so the launches after the first five levels
// take one level each.
// LEFT: out(row, col) at alt[row + m*col];  RIGHT_T: alt[row*k + col]
constexpr int APPLY_LEAVES = 32;
template <int CT>
__global__ void __launch_bounds__(NT) k_apply(const DevDesc* D, int kcore, int mode, Plan pl, double* ws,
                                              const int* kptr, int l0, int l1) {
    PTT_PDL_ENTRY();
    if (gq_finished(pl)) return;
    extern __shared__ double sm[];
    constexpr int S = CT + 1;
    constexpr int VR = CT > H ? CT : H;
    constexpr int NHC = (CT + H - 1) / H;  // chunks of a node
    double* Rp = sm;             // CT x KG
    double* Vs = Rp + CT * KG;   // VR x S
    const int p = blockIdx.x;
    const int kg0 = blockIdx.y * KG;
    const int kk = *kptr;
    if (pl.info->status || kg0 >= kk) return;
    const int tid = threadIdx.x, col = tid >> 3, part = tid & 7;
    const int m = pl.info->m, c = pl.info->c, q = pl.info->q;
    // the unfolding the factorisation recorded (m x c), not the descriptor's
    // ranks: in the truncation sweep this runs on the side stream while the
    // main stream has already published the bond's new rank
    View A;
    A.p = D->core[kcore];
    A.m = m;
    A.c = c;
    A.rs = (mode == LEFT) ? 1 : c;
    A.cs = (mode == LEFT) ? m : 1;
    double* outp = D->alt[kcore];
    const long long ors = (mode == LEFT) ? 1 : kk;
    const long long ocs = (mode == LEFT) ? m : 1;
    int r0, r1;  // rows of the leaf, or of the node's first leaf (the empty leaves come last)
    const int below = 31 - __clz(pl.P) - l1;
    leaf_range(m, pl.L, pl.P, p << below, &r0, &r1);
    const int rows = r1 - r0;
    if (rows <= 0) return;
    const int rb = rows < c ? rows : c;
    const int slot = (1 << l1) - 1 + p;
    double* Bn = ws + pl.o_Bn;  // CT x KC a slot
    const double* B = Bn + (long long)(((slot + 1) >> (l1 - l0)) - 1) * CT * pl.KC;
    for (int e = tid; e < CT * KG; e += NT) {
        const int a = e / KG, b = kg0 + e - a * KG;
        Rp[e] = mode == LEFT && l0 == 0 ? (a == b && a < q ? 1.0 : 0.0) : B[(long long)a * pl.KC + b];
    }
    for (int l = l1 - l0; l >= (below > 0 ? 0 : 1); l--) {
        const int node = ((slot + 1) >> l) - 1;                                // ancestor l levels up, or the node
        const bool right = l > 0 && ((((slot + 1) >> (l - 1)) - 1) & 1) == 0;  // its child on the path
        if (pl.pass[node] != 0) continue;  // the right child has no rows: nothing was eliminated
        const double* RR = ws + pl.o_Rn + (long long)(2 * node + 2) * CT * CT;
        double out[NHC][H / 8];
#pragma unroll
        for (int half = NHC - 1; half >= 0; half--) {
            const int h0 = half * H;
#pragma unroll
            for (int v = 0; v < H / 8; v++) out[half][v] = 0.0;
            if (h0 >= c) continue;
            __syncthreads();
            for (int e = tid; e < H * CT; e += NT) {
                const int t = e / CT, j = e - (e / CT) * CT;
                Vs[t * S + j] = (h0 + t < c) ? RR[(long long)(h0 + t) * CT + j] : 0.0;
            }
            __syncthreads();
            replay_tsqrt<CT>(Rp, Vs, ws + pl.o_tau_node + ((long long)node * pl.NH + half) * CT, c, out[half], col,
                             part);
        }
        __syncthreads();
        if (right) {
#pragma unroll
            for (int half = 0; half < NHC; half++)
#pragma unroll
                for (int v = 0; v < H / 8; v++) {
                    const int t = half * H + part + 8 * v;
                    if (t < CT) Rp[t * KG + col] = out[half][v];
                }
        } else if (l == 0) {
            double* Bcr = Bn + (long long)(2 * node + 2) * CT * pl.KC;
#pragma unroll
            for (int half = 0; half < NHC; half++)
#pragma unroll
                for (int v = 0; v < H / 8; v++) {
                    const int t = half * H + part + 8 * v;
                    if (t < CT) Bcr[(long long)t * pl.KC + kg0 + col] = out[half][v];
                }
        }
    }
    if (below > 0) {
        double* Bcl = Bn + (long long)(2 * slot + 1) * CT * pl.KC;
        __syncthreads();
        for (int e = tid; e < CT * KG; e += NT) Bcl[(long long)(e / KG) * pl.KC + kg0 + e % KG] = Rp[e];
        return;
    }
    const double* tau_leaf = ws + pl.o_tau_leaf + (long long)p * pl.KL * CT;
    const int ocol = kg0 + col;
    const bool colok = ocol < kk;
    const int nch = (rows - rb + H - 1) / H;
    for (int s = nch - 1; s >= 0; s--) {
        const int t0 = r0 + rb + s * H;
        const int h = (r1 - t0) < H ? (r1 - t0) : H;
        __syncthreads();
        for (int e = tid; e < H * CT; e += NT) {
            const int t = e / CT, l = e - (e / CT) * CT;
            Vs[t * S + l] = (t < h && l < c) ? A.p[(long long)(t0 + t) * A.rs + (long long)l * A.cs] : 0.0;
        }
        __syncthreads();
        double out[H / 8];
#pragma unroll
        for (int v = 0; v < H / 8; v++) out[v] = 0.0;
        replay_tsqrt<CT>(Rp, Vs, tau_leaf + (long long)(1 + s) * CT, c, out, col, part);
#pragma unroll
        for (int v = 0; v < H / 8; v++) {
            const int t = part + 8 * v;
            if (t < h && colok) outp[(long long)(t0 + t) * ors + (long long)ocol * ocs] = out[v];
        }
    }
    __syncthreads();
    for (int e = tid; e < CT * CT; e += NT) {
        const int t = e / CT, l = e - (e / CT) * CT;
        Vs[t * S + l] = (t < rb && l < c && t > l) ? A.p[(long long)(r0 + t) * A.rs + (long long)l * A.cs] : 0.0;
    }
    __syncthreads();
    replay_geqrt<CT>(Rp, Vs, tau_leaf, c, col, part);
    __syncthreads();
    for (int e = tid; e < CT * KG; e += NT) {
        const int t = e / KG, b = e - (e / KG) * KG;
        if (t < rb && kg0 + b < kk) outp[(long long)(r0 + t) * ors + (long long)(kg0 + b) * ocs] = Rp[e];
    }
}

#include "ptt_svd.cuh"

// Rebuild rows of V (q x q, V = product of the recorded rotations) and write
// V_r = V[:, order[0:rank]] into Bn[root].  One warp per row, PP pairs a lane.
// The chain of a row is what counts (a step reads two entries, multiplies and
// writes them: about 100 cycles, 500 steps at 64 columns), so everything else
// is off it: the rotations come from memory into registers RD steps ahead, the
// pair's columns (tabulated once for all sweeps) one step ahead.  With the
// table of each sweep staged in shared memory and both looked up inside the
// step it took 117 us at 64 columns, now 49.
template <int PP>
__device__ __forceinline__ void svd_replay_rows(double* vrow, const unsigned short* cols, int npair, int npr, int nrd,
                                                int sweeps, const double2* rot, long long per_sweep) {
    constexpr int RD = 8;
    const int lane = threadIdx.x & 31, total = sweeps * nrd;
    double2 r[RD][PP];
    const double2* next = rot + lane;  // rotations of the next step to request
    int nleft = nrd;                   // steps left in its sweep
    auto request = [&](double2 (&d)[PP]) {
#pragma unroll
        for (int u = 0; u < PP; u++) d[u] = lane + 32 * u < npr ? next[32 * u] : make_double2(1.0, 0.0);
        next += npair;
        if (--nleft == 0) {
            nleft = nrd;
            next += per_sweep - (long long)nrd * npair;
        }
    };
#pragma unroll
    for (int t = 0; t < RD; t++)
        if (t < total) request(r[t]);
    unsigned short pq[PP];
    int rd = 0;
    auto columns = [&]() {
#pragma unroll
        for (int u = 0; u < PP; u++) pq[u] = lane + 32 * u < npr ? cols[rd * npair + lane + 32 * u] : 0;
        rd = rd + 1 == nrd ? 0 : rd + 1;
    };
    columns();
    for (int t0 = 0; t0 < total; t0 += RD) {
#pragma unroll
        for (int u8 = 0; u8 < RD; u8++) {
            if (t0 + u8 >= total) break;  // uniform
            double2 w[PP];
            unsigned short c[PP];
#pragma unroll
            for (int u = 0; u < PP; u++) {
                w[u] = r[u8][u];
                c[u] = pq[u];
            }
#pragma unroll
            for (int u = 0; u < PP; u++)
                if (w[u].y != 0.0) {  // (cos, tan)
                    const int pc = c[u] & 255, qc = c[u] >> 8;
                    const double x = vrow[pc], y = vrow[qc];
                    vrow[pc] = w[u].x * fma(-w[u].y, y, x);
                    vrow[qc] = w[u].x * fma(w[u].y, x, y);
                }
            if (t0 + u8 + RD < total) request(r[u8]);
            columns();
            __syncwarp();
        }
    }
}

__device__ void svd_replay_body(const Plan& pl, double* ws, const Info* info, int bx) {
    extern __shared__ double sm[];
    const int CT = pl.CT, KC = pl.KC;
    const int SR = CT + 2;
    const int npair = (CT + 2) / 2;
    double* vrow = sm + (threadIdx.x >> 5) * SR;  // 8 rows
    unsigned short* cols = (unsigned short*)(sm + 8 * SR);  // (CT + 1) steps x npair
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int row = bx * 8 + warp;
    if (info->status) return;
    const int q = info->q, sweeps = info->sweeps, rank = info->rank, order = info->order;
    // pairs and steps of a sweep: two pairs for each of the G groups
    const int qa = info->qa, Gc = qa > 4 ? (qa + 3) >> 2 : 1;
    const int G = order == ORD_RING ? (Gc > 1 ? 1 << (32 - __clz(Gc - 1)) : 1) : Gc;
    const int npr = 2 * G, nrd = 4 * G - 1;
    const int* perm = (const int*)(ws + pl.o_sig + CT) + CT;
    // the columns of V of every (step, pair) slot; beyond qa (never rotated): CT
    for (int e = threadIdx.x; e < nrd * npr; e += blockDim.x) {
        const int rd = e / npr, i = e - (e / npr) * npr;
        int pc, qc;
        svd_pair(i, rd, G, order, &pc, &qc);
        cols[rd * npair + i] = (unsigned short)((pc < qa ? perm[pc] : CT) | (qc < qa ? perm[qc] : CT) << 8);
    }
    for (int j = lane; j < SR; j += 32) vrow[j] = (j == row) ? 1.0 : 0.0;
    __syncthreads();
    if (row < q && sweeps > 0) {
        const double2* rot = (const double2*)(ws + pl.o_rot);
        const long long per = (long long)(CT + 1) * npair;
        if (npr <= 32)
            svd_replay_rows<1>(vrow, cols, npair, npr, nrd, sweeps, rot, per);
        else
            svd_replay_rows<2>(vrow, cols, npair, npr, nrd, sweeps, rot, per);
    }
    __syncwarp();
    if (row >= CT) return;
    const int* ord = (const int*)(ws + pl.o_sig + CT);
    double* B = ws + pl.o_Bn + (long long)row * KC;
    for (int b = lane; b < KC; b += 32) B[b] = (row < q && b < rank) ? vrow[ord[b]] : 0.0;
}

__global__ void __launch_bounds__(256) k_svd_replay(Plan pl, double* ws) {
    PTT_PDL_ENTRY();
    svd_replay_body(pl, ws, pl.info, blockIdx.x);
}

// the same for bonds k0 .. k0 + gridDim.y - 1, bond k's records at ws + k * stride
__global__ void __launch_bounds__(256) k_svd_replay_b(Plan pl, double* ws, long long stride, int k0) {
    PTT_PDL_ENTRY();
    double* wsb = ws + (long long)(k0 + blockIdx.y) * stride;
    svd_replay_body(pl, wsb, (const Info*)(wsb + pl.o_info_d), blockIdx.x);
}

// ---------------------------------------------------------------------------
// A small matrix times a long one on the FP64 tensor cores: C(row, n) =
// sum_k S(row, k) B(k, n), S s x c with s, c <= CB (R, U_r S_r or V_r of a
// bond), n < N in the tens of thousands (a core's columns or rows).
//
// Memory is the bound at CB = 64 (16384 columns: 16 MB, 2.5 us, against 3.6 of
// DMMAs at their peak).  S is laid out once per CTA in fragment order (one
// conflict-free read per product); a warp takes 8 columns of B at a time,
// fragments straight from memory, all of a tile's loads in flight and the next
// tile's issued as the products use up this one's.  k runs in the order 8 b + 2 q
// + s (lane q of four, step s), so a group of four lanes reads 64 contiguous
// bytes whichever index of B is contiguous.  64 x 64 x 16 tiles staged through
// shared memory took 18.4 us (R x core), 14.7 (core x U_r S_r) and 12.1 (Q V_r)
// at 16384 x 64; now 11.2, 11.3 and 6.9.
// ---------------------------------------------------------------------------
template <int CB>
struct Slab {
    static constexpr int T = CB / 8;                                // tile rows of S, blocks of 8 of k
    static constexpr size_t SMEM = sizeof(double) * T * T * 64;
    static constexpr int PER_SM = CB <= 64 ? 2 : 1;                 // CTAs
};

template <int CB>
__device__ __forceinline__ void slab_mul(const double* S, int srs, int scs, int s, int c, const double* B, long long brs,
                                         long long bcs, long long N, double* C, long long crs, long long ccs, int blk,
                                         int nblk, double* Ss) {
    constexpr int T = Slab<CB>::T;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lr = lane >> 2, q = lane & 3;
    const int st = (s + 7) >> 3, kt = (c + 7) >> 3;
    double b[T][2];
    const double* bp = B + 2 * q * brs + lr * bcs;
    auto load = [&](long long n0, int kb) {
#pragma unroll
        for (int h = 0; h < 2; h++)
            b[kb][h] = (8 * kb + 2 * q + h < c && n0 + lr < N) ? bp[(8 * kb + h) * brs + n0 * bcs] : 0.0;
    };
    long long n0 = 8LL * (8 * blk + warp);
    const long long step = 64LL * nblk;
    if (n0 < N) {
#pragma unroll
        for (int kb = 0; kb < T; kb++) load(n0, kb);
    }
    for (int e = tid; e < 64 * st * kt; e += 256) {
        int row, k;
        if (scs == 1) {
            k = e % (8 * kt);
            row = e / (8 * kt);
        } else {
            row = e % (8 * st);
            k = e / (8 * st);
        }
        const double v = (row < s && k < c) ? S[(long long)row * srs + (long long)k * scs] : 0.0;
        Ss[((((k >> 3) * 2 + (k & 1)) * T + (row >> 3)) << 5) + ((row & 7) << 2) + ((k & 7) >> 1)] = v;
    }
    __syncthreads();
    for (; n0 < N; n0 += step) {
        double d[T][2];
#pragma unroll
        for (int r = 0; r < T; r++) d[r][0] = d[r][1] = 0.0;
        const bool more = n0 + step < N;
#pragma unroll
        for (int kb = 0; kb < T; kb++) {
            if (kb < kt) {
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < T; r++)
                        if (r < st) {
                            const double a = Ss[(((kb * 2 + h) * T + r) << 5) + lane];
                            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                                         : "+d"(d[r][0]), "+d"(d[r][1])
                                         : "d"(a), "d"(b[kb][h]));
                        }
                if (more) load(n0 + step, kb);
            }
        }
        const long long col = n0 + 2 * q;
#pragma unroll
        for (int r = 0; r < T; r++) {
            const int row = 8 * r + lr;
            if (row < s && col < N) C[row * crs + col * ccs] = d[r][0];
            if (row < s && col + 1 < N) C[row * crs + (col + 1) * ccs] = d[r][1];
        }
    }
}

// f(std::integral_constant<int, CB>) with the smallest CB that holds the bond's
// ranks: a small bond of a wide train then leaves shared memory and registers to
// the kernels beside it (the lanes of a batch: 12 trains of ranks to 96 in 55.6
// ms, 58.0 with the 128-wide kernels for every bond).
template <typename F>
static int slab_dispatch(int bound, F f) {
    if (bound <= 32) return f(std::integral_constant<int, 32>{});
    if (bound <= 64) return f(std::integral_constant<int, 64>{});
    if (bound <= 96) return f(std::integral_constant<int, 96>{});
    return f(std::integral_constant<int, 128>{});
}

// CTAs of such a launch for at most ncap columns
template <int CB>
static int slab_ctas(long long ncap, int nsm) {
    const long long t = (ncap + 63) / 64, w = (long long)Slab<CB>::PER_SM * nsm;
    return (int)(t < 1 ? 1 : (t < w ? t : w));
}

// The bookkeeping that follows a bond's contraction: publish the bond's new
// rank (D->r[kq] = *val; kq < 0: none) and swap core[ka], and core[kb] unless
// kb < 0, with the buffers just written.  With a ticket (a zero-initialised
// counter) the last block of the contraction does it, so it needs no launch of
// its own; without one the caller launches k_bond_finalize.
struct Fin {
    int* ticket;
    int kq, ka;
    const int* val;
    int kb = -1;
};

__device__ __forceinline__ void fin_last_block(DevDesc* D, const Fin& f, const Info* info) {
    if (!f.ticket) return;
    __shared__ int s_last;
    __syncthreads();
    __threadfence();  // this block's output is visible before its ticket
    if (threadIdx.x == 0) s_last = atomicAdd(f.ticket, 1) == (int)(gridDim.x * gridDim.y) - 1;
    __syncthreads();
    if (s_last && threadIdx.x == 0) {
        *f.ticket = 0;
        __threadfence();
        if (info->status == 0) {
            if (f.kq >= 0) D->r[f.kq] = *f.val;
            double* t = D->core[f.ka];
            D->core[f.ka] = D->alt[f.ka];
            D->alt[f.ka] = t;
            if (f.kb >= 0) {
                t = D->core[f.kb];
                D->core[f.kb] = D->alt[f.kb];
                D->alt[f.kb] = t;
            }
        }
    }
}

// core[i+1] <- R * core[i+1]   (R = root factor, q x c, row-major CT)
template <int CB>
__global__ void __launch_bounds__(256, Slab<CB>::PER_SM) k_gemm_rx(DevDesc* D, int i1, Plan pl, double* ws, Fin fin) {
    PTT_PDL_ENTRY();
    extern __shared__ double sm[];
    const int q = pl.info->q, c = pl.info->c;
    const long long N = (long long)D->n[i1] * D->r[i1 + 1];
    if (pl.info->status == 0)
        slab_mul<CB>(ws + pl.o_Rn, pl.CT, 1, q, c, D->core[i1], 1, c, N, D->alt[i1], 1, q, blockIdx.x, gridDim.x, sm);
    fin_last_block(D, fin, pl.info);
}

// core[i-1] <- core[i-1] * US   (US = c x rank, column-major ld CT), as its transpose US^T core^T
template <int CB>
__global__ void __launch_bounds__(256, Slab<CB>::PER_SM) k_gemm_xm(DevDesc* D, int im1, Plan pl, double* ws, Fin fin) {
    PTT_PDL_ENTRY();
    extern __shared__ double sm[];
    const int c = pl.info->c, rank = pl.info->rank;
    const long long M = (long long)D->r[im1] * D->n[im1];
    if (pl.info->status == 0)
        slab_mul<CB>(ws + pl.o_US, pl.CT, 1, rank, c, D->core[im1], M, 1, M, D->alt[im1], M, 1, blockIdx.x, gridDim.x,
                     sm);
    fin_last_block(D, fin, pl.info);
}

// The same two contractions for a train whose ranks stay <= 8 NT <= 32, with
// the rank update and the swap (kq, core i).  Latency bounds them: 2560 x 10
// columns are 0.4 us of DMMAs and of memory, a launch 0.8 us, the pointer chase
// (record, descriptor, data) 0.35 us a step and the ticket 0.7.  So the record
// and the descriptor are read together, every warp takes 8 columns (rows) with
// both operands' fragments straight from memory -- all its loads in flight at
// once, no shared memory, no barrier before the ticket -- and only the tiles
// that exist are multiplied.  A
// launch of a 40-dimensional step (n = 256, ranks to 16) in its chain: 5.3 us
// with 64 x 64 tiles, 2.6 here; 5120 x 20 columns 7.1 and 3.8.
struct WGemm {
    int status, c, q, rank, nk, r0, r1;
    double *core, *alt;
};
__device__ __forceinline__ WGemm wgemm_sizes(const DevDesc* D, int i, const Info* info) {
    WGemm g;
    g.status = info->status;
    g.c = info->c;
    g.q = info->q;
    g.rank = info->rank;
    g.nk = D->n[i];
    g.r0 = D->r[i];
    g.r1 = D->r[i + 1];
    g.core = D->core[i];
    g.alt = D->alt[i];
    return g;
}
__device__ __forceinline__ void wgemm_finish(DevDesc* D, int* ticket, int kq, int i, const WGemm& g, int val) {
    __threadfence();  // this block's output is visible before its ticket
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(ticket, 1) == (int)gridDim.x - 1) {
        *ticket = 0;
        if (g.status == 0) {
            D->r[kq] = val;
            D->core[i] = g.alt;
            D->alt[i] = g.core;
        }
    }
}

// core i <- R core i (R = root factor, q x c, row-major CT), r_i <- q
template <int NT8>
__global__ void __launch_bounds__(256) k_wgemm_rx(DevDesc* D, int i, Plan pl, const double* ws, int* ticket) {
    PTT_PDL_ENTRY();
    const WGemm g = wgemm_sizes(D, i, pl.info);
    const int lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    const int N = g.nk * g.r1, q = g.q, c = g.c;
    const double* R = ws + pl.o_Rn;
    const int t0 = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (g.status == 0 && 8 * t0 < N) {
        double a[NT8][2 * NT8], b[2 * NT8];
        auto load_b = [&](int t) {
#pragma unroll
            for (int k4 = 0; k4 < 2 * NT8; k4++) {
                const int kk = 4 * k4 + lk, col = 8 * t + lr;
                b[k4] = (kk < c && col < N) ? g.core[kk + (long long)c * col] : 0.0;
            }
        };
        load_b(t0);
#pragma unroll
        for (int r = 0; r < NT8; r++)
#pragma unroll
            for (int k4 = 0; k4 < 2 * NT8; k4++) {
                const int row = 8 * r + lr, kk = 4 * k4 + lk;
                a[r][k4] = (row < q && kk < c) ? R[row * pl.CT + kk] : 0.0;
            }
        for (int t = t0; 8 * t < N; t += 8 * gridDim.x) {
            if (t != t0) load_b(t);
#pragma unroll
            for (int r = 0; r < NT8; r++) {
                if (8 * r >= q) continue;
                double d0 = 0.0, d1 = 0.0;
#pragma unroll
                for (int k4 = 0; k4 < 2 * NT8; k4++)
                    if (4 * k4 < c)
                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                                     : "+d"(d0), "+d"(d1)
                                     : "d"(a[r][k4]), "d"(b[k4]));
                const int row = 8 * r + lr, col = 8 * t + 2 * lk;
                if (row < q && col < N) g.alt[row + (long long)q * col] = d0;
                if (row < q && col + 1 < N) g.alt[row + (long long)q * (col + 1)] = d1;
            }
        }
    }
    wgemm_finish(D, ticket, i, i, g, q);
}

// core i <- core i US (US = c x rank, column-major, leading dimension CT), r_{i+1} <- rank
template <int NT8>
__global__ void __launch_bounds__(256) k_wgemm_xm(DevDesc* D, int i, Plan pl, const double* ws, int* ticket) {
    PTT_PDL_ENTRY();
    const WGemm g = wgemm_sizes(D, i, pl.info);
    const int lane = threadIdx.x & 31, lr = lane >> 2, lk = lane & 3;
    const int M = g.r0 * g.nk, c = g.c, rank = g.rank;
    const double* US = ws + pl.o_US;
    const int t0 = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (g.status == 0 && 8 * t0 < M) {
        double a[2 * NT8], b[NT8][2 * NT8];
        auto load_a = [&](int t) {
#pragma unroll
            for (int k4 = 0; k4 < 2 * NT8; k4++) {
                const int row = 8 * t + lr, kk = 4 * k4 + lk;
                a[k4] = (row < M && kk < c) ? g.core[row + (long long)M * kk] : 0.0;
            }
        };
        load_a(t0);
#pragma unroll
        for (int v = 0; v < NT8; v++)
#pragma unroll
            for (int k4 = 0; k4 < 2 * NT8; k4++) {
                const int col = 8 * v + lr, kk = 4 * k4 + lk;
                b[v][k4] = (col < rank && kk < c) ? US[kk + pl.CT * col] : 0.0;
            }
        for (int t = t0; 8 * t < M; t += 8 * gridDim.x) {
            if (t != t0) load_a(t);
#pragma unroll
            for (int v = 0; v < NT8; v++) {
                if (8 * v >= rank) continue;
                double d0 = 0.0, d1 = 0.0;
#pragma unroll
                for (int k4 = 0; k4 < 2 * NT8; k4++)
                    if (4 * k4 < c)
                        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                                     : "+d"(d0), "+d"(d1)
                                     : "d"(a[k4]), "d"(b[v][k4]));
                const int row = 8 * t + lr, col = 8 * v + 2 * lk;
                if (row < M && col < rank) g.alt[row + (long long)M * col] = d0;
                if (row < M && col + 1 < rank) g.alt[row + (long long)M * (col + 1)] = d1;
            }
        }
    }
    wgemm_finish(D, ticket, i + 1, i, g, rank);
}

#include "ptt_ozaki.cuh"

// k_gemm_rx of the block-level path with the product as an Ozaki
// split-precision product on the fifth-generation tensor cores
// (oz::gemm_tiles): R (q x c, row-major, leading dimension CT) times core
// i1 (c x N, column-major) into alt[i1] (q x N); CTA y takes the 64-column
// tiles y, y + gridDim.y, ...
__global__ void __launch_bounds__(256, 1) k_gemm_rx_oz(DevDesc* D, int i1, Plan pl, double* ws) {
    PTT_PDL_ENTRY();
    extern __shared__ __align__(128) unsigned char osm[];
    if (pl.info->status != 0) return;
    const int q = pl.info->q, c = pl.info->c;
    const int N = D->n[i1] * D->r[i1 + 1];
    if (q > oz::KG || c > oz::KG || 64 * (int)blockIdx.y >= N) return;  // uniform
    oz::gemm_tiles<256>(ws + pl.o_Rn, pl.CT, 1, D->core[i1], 1, c, D->alt[i1], q, q, N, c, osm, false);
}

// k_gemm_xm of the block-level path as an Ozaki product: core[i-1] (M x c,
// column-major) times U_r S_r (c x rank, column-major, leading dimension CT)
// into alt[i-1], formed as its transpose (U_r S_r)^T core^T so that the
// 64-wide tiles run along the M rows
__global__ void __launch_bounds__(256, 1) k_gemm_xm_oz(DevDesc* D, int im1, Plan pl, double* ws) {
    PTT_PDL_ENTRY();
    extern __shared__ __align__(128) unsigned char osm[];
    if (pl.info->status != 0) return;
    const int c = pl.info->c, rank = pl.info->rank;
    const int M = D->r[im1] * D->n[im1];
    if (rank > oz::KG || c > oz::KG || 64 * (int)blockIdx.y >= M) return;  // uniform
    oz::gemm_tiles<256>(ws + pl.o_US, pl.CT, 1, D->core[im1], M, 1, D->alt[im1], M, rank, M, c, osm, true);
}

// publish a bond's new rank (kq < 0: none) and swap the rewritten cores (kb < 0: one)
__global__ void k_bond_finalize(DevDesc* D, int kq, int ka, int kb, const int* val, const Info* info) {
    PTT_PDL_ENTRY();
    if (threadIdx.x == 0 && info->status == 0) {
        if (kq >= 0) D->r[kq] = *val;
        double* t = D->core[ka];
        D->core[ka] = D->alt[ka];
        D->alt[ka] = t;
        if (kb >= 0) {
            t = D->core[kb];
            D->core[kb] = D->alt[kb];
            D->alt[kb] = t;
        }
    }
}

#include "ptt_wtsqr.cuh"
#include "ptt_gramstage.cuh"
#include "ptt_cholqr.cuh"
#include "ptt_gridqr.cuh"

// ---------------------------------------------------------------------------
// host planning
// ---------------------------------------------------------------------------
static int next_pow2(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

struct Layout {
    Plan pl;
    long long bytes;
};

// pmax bounds the leaves (and so the tree levels): the Householder TSQR behind
// the grid Cholesky QR only runs for a bond that falls back, so there it takes
// few, long leaves and its skipped launches stay small.
static void plan_bond(int CT, long long mcap, int KC, Plan* pl, int pmax = 512) {
    int L = 2 * CT;
    if (L < 128) L = 128;
    L = (L + H - 1) / H * H;
    long long P = (mcap + L - 1) / L;
    while (P > pmax) {
        L *= 2;
        P = (mcap + L - 1) / L;
    }
    pl->CT = CT;
    pl->L = L;
    pl->P = next_pow2((int)(P < 1 ? 1 : P));
    pl->KL = 1 + (2 * L - 1 + H - 1) / H;
    pl->NH = (CT + H - 1) / H;
    pl->KC = KC;
    pl->gqstate = nullptr;
}

static long long carve(Plan* pl, int PMAX, int LMAXKL) {
    const int CT = pl->CT, KC = pl->KC;
    long long o = 0;
    auto take = [&](long long n) {
        long long r = o;
        o += (n + 31) / 32 * 32;
        return r;
    };
    pl->o_tau_leaf = take((long long)PMAX * LMAXKL * CT);
    pl->o_Rn = take((long long)(2 * PMAX - 1) * CT * CT);
    pl->o_tau_node = take((long long)PMAX * pl->NH * CT);
    pl->o_Bn = take((long long)(PMAX > APPLY_LEAVES ? 2 * PMAX - 1 : 1) * CT * KC);
    pl->o_US = take((long long)CT * CT);
    pl->o_rot = take((long long)MAXSW * (CT + 1) * ((CT + 2) / 2) * 2);
    pl->o_sig = take(2LL * CT + 64);
    pl->o_info_d = take(64);
    pl->o_nodes = take((long long)(3 * PMAX + 64) / 2 + 1);  // qn [2P-1] and pass [P] as ints
    pl->total = o;
    return o;
}

template <int CT>
static size_t factor_smem() {
    return sizeof(double) * ((size_t)CT * CT + 2 * (size_t)FCfg<CT>::VB + CT);
}
template <int CT>
static size_t apply_smem() {
    const int VR = CT > H ? CT : H;
    return sizeof(double) * ((size_t)CT * KG + (size_t)VR * (CT + 1));
}
// 8 rows of V and the columns (two bytes) of a sweep's (CT + 1) x (CT + 2) / 2 pairs
template <int CT>
static size_t replay_smem() {
    return sizeof(double) * 8 * (size_t)(CT + 2) + 2 * (size_t)(CT + 1) * ((CT + 2) / 2);
}

template <int CT>
static int set_attrs() {
    static std::atomic<unsigned long long> done{0};
    unsigned long long bit;
    if (ptt_device_done(done, &bit)) return PTT_OK;
    PTT_CUDA(cudaFuncSetAttribute(k_tsqr_factor<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)factor_smem<CT>()));
    PTT_CUDA(cudaFuncSetAttribute(k_apply<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)apply_smem<CT>()));
    PTT_CUDA(cudaFuncSetAttribute(k_svd_jacobi<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)svd_smem<64>()));
    if constexpr (CT == 128) {
        PTT_CUDA(cudaFuncSetAttribute(k_svd_jacobi<96>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)svd_smem<96>()));
        PTT_CUDA(cudaFuncSetAttribute(k_svd_jacobi<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)svd_smem<128>()));
    }
    PTT_CUDA(cudaFuncSetAttribute(k_svd_replay, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)replay_smem<128>()));
    if constexpr (CT == 128) {
        for (int cb : {96, 128}) {
            const int err = slab_dispatch(cb, [&](auto b) -> int {
                constexpr int CB = decltype(b)::value;
                for (auto f : {(const void*)k_gemm_rx<CB>, (const void*)k_gemm_xm<CB>, (const void*)gq::k_gq_write<CB>})
                    PTT_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Slab<CB>::SMEM));
                return PTT_OK;
            });
            if (err) return err;
        }
    }
    if constexpr (CT >= 64) {
        PTT_CUDA(cudaFuncSetAttribute(gq::k_gq_rows<CT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)gq::Cfg<CT>::SM_ROWS));
        PTT_CUDA(cudaFuncSetAttribute(gq::k_gq_decide<CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)gq::Cfg<CT>::SM_DEC));
    }
    if constexpr (CT == 64)
        PTT_CUDA(cudaFuncSetAttribute(gq::k_gq_rows<64, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)gq::SM_ROWS_OZ));
    PTT_CUDA(cudaFuncSetAttribute(k_gemm_rx_oz, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)oz::SMEM_GEMM));
    PTT_CUDA(cudaFuncSetAttribute(k_gemm_xm_oz, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)oz::SMEM_GEMM));
    done.fetch_or(bit);
    return PTT_OK;
}

// SVD of a bond's factor (at most rk rows and columns): the kernel for the
// smallest row bound that holds it, so that a small bond pays for no idle
// lanes and rows.
static int launch_svd(ptt_ctx* c, int rk, const Plan& pl, double* ws, double delta, int mr, int bond) {
    auto go = [&](auto kernel, int nt, size_t smem) -> int {
        PTT_CUDA(ptt_launch(c, kernel, dim3(1), dim3(nt), smem, pl, ws, delta, mr, bond, c->d_status));
        return PTT_OK;
    };
    if (rk <= 16) return go(k_svd_jacobi<16>, svd_nt<16>(), svd_smem<16>());
    if (rk <= 32) return go(k_svd_jacobi<32>, svd_nt<32>(), svd_smem<32>());
    if (rk <= 48) return go(k_svd_jacobi<48>, svd_nt<48>(), svd_smem<48>());
    if (rk <= 64) return go(k_svd_jacobi<64>, svd_nt<64>(), svd_smem<64>());
    if (rk <= 96) return go(k_svd_jacobi<96>, svd_nt<96>(), svd_smem<96>());
    return go(k_svd_jacobi<128>, svd_nt<128>(), svd_smem<128>());
}

// Factor the unfolding (mode) of core k; R lands at the root slot.  With the
// grid Cholesky QR (g != null) its stage launches go first and the Householder
// TSQR only factors a bond they did not finish.
template <int CT>
static int launch_factor(ptt_ctx* c, ptt_tt* x, int k, int mode, Plan& pl, double* ws, gq::GQ* g, long long mcap) {
    ptt_time_begin(c, PTT_TIME_TSQR);
    if constexpr (CT >= 64) {
        if (g) {
            using C = gq::Cfg<CT>;
            g->rpb = gq::rows_per_cta(mcap, c->nsm, C::RPB_MAX);
            g->nb = gq::ctas(mcap, g->rpb);
            pl.gqstate = (const int*)g->rec;
            for (int s = 0; s < gq::MAXST; s++) {
                if (CT == 64 && c->ozaki)
                    PTT_CUDA(ptt_launch(c, gq::k_gq_rows<64, true>, dim3(g->nb), dim3(gq::NT), gq::SM_ROWS_OZ,
                                        (const DevDesc*)x->dd, k, mode, pl, *g, s));
                else
                    PTT_CUDA(ptt_launch(c, gq::k_gq_rows<CT, false>, dim3(g->nb), dim3(gq::NT), C::SM_ROWS,
                                        (const DevDesc*)x->dd, k, mode, pl, *g, s));
                PTT_LAUNCHED(c);
                PTT_CUDA(ptt_launch(c, gq::k_gq_decide<CT>, dim3(C::NTI), dim3(gq::NT), C::SM_DEC,
                                    (const DevDesc*)x->dd, k, mode, pl, *g, ws, s, c->d_qrstat));
                PTT_LAUNCHED(c);
            }
        }
    }
    PTT_CUDA(ptt_launch(c, k_tsqr_factor<CT>, dim3(pl.P), dim3(NT), factor_smem<CT>(), (const DevDesc*)x->dd, k, mode,
                        pl, ws, c->d_status));
    ptt_time_end(c, PTT_TIME_TSQR);
    PTT_LAUNCHED(c);
    return PTT_OK;
}

// out = Q B (k_apply); B and out have k columns, read from *kptr, at most kcap.
template <int CT>
static int launch_apply(ptt_ctx* c, ptt_tt* x, int k, int mode, Plan& pl, double* ws, const int* kptr, int kcap) {
    const int depth = 31 - __builtin_clz((unsigned)pl.P);
    for (int l0 = 0, l1; l0 <= depth; l0 = l1 + 1) {
        l1 = pl.P <= APPLY_LEAVES ? depth : (l0 == 0 ? 4 : l0);
        PTT_CUDA(ptt_launch(c, k_apply<CT>, dim3(1 << l1, (kcap + KG - 1) / KG), dim3(NT), apply_smem<CT>(),
                            (const DevDesc*)x->dd, k, mode, pl, ws, kptr, l0, l1));
        PTT_LAUNCHED(c);
    }
    return PTT_OK;
}

// phases: 1 = left-to-right orthogonalisation, 2 = right-to-left truncation,
// 4 = QR of the single core `only` (left unfolding; core <- Q, r_{only+1} <- q).
// rk[k]: upper bound of rank k for the whole call (the capacity, or the
// actual ranks when they were read back; ranks only shrink while rounding).
// At CT = 64 and 128 every factorisation first runs the grid Cholesky QR
// (ptt_gridqr.cuh) unless the context is set to Householder only.
template <int CT>
static int round_impl(ptt_tt* x, const int* rk, double delta, const int* maxr, int phases, int only) {
    ptt_ctx* c = x->ctx;
    const int d = x->d;
    int rc = set_attrs<CT>();
    if (rc) return rc;
    bool use_gq = CT >= 64 && !c->no_cholqr;
    const int KC = (CT + KG - 1) / KG * KG;
    using GC = gq::Cfg<CT >= 64 ? CT : 64>;
    const long long gq_rec = (GC::REC + 31) / 32 * 32;
    int PMAX, KLMAX, NBMAX, pmax;
    long long MQMAX, o_gq, SLOT;
    Plan base;
    for (;;) {
        // plan: largest leaf count over all bonds decides the workspace
        PMAX = KLMAX = NBMAX = 1;
        MQMAX = 1;
        pmax = use_gq ? APPLY_LEAVES : 512;
        for (int i = 0; i < d; i++) {
            Plan t;
            long long ml = (long long)rk[i] * x->n[i], mr = (long long)x->n[i] * rk[i + 1];
            plan_bond(CT, ml > mr ? ml : mr, KC, &t, pmax);
            if (t.P > PMAX) PMAX = t.P;
            if (t.KL > KLMAX) KLMAX = t.KL;
            for (long long mm : {ml, mr}) {
                const int nb = gq::ctas(mm, gq::rows_per_cta(mm, c->nsm, GC::RPB_MAX));
                NBMAX = nb > NBMAX ? nb : NBMAX;
            }
            MQMAX = mr > MQMAX ? mr : MQMAX;
        }
        plan_bond(CT, 1, KC, &base);
        base.NH = (CT + H - 1) / H;
        o_gq = (carve(&base, PMAX, KLMAX) + 31) / 32 * 32;
        // two slots of the whole region (bond parity): the truncation sweep runs
        // the tail of bond i (V replay, Q V_r, swap of core i) on the side stream
        // while bond i - 1 is factored in the other slot
        SLOT = o_gq;
        // grid Cholesky QR: record, partial Gram matrices, Q rows of RIGHT_T bonds
        if (use_gq) SLOT += (gq_rec + (long long)NBMAX * GC::UP + MQMAX * CT + 31) / 32 * 32;
        if (!(rc = ptt_ws_reserve(c, (size_t)(2 * SLOT) * sizeof(double) + 256))) break;
        if (!use_gq) return rc;
        // the grid's share grows with rows x columns, the Householder tree's
        // hardly: where the first does not fit the GPU beside the train, the
        // tree alone factors the bonds
        cudaGetLastError();
        ptt_set_error(PTT_OK, "");
        use_gq = false;
    }
    const size_t cnt_tree = (size_t)PMAX * 4 + 64;
    if ((rc = ptt_counters_reserve(c, cnt_tree + 3))) return rc;
    int* const tick_main = c->d_counters + cnt_tree + 1;  // Fin tickets: the contractions of the main stream,
    int* const tick_tail = c->d_counters + cnt_tree + 2;  // and the tails' (one stream each)
    double* const ws0 = (double*)c->ws;
    // ints live after the doubles: qn [2P-1], pass [P], Info
    // Tree counters live alone in ctx->d_counters (zero between launches,
    // reset by the combining block); node ranks and pass flags in ws.
    double* wss[2] = {ws0, ws0 + SLOT};
    gq::GQ gqs[2] = {};
    for (int sl = 0; sl < 2 && use_gq; sl++) {
        gqs[sl].rec = wss[sl] + o_gq;
        gqs[sl].part = gqs[sl].rec + gq_rec;
        gqs[sl].qscr = gqs[sl].part + (long long)NBMAX * GC::UP;
        gqs[sl].cnt = c->d_counters + cnt_tree;  // main stream only
    }
    double* ws = ws0;
    Info* info = (Info*)(ws0 + base.o_info_d);
    gq::GQ* g = use_gq ? &gqs[0] : nullptr;

    auto mkplan = [&](long long mcap, int sl = 0) {
        Plan pl = base;
        Plan t;
        plan_bond(CT, mcap, KC, &t, pmax);
        int* ints = (int*)(wss[sl] + base.o_nodes);
        pl.L = t.L;
        pl.P = t.P;
        pl.KL = KLMAX;
        pl.cnt = c->d_counters;
        pl.qn = ints;
        pl.pass = ints + 2 * PMAX;
        pl.info = (Info*)(wss[sl] + base.o_info_d);
        pl.stats = c->d_stats;
        pl.work = (c->tkind == PTT_TIME_TSQR) ? c->d_work + PTT_TIME_TSQR : nullptr;
        return pl;
    };
    const DevDesc* dd = x->dd;

    if (phases & 4) {
        const int i = only;
        const long long mcap = (long long)rk[i] * x->n[i];
        Plan pl = mkplan(mcap);
        if ((rc = launch_factor<CT>(c, x, i, LEFT, pl, ws, g, mcap))) return rc;
        if ((rc = launch_apply<CT>(c, x, i, LEFT, pl, ws, &info->q, CT))) return rc;
        PTT_CUDA(ptt_launch(c, k_bond_finalize, dim3(1), dim3(32), 0, x->dd, i + 1, i, -1, (const int*)&info->q,
                            (const Info*)info));
        PTT_LAUNCHED(c);
        return PTT_OK;
    }
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    PTT_CUDA(cudaStreamIsCapturing(c->stream, &cap));
    const bool ovl = cap == cudaStreamCaptureStatusNone && !c->capturing && !c->lane;
    // The rank update and swaps ride in the contraction's last block where
    // launches are plain (a batch's lanes, a capture): one launch less a bond
    // is 2 to 5 us there.  With programmatic launches a separate
    // k_bond_finalize costs 1.2 us, the tickets of 256 blocks 1.7.
    int* const tmain = ovl ? nullptr : tick_main;
    int* const ttail = ovl ? nullptr : tick_tail;
    auto finalize = [&](int kq, int ka, int kb, const int* val, const Info* inf) -> int {
        PTT_CUDA(ptt_launch(c, k_bond_finalize, dim3(1), dim3(32), 0, x->dd, kq, ka, kb, val, inf));
        PTT_LAUNCHED(c);
        return PTT_OK;
    };
    // left-to-right orthogonalisation
    for (int i = 0; i < d - 1 && (phases & 1); i++) {
        const long long mcap = (long long)rk[i] * x->n[i];
        Plan pl = mkplan(mcap);
        if ((rc = launch_factor<CT>(c, x, i, LEFT, pl, ws, g, mcap))) return rc;
        if ((rc = launch_apply<CT>(c, x, i, LEFT, pl, ws, &info->q, CT))) return rc;
        const long long ncap = (long long)x->n[i + 1] * rk[i + 2];
        const int gy = (int)((ncap + 63) / 64 > 4096 ? 4096 : (ncap + 63) / 64);
        // then the rank q and the swap of both rewritten cores
        if (c->ozaki && CT <= oz::KG) {  // one wave, R split once per CTA
            PTT_CUDA(ptt_launch(c, k_gemm_rx_oz, dim3(1, gy < c->nsm ? gy : c->nsm), dim3(256), oz::SMEM_GEMM,
                                x->dd, i + 1, pl, ws));
            PTT_LAUNCHED(c);
            if ((rc = finalize(i + 1, i, i + 1, &info->q, info))) return rc;
        } else {
            rc = slab_dispatch(rk[i + 1], [&](auto b) -> int {
                constexpr int CB = decltype(b)::value;
                PTT_CUDA(ptt_launch(c, k_gemm_rx<CB>, dim3(slab_ctas<CB>(ncap, c->nsm)), dim3(256), Slab<CB>::SMEM,
                                    x->dd, i + 1, pl, ws, Fin{tmain, i + 1, i + 1, &info->q, i}));
                return PTT_OK;
            });
            if (rc) return rc;
            PTT_LAUNCHED(c);
            if (!tmain && (rc = finalize(i + 1, i, i + 1, &info->q, info))) return rc;
        }
    }
    // right-to-left truncation.  The tail of bond i (V replay, Q V_r into
    // core i, swap of core i) is not needed by bond i - 1, which only reads
    // core i - 1 and the new rank r_i: it runs on the side stream from the
    // bond's slot (bond parity) while the main stream carries on; the main
    // stream waits for a slot's previous tail before reusing it, and for both
    // at the end.  Inside a caller's stream capture, and on the worker
    // contexts of a batch (which overlap whole roundings already: measured
    // 1.22 s against 0.98 s for 64 trains with the side stream), the sweep
    // stays serial.
    bool pending[2] = {false, false};
    for (int i = d - 1; i >= 1 && (phases & 2); i--) {
        const int sl = ovl ? (i & 1) : 0;
        if (pending[sl]) {
            PTT_CUDA(cudaStreamWaitEvent(c->stream, c->ev_tail[sl], 0));
            pending[sl] = false;
        }
        ws = wss[sl];
        info = (Info*)(ws + base.o_info_d);
        g = use_gq ? &gqs[sl] : nullptr;
        const long long mcap = (long long)x->n[i] * rk[i + 1];
        Plan pl = mkplan(mcap, sl);
        if ((rc = launch_factor<CT>(c, x, i, RIGHT_T, pl, ws, g, mcap))) return rc;
        const int mr = maxr ? maxr[i] : rk[i];
        ptt_time_begin(c, PTT_TIME_SVD);
        if ((rc = launch_svd(c, rk[i], pl, ws, delta, mr, i))) return rc;
        ptt_time_end(c, PTT_TIME_SVD);
        PTT_LAUNCHED(c);
        // the tail: V_r, then Q V_r (Householder tree or grid Cholesky QR) into alt[i], the swap of core i
        auto tail = [&]() -> int {
            PTT_CUDA(ptt_launch(c, k_svd_replay, dim3((CT + 7) / 8), dim3(256), replay_smem<CT>(), pl, ws));
            PTT_LAUNCHED(c);
            int r2 = launch_apply<CT>(c, x, i, RIGHT_T, pl, ws, &info->rank, CT);
            if (r2) return r2;
            if (g) {  // Q V_r for a bond the grid Cholesky QR finished
                r2 = slab_dispatch(rk[i], [&](auto b) -> int {
                    constexpr int CB = decltype(b)::value;
                    PTT_CUDA(ptt_launch(c, gq::k_gq_write<CB>, dim3(slab_ctas<CB>(mcap, c->nsm)), dim3(256),
                                        Slab<CB>::SMEM, x->dd, i, pl, *g, ws, Fin{ttail, -1, i, &info->rank}));
                    return PTT_OK;
                });
                if (r2) return r2;
                PTT_LAUNCHED(c);
                if (ttail) return PTT_OK;
            }
            return finalize(-1, i, -1, &info->rank, info);
        };
        if (ovl) {
            PTT_CUDA(cudaEventRecord(c->ev_svd[sl], c->stream));
            PTT_CUDA(cudaStreamWaitEvent(c->side, c->ev_svd[sl], 0));
            // the launch helpers issue on c->stream: point it at the side
            // stream; plain launches there (full stream order after the
            // event wait, no programmatic early start)
            cudaStream_t mainst = c->stream;
            const int pdl = c->no_pdl;
            c->stream = c->side;
            c->no_pdl = 1;
            rc = tail();
            if (!rc) {
                const cudaError_t e = cudaEventRecord(c->ev_tail[sl], c->side);
                rc = e == cudaSuccess ? PTT_OK : ptt_set_error(PTT_ERR_CUDA, "CUDA: %s", cudaGetErrorString(e));
            }
            c->stream = mainst;
            c->no_pdl = pdl;
            if (rc) return rc;
            pending[sl] = true;
        } else if ((rc = tail())) {
            return rc;
        }
        // core i - 1 times U_r S_r, then the new rank r_i and the swap of core i - 1
        const long long mcap2 = (long long)rk[i - 1] * x->n[i - 1];
        const int gx = (int)((mcap2 + 63) / 64 > 4096 ? 4096 : (mcap2 + 63) / 64);
        if (c->ozaki && CT <= oz::KG) {  // one wave, U_r S_r split once per CTA
            PTT_CUDA(ptt_launch(c, k_gemm_xm_oz, dim3(1, gx < c->nsm ? gx : c->nsm), dim3(256), oz::SMEM_GEMM, x->dd,
                                i - 1, pl, ws));
            PTT_LAUNCHED(c);
            if ((rc = finalize(i, i - 1, -1, &info->rank, info))) return rc;
        } else {
            rc = slab_dispatch(rk[i], [&](auto b) -> int {
                constexpr int CB = decltype(b)::value;
                PTT_CUDA(ptt_launch(c, k_gemm_xm<CB>, dim3(slab_ctas<CB>(mcap2, c->nsm)), dim3(256), Slab<CB>::SMEM,
                                    x->dd, i - 1, pl, ws, Fin{tmain, i, i - 1, &info->rank}));
                return PTT_OK;
            });
            if (rc) return rc;
            PTT_LAUNCHED(c);
            if (!tmain && (rc = finalize(i, i - 1, -1, &info->rank, info))) return rc;
        }
    }
    for (int sl = 0; sl < 2; sl++)
        if (pending[sl]) PTT_CUDA(cudaStreamWaitEvent(c->stream, c->ev_tail[sl], 0));
    return PTT_OK;
}


// Rounding of a train whose ranks stay <= 32 on the warp-level TSQR.
// Per bond only the factorisation, the small product that moves R (or U S)
// into the neighbour core and the rank update run in sequence; Q (and V_r Q)
// is formed for all bonds of a sweep in one launch after the sweep, and the
// SVD rotations are replayed for all bonds in one launch.
// Every bond k has its own record region (ws + k * stride) so the deferred
// launches find each bond's reflectors.  Same phases as round_impl.
static bool wt_fits(const ptt_tt* x, const int* rk) {
    for (int i = 0; i < x->d; i++) {
        const long long ml = (long long)rk[i] * x->n[i], mr = (long long)x->n[i] * rk[i + 1];
        const long long mx = ml > mr ? ml : mr;
        if (mx > 32LL * wt::PMAX) return false;
    }
    return true;
}

static int g_cq_csmax[64];  // per device: cluster size it can schedule

// rows bucket of the autotuner's table: <= 512, 1024, ..., > 8192
static int cq_bucket(int mp) {
    int b = 0, lim = 512;
    while (b < 5 && mp > lim) {
        b++;
        lim <<= 1;
    }
    return b;
}

static int round_impl_w(ptt_tt* x, const int* rk, double delta, const int* maxr, int phases, int only) {
    using namespace wt;
    ptt_ctx* c = x->ctx;
    const int d = x->d;
    int rc = set_attrs<32>();
    if (rc) return rc;
    static std::atomic<unsigned long long> wattr{0};
    unsigned long long wbit;
    int dev = 0;
    cudaGetDevice(&dev);
    dev &= 63;
    if (!ptt_device_done(wattr, &wbit)) {
        g_cq_csmax[dev] = cq::CSMAX;
        PTT_CUDA(cudaFuncSetAttribute(k_wfactor<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wfactor_smem()));
        PTT_CUDA(cudaFuncSetAttribute(k_wfactor<24>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wfactor_smem()));
        PTT_CUDA(cudaFuncSetAttribute(k_wfactor<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)wfactor_smem()));
        for (auto f : {(const void*)cq::k_cq_factor<16>, (const void*)cq::k_cq_factor<24>,
                       (const void*)cq::k_cq_factor<32>}) {
            PTT_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cq::SMEM_MAX));
            PTT_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        }
        // largest cluster the device can hold with one full-size CTA per SM
        cudaLaunchConfig_t qc = {};
        qc.gridDim = dim3(cq::CSMAX);
        qc.blockDim = dim3(cq::NT);
        qc.dynamicSmemBytes = cq::SMEM_MAX;
        cudaLaunchAttribute qa[1];
        qa[0].id = cudaLaunchAttributeClusterDimension;
        qa[0].val.clusterDim.x = cq::CSMAX;
        qa[0].val.clusterDim.y = 1;
        qa[0].val.clusterDim.z = 1;
        qc.attrs = qa;
        qc.numAttrs = 1;
        int ncl = 0;
        if (cudaOccupancyMaxActiveClusters(&ncl, (const void*)cq::k_cq_factor<32>, &qc) != cudaSuccess || ncl < 1) {
            cudaGetLastError();
            g_cq_csmax[dev] = 8;
        }
        wattr.fetch_or(wbit);
    }
    int Wl[PTT_MAX_DIM], Wr[PTT_MAX_DIM], Pcap = 1;
    for (int i = 0; i < d; i++) {
        const long long ml = (long long)rk[i] * x->n[i], mr = (long long)x->n[i] * rk[i + 1];
        Wl[i] = (int)((ml + 31) / 32);
        Wr[i] = (int)((mr + 31) / 32);
        const int pw = pow2_ge(Wl[i] > Wr[i] ? Wl[i] : Wr[i]);
        if (pw > Pcap) Pcap = pw;
    }
    Plan base;
    plan_bond(32, 1, 32, &base);
    base.NH = 1;
    long long o = carve(&base, 1, 1);
    WP wp;
    wp.o_R = o;
    o += (2LL * Pcap - 1) * SLOT;
    wp.o_tl = o;
    o += (long long)Pcap * 32;
    wp.o_tn = o;
    o += (long long)Pcap * 32;
    // Cholesky-QR record
    const int use_cq = c->no_cholqr ? 0 : 1;
    wp.o_cq = o;
    o += cq::REGION;
    wp.stride = (o + 31) / 32 * 32;
    wp.Pcap = Pcap;
    base.o_Rn = wp.o_R;  // root R = slot 0 (read by the SVD and the R product)
    if ((rc = ptt_ws_reserve(c, (size_t)wp.stride * d * sizeof(double) + 256))) return rc;
    if ((rc = ptt_counters_reserve(c, (size_t)Pcap * d + 64))) return rc;
    double* ws = (double*)c->ws;
    wp.cnt = c->d_counters;
    base.cnt = c->d_counters;
    int* fin_ticket = c->d_counters + (long long)Pcap * d;  // past the bonds' tree counters
    base.qn = nullptr;
    base.pass = nullptr;
    base.stats = c->d_stats;
    base.work = (c->tkind == PTT_TIME_TSQR) ? c->d_work + PTT_TIME_TSQR : nullptr;
    auto bond = [&](int i, double** wsb) {
        Plan pl = base;
        *wsb = ws + (long long)i * wp.stride;
        pl.info = (Info*)(*wsb + base.o_info_d);
        return pl;
    };
    // column bound of the unrolled Householder loops: the bond's rank bound
    auto cbound = [](int cols) { return cols <= 16 ? 16 : (cols <= 24 ? 24 : 32); };
    auto factor = [&](int i, int mode, int W, const Plan& pl, double* wsb) -> int {
        const int cb = cbound(mode == LEFT ? rk[i + 1] : rk[i]);
        const dim3 g((W + FPB - 1) / FPB), b(32 * FPB);
        const size_t sm = wfactor_smem();
        ptt_time_begin(c, PTT_TIME_TSQR);
        if (use_cq) {
            // Cholesky QR by one cluster; the TSQR below only runs for a bond
            // it did not finish
            const int mp = W * 32;  // bound on the unfolding's rows
            int cs = 1;
            if (c->cq_cs_force) {
                cs = c->cq_cs_force;
            } else if (c->cq_tuned && c->cq_cs[cb == 16 ? 0 : (cb == 24 ? 1 : 2)][cq_bucket(mp)]) {
                cs = c->cq_cs[cb == 16 ? 0 : (cb == 24 ? 1 : 2)][cq_bucket(mp)];
            } else {  // row-count rule: about RTARGET rows per CTA
                while (cs < g_cq_csmax[dev] && (long long)cs * cq::RTARGET < mp) cs <<= 1;
            }
            if (cs > g_cq_csmax[dev]) cs = g_cq_csmax[dev];
            const int rmax = cb == 16 ? cq::rpb_max<16>() : (cb == 24 ? cq::rpb_max<24>() : cq::rpb_max<32>());
            while (cs < g_cq_csmax[dev] && (mp + cs - 1) / cs > rmax) cs <<= 1;  // fit the rows
            int rpb = (mp + cs - 1) / cs;
            if (rpb > rmax) {  // too tall for the cluster's shared memory: falls back at once
                cs = 1;
                rpb = 1;
            }
            cudaLaunchConfig_t lc = {};
            lc.gridDim = dim3(cs);
            lc.blockDim = dim3(cq::NT);
            lc.dynamicSmemBytes = cb == 16 ? cq::smem<16>(rpb) : (cb == 24 ? cq::smem<24>(rpb) : cq::smem<32>(rpb));
            lc.stream = c->stream;
            cudaLaunchAttribute la[2];
            la[0].id = cudaLaunchAttributeClusterDimension;
            la[0].val.clusterDim.x = cs;
            la[0].val.clusterDim.y = 1;
            la[0].val.clusterDim.z = 1;
            la[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            la[1].val.programmaticStreamSerializationAllowed = 1;
            lc.attrs = la;
            lc.numAttrs = (c->no_pdl || c->capturing) ? 1 : 2;
            const DevDesc* dd = x->dd;
            if (cb == 16)
                PTT_CUDA(cudaLaunchKernelEx(&lc, cq::k_cq_factor<16>, dd, i, mode, pl, wp, wsb, rpb, c->d_qrstat));
            else if (cb == 24)
                PTT_CUDA(cudaLaunchKernelEx(&lc, cq::k_cq_factor<24>, dd, i, mode, pl, wp, wsb, rpb, c->d_qrstat));
            else
                PTT_CUDA(cudaLaunchKernelEx(&lc, cq::k_cq_factor<32>, dd, i, mode, pl, wp, wsb, rpb, c->d_qrstat));
            PTT_LAUNCHED(c);
        }
        if (cb == 16)
            PTT_CUDA(ptt_launch(c, k_wfactor<16>, dim3(g), dim3(b), sm, x->dd, i, mode, pl, wp, wsb, use_cq, c->d_status));
        else if (cb == 24)
            PTT_CUDA(ptt_launch(c, k_wfactor<24>, dim3(g), dim3(b), sm, x->dd, i, mode, pl, wp, wsb, use_cq, c->d_status));
        else
            PTT_CUDA(ptt_launch(c, k_wfactor<32>, dim3(g), dim3(b), sm, x->dd, i, mode, pl, wp, wsb, use_cq, c->d_status));
        ptt_time_end(c, PTT_TIME_TSQR);
        PTT_LAUNCHED(c);
        return PTT_OK;
    };
    auto apply = [&](int k0, int nb, int mode, int Wmax, int cmax, Fin fin = Fin{}) -> int {
        const int cb = cbound(cmax);
        const dim3 g((Wmax + WPB - 1) / WPB, nb), b(32 * WPB);
        if (cb == 16)
            PTT_CUDA(ptt_launch(c, k_wapply<16>, dim3(g), dim3(b), 0, x->dd, k0, mode, base, wp, ws, use_cq, fin));
        else if (cb == 24)
            PTT_CUDA(ptt_launch(c, k_wapply<24>, dim3(g), dim3(b), 0, x->dd, k0, mode, base, wp, ws, use_cq, fin));
        else
            PTT_CUDA(ptt_launch(c, k_wapply<32>, dim3(g), dim3(b), 0, x->dd, k0, mode, base, wp, ws, use_cq, fin));
        PTT_LAUNCHED(c);
        if (use_cq && mode == RIGHT_T) {  // LEFT: the cluster wrote Q already
            long long gx = ((long long)Wmax * 32 + cq::NT - 1) / cq::NT;
            gx = gx < 1 ? 1 : (gx > 4096 ? 4096 : gx);
            const dim3 gw((unsigned)gx, nb);
            if (cb == 16)
                PTT_CUDA(ptt_launch(c, cq::k_cq_write<16>, dim3(gw), dim3(cq::NT), 0, x->dd, k0, base, wp, ws));
            else if (cb == 24)
                PTT_CUDA(ptt_launch(c, cq::k_cq_write<24>, dim3(gw), dim3(cq::NT), 0, x->dd, k0, base, wp, ws));
            else
                PTT_CUDA(ptt_launch(c, cq::k_cq_write<32>, dim3(gw), dim3(cq::NT), 0, x->dd, k0, base, wp, ws));
            PTT_LAUNCHED(c);
        }
        return PTT_OK;
    };
    // the launches below, as one unit that can be captured and replayed;
    // the key holds every value they bake in
    struct Key {
        int tag, d, phases, only, use_cq, tuned;
        const void *dd, *ws, *cnt, *status, *stats;
        long long stride;
        int Pcap;
        double delta;
        int n[PTT_MAX_DIM], rk[PTT_MAX_DIM + 1], mr[PTT_MAX_DIM + 1];
    } key;
    memset(&key, 0, sizeof(key));
    key.tag = 1;
    key.d = d;
    key.phases = phases;
    key.only = only;
    key.use_cq = use_cq;
    key.tuned = c->cq_tuned;
    key.dd = x->dd;
    key.ws = ws;
    key.cnt = c->d_counters;
    key.status = c->d_status;
    key.stats = c->d_stats;
    key.stride = wp.stride;
    key.Pcap = wp.Pcap;
    key.delta = delta;
    for (int i = 0; i < d; i++) key.n[i] = x->n[i];
    for (int i = 0; i <= d; i++) {
        key.rk[i] = rk[i];
        key.mr[i] = maxr ? maxr[i] : -1;
    }
    auto issue = [&]() -> int {
        if (phases & 4) {
            const int i = only;
            double* wsb;
            Plan pl = bond(i, &wsb);
            if ((rc = factor(i, LEFT, Wl[i], pl, wsb))) return rc;
            // the apply's last block publishes the rank and swaps the core
            if ((rc = apply(i, 1, LEFT, Wl[i], rk[i + 1], Fin{fin_ticket, i + 1, i, &pl.info->q}))) return rc;
            return PTT_OK;
        }
        if (phases & 1) {
            int Wmax = 1, cmax = 1;
            for (int i = 0; i < d - 1; i++) {
                cmax = rk[i + 1] > cmax ? rk[i + 1] : cmax;
                double* wsb;
                Plan pl = bond(i, &wsb);
                if ((rc = factor(i, LEFT, Wl[i], pl, wsb))) return rc;
                Wmax = Wl[i] > Wmax ? Wl[i] : Wmax;
                const long long ncap = (long long)x->n[i + 1] * rk[i + 2];
                int gy = (int)((ncap + 63) / 64);
                if (gy > 4096) gy = 4096;
                // the contraction's last block publishes the rank and swaps the core
                const int cb = cbound(rk[i + 1]);
                auto kern = cb == 16 ? k_wgemm_rx<2> : (cb == 24 ? k_wgemm_rx<3> : k_wgemm_rx<4>);
                PTT_CUDA(ptt_launch(c, kern, dim3(gy), dim3(256), 0, x->dd, i + 1, pl, (const double*)wsb, fin_ticket));
                PTT_LAUNCHED(c);
            }
            if (d > 1) {
                if ((rc = apply(0, d - 1, LEFT, Wmax, cmax))) return rc;
                PTT_CUDA(ptt_launch(c, k_wswap, dim3(1), dim3(64), 0, x->dd, 0, d - 1, c->d_status));
                PTT_LAUNCHED(c);
            }
        }
        if (phases & 2) {
            int Wmax = 1, cmax = 1;
            for (int i = d - 1; i >= 1; i--) {
                cmax = rk[i] > cmax ? rk[i] : cmax;
                double* wsb;
                Plan pl = bond(i, &wsb);
                if ((rc = factor(i, RIGHT_T, Wr[i], pl, wsb))) return rc;
                Wmax = Wr[i] > Wmax ? Wr[i] : Wmax;
                const int mr = maxr ? maxr[i] : rk[i];
                ptt_time_begin(c, PTT_TIME_SVD);
                if ((rc = launch_svd(c, rk[i], pl, wsb, delta, mr, i))) return rc;
                ptt_time_end(c, PTT_TIME_SVD);
                PTT_LAUNCHED(c);
                const long long mcap = (long long)rk[i - 1] * x->n[i - 1];
                int gx = (int)((mcap + 63) / 64);
                if (gx > 4096) gx = 4096;
                const int cb = cbound(rk[i]);
                auto kern = cb == 16 ? k_wgemm_xm<2> : (cb == 24 ? k_wgemm_xm<3> : k_wgemm_xm<4>);
                PTT_CUDA(ptt_launch(c, kern, dim3(gx), dim3(256), 0, x->dd, i - 1, pl, (const double*)wsb, fin_ticket));
                PTT_LAUNCHED(c);
            }
            if (d > 1) {
                PTT_CUDA(ptt_launch(c, k_svd_replay_b, dim3(dim3(4, d - 1)), dim3(256), replay_smem<32>(), base, ws, wp.stride, 1));
                PTT_LAUNCHED(c);
                if ((rc = apply(1, d - 1, RIGHT_T, Wmax, cmax))) return rc;
                PTT_CUDA(ptt_launch(c, k_wswap, dim3(1), dim3(64), 0, x->dd, 1, d, c->d_status));
                PTT_LAUNCHED(c);
            }
        }
        return PTT_OK;
    };
    return ptt_graph_run(c, &key, sizeof(key), issue);
}

}  // namespace

// Per-bond threshold of the reference applied to the unnormalised tensor.
double ptt_round_threshold(const ptt_tt* x, double tol) {
    const int d = x->d;
    if (d < 2) return INFINITY;
    double lg = 0.0;
    for (int k = 0; k < d; k++) lg += log((double)x->n[k]);
    return tol / sqrt(d - 1.0) * exp(0.5 * lg);
}

extern "C" int ptt_round_stats(ptt_ctx* c, int d, double* out) {
    if (!c || !out || d < 1 || d > PTT_MAX_DIM) return ptt_set_error(PTT_ERR_ARG, "ptt_round_stats: bad arguments");
    PTT_CUDA(cudaStreamSynchronize(c->stream));
    PTT_CUDA(cudaMemcpy(out, c->d_stats, sizeof(double) * PTT_STAT_LEN * (size_t)d, cudaMemcpyDeviceToHost));
    return PTT_OK;
}

int ptt_round_phases(ptt_tt* x, double tol, const int* maxrank, int phases, int only) {
    if (!x) return ptt_set_error(PTT_ERR_ARG, "ptt_round: null tt");
    if (x->d < 2) return PTT_OK;
    int rk[PTT_MAX_DIM + 1];
    cudaSetDevice(x->ctx->device);
    if (x->ctx->fixed_plans) {
        // capacity-sized plan: no host synchronisation (stream capture)
        for (int k = 0; k <= x->d; k++) rk[k] = x->rcap[k];
    } else {
        // plan from the actual ranks (one read-back): tiles, trees and grids
        // then match the tensor instead of its capacity
        int rc = ptt_tt_get_ranks(x, rk);
        if (rc) return rc;
    }
    return ptt_round_phases_rk(x, rk, tol, maxrank, phases, only);
}

// The same with upper bounds rk[0..d] of the ranks known to the caller (no
// read-back).
int ptt_round_phases_rk(ptt_tt* x, const int* rk, double tol, const int* maxrank, int phases, int only) {
    if (!x) return ptt_set_error(PTT_ERR_ARG, "ptt_round: null tt");
    if (x->d < 2) return PTT_OK;
    if (!(tol >= 0.0)) return ptt_set_error(PTT_ERR_ARG, "ptt_round: tol must be >= 0");
    cudaSetDevice(x->ctx->device);
    int rmax = 1;
    for (int k = 0; k <= x->d; k++) rmax = rk[k] > rmax ? rk[k] : rmax;
    const double delta = ptt_round_threshold(x, tol);
    if (rmax <= 32 && wt_fits(x, rk)) return round_impl_w(x, rk, delta, maxrank, phases, only);
    if (rmax <= 32) return round_impl<32>(x, rk, delta, maxrank, phases, only);
    if (rmax <= 64) return round_impl<64>(x, rk, delta, maxrank, phases, only);
    if (rmax <= 128) return round_impl<128>(x, rk, delta, maxrank, phases, only);
    return ptt_set_error(PTT_ERR_CAPACITY, "ptt_round: rank %d > 128 not supported", rmax);
}

extern "C" int ptt_ctx_fixed_plans(ptt_ctx* c, int on) {
    if (!c) return ptt_set_error(PTT_ERR_ARG, "null context");
    c->fixed_plans = on ? 1 : 0;
    return PTT_OK;
}

extern "C" int ptt_round(ptt_tt* x, double tol, const int* maxrank) {
    return ptt_round_phases(x, tol, maxrank, 3, 0);
}

extern "C" int ptt_ctx_ozaki(ptt_ctx* c, int on) {
    if (!c) return ptt_set_error(PTT_ERR_ARG, "null context");
    c->ozaki = on ? 1 : 0;
    for (int l = 0; l < c->nlanes; l++)
        if (c->lanes[l]) c->lanes[l]->ozaki = c->ozaki;
    return PTT_OK;
}

// G = A^T A of a device m x c column-major matrix (c <= 64): method 0 on the
// FP64 tensor cores, 1 by the Ozaki split on the fifth-generation tensor
// cores (the two Gram kernels of the grid Cholesky QR, ptt_gridqr.cuh and
// ptt_ozaki.cuh).
extern "C" int ptt_gram(ptt_ctx* c, const double* A, long long m, int cols, long long lda, double* G, int method) {
    if (!c || !A || !G || m < 1 || cols < 1 || cols > 64 || lda < m || (method != 0 && method != 1))
        return ptt_set_error(PTT_ERR_ARG, "ptt_gram: bad arguments");
    const long long nbl = (m + gq::Cfg<64>::RPB_MAX - 1) / gq::Cfg<64>::RPB_MAX;
    if (nbl > (1ll << 24)) return ptt_set_error(PTT_ERR_CAPACITY, "ptt_gram: %lld rows", m);
    cudaSetDevice(c->device);
    int rc;
    const int nb = (int)nbl, ng = (nb + gq::GROUP - 1) / gq::GROUP;
    if ((rc = ptt_ws_reserve(c, sizeof(double) * (size_t)(nb + ng) * gq::Cfg<64>::UP + 256))) return rc;
    if ((rc = ptt_counters_reserve(c, (size_t)ng + 1))) return rc;
    double* part = (double*)c->ws;
    double* gpart = part + (long long)nb * gq::Cfg<64>::UP;
    if (method == 1) {
        PTT_CUDA(cudaFuncSetAttribute(gq::k_gram<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)gq::SM_ROWS_OZ));
        gq::k_gram<true><<<nb, gq::NT, gq::SM_ROWS_OZ, c->stream>>>(A, m, cols, lda, part, gpart, c->d_counters, G);
    } else {
        PTT_CUDA(cudaFuncSetAttribute(gq::k_gram<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)gq::SM_GRAM));
        gq::k_gram<false><<<nb, gq::NT, gq::SM_GRAM, c->stream>>>(A, m, cols, lda, part,
                                                                                          gpart, c->d_counters, G);
    }
    PTT_LAUNCHED(c);
    return PTT_OK;
}

// ---------------------------------------------------------------------------
// autotuner of the Cholesky-QR cluster size
// ---------------------------------------------------------------------------
namespace {
__global__ void k_tune_fill(double* p, long long cnt, unsigned long long seed) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt;
         e += (long long)gridDim.x * blockDim.x) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(e + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        p[e] = (double)(z >> 11) * 1.1102230246251565e-16 - 0.5;  // uniform in [-0.5, 0.5)
    }
}
}  // namespace

// For each column bound (16, 24, 32) and rows bucket (512 ... 16384), time the
// QR of one core (the single-core phase of a rounding, the path the sketch
// uses per core) of a random m x c unfolding with every cluster size the
// device can hold, and keep the fastest in the context's table.
extern "C" int ptt_ctx_autotune(ptt_ctx* c) {
    if (!c) return ptt_set_error(PTT_ERR_ARG, "null context");
    cudaSetDevice(c->device);
    const int graphs = c->graphs, tkind = c->tkind;
    c->graphs = 0;
    c->tkind = 0;
    int rc = PTT_OK;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    ptt_tt *x = nullptr, *x0 = nullptr;
    PTT_CUDA(cudaEventCreate(&e0));
    PTT_CUDA(cudaEventCreate(&e1));
    static const int cbs[3] = {16, 24, 32};
    for (int ci = 0; ci < 3 && !rc; ci++) {
        for (int bi = 0; bi < 6 && !rc; bi++) {
            const int cb = cbs[ci], m = 512 << bi;
            int n[2] = {m, 1}, cap[3] = {1, cb, 1}, rk[3] = {1, cb, 1};
            x = ptt_tt_create(c, 2, n, cap);
            x0 = ptt_tt_create(c, 2, n, cap);
            if (!x || !x0) {
                rc = ptt_last_error() ? ptt_last_error() : PTT_ERR_CUDA;
                break;
            }
            if ((rc = ptt_pull_desc(x0))) break;
            k_tune_fill<<<148, 256, 0, c->stream>>>(x0->hd.core[0], (long long)m * cb, 1234567ull + 977ull * bi + ci);
            k_tune_fill<<<1, 32, 0, c->stream>>>(x0->hd.core[1], cb, 7654321ull + ci);
            if ((rc = ptt_cuda_check(cudaGetLastError(), "tune fill"))) break;
            float best = 1e30f, theur = 1e30f;
            int bestcs = 1;
            // the size the row-count heuristic would take
            int hcs = 1;
            {
                const int dev = c->device & 63;
                const int csmax = g_cq_csmax[dev] ? g_cq_csmax[dev] : cq::CSMAX;
                while (hcs < csmax && (long long)hcs * cq::RTARGET < m) hcs <<= 1;
            }
            for (int cs = 1; cs <= cq::CSMAX && !rc; cs <<= 1) {
                int dev = c->device & 63;
                if (g_cq_csmax[dev] && cs > g_cq_csmax[dev]) break;
                const int rmax = cb == 16 ? cq::rpb_max<16>() : (cb == 24 ? cq::rpb_max<24>() : cq::rpb_max<32>());
                if ((m + cs - 1) / cs > rmax) continue;
                c->cq_cs_force = cs;
                float tmin = 1e30f;
                for (int rep = 0; rep < 7 && !rc; rep++) {
                    if ((rc = ptt_tt_copy(x, x0))) break;
                    if ((rc = ptt_ctx_synchronize(c))) break;
                    PTT_CUDA(cudaEventRecord(e0, c->stream));
                    if ((rc = ptt_round_phases_rk(x, rk, 0.0, NULL, 4, 0))) break;
                    PTT_CUDA(cudaEventRecord(e1, c->stream));
                    PTT_CUDA(cudaEventSynchronize(e1));
                    float ms = 0.f;
                    PTT_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                    if (rep > 0 && ms < tmin) tmin = ms;  // rep 0 warms up
                }
                if (tmin < best) {
                    best = tmin;
                    bestcs = cs;
                }
                if (cs == hcs) theur = tmin;
            }
            // a single timed QR is noisy: leave the heuristic's size unless
            // another one is clearly faster
            if (theur < 1e30f && !(best < 0.85f * theur)) bestcs = 0;  // 0: keep the row-count rule
            c->cq_cs[ci][bi] = (unsigned char)bestcs;
            ptt_tt_destroy(x);
            ptt_tt_destroy(x0);
            x = x0 = nullptr;
        }
    }
    if (x) ptt_tt_destroy(x);
    if (x0) ptt_tt_destroy(x0);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    c->cq_cs_force = 0;
    c->graphs = graphs;
    c->tkind = tkind;
    if (rc) return rc;
    c->cq_tuned++;
    if ((rc = ptt_gemm_autotune(c))) return rc;
    return ptt_ctx_synchronize(c);
}

extern "C" int ptt_ctx_autotune_table(const ptt_ctx* c, int* out) {
    if (!c || !out) return ptt_set_error(PTT_ERR_ARG, "ptt_ctx_autotune_table: bad arguments");
    for (int i = 0; i < 18; i++) out[i] = c->cq_tuned ? c->cq_cs[i / 6][i % 6] : 0;
    return PTT_OK;
}
