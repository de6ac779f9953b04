// What the Cholesky-QR factorisations share (ptt_cholqr.cuh: one cluster, up
// to 32 columns; ptt_gridqr.cuh: the whole GPU, up to 128): the Gram stages'
// rules, the tile layout of their small matrices and the 8 x 8 factor step.
//
// A = Q R is a sequence of Gram stages: stage s has Q_s = A R_1^{-1} ...
// R_s^{-1} (Q_0 = A), its Gram matrix G = Q_s^T Q_s and the accumulated R = T
// (A = Q_s T), and from them
//   * columns whose part of A is below the rounding of A are dropped: column
//     j of Q_s adds q_j T_j: to A, at most |q_j| max_i |T_ji| / |a_i| of each
//     column a_i; where that is below 0.5 sqrt(c) u it is rounding noise of A,
//     and q_j and T_j: are set to zero (exactly zero columns of A likewise).
//     Unfoldings of sums are numerically rank-deficient: without this the
//     noise directions kept the sequence busy for up to eight stages, and 11
//     of the 78 factorisations of a rank-64 rounding with d = 40 fell back;
//   * s >= 1 and max|G - I| <= TAU over the other columns: done, R = T.  A
//     column that this very stage drops was not part of that test and may lie
//     along the others (|q_j q_i| to 1e-8 seen), and a caller may use Q as a
//     projector without R: it is cleared before Q is final (the cluster masks
//     it as it writes Q; the grid, whose Q_s is in memory already, finishes by
//     the first-order factor, whose inverse pivot is zero there);
//   * s >= 1 and max|G - I| <= FIRST: R_{s+1} = I + striu(E) + diag(E)/2 with E
//     = G - I, the Cholesky factor of I + E to first order; when max|E| <=
//     FIRST_DONE that finishes without another Gram stage;
//   * otherwise R_{s+1} = chol(H) D with H = D^-1 G D^-1 and D = diag(the power
//     of two above |q_j|) (a diagonal in [1/4, 1], so the scale of a column does
//     not matter, and no rounding: with D = diag(|q_j|) the pivots and their
//     inverses were each off by the roundings of |q_j|, 1 / |q_j| and H, whose
//     product is 1 + 1.2e-16 on average, not 1, and a time step added that up to
//     an error of 5e-15).  A pivot
//     below PIV is set to PIV and the rest of its row of R to zero: the column
//     is only rescaled and is orthogonalised against the others in the next
//     stage, where it has unit norm again.  So every stage resolves another
//     seven decades of the spectrum, whatever the condition: condition 1e25
//     and exactly repeated columns take four or five stages.  (Shifted
//     Cholesky QR -- Fukaya, Kannan, Nakatsukasa, Yamamoto, Yanagisawa, SIAM
//     J. Sci. Comput. 42 (2020) -- resolves five decades a stage at 16384 x 64
//     and perturbs the columns that need no shift.)
// The row-wise triangular solve changes A = Q R by O(u |a_j|) per column and
// stage, so R carries the singular values to the accuracy of a Householder R.
#pragma once

namespace gst {

constexpr double TAU = 1e-14;
constexpr double FIRST = 1e-7;
constexpr double FIRST_DONE = 1e-8;
constexpr double U = 1.1102230246251565e-16;
constexpr double PIV = 1e-13;          // smallest pivot of the equilibrated Gram matrix that is trusted: its
                                       // relative error is ~1e-15 / PIV, so the next stage sees max|E| ~ 1e-2
constexpr double RPIV = 3.1622776601683795e-7;  // its root
constexpr double DROP = 0.5 * U;       // times sqrt(c): a column's part of A that is rounding noise
constexpr double SMALL = 1e-280;       // squared norms below this lose digits to underflow: fall back
constexpr double LARGE = 1e300;        // and above this are near overflow

enum { RUN = 0, DONE = 1, FALLBACK = 2, FINISH = 4 };

// the power of two above a column norm d > 0, and its inverse
__device__ __forceinline__ void pow2_above(double d, double* p, double* ip) {
    const int e = (__double2hiint(d) & 0x7ff00000) + 0x00100000;
    *p = __hiloint2double(e, 0);
    *ip = __hiloint2double(0x7fe00000 - e, 0);
}

// A symmetric or upper triangular matrix is kept as its upper 8 x 8 tiles:
// tile (I, J), I <= J, is number J (J + 1) / 2 + I (so c columns use the first
// tiles, whatever the bound), entry (i, j) of a tile at tix(i, j).  The swizzle
// puts the four rows of an mma fragment load, and the four columns of a
// transposed one, in different banks.
__host__ __device__ __forceinline__ constexpr int tix(int i, int j) { return i * 8 + (j ^ ((i & 2) << 1)); }
__host__ __device__ __forceinline__ constexpr int tnum(int I, int J) { return (J * (J + 1)) / 2 + I; }
__host__ __device__ __forceinline__ constexpr int telem(int i, int j) {
    return tnum(i >> 3, j >> 3) * 64 + tix(i & 7, j & 7);
}
__device__ __forceinline__ void tile_of(int t, int* I, int* J) {
    int j = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((j + 1) * (j + 2) / 2 <= t) j++;
    while (j * (j + 1) / 2 > t) j--;
    *J = j;
    *I = t - j * (j + 1) / 2;
}
__device__ __forceinline__ void mma884(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// Cholesky factor of the 8 x 8 block at G (tile layout, upper half read) in
// the caller's registers -- every thread does the same 8 steps, so nothing is
// broadcast: r[i][j], j >= i, and inv[i] = 1 / r[i][i].  `live`: bits of the
// columns that are kept; a dropped one gets a zero row and inv 0, a pivot not
// above PIV (NaN included) PIV and a zero rest of its row.  Returns the bits
// of the rows that are zero beyond the diagonal.
__device__ __forceinline__ unsigned chol8(const double* G, unsigned live, double (&r)[8][8], double (&inv)[8]) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = i; j < 8; j++) r[i][j] = G[tix(i, j)];
    unsigned weak = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const bool on = (live >> j) & 1u;
        const double p = r[j][j];
        const bool good = p > PIV;
        const double iv = on ? (good ? rsqrt(p) : 1.0 / RPIV) : 0.0;  // the test runs beside the root
        const double io = good ? iv : 0.0;
        r[j][j] = on ? (good ? p * iv : RPIV) : 0.0;
        inv[j] = iv;
        if (!(on && good)) weak |= 1u << j;
#pragma unroll
        for (int l = j + 1; l < 8; l++) r[j][l] *= io;
#pragma unroll
        for (int i = j + 1; i < 8; i++)
#pragma unroll
            for (int l = i; l < 8; l++) r[i][l] = fma(-r[j][i], r[j][l], r[i][l]);
    }
    return weak;
}
// Column `j` (0..7) of the tile at Gc, solved against that factor in place.
__device__ __forceinline__ void solve8(double* Gc, int j, const double (&r)[8][8], const double (&inv)[8], unsigned weak) {
    double y[8];
#pragma unroll
    for (int i = 0; i < 8; i++) y[i] = Gc[tix(i, j)];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        y[i] = ((weak >> i) & 1u) ? 0.0 : y[i] * inv[i];
#pragma unroll
        for (int l = i + 1; l < 8; l++) y[l] = fma(-r[i][l], y[i], y[l]);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) Gc[tix(i, j)] = y[i];
}
// Trailing tile (I, K) -= R_{J,I}^T R_{J,K} by one warp.
__device__ __forceinline__ void trail8(double* sG, int J, int I, int K, int li, int lk) {
    const double* Ra = sG + tnum(J, I) * 64;
    const double* Rb = sG + tnum(J, K) * 64;
    double2* Ct = (double2*)(sG + tnum(I, K) * 64 + tix(li, 2 * lk));
    double2 v = *Ct;
    mma884(v.x, v.y, -Ra[tix(lk, li)], Rb[tix(lk, li)]);
    mma884(v.x, v.y, -Ra[tix(lk + 4, li)], Rb[tix(lk + 4, li)]);
    *Ct = v;
}
// Tile (I, J) of F T, both upper triangular in tiles, by one warp: entries
// (li, 2 lk) and the next.
__device__ __forceinline__ double2 tile_product(const double* F, const double* T, int I, int J, int li, int lk) {
    double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
    for (int K = I; K <= J; K++) {
        const double* Fk = F + tnum(I, K) * 64;
        const double* Tk = T + tnum(K, J) * 64;
        mma884(a0, a1, Fk[tix(li, lk)], Tk[tix(lk, li)]);
        mma884(b0, b1, Fk[tix(li, lk + 4)], Tk[tix(lk + 4, li)]);
    }
    return make_double2(a0 + b0, a1 + b1);
}

// x <- x R^{-1} for the CTA's rows (h of them, zero rows up to a multiple of
// 16), one warp per 16 rows, by 8-column blocks in order: the update of block
// J by the solved blocks, X_J - Y_{<J} R_{<J,J}, on the FP64 tensor cores
// (two accumulators a tile, so the chain is J products long), then forward
// substitution in the 8 x 8 diagonal block with one lane per row, the block
// passed through shared memory: 8 dependent multiply-add pairs, where passing
// each solved entry between the row's four lanes by shuffles took ~65 cycles
// an entry.  Rows are independent, so a warp needs no block barrier.  R upper
// triangular in tiles, iv = inverse pivots, zero beyond c and for a dropped
// column.  XP: row pitch (even), NW: warps.
template <int XP, int NW>
__device__ __forceinline__ void tile_solve(double* Xs, int h, const double* R, const double* iv, int nbc) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int li = lane >> 2, lk = lane & 3;
    for (int u = warp; u * 16 < h; u += NW) {
        double* xa = Xs + (u * 16 + li) * XP;  // this lane's fragment rows
        double* xb = xa + 8 * XP;
        double* xr = Xs + (u * 16 + (lane & 15)) * XP;
        for (int J = 0; J < nbc; J++) {
            const double2 ca = *(const double2*)(xa + 8 * J + 2 * lk);
            const double2 cb = *(const double2*)(xb + 8 * J + 2 * lk);
            double a0 = ca.x, a1 = ca.y, b0 = cb.x, b1 = cb.y;
            double e0 = 0.0, e1 = 0.0, f0 = 0.0, f1 = 0.0;
            if (J > 0) {
                for (int I = 0; I < J; I++) {
                    const double* Rt = R + tnum(I, J) * 64;
                    const double r0 = Rt[tix(lk, li)], r1 = Rt[tix(lk + 4, li)];
                    mma884(a0, a1, -xa[8 * I + lk], r0);
                    mma884(b0, b1, -xb[8 * I + lk], r0);
                    mma884(e0, e1, -xa[8 * I + 4 + lk], r1);
                    mma884(f0, f1, -xb[8 * I + 4 + lk], r1);
                }
                *(double2*)(xa + 8 * J + 2 * lk) = make_double2(a0 + e0, a1 + e1);
                *(double2*)(xb + 8 * J + 2 * lk) = make_double2(b0 + f0, b1 + f1);
                __syncwarp();
            }
            if (lane < 16) {
                const double* Rd = R + tnum(J, J) * 64;
                double x[8];
#pragma unroll
                for (int j = 0; j < 8; j += 2) {
                    const double2 v = *(const double2*)(xr + 8 * J + j);
                    x[j] = v.x;
                    x[j + 1] = v.y;
                }
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const double y = x[j] * iv[8 * J + j];
                    x[j] = y;
#pragma unroll
                    for (int l = j + 1; l < 8; l++) x[l] = fma(-y, Rd[tix(j, l)], x[l]);
                }
#pragma unroll
                for (int j = 0; j < 8; j += 2) *(double2*)(xr + 8 * J + j) = make_double2(x[j], x[j + 1]);
            }
            __syncwarp();
        }
    }
}

}  // namespace gst
