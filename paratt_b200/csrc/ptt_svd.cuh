// One-sided Jacobi SVD of a bond's factor (included by ptt_round.cu inside
// its anonymous namespace): L = R^T (c x q, R the root factor of the LQ), the
// rank rule, U S, and a log of the rotations from which k_svd_replay(_b)
// rebuilds V row by row.
//
// The columns are taken in blocks of two.  A group of LP lanes holds two
// blocks -- four columns, rows p + LP v in lane p's registers -- and a
// super-round rotates their four cross pairs in two steps of two independent
// pairs; then the blocks move on.  Every pair of blocks meets once per sweep,
// and one step at the end of the sweep rotates the two columns inside each
// block: nblk - 1 super-rounds of nblk blocks, 4 G - 1 steps for G groups.
//
// A step is one dependent chain on one SM (dot product, shuffle sum, rotation
// angle, its application), beside ~5 c^2 / 2 FP64 operations, so the design is
// about what is on that chain and about the traffic beside it:
//   * with the columns in shared memory every round moved all of L in and out
//     (at 64 columns 512 cycles of shared-memory bandwidth); in registers only
//     the blocks that move travel, through shared memory once per two steps,
//     with the one barrier that orders them (a warp barrier up to 16 columns);
//   * two pairs per step, and two or more warps per scheduler from 48 columns
//     on, overlap their chains;
//   * the angle and the tests come from single precision: FP64 instructions
//     take two issue slots each and every lane of a group repeats the pair's
//     scalar work.  tan theta = t only has to be close: a pair's remaining
//     cosine is the old one times t's relative error, ~1e-7, and the sweeps go
//     on until the cosines (of FP64 dot products) meet the tolerance.  But the
//     rotation must be one to FP64: with t exact in double, cos = (1 +
//     t^2)^(-1/2) by one third-order Newton step (error (1e-7)^3) from the
//     single-precision value.  x' = cos (x - t y), y' = cos (y + t x): the
//     differences do not wait for cos.  L is scaled by a power of two to a
//     largest column norm of about one, so the single-precision values do not
//     overflow;
//   * a warp whose pairs are all orthogonal already skips the application.
//
// The figures of a bond's SVD against the kernels before (columns in shared
// memory, or one column per group moved by shuffles, FP64 reciprocal square
// roots on the chain): 20 columns 81 -> 50 us, 64 columns of a rank-32 sum 283 ->
// 133 us (99 where half of them are noise), 95 columns with a spectrum of 2^-j
// 531 -> 130 us, 14 columns of a time step 31 -> 20.
#pragma once

constexpr int MAXSW = 40;  // Jacobi sweep limit

// Pair orders of a recorded rotation log (Info::order).
enum { ORD_CIRCLE = 2, ORD_RING = 3 };

// Blocks of group g in super-round s of the circle (round-robin) order over
// nblk = 2 G blocks: position 0 stays, every other block moves one position.
__device__ __forceinline__ int circle_blk(int pos, int s, int nblk) {
    return pos == 0 ? 0 : 1 + (pos - 1 + s) % (nblk - 1);
}
// Stationary-ring order, G a power of two.  Level l (ring size hb = G >> l,
// super-rounds [2G - 2hb, 2G - hb)): ring b of hb consecutive groups owns
// blocks [2 hb b, 2 hb (b + 1)); group i of the ring keeps block 2 hb b + i
// and meets 2 hb b + hb + (i + s) mod hb at shift s, so the second blocks move
// one group along the ring while the first ones stay.  Between levels each
// ring splits in two: the first half pairs its first blocks among themselves,
// the second half its second blocks (one block swapped between groups i and
// i + hb / 2).
__device__ __forceinline__ void ring_blks(int g, int s, int G, int* a, int* b) {
    const int x = 2 * G - 1 - s, lg = 31 - __clz(x), hb = 1 << lg;
    const int sh = s - (2 * G - 2 * hb), i = g & (hb - 1), b0 = (g >> lg) << (lg + 1);
    *a = b0 + i;
    *b = b0 + hb + ((i + sh) & (hb - 1));
}
// Columns of pair `pr` (two per group) in step st of a sweep over G groups.
__device__ __forceinline__ void svd_pair(int pr, int st, int G, int order, int* pc, int* qc) {
    const int g = pr >> 1, k = pr & 1, ns = 2 * G - 1;
    if (st == 2 * ns) {  // inside the blocks
        const int blk = order == ORD_RING ? pr : (k ? 2 * G - 1 - g : g);
        *pc = 2 * blk;
        *qc = 2 * blk + 1;
        return;
    }
    int a, b;
    if (order == ORD_RING) {
        ring_blks(g, st >> 1, G, &a, &b);
    } else {
        a = circle_blk(g, st >> 1, 2 * G);
        b = circle_blk(2 * G - 1 - g, st >> 1, 2 * G);
    }
    *pc = 2 * a + k;
    *qc = 2 * b + (k ^ (st & 1));
}

__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

constexpr int SVD_LP = 8;  // lanes per group: 16 took 888-946 cycles a step at 64 columns where 8 take 800
template <int RB>
__host__ __device__ constexpr int svd_nt() {
    return RB / 4 * SVD_LP;
}
// buffers of the moving blocks: two where they fit (one barrier a move), else one
template <int RB>
__host__ __device__ constexpr int svd_nb() {
    return RB <= 96 ? 2 : 1;
}
// the moving blocks, [buffer][block][row][lane] pairs of the block's columns,
// so the lanes of a group touch consecutive 16-byte words; in the same place
// the columns for the epilogue
template <int RB>
static size_t svd_smem() {
    const size_t cols = (size_t)RB * (RB + 2), x = (size_t)svd_nb<RB>() * RB * RB;
    return sizeof(double) * (cols > x ? cols : x);
}

// v divided by the power of two of exponent field E (bits 20..30 of a double's
// high word), truncated to single precision; below its range: 0.  By integer
// operations: a conversion instruction takes eight issue slots of a pipe that
// the reciprocal square roots need too (18 conversions and square roots a
// step held it for 144 cycles).
__device__ __forceinline__ float scaled_float(double v, int E) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int m = (hi & 0x7fffffff) - (E - 0x07f00000);
    const int b = (int)__funnelshift_l((unsigned)lo, (unsigned)m, 3);
    return __int_as_float((m < 0x00100000 ? 0 : b) | (hi & 0x80000000));
}
// a normal single-precision value as a double (0 where !on)
__device__ __forceinline__ double widen(float f, bool on) {
    const int b = __float_as_int(f);
    const int hi = (((b & 0x7fffffff) >> 3) + 0x38000000) | (b & 0x80000000);
    return __hiloint2double(on ? hi : 0, on ? b << 29 : 0);
}

// The pair's rotation from its squared norms and dot product: t = tan theta (0
// for a pair left alone) and cos theta.  With dd = be - al, g2 = 2 ga, r =
// sqrt(dd^2 + g2^2): cos 2theta = |dd| / r, sin 2theta = sign(dd) g2 / r, cos
// theta = sqrt((1 + cos 2theta) / 2), tan theta = sin 2theta / (1 + cos
// 2theta) -- dd and ga scaled by the exponent of max(al, be).
struct Pre {
    double lim, small;  // squared dot products: of a cosine of tol, and of a rotation that leaves the others alone
    float ds;           // dd, scaled
    int E;              // exponent field of max(al, be)
    bool big;
};
// gap2: see the stop rule of the sweeps
__device__ __forceinline__ Pre svd_pre(double al, double be, int thr, double tol2, double gap2, bool act) {
    Pre r;
    const int ha = __double2hiint(al), hb = __double2hiint(be);
    r.big = act && min(ha, hb) > thr;
    r.E = max(ha, hb) & 0x7ff00000;
    const double dd = be - al, ab = al * be;
    r.ds = scaled_float(dd, r.E);
    r.lim = tol2 * ab;
    r.small = fmin(1e-18 * ab, gap2 * (dd * dd));
    return r;
}
__device__ __forceinline__ void svd_angle(const Pre& r, double ga, bool on, double* t, double* cs) {
    const float w = 2.0f * scaled_float(ga, r.E);
    const float ri = rsqrt_ftz(fmaf(w, w, fmaf(r.ds, r.ds, 1e-36f)));
    const float hc = fmaf(0.5f * fabsf(r.ds), ri, 0.5f);  // (1 + cos 2theta) / 2, in [1/2, 1]
    const float ic = rsqrt_ftz(hc);                        // 1 / cos theta
    const float tf = (copysignf(0.5f, r.ds) * w * ri) * (ic * ic);
    *t = widen(tf, on && tf != 0.0f);
    const double y = widen(on ? hc * ic : 1.0f, true);
    const double e = fma(-fma(*t, *t, 1.0) * y, y, 1.0);
    *cs = fma(y * e, fma(0.375, e, 0.5), y);
}

template <int NR>
__device__ __forceinline__ double dot_rows(const double (&x)[NR], const double (&y)[NR]) {
    constexpr int NA = NR < 4 ? (NR < 2 ? 1 : 2) : 4;
    double a[NA];
#pragma unroll
    for (int v = 0; v < NR; v++) a[v % NA] = v < NA ? x[v] * y[v] : fma(x[v], y[v], a[v % NA]);
    if (NA == 4) return (a[0] + a[1]) + (a[2 % NA] + a[3 % NA]);
    return NA == 2 ? a[0] + a[1 % NA] : a[0];
}

// RB bounds c and q (a multiple of 16; RB / 4 groups).
template <int RB>
__global__ void __launch_bounds__(svd_nt<RB>(), 1) k_svd_jacobi(Plan pl, double* ws, double delta, int maxr, int bond,
                                                                int* status) {
    PTT_PDL_ENTRY();
    constexpr int LP = SVD_LP, NTH = svd_nt<RB>(), NW = NTH / 32, NR = RB / LP;
    constexpr int S = RB + 2, NBLK = RB / 2, NBUF = svd_nb<RB>();
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ __align__(16) double sm[];
    double* Lc = sm;   // RB columns x S
    double2* xch = (double2*)sm;
    __shared__ double2 s_xn[NBUF][NBLK];  // norms of the moving blocks
    __shared__ double s_sig[RB], s_srt[RB], s_suf[RB];
    __shared__ double s_nrm[RB];
    __shared__ int s_ord[RB], s_perm[RB], s_slot[RB];
    __shared__ int s_rot, s_rank;
    __shared__ double s_wmax[NW > 0 ? NW : 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int grp = tid / LP, p = tid % LP;
    Info* info = pl.info;
    if (info->status) return;
    const int CT = pl.CT, c = info->c, q = info->q;
    if (c > RB || q > RB) {  // uniform; the host sizes RB by the bond's rank bound
        if (tid == 0) PTT_STATUS_SET(status, PTT_ERR_CAPACITY);
        return;
    }
    const double* R = ws + pl.o_Rn;  // root factor, row-major CT x CT; L = R^T: column j of L = row j of R
    double A0[NR], A1[NR], B0[NR], B1[NR];
    auto gsum = [&](double v) {
#pragma unroll
        for (int o = LP / 2; o >= 1; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        return v;
    };
    auto sync = [&]() {
        if (NW > 1)
            __syncthreads();
        else
            __syncwarp();
    };
    double a0, a1, b0, b1;  // squared norms of the group's columns
    // The columns as they come (group g: 4 g .. 4 g + 3), their norms, and from
    // them the columns that take part.  Columns below the numerical-rank
    // threshold (sqrt(q) eps_LAPACK times the largest column norm) are
    // rounding noise: rotating noise against noise is a random walk that never
    // meets the relative criterion, and their values are discarded by the rank
    // rule anyway, so they are left alone -- and, since the largest norm only
    // grows, for good: the sweeps run over the qa others alone (half of 64 in
    // the truncation of a rank-32 sum, 50 of 95 in a spectrum of 2^-j).
#pragma unroll
    for (int v = 0; v < NR; v++) {
        const int t = p + LP * v, j = 4 * grp;
        A0[v] = (t < c && j < q) ? R[(long long)j * CT + t] : 0.0;
        A1[v] = (t < c && j + 1 < q) ? R[(long long)(j + 1) * CT + t] : 0.0;
        B0[v] = (t < c && j + 2 < q) ? R[(long long)(j + 2) * CT + t] : 0.0;
        B1[v] = (t < c && j + 3 < q) ? R[(long long)(j + 3) * CT + t] : 0.0;
    }
    a0 = gsum(dot_rows(A0, A0));
    a1 = gsum(dot_rows(A1, A1));
    b0 = gsum(dot_rows(B0, B0));
    b1 = gsum(dot_rows(B1, B1));
    if (p < 4) s_nrm[4 * grp + p] = p == 0 ? a0 : (p == 1 ? a1 : (p == 2 ? b0 : b1));
#pragma unroll
    for (int v = 0; v < NR; v++) {
        const int t = p + LP * v, j = 4 * grp;
        Lc[j * S + t] = A0[v];
        Lc[(j + 1) * S + t] = A1[v];
        Lc[(j + 2) * S + t] = B0[v];
        Lc[(j + 3) * S + t] = B1[v];
    }
    if (tid == 0) s_rot = 0;
    sync();
    double mx = 0.0;
    int qa = 0;
    {
        for (int j = lane; j < RB; j += 32) mx = fmax(mx, s_nrm[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
        const int thr = __double2hiint((double)q * 1.232595164407831e-32 * mx);  // (sqrt(q) * 2^-53)^2 * max |a_j|^2
        for (int j0 = 0; j0 < RB; j0 += 32) {
            const int j = j0 + lane;
            const bool in = j < RB && j < q && s_nrm[j < RB ? j : 0] > 0.0 && __double2hiint(s_nrm[j < RB ? j : 0]) > thr;
            const unsigned m = __ballot_sync(FULL, in);
            const int at = qa + __popc(m & ((1u << lane) - 1u));
            if (warp == 0 && j < RB) {
                s_slot[j] = in ? at : -1;
                if (in) s_perm[at] = j;
            }
            qa += __popc(m);
        }
    }
    // the stationary ring where its power-of-two block count costs at most 15 %
    // more steps than the circle: it takes one sweep in eight less (8.5 against
    // 9.7 at 64 columns, 6.3 against 6.7 at 32) and moves half as many blocks
    const int Gc = qa > 4 ? (qa + 3) >> 2 : 1;                  // groups of the circle order
    const int Gr = Gc > 1 ? 1 << (32 - __clz(Gc - 1)) : 1;      // of the ring order
    const bool ring = 4 * Gr <= RB && 20 * (4 * Gr - 1) <= 23 * (4 * Gc - 1);
    const int G = ring ? Gr : Gc, ns = 2 * G - 1;
    const bool act = grp < G;
    // slots of this group: blocks grp and G + grp (ring) or 2 G - 1 - grp (circle)
    const int ja = 2 * grp, jb = 2 * (ring ? G + grp : 2 * G - 1 - grp);
    int sh = 0;  // L is held as 2^-sh L
    if (mx > 0.0 && mx < 1.0 / 0.0) sh = ilogb(mx) >> 1;
    const double down = scalbn(1.0, -sh);
    sync();
    if (act) {
        auto fetch = [&](int slot, double(&x)[NR]) {
            const double* col = Lc + s_perm[slot < qa ? slot : 0] * S;
#pragma unroll
            for (int v = 0; v < NR; v++) x[v] = slot < qa ? col[p + LP * v] * down : 0.0;
        };
        if (qa > 0) {
            fetch(ja, A0);
            fetch(ja + 1, A1);
            fetch(jb, B0);
            fetch(jb + 1, B1);
        }
    }
    sync();  // the moving blocks take the columns' place
    // exact norms of all columns; returns the largest
    auto norms = [&]() {
        a0 = gsum(dot_rows(A0, A0));
        a1 = gsum(dot_rows(A1, A1));
        b0 = gsum(dot_rows(B0, B0));
        b1 = gsum(dot_rows(B1, B1));
        double mx = act ? fmax(fmax(a0, a1), fmax(b0, b1)) : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(FULL, mx, o));
        if (NW > 1) {
            if (lane == 0) s_wmax[warp] = mx;
            __syncthreads();
#pragma unroll
            for (int w = 0; w < NW; w++) mx = fmax(mx, s_wmax[w]);
        }
        return mx;
    };
    double2* rot = (double2*)(ws + pl.o_rot);
    const int npair = (CT + 2) / 2;
    const double tol = (double)(c < 16 ? 16 : c) * 2.220446049250313e-16;
    const double tol2 = tol * tol;  // |ga| > tol sqrt(al be), compared in squares
    int sweeps = 0;
    bool conv = qa < 2;
    for (int sw = 0; sw < MAXSW && !conv; sw++) {
        mx = norms();
        // (sqrt(q) * 2^-53)^2 * max |a_j|^2, compared by the high words
        const int thr = __double2hiint((double)q * 1.232595164407831e-32 * mx);
        // The sweeps may end after one whose rotations all were small: cosine
        // <= 1e-9 and tangent (ga / |dd| at that size) <= 1e-7.  A rotation by t
        // adds t times the cosine of (q, r) to that of a pair (p, r) already
        // zeroed, so what they leave is ~1e-16, as the single-precision angle
        // leaves 1e-7 of each cosine.  The cosines alone do not tell: equal
        // singular values make a tangent O(1) at any cosine, and stopping on
        // them left a cluster's values wrong by 1e-10.  Only the sweep limit
        // does without the tangents (infinity: fmin takes the other).
        const double gap2 = sw < MAXSW - 1 ? 1e-14 : 1.0 / 0.0;
        int myrot = 0;
        double2* lg = rot + (long long)sw * (CT + 1) * npair + 2 * grp;
        // rotate two independent pairs of the group; log them as pairs 2 grp, 2 grp + 1
        auto step = [&](double(&x0)[NR], double(&y0)[NR], double& nx0, double& ny0, double(&x1)[NR], double(&y1)[NR],
                        double& nx1, double& ny1) {
            double g0 = dot_rows(x0, y0), g1 = dot_rows(x1, y1);
            const Pre r0 = svd_pre(nx0, ny0, thr, tol2, gap2, act), r1 = svd_pre(nx1, ny1, thr, tol2, gap2, act);
#pragma unroll
            for (int o = LP / 2; o >= 1; o >>= 1) {
                g0 += __shfl_xor_sync(FULL, g0, o);
                g1 += __shfl_xor_sync(FULL, g1, o);
            }
            const double q0 = g0 * g0, q1 = g1 * g1;
            const bool on0 = r0.big && q0 > r0.lim, on1 = r1.big && q1 > r1.lim;
            double t0 = 0.0, t1 = 0.0, c0 = 1.0, c1 = 1.0;
            if (__any_sync(FULL, on0 || on1)) {
                svd_angle(r0, g0, on0, &t0, &c0);
                svd_angle(r1, g1, on1, &t1, &c1);
#pragma unroll
                for (int v = 0; v < NR; v++) {
                    const double u0 = fma(-t0, y0[v], x0[v]), w0 = fma(t0, x0[v], y0[v]);
                    const double u1 = fma(-t1, y1[v], x1[v]), w1 = fma(t1, x1[v], y1[v]);
                    x0[v] = c0 * u0;
                    y0[v] = c0 * w0;
                    x1[v] = c1 * u1;
                    y1[v] = c1 * w1;
                }
                nx0 = fma(-t0, g0, nx0);
                ny0 = fma(t0, g0, ny0);
                nx1 = fma(-t1, g1, nx1);
                ny1 = fma(t1, g1, ny1);
                // bit 1: a rotation that was not small
                myrot |= (on0 ? (q0 > r0.small ? 3 : 1) : 0) | (on1 ? (q1 > r1.small ? 3 : 1) : 0);
            }
            if (p == 0 && act) {
                lg[0] = make_double2(c0, t0);
                lg[1] = make_double2(c1, t1);
            }
            lg += npair;
        };
        // a block to / from slot b (0 .. 2 G - 1) of a buffer
        auto put = [&](int buf, int b, const double(&x0)[NR], const double(&x1)[NR], double n0, double n1) {
            double2* w = xch + ((size_t)(buf * NBLK + b) * NR) * LP + p;
#pragma unroll
            for (int v = 0; v < NR; v++) w[v * LP] = make_double2(x0[v], x1[v]);
            if (p == 0) s_xn[buf][b] = make_double2(n0, n1);
        };
        auto take = [&](int buf, int b, double(&x0)[NR], double(&x1)[NR], double& n0, double& n1) {
            const double2* w = xch + ((size_t)(buf * NBLK + b) * NR) * LP + p;
#pragma unroll
            for (int v = 0; v < NR; v++) {
                const double2 t = w[v * LP];
                x0[v] = t.x;
                x1[v] = t.y;
            }
            const double2 t = s_xn[buf][b];
            n0 = t.x;
            n1 = t.y;
        };
        int buf = 0;
        auto next = [&]() {  // after a move's reads
            if (NBUF > 1)
                buf ^= 1;
            else
                sync();
        };
        if (ring) {
            for (int hb = G; hb >= 1; hb >>= 1) {
                const int i = grp & (hb - 1), up = grp - i + ((i + 1) & (hb - 1));
                for (int s = 0; s < hb; s++) {
                    step(A0, B0, a0, b0, A1, B1, a1, b1);
                    step(A0, B1, a0, b1, A1, B0, a1, b0);
                    if (hb == 1) continue;
                    // second blocks one group back along the ring (the last
                    // move of a level brings them home)
                    if (act) put(buf, grp, B0, B1, b0, b1);
                    sync();
                    if (act) take(buf, up, B0, B1, b0, b1);
                    next();
                }
                if (hb >= 2) {
                    // split: group i < h takes the first block of group i + h as
                    // its second, group i + h the second block of group i as its
                    // first (h = hb / 2)
                    const int h = hb >> 1;
                    if (act) {
                        if (i < h)
                            put(buf, grp, B0, B1, b0, b1);
                        else
                            put(buf, grp, A0, A1, a0, a1);
                    }
                    sync();
                    if (act) {
                        if (i < h)
                            take(buf, grp ^ h, B0, B1, b0, b1);
                        else
                            take(buf, grp ^ h, A0, A1, a0, a1);
                    }
                    next();
                }
            }
            step(A0, A1, a0, a1, B0, B1, b0, b1);
            // group g holds blocks 2g, 2g + 1 after the last level: back to g, G + g
            if (act) {
                put(buf, 2 * grp, A0, A1, a0, a1);
                put(buf, 2 * grp + 1, B0, B1, b0, b1);
            }
            sync();
            if (act) {
                take(buf, grp, A0, A1, a0, a1);
                take(buf, G + grp, B0, B1, b0, b1);
            }
        } else {
            // blocks to the next super-round's positions: group 0's first
            // block stays, the other first blocks go one group down (group
            // 1's becomes group 0's second), second blocks one group up (the
            // last group's becomes its own first).  Slot g: first block of
            // group g, slot G + g: second block.
            const int sa = grp == G - 1 ? G + grp : grp + 1, sb = grp > 0 ? G + grp - 1 : 1;
            for (int s = 0; s < ns; s++) {
                step(A0, B0, a0, b0, A1, B1, a1, b1);
                step(A0, B1, a0, b1, A1, B0, a1, b0);
                if (G == 1) break;
                if (act) {
                    if (grp > 0) put(buf, grp, A0, A1, a0, a1);
                    put(buf, G + grp, B0, B1, b0, b1);
                }
                sync();
                if (act) {
                    if (grp > 0) take(buf, sa, A0, A1, a0, a1);
                    take(buf, sb, B0, B1, b0, b1);
                }
                next();
            }
            step(A0, A1, a0, a1, B0, B1, b0, b1);
        }
        sync();  // the buffers are read before the next sweep (or the epilogue) writes them
        int any = __reduce_or_sync(FULL, myrot);
        if (NW > 1) {
            if (lane == 0 && any) atomicOr(&s_rot, any);
            __syncthreads();
            any = s_rot;
            __syncthreads();
            if (tid == 0) s_rot = 0;
        }
        if (any == 0) {
            conv = true;
        } else {
            sweeps = sw + 1;
            if (!(any & 2)) conv = true;  // the next one would only meet cosines ~1e-16
        }
    }
    if (!conv && tid == 0) PTT_STATUS_SET(status, PTT_ERR_NUMERIC);
    const double back = scalbn(1.0, sh);
    // singular values (column norms), the columns back to shared memory
    a0 = gsum(dot_rows(A0, A0));
    a1 = gsum(dot_rows(A1, A1));
    b0 = gsum(dot_rows(B0, B0));
    b1 = gsum(dot_rows(B1, B1));
    if (act) {
        auto store = [&](int slot, const double(&x)[NR]) {
            if (slot >= qa) return;
            double* col = Lc + s_perm[slot] * S;
#pragma unroll
            for (int v = 0; v < NR; v++) col[p + LP * v] = x[v];
        };
        store(ja, A0);
        store(ja + 1, A1);
        store(jb, B0);
        store(jb + 1, B1);
        if (p < 4) {  // lane p: one of the four columns
            const int slot = (p & 2 ? jb : ja) + (p & 1);
            const double s2 = p == 0 ? a0 : (p == 1 ? a1 : (p == 2 ? b0 : b1));
            if (slot < qa) s_nrm[s_perm[slot]] = s2;
        }
    }
    for (int j = warp; j < q; j += NW) {  // the columns that took no part
        if (s_slot[j] < 0)
            for (int t = lane; t < c; t += 32) Lc[j * S + t] = R[(long long)j * CT + t] * down;
    }
    __syncthreads();
    for (int j = tid; j < q; j += NTH) {
        const double s2 = s_nrm[j];
        // a NaN (corrupt input) would break the strict order below and leave
        // order slots unset; it sorts last and is reported instead
        const bool nan = !(s2 == s2);
        if (nan) PTT_STATUS_SET(status, PTT_ERR_NUMERIC);
        s_sig[j] = nan ? -1.0 : sqrt(s2) * (s_slot[j] < 0 ? 1.0 : back);
    }
    __syncthreads();
    for (int j = tid; j < q; j += NTH) {  // descending order
        const double sj = s_sig[j];
        int pos = 0;
#pragma unroll 4
        for (int i = 0; i < q; i++) {
            const double si = s_sig[i];
            pos += (si > sj) || (si == sj && i < j);
        }
        s_ord[pos] = j;
        s_srt[pos] = sj < 0.0 ? 0.0 / 0.0 : sj;  // a NaN stays one for the rank rule
    }
    __syncthreads();
    double* sig_out = ws + pl.o_sig;
    if (warp == 0) {
        const double s0 = q > 0 ? s_srt[0] : 0.0;
        // numerical rank kept by LAPACK dgesvdq(JOBA='A'): sqrt(N)*eps*s0
        const double thr = sqrt((double)q) * 1.1102230246251565e-16 * s0;
        int nsv = 0;  // leading run of values >= thr, at least one
        for (int j0 = 0; j0 < q; j0 += 32) {
            const unsigned lo = __ballot_sync(FULL, !(j0 + lane < q && s_srt[j0 + lane] >= thr));
            nsv = j0 + (lo ? __ffs(lo) - 1 : 32);
            if (lo) break;
        }
        nsv = nsv < 1 ? (q > 0 ? 1 : 0) : nsv;
        if (!(s0 == s0) && lane == 0) PTT_STATUS_SET(status, PTT_ERR_NUMERIC);
        // tail-sum rule, pattac.c:468-481: sums from the smallest kept value up,
        // then the largest index whose tail reaches delta
        if (lane == 0) {
            double ssum = 0.0;
#pragma unroll 8
            for (int j = nsv - 1; j >= 0; j--) {
                ssum = fma(s_srt[j], s_srt[j], ssum);
                s_suf[j] = ssum;
            }
        }
        __syncwarp();
        int rank = 0;
        double tail = 0.0;
        for (int j0 = 0; j0 < nsv; j0 += 32) {
            const unsigned hi = __ballot_sync(FULL, j0 + lane < nsv && !(sqrt(s_suf[j0 + lane]) < delta));
            if (hi) rank = j0 + 32 - __clz(hi);
        }
        if (rank > q) rank = q;
        if (rank > maxr) rank = maxr;
        if (rank < 1) rank = 1;
        for (int j = rank + lane; j < q; j += 32) tail += s_srt[j] * s_srt[j];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tail += __shfl_xor_sync(FULL, tail, o);
        if (lane == 0) {
            s_rank = rank;
            info->rank = rank;
            info->nsv = nsv;
            info->sweeps = sweeps;
            info->order = ring ? ORD_RING : ORD_CIRCLE;
            info->qa = qa;
            info->tail = tail;
            if (pl.stats) {
                double* st = pl.stats + (long long)bond * PTT_STAT_LEN;
                st[0] = rank;
                st[1] = nsv;
                st[2] = sweeps;
                st[3] = q;
                st[4] = c;
                st[5] = tail;
                st[6] = delta;
                st[7] = 0.0;
            }
        }
        if (pl.stats && lane < PTT_STAT_NSIG)
            pl.stats[(long long)bond * PTT_STAT_LEN + 8 + lane] = lane < q ? s_srt[lane] : 0.0;
    }
    for (int j = tid; j < CT; j += NTH) {
        sig_out[j] = j < q ? s_srt[j] : 0.0;
        int* ord = (int*)(sig_out + CT);
        ord[j] = j < q ? s_ord[j] : 0;
        ord[CT + j] = j < qa ? s_perm[j] : CT;  // slot of the rotation log -> column (CT: none)
    }
    __syncthreads();
    const int rank = s_rank;
    double* US = ws + pl.o_US;  // c x rank, column-major ld CT
    for (int b = warp; b < rank; b += NW) {
        const double* col = Lc + s_ord[b] * S;
        for (int t = lane; t < c; t += 32) US[(long long)b * CT + t] = col[t] * back;
    }
}
