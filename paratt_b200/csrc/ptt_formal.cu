// Formal TT arithmetic and mode-local operators (HBM-bound kernels).
//
//  axpby     attacFormalAXPBY   attac.c:81-112, wrapper paratt.c:237-268
//  hadamard  attacHadamard      attac.c:128-136 with attacKron utilities.c:112-129
//  square_sym  x (.) x at rank r(r+1)/2 (no reference counterpart; same tensor)
//  scale     attac_tt_scale     paratt.c:271-281
//  diag      attac_mult_diag_mat paratt.c:571-581
//  stencil   attac_apply_periodic_stencil paratt.c:584-661
//
// Every kernel reads ranks from the device descriptors, writes its result to
// the output's second buffer and the new ranks to a scratch array; a one-block
// finalize kernel then swaps the buffers and publishes the ranks.  This keeps
// the ops safe when the output aliases an input and free of host syncs.
#include "ptt_common.cuh"

#include <string.h>

#define PTT_MAX_STENCIL 15

struct Stencil {
    double s[PTT_MAX_STENCIL];
    int len;
};

// grid: (blocks, cores). One block per (slab chunk, core).
static inline int elem_blocks(long long maxcnt) {
    long long b = (maxcnt + 255) / 256;
    if (b > 2048) b = 2048;
    if (b < 1) b = 1;
    return (int)b;
}

// Blocks per core of an element-wise launch over all d cores (grid y =
// core): sized by the largest capacity, capped at a few waves over the
// device; the grid-stride loops cover any core with any grid.
static inline int core_blocks(const ptt_ctx* c, long long maxcnt, int d) {
    const int b = elem_blocks(maxcnt);
    const int cap = ptt_core_grid_cap(c, d);
    return b < cap ? b : cap;
}

// Fibers of a core: element (i, f) at i + R f, f = j + n l (the column-major
// core seen as R x (n R1)).  A group of G lanes (a power of two; 32 once
// R >= 32) takes one fiber at a time, so a fiber's rows are contiguous
// accesses of consecutive lanes and (j, l) cost one 32-bit division per
// fiber instead of 64-bit divisions per element.
struct FiberIter {
    int G, li;
    long long f0, fstep;
};
__device__ __forceinline__ FiberIter fiber_iter(int R) {
    FiberIter it;
    int G = 32;
    if (R < 32) {
        G = 1;
        while (G < R) G <<= 1;
    }
    const int lane = threadIdx.x & 31;
    const int per = 32 / G;
    it.G = G;
    it.li = lane & (G - 1);
    const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    it.f0 = warp * per + lane / G;
    it.fstep = nw * per;
    return it;
}

// Walk of a core by runs of JRUN consecutive fibers of one slab l, one warp
// per run: one division per run instead of one per fiber, and the next
// fiber's addresses by addition.  It pays for even ranks from 32 on, with runs
// enough to occupy the GPU (counted over the launch as if its d cores were
// alike).  The ranks are only known on the device, so a kernel that may walk by
// runs holds the walk fiber by fiber as well; it is launched where a core's
// capacities qualify, and its registers are held to 40 and 48 (six and five
// blocks an SM): with 56 and 64 every other rank of such a train lost up to 13 %.
constexpr int JRUN = 16;
__host__ __device__ __forceinline__ bool by_runs(int d, int n, int rows, int slabs, int least) {
    return (rows & 1) == 0 && rows >= 32 && (long long)((n + JRUN - 1) / JRUN) * slabs * d >= least;
}
struct RunIter {
    int t, step, runs, total;  // run t of `runs` per slab
};
__device__ __forceinline__ RunIter run_iter(int n, int slabs) {
    RunIter it;
    it.t = (int)(((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    it.step = (int)(((long long)gridDim.x * blockDim.x) >> 5);
    it.runs = (n + JRUN - 1) / JRUN;
    it.total = it.runs * slabs;
    return it;
}

// Blocks per core of a fiber launch over d cores (grid y = core): enough for
// the largest core's fibers at 8 per block (one per warp of 256 threads),
// capped at 32 blocks per SM over the whole grid.
static inline int fiber_blocks(const ptt_ctx* c, const ptt_tt* z, int d) {
    long long nf = 1;
    for (int k = 0; k < d; k++) {
        const long long f = (long long)z->n[k] * z->rcap[k + 1];
        nf = f > nf ? f : nf;
    }
    long long b = (nf + 7) / 8;
    const long long cap = ptt_core_grid_cap(c, d);
    if (b > cap) b = cap;
    return (int)(b < 1 ? 1 : b);
}

// ---------------------------------------------------------------------------
// finalize: publish ranks computed by a kernel and swap the written cores
// ---------------------------------------------------------------------------
__global__ void k_finalize(DevDesc* Z, const int* newr, int k0, int k1, int set_ranks) {
    int d = Z->d;
    for (int k = threadIdx.x; k <= d; k += blockDim.x)
        if (set_ranks) Z->r[k] = newr[k];
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) {
        double* a = Z->core[k];
        Z->core[k] = Z->alt[k];
        Z->alt[k] = a;
    }
}

static int finalize(ptt_tt* z, int* newr, int k0, int k1, int set_ranks) {
    k_finalize<<<1, 128, 0, z->ctx->stream>>>(z->dd, newr, k0, k1, set_ranks);
    PTT_LAUNCHED(z->ctx);
    return PTT_OK;
}

// new ranks of an op, published by the finalize kernel (512 doubles = 1024 ints)
static int* ranks_scratch(ptt_ctx* c, int d) {
    if (d + 1 <= 1024) return (int*)c->d_scalars;
    return NULL;
}

// ---------------------------------------------------------------------------
// axpby
// ---------------------------------------------------------------------------
__global__ void k_axpby(const DevDesc* X, const DevDesc* Y, DevDesc* Z, double a, double b, int* newr,
                        int* status) {
    const int k = blockIdx.y;
    const int d = X->d;
    const int rx = X->r[k], rx1 = X->r[k + 1], ry = Y->r[k], ry1 = Y->r[k + 1];
    const int n = X->n[k];
    int rz, rz1;
    if (d == 1) {
        rz = 1;
        rz1 = 1;
    } else {
        rz = (k == 0) ? 1 : rx + ry;
        rz1 = (k == d - 1) ? 1 : rx1 + ry1;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        newr[k] = rz;
        if (k == d - 1) newr[d] = 1;
    }
    const long long cnt = (long long)rz * n * rz1;
    if (rz > Z->rcap[k] || rz1 > Z->rcap[k + 1] || cnt > Z->cap[k]) {
        if (blockIdx.x == 0 && threadIdx.x == 0) PTT_STATUS_SET(status, PTT_ERR_CAPACITY);
        return;
    }
    const double* xc = X->core[k];
    const double* yc = Y->core[k];
    double* zc = Z->alt[k];
    if (d == 1) {
        const long long stride = (long long)gridDim.x * blockDim.x;
        for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt; e += stride)
            zc[e] = a * xc[e] + b * yc[e];
        return;
    }
    // fiber (j, l) of z: x's fiber over zeros (l < rx1), zeros over y's fiber
    // (l >= rx1); core 0 is [a x_0 | b y_0], the last core stacks x over y
    const int NF = n * rz1;
    const FiberIter it = fiber_iter(rz);
    for (long long f = it.f0; f < NF; f += it.fstep) {
        const int fi = (int)f, l = fi / n, j = fi - l * n;
        double* zf = zc + (long long)rz * fi;
        if (k == 0) {
            if (it.li == 0) zf[0] = (l < rx1) ? a * xc[j + (long long)n * l] : b * yc[j + (long long)n * (l - rx1)];
        } else if (k == d - 1) {
#pragma unroll 4
            for (int i = it.li; i < rz; i += it.G)
                zf[i] = (i < rx) ? xc[i + (long long)rx * j] : yc[(i - rx) + (long long)ry * j];
        } else if (l < rx1) {
            const double* src = xc + (long long)rx * (j + (long long)n * l);
#pragma unroll 4
            for (int i = it.li; i < rz; i += it.G) zf[i] = (i < rx) ? src[i] : 0.0;
        } else {
            const double* src = yc + (long long)ry * (j + (long long)n * (l - rx1));
#pragma unroll 4
            for (int i = it.li; i < rz; i += it.G) zf[i] = (i >= rx) ? src[i - rx] : 0.0;
        }
    }
}

// Make z's rank capacity cover an op's output.  need[] is the bound from the
// inputs' capacities; when z already covers it nothing happens (no sync).
// Otherwise the inputs' actual ranks are read back (synchronises) and z is
// grown only to the exact output ranks: op 0 = sum (r_x + r_y), 1 = product,
// 2 = operator sum (2 r_x; y unused), 3 = symmetric square (r_x (r_x + 1) / 2).
static int fit_output(ptt_tt* z, const int* need, const ptt_tt* x, const ptt_tt* y, int op) {
    const int d = z->d;
    int ok = 1;
    for (int k = 0; k <= d; k++) ok &= need[k] <= z->rcap[k];
    if (ok) return PTT_OK;
    int rx[PTT_MAX_DIM + 1], ry[PTT_MAX_DIM + 1], ex[PTT_MAX_DIM + 1];
    int rc;
    if ((rc = ptt_tt_get_ranks((ptt_tt*)x, rx))) return rc;
    if (op < 2 && (rc = ptt_tt_get_ranks((ptt_tt*)y, ry))) return rc;
    for (int k = 0; k <= d; k++) {
        if (op == 0)
            ex[k] = (k == 0 || k == d) ? 1 : rx[k] + ry[k];
        else if (op == 1)
            ex[k] = rx[k] * ry[k];
        else if (op == 3)
            ex[k] = rx[k] * (rx[k] + 1) / 2;
        else
            ex[k] = (k == 0 || k == d) ? 1 : 2 * rx[k];
        if (ex[k] < z->rcap[k]) ex[k] = z->rcap[k];
    }
    return ptt_tt_reserve(z, ex);
}

static int check_same_modes(const ptt_tt* x, const ptt_tt* y) {
    if (!x || !y || x->d != y->d) return ptt_set_error(PTT_ERR_ARG, "mode count mismatch");
    for (int k = 0; k < x->d; k++)
        if (x->n[k] != y->n[k]) return ptt_set_error(PTT_ERR_ARG, "mode %d size mismatch", k);
    return PTT_OK;
}

extern "C" int ptt_axpby(double a, const ptt_tt* x, double b, const ptt_tt* y, ptt_tt* z) {
    int rc = check_same_modes(x, y);
    if (rc || (rc = check_same_modes(x, z))) return rc;
    const int d = x->d;
    int need[PTT_MAX_DIM + 1];
    need[0] = need[d] = 1;
    for (int k = 1; k < d; k++) need[k] = x->rcap[k] + y->rcap[k];
    if ((rc = fit_output(z, need, x, y, 0))) return rc;
    ptt_ctx* c = z->ctx;
    int* newr = ranks_scratch(c, d);
    if (!newr) return ptt_set_error(PTT_ERR_ARG, "d too large");
    long long mx = 0;
    for (int k = 0; k < d; k++) mx = z->cap[k] > mx ? z->cap[k] : mx;
    (void)mx;
    k_axpby<<<dim3(fiber_blocks(c, z, d), d), 256, 0, c->stream>>>(x->dd, y->dd, z->dd, a, b, newr, c->d_status);
    PTT_LAUNCHED(c);
    return finalize(z, newr, 0, d, 1);
}

// ---------------------------------------------------------------------------
// hadamard: z_k[(ky + ry*ix), j, (ly + ry1*jx)] = x_k[ix, j, jx] * y_k[ky, j, ly]
// ---------------------------------------------------------------------------
// RUNS: a warp walks runs of fibers (j, lz), lz = ly + ry1 jx; lane: rows iz = 2
// lane + 64 b and the next, iz = ky + ry ix, so the row's factors are found once
// and every store is 16 bytes.  Bound by the writes (8 bytes per element; x and y
// come from L1/L2): d = 40, n = 256, ranks 8 x 8, 329 MB: 140 us with a division
// and an 8-byte store per element, 73 now (4.5 TB/s, 59 back to back).  With few
// runs it is slower: 10 modes of 17, ranks 8 x 16 (2560 runs) 20.6 us a product,
// 16.6 fiber by fiber; 20 modes of 100, ranks 4 x 8 (4480) 18.8 and 23.4.
constexpr int RUNS_HADAMARD = 4096;
template <bool RUNS>
__device__ __forceinline__ void hadamard_core(const DevDesc* X, const DevDesc* Y, DevDesc* Z, int* newr, int* status) {
    const int k = blockIdx.y;
    const int d = X->d;
    const int rx = X->r[k], rx1 = X->r[k + 1], ry = Y->r[k], ry1 = Y->r[k + 1];
    const int n = X->n[k];
    const int rz = rx * ry, rz1 = rx1 * ry1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        newr[k] = rz;
        if (k == d - 1) newr[d] = rz1;
    }
    const long long cnt = (long long)rz * n * rz1;
    if (rz > Z->rcap[k] || rz1 > Z->rcap[k + 1] || cnt > Z->cap[k]) {
        if (blockIdx.x == 0 && threadIdx.x == 0) PTT_STATUS_SET(status, PTT_ERR_CAPACITY);
        return;
    }
    const double* xc = X->core[k];
    const double* yc = Y->core[k];
    double* zc = Z->alt[k];
    if (RUNS && by_runs(d, n, rz, rz1, RUNS_HADAMARD)) {
        const RunIter it = run_iter(n, rz1);
        const int lane = threadIdx.x & 31;
        for (int b = 2 * lane; b < rz; b += 64) {
            const int i0 = b / ry, k0 = b - i0 * ry, i1 = (b + 1) / ry, k1 = (b + 1) - i1 * ry;
            for (int t = it.t; t < it.total; t += it.step) {
                const int lz = t / it.runs, j0 = (t - lz * it.runs) * JRUN, h = min(JRUN, n - j0);
                const int jx = lz / ry1, ly = lz - jx * ry1;
                const double* xf = xc + (long long)rx * (j0 + (long long)n * jx);
                const double* yf = yc + (long long)ry * (j0 + (long long)n * ly);
                double2* zf = (double2*)(zc + (long long)rz * (j0 + (long long)n * lz) + b);
#pragma unroll 2
                for (int j = 0; j < h; j++)
                    __stcs(zf + (long long)(rz / 2) * j, make_double2(xf[rx * j + i0] * yf[ry * j + k0],
                                                                      xf[rx * j + i1] * yf[ry * j + k1]));
            }
        }
        return;
    }
    // fiber (j, lz), lz = ly + ry1 jx: rows iz = ky + ry ix
    const int NF = n * rz1;
    const FiberIter it = fiber_iter(rz);
    for (long long f = it.f0; f < NF; f += it.fstep) {
        const int fi = (int)f, lz = fi / n, j = fi - lz * n;
        const int jx = lz / ry1, ly = lz - jx * ry1;
        const double* xf = xc + (long long)rx * (j + (long long)n * jx);
        const double* yf = yc + (long long)ry * (j + (long long)n * ly);
        double* zf = zc + (long long)rz * fi;
        for (int iz = it.li; iz < rz; iz += it.G) {
            const int ix = iz / ry, ky = iz - ix * ry;
            zf[iz] = xf[ix] * yf[ky];
        }
    }
}
__global__ void k_hadamard(const DevDesc* X, const DevDesc* Y, DevDesc* Z, int* newr, int* status) {
    hadamard_core<false>(X, Y, Z, newr, status);
}
__global__ void __launch_bounds__(256, 6) k_hadamard_runs(const DevDesc* X, const DevDesc* Y, DevDesc* Z, int* newr,
                                                          int* status) {
    hadamard_core<true>(X, Y, Z, newr, status);
}

extern "C" int ptt_hadamard(const ptt_tt* x, const ptt_tt* y, ptt_tt* z) {
    int rc = check_same_modes(x, y);
    if (rc || (rc = check_same_modes(x, z))) return rc;
    const int d = x->d;
    int need[PTT_MAX_DIM + 1];
    for (int k = 0; k <= d; k++) need[k] = x->rcap[k] * y->rcap[k];
    if ((rc = fit_output(z, need, x, y, 1))) return rc;
    ptt_ctx* c = z->ctx;
    int* newr = ranks_scratch(c, d);
    if (!newr) return ptt_set_error(PTT_ERR_ARG, "d too large");
    long long mx = 0;
    for (int k = 0; k < d; k++) mx = z->cap[k] > mx ? z->cap[k] : mx;
    (void)mx;
    bool runs = false;
    for (int k = 0; k < d; k++) runs = runs || by_runs(d, x->n[k], need[k], need[k + 1], RUNS_HADAMARD);
    auto kern = runs ? k_hadamard_runs : k_hadamard;
    kern<<<dim3(fiber_blocks(c, z, d), d), 256, 0, c->stream>>>(x->dd, y->dd, z->dd, newr, c->d_status);
    PTT_LAUNCHED(c);
    return finalize(z, newr, 0, d, 1);
}

// ---------------------------------------------------------------------------
// symmetric square: x (.) x restricted to the symmetric subspace.
// The formal core x_k (x) x_k (per mode index j) maps Sym^2(R^r) into
// Sym^2(R^r') and both interface vectors of x (.) x are symmetric, so with
// the orthonormal basis e_(a,a) and (e_(a,b) + e_(b,a))/sqrt2 (a < b) of
// Sym^2 the compressed core
//   z[s, j, s'] = (x[a,j,a'] x[b,j,b'] + x[a,j,b'] x[b,j,a']) f(s) f(s'),
//   f(s) = 1/sqrt2 if a == b else 1,
// gives exactly the same tensor at rank r (r + 1) / 2 instead of r^2.
// Pairs are packed s = b (b + 1) / 2 + a, a <= b.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void sym_pair(int s, int* a, int* b) {
    int bb = (int)((sqrt(8.0 * s + 1.0) - 1.0) * 0.5);
    while ((bb + 1) * (bb + 2) / 2 <= s) bb++;
    while (bb * (bb + 1) / 2 > s) bb--;
    *b = bb;
    *a = s - bb * (bb + 1) / 2;
}

__global__ void k_square_sym(const DevDesc* X, DevDesc* Z, int* newr, int* status) {
    const int k = blockIdx.y;
    const int d = X->d;
    const int rx = X->r[k], rx1 = X->r[k + 1];
    const int n = X->n[k];
    const int rz = rx * (rx + 1) / 2, rz1 = rx1 * (rx1 + 1) / 2;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        newr[k] = rz;
        if (k == d - 1) newr[d] = rz1;
    }
    const long long cnt = (long long)rz * n * rz1;
    if (rz > Z->rcap[k] || rz1 > Z->rcap[k + 1] || cnt > Z->cap[k]) {
        if (blockIdx.x == 0 && threadIdx.x == 0) PTT_STATUS_SET(status, PTT_ERR_CAPACITY);
        return;
    }
    const double* xc = X->core[k];
    double* zc = Z->alt[k];
    const long long rzn = (long long)rz * n;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const double h = 0.70710678118654752440;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt; e += stride) {
        const int sz1 = (int)(e / rzn);
        const long long rem = e - sz1 * rzn;
        const int j = (int)(rem / rz);
        const int sz = (int)(rem - (long long)j * rz);
        int a, b, a1, b1;
        sym_pair(sz, &a, &b);
        sym_pair(sz1, &a1, &b1);
        const double* xj = xc + (long long)rx * j;
        const long long ls = (long long)rx * n;
        const double v = xj[a + ls * a1] * xj[b + ls * b1] + xj[a + ls * b1] * xj[b + ls * a1];
        zc[e] = v * (a == b ? h : 1.0) * (a1 == b1 ? h : 1.0);
    }
}

extern "C" int ptt_square_sym(const ptt_tt* x, ptt_tt* z) {
    int rc = check_same_modes(x, z);
    if (rc) return rc;
    const int d = x->d;
    int need[PTT_MAX_DIM + 1];
    for (int k = 0; k <= d; k++) need[k] = x->rcap[k] * (x->rcap[k] + 1) / 2;
    if ((rc = fit_output(z, need, x, x, 3))) return rc;
    ptt_ctx* c = z->ctx;
    int* newr = ranks_scratch(c, d);
    if (!newr) return ptt_set_error(PTT_ERR_ARG, "d too large");
    long long mx = 0;
    for (int k = 0; k < d; k++) mx = z->cap[k] > mx ? z->cap[k] : mx;
    k_square_sym<<<dim3(core_blocks(c, mx, d), d), 256, 0, c->stream>>>(x->dd, z->dd, newr, c->d_status);
    PTT_LAUNCHED(c);
    return finalize(z, newr, 0, d, 1);
}

// ---------------------------------------------------------------------------
// scale core 0, diagonal multiply along one mode (in place)
// ---------------------------------------------------------------------------
__global__ void k_scale_core(DevDesc* X, int k, double a) {
    const long long cnt = (long long)X->r[k] * X->n[k] * X->r[k + 1];
    double* xc = X->core[k];
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt;
         e += (long long)gridDim.x * blockDim.x)
        xc[e] *= a;
}

extern "C" int ptt_scale(double a, ptt_tt* x) {
    if (!x) return ptt_set_error(PTT_ERR_ARG, "null tt");
    k_scale_core<<<elem_blocks(x->cap[0]), 256, 0, x->ctx->stream>>>(x->dd, 0, a);
    PTT_LAUNCHED(x->ctx);
    return PTT_OK;
}

__global__ void k_diag(DevDesc* X, int k, const double* vec) {
    const int r = X->r[k], n = X->n[k];
    const long long cnt = (long long)r * n * X->r[k + 1];
    double* xc = X->core[k];
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt;
         e += (long long)gridDim.x * blockDim.x) {
        const int j = (int)((e / r) % n);
        xc[e] *= vec[j];
    }
}

extern "C" int ptt_mult_diag(ptt_tt* x, int mode, const double* vec) {
    if (!x || !vec || mode < 0 || mode >= x->d) return ptt_set_error(PTT_ERR_ARG, "ptt_mult_diag: bad arguments");
    ptt_ctx* c = x->ctx;
    size_t bytes = sizeof(double) * x->n[mode];
    int rc = ptt_ws_reserve(c, bytes);
    if (rc) return rc;
    PTT_CUDA(cudaMemcpyAsync(c->ws, vec, bytes, cudaMemcpyHostToDevice, c->stream));
    k_diag<<<elem_blocks(x->cap[mode]), 256, 0, c->stream>>>(x->dd, mode, (const double*)c->ws);
    PTT_LAUNCHED(c);
    return PTT_OK;
}

// ---------------------------------------------------------------------------
// periodic centred stencil along one mode:
//   out[i, a, l] = sum_t s_t f[i, (a + t - h) mod n, l],  h = (len-1)/2
// Block = one (l) slab of r*n contiguous doubles; i fastest -> coalesced.
// ---------------------------------------------------------------------------
__global__ void k_stencil(DevDesc* X, int k, Stencil st) {
    const int r = X->r[k], n = X->n[k], r1 = X->r[k + 1];
    const int h = (st.len - 1) / 2;
    const double* in = X->core[k];
    double* out = X->alt[k];
    // fiber (a, l): out[:, a, l] = sum_t s_t in[:, (a + t - h) mod n, l]
    const int NF = n * r1;
    const FiberIter it = fiber_iter(r);
    for (long long f = it.f0; f < NF; f += it.fstep) {
        const int fi = (int)f, l = fi / n, a = fi - l * n;
        const double* fl = in + (long long)r * n * l;
        double* fo = out + (long long)r * fi;
        for (int i = it.li; i < r; i += it.G) {
            double acc = 0.0;
            for (int t = 0; t < st.len; t++) {
                int src = a + t - h;
                src = src < 0 ? src + n : (src >= n ? src - n : src);
                acc += st.s[t] * fl[i + (long long)r * src];
            }
            fo[i] = acc;
        }
    }
}

int ptt_make_stencil(const double* sten, int slen, Stencil* st) {
    if (slen % 2 == 0) slen -= 1;  // paratt.c:586: even lengths drop the last tap
    if (slen < 1 || slen > PTT_MAX_STENCIL) return ptt_set_error(PTT_ERR_ARG, "stencil length %d", slen);
    memset(st, 0, sizeof(*st));
    st->len = slen;
    for (int t = 0; t < slen; t++) st->s[t] = sten[t];
    return PTT_OK;
}

extern "C" int ptt_stencil(ptt_tt* x, int mode, const double* sten, int slen) {
    if (!x || !sten || mode < 0 || mode >= x->d) return ptt_set_error(PTT_ERR_ARG, "ptt_stencil: bad arguments");
    Stencil st;
    int rc = ptt_make_stencil(sten, slen, &st);
    if (rc) return rc;
    if ((st.len - 1) / 2 >= x->n[mode] && st.len > 1)
        return ptt_set_error(PTT_ERR_ARG, "stencil half-width exceeds mode size");
    ptt_ctx* c = x->ctx;
    long long bx = ((long long)x->n[mode] * x->rcap[mode + 1] + 7) / 8;  // 8 fibers per block
    if (bx > 8LL * c->nsm) bx = 8LL * c->nsm;
    if (bx < 1) bx = 1;
    k_stencil<<<dim3((unsigned)bx), 256, 0, c->stream>>>(x->dd, mode, st);
    PTT_LAUNCHED(c);
    k_finalize<<<1, 32, 0, c->stream>>>(x->dd, NULL, mode, mode + 1, 0);
    PTT_LAUNCHED(c);
    return PTT_OK;
}

// ---------------------------------------------------------------------------
// Y = sum_i S_i X + shift * X, S_i = the periodic stencil on mode i.
// Exact rank-2r TT (the formal sum of the d single-mode stencil applications,
// attac_apply_periodic_stencil paratt.c:584-661 summed with attacFormalSum,
// represents the same tensor at rank d*r).  Core k in 2x2 blocks indexed by
// (applied-before-k, applied-up-to-k): [[x_k, S x_k], [0, x_k]]; the first
// core keeps block row 0 with the shift added to S x_0, the last core keeps
// block column 1.  For d == 1: (S + shift) x_0.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double sten_at(const double* xc, int r, int n, int i, int j, int l, const Stencil& st) {
    const int h = (st.len - 1) / 2;
    double acc = 0.0;
    for (int t = 0; t < st.len; t++) {
        int s = j + t - h;
        s = s < 0 ? s + n : (s >= n ? s - n : s);
        acc += st.s[t] * xc[i + (long long)r * (s + (long long)n * l)];
    }
    return acc;
}

// RUNS, a middle core and three points: a warp walks runs of fibers (j, l') of x
// and writes both of y's fibers that come from each, [x; 0] and [S x; x]; the
// stencil slides along the run in registers, so every fiber of x is read once
// (plus two per run) and all accesses are 16 bytes.  Bound by HBM, four bytes
// written per byte read: d = 40, n = 256, r = 64, 1.59 GB: 499 us with 8-byte
// accesses, a division per fiber and the stencil's neighbours re-read, 267 now (6.0
// TB/s).  At 2000 runs both take as long (10 modes of 17, rank 100: 25.6 us an
// operator; fiber by fiber rank 96 takes 23.1); 40 modes of 32, rank 32 (2560)
// 21.5, and rank 31 27.0 fiber by fiber.
//   The stencil stays in the parameters (__grid_constant__): indexed through its
// address, a plain parameter was first copied to 128 bytes of local memory by
// every thread, 14 us of a launch of 4700 blocks.
constexpr int RUNS_OPSUM = 2000;
template <bool RUNS>
__device__ __forceinline__ void opsum_core(const DevDesc* X, DevDesc* Y, const Stencil& st, double shift, int* newr,
                                           int* status) {
    const int k = blockIdx.y;
    const int d = X->d;
    const int r = X->r[k], r1 = X->r[k + 1], n = X->n[k];
    const int ry = (d == 1 || k == 0) ? 1 : 2 * r;
    const int ry1 = (d == 1 || k == d - 1) ? 1 : 2 * r1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        newr[k] = ry;
        if (k == d - 1) newr[d] = 1;
    }
    const long long cnt = (long long)ry * n * ry1;
    if (ry > Y->rcap[k] || ry1 > Y->rcap[k + 1] || cnt > Y->cap[k]) {
        if (blockIdx.x == 0 && threadIdx.x == 0) PTT_STATUS_SET(status, PTT_ERR_CAPACITY);
        return;
    }
    const double* xc = X->core[k];
    double* yc = Y->alt[k];
    if (RUNS && k > 0 && k < d - 1 && st.len == 3 && by_runs(d, n, r, r1, RUNS_OPSUM)) {
        const RunIter it = run_iter(n, r1);
        const int lane = threadIdx.x & 31, r2 = r >> 1;
        const double s0 = st.s[0], s1 = st.s[1], s2 = st.s[2];
        for (int b = 2 * lane; b < r; b += 64) {
            for (int t = it.t; t < it.total; t += it.step) {
                const int l = t / it.runs, j0 = (t - l * it.runs) * JRUN, h = min(JRUN, n - j0);
                const double2* xs = (const double2*)(xc + (long long)r * n * l + b);  // fiber j at xs[j r / 2]
                double2* ya = (double2*)(yc + (long long)ry * (j0 + (long long)n * l) + b);
                double2* yb = ya + (long long)r * n * r1;  // the fiber l + r1
                double2 xm = __ldg(xs + (long long)r2 * (j0 > 0 ? j0 - 1 : n - 1)), x0 = __ldg(xs + (long long)r2 * j0);
#pragma unroll 4
                for (int j = 0; j < h; j++) {
                    const int jn = j0 + j + 1 < n ? j0 + j + 1 : 0;
                    const double2 xp = __ldg(xs + (long long)r2 * jn);
                    const double2 sx = make_double2(fma(s2, xp.x, fma(s1, x0.x, fma(s0, xm.x, 0.0))),
                                                    fma(s2, xp.y, fma(s1, x0.y, fma(s0, xm.y, 0.0))));
                    __stcs(ya + (long long)r * j, x0);
                    __stcs(ya + (long long)r * j + r2, make_double2(0.0, 0.0));
                    __stcs(yb + (long long)r * j, sx);
                    __stcs(yb + (long long)r * j + r2, x0);
                    xm = x0;
                    x0 = xp;
                }
            }
        }
        return;
    }
    // fiber (j, l) of y; l' = l - r1 for the second block column
    const int NF = n * ry1;
    const FiberIter it = fiber_iter(ry);
    for (long long f = it.f0; f < NF; f += it.fstep) {
        const int fi = (int)f, l = fi / n, j = fi - l * n;
        double* yf = yc + (long long)ry * fi;
        if (d == 1) {
            if (it.li == 0) yf[0] = sten_at(xc, 1, n, 0, j, 0, st) + shift * xc[j];
        } else if (k == 0) {
            if (it.li == 0)
                yf[0] = (l < r1) ? xc[j + (long long)n * l]
                                 : sten_at(xc, 1, n, 0, j, l - r1, st) + shift * xc[j + (long long)n * (l - r1)];
        } else if (k == d - 1) {
            for (int i = it.li; i < ry; i += it.G)
                yf[i] = (i < r) ? sten_at(xc, r, n, i, j, 0, st) : xc[(i - r) + (long long)r * j];
        } else if (l < r1) {
            const double* src = xc + (long long)r * (j + (long long)n * l);
#pragma unroll 4
            for (int i = it.li; i < ry; i += it.G) yf[i] = (i < r) ? src[i] : 0.0;
        } else {
            const int lp = l - r1;
            const double* src = xc + (long long)r * (j + (long long)n * lp);
            for (int i = it.li; i < ry; i += it.G) yf[i] = (i < r) ? sten_at(xc, r, n, i, j, lp, st) : src[i - r];
        }
    }
}
__global__ void k_opsum(const DevDesc* X, DevDesc* Y, const __grid_constant__ Stencil st, double shift, int* newr,
                        int* status) {
    opsum_core<false>(X, Y, st, shift, newr, status);
}
__global__ void __launch_bounds__(256, 5) k_opsum_runs(const DevDesc* X, DevDesc* Y, const __grid_constant__ Stencil st,
                                                       double shift, int* newr, int* status) {
    opsum_core<true>(X, Y, st, shift, newr, status);
}

extern "C" int ptt_op_sum(const ptt_tt* x, const double* sten, int slen, double shift, ptt_tt* y) {
    int rc = check_same_modes(x, y);
    if (rc) return rc;
    Stencil st;
    if ((rc = ptt_make_stencil(sten, slen, &st))) return rc;
    const int d = x->d;
    for (int k = 0; k < d; k++)
        if ((st.len - 1) / 2 >= x->n[k] && st.len > 1)
            return ptt_set_error(PTT_ERR_ARG, "stencil half-width exceeds mode %d size", k);
    int need[PTT_MAX_DIM + 1];
    for (int k = 0; k <= d; k++) need[k] = (k == 0 || k == d) ? 1 : 2 * x->rcap[k];
    if ((rc = fit_output(y, need, x, x, 2))) return rc;
    ptt_ctx* c = y->ctx;
    int* newr = ranks_scratch(c, d);
    long long mx = 0;
    for (int k = 0; k < d; k++) mx = y->cap[k] > mx ? y->cap[k] : mx;
    (void)mx;
    bool runs = false;
    for (int k = 1; k < d - 1 && st.len == 3; k++)
        runs = runs || by_runs(d, x->n[k], x->rcap[k], x->rcap[k + 1], RUNS_OPSUM);
    auto kern = runs ? k_opsum_runs : k_opsum;
    kern<<<dim3(fiber_blocks(c, y, d), d), 256, 0, c->stream>>>(x->dd, y->dd, st, shift, newr, c->d_status);
    PTT_LAUNCHED(c);
    return finalize(y, newr, 0, d, 1);
}
