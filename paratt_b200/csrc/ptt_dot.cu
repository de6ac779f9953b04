// Contractions: inner product, norm, single entry.
//
//  ptt_dot    paratt_dotprod (paratt.c:412-469) via transfer matrices as in
//             pattacInnerProduct (pattac.c:693-741); each step is divided by
//             n_k, which is the reference's 1/sqrt(n_k) scaling of both
//             arguments, so the result is <X, Y> / prod(n).
//  ptt_norm   paratt_norm (paratt.c:369-409) returns ||X||_F / sqrt(prod n);
//             computed here as sqrt(<X,X>/prod n) without touching the gauge
//             (the reference left-orthogonalises its argument in place).
//  ptt_entry  paratt_entry (paratt.c:471-499) -> pattacValue (pattac.c:82-121).
#include "ptt_common.cuh"

#include <mutex>

#include <string.h>

// T[i, j, e] = sum_k a[i, k] * y[k, j, e]      (a: rx x ry, column-major ld rx)
__global__ void k_dot_t(const DevDesc* X, const DevDesc* Y, int k, const double* a, double* T) {
    const int rx = X->r[k], ry = Y->r[k], n = X->n[k], ry1 = Y->r[k + 1];
    const long long cnt = (long long)rx * n * ry1;
    const double* y = Y->core[k];
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < cnt;
         e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e % rx);
        const long long je = e / rx;  // j + n*e'
        double acc = 0.0;
        for (int kk = 0; kk < ry; kk++) acc += a[i + (long long)rx * kk] * y[kk + (long long)ry * je];
        T[e] = acc;
    }
}

// a'[b, e] = (1/n) sum_{i,j} x[i, j, b] * T[i, j, e]; one block per (b, e).
__global__ void k_dot_a(const DevDesc* X, const DevDesc* Y, int k, const double* T, double* anew) {
    const int rx = X->r[k], n = X->n[k], rx1 = X->r[k + 1], ry1 = Y->r[k + 1];
    const int b = blockIdx.y, e = blockIdx.x;
    if (b >= rx1 || e >= ry1) return;
    const long long len = (long long)rx * n;
    const double* xb = X->core[k] + len * b;
    const double* te = T + len * e;
    double acc = 0.0;
    for (long long t = threadIdx.x; t < len; t += blockDim.x) acc += xb[t] * te[t];
    __shared__ double red[32];
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        double v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        v = warp_sum(v);
        if (threadIdx.x == 0) anew[b + (long long)rx1 * e] = v / (double)n;
    }
}

// Both contractions of a core in one kernel, for ranks up to DR: CTA p takes
// mode indices j = p, p + P, ...: T_j = a y_j (rx x ry1) and then its share of
// a'[b, e] += sum_i x_j[i, b] T_j[i, e], both on the FP64 tensor cores
// (mma.m8n8k4), T_j never leaving shared memory, the cores' slices x_j, y_j of
// the next j loaded (cp.async) during the products of this one.  The partial
// a' of the P CTAs are summed in order by k_dot_sum.
// One inner product needs 4 n r^3 operations and 16 n r^2 bytes per core: at r
// = 64 it is bound by the FP64 rate (7 us a core at n = 256), below r ~ 20 by
// latency.  d = 40, n = 256, r = 64: 116 us a core with one thread per element
// of T and one block per element of a' (each block re-reading T and x from
// L2), 19 us now.
constexpr int DR = 64, DP = DR + 4;  // rank bound; pitch: 4 mod 16 doubles, conflict-free fragments
constexpr int DNT = 256;
constexpr size_t DOT_SMEM = sizeof(double) * 6 * DR * DP;

__device__ __forceinline__ void dot_mma(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}
// slice j of a core (r x n x r1) to dst[l * DP + i]
__device__ __forceinline__ void dot_load(const double* core, int r, int n, int r1, int j, double* dst) {
    const unsigned d0 = (unsigned)__cvta_generic_to_shared(dst);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (((r & 1) | (int)((size_t)core & 15)) == 0) {  // every fiber starts on 16 bytes
        for (int l = warp; l < r1; l += DNT / 32) {
            const double* g = core + (long long)r * (j + (long long)n * l);
            for (int i = 2 * lane; i < r; i += 64)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d0 + 8u * (unsigned)(l * DP + i)), "l"(g + i)
                             : "memory");
        }
    } else {
        for (int l = warp; l < r1; l += DNT / 32) {
            const double* g = core + (long long)r * (j + (long long)n * l);
            for (int i = lane; i < r; i += 32)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d0 + 8u * (unsigned)(l * DP + i)), "l"(g + i)
                             : "memory");
        }
    }
}

__global__ void __launch_bounds__(DNT, 1) k_dot_part(const DevDesc* X, const DevDesc* Y, int k, const double* a, double* part,
                                                     int* status) {
    extern __shared__ __align__(16) double dsm[];
    double* As = dsm;                // a[i, kk] at kk * DP + i
    double* Ts = As + DR * DP;       // T[i, e] at i * DP + e
    double* XY = Ts + DR * DP;       // two buffers of x_j[i, b] at b * DP + i, y_j[kk, e] at e * DP + kk
    const int rx = X->r[k], ry = Y->r[k], n = X->n[k], rx1 = X->r[k + 1], ry1 = Y->r[k + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, li = lane >> 2, lk = lane & 3;
    if (rx > DR || ry > DR || rx1 > DR || ry1 > DR) {  // uniform; the host checks the capacities
        if (blockIdx.x == 0 && tid == 0) PTT_STATUS_SET(status, PTT_ERR_CAPACITY);
        return;
    }
    const double *xc = X->core[k], *yc = Y->core[k];
    if ((rx | ry | rx1 | ry1) & 7) {  // zero padding up to whole tiles (the loads leave it alone)
        const int mx = max(max(rx, ry), max(rx1, ry1)), r8 = (mx + 7) & ~7;
        for (int e = tid; e < 6 * r8 * (r8 / 2); e += DNT) {
            const int row = e / (r8 / 2), col = 2 * (e - row * (r8 / 2)), arr = row / r8;
            *(double2*)(dsm + (arr * DR + row - arr * r8) * DP + col) = make_double2(0.0, 0.0);
        }
        __syncthreads();
    }
    int j = blockIdx.x, buf = 0;
    if (j < n) {
        dot_load(xc, rx, n, rx1, j, XY);
        dot_load(yc, ry, n, ry1, j, XY + DR * DP);
    }
    // only a comes from the kernel before: the trains were complete before the
    // chain's first kernel started, so their first slices are requested while
    // that kernel finishes
    PTT_PDL_ENTRY();
    dot_load(a, rx, 1, ry, 0, As);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    double d0[8], d1[8];  // rows 8 warp .. of a', all columns
#pragma unroll
    for (int t = 0; t < 8; t++) d0[t] = d1[t] = 0.0;
    const int nb1 = (ry1 + 7) >> 3;
    for (; j < n; j += gridDim.x, buf ^= 1) {
        const int jn = j + gridDim.x;
        double* Xs = XY + buf * 2 * DR * DP;
        double* Ys = Xs + DR * DP;
        if (jn < n) {
            double* nx = XY + (buf ^ 1) * 2 * DR * DP;
            dot_load(xc, rx, n, rx1, jn, nx);
            dot_load(yc, ry, n, ry1, jn, nx + DR * DP);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();  // this j's slices (and a) are in place, the last j's T is read
        if (8 * warp < rx) {
            double c0[8], c1[8];
#pragma unroll
            for (int t = 0; t < 8; t++) c0[t] = c1[t] = 0.0;
            for (int k4 = 0; k4 < ry; k4 += 4) {
                const double av = As[(k4 + lk) * DP + 8 * warp + li];
#pragma unroll
                for (int t = 0; t < 8; t++)
                    if (t < nb1) dot_mma(c0[t], c1[t], av, Ys[(8 * t + li) * DP + k4 + lk]);
            }
#pragma unroll
            for (int t = 0; t < 8; t++) {
                // rows past rx: zero, not the padding's 0 x y_j (NaN where y_j is not finite), which the
                // second product would carry into a'
                if (t < nb1)
                    *(double2*)(Ts + (8 * warp + li) * DP + 8 * t + 2 * lk) =
                        8 * warp + li < rx ? make_double2(c0[t], c1[t]) : make_double2(0.0, 0.0);
            }
        }
        __syncthreads();
        if (8 * warp < rx1) {
            for (int k4 = 0; k4 < rx; k4 += 4) {
                const double av = Xs[(8 * warp + li) * DP + k4 + lk];
#pragma unroll
                for (int t = 0; t < 8; t++)
                    if (t < nb1) dot_mma(d0[t], d1[t], av, Ts[(k4 + lk) * DP + 8 * t + li]);
            }
        }
        __syncthreads();  // the buffer of this j is free for the load after next
    }
    double* out = part + (long long)blockIdx.x * rx1 * ry1;
    const int b = 8 * warp + li;
    if (b < rx1) {
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int e = 8 * t + 2 * lk;
            if (e < ry1) out[b + (long long)rx1 * e] = d0[t];
            if (e + 1 < ry1) out[b + (long long)rx1 * (e + 1)] = d1[t];
        }
    }
}

// a'[u] = (1/n) sum_p part[p][u]: eight eighths of the partials per entry,
// each in order, the eighths in order
__global__ void __launch_bounds__(DNT) k_dot_sum(const DevDesc* X, const DevDesc* Y, int k, const double* part, int P,
                                                 double* anew) {
    PTT_PDL_ENTRY();
    __shared__ double red[DNT];
    const int cnt = X->r[k + 1] * Y->r[k + 1];
    const int tid = threadIdx.x, q = tid >> 5, u = blockIdx.x * 32 + (tid & 31);
    if (blockIdx.x * 32 >= cnt) return;
    double acc = 0.0;
    if (u < cnt) {
        const double* s = part + u;
        int p = P * q / 8;
        const int p1 = P * (q + 1) / 8;
        for (; p < p1; p += 10) {
            double v[10];
#pragma unroll
            for (int t = 0; t < 10; t++) v[t] = p + t < p1 ? s[(long long)(p + t) * cnt] : 0.0;
#pragma unroll
            for (int t = 0; t < 10; t++) acc += v[t];
        }
    }
    red[tid] = acc;
    __syncthreads();
    if (tid < 32 && u < cnt) {
        double a = red[tid];
#pragma unroll
        for (int t = 1; t < 8; t++) a += red[32 * t + tid];
        anew[u] = a / (double)X->n[k];
    }
}

// The transfer matrices through all cores: a0 holds 1 on entry; returns the
// buffer of the result.  rx, ry bound the ranks; t holds tcap doubles, at
// least rx_k n_k ry_{k+1} for every core.
static int dot_chain(ptt_ctx* c, const ptt_tt* x, const ptt_tt* y, const int* rx, const int* ry, double* a0, double* a1,
                     double* t, long long tcap, double** res) {
    int rmax = 1;
    for (int k = 0; k <= x->d; k++) {
        rmax = rx[k] > rmax ? rx[k] : rmax;
        rmax = ry[k] > rmax ? ry[k] : rmax;
    }
    if (rmax <= DR) {
        static std::atomic<unsigned long long> attr{0};
        unsigned long long bit;
        if (!ptt_device_done(attr, &bit)) {
            PTT_CUDA(cudaFuncSetAttribute(k_dot_part, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DOT_SMEM));
            attr.fetch_or(bit);
        }
    }
    for (int k = 0; k < x->d; k++) {
        const long long tc = (long long)rx[k] * x->n[k] * ry[k + 1], ac = (long long)rx[k + 1] * ry[k + 1];
        if (rmax <= DR) {
            // partials of the CTAs in t: as many as it holds
            long long P = x->n[k] < c->nsm ? x->n[k] : c->nsm;
            if (P * ac > tcap) P = tcap / ac;
            if (P < 1) P = 1;
            PTT_CUDA(ptt_launch(c, k_dot_part, dim3((unsigned)P), dim3(DNT), DOT_SMEM, x->dd, y->dd, k, a0, t, c->d_status));
            PTT_LAUNCHED(c);
            PTT_CUDA(ptt_launch(c, k_dot_sum, dim3((unsigned)((ac + 31) / 32)), dim3(DNT), 0, x->dd, y->dd, k, t, (int)P, a1));
            PTT_LAUNCHED(c);
        } else {
            int bx = (int)((tc + 255) / 256);
            if (bx > 4096) bx = 4096;
            k_dot_t<<<bx, 256, 0, c->stream>>>(x->dd, y->dd, k, a0, t);
            PTT_LAUNCHED(c);
            k_dot_a<<<dim3(ry[k + 1], rx[k + 1]), 256, 0, c->stream>>>(x->dd, y->dd, k, t, a1);
            PTT_LAUNCHED(c);
        }
        double* s = a0;
        a0 = a1;
        a1 = s;
    }
    *res = a0;
    return PTT_OK;
}

// The start of a chain of products, to be launched without the programmatic
// attribute: k_dot_part reads the trains before its wait, which is only safe
// behind a launch that waited for everything before it.
__global__ void k_set_one(double* a) { a[0] = 1.0; }

extern "C" int ptt_dot(const ptt_tt* x, const ptt_tt* y, double* out) {
    if (!x || !y || !out || x->d != y->d) return ptt_set_error(PTT_ERR_ARG, "ptt_dot: bad arguments");
    for (int k = 0; k < x->d; k++)
        if (x->n[k] != y->n[k]) return ptt_set_error(PTT_ERR_ARG, "ptt_dot: mode %d differs", k);
    ptt_ctx* c = x->ctx;
    if (y->ctx != c) {
        PTT_CUDA(cudaEventRecord(y->ctx->ev_fork, y->ctx->stream));
        PTT_CUDA(cudaStreamWaitEvent(c->stream, y->ctx->ev_fork, 0));
    }
    // The ranks decide, not the capacities: a state of rank 7 in buffers for 128
    // takes the fused kernel, and the value does not depend on the buffers.  They
    // are read back (two small copies, one wait) only where a capacity leaves it
    // open.
    int rx[PTT_MAX_DIM + 1], ry[PTT_MAX_DIM + 1], rc;
    bool known = true;
    for (int k = 0; k <= x->d; k++) {
        rx[k] = x->rcap[k];
        ry[k] = y->rcap[k];
        known = known && rx[k] <= DR && ry[k] <= DR;
    }
    if (!known) {
        const size_t bytes = sizeof(int) * (size_t)(x->d + 1);
        int* h = (int*)c->h_scalars;  // 512 doubles
        PTT_CUDA(cudaMemcpyAsync(h, x->dd->r, bytes, cudaMemcpyDeviceToHost, c->stream));
        PTT_CUDA(cudaMemcpyAsync(h + PTT_MAX_DIM + 1, y->dd->r, bytes, cudaMemcpyDeviceToHost, c->stream));
        PTT_CUDA(cudaStreamSynchronize(c->stream));
        memcpy(rx, h, bytes);
        memcpy(ry, h + PTT_MAX_DIM + 1, bytes);
    }
    long long amax = 1, tmax = 1;
    for (int k = 0; k <= x->d; k++) amax = (long long)rx[k] * ry[k] > amax ? (long long)rx[k] * ry[k] : amax;
    for (int k = 0; k < x->d; k++) {
        long long t = (long long)rx[k] * x->n[k] * ry[k + 1];
        tmax = t > tmax ? t : tmax;
    }
    if (amax <= DR * DR && tmax < c->nsm * amax) tmax = c->nsm * amax;  // room for every CTA's partial
    size_t bytes = sizeof(double) * (size_t)(2 * amax + tmax) + 1024;
    if ((rc = ptt_ws_reserve(c, bytes))) return rc;
    double* A0 = (double*)c->ws;
    double* A1 = A0 + amax;
    double* T = A1 + amax;
    k_set_one<<<1, 1, 0, c->stream>>>(A0);
    PTT_LAUNCHED(c);
    if ((rc = dot_chain(c, x, y, rx, ry, A0, A1, T, tmax, &A0))) return rc;
    PTT_CUDA(cudaMemcpyAsync(c->h_scalars, A0, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    rc = ptt_ctx_synchronize(c);
    if (rc) return rc;
    *out = c->h_scalars[0];
    return PTT_OK;
}

extern "C" int ptt_norm(const ptt_tt* x, double* out) {
    double v = 0.0;
    int rc = ptt_dot(x, x, &v);
    if (rc) return rc;
    *out = sqrt(v > 0.0 ? v : 0.0);
    return PTT_OK;
}

// v <- v * core[k][:, idx, :]  (one block; v has r_k entries)
__global__ void k_entry_step(const DevDesc* X, int k, int idx, const double* vin, double* vout) {
    const int r = X->r[k], n = X->n[k], r1 = X->r[k + 1];
    const double* ck = X->core[k];
    for (int l = threadIdx.x; l < r1; l += blockDim.x) {
        double acc = 0.0;
        for (int i = 0; i < r; i++) acc += vin[i] * ck[i + (long long)r * (idx + (long long)n * l)];
        vout[l] = acc;
    }
}

extern "C" int ptt_entry(const ptt_tt* x, const int* idx, double* out) {
    if (!x || !idx || !out) return ptt_set_error(PTT_ERR_ARG, "ptt_entry: bad arguments");
    for (int k = 0; k < x->d; k++)
        if (idx[k] < 0 || idx[k] >= x->n[k]) return ptt_set_error(PTT_ERR_ARG, "ptt_entry: index %d out of range", k);
    ptt_ctx* c = x->ctx;
    int rmax = 1;
    for (int k = 0; k <= x->d; k++) rmax = x->rcap[k] > rmax ? x->rcap[k] : rmax;
    int rc = ptt_ws_reserve(c, sizeof(double) * 2 * (size_t)rmax + 256);
    if (rc) return rc;
    double* v0 = (double*)c->ws;
    double* v1 = v0 + rmax;
    k_set_one<<<1, 1, 0, c->stream>>>(v0);
    PTT_LAUNCHED(c);
    for (int k = 0; k < x->d; k++) {
        k_entry_step<<<1, 128, 0, c->stream>>>(x->dd, k, idx[k], v0, v1);
        PTT_LAUNCHED(c);
        double* s = v0;
        v0 = v1;
        v1 = s;
    }
    PTT_CUDA(cudaMemcpyAsync(c->h_scalars, v0, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    rc = ptt_ctx_synchronize(c);
    if (rc) return rc;
    *out = c->h_scalars[0];
    return PTT_OK;
}

// ---------------------------------------------------------------------------
// ptt_dot_noalloc: the same inner product with no device allocation.
//
// Some callers cannot let a library call cudaMalloc: a host framework that
// has already reserved the GPU's memory for its own pool, a latency-bound
// loop where cudaMalloc's implicit device-wide synchronisation would stall
// work on other streams, or an embedding that forbids allocation after
// start-up.  This variant keeps its scratch (two transfer matrices and the
// partial contraction T) in a fixed file-scope device array instead of the
// context workspace.  The array is PTT_DOT_NOALLOC_MAX_DOUBLES doubles
// (4 MiB) and exists on every GPU that loads the library until the process
// exits.  Requests that do not fit are rejected with PTT_ERR_CAPACITY.
//
// The array is shared by every call: it keeps the last call's contents, and
// nothing in it has to start at zero (the start value of the transfer matrix
// is written by a kernel of each call).  Two calls whose kernels overlap on
// the GPU (different streams or contexts on one device) race on it.
//
// Host code cannot use the array's name as a device address, so its address
// is looked up once per device (cudaGetSymbolAddress, with that device
// current).  ptt_ctx_create does that lookup for its device, which also loads
// this module (and so reserves the array) while the context is created:
// create the context before handing the GPU's memory to another allocator.
// A call on a device whose address is not known yet (not possible through
// ptt_ctx_create) looks it up itself, so make the first call before any
// stream capture.  The lookup restores the caller's current device and is
// serialised by a mutex, so threads making their first calls at once agree.
// ---------------------------------------------------------------------------
static __device__ __align__(256) double g_dot_scratch[PTT_DOT_NOALLOC_MAX_DOUBLES];

#define PTT_NOALLOC_MAX_DEVICES 64
static std::atomic<double*> g_dot_scratch_addr[PTT_NOALLOC_MAX_DEVICES];
static std::mutex g_dot_scratch_mu;

int ptt_dot_scratch_init(int device, double** out) {
    if (device < 0 || device >= PTT_NOALLOC_MAX_DEVICES)
        return ptt_set_error(PTT_ERR_ARG, "ptt_dot_noalloc: device %d out of range", device);
    double* a = g_dot_scratch_addr[device].load(std::memory_order_acquire);
    if (!a) {
        std::lock_guard<std::mutex> lock(g_dot_scratch_mu);
        a = g_dot_scratch_addr[device].load(std::memory_order_acquire);
        if (!a) {
            int prev = 0;
            PTT_CUDA(cudaGetDevice(&prev));
            void* p = NULL;
            cudaError_t e = cudaSetDevice(device);
            if (e == cudaSuccess) e = cudaGetSymbolAddress(&p, g_dot_scratch);
            const cudaError_t e2 = cudaSetDevice(prev);  // the caller's device, whatever happened
            if (e != cudaSuccess) return ptt_cuda_check(e, "cudaGetSymbolAddress(g_dot_scratch)");
            if (e2 != cudaSuccess) return ptt_cuda_check(e2, "cudaSetDevice (restore)");
            a = (double*)p;
            g_dot_scratch_addr[device].store(a, std::memory_order_release);
        }
    }
    if (out) *out = a;
    return PTT_OK;
}

extern "C" int ptt_dot_noalloc(const ptt_tt* x, const ptt_tt* y, double* out) {
    if (!x || !y || !out || x->d != y->d) return ptt_set_error(PTT_ERR_ARG, "ptt_dot_noalloc: bad arguments");
    for (int k = 0; k < x->d; k++)
        if (x->n[k] != y->n[k]) return ptt_set_error(PTT_ERR_ARG, "ptt_dot_noalloc: mode %d differs", k);
    ptt_ctx* c = x->ctx;
    if (y->ctx != c) {
        PTT_CUDA(cudaEventRecord(y->ctx->ev_fork, y->ctx->stream));
        PTT_CUDA(cudaStreamWaitEvent(c->stream, y->ctx->ev_fork, 0));
    }
    double* scratch = NULL;
    int rc = ptt_dot_scratch_init(c->device, &scratch);
    if (rc) return rc;
    // size the scratch from the actual ranks (reading them synchronises)
    int rx[PTT_MAX_DIM + 1], ry[PTT_MAX_DIM + 1];
    if ((rc = ptt_tt_get_ranks((ptt_tt*)x, rx)) || (rc = ptt_tt_get_ranks((ptt_tt*)y, ry))) return rc;
    long long amax = 1, tmax = 1;
    for (int k = 0; k <= x->d; k++) amax = (long long)rx[k] * ry[k] > amax ? (long long)rx[k] * ry[k] : amax;
    for (int k = 0; k < x->d; k++) {
        const long long t = (long long)rx[k] * x->n[k] * ry[k + 1];
        tmax = t > tmax ? t : tmax;
    }
    if (2 * amax + tmax > PTT_DOT_NOALLOC_MAX_DOUBLES)
        return ptt_set_error(PTT_ERR_CAPACITY,
                             "ptt_dot_noalloc: needs %lld doubles of scratch, the fixed array holds %d "
                             "(use ptt_dot, which allocates)",
                             2 * amax + tmax, (int)PTT_DOT_NOALLOC_MAX_DOUBLES);
    double* A0 = scratch;
    double* A1 = A0 + amax;
    double* T = A1 + amax;
    k_set_one<<<1, 1, 0, c->stream>>>(A0);
    PTT_LAUNCHED(c);
    // all the array has left: as many partials as ptt_dot takes, so the same sums (148 SMs x 64 x 64 would be more)
    if ((rc = dot_chain(c, x, y, rx, ry, A0, A1, T, PTT_DOT_NOALLOC_MAX_DOUBLES - 2 * amax, &A0))) return rc;
    PTT_CUDA(cudaMemcpyAsync(c->h_scalars, A0, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    rc = ptt_ctx_synchronize(c);
    if (rc) return rc;
    *out = c->h_scalars[0];
    return PTT_OK;
}
