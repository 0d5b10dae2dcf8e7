// FP64 CSR sparse matrix-vector product for the circuit simulator, with the matrix resident on the
// device, and a Jacobi-preconditioned BiCGSTAB built on it.
//
// Role in the reference: nangila-spice/nangila-node/cuda/cusparse_solver.cu:17-123 (a cuSPARSE SpMV
// behind four C calls: init / load_matrix / spmv / free, with the vectors copied over PCIe on every
// call). Here the product is a hand-written kernel and the vectors can stay on the device.
//
// Two designs. Matrices of short rows only (ladders and meshes) take one thread per row: spmv_short_rows_kernel, where the rule
// stands. All others take "row blocks", as do arrays that the caller owns (nangila_spmv_launch) and matrices loaded under
// NANGILA_SPMV_PLAIN=1: at load time the host packs consecutive rows into blocks of at most
// kCap non-zeros. A CTA streams its block's values and column indices with coalesced loads, gathers
// x through the read-only path, parks the products in shared memory and then reduces each row from
// there with 1..32 lanes per row (chosen from the block's mean row length), so that rows of a few
// entries cost no idle lanes and long rows still reduce in parallel. A row
// longer than kCap gets a block of its own and a CTA-wide strided reduction.
//
// Row blocks have two variants of the staging step. The context-owned matrix (nangila_spmv_load) is stored padded
// to a multiple of four entries, so a CTA fetches its slice of `val` and `col` with two
// cp.async.bulk copies completing on an mbarrier: the copy engine keeps 24 KB per CTA in flight
// without spending registers or issue slots, where the plain-load variant was bound by load latency
// (long-scoreboard stalls at 41 % of DRAM throughput; tridiagonal, before those took the other design.
// Nine diagonals, 10^6 rows: 51 us, plain loads 53, blocks of 1024 entries 47). A further variant that also staged the
// block's window of x in shared memory was measured and dropped: 41 KB and 48 registers per CTA cut
// residency from 8 to 5 CTAs per SM and the 16 M-row product went from 0.199 ms to 0.254 ms; with
// one copy per CTA the overlap comes from resident CTAs, so residency matters more than the
// gathers. Arrays owned by the caller
// (nangila_spmv_launch) carry no padding guarantee and use the plain-load variant.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>
#include <new>
#include <vector>

#include "bicgstab.cuh"
#include "nangila_spice_kernels.h"
#include "ptx_sm100.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kCap = 2048;  // products staged per CTA: 16 KB of shared memory

__global__ void __launch_bounds__(kThreads) spmv_row_blocks_kernel(const int* __restrict__ row_ptr, const int* __restrict__ col,
                                                                    const double* __restrict__ val, const double* __restrict__ x,
                                                                    double* __restrict__ y, const int* __restrict__ row_blocks) {
    __shared__ double prod[kCap];
    __shared__ double warp_sums[kThreads / 32];
    const int tid = threadIdx.x;
    const int r0 = row_blocks[blockIdx.x], r1 = row_blocks[blockIdx.x + 1];
    const int k0 = row_ptr[r0], k1 = row_ptr[r1];
    const int nnz = k1 - k0, nrows = r1 - r0;
    if (nnz <= kCap) {
        // stage products; four independent loads per thread in flight
        int k = tid;
        for (; k + 3 * kThreads < nnz; k += 4 * kThreads) {
            int c0 = __ldg(col + k0 + k), c1 = __ldg(col + k0 + k + kThreads), c2 = __ldg(col + k0 + k + 2 * kThreads),
                c3 = __ldg(col + k0 + k + 3 * kThreads);
            double v0 = __ldg(val + k0 + k), v1 = __ldg(val + k0 + k + kThreads), v2 = __ldg(val + k0 + k + 2 * kThreads),
                   v3 = __ldg(val + k0 + k + 3 * kThreads);
            prod[k] = v0 * __ldg(x + c0);
            prod[k + kThreads] = v1 * __ldg(x + c1);
            prod[k + 2 * kThreads] = v2 * __ldg(x + c2);
            prod[k + 3 * kThreads] = v3 * __ldg(x + c3);
        }
        for (; k < nnz; k += kThreads) prod[k] = __ldg(val + k0 + k) * __ldg(x + __ldg(col + k0 + k));
        __syncthreads();
        // lanes per row: largest power of two not above the mean row length, 1..32
        int mean = nrows > 0 ? nnz / nrows : 1;
        int lanes = 1;
        while (lanes < 32 && lanes * 2 <= mean) lanes *= 2;
        const int group = tid / lanes, lane = tid % lanes, groups = kThreads / lanes;
        // every lane of a warp runs the same number of iterations, so the shuffles below are uniform
        const int iters = (nrows + groups - 1) / groups;
        for (int it = 0; it < iters; ++it) {
            const int r = r0 + it * groups + group;
            double acc = 0.0;
            if (r < r1) {
                const int s = __ldg(row_ptr + r) - k0, e = __ldg(row_ptr + r + 1) - k0;
                for (int j = s + lane; j < e; j += lanes) acc += prod[j];
            }
            for (int off = lanes >> 1; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off, lanes);
            if (lane == 0 && r < r1) y[r] = acc;
        }
    } else {
        // one long row (the builder never mixes a long row with others)
        double acc = 0.0;
        for (int k = tid; k < nnz; k += kThreads) acc += __ldg(val + k0 + k) * __ldg(x + __ldg(col + k0 + k));
        for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
        if ((tid & 31) == 0) warp_sums[tid >> 5] = acc;
        __syncthreads();
        if (tid == 0) {
            double s = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) s += warp_sums[w];
            y[r0] = s;
        }
    }
}

// Bulk-copy variant: `val` and `col` must be readable up to the next multiple of four entries past
// the end of every block (the context pads its arrays). status[0] is set to 1 when a copy did not
// land within the time limit; the CTA then leaves its rows unwritten.
template <int T, int CAP>
__global__ void __launch_bounds__(T) spmv_row_blocks_bulk_kernel(const int* __restrict__ row_ptr, const int* __restrict__ col,
                                                                         const double* __restrict__ val, const double* __restrict__ x,
                                                                         double* __restrict__ y, const int* __restrict__ row_blocks,
                                                                         int* __restrict__ status, unsigned long long timeout_ns) {
    __shared__ __align__(16) double s_val[CAP + 8];
    __shared__ __align__(16) int s_col[CAP + 8];
    __shared__ __align__(8) uint64_t bar;
    __shared__ double warp_sums[T / 32];
    const int tid = threadIdx.x;
    const int r0 = row_blocks[blockIdx.x], r1 = row_blocks[blockIdx.x + 1];
    const int k0 = row_ptr[r0], k1 = row_ptr[r1];
    const int nnz = k1 - k0, nrows = r1 - r0;
    if (nnz <= CAP) {
        const int ka = k0 & ~3, kb = (k1 + 3) & ~3;  // 16-byte aligned in both arrays
        const int cnt = kb - ka, off = k0 - ka;
        if (tid == 0) {
            nangila::sm100::mbar_init(&bar, 1);
            nangila::sm100::fence_barrier_init();
        }
        __syncthreads();
        if (tid == 0 && cnt > 0) {
            nangila::sm100::mbar_arrive_expect_tx(&bar, uint32_t(cnt) * 12u);
            nangila::sm100::bulk_load(s_val, val + ka, uint32_t(cnt) * 8u, &bar);
            nangila::sm100::bulk_load(s_col, col + ka, uint32_t(cnt) * 4u, &bar);
        }
        if (cnt > 0 && !nangila::sm100::mbar_wait(&bar, 0, timeout_ns)) {
            if (tid == 0) atomicExch(status, 1);
            // the copies still target this CTA's shared memory: give them one more bounded wait
            nangila::sm100::mbar_wait(&bar, 0, timeout_ns);
            return;
        }
        int k = tid;
        for (; k + 3 * T < nnz; k += 4 * T) {
            const int j = off + k;
            double x0 = __ldg(x + s_col[j]), x1 = __ldg(x + s_col[j + T]), x2 = __ldg(x + s_col[j + 2 * T]),
                   x3 = __ldg(x + s_col[j + 3 * T]);
            s_val[j] *= x0;
            s_val[j + T] *= x1;
            s_val[j + 2 * T] *= x2;
            s_val[j + 3 * T] *= x3;
        }
        for (; k < nnz; k += T) s_val[off + k] *= __ldg(x + s_col[off + k]);
        __syncthreads();
        const double* prod = s_val + off;
        int mean = nrows > 0 ? nnz / nrows : 1;
        int lanes = 1;
        while (lanes < 32 && lanes * 2 <= mean) lanes *= 2;
        const int group = tid / lanes, lane = tid % lanes, groups = T / lanes;
        const int iters = (nrows + groups - 1) / groups;
        for (int it = 0; it < iters; ++it) {
            const int r = r0 + it * groups + group;
            double acc = 0.0;
            if (r < r1) {
                const int s = __ldg(row_ptr + r) - k0, e = __ldg(row_ptr + r + 1) - k0;
                for (int j = s + lane; j < e; j += lanes) acc += prod[j];
            }
            for (int o = lanes >> 1; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o, lanes);
            if (lane == 0 && r < r1) y[r] = acc;
        }
    } else {
        double acc = 0.0;
        for (int k = tid; k < nnz; k += T) acc += __ldg(val + k0 + k) * __ldg(x + __ldg(col + k0 + k));
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        if ((tid & 31) == 0) warp_sums[tid >> 5] = acc;
        __syncthreads();
        if (tid == 0) {
            double t = 0.0;
            for (int w = 0; w < T / 32; ++w) t += warp_sums[w];
            y[r0] = t;
        }
    }
}

// Short rows: one thread per row, no staging, no barrier. Four entries of the row are in flight at once; a warp's loads of one
// entry are strided by the row length, but the lines they touch are the ones its next entries need, so L1 serves them.
// Bound by HBM where the matrix does not fit L2, by the chain row_ptr -> col -> x otherwise; the staged kernel adds to that chain
// the block table, a barrier initialisation, a copy of the slice and two block barriers, and gives a CTA so much of the matrix that a
// ladder of 10^6 rows is 1.2 waves of CTAs. Products are rounded and added in the staged kernel's order for two and four lanes a row, so
// that ladders and meshes keep their bits. Measured on B200, staged kernel and this one, repeated products (10^6 rows lie in L2, 4 10^6 do not):
// ladder of 10^6 rows 24 -> 14 us, of 4 10^6 59 -> 41 us (5.5 TB/s); mesh of 10^6 nodes 35 -> 19, of 4 10^6 100 -> 56 us. With nothing in L2:
// rows of 1, 3, 5, 6 entries near the diagonal, 10^6 rows: 23 -> 16, 39 -> 23, 52 -> 35, 55 -> 39 us; anywhere: 31 -> 17, 56 -> 28, 77 -> 39, 83 -> 45.
// While the row pointers are on their way, a thread of each CTA has L2 fetch what the CTA would need if all rows were of the same length (`mean`): whole
// lines in one bulk prefetch, which every CTA's neighbours want soon if the guess is off. The columns alone, since these are what x waits for, or all of it.
// us without it / as chosen, in captured products: matrices in turn, and one again and again:
//   columns: ladder of 10^6 rows (55 MB)   12.0 / 11.3,  5.9 / 6.1     mesh of 10^6 (79 MB)     18.3 / 17.6,  11.6 / 11.6
//   all:     ladder of 4 10^6 (223 MB)     38.4 / 34.3,  38.1 / 33.9   mesh of 4 10^6 (319 MB)  59.4 / 54.7,  59.4 / 51.2
// So all of it where the matrix is larger than L2; the columns where a product may find it there or not (all of it there: 10.3, 7.0 and 17.0, 12.5 for the
// first line); nothing below 40 MB, where there is hardly anything to gain. (A prefetch by every row's thread for its own entries cost a product that
// finds its matrix in L2 more and gained less elsewhere: 11.3, 6.8 and 17.3, 11.8; 36.9, 36.1 and 60.0, 59.2.)
//
// The rule: no row above 16 entries, and at most 6 on average. Uneven rows cost a warp the time of its longest; at the corner of the rule
// (rows of 1 and of 16, mean 6) what is left is 43.5 -> 41.4 us near the diagonal and 150 -> 142 for 4 10^6 rows, so longer rows and higher means
// stay with the staged kernel; within it this kernel was the faster one for means 1 to 6, even and uneven, 10^4 to 4 10^6 rows.
constexpr int kShortRow = 16;
constexpr int kShortMean = 6;
enum Ahead { kNothing, kColumns, kAll };
constexpr int64_t kColumnsAhead = 40000000, kAllAhead = 126 << 20;  // bytes of matrix and vectors
template <Ahead AHEAD>
__global__ void __launch_bounds__(kThreads) spmv_short_rows_kernel(const int* __restrict__ row_ptr, const int* __restrict__ col,
                                                                   const double* __restrict__ val, const double* __restrict__ x,
                                                                   double* __restrict__ y, int n, int nnz, float mean) {
    const int r = int(blockIdx.x * unsigned(kThreads) + threadIdx.x);
    if (unsigned(r) >= unsigned(n)) return;
    if (AHEAD != kNothing && threadIdx.x == 0) {
        const int rows = min(kThreads, n - r);
        const int64_t from = int64_t(float(r) * mean), to = int64_t(float(r + rows) * mean);
        auto fetch = [](const void* first, const void* last) {  // whole 16-byte units between the two
            const uint64_t a = (reinterpret_cast<uint64_t>(first) + 15) & ~uint64_t(15), z = reinterpret_cast<uint64_t>(last) & ~uint64_t(15);
            if (a < z) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(uint32_t(z - a)) : "memory");
        };
        const int64_t f = min(from, int64_t(nnz)), t = min(to, int64_t(nnz));
        fetch(col + f, col + t);
        if (AHEAD == kAll) {
            fetch(val + f, val + t);
            fetch(x + r, x + r + rows);
        }
    }
    if (AHEAD != kNothing) __syncwarp();  // before the warp's loads: behind them it gains nothing
    const int s = __ldg(row_ptr + r), e = __ldg(row_ptr + r + 1);
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int j = s; j < e; j += 4) {
        int c[4];
        double v[4], g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            c[u] = j + u < e ? __ldg(col + j + u) : -1;
            v[u] = j + u < e ? __ldg(val + j + u) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) g[u] = c[u] >= 0 ? __ldg(x + c[u]) : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c[u] >= 0) acc[u] = __dadd_rn(acc[u], __dmul_rn(v[u], g[u]));
    }
    y[r] = (acc[0] + acc[2]) + (acc[1] + acc[3]);
}

// ---- vector kernels of the Krylov solver -------------------------------------------------------

constexpr int kRedBlocks = 296;  // two CTAs per SM

// partial[2 * b + {0, 1}] = sum over the CTA's slice of a1*b1 and a2*b2 (a2 may be null)
__global__ void __launch_bounds__(kThreads) dot2_partial_kernel(const double* __restrict__ a1, const double* __restrict__ b1,
                                                                 const double* __restrict__ a2, const double* __restrict__ b2, int n,
                                                                 double* __restrict__ partial) {
    __shared__ double s1[kThreads / 32], s2[kThreads / 32];
    double p = 0.0, q = 0.0;
    for (int i = blockIdx.x * kThreads + threadIdx.x; i < n; i += gridDim.x * kThreads) {
        p += a1[i] * b1[i];
        if (a2) q += a2[i] * b2[i];
    }
    for (int off = 16; off > 0; off >>= 1) { p += __shfl_down_sync(0xffffffffu, p, off); q += __shfl_down_sync(0xffffffffu, q, off); }
    if ((threadIdx.x & 31) == 0) { s1[threadIdx.x >> 5] = p; s2[threadIdx.x >> 5] = q; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t1 = 0.0, t2 = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) { t1 += s1[w]; t2 += s2[w]; }
        partial[2 * blockIdx.x] = t1;
        partial[2 * blockIdx.x + 1] = t2;
    }
}

// fixed-order sum of the partials: the same inputs give the same bits on every run
__global__ void dot2_final_kernel(const double* __restrict__ partial, int blocks, double* __restrict__ out) {
    if (threadIdx.x < 2) {
        double s = 0.0;
        for (int b = 0; b < blocks; ++b) s += partial[2 * b + threadIdx.x];
        out[threadIdx.x] = s;
    }
}

// p = r + beta (p - omega v);  ph = p / diag
__global__ void update_p_kernel(double* p, double* ph, const double* r, const double* v, const double* inv_diag, double beta,
                                double omega, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { double t = r[i] + beta * (p[i] - omega * v[i]); p[i] = t; ph[i] = t * inv_diag[i]; }
}
// s = r - alpha v;  sh = s / diag
__global__ void update_s_kernel(double* s, double* sh, const double* r, const double* v, const double* inv_diag, double alpha, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { double t = r[i] - alpha * v[i]; s[i] = t; sh[i] = t * inv_diag[i]; }
}
// x += alpha ph + omega sh;  r = s - omega t
__global__ void update_xr_kernel(double* x, double* r, const double* ph, const double* sh, const double* s, const double* t, double alpha,
                                 double omega, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { x[i] += alpha * ph[i] + omega * sh[i]; r[i] = s[i] - omega * t[i]; }
}
__global__ void residual_init_kernel(double* r, double* r0, const double* b, const double* ax, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { double t = b[i] - ax[i]; r[i] = t; r0[i] = t; }
}

}  // namespace

struct NangilaSpmv {
    int n = 0, nnz = 0, n_blocks = 0;
    int *d_row_ptr = nullptr, *d_col = nullptr, *d_blocks = nullptr;
    double *d_val = nullptr, *d_x = nullptr, *d_y = nullptr;
    int* d_status = nullptr;  // set by a kernel whose bulk copy timed out
    bool plain_loads = false;  // NANGILA_SPMV_PLAIN=1: use the plain-load kernel
    bool short_rows = false;   // every row suits one thread: spmv_short_rows_kernel
    Ahead ahead = kNothing;    // what it fetches ahead
    int cap = kCap;            // non-zeros per staged row block: 2048 (256 threads) or 1024 (128 threads, NANGILA_SPMV_TILE=1024)
    double* d_work = nullptr;   // solver vectors (kWorkVectors), allocated on first solve
    double* d_partial = nullptr;  // partial sums, then results and counter of the solver kernel
    std::vector<double> h_inv_diag;
    bool inv_diag_on_device = false;  // d_work holds h_inv_diag
    cudaStream_t solve_stream = nullptr;
    // the solver kernel's split of the rows: see bicgstab.cuh
    int ctas = 0, max_rows = 0, max_entries = 0;
    bool resident = false;
    double* d_scaled = nullptr;  // the solver's scaled values where they do not fit into shared memory
    int* d_plan = nullptr;  // first_row [ctas + 1], first_long [ctas + 1], long_rows
    std::vector<int> h_row_ptr, h_diag_slot;  // kept on the host to refresh the preconditioner when values change
};

// Jacobi preconditioner: 1 / diagonal where the diagonal carries weight in its row (at least 1e-3 of
// the row's largest entry), else 1 / that largest entry (branch-current rows of an MNA matrix have a
// zero or tiny diagonal).
static void refresh_preconditioner(NangilaSpmv* c, const double* val) {
    const int n = c->n;
    c->inv_diag_on_device = false;
    c->h_inv_diag.assign(size_t(n), 1.0);
    for (int r = 0; r < n; ++r) {
        double mx = 0.0;
        for (int k = c->h_row_ptr[size_t(r)]; k < c->h_row_ptr[size_t(r) + 1]; ++k) mx = fmax(mx, fabs(val[k]));
        const int d = c->h_diag_slot[size_t(r)];
        if (d >= 0 && fabs(val[d]) >= 1e-3 * mx && fabs(val[d]) > 1e-300) c->h_inv_diag[size_t(r)] = 1.0 / val[d];
        else if (mx > 1e-300) c->h_inv_diag[size_t(r)] = 1.0 / mx;
    }
}

static void free_arrays(NangilaSpmv* c) {
    cudaFree(c->d_row_ptr); cudaFree(c->d_col); cudaFree(c->d_blocks); cudaFree(c->d_val); cudaFree(c->d_x); cudaFree(c->d_y);
    cudaFree(c->d_work); cudaFree(c->d_partial); cudaFree(c->d_status); cudaFree(c->d_plan);
    cudaFree(c->d_scaled);
    if (c->solve_stream) cudaStreamDestroy(c->solve_stream);
    c->solve_stream = nullptr;
    c->d_plan = nullptr;
    c->d_scaled = nullptr;
    c->inv_diag_on_device = false;
    c->d_status = nullptr;
    c->d_row_ptr = c->d_col = c->d_blocks = nullptr;
    c->d_val = c->d_x = c->d_y = c->d_work = c->d_partial = nullptr;
}

// The matrix is uploaded on the legacy stream, where a copy from pageable memory may return before it has reached the device and a
// memset before it has run; solve_stream, and products on streams of the caller's, do not wait for that stream by themselves.
static cudaError_t uploads_landed() { return cudaStreamSynchronize(cudaStreamLegacy); }

static int build_row_blocks(const int* row_ptr, int n, int cap, int* out, int max_out);

extern "C" int nangila_spmv_build_row_blocks(const int* row_ptr, int n, int* out, int max_out) {
    return build_row_blocks(row_ptr, n, kCap, out, max_out);
}

static int build_row_blocks(const int* row_ptr, int n, int cap, int* out, int max_out) {
    // out[0] = 0, out[b + 1] = first row after block b; returns the number of blocks (or the number
    // needed when out is null / too small)
    int count = 0, r = 0;
    auto emit = [&](int v) { if (out && count + 1 < max_out) out[count + 1] = v; ++count; };
    if (out && max_out > 0) out[0] = 0;
    while (r < n) {
        int start = r;
        int base = row_ptr[r];
        if (row_ptr[r + 1] - base > cap) { ++r; emit(r); continue; }
        while (r < n && row_ptr[r + 1] - base <= cap) ++r;
        if (r == start) ++r;
        emit(r);
    }
    return count;
}

extern "C" NangilaSpmv* nangila_spmv_create(void) { return new (std::nothrow) NangilaSpmv(); }

extern "C" void nangila_spmv_destroy(NangilaSpmv* c) {
    if (!c) return;
    free_arrays(c);
    delete c;
}

extern "C" int nangila_spmv_load(NangilaSpmv* c, int n, int nnz, const int* row_ptr, const int* col, const double* val) {
    if (!c || n <= 0 || nnz < 0 || !row_ptr || !col || !val) return int(cudaErrorInvalidValue);
    if (row_ptr[0] != 0 || row_ptr[n] != nnz) return int(cudaErrorInvalidValue);
    for (int r = 0; r < n; ++r) if (row_ptr[r + 1] < row_ptr[r]) return int(cudaErrorInvalidValue);
    for (int k = 0; k < nnz; ++k) if (col[k] < 0 || col[k] >= n) return int(cudaErrorInvalidValue);
    free_arrays(c);
    c->n = n; c->nnz = nnz;
    {
        const char* tile = getenv("NANGILA_SPMV_TILE");
        c->cap = (tile && atoi(tile) == 1024) ? 1024 : kCap;
    }
    int nb = build_row_blocks(row_ptr, n, c->cap, nullptr, 0);
    std::vector<int> blocks(size_t(nb) + 1);
    build_row_blocks(row_ptr, n, c->cap, blocks.data(), nb + 1);
    c->n_blocks = nb;
    c->h_row_ptr.assign(row_ptr, row_ptr + n + 1);
    {
        int longest = 0;
        for (int r = 0; r < n; ++r) longest = std::max(longest, row_ptr[r + 1] - row_ptr[r]);
        c->short_rows = longest <= kShortRow && nnz <= int64_t(kShortMean) * n;
        const int64_t bytes = 12 * int64_t(nnz) + 20 * int64_t(n);
        c->ahead = bytes > kAllAhead ? kAll : bytes > kColumnsAhead ? kColumns : kNothing;
    }
    c->h_diag_slot.assign(size_t(n), -1);
    for (int r = 0; r < n; ++r)
        for (int k = row_ptr[r]; k < row_ptr[r + 1]; ++k)
            if (col[k] == r) c->h_diag_slot[size_t(r)] = k;
    refresh_preconditioner(c, val);
    cudaError_t e;
#define NG_TRY(call) do { e = (call); if (e != cudaSuccess) { free_arrays(c); return int(e); } } while (0)
    NG_TRY(cudaMalloc(&c->d_row_ptr, sizeof(int) * (size_t(n) + 1)));
    // padded so that a block's slice can be fetched in whole 16-byte units
    const size_t padded = (size_t(nnz) + 3) / 4 * 4 + 4;
    NG_TRY(cudaMalloc(&c->d_col, sizeof(int) * padded));
    NG_TRY(cudaMalloc(&c->d_val, sizeof(double) * padded));
    NG_TRY(cudaMemset(c->d_col, 0, sizeof(int) * padded));
    NG_TRY(cudaMemset(c->d_val, 0, sizeof(double) * padded));
    NG_TRY(cudaMalloc(&c->d_status, sizeof(int)));
    NG_TRY(cudaMemset(c->d_status, 0, sizeof(int)));
    {
        const char* env = getenv("NANGILA_SPMV_PLAIN");
        c->plain_loads = env && env[0] == '1';
    }
    NG_TRY(cudaMalloc(&c->d_blocks, sizeof(int) * (size_t(nb) + 1)));
    NG_TRY(cudaMalloc(&c->d_x, sizeof(double) * size_t(n)));
    NG_TRY(cudaMalloc(&c->d_y, sizeof(double) * size_t(n)));
    NG_TRY(cudaMemcpy(c->d_row_ptr, row_ptr, sizeof(int) * (size_t(n) + 1), cudaMemcpyHostToDevice));
    NG_TRY(cudaMemcpy(c->d_col, col, sizeof(int) * size_t(nnz), cudaMemcpyHostToDevice));
    NG_TRY(cudaMemcpy(c->d_val, val, sizeof(double) * size_t(nnz), cudaMemcpyHostToDevice));
    NG_TRY(cudaMemcpy(c->d_blocks, blocks.data(), sizeof(int) * (size_t(nb) + 1), cudaMemcpyHostToDevice));
    NG_TRY(uploads_landed());
    return 0;
}

extern "C" int nangila_spmv_update_values(NangilaSpmv* c, const double* val) {
    if (!c || !c->d_val || !val) return int(cudaErrorInvalidValue);
    refresh_preconditioner(c, val);
    const cudaError_t e = cudaMemcpy(c->d_val, val, sizeof(double) * size_t(c->nnz), cudaMemcpyHostToDevice);
    return int(e != cudaSuccess ? e : uploads_landed());
}

extern "C" int nangila_spmv_launch(const int* d_row_ptr, const int* d_col, const double* d_val, const double* d_x, double* d_y,
                                   const int* d_row_blocks, int n_blocks, cudaStream_t stream) {
    if (n_blocks <= 0) return 0;
    spmv_row_blocks_kernel<<<n_blocks, kThreads, 0, stream>>>(d_row_ptr, d_col, d_val, d_x, d_y, d_row_blocks);
    return int(cudaGetLastError());
}

extern "C" int nangila_spmv_device(NangilaSpmv* c, const double* d_x, double* d_y, cudaStream_t stream) {
    if (!c || !c->d_val || !d_x || !d_y) return int(cudaErrorInvalidValue);
    if (c->plain_loads) return nangila_spmv_launch(c->d_row_ptr, c->d_col, c->d_val, d_x, d_y, c->d_blocks, c->n_blocks, stream);
    if (c->n_blocks <= 0) return 0;
    if (c->short_rows) {
        auto* kernel = c->ahead == kAll ? spmv_short_rows_kernel<kAll> : c->ahead == kColumns ? spmv_short_rows_kernel<kColumns> : spmv_short_rows_kernel<kNothing>;
        kernel<<<unsigned((int64_t(c->n) + kThreads - 1) / kThreads), kThreads, 0, stream>>>(c->d_row_ptr, c->d_col, c->d_val, d_x, d_y, c->n, c->nnz,
                                                                                           float(c->nnz) / float(c->n));
        return int(cudaGetLastError());
    }
    if (c->cap == 1024)
        spmv_row_blocks_bulk_kernel<128, 1024><<<c->n_blocks, 128, 0, stream>>>(c->d_row_ptr, c->d_col, c->d_val, d_x, d_y, c->d_blocks,
                                                                               c->d_status, 2000000000ull);
    else
        spmv_row_blocks_bulk_kernel<kThreads, kCap><<<c->n_blocks, kThreads, 0, stream>>>(c->d_row_ptr, c->d_col, c->d_val, d_x, d_y,
                                                                                         c->d_blocks, c->d_status, 2000000000ull);
    return int(cudaGetLastError());
}

extern "C" int nangila_spmv_host(NangilaSpmv* c, const double* h_x, double* h_y) {
    if (!c || !c->d_val || !h_x || !h_y) return int(cudaErrorInvalidValue);
    cudaError_t e = cudaMemcpy(c->d_x, h_x, sizeof(double) * size_t(c->n), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return int(e);
    int rc = nangila_spmv_device(c, c->d_x, c->d_y, 0);
    if (rc) return rc;
    cudaError_t e2 = cudaMemcpy(h_y, c->d_y, sizeof(double) * size_t(c->n), cudaMemcpyDeviceToHost);
    if (e2 != cudaSuccess) return int(e2);
    return nangila_spmv_status(c);
}

extern "C" int nangila_spmv_status(NangilaSpmv* c) {
    if (!c || !c->d_status) return int(cudaErrorInvalidValue);
    int st = 0;
    cudaError_t e = cudaMemcpy(&st, c->d_status, sizeof(int), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return int(e);
    return st ? int(cudaErrorTimeout) : 0;
}

extern "C" int nangila_spmv_dims(const NangilaSpmv* c, int* n, int* nnz, int* n_blocks) {
    if (!c) return int(cudaErrorInvalidValue);
    if (n) *n = c->n;
    if (nnz) *nnz = c->nnz;
    if (n_blocks) *n_blocks = c->n_blocks;
    return 0;
}

// ---- BiCGSTAB ---------------------------------------------------------------------------------------
constexpr int kWorkVectors = 11;  // inverse diagonal, right-hand side, then nine that either form of the solver uses as it needs

// Splits the rows over the CTAs of the solver kernel: contiguous ranges of about equal cost (an entry counts one, a row
// three more for its vector work).
static cudaError_t plan_solver(NangilaSpmv* c) {
    using namespace nangila::krylov;
    int dev = 0, sms = 0, smem_max = 0;
    cudaError_t e;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    const int n = c->n;
    const int ctas = c->nnz <= kOneCta ? 1 : std::min({sms, kMaxCtas, c->nnz / kEntriesPerCta});
    std::vector<int> first_row(size_t(ctas) + 1, n), first_long(size_t(ctas) + 1, 0), long_rows;
    const double total = double(c->nnz) + 3.0 * n;
    int row = 0, max_rows = 0, max_entries = 0;
    first_row[0] = 0;
    for (int b = 0; b < ctas; ++b) {
        const int begin = row;
        first_long[size_t(b)] = int(long_rows.size());
        const double until = total * (b + 1) / ctas;
        while (row < n && (b == ctas - 1 || double(c->h_row_ptr[size_t(row)]) + 3.0 * row < until)) {
            if (c->h_row_ptr[size_t(row) + 1] - c->h_row_ptr[size_t(row)] > kLongRow) long_rows.push_back(row);
            ++row;
        }
        first_row[size_t(b) + 1] = row;
        max_rows = std::max(max_rows, row - begin);
        max_entries = std::max(max_entries, c->h_row_ptr[size_t(row)] - c->h_row_ptr[size_t(begin)]);
    }
    first_long[size_t(ctas)] = int(long_rows.size());
    std::vector<int> plan(first_row);
    plan.insert(plan.end(), first_long.begin(), first_long.end());
    plan.insert(plan.end(), long_rows.begin(), long_rows.end());
    if ((e = cudaMalloc(&c->d_plan, sizeof(int) * plan.size())) != cudaSuccess) return e;
    if ((e = cudaMemcpy(c->d_plan, plan.data(), sizeof(int) * plan.size(), cudaMemcpyHostToDevice)) != cudaSuccess) return e;
    if ((e = uploads_landed()) != cudaSuccess) return e;
    c->ctas = ctas;
    c->max_rows = max_rows;
    c->max_entries = max_entries;
    const size_t room = size_t(smem_max) - 4096;  // the kernel's static shared memory, and what the runtime keeps
    c->resident = solver_smem(true, max_rows, max_entries) <= room;
    if (!c->resident) return cudaSuccess;
    return cudaFuncSetAttribute(bicgstab_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(room));
}

// The solver kernel: one launch for the whole solve (bicgstab.cuh).
static int solve_on_device(NangilaSpmv* c, double* h_x, double tol, int max_iter, int* iterations, double* rel_residual) {
    using namespace nangila::krylov;
    const size_t N = size_t(c->n), S = (N + 1) & ~size_t(1);
    cudaStream_t st = c->solve_stream;
    double* w = c->d_work + 2 * S;
    const size_t sums = 2 * kSlot * size_t(c->ctas);
    SolverArgs a;
    a.row_ptr = c->d_row_ptr; a.col = c->d_col; a.val = c->d_val;
    a.first_row = c->d_plan; a.first_long = c->d_plan + c->ctas + 1; a.long_rows = c->d_plan + 2 * (c->ctas + 1);
    a.inv_diag = c->d_work; a.b = c->d_work + S;
    a.status = c->d_status;
    a.parts = reinterpret_cast<Parts*>(w); a.rv = reinterpret_cast<double2*>(w + 4 * S);
    a.x = w + 6 * S; a.r0 = w + 7 * S; a.p = w + 8 * S;
    a.scaled = c->d_scaled;
    a.partial = c->d_partial;
    a.out = c->d_partial + sums;
    a.arrived = reinterpret_cast<uint32_t*>(a.out + 4);
    a.max_iter = max_iter; a.max_entries = c->max_entries;
    a.tol = tol;
    a.timeout_ns = 2000000000ull;
    cudaError_t e;
    if ((e = cudaMemsetAsync(a.out, 0, 5 * sizeof(double), st)) != cudaSuccess) return int(e);
    void* args[] = {&a};
    const void* fn = c->resident ? reinterpret_cast<const void*>(&bicgstab_kernel<true>) : reinterpret_cast<const void*>(&bicgstab_kernel<false>);
    e = cudaLaunchCooperativeKernel(fn, dim3(unsigned(c->ctas)), dim3(unsigned(solver_threads(c->resident))), args, solver_smem(c->resident, c->max_rows, c->max_entries), st);
    if (e != cudaSuccess) return int(e);
    double out[4];
    if ((e = cudaMemcpyAsync(out, a.out, sizeof out, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return int(e);
    if ((e = cudaMemcpyAsync(h_x, a.x, sizeof(double) * N, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return int(e);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return int(e);
    const double rel = sqrt(out[0]) / out[1];
    if (iterations) *iterations = int(out[2]);
    if (rel_residual) *rel_residual = rel;
    if (out[3] != 0.0) return int(cudaErrorTimeout);
    return rel < tol ? 0 : -1;
}

// Solves A x = b (x starts at 0) with vectors resident on the device: one kernel for the whole solve, which tests the
// residual every fourth iteration. NANGILA_SPMV_GRAPH=0: per iteration two SpMVs, three fused vector kernels and four 16-byte reads
// of reduction results by the host, the residual tested after every one.
extern "C" int nangila_spmv_bicgstab(NangilaSpmv* c, const double* h_b, double* h_x, double tol, int max_iter, int* iterations,
                                     double* rel_residual) {
    if (!c || !c->d_val || !h_b || !h_x) return int(cudaErrorInvalidValue);
    const int n = c->n;
    const size_t N = size_t(n);
    const size_t S = (N + 1) & ~size_t(1);  // vector stride: keeps every work vector 16-byte aligned
    cudaError_t e;
    if (!c->d_work) {
        if (!c->d_plan && (e = plan_solver(c)) != cudaSuccess) return int(e);
        if (!c->solve_stream && (e = cudaStreamCreateWithFlags(&c->solve_stream, cudaStreamNonBlocking)) != cudaSuccess) return int(e);
        // sums of either form, results and the counter
        const size_t doubles = std::max(size_t(2) * kRedBlocks + 2, 2 * nangila::krylov::kSlot * size_t(c->ctas) + 5);
        if (!c->d_partial && (e = cudaMalloc(&c->d_partial, sizeof(double) * doubles)) != cudaSuccess) return int(e);
        if (!c->resident && !c->d_scaled && (e = cudaMalloc(&c->d_scaled, sizeof(double) * size_t(c->nnz))) != cudaSuccess) return int(e);
        if ((e = cudaMalloc(&c->d_work, sizeof(double) * S * kWorkVectors)) != cudaSuccess) return int(e);
    }
    double *inv = c->d_work, *b = inv + S;
    const char* genv = getenv("NANGILA_SPMV_GRAPH");
    if (!(genv && genv[0] == '0')) {
        cudaStream_t st = c->solve_stream;
        if (!c->inv_diag_on_device && (e = cudaMemcpyAsync(inv, c->h_inv_diag.data(), sizeof(double) * N, cudaMemcpyHostToDevice, st)) != cudaSuccess)
            return int(e);
        c->inv_diag_on_device = true;
        if ((e = cudaMemcpyAsync(b, h_b, sizeof(double) * N, cudaMemcpyHostToDevice, st)) != cudaSuccess) return int(e);
        return solve_on_device(c, h_x, tol, max_iter, iterations, rel_residual);
    }
    double *x = b + S, *r = x + S, *r0 = r + S, *p = r0 + S, *v = p + S, *s = v + S, *t = s + S, *ph = t + S, *sh = ph + S;
    double* out = c->d_partial + 2 * kRedBlocks;
    const int grid = (n + kThreads - 1) / kThreads;
    auto dots = [&](const double* a1, const double* b1, const double* a2, const double* b2, double res[2]) -> cudaError_t {
        dot2_partial_kernel<<<kRedBlocks, kThreads>>>(a1, b1, a2, b2, n, c->d_partial);
        dot2_final_kernel<<<1, 32>>>(c->d_partial, kRedBlocks, out);
        return cudaMemcpy(res, out, 2 * sizeof(double), cudaMemcpyDeviceToHost);
    };
    if ((e = cudaMemcpy(b, h_b, sizeof(double) * N, cudaMemcpyHostToDevice)) != cudaSuccess) return int(e);
    if ((e = cudaMemcpy(inv, c->h_inv_diag.data(), sizeof(double) * N, cudaMemcpyHostToDevice)) != cudaSuccess) return int(e);
    if ((e = cudaMemset(x, 0, sizeof(double) * S * 9)) != cudaSuccess) return int(e);
    residual_init_kernel<<<grid, kThreads>>>(r, r0, b, v, n);  // x = 0, so A x = v = 0
    double d[2];
    if ((e = dots(b, b, r, r, d)) != cudaSuccess) return int(e);
    double bnorm = sqrt(d[0]);
    if (bnorm == 0.0) bnorm = 1.0;
    double rel = sqrt(d[1]) / bnorm, rho = 1.0, alpha = 1.0, omega = 1.0;
    int it = 0;
    bool ok = rel < tol;
    while (!ok && it < max_iter) {
        if ((e = dots(r0, r, nullptr, nullptr, d)) != cudaSuccess) return int(e);
        double rho_new = d[0];
        if (fabs(rho_new) < 1e-300) break;
        double beta = (rho_new / rho) * (alpha / omega);
        rho = rho_new;
        update_p_kernel<<<grid, kThreads>>>(p, ph, r, v, inv, beta, omega, n);
        nangila_spmv_device(c, ph, v, 0);
        if ((e = dots(r0, v, nullptr, nullptr, d)) != cudaSuccess) return int(e);
        if (fabs(d[0]) < 1e-300) break;
        alpha = rho / d[0];
        update_s_kernel<<<grid, kThreads>>>(s, sh, r, v, inv, alpha, n);
        nangila_spmv_device(c, sh, t, 0);
        if ((e = dots(t, s, t, t, d)) != cudaSuccess) return int(e);
        omega = d[1] > 0.0 ? d[0] / d[1] : 0.0;
        update_xr_kernel<<<grid, kThreads>>>(x, r, ph, sh, s, t, alpha, omega, n);
        ++it;
        if ((e = dots(r, r, nullptr, nullptr, d)) != cudaSuccess) return int(e);
        rel = sqrt(d[0]) / bnorm;
        if (rel < tol) { ok = true; break; }
        if (omega == 0.0) break;
    }
    if ((e = cudaMemcpy(h_x, x, sizeof(double) * N, cudaMemcpyDeviceToHost)) != cudaSuccess) return int(e);
    if (iterations) *iterations = it;
    if (rel_residual) *rel_residual = rel;
    e = cudaGetLastError();
    if (e != cudaSuccess) return int(e);
    if (int st = nangila_spmv_status(c)) return st;
    return ok ? 0 : -1;
}
