// Jacobi-preconditioned BiCGSTAB as ONE kernel: the CTAs of the launch are all resident (cooperative launch), every CTA owns
// a contiguous range of rows for the whole solve, and an iteration is two phases with one grid-wide sum after each.
//
//   A   r = s - omega t, p <- r + beta (p - omega v), v <- A D p     -> <r0, v>                              -> alpha
//   B   s = r - alpha v, t = A D s                                   -> <t,s> <t,t> <r0,s> <r0,t> <s,s>      -> omega, beta, |r|
//
// (D: the inverse diagonal; its product with the matrix's columns is taken once per solve.) The vectors that a product needs at
// other rows depend on scalars that are known only after the sum before it, so what is left in memory are the parts:
// phase B leaves (s, t, p, v) of a row as 32 bytes, one memory sector, and phase A puts r and p together from them at every
// column it gathers; phase A leaves (r, v). <r0, r> and <r, r> follow from the five sums of phase B (r = s - omega t), and x
// is advanced one phase late. That makes two grid-wide sums per iteration where the textbook order needs five barriers.
//
// Those two are differences: their errors are rounding of |s|^2 and |r0| |s|, not of what is left. Where the step by omega removes
// most of s (matrices that couple mostly one way, as amplifier chains do), or <r0, r> cancels, a third sum takes both from the elements
// of r; no convergence and no breakdown is concluded from a value that has lost more than about two of its 16 digits. On meshes and
// ladders that happens in none to two of some hundred iterations.
//
// What bounds it: for circuit sizes (10^2 to 10^6 unknowns, vectors in L2) latency. A phase is one chain of an L2 gather, about 1 us;
// a grid-wide sum on 148 CTAs 2.4 (one value) to 3.3 us (five): two block reductions, one counter that one thread per CTA polls,
// one slot of partial sums read per thread. (A flag per CTA that every CTA polls: 8 us; the slots of all CTAs read by one warp,
// their values interleaved in shared lines: 4.5 to 9 us.) So a CTA's slice of the matrix stays in shared memory over all iterations where it fits,
// and small systems run on few CTAs, or on one. Measured on B200, us per iteration of whole calls, copies included, against
// one CUDA graph of 13 kernels per iteration: mesh of 400 nodes 59 -> 3.9, 2500: 57 -> 7.0, 65 536: 70 -> 8.9, 400 000: 83 -> 22, 10^6: 180 -> 69.
// With the values of a sum shared out among the lanes while a warp adds them up, a barrier less, and all entries of a row gathered at once:
// 10 000 nodes 7.19 -> 6.81, 65 536: 8.86 -> 8.40, 300 000: 16.6 -> 15.9; ladders of 10 000: 8.07 -> 7.68, 300 000: 15.9 -> 14.8; random rows of about six
// entries, 65 536: 12.0 -> 11.8, 300 000: 28.1 -> 28.6 to 29.2; uneven rows, 65 536 (mean 4.5): 14.2 -> 13.6. (Partial sums that carry their number, which every CTA looks at itself instead of
// a counter, took 10 us at 65 536 nodes.)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "signal.cuh"

namespace nangila {
namespace krylov {

// Threads per CTA. Where the slices fit into shared memory an iteration is latency, and 16 warps reduce faster than 32 (65 536 nodes:
// 8.8 us an iteration against 11.2); larger matrices are streamed, which wants more loads in flight (10^6 nodes: 65 against 88 us).
__host__ __device__ constexpr int solver_threads(bool resident) { return resident ? 512 : 1024; }
// Split of a matrix of nnz entries over CTAs. One CTA up to kOneCta entries: its sums are block barriers (1000 nodes, 4.9 K entries:
// 5.6 us an iteration, 6.5 on two CTAs); beyond that 2048 entries a CTA (2500 nodes: 6.3 us on 6 CTAs, 9.0 on 3, 7.4 on 12).
constexpr int kOneCta = 6144;
constexpr int kEntriesPerCta = 2048;
constexpr int kMaxCtas = 512;         // a sum reads the CTAs' slots with one thread each
constexpr int kLongRow = 64;          // rows above this many entries are summed by a whole warp each
constexpr int kCheckEvery = 4;        // iterations between two tests of the residual
// Below these shares of what they are differences of, <r, r> and <r0, r> are summed from r itself. |r| < 0.1 |s|: an error of about
// 1e-16 |s|^2 is then 1e-14 of |r|^2. <r0, r> may be small of itself; its line only has to catch what is nothing but rounding.
constexpr double kCancelled = 1e-2;
constexpr double kCancelledRho = 1e-6;
constexpr int kSums = 5;
constexpr int kSlot = 8;              // doubles a CTA's partial sums take: a line half of its own

struct __align__(32) Parts {
  double s, t, p, v;
};

struct SolverArgs {
  const int* row_ptr;
  const int* col;
  const double* val;
  const int* first_row;   // [ctas + 1]
  const int* long_rows;   // rows above kLongRow entries, ascending
  const int* first_long;  // [ctas + 1] into long_rows
  const double* b;
  const double* inv_diag;
  const int* status;      // set when a product of this matrix gave up waiting for one of its copies
  double *x, *r0, *p;
  Parts* parts;
  double2* rv;            // (r, v)
  double* scaled;         // value * inv_diag[column], where the slices do not fit into shared memory
  double* partial;        // [2][ctas][kSlot]: partial sums, by parity of the sum's number
  uint32_t* arrived;      // zero: CTAs that have contributed, over all sums
  double* out;            // <r, r>, ||b|| (1 for a zero right-hand side), iterations, 1 if a wait ran out (zero at first)
  int max_iter, max_entries;
  double tol;
  uint64_t timeout_ns;
};

__host__ __device__ inline size_t solver_smem(bool resident, int max_rows, int max_entries) {
  return resident ? size_t(max_entries) * 12 + size_t(max_rows + 1) * 4 : 0;
}

// Sums of N values over all threads of the grid, the same bits in every thread: partial sums are added in a fixed order. Also
// the grid-wide barrier between the phases (what a thread wrote before it is seen by every thread after it). False if the
// other CTAs did not arrive within the time limit.
template <int WARPS>
struct GridSum {
  double* partial;
  uint32_t* arrived;
  uint64_t timeout_ns;
  double (*twice)[WARPS][kSums];  // by parity of the sum's number: a thread may be a sum ahead of another's last look
  int* failed;
  uint32_t k = 0;
  // The sum over a warp of each of N values: value i in lane 4 i. The values are shared out among the lanes as they are added up
  // (nine exchanges for five values; each on its own takes 25).
  template <int N>
  static __device__ __forceinline__ double warp_sums(const double (&v)[N]) {
    const int lane = threadIdx.x & 31;
    double a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = i < N ? v[i < N ? i : 0] : 0.0;
#pragma unroll
    for (int half = 4; half >= 1; half >>= 1) {
      const bool upper = (lane & (4 * half)) != 0;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        if (i < N) {  // (above N only zeros would meet)
          const double other = __shfl_xor_sync(0xffffffffu, upper ? a[i] : a[i + half], 4 * half);
          a[i] = (upper ? a[i + half] : a[i]) + other;
        }
      }
    }
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 2);
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], 1);
    return a[0];
  }
  template <int N>
  __device__ __forceinline__ bool operator()(double (&v)[N]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ctas = int(gridDim.x);
    ++k;
    double (*sh)[kSums] = twice[k & 1u];
    const double mine = warp_sums(v);
    if ((lane & 3) == 0 && lane / 4 < N) sh[warp][lane / 4] = mine;
    __syncthreads();
    if (ctas == 1) {
      if (warp == 0 && lane < N) {
        double a = 0.0;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) a += sh[w][lane];
        sh[0][lane] = a;  // no other lane reads this column
      }
      __syncthreads();
    }
    int groups = 1;
    if (ctas > 1) {
      double* slots = partial + size_t(k & 1u) * kSlot * ctas;
      if (warp == 0) {
        if (lane < N) {
          double a = 0.0;
#pragma unroll
          for (int w = 0; w < WARPS; ++w) a += sh[w][lane];
          __stcg(slots + blockIdx.x * kSlot + lane, a);
        }
        __syncwarp();
        if (lane == 0) {
          comm::red_release_gpu_add(arrived, 1u);
          uint64_t t0 = 0;
          uint32_t spins = 0;
          while (int32_t(comm::ld_acquire_gpu(arrived) - k * uint32_t(ctas)) < 0) {
            if ((++spins & 255u) == 0u) {
              const uint64_t now = comm::globaltimer_ns();
              if (t0 == 0) t0 = now;
              if (now - t0 > timeout_ns) {
                *failed = 1;
                break;
              }
            }
          }
        }
      }
      __syncthreads();
      // one slot a thread (a CTA that is one sum ahead has not touched this one's set of slots: there are two)
      groups = (ctas + 31) / 32;
      if (warp < groups) {
        const double2* slot = reinterpret_cast<const double2*>(slots + tid * kSlot);
        const bool have = tid < ctas;
#pragma unroll
        for (int i = 0; i < N; i += 2) {
          const double2 w = have ? __ldcg(slot + i / 2) : make_double2(0.0, 0.0);
          v[i] = w.x;
          if (i + 1 < N) v[i + 1] = w.y;
        }
        const double part = warp_sums(v);
        if ((lane & 3) == 0 && lane / 4 < N) sh[warp][lane / 4] = part;
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = sh[0][i];
    for (int w = 1; w < groups; ++w) {
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += sh[w][i];
    }
    return *reinterpret_cast<volatile int*>(failed) == 0;
  }
};

template <bool RESIDENT>
__global__ void __launch_bounds__(solver_threads(RESIDENT), 1) bicgstab_kernel(const __grid_constant__ SolverArgs a) {
  constexpr int kThreads = solver_threads(RESIDENT), kWarps = kThreads / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double sh[2][kWarps][kSums];
  __shared__ int failed;
  const int tid = threadIdx.x;
  const int r0 = a.first_row[blockIdx.x], r1 = a.first_row[blockIdx.x + 1], rows = r1 - r0;
  const int l0 = a.first_long[blockIdx.x], l1 = a.first_long[blockIdx.x + 1];
  const int k0 = a.row_ptr[r0], entries = a.row_ptr[r1] - k0;
  // this CTA's slice, indexed from its first row and entry: the values times the inverse diagonal of their columns
  double* val = RESIDENT ? reinterpret_cast<double*>(smem) : a.scaled + k0;
  const int* col = a.col + k0;
  const int* start = a.row_ptr + r0;
  const int base = RESIDENT ? 0 : k0;
  for (int k = tid; k < entries; k += kThreads) val[k] = a.val[k0 + k] * a.inv_diag[col[k]];
  if (RESIDENT) {
    int* s_col = reinterpret_cast<int*>(val + a.max_entries);
    int* s_start = s_col + a.max_entries;
    for (int k = tid; k < entries; k += kThreads) s_col[k] = col[k];
    for (int k = tid; k <= rows; k += kThreads) s_start[k] = start[k] - k0;
    col = s_col;
    start = s_start;
  }
  // Lanes per row: one, unless rows are long (eight entries a lane) or there are lanes to spare.
  const int mean = rows > 0 ? entries / rows : 1;
  int lanes = 1;
  while (lanes < 32 && lanes * 2 <= mean && (mean > 8 * lanes || rows * lanes * 2 <= kThreads)) lanes *= 2;
  const int group = tid / lanes, lane = tid % lanes, groups = kThreads / lanes;
  const int turns = (rows + groups - 1) / groups;  // every lane of a warp takes part in the same shuffles

  // For every row of this CTA: own = load(row); sum = sum over the row's entries of value * gather(column); then
  // finish(row, own, sum), the first and the last by one lane.
  auto product = [&](auto load, auto gather, auto finish) {
    if (l1 > l0) {
      for (int l = l0 + (tid >> 5); l < l1; l += kWarps) {
        const int i = a.long_rows[l] - r0;
        double sum = 0.0;
#pragma unroll 4
        for (int j = start[i] - base + (tid & 31), e = start[i + 1] - base; j < e; j += 32) sum += val[j] * gather(col[j]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off);
        if ((tid & 31) == 0) finish(r0 + i, load(r0 + i), sum);
      }
    }
    for (int it = 0; it < turns; ++it) {
      const int i = it * groups + group;
      int s = 0, e = 0;
      if (i < rows) {
        s = start[i] - base;
        e = start[i + 1] - base;
      }
      const bool mine = i < rows && e - s <= kLongRow;
      decltype(load(0)) own{};
      if (mine && lane == 0) own = load(r0 + i);
      double sum = 0.0;
      // All gathers of a short row at once, at a valid place whatever its length: the next one would wait for a trip to L2 otherwise. As many as the warp's
      // longest row has, since a gather that nobody needs takes its time too (five for every row: ladders 2 to 8 % slower than with one behind the other).
      const int most = __reduce_max_sync(0xffffffffu, mine ? e - s : 0);
      auto row = [&](auto n) {
        constexpr int N = decltype(n)::value;
        if (mine) {
          for (int j = s + lane; j < e; j += N * lanes) {
            double g[N], w[N];
#pragma unroll
            for (int u = 0; u < N; ++u) {
              const int at = min(j + u * lanes, e - 1);
              g[u] = gather(col[at]);
              w[u] = val[at];
            }
#pragma unroll
            for (int u = 0; u < N; ++u)
              if (j + u * lanes < e) sum += w[u] * g[u];
          }
        }
      };
      if (most <= 3 * lanes) row(std::integral_constant<int, 3>{});
      else if (most <= 5 * lanes) row(std::integral_constant<int, 5>{});
      else row(std::integral_constant<int, 4>{});
      for (int off = lanes >> 1; off > 0; off >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, off, lanes);
      if (mine && lane == 0) finish(r0 + i, own, sum);
    }
  };

  GridSum<kWarps> sum{a.partial, a.arrived, a.timeout_ns, sh, &failed};
  if (tid == 0) failed = 0;
  double bb[1] = {0.0};
  for (int i = r0 + tid; i < r1; i += kThreads) {
    const double bi = a.b[i];
    a.x[i] = 0.0;
    a.r0[i] = bi;
    a.parts[i] = Parts{bi, 0.0, 0.0, 0.0};
    bb[0] += bi * bi;
  }
  __syncthreads();  // the slice in shared memory (and, where it is in memory, this CTA's writes) are complete
  bool alive = sum(bb);
  double bnorm = sqrt(bb[0]);
  if (bnorm == 0.0) bnorm = 1.0;
  double rr = bb[0], rho_next = bb[0], rho = 1.0, alpha = 0.0, omega = 1.0, beta = 0.0;
  bool first = true;
  int it = 0;
  bool done = sqrt(rr) / bnorm < a.tol;
  while (alive && !done && it < a.max_iter) {
    for (int k = 0; k < kCheckEvery; ++k) {
      if (fabs(rho_next) < 1e-300) {  // breakdown: what there is is the answer
        done = true;
        break;
      }
      // (in the first iteration t, p and v are zero: r = s = b, p = b, and x has no step to take)
      beta = first ? 0.0 : (rho_next / rho) * (alpha / omega);
      rho = rho_next;
      // ---- A ----
      struct RowA {
        Parts q;
        double x, r0, inv;
      };
      double rv[1] = {0.0};
      const double om = omega, be = beta, xp = first ? 0.0 : alpha, xs = first ? 0.0 : omega;
      product([&](int i) { return RowA{a.parts[i], a.x[i], a.r0[i], a.inv_diag[i]}; },
              [&](int j) {
                const Parts q = a.parts[j];
                return q.s - om * q.t + be * (q.p - om * q.v);
              },
              [&](int i, const RowA& o, double v) {
                a.x[i] = o.x + o.inv * (xp * o.q.p + xs * o.q.s);
                const double r = o.q.s - om * o.q.t;
                a.p[i] = r + be * (o.q.p - om * o.q.v);
                a.rv[i] = make_double2(r, v);
                rv[0] += o.r0 * v;
              });
      if (!(alive = sum(rv))) break;
      first = false;
      if (fabs(rv[0]) < 1e-300) {
        done = true;
        alpha = omega = 0.0;  // x has had its last step
        break;
      }
      alpha = rho / rv[0];
      // ---- B ----
      struct RowB {
        double2 rv;
        double r0, p;
      };
      double d[kSums] = {0.0, 0.0, 0.0, 0.0, 0.0};
      const double step = alpha;
      product([&](int i) { return RowB{a.rv[i], a.r0[i], a.p[i]}; },
              [&](int j) {
                const double2 w = a.rv[j];
                return w.x - step * w.y;
              },
              [&](int i, const RowB& o, double t) {
                const double s = o.rv.x - step * o.rv.y;
                a.parts[i] = Parts{s, t, o.p, o.rv.y};
                d[0] += t * s;
                d[1] += t * t;
                d[2] += o.r0 * s;
                d[3] += o.r0 * t;
                d[4] += s * s;
              });
      if (!(alive = sum(d))) break;
      omega = d[1] > 0.0 ? d[0] / d[1] : 0.0;
      rho_next = d[2] - omega * d[3];
      rr = d[4] - omega * (2.0 * d[0] - omega * d[1]);
      if (rr < kCancelled * d[4] || fabs(rho_next) <= kCancelledRho * (fabs(d[2]) + fabs(omega * d[3]))) {
        double m[2] = {0.0, 0.0};
        for (int i = r0 + tid; i < r1; i += kThreads) {  // this CTA's rows: its own writes
          const Parts q = a.parts[i];
          const double r = q.s - omega * q.t;
          m[0] += r * r;
          m[1] += a.r0[i] * r;
        }
        if (!(alive = sum(m))) break;
        rr = m[0];
        rho_next = m[1];
      }
      ++it;
      if (omega == 0.0) {
        done = true;
        break;
      }
    }
    done = done || sqrt(rr) / bnorm < a.tol;
  }
  // the step of the last whole iteration
  if (it > 0) {
    for (int i = r0 + tid; i < r1; i += kThreads) a.x[i] += a.inv_diag[i] * (alpha * a.parts[i].p + omega * a.parts[i].s);
  }
  if (blockIdx.x == 0 && tid == 0) {
    a.out[0] = rr;
    a.out[1] = bnorm;
    a.out[2] = double(it);
    if (*a.status != 0) a.out[3] = 1.0;
  }
  if (tid == 0 && failed) a.out[3] = 1.0;
}

}  // namespace krylov
}  // namespace nangila
