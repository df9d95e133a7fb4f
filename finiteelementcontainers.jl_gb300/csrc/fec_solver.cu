// fec_solver.cu -- the linear solve after assembly: preconditioned conjugate
// gradients on the assembled CSC stiffness over the unknowns (the reference's
// IterativeLinearSolver, src/Solvers.jl:88-152, which hands K and R to a Krylov
// CG), on the device.
//
// K is symmetric, so its CSC columns are its rows.  A matrix that fits the SMs' shared
// memory is solved in one cooperative launch (cg_solve_kernel); else an iteration is three
// kernels: y = K p with the partial sums of p.y, x and r updated with the
// partial sums of r.z and r.r, and the new direction.  The partial sums of a
// kernel (one per CTA) are added by every CTA of the next one in the same fixed
// order, so there is no reduction kernel, the scalars never leave the device and
// a solve is bitwise repeatable.
//
// What bounds it: up to some 100k unknowns launches, the latency of dependent
// loads and the FP64 pipe, which takes an SM 16 clocks per warp instruction
// however few lanes are active (the matrix of a 36 x 32 x 34 box, 11 MB, stays in
// L2); beyond, the matrix from memory.  Hence three launches an iteration instead
// of eight, chained by programmatic dependent launch; a product with one FP64
// instruction per entry and no shuffle tree (a warp copies the entries of its
// next 32 rows to shared memory, coalesced and asynchronous, while each lane adds
// a row of the last 32, whose x entries are mostly neighbours' too); sums
// through shared memory and one warp; and the stopping test on the device, which
// the host reads one batch of iterations behind, so the stream never runs dry and
// the kernels of a batch that follow the converged iteration return at once.
// Per iteration, Poisson: 36 x 32 x 34 elements 55 -> 15 us (product 7, update 4,
// direction 4; 11 in one launch), 70^3 elements 59 us (product 44: 2.5 TB/s of matrix).
#include <cmath>
#include <cstdlib>
#include <cstring>
#include "fec_launch.h"
#include "fec_solver.h"

namespace fec {
namespace {

constexpr int THREADS = 256;
constexpr int MAX_CTAS = 304;  // the partial sums of one kernel
constexpr int WARPS = THREADS / 32;
constexpr int CAP = 896;       // entries a warp stages at once (32 rows of 27 fit; longer rows take more rounds)
constexpr size_t ROWS_SMEM = size_t(WARPS) * 2 * CAP * 12;  // (value, row) double-buffered

// scalars on the device
struct CgScalars {
  double rz[2];      // r.z of the iteration, by parity
  double bb, rr;     // b.b; r.r of the last stopping test
  int it;            // iterations of the last stopping test
  int done;          // 1: converged (or b = 0); the iteration kernels return
};

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The step length, and the factor of the old direction in the new one: a / b, and 0 where b
// is.  That is where the residual has become exactly zero (r.z = 0; p = 0 an iteration
// later): x stays.  (Compared as an integer: off the FP64 pipe.)
__device__ __forceinline__ double quotient(double a, double b) {
  return (__double_as_longlong(b) << 1) == 0 ? 0.0 : a / b;
}
// The stopping test (rtol 0: none, every iteration asked for).
__device__ __forceinline__ bool converged(double rr, double bb, double rtol) {
  return rtol > 0.0 && sqrt(rr) / sqrt(bb) <= rtol;
}

// Sums over the CTA of a and b (fixed order), to thread 0 (a) and thread 32 (b).
// Through shared memory: a shuffle tree in every warp would issue three times the
// FP64 instructions.
struct SumBuf {
  double a[THREADS], b[THREADS];
};
// (in pairs: a dependent FP64 addition takes over a hundred clocks, and these sums are a
// third of an iteration)
template <int N>
__device__ __forceinline__ double pair_sum(double (&t)[N]) {
  static_assert((N & (N - 1)) == 0, "pairs");
#pragma unroll
  for (int h = N / 2; h > 0; h /= 2)
#pragma unroll
    for (int k = 0; k < h; ++k) t[k] += t[k + h];
  return t[0];
}
__device__ __forceinline__ double lanes_total(double t) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}
__device__ __forceinline__ double warp_total(const double* v) {
  const int lane = threadIdx.x & 31;
  double t[THREADS / 32];
#pragma unroll
  for (int k = 0; k < THREADS / 32; ++k) t[k] = v[lane + 32 * k];
  return lanes_total(pair_sum(t));
}
__device__ __forceinline__ void cta_sums(SumBuf& buf, double a, double b, double* out_a, double* out_b) {
  buf.a[threadIdx.x] = a;
  buf.b[threadIdx.x] = b;
  __syncthreads();
  if (threadIdx.x < 32) {
    const double t = warp_total(buf.a);
    if (threadIdx.x == 0) *out_a = t;
  } else if (threadIdx.x < 64) {
    const double t = warp_total(buf.b);
    if (threadIdx.x == 32) *out_b = t;
  }
}
// The partial sums part[0 .. count), added in the same order by every CTA, on
// every thread.
__device__ __forceinline__ double total(const double* part, int count, double* slot) {
  if (threadIdx.x < 32) {
    // (every load before the first addition)
    double v[8], w[2] = {0.0, 0.0};
    static_assert(MAX_CTAS <= 320, "ten a lane");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = int(threadIdx.x) + 32 * i < count ? __ldcg(part + threadIdx.x + 32 * i) : 0.0;
    if (count > 256)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (int(threadIdx.x) + 32 * (8 + i) < count) w[i] = __ldcg(part + threadIdx.x + 32 * (8 + i));
    double s = pair_sum(v);
    if (count > 256) s += w[0] + w[1];
    s = lanes_total(s);
    if (threadIdx.x == 0) *slot = s;
  }
  __syncthreads();
  return *slot;
}

// Entries [c0, c0 + CAP) of the 32 rows 32 rc .. of a warp; this lane's row is
// 32 rc + lane and has the entries [lo, hi).
struct Round {
  int64_t rc, lo, hi, c0, end;
};

// f(j, (K x)_j, K_jj) for the rows of this warp (WANT_DIAG, else 0): a lane adds a
// row in its order; the entries of the next round are on their way meanwhile.
template <bool WANT_DIAG, class F>
__device__ __forceinline__ void rows_product(const CscSym& A, const double* x, unsigned char* sm, F f) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* val = reinterpret_cast<double*>(sm) + warp * 2 * CAP;
  int32_t* row = reinterpret_cast<int32_t*>(sm + size_t(WARPS) * 2 * CAP * 8) + warp * 2 * CAP;
  const int64_t GW = int64_t(gridDim.x) * WARPS, n = A.n;
  auto ptr = [&](int64_t j) { return __ldg(A.colptr + (j < n ? j : n)); };
  auto start = [&](int64_t rc, int64_t lo, int64_t hi) {
    Round r;
    r.rc = rc;
    r.lo = lo;
    r.hi = hi;
    r.c0 = __shfl_sync(0xffffffffu, lo, 0);
    r.end = __shfl_sync(0xffffffffu, hi, 31);
    return r;
  };
  auto issue = [&](const Round& r, int st) {
    if (r.rc * 32 < n) {
      const int cnt = int(r.end - r.c0 < CAP ? r.end - r.c0 : CAP);
      for (int i = lane; i < cnt; i += 32) {
        gp::cp_small<8>(val + st * CAP + i, A.val + r.c0 + i);
        gp::cp_small<4>(row + st * CAP + i, A.rowval + r.c0 + i);
      }
    }
    gp::commit();
  };
  int64_t rc = int64_t(blockIdx.x) * WARPS + warp;
  Round cur = start(rc, ptr(rc * 32 + lane), ptr(rc * 32 + lane + 1));
  issue(cur, 0);
  int64_t rc1 = rc + GW, lo1 = ptr(rc1 * 32 + lane), hi1 = ptr(rc1 * 32 + lane + 1);  // the chunk after
  double s = 0.0, d = 0.0;
  for (int it = 0; cur.rc * 32 < n; ++it) {
    const int st = it & 1;
    Round nxt = cur;
    const bool last = cur.c0 + CAP >= cur.end;  // of these 32 rows
    if (last) {
      nxt = start(rc1, lo1, hi1);
      rc1 += GW;
      lo1 = ptr(rc1 * 32 + lane);
      hi1 = ptr(rc1 * 32 + lane + 1);
    } else {
      nxt.c0 += CAP;
    }
    issue(nxt, st ^ 1);
    gp::wait_prev();
    __syncwarp();
    const int64_t j = cur.rc * 32 + lane;
    const int b = int((cur.lo > cur.c0 ? cur.lo : cur.c0) - cur.c0);
    const int e = int((cur.hi < cur.c0 + CAP ? cur.hi : cur.c0 + CAP) - cur.c0);
    const double* v = val + st * CAP;
    const int32_t* c = row + st * CAP;
    constexpr int U = 9;
    for (int i = b; i < e; i += U) {
      double xv[U];
#pragma unroll
      for (int k = 0; k < U; ++k) {
        const int cc = i + k < e ? c[i + k] : -1;
        xv[k] = cc >= 0 ? x[cc] : 0.0;
        if (WANT_DIAG && cc == j) d = v[i + k];
      }
#pragma unroll
      for (int k = 0; k < U; ++k)
        if (i + k < e) s = fma(v[i + k], xv[k], s);
    }
    if (last) {
      if (j < n) f(j, s, d);
      s = d = 0.0;
    }
    __syncwarp();  // every lane has read this stage
    cur = nxt;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// r = b - K x; z = M^-1 r; p = z; partial sums of r.z and b.b.  inv_diag: filled
// here when the preconditioner is Jacobi's, else null (M = 1).
__global__ void __launch_bounds__(THREADS) cg_init_kernel(CscSym A, const double* __restrict__ b, const double* x,
                                                          double* r, double* z, double* p, double* inv_diag,
                                                          double* part_rz, double* part_bb) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SumBuf buf;
  double rz = 0.0, bb = 0.0;
  auto put = [&](int64_t j, double s, double d) {
    const double bj = b[j], rj = bj - s;
    double zj = rj;
    if (inv_diag) {
      const double m = d != 0.0 ? 1.0 / d : 1.0;
      inv_diag[j] = m;
      zj = m * rj;
    }
    r[j] = rj;
    z[j] = zj;
    p[j] = zj;
    rz = fma(rj, zj, rz);
    bb = fma(bj, bj, bb);
  };
  if (inv_diag)
    rows_product<true>(A, x, sm, put);
  else
    rows_product<false>(A, x, sm, put);
  cta_sums(buf, rz, bb, part_rz + blockIdx.x, part_bb + blockIdx.x);
}

// b.b and whether it is zero (one CTA)
__global__ void __launch_bounds__(THREADS) cg_start_kernel(const double* part_rz, const double* part_bb, int count,
                                                           CgScalars* sc) {
  __shared__ double slot[2];
  const double rz = total(part_rz, count, slot), bb = total(part_bb, count, slot + 1);
  if (threadIdx.x == 0) {
    sc->rz[0] = rz;
    sc->bb = bb;
    sc->rr = 0.0;
    sc->it = 0;
    sc->done = bb == 0.0 ? 1 : 0;
  }
}

// y = K p; partial sums of p.y
__global__ void __launch_bounds__(THREADS) cg_product_kernel(CscSym A, const double* p, double* y, double* part,
                                                             const CgScalars* sc) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SumBuf buf;
  grid_wait();
  grid_next();
  if (__ldcg(&sc->done)) return;
  double py = 0.0;
  rows_product<false>(A, p, sm, [&](int64_t j, double s, double) {
    y[j] = s;
    py = fma(p[j], s, py);
  });
  buf.a[threadIdx.x] = py;
  __syncthreads();
  if (threadIdx.x < 32) {
    const double t = warp_total(buf.a);
    if (threadIdx.x == 0) part[blockIdx.x] = t;
  }
}

// alpha = r.z / p.y; x += alpha p; r -= alpha y; z = M^-1 r; partial sums of the
// new r.z and r.r.  (A thread's next entries are loaded before it waits for the
// sum or uses those it has.)
__global__ void __launch_bounds__(THREADS) cg_update_kernel(int64_t n, const CgScalars* sc, int parity,
                                                            const double* part_py, int count, double* x, double* r,
                                                            double* z, const double* p, const double* y,
                                                            const double* inv_diag, double* part_rz, double* part_rr) {
  __shared__ SumBuf buf;
  __shared__ double slot;
  grid_wait();
  grid_next();
  if (__ldcg(&sc->done)) return;
  int64_t i = int64_t(blockIdx.x) * THREADS + threadIdx.x;
  double pi = 0.0, yi = 0.0, xi = 0.0, ri = 0.0, mi = 1.0;
  auto load = [&] {
    if (i >= n) return;
    pi = p[i];
    yi = y[i];
    xi = x[i];
    ri = r[i];
    if (inv_diag) mi = inv_diag[i];
  };
  load();
  const double alpha = quotient(__ldcg(&sc->rz[parity]), total(part_py, count, &slot));
  double rz = 0.0, rr = 0.0;
  while (i < n) {
    const int64_t k = i;
    const double xk = fma(alpha, pi, xi), rk = fma(-alpha, yi, ri), zk = mi * rk;
    i += int64_t(gridDim.x) * THREADS;
    load();
    x[k] = xk;
    r[k] = rk;
    z[k] = zk;
    rz = fma(rk, zk, rz);
    rr = fma(rk, rk, rr);
  }
  cta_sums(buf, rz, rr, part_rz + blockIdx.x, part_rr + blockIdx.x);
}

// beta = new r.z / r.z; p = z + beta p; the new r.z for the next iteration
__global__ void __launch_bounds__(THREADS) cg_direction_kernel(int64_t n, CgScalars* sc, int parity,
                                                               const double* part_rz, int count, const double* z,
                                                               double* p) {
  __shared__ double slot;
  grid_wait();
  grid_next();
  if (__ldcg(&sc->done)) return;
  int64_t i = int64_t(blockIdx.x) * THREADS + threadIdx.x;
  double zi = 0.0, pi = 0.0;
  auto load = [&] {
    if (i >= n) return;
    zi = z[i];
    pi = p[i];
  };
  load();
  const double rz = total(part_rz, count, &slot);
  const double beta = quotient(rz, __ldcg(&sc->rz[parity]));
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->rz[parity ^ 1] = rz;
  while (i < n) {
    const int64_t k = i;
    const double pk = fma(beta, pi, zi);
    i += int64_t(gridDim.x) * THREADS;
    load();
    p[k] = pk;
  }
}

// The stopping test after `it` iterations: sqrt(r.r) / sqrt(b.b) <= rtol (one CTA).
__global__ void __launch_bounds__(THREADS) cg_test_kernel(CgScalars* sc, const double* part_rr, int count, int it,
                                                          double rtol) {
  __shared__ double slot;
  grid_wait();
  grid_next();
  if (__ldcg(&sc->done)) return;
  const double rr = total(part_rr, count, &slot);
  if (threadIdx.x == 0) {
    sc->rr = rr;
    sc->it = it;
    if (converged(rr, sc->bb, rtol)) sc->done = 1;
  }
}

// The whole solve in one cooperative launch, for matrices that fit the SMs' shared
// memory.  A CTA keeps its rows' entries there and their vectors in registers (KR rows a
// thread); only p, which other rows read, and the partial sums go through memory.  An
// iteration is three barriers over the grid -- the sums of p.y, those of r.z and r.r,
// the new p -- and the arithmetic of the three kernels above.  A barrier is one atomic a
// CTA and a bounded wait; a CTA that gives up reports through sc->done.
//
// What bounds it: latency -- three barriers (2,500 clocks each), the FP64 sums on their way
// (eight dependent additions each) and the gathers of p from L2 -- and the FP64 pipe in the
// product.  (The next nine gathers in flight during the additions: no faster.)  Whole
// solves, three kernels an iteration against this: 60 elements 364 -> 308 us, 36 x 32 x 34
// (35,805 unknowns) 1.98 -> 1.61 ms, 44 x 45 x 46 3.77 -> 2.77 ms: faster wherever it
// applies.
constexpr int KR = 4, COOP_CAP = 16384;  // entries of a CTA (one with more reads them from memory)
constexpr size_t COOP_SMEM = size_t(COOP_CAP) * 12;
constexpr long long COOP_BUDGET = 2000000000LL;  // clocks a barrier waits when no budget is set
struct CoopShape {
  int64_t rows;  // of a CTA
  unsigned grid;
};
__global__ void __launch_bounds__(THREADS, 1) cg_solve_kernel(CscSym A, int64_t rows, const double* __restrict__ b,
                                                              double* x, double* p, int jacobi, double* parts,
                                                              CgScalars* sc, unsigned long long* bar, int max_iter,
                                                              int check_every, double rtol, long long budget) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SumBuf buf;
  __shared__ double slot[2];
  __shared__ int s_fail;
  const int tid = threadIdx.x;
  const int64_t r0 = int64_t(blockIdx.x) * rows, r1 = r0 + rows < A.n ? r0 + rows : A.n;
  const int64_t base = A.colptr[r0];
  const int cnt = int(A.colptr[r1] - base);
  const double* val = A.val + base;
  const int32_t* col = A.rowval + base;
  if (cnt <= COOP_CAP) {
    double* v = reinterpret_cast<double*>(sm);
    int32_t* c = reinterpret_cast<int32_t*>(sm + size_t(COOP_CAP) * 8);
    for (int i = tid; i < cnt; i += THREADS) {
      v[i] = val[i];
      c[i] = col[i];
    }
    val = v;
    col = c;
  }
  if (tid == 0) s_fail = 0;
  __syncthreads();
  double* part_py = parts;
  double* part_rz = parts + MAX_CTAS;
  double* part_rr = parts + 2 * MAX_CTAS;
  unsigned long long target = 0;
  // false: a wait gave up, here or elsewhere
  auto barrier = [&] {
    target += gridDim.x;
    __syncthreads();
    if (tid == 0) {
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(bar), "l"(1ull) : "memory");
      const long long t0 = clock64();
      for (;;) {
        unsigned long long seen;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(bar) : "memory");
        if (seen >= target) break;
        if (clock64() - t0 > budget) {
          s_fail = 1;
          atomicExch(&sc->done, -1);
          break;
        }
      }
    }
    __syncthreads();
    return s_fail == 0;
  };
  int lo[KR], hi[KR];
  double xk[KR], rk[KR], pk[KR], yk[KR], mk[KR];
  // sum over row k of this thread of K_jc src_c; d: its diagonal entry
  auto product = [&](const double* src, int k, double& d) {
    const int64_t j = r0 + tid + k * THREADS;
    double s = 0.0;
    constexpr int U = 9;
    for (int i = lo[k]; i < hi[k]; i += U) {
      double xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int cc = i + u < hi[k] ? col[i + u] : -1;
        xv[u] = cc >= 0 ? __ldcg(src + cc) : 0.0;
        if (cc == j) d = val[i + u];
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (i + u < hi[k]) s = fma(val[i + u], xv[u], s);
    }
    return s;
  };
  double rz = 0.0, bb = 0.0;
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const int64_t j = r0 + tid + k * THREADS;
    lo[k] = hi[k] = 0;
    xk[k] = rk[k] = pk[k] = yk[k] = 0.0;
    mk[k] = 1.0;
    if (j >= r1) continue;
    lo[k] = int(A.colptr[j] - base);
    hi[k] = int(A.colptr[j + 1] - base);
    double d = 0.0;
    const double bj = b[j];
    rk[k] = bj - product(x, k, d);
    xk[k] = x[j];
    if (jacobi) mk[k] = d != 0.0 ? 1.0 / d : 1.0;
    pk[k] = mk[k] * rk[k];
    p[j] = pk[k];
    rz = fma(rk[k], pk[k], rz);
    bb = fma(bj, bj, bb);
  }
  cta_sums(buf, rz, bb, part_rz + blockIdx.x, part_rr + blockIdx.x);
  if (!barrier()) return;
  rz = total(part_rz, int(gridDim.x), slot);
  bb = total(part_rr, int(gridDim.x), slot + 1);
  double rr_test = 0.0;
  int it_test = 0, done = bb == 0.0;
  for (int it = 0; it < max_iter && !done;) {
    double py = 0.0;
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      if (r0 + tid + k * THREADS >= r1) continue;
      double d = 0.0;
      yk[k] = product(p, k, d);
      py = fma(pk[k], yk[k], py);
    }
    buf.a[tid] = py;
    __syncthreads();
    if (tid < 32) {
      const double t = warp_total(buf.a);
      if (tid == 0) part_py[blockIdx.x] = t;
    }
    if (!barrier()) return;
    const double alpha = quotient(rz, total(part_py, int(gridDim.x), slot));
    double rz1 = 0.0, rr = 0.0;
    double zk[KR];
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      zk[k] = 0.0;
      if (k * THREADS >= rows) continue;  // (an FP64 instruction costs the same with no lane active)
      xk[k] = fma(alpha, pk[k], xk[k]);
      rk[k] = fma(-alpha, yk[k], rk[k]);
      zk[k] = mk[k] * rk[k];
      rz1 = fma(rk[k], zk[k], rz1);
      rr = fma(rk[k], rk[k], rr);
    }
    cta_sums(buf, rz1, rr, part_rz + blockIdx.x, part_rr + blockIdx.x);
    if (!barrier()) return;
    rz1 = total(part_rz, int(gridDim.x), slot);
    ++it;
    if (it % check_every == 0 || it == max_iter) {  // the stopping test
      rr_test = total(part_rr, int(gridDim.x), slot + 1);
      it_test = it;
      done = converged(rr_test, bb, rtol);
      if (done || it == max_iter) break;
    }
    const double beta = quotient(rz1, rz);
    rz = rz1;
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      const int64_t j = r0 + tid + k * THREADS;
      if (k * THREADS >= rows) continue;
      pk[k] = fma(beta, pk[k], zk[k]);
      if (j < r1) p[j] = pk[k];
    }
    if (!barrier()) return;
  }
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const int64_t j = r0 + tid + k * THREADS;
    if (j < r1) x[j] = xk[k];
  }
  if (blockIdx.x == 0 && tid == 0) {
    sc->bb = bb;
    sc->rr = rr_test;
    sc->it = it_test;
  }
}

// A launch that may start while the kernel before it on the stream drains; its
// kernels wait (grid_wait) before they read what that one wrote.
template <typename... P, typename... Q>
cudaError_t launch_next(void (*kern)(P...), unsigned grid, size_t smem, cudaStream_t s, Q... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

constexpr size_t SC_DOUBLES = (sizeof(CgScalars) + 7) / 8;

}  // namespace

cudaError_t PcgHost::ensure() {
  cudaError_t e;
  if (!pinned && (e = cudaMallocHost(&pinned, 2 * SLOT)) != cudaSuccess) return e;
  for (cudaEvent_t& d : done)
    if (!d && (e = cudaEventCreateWithFlags(&d, cudaEventDisableTiming)) != cudaSuccess) return e;
  return cudaSuccess;
}

void PcgHost::release() {
  if (pinned) cudaFreeHost(pinned);
  pinned = nullptr;
  for (cudaEvent_t& d : done) {
    if (d) cudaEventDestroy(d);
    d = nullptr;
  }
}

// Where the one-launch solve applies: the entries in the SMs' shared memory, at most KR
// rows a thread.  FEC_CG_COOP=0 keeps the three kernels an iteration.
static bool coop_shape(const CscSym& A, CoopShape* out) {
  const char* v = std::getenv("FEC_CG_COOP");
  const int64_t sms = num_sms() < MAX_CTAS ? num_sms() : MAX_CTAS;
  const int64_t by_rows = (A.n + THREADS - 1) / THREADS, by_nnz = A.nnz / (COOP_CAP / 10 * 9) + 1;
  int64_t grid = by_rows > by_nnz ? by_rows : by_nnz;
  if (grid > sms) grid = sms;
  if ((v && v[0] == '0') || A.nnz > grid * COOP_CAP || A.n > grid * KR * THREADS) return false;
  int dev = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) {
    cudaGetLastError();
    return false;
  }
  out->rows = (A.n + grid - 1) / grid;
  out->grid = unsigned((A.n + out->rows - 1) / out->rows);
  return true;
}

size_t pcg_scratch_doubles(int64_t n) { return size_t(5) * size_t(n) + 3 * MAX_CTAS + SC_DOUBLES + 1; }

// Reads the scalars of a finished solve.
static cudaError_t finish(CgScalars& st, const CgScalars* sc, PcgHost& host, double* x, int64_t n, int max_iter,
                          int* iterations, double* rel_residual, cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemcpyAsync(host.pinned, sc, sizeof(CgScalars), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return e;
  memcpy(&st, host.pinned, sizeof st);
  if (st.done < 0) return cudaErrorLaunchTimeout;  // a barrier of the one-launch solve gave up
  if (st.bb == 0.0) {  // x = 0 solves it
    *iterations = 0;
    *rel_residual = 0.0;
    return cudaMemsetAsync(x, 0, sizeof(double) * size_t(n), s);
  }
  *iterations = st.it;
  *rel_residual = max_iter > 0 ? std::sqrt(st.rr) / std::sqrt(st.bb) : 0.0;
  return cudaSuccess;
}

cudaError_t pcg(const CscSym& A, const double* b, double* x, double* scratch, int max_iter, double rtol,
                int check_every, bool jacobi, long long wait_budget, PcgHost& host, int* iterations,
                double* rel_residual, cudaStream_t s) {
  static_assert(sizeof(CgScalars) <= PcgHost::SLOT, "host slot");
  *iterations = 0;
  *rel_residual = 0.0;
  if (A.n == 0) return cudaSuccess;
  const int64_t n = A.n;
  double* r = scratch;
  double* z = r + n;
  double* p = z + n;
  double* y = p + n;
  double* inv_diag = jacobi ? y + n : nullptr;
  double* part_py = y + 2 * n;
  double* part_rz = part_py + MAX_CTAS;
  double* part_rr = part_rz + MAX_CTAS;
  CgScalars* sc = reinterpret_cast<CgScalars*>(part_rr + MAX_CTAS);
  const int64_t groups = (n + THREADS - 1) / THREADS, sms = num_sms() < MAX_CTAS ? num_sms() : MAX_CTAS;
  const unsigned gm = unsigned(groups < sms ? groups : sms);  // one CTA of the product per SM (shared memory)
  const unsigned gv = unsigned(groups < MAX_CTAS ? groups : MAX_CTAS);
  cudaError_t e;
  if ((e = host.ensure()) != cudaSuccess || (e = ensure_smem<cg_init_kernel>(ROWS_SMEM)) != cudaSuccess ||
      (e = ensure_smem<cg_product_kernel>(ROWS_SMEM)) != cudaSuccess)
    return e;
  CgScalars st;
  CoopShape shape;
  if (coop_shape(A, &shape)) {
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(sc) + SC_DOUBLES;
    if ((e = ensure_smem<cg_solve_kernel>(COOP_SMEM)) != cudaSuccess ||
        (e = cudaMemsetAsync(sc, 0, 8 * (SC_DOUBLES + 1), s)) != cudaSuccess)
      return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(shape.grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = COOP_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, cg_solve_kernel, A, shape.rows, b, x, p, jacobi ? 1 : 0, part_py, sc, bar, max_iter,
                           check_every, rtol, wait_budget > 0 ? wait_budget : COOP_BUDGET);
    if (e == cudaSuccess) return finish(st, sc, host, x, n, max_iter, iterations, rel_residual, s);
    if (e != cudaErrorCooperativeLaunchTooLarge) return e;
    cudaGetLastError();  // (a share of the device: fewer CTAs resident than SMs) the three kernels
  }
  cg_init_kernel<<<gm, THREADS, ROWS_SMEM, s>>>(A, b, x, r, z, p, inv_diag, part_rz, part_py);
  cg_start_kernel<<<1, THREADS, 0, s>>>(part_rz, part_py, int(gm), sc);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  // the scalars after batch k land in host slot k & 1
  auto read_back = [&](int k) {
    const cudaError_t e1 = cudaMemcpyAsync(static_cast<char*>(host.pinned) + (k & 1) * PcgHost::SLOT, sc,
                                           sizeof(CgScalars), cudaMemcpyDeviceToHost, s);
    return e1 != cudaSuccess ? e1 : cudaEventRecord(host.done[k & 1], s);
  };
  auto scalars = [&](int k, CgScalars* out) {
    const cudaError_t e1 = cudaEventSynchronize(host.done[k & 1]);
    if (e1 == cudaSuccess) memcpy(out, static_cast<char*>(host.pinned) + (k & 1) * PcgHost::SLOT, sizeof(CgScalars));
    return e1;
  };
  int it = 0, batch = 0;
  while (it < max_iter) {
    const int end = max_iter - it < check_every ? max_iter : it + check_every;
    while (it < end) {
      const int par = it & 1;
      if ((e = launch_next(cg_product_kernel, gm, ROWS_SMEM, s, A, p, y, part_py, sc)) != cudaSuccess) return e;
      if ((e = launch_next(cg_update_kernel, gv, 0, s, n, sc, par, part_py, int(gm), x, r, z, p, y, inv_diag, part_rz,
                           part_rr)) != cudaSuccess)
        return e;
      ++it;
      if (it == end && (e = launch_next(cg_test_kernel, 1u, 0, s, sc, part_rr, int(gv), it, rtol)) != cudaSuccess)
        return e;
      if ((e = launch_next(cg_direction_kernel, gv, 0, s, n, sc, par, part_rz, int(gv), z, p)) != cudaSuccess) return e;
    }
    if ((e = read_back(batch)) != cudaSuccess) return e;
    if (batch > 0) {  // the test of the batch before, while this one runs
      if ((e = scalars(batch - 1, &st)) != cudaSuccess) return e;
      if (st.done) break;
    }
    ++batch;
  }
  // (after a break the batch just enqueued changed nothing)
  return finish(st, sc, host, x, n, max_iter, iterations, rel_residual, s);
}

}  // namespace fec
