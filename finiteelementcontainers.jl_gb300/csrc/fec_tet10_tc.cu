// fec_tet10_tc.cu -- FP64 tet10 Neo-Hookean element stiffness on the tensor cores,
// for elements of any shape: the exact-digit contraction of fec_hex8_affine_tc.cu in
// reference coordinates (GenNeoHookean), whose constant operand
//     W[n, r] = dN_qaJ dN_qbL,   n = (a, b), a <= b (55 pairs),  r = (J, L, q) (36 values)
// is that of the reference element.
//
// Quadratic tets have a structure of their own.  The points of the symmetric 4-point
// rule each lie towards one vertex: with barycentrics a there and b towards the others
// (vertex_rule below), and x_mn the value at the mid node of edge mn (x_mm: at vertex m),
//     d x / d lambda_m at point q = B_m + c x_mq,   B_m = 4b sum_n x_mn - x_m,  c = 4 (a - b),
// so the four lanes of an element each load their vertex and its three edges, form one
// B, and share it: 15 FP64 operations a component instead of 30.  The residual is the
// transpose: with S = sum_q P_q and Y_m = 4b S + c P_m (JxW P in reference coordinates),
//     R_m = (Y_m - S) . grad lambda_m,   R_mn = Y_m . grad lambda_n + Y_n . grad lambda_m.
//
// One persistent CTA per SM, tiles of 24 elements (96 points, a thread each), which the
// MMAs take in two halves of 12 elements (M = 128 rows, laid out as in the hex8 kernel):
//   9 producers point phase in FP64, then, while the slicers work on the staging, the
//               residual;
//   6 slicers   a point's 45 unique tangent entries by two threads, parked in shared
//               memory; then, a half tile at a time, their digits into the A slices: a
//               thread takes one entry of an element at its four points, which are
//               neighbours in r, and stores 8 bytes per digit;
//   4 warps     the epilogue into the symmetric half (KE_PAIRS);
//   1 warp      issues 30 MMAs a half tile.
// What bounds it: the FP64 point phase, about 400 operations a point at 64 clocks a warp
// instruction and sub-partition (two thirds of the time a tile takes); the epilogue, the
// MMAs and the slicers each need about half of it.  55,062 distorted elements 0.252 ms
// (the per-element kernel 1.37), 82,368 of six translation classes 0.364 (the class
// kernel 1.19).
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "fec_digits.cuh"
#include "fec_kernels.cuh"
#include "fec_launch.h"
#include "fec_tc.cuh"

namespace fec {
namespace tet {

using namespace aff;
using Model = GenNeoHookean;

constexpr int NQ = 4, NNODE = 10, EPT = 24, HALF_EL = 12, NPT = EPT * NQ;
constexpr int KR = 36, KP = 48, NPAIR = 55, NPAD = 64;
constexpr int SBO = KP * 16;
constexpr int A_SLICE = 128 * KP * 2, W_SLICE = NPAD * KP * 2, W_BYTES = ND * W_SLICE;
constexpr int MAXS = 256 / NPAD;  // W digits in one MMA (N <= 256)
// table (tet10_general_table)
constexpr int T_W = 0, T_SIG = W_BYTES, T_B4 = T_SIG + NPAD * 4;  // 4b, c, weights [4] (double)
constexpr int T_BYTES = (T_B4 + 6 * 8 + 15) / 16 * 16;

// Producer warps take units of 8 elements (32 points), three to a tile, whichever the
// tile, and stage a unit in a buffer of their own.  Nine of them: with eight (two a
// sub-partition) the FP64 pipe idles for latency (8% longer on 55,062 elements;
// three groups of three warps, a tile each: 1%).
constexpr int NPROD = 9, UNITS = NPT / 32, UEL = EPT / UNITS, SL_W = 2 * UNITS, EP_W = 4;
constexpr int T_SL = 32 * NPROD, NSL = 32 * SL_W, T_EP = T_SL + NSL, T_MMA = T_EP + 32 * EP_W, NTHR = T_MMA + 32;
static_assert(NTHR <= 640, "roles");
constexpr int BAR_PARK = 1, BAR_DIGITS = 2;  // among the slicers: a tile parked, its digits done
constexpr int NENT = 45, N_HALF = 24;  // unique entries of a point; those of the first slicer thread (i = 0)

struct Lay {
  static constexpr int W = 0;
  static constexpr int A = W + W_BYTES;
  static constexpr int PARK = A + ND * A_SLICE;              // float2 [45][96]
  static constexpr int P = PARK + NENT * NPT * 8;            // float2 [NPROD][32][9]
  static constexpr int SCR = P + NPROD * 32 * 9 * 8;           // float2 [NPROD][32][SCR2]
  static constexpr int SIG = SCR + NPROD * 32 * Model::SCR2 * 8;  // float [64]: 2^(sigma - 7)
  static constexpr int TAUST = SIG + NPAD * 4;               // int [NPROD][8]: the staged units' scales
  static constexpr int TAUT = TAUST + NPROD * UEL * 4;       // int [24]: the parked tile's
  static constexpr int TAU = TAUT + EPT * 4;                 // int [2][12]: per half-tile parity
  static constexpr int CODE = TAU + 2 * HALF_EL * 4;         // uint32 [45][12]: where an entry's digits go
  static constexpr int BAR = (CODE + NENT * HALF_EL * 4 + 15) / 16 * 16;
  static constexpr int TSLOT = BAR + (3 + 2 * NPROD) * 8;
  static constexpr int SMEM = TSLOT + 16;
  static_assert(SMEM <= 232448 && PARK % 16 == 0, "shared memory");
};

// MMA row of element el of a half tile (as in the hex8 kernel: the odd quarters of 32
// rows start at row 3, which spreads the digit stores over the banks)
__host__ __device__ __forceinline__ int first_row(int el) { return el / 3 * 32 + 3 * (el / 3 & 1) + 9 * (el % 3); }
// byte offset of (row, col) in a K-major operand tile with K = 48
__host__ __device__ __forceinline__ uint32_t op_off(int row, int col) {
  return uint32_t(row >> 3) * SBO + uint32_t(col >> 3) * 128 + uint32_t(row & 7) * 16 + uint32_t(col & 7) * 2;
}
// the node at vertex m and vertex n (edge mn's mid node, or the vertex m = n)
__host__ __device__ __forceinline__ int node_at(int m, int n) {
  return int(0x3987925685147640ull >> (16 * m + 4 * n)) & 15;
}

struct Coef {
  double b4, c;
};
// d v / d xi at point q (lane q of the element's four), v[m]: the value at node_at(q, m)
// less node 0's
__device__ __forceinline__ void gradient(const Coef& k, int q, const double (&v)[4], double (&g)[3]) {
  const double own = q == 0 ? v[0] : q == 1 ? v[1] : q == 2 ? v[2] : v[3];
  const double B = fma(k.b4, (v[0] + v[1]) + (v[2] + v[3]), -own);
  double D[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) D[m] = fma(k.c, v[m], __shfl_sync(0xffffffffu, B, m, 4));
#pragma unroll
  for (int j = 0; j < 3; ++j) g[j] = D[j + 1] - D[0];
}

// Gradient of one component of nodal values x (the lane's four nodes).
__device__ __forceinline__ void gradient_of(const Coef& k, int q, const double (&x)[4], double (&g)[3]) {
  const double x0 = __shfl_sync(0xffffffffu, x[0], 0, 4);
  const double v[4] = {x[0] - x0, x[1] - x0, x[2] - x0, x[3] - x0};
  gradient(k, q, v, g);
}

// Point phase of point q of an element; X, uo: coordinates and displacements of the
// lane's four nodes (0 where not live).  Every lane of the warp calls it.
__device__ __forceinline__ void point_phase(const ElemArgs& g, const Coef& k, double w, int q, bool live,
                                            const double (&X)[3][4], const double (&uo)[3][4], Model::Mid& m) {
  double G[3][3], D[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) gradient_of(k, q, X[d], G[d]);
#pragma unroll
  for (int d = 0; d < 3; ++d) gradient_of(k, q, uo[d], D[d]);
  if (live) ref_point(g.props, G, D, w, m);
}

// Component i of the element's residual from row i of JxW P at the lane's point, in FP64
// (the double-float sums' own rounding showed in the assembled residual): the lane's
// vertex, and the edges to the vertices after its own.
__device__ __forceinline__ void residual_row(const Coef& k, int q, bool live, const double (&p)[3], double* Re) {
  double z[4], own[3];  // grad lambda_m . Y
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    double S = p[j] + __shfl_xor_sync(0xffffffffu, p[j], 1);
    S = S + __shfl_xor_sync(0xffffffffu, S, 2);
    z[j + 1] = fma(k.b4, S, mul_rn(k.c, p[j]));
    own[j] = z[j + 1] - S;
  }
  z[0] = -((z[1] + z[2]) + z[3]);
  const double o0 = -((own[0] + own[1]) + own[2]);
  if (live) Re[q * 3] = q == 0 ? o0 : q == 1 ? own[0] : q == 2 ? own[1] : own[2];
#pragma unroll
  for (int d = 1; d < 4; ++d) {
    // (the lane across wants its own gradient of this lane's Y)
    const int m = q ^ d;
    const double t = m == 0 ? z[0] : m == 1 ? z[1] : m == 2 ? z[2] : z[3];
    const double e = t + __shfl_xor_sync(0xffffffffu, t, d);
    if (live && q < m) Re[node_at(q, m) * 3] = e;
  }
}

// A point's scaled entries of one half into the parking space (stride NPT).
template <int HALF>
__device__ __forceinline__ void park(const float2* scr, const float2* P, float fs, float2* out) {
  Model::Tangent t;
  Model::load(scr, P, t);
#pragma unroll
  for (int r1 = 0; r1 < 9; ++r1)
#pragma unroll
    for (int r2 = r1; r2 < 9; ++r2) {
      const int c = r1 * 9 - r1 * (r1 - 1) / 2 + r2 - r1;
      if ((c >= N_HALF) != (HALF == 1)) continue;
      const float2 a = Model::entry(t, r1 / 3, r1 % 3, r2 / 3, r2 % 3);
      out[c * NPT] = make_float2(a.x * fs, a.y * fs);
    }
}

// the part of (xh, xl) at or above 2^(-8s), taken off (by adding and subtracting
// 1.5 2^(23-8s)); |xl| <= 2^-18 has no digits before the third
__device__ __forceinline__ uint32_t take_digit(int s, float& xh, float& xl) {
  const float big = pow2f(23 - 8 * s) * 1.5f;
  float d = __fsub_rn(__fadd_rn(xh, big), big);
  xh = __fsub_rn(xh, d);
  if (s >= 3) {
    const float dl = __fsub_rn(__fadd_rn(xl, big), big);
    xl = __fsub_rn(xl, dl);
    d = __fadd_rn(d, dl);
  }
  return __float_as_uint(d);
}

template <bool WANT_R>
__global__ void __launch_bounds__(NTHR, 1) tet10_tc_kernel(ElemArgs g, const unsigned char* __restrict__ tab) {
  using namespace tc;
  constexpr int SCR2 = Model::SCR2;
  extern __shared__ __align__(1024) unsigned char sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t s0 = smem_u32(sm);
  float2* s_park = reinterpret_cast<float2*>(sm + Lay::PARK);
  float2* s_P = reinterpret_cast<float2*>(sm + Lay::P);
  float2* s_scr = reinterpret_cast<float2*>(sm + Lay::SCR);
  float* s_sig = reinterpret_cast<float*>(sm + Lay::SIG);
  int* s_taust = reinterpret_cast<int*>(sm + Lay::TAUST);
  int* s_taut = reinterpret_cast<int*>(sm + Lay::TAUT);
  int* s_tau = reinterpret_cast<int*>(sm + Lay::TAU);
  uint32_t* s_code = reinterpret_cast<uint32_t*>(sm + Lay::CODE);
  uint64_t* bar_sl = reinterpret_cast<uint64_t*>(sm + Lay::BAR);  // slices of a half tile written
  uint64_t* bar_mma = bar_sl + 1;                                  // its MMAs complete (and their issuer saw its slices)
  uint64_t* bar_tfree = bar_sl + 2;                                // the epilogue read its accumulators
  uint64_t* bar_full = bar_sl + 3;                                 // per producer: a unit staged
  uint64_t* bar_empty = bar_full + NPROD;                          // and read by the slicers

  // ---- setup: A slices zero (padding rows and columns stay zero), W digits, tables ----
  for (int i = tid; i < ND * A_SLICE / 16; i += NTHR)
    reinterpret_cast<uint4*>(sm + Lay::A)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < W_BYTES / 16; i += NTHR)
    reinterpret_cast<uint4*>(sm + Lay::W)[i] = __ldg(reinterpret_cast<const uint4*>(tab + T_W) + i);
  if (tid < NPAD) s_sig[tid] = pow2f(__ldg(reinterpret_cast<const int*>(tab + T_SIG) + tid) - 7);
  if (tid < NENT * HALF_EL) {
    // unique entry (r1, r2), r1 = 3i + J <= r2 = 3k + L, of element el: the operand
    // positions (row 3i + k, columns of (J, L)) and (row 3k + i, columns of (L, J)) as
    // byte offsets, low and high half
    const int r0 = first_row(tid % HALF_EL);
    int m = tid / HALF_EL, r = 0;
    for (int c = 0; c < 9; ++c)
      if (m >= 9 - r) { m -= 9 - r; ++r; }
    const int i = r / 3, J = r % 3, k = (r + m) / 3, L = (r + m) % 3;
    s_code[tid] = op_off(r0 + i * 3 + k, (J * 3 + L) * NQ) | op_off(r0 + k * 3 + i, (L * 3 + J) * NQ) << 16;
  }
  if (tid == 0) {
    mbar_init(bar_sl, NSL);
    mbar_init(bar_mma, 2);
    mbar_init(bar_tfree, 32 * EP_W);
    for (int i = 0; i < NPROD; ++i) {
      mbar_init(bar_full + i, 32);
      mbar_init(bar_empty + i, 64);
    }
    mbar_fence_init();
  }
  if (warp == T_EP / 32) tmem_alloc(reinterpret_cast<uint32_t*>(sm + Lay::TSLOT), 512);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(sm + Lay::TSLOT);
  const int64_t ntiles = (g.ne + EPT - 1) / EPT;
  const long long budget = g.wait_budget > 0 ? g.wait_budget : WAIT_BUDGET;
  // a wait that gave up reports through the flag and waits again (the long
  // budget) so that no buffer is reused under an operation in flight
  auto wait_or_report = [&](uint64_t* bar, uint32_t par) {
    if (!mbar_wait(bar, par, budget)) {
      if (g.wait_err) atomicExch(g.wait_err, 1);
      mbar_wait(bar, par, WAIT_BUDGET);
    }
  };
  // half tiles of a tile (the second one of the last tile may be empty)
  auto halves = [&](int64_t tile) { return tile * EPT + HALF_EL < g.ne ? 2 : 1; };

  if (tid < T_SL) {
    // ---------------- producers: warp p takes the units p, p + NPROD, ...; lane (el, q) ----------------
    const int q = lane & 3, sp = tid;  // the staged point
    const double* T = reinterpret_cast<const double*>(tab + T_B4);
    const Coef co = {__ldg(T), __ldg(T + 1)};
    const double w = __ldg(T + 2 + q);
    // the nodes of the warp's next unit are fetched while it computes this one
    int node[4];
    auto element_of = [&](int u) {
      const int64_t tile = blockIdx.x + int64_t(u / UNITS) * gridDim.x;
      return tile < ntiles ? tile * EPT + u % UNITS * UEL + (lane >> 2) : int64_t(-1);
    };
    auto nodes_of = [&](int64_t e) {
#pragma unroll
      for (int m = 0; m < 4; ++m) node[m] = e >= 0 && e < g.ne ? g.conn[e * NNODE + node_at(q, m)] : 0;
    };
    nodes_of(element_of(warp));
    for (int u = warp, use = 0;; u += NPROD, ++use) {
      const int64_t e = element_of(u);
      if (e < 0) break;
      const bool live = e < g.ne;
      double X[3][4], uo[3][4];
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          X[d][m] = live ? __ldg(&g.coords[int64_t(node[m]) * 3 + d]) : 0.0;
          uo[d][m] = live ? __ldg(&g.U[int64_t(node[m]) * 3 + d]) : 0.0;
        }
      nodes_of(element_of(u + NPROD));
      Model::Mid mid;
      point_phase(g, co, w, q, live, X, uo, mid);
      if (use) wait_or_report(bar_empty + warp, uint32_t((use - 1) & 1));  // the last unit has been read
      float bnd = 0.f;
      double P[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) P[i] = 0.0;
      if (live) {
        float2 P2[9];
        bnd = Model::stage(mid, P2, s_scr + sp * SCR2) * 1.0001f;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          s_P[sp * 9 + i] = P2[i];
          P[i] = mid.P[i];
        }
      }
      // the element's scale 2^tau > |every tangent entry|
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) bnd = fmaxf(bnd, __shfl_xor_sync(0xffffffffu, bnd, o));
      if (q == 0) {
        int tau = 0;
        if (bnd > 0.f) frexpf(bnd, &tau);
        s_taust[warp * UEL + (lane >> 2)] = tau < -119 ? -119 : (tau > 126 ? 126 : tau);
      }
      mbar_arrive(bar_full + warp);
      if (WANT_R) {  // while the slicers work on the staging
        double* Re = static_cast<double*>(g.Re) + e * (3 * NNODE);
#pragma unroll 1
        for (int i = 0; i < 3; ++i) {
          const double p[3] = {P[0], P[1], P[2]};
          residual_row(co, q, live, p, Re + i);
#pragma unroll
          for (int j = 0; j < 6; ++j) P[j] = P[j + 3];
        }
      }
    }
  } else if (tid < T_EP) {
    // ---------------- slicers ----------------
    const int ts = tid - T_SL, half = ts / NPT, p = ts - half * NPT;
    int hh = 0;  // half tiles done
    for (int k = 0;; ++k) {
      const int64_t tile = blockIdx.x + int64_t(k) * gridDim.x;
      if (tile >= ntiles) break;
      // pass 1 (overlaps the last half tile's MMAs): lane = point of a unit, the scaled entries parked
      const int u = k * UNITS + p / 32, buf = u % NPROD, sp = buf * 32 + lane;
      wait_or_report(bar_full + buf, uint32_t(u / NPROD & 1));
      const int tau = s_taust[buf * UEL + (lane >> 2)];
      const float fs = tile * EPT + (p >> 2) < g.ne ? pow2f(7 - tau) : 0.f;  // entries scaled to |x| < 128
      if (k) named_sync(BAR_DIGITS, NSL);
      if (half == 0) {
        if ((lane & 3) == 0) s_taut[p >> 2] = tau;
        park<0>(s_scr + sp * SCR2, s_P + sp * 9, fs, s_park + p);
      } else {
        park<1>(s_scr + sp * SCR2, s_P + sp * 9, fs, s_park + p);
      }
      mbar_arrive(bar_empty + buf);
      named_sync(BAR_PARK, NSL);
      // pass 2: the digits of each half tile, once the MMAs before it have read the slices
      const int nh = halves(tile);
      for (int h = 0; h < nh; ++h, ++hh) {
        if (hh >= 1) wait_or_report(bar_mma, uint32_t((hh - 1) & 1));
        if (ts < HALF_EL) s_tau[(hh & 1) * HALF_EL + ts] = s_taut[h * HALF_EL + ts];
#pragma unroll 1
        for (int it = ts; it < NENT * HALF_EL; it += NSL) {
          const int c = it / HALF_EL, el = it - c * HALF_EL;
          const float4* src = reinterpret_cast<const float4*>(s_park + c * NPT + (h * HALF_EL + el) * NQ);
          const float4 a = src[0], b = src[1];
          float xh[4] = {a.x, a.z, b.x, b.z}, xl[4] = {a.y, a.w, b.y, b.w};
          const uint32_t at = s_code[it];
          unsigned char* p1 = sm + Lay::A + (at & 0xffffu);
          unsigned char* p2 = sm + Lay::A + (at >> 16);
          const bool twin = p1 != p2;
#pragma unroll
          for (int s = 0; s < ND; ++s) {
            uint32_t u[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = take_digit(s, xh[j], xl[j]);
            const uint2 d = make_uint2(__byte_perm(u[0], u[1], 0x7632), __byte_perm(u[2], u[3], 0x7632));
            *reinterpret_cast<uint2*>(p1 + s * A_SLICE) = d;
            if (twin) *reinterpret_cast<uint2*>(p2 + s * A_SLICE) = d;
          }
        }
        fence_async_smem();
        mbar_arrive(bar_sl);
      }
    }
  } else if (tid < T_MMA) {
    // ---------------- epilogue: thread = TMEM lane = row (el, i, k) ----------------
    const int qw = warp & 3;
    const int row = lane - 3 * (qw & 1);  // of the quarter's 27
    const bool used = row >= 0 && row < 27;
    const int el = qw * 3 + (used ? row / 9 : 0), ik = used ? row % 9 : 0;
    const uint32_t lane_addr = tmem + (uint32_t(qw * 32) << 16);
    int hh = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const int nh = halves(tile);
      for (int h = 0; h < nh; ++h, ++hh) {
        const uint32_t par = uint32_t(hh & 1);
        const int64_t e = tile * EPT + h * HALF_EL + el;
        const bool live = used && e < g.ne;
        wait_or_report(bar_mma, par);  // (alone, as in the hex8 kernel)
        tc_fence_after();
        const float f1 = pow2f(s_tau[par * HALF_EL + el] - 7);
        float2* dst = static_cast<float2*>(g.Ke) + e * (NPAIR * 9) + ik;
#pragma unroll 1
        for (int n0 = 0; n0 < NPAIR; n0 += 4) {
          float v[NLEV][4];
          tmem_ld4x7<NPAD>(lane_addr + uint32_t(n0), v);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 hl = combine_levels(v, j);
            const float f = f1 * s_sig[n0 + j];
            if (live && n0 + j < NPAIR) dst[(n0 + j) * 9] = make_float2(hl.x * f, hl.y * f);
          }
        }
        tc_fence_before();
        mbar_arrive(bar_tfree);  // the accumulators may be overwritten
      }
    }
  } else {
    // ---------------- MMA warp: lane 0 issues, the warp waits together ----------------
    const uint64_t dA = smem_desc(s0 + Lay::A, 128, SBO), dW = smem_desc(s0 + Lay::W, 128, SBO);
    int hh = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
      const int nh = halves(tile);
      for (int h = 0; h < nh; ++h, ++hh) {
        wait_or_report(bar_sl, uint32_t(hh & 1));  // the slices are written
        tc_fence_after();
        if (hh >= 1) {
          wait_or_report(bar_tfree, uint32_t((hh - 1) & 1));  // the accumulators are free
          tc_fence_after();
        }
        if (lane == 0) {
          // A digit t against up to four W digits s .. at once; every pair s + t <= 6 once
#pragma unroll 1
          for (int t = 0; t < ND; ++t)
#pragma unroll 1
            for (int s = 0; s < ND - t; s += MAXS) {
              const int ns = ND - t - s < MAXS ? ND - t - s : MAXS;
              const uint32_t idesc = idesc_bf16(128, NPAD * ns);
              const uint64_t a0 = dA + uint64_t((t * A_SLICE) >> 4), ws = dW + uint64_t((s * W_SLICE) >> 4);
#pragma unroll
              for (int kk = 0; kk < KP / 16; ++kk)
                mma_bf16(tmem + uint32_t((s + t) * NPAD), a0 + uint64_t(kk * 16), ws + uint64_t(kk * 16), idesc,
                         (t == 0 && kk == 0) ? 0u : 1u);
            }
          mma_commit(bar_mma);
          mbar_arrive(bar_mma);  // (passes on what the slicers wrote before the slices: the scales)
        }
        __syncwarp();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == T_EP / 32) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Residual only: the same point phase and residual arithmetic, so the same bits.  One
// thread per point.
constexpr int R_THR = 128;
__global__ void __launch_bounds__(R_THR) tet10_r_kernel(ElemArgs g, const unsigned char* __restrict__ tab) {
  const int64_t p = int64_t(blockIdx.x) * R_THR + threadIdx.x, e = p >> 2;
  const int q = int(p & 3);
  const bool live = e < g.ne;
  const double* T = reinterpret_cast<const double*>(tab + T_B4);
  const Coef co = {__ldg(T), __ldg(T + 1)};
  double X[3][4], uo[3][4];
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int64_t n = live ? g.conn[e * NNODE + node_at(q, m)] : 0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      X[d][m] = live ? __ldg(&g.coords[n * 3 + d]) : 0.0;
      uo[d][m] = live ? __ldg(&g.U[n * 3 + d]) : 0.0;
    }
  }
  Model::Mid mid;
  point_phase(g, co, __ldg(T + 2 + q), q, live, X, uo, mid);
  double* Re = static_cast<double*>(g.Re) + e * (3 * NNODE);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double p[3] = {0.0, 0.0, 0.0};
    if (live)
#pragma unroll
      for (int j = 0; j < 3; ++j) p[j] = mid.P[i * 3 + j];
    residual_row(co, q, live, p, Re + i);
  }
}

template <bool WANT_R>
cudaError_t launch(const ElemArgs& a, cudaStream_t s) {
  const cudaError_t e = ensure_smem<tet10_tc_kernel<WANT_R>>(Lay::SMEM);
  if (e != cudaSuccess) return e;
  const int64_t ntiles = (a.ne + EPT - 1) / EPT;
  const int grid = int(ntiles < num_sms() ? ntiles : num_sms());
  tet10_tc_kernel<WANT_R><<<grid, NTHR, Lay::SMEM, s>>>(a, static_cast<const unsigned char*>(a.general));
  return cudaGetLastError();
}

// d N_a / d xi_j at barycentrics l
double shape_gradient(int a, int j, const double l[4]) {
  for (int m = 0; m < 4; ++m)
    for (int n = m; n < 4; ++n) {
      if (node_at(m, n) != a) continue;
      auto gl = [&](int v) { return v == 0 ? -1.0 : (v == j + 1 ? 1.0 : 0.0); };  // d lambda_v / d xi_j
      return m == n ? (4.0 * l[m] - 1.0) * gl(m) : 4.0 * (l[m] * gl(n) + l[n] * gl(m));
    }
  return 0.0;
}

// Whether the reference tables are those of the quadratic tet at four points, one
// towards each vertex (barycentrics 1 - 3b there and b towards the others): the point of
// each vertex, and b.
bool vertex_rule(const double* ref, int point[4], double& b) {
  const double* dN = ref + RefLayout<7>::DN_OFF;
  bool have[4] = {false, false, false, false};
  double l[4][4];
  for (int q = 0; q < NQ; ++q) {
    const double* D = dN + q * NNODE * 3;
    l[q][0] = 0.25 * (1.0 - D[0]);
    for (int m = 1; m < 4; ++m) l[q][m] = 0.25 * (1.0 + D[m * 3 + m - 1]);
    int v = 0;
    for (int m = 1; m < 4; ++m)
      if (l[q][m] > l[q][v]) v = m;
    if (have[v]) return false;
    have[v] = true;
    point[v] = q;
  }
  b = l[point[0]][1];
  for (int v = 0; v < 4; ++v) {
    double at[4] = {b, b, b, b};
    at[v] = 1.0 - 3.0 * b;
    for (int a = 0; a < NNODE; ++a)
      for (int j = 0; j < 3; ++j)
        if (!(std::fabs(dN[(point[v] * NNODE + a) * 3 + j] - shape_gradient(a, j, at)) <= 4e-15)) return false;
  }
  return true;
}

}  // namespace tet

bool tet10_general_enabled() {
  const char* v = std::getenv("FEC_TET10_GENERAL");
  return !(v && v[0] == '0');
}

cudaError_t launch_tet10_general(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (!a.general || (want_k && !a.Ke) || (want_r && !a.Re)) return cudaErrorInvalidValue;
  if (a.ne <= 0 || (!want_r && !want_k)) return cudaSuccess;
  ++*launches;
  if (want_k) return want_r ? tet::launch<true>(a, s) : tet::launch<false>(a, s);
  const int64_t nb = (a.ne * tet::NQ + tet::R_THR - 1) / tet::R_THR;
  tet::tet10_r_kernel<<<unsigned(nb), tet::R_THR, 0, s>>>(a, static_cast<const unsigned char*>(a.general));
  return cudaGetLastError();
}

bool tet10_general_table(const double* ref, std::vector<unsigned char>& out) {
  using namespace tet;
  int point[4];
  double b;
  if (!vertex_rule(ref, point, b)) return false;
  out.assign(T_BYTES, 0);
  const double* dN = ref + RefLayout<7>::DN_OFF;
  const double* wq = ref + RefLayout<7>::W_OFF;
  int32_t sig[NPAD] = {0};
  for (int a = 0, n = 0; a < NNODE; ++a)
    for (int bb = a; bb < NNODE; ++bb, ++n) {
      double w[KR], mx = 0.0;
      for (int r = 0; r < KR; ++r) {  // r = (J, L, q), q the point's vertex
        const int q = point[r % NQ], J = r / NQ / 3, L = r / NQ % 3;
        w[r] = dN[(q * NNODE + a) * 3 + J] * dN[(q * NNODE + bb) * 3 + L];
        mx = std::fmax(mx, std::fabs(w[r]));
      }
      int e = 0;
      if (mx > 0.0) std::frexp(mx, &e);  // |w| < 2^e
      if (e < -119 || e > 134) return false;  // the epilogue scales by 2^(e - 7) in FP32
      sig[n] = e;
      for (int r = 0; r < KR; ++r) {
        uint16_t bits[ND];
        bf16_digits(w[r], e, bits);
        for (int s = 0; s < ND; ++s) std::memcpy(out.data() + T_W + s * W_SLICE + op_off(n, r), &bits[s], 2);
      }
    }
  double co[6] = {4.0 * b, 4.0 * (1.0 - 4.0 * b), wq[point[0]], wq[point[1]], wq[point[2]], wq[point[3]]};
  std::memcpy(out.data() + T_SIG, sig, sizeof sig);
  std::memcpy(out.data() + T_B4, co, sizeof co);
  return true;
}

}  // namespace fec
