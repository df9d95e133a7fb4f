// fec_hex8_affine_tc.cu -- FP64-accurate hex8 element stiffness on the tensor
// cores for blocks whose elements are translates of one another (structured
// meshes), by exact integer slicing of both operands (the Ozaki scheme: Ozaki,
// Ogita, Oishi and Rump, Numer. Algorithms 59 (2012) 95-118, restated here for
// BF16 digits and FP32 accumulation).
//
// The tangent of element e is (src/Formulations.jl:462-576)
//     K_(a,i),(b,k) = sum_q sum_(J,L) dNX_qaJ * JxW A_q,iJkL * dNX_qbL .
// With every element a translate of the first, dNX_q and JxW_q are the same for
// all elements, so with r = (q, J, L) (72 values) and the node pair n = (a, b),
// a <= b (36 pairs: the rest follow from K = K^T),
//     D[(e, i, k), n] = sum_r A_e[(e, i, k), r] * W[n, r],   W[n, r] = dNX_qaJ dNX_qbL,
// one GEMM over all elements with a constant right operand.  Each A row (one
// element, scaled by a power of two 2^tau_e over the element's largest entry)
// and each W row (2^sigma_n) is written as seven signed 8-bit digits,
//     x = 2^tau * sum_t d_t 2^(-7-8t),  |d_t| <= 256,
// every digit exact in BF16.  A digit product is an integer below 2^16 and a
// 72-term dot product of digits below 2^23, so the sums over r of all digit
// pairs with s + t = L (at most seven pairs, each with |d| <= 256 in one digit
// position per value at most) stay below 2^24: each level L = 0..6 accumulates
// exactly in its own FP32 TMEM accumulator.  Levels above 6 are dropped
// (contributions below 2^-56 of the scales); the epilogue sums the seven levels
// in double-float and scales by 2^(tau_e + sigma_n - 14).
//
// One persistent CTA per SM, tiles of 12 elements.  MMA row 32 w + 9 j + ik (3 more
// where w is odd, see quarter_start) holds (element 3 w + j, ik = 3 i + k): every
// element's nine rows lie in one warp's TMEM lanes, the other five are padding.
//   producers   FP64 point phase (displacement gradient, constitutive update),
//               one thread per quadrature point: two or three groups of three warps
//               take the tiles in turn, each with a staging buffer of its own; then,
//               while the slicers read it, the residual R = sum_q dNX P in
//               double-float;
//   6 slicers   two threads per point: tangent entries (45 unique, double-float),
//               parked in TMEM, then (once the previous tile's MMAs read the
//               slices) their digits into the seven A slices;
//   4 warps     the epilogue: TMEM -> double-float values (row (e, i, k) holds
//               K_(a,i),(b,k) for a <= b), stored as they leave tensor memory:
//               the symmetric half (KE_PAIRS, entry 9n + 3i + k of pair n), or
//               each value at its two places in the node rows of the whole K_e;
//   1 warp      issues the tile's 45 MMAs.
// The A slices are rewritten as soon as the MMAs that read them completed; the
// next MMAs wait only for the epilogue's reads of the accumulators.
//
// What bounds it: every role is near the tile period (about 14k SM clocks a tile of
// 12 elements), and straight-line code is what they all pay for -- five warps of a
// sub-partition run different code, which does not fit the instruction cache, at
// about five clocks an instruction.  So the loops that can be small are kept small: one
// entry's digits (four at once: 9.0 ms instead of 8.1), the MMA issue (unrolled: 9.4), one
// residual component (three: 8.7); ncu's no-instruction stalls went from 3.3 to 0.9 per
// issue.  Now FP64 pipe 49%, 2.3 instructions a clock, tensor pipe 23%.  128^3 Neo-Hookean: 8.1 ms; 64 x 56 x 60 J2: 0.85 ms.
// Elements of any shape (GenNeoHookean) map every point in FP64 too: 61 x 53 x 47 0.98 ms, the
// FP64 pipe 78% (the per-element kernel 1.60).
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <cmath>
#include <type_traits>
#include <vector>

#include "fec_digits.cuh"
#include "fec_kernels.cuh"
#include "fec_launch.h"
#include "fec_tc.cuh"

namespace fec {
namespace aff {

constexpr int EPT = 12;              // elements per tile (three per 32-row quarter)
constexpr int NQ = 8;
constexpr int NPT = EPT * NQ;        // quadrature points per tile (96)
constexpr int KR = 72, KP = 80;      // reduction length r = (J, L, q), q fastest, padded to 5 K steps
constexpr int NPAIR = 36, NPAD = 48; // node pairs a <= b, padded N
constexpr int SBO = KP * 16;         // bytes between 8-row groups of an operand tile
constexpr int A_SLICE = 128 * KP * 2;
constexpr int W_SLICE = NPAD * KP * 2;
constexpr int MAXS = 256 / NPAD;     // W digits in one MMA (N <= 256)
constexpr int W_BYTES = ND * W_SLICE;
// table built on the host (hex8_affine_table): W digits, sigma, dNX, JxW
constexpr int T_W = 0;
constexpr int T_SIG = W_BYTES;
constexpr int T_G = T_SIG + NPAD * 4;
constexpr int T_JXW = T_G + NQ * 24 * 8;
constexpr int T_TEN = T_JXW + NQ * 8;           // TEN_N doubles, see tensor_gradient
constexpr int TEN_N = 10 + 2 + NQ * 9;          // coefficients, box flag, separable-point flag, Ji [q][k][j]
constexpr int T_OFF = T_TEN + TEN_N * 8;        // X_q - X_0 [q][3]
constexpr int T_N = T_OFF + NQ * 24;            // shape functions [q][a]
constexpr int T_K = T_N + NQ * 64;              // Poisson's element matrix [a][b]
constexpr int T_BYTES = T_K + 64 * 8;
static_assert(T_BYTES % 16 == 0 && T_G % 8 == 0, "table layout");
constexpr int TMEM_COLS = 512;
constexpr int TM_ENT = NLEV * NPAD;  // 96 columns after the accumulators: the slicers' scaled tangent entries (hi, lo)
static_assert(TM_ENT + 96 <= TMEM_COLS, "tensor memory columns");

// Warps.  Five warps a sub-partition leave 96 registers a thread.  Two or three
// groups of producers, by what the physics costs them; a slicer thread takes half of
// a point's entries.
constexpr int PROD_W = 3, EP_W = 4, MMA_W = 1, NSL = 2 * NPT;
template <class Model>
struct Roles {
  static constexpr int PG = Model::PROD_GROUPS;
  static constexpr int T_SL = 32 * PROD_W * PG, T_EP = T_SL + NSL, T_MMA = T_EP + 32 * EP_W, NTHR = T_MMA + 32 * MMA_W;
  static constexpr int N_SL = 32 * PROD_W + NSL;  // a producer group and the slicers
  static constexpr int EMPTY = 1 + PG;            // first EMPTY barrier
  static_assert(32 * PROD_W == NPT && NTHR <= 640, "roles");
};
// named barriers (0 is __syncthreads), each + the producer group
constexpr int BAR_FULL = 1;  // the group arrives, slicers sync: a tile staged
                             // Roles::EMPTY: slicers arrive, the group syncs: the buffer of its next tile read

// The MMAs of a tile: A digit t against up to five W digits s0 .. at once
// (consecutive W slices are consecutive 48-row blocks, one N = 48 ns operand),
// accumulating into levels s0+t .. (consecutive 48-column blocks).  Every pair s + t <=
// 6 once; the t = 0 ones write each level first.  (The pairs in three subsets of 16
// with barriers of their own, so that the epilogue of one overlaps the MMAs of the
// next, were slower: 105 MMAs read A from shared memory 105 instead of 45 times,
// 9-10k against 5k clocks a tile.)

// MMA row of (element el of the tile, ik = 3 i + k) within its quarter of 32 rows.
// The odd quarters start at row 3: the four elements of a slicer warp then lie in
// different eighths of the 128-byte core matrices, so their digit stores hit
// different banks (the stores share the shared-memory pipe with the MMAs' reads).
__host__ __device__ __forceinline__ int quarter_start(int quarter) { return 3 * (quarter & 1); }

struct AffJ2 {
  static constexpr int NS = J2::NS, SCR2 = J2::SCR2;
  static constexpr bool TANGENT_P = false;
  static constexpr bool GENERAL = false, TENSOR = true;
  static constexpr int PROD_GROUPS = 3, STAGES = 3;
  struct Mid {
    double P[9], scr[J2::SCR];
  };
  __device__ static void point(const double* props, double (&gu)[3][3], double jxw, const double* so, double* sn,
                               Mid& m) {
    J2::point(props, gu, jxw, so, sn, m.P, m.scr);
  }
  __device__ static void stress(const Mid& m, float2* P) {
#pragma unroll
    for (int i = 0; i < 9; ++i) P[i] = df64_split(m.P[i]);
  }
  __device__ static void action(const Mid& m, const double (&D)[3][3], double (&out)[3][3]) {
    J2::action(m.scr, D, out);
  }
  __device__ static float stage(const Mid& m, float2* P, float2* scr) {
    stress(m, P);
    J2::split_scratch(m.scr, scr);
    return J2::abound(scr);
  }
  struct Tangent {
    float2 s[SCR2];
  };
  __device__ static void load(const float2* scr, const float2*, Tangent& t) {
#pragma unroll
    for (int i = 0; i < SCR2; ++i) t.s[i] = scr[i];
  }
  __device__ static float2 entry(const Tangent& t, int i, int J, int k, int L) {
    return J2::aentry_df64(t.s, i, J, k, L);
  }
};

// The same on a block of translated elements with 8-point tables that are not a symmetric
// rule's (points in another order, any other points): gradients and residual by sums over
// the block's own dNX, read from its table.  An assembly of 128^3 such elements 17.2 ms
// (11.6 with a symmetric rule's tables, 25.4 with the per-element kernels).
template <class Model>
struct AnyRule : Model {
  static constexpr bool TENSOR = false;
};

template <class Model>
struct Layout {
  static constexpr int W = 0;
  static constexpr int A = W + W_BYTES;
  static constexpr int NB = Model::STAGES;                        // staging buffers
  static constexpr int P = A + ND * A_SLICE;                      // float2 [NB][96][9] (where the slicers read it)
  static constexpr int SCR = P + (Model::TANGENT_P ? NB * NPT * 9 * 8 : 0);  // float2 [NB][96][SCR2]
  static constexpr int TEN = (SCR + NB * NPT * Model::SCR2 * 8 + 15) / 16 * 16;  // double [TEN_N]
  static constexpr int TEN2 = TEN + TEN_N * 8;                    // float2 [10]: the coefficients split
  static constexpr int JXW = TEN2 + 10 * 8;                    // double [8]
  static constexpr int SIG = JXW + NQ * 8;                        // float [48]: 2^(sigma - 7)
  static constexpr int TAU = SIG + NPAD * 4;                      // int [2][12]: per tile parity
  static constexpr int TAUST = TAU + 2 * 16 * 4;                  // int [NB][12]: the staged tiles' scales
  static constexpr int CODE = TAUST + NB * 16 * 4;                     // uint32 [6][48] where an entry's digits go
  static constexpr int BAR = (CODE + 6 * 48 * 4 + 15) / 16 * 16;  // mbarriers: slices, MMAs, TMEM read
  static constexpr int TSLOT = BAR + 32;
  static constexpr int SMEM = TSLOT + 16;
  static_assert(SMEM <= 232448, "shared memory");
};

// byte offset of element (row, col) in a K-major operand tile with K = 80
__host__ __device__ __forceinline__ uint32_t op_off(int row, int col) {
  return uint32_t(row >> 3) * SBO + uint32_t(col >> 3) * 128 + uint32_t(row & 7) * 16 + uint32_t(col & 7) * 2;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
               "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
               "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
               : "memory");
}
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, float& a, float& b) {
  uint32_t r[2];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(taddr)
               : "memory");
  a = __uint_as_float(r[0]);
  b = __uint_as_float(r[1]);
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }


// Node of an element at the corner in point q's octant (bits x, y, z of q).
__device__ __forceinline__ int corner_node(int q) { return q ^ ((q >> 1) & 1); }

// -d where the bit is clear
__device__ __forceinline__ double signed_by(double d, unsigned bit) {
  return __hiloint2double(__double2hiint(d) ^ int(bit ? 0u : 0x80000000u), __double2loint(d));
}

// Gradient at point q of the nodal values of an element, shared by its eight
// lanes (consecutive, aligned to 8): lane q holds v = the value at corner q minus
// node 0's.  The point rule is symmetric (points at -t_d, t_d per direction), so a
// trilinear value is interpolated (I) or differenced (D) one direction at a time,
// the other value coming from the lane across: gx = I_z I_y D_x v, gy = I_z D_y
// I_x v, gz = D_z I_y I_x v.  13 FP64 operations per component instead of the 24 of
// sum_a v_a dN_a, which is what counts: the FP64 pipe takes a sub-partition 64
// clocks per warp instruction.  Differences of values come first, so the
// result is no further from the exact gradient.  co: I_x (own, across), I_y, then
// I_y, I_z, I_z with the scales of gz, gy, gx folded in.
__device__ __forceinline__ void tensor_gradient1(const double* co, int q, double v, double& gx, double& gy, double& gz) {
  const double vx = __shfl_xor_sync(0xffffffffu, v, 1);
  const double A = fma(co[0], v, mul_rn(co[1], vx)), B = signed_by(v - vx, q & 1);
  const double Ay = __shfl_xor_sync(0xffffffffu, A, 2), By = __shfl_xor_sync(0xffffffffu, B, 2);
  const double C = fma(co[4], A, mul_rn(co[5], Ay)), D = signed_by(A - Ay, q & 2);
  const double E = fma(co[2], B, mul_rn(co[3], By));
  const double Cz = __shfl_xor_sync(0xffffffffu, C, 4), Dz = __shfl_xor_sync(0xffffffffu, D, 4),
               Ez = __shfl_xor_sync(0xffffffffu, E, 4);
  gx = fma(co[8], E, mul_rn(co[9], Ez));
  gy = fma(co[6], D, mul_rn(co[7], Dz));
  gz = signed_by(C - Cz, q & 4);
}
__device__ __forceinline__ void tensor_gradient(const double* co, int q, const double (&v)[3], double (&g)[3][3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) tensor_gradient1(co, q, v[i], g[i][0], g[i][1], g[i][2]);
}

// Point phase of quadrature point q of element e (FP64): the displacement gradient
// and the constitutive update.  Every lane of the warp calls it (the shuffles);
// uo: the displacement of the lane's corner node (0 where not live); dNX: the block's gradients.
template <class Model>
__device__ __forceinline__ void point_phase(const ElemArgs& g, const double* s_ten, const double* s_jxw,
                                            const double* __restrict__ dNX, int64_t e, int q, bool live,
                                            const double (&uo)[3], typename Model::Mid& m) {
  const int lane = threadIdx.x & 31;
  double st[Model::NS ? Model::NS : 1];
  double* sn = nullptr;
  if (Model::NS && live) {  // (the state on its way during the gradient)
    const double* so = g.state_old + (e * NQ + q) * Model::NS;
#pragma unroll
    for (int k = 0; k < Model::NS; ++k) st[k] = so[k];
    if (g.state_new) sn = g.state_new + (e * NQ + q) * Model::NS;
  }
  double v[3], gu[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = uo[d] - __shfl_sync(0xffffffffu, uo[d], lane & ~7);
  if constexpr (!Model::TENSOR) {
#pragma unroll
    for (int i = 0; i < 9; ++i) gu[i / 3][i % 3] = 0.0;
#pragma unroll 1
    for (int a = 1; a < 8; ++a) {
      const double* ga = dNX + q * 24 + a * 3;
      const int src = (lane & ~7) | corner_node(a);
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double t = __shfl_sync(0xffffffffu, v[i], src);
#pragma unroll
        for (int j = 0; j < 3; ++j) gu[i][j] = fma(t, __ldg(ga + j), gu[i][j]);
      }
    }
  } else {
    tensor_gradient(s_ten, q, v, gu);
  }
  if (Model::TENSOR && s_ten[10] == 0.0) {  // not an axis-aligned box: reference gradient times dxi/dX
    const double* Ji = s_ten + 12 + q * 9;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double r0 = gu[i][0], r1 = gu[i][1], r2 = gu[i][2];
#pragma unroll
      for (int j = 0; j < 3; ++j) gu[i][j] = fma(r0, Ji[j], fma(r1, Ji[3 + j], mul_rn(r2, Ji[6 + j])));
    }
  }
  if (live) Model::point(g.props, gu, s_jxw[q], st, sn, m);
}

// Its inputs on an element of any shape, X: its corner node's coordinates; s_ten: the
// reference element's coefficients: dX/dxi and du/dxi at point q.
__device__ __forceinline__ void general_gradients(const double* s_ten, int q, const double (&X)[3], const double (&uo)[3],
                                                  double (&G)[3][3], double (&D)[3][3]) {
  const int l0 = threadIdx.x & 24;
  double v[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = X[d] - __shfl_sync(0xffffffffu, X[d], l0);
  tensor_gradient(s_ten, q, v, G);
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] = uo[d] - __shfl_sync(0xffffffffu, uo[d], l0);
  tensor_gradient(s_ten, q, v, D);
}
__device__ __forceinline__ void general_point(const ElemArgs& g, const double* s_ten, double w, int q, bool live,
                                              const double (&X)[3], const double (&uo)[3], RefPoint& m) {
  double G[3][3], D[3][3];
  general_gradients(s_ten, q, X, uo, G, D);
  if (live) ref_point(g.props, G, D, w, m);
}

// node pair n = (a, b), a <= b, as a << 4 | b
__constant__ unsigned char kPairNodes[NPAIR] = {0x00, 0x01, 0x02, 0x03, 0x04, 0x05, 0x06, 0x07, 0x11, 0x12, 0x13, 0x14, 0x15, 0x16, 0x17, 0x22, 0x23, 0x24, 0x25, 0x26, 0x27, 0x33, 0x34, 0x35, 0x36, 0x37, 0x44, 0x45, 0x46, 0x47, 0x55, 0x56, 0x57, 0x66, 0x67, 0x77};

// The unique tangent entries (r1, r2), r1 <= r2, of a point in two halves, each by
// a warp of its own: with the point's vectors in registers and the entry a
// constant an entry is its arithmetic and no more.  The first half are the 24 entries
// with i = 0, the second the 21 with i, k in {1, 2}: neither reads every vector.
constexpr int N_HALF = 24;
template <class Model, int HALF>
__device__ __forceinline__ void park_entries(const float2* scr, const float2* P, float fs, uint32_t ent) {
  constexpr int W0 = HALF ? N_HALF : 0, CNT = HALF ? 45 - N_HALF : N_HALF;
  typename Model::Tangent t;
  Model::load(scr, P, t);
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int r1 = 0; r1 < 9; ++r1)
#pragma unroll
    for (int r2 = r1; r2 < 9; ++r2) {
      const int c = r1 * 9 - r1 * (r1 - 1) / 2 + r2 - r1 - W0;
      if (c < 0 || c >= CNT) continue;
      const float2 a = Model::entry(t, r1 / 3, r1 % 3, r2 / 3, r2 % 3);
      v[2 * (c & 3)] = a.x * fs;
      v[2 * (c & 3) + 1] = a.y * fs;
      if ((c & 3) == 3 || c == CNT - 1) tmem_st8(ent + uint32_t(2 * (c & ~3)), v);
    }
}

__device__ __forceinline__ float2 df64_across(float2 v, int bit) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, bit), __shfl_xor_sync(0xffffffffu, v.y, bit));
}
// (v + across) where the lane's bit is set, its negative else: the transpose of a difference
__device__ __forceinline__ float2 df64_spread(float2 v, int q, int bit) {
  const float2 t = df64_add(v, df64_across(v, bit));
  return (q & bit) ? t : df64_neg(t);
}

// R_(a,i) = sum_q sum_J dNX_qaJ JxW P_iJ at node a = corner_node(q), from the row i of
// JxW P of the lane's point q (double-float): the transpose of tensor_gradient, one
// direction at a time across the element's eight lanes -- 150 FP32 operations per
// entry instead of the 290 of the sum over points, and no gradient table.  Every
// lane of the warp calls it.
template <class Model>
__device__ __forceinline__ double residual_entry(const double* ten, const float2* ten2, const double* __restrict__ dNX,
                                                 int q, float2 p0, float2 p1, float2 p2) {
  if constexpr (!Model::TENSOR) {  // the sum over points
    const double* ga = dNX + corner_node(q) * 3;
    const int l0 = threadIdx.x & 24;
    auto at = [](float2 v, int l) {
      return make_float2(__shfl_sync(0xffffffffu, v.x, l), __shfl_sync(0xffffffffu, v.y, l));
    };
    float2 R = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int k = 0; k < NQ; ++k)
      R = df64_dot3_acc(R, df64_split(__ldg(ga + k * 24)), at(p0, l0 + k), df64_split(__ldg(ga + k * 24 + 1)),
                        at(p1, l0 + k), df64_split(__ldg(ga + k * 24 + 2)), at(p2, l0 + k));
    return widen(R.x) + widen(R.y);
  }
  if (ten[10] == 0.0) {  // not a box: to the reference element
    float2 Ji[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) Ji[m] = df64_split(ten[12 + q * 9 + m]);
    const float2 x = df64_dot3(Ji[0], p0, Ji[1], p1, Ji[2], p2), y = df64_dot3(Ji[3], p0, Ji[4], p1, Ji[5], p2),
                 z = df64_dot3(Ji[6], p0, Ji[7], p1, Ji[8], p2);
    p0 = x;
    p1 = y;
    p2 = z;
  }
  const float2 E = df64_dot2(ten2[8], p0, ten2[9], df64_across(p0, 4));
  const float2 D = df64_dot2(ten2[6], p1, ten2[7], df64_across(p1, 4));
  const float2 C = df64_spread(p2, q, 4);
  const float2 A = df64_add(df64_dot2(ten2[4], C, ten2[5], df64_across(C, 2)), df64_spread(D, q, 2));
  const float2 B = df64_dot2(ten2[2], E, ten2[3], df64_across(E, 2));
  const float2 R = df64_add(df64_dot2(ten2[0], A, ten2[1], df64_across(A, 1)), df64_spread(B, q, 1));
  return widen(R.x) + widen(R.y);
}

template <class Model, bool WANT_R>
__global__ void __launch_bounds__(Roles<Model>::NTHR, 1) hex8_affine_tc_kernel(ElemArgs g, const unsigned char* __restrict__ tab) {
  using namespace tc;
  using Lay = Layout<Model>;
  using Ro = Roles<Model>;
  constexpr int SCR2 = Model::SCR2, PG = Ro::PG, NB = Model::STAGES, NTHR = Ro::NTHR, N_SL = Ro::N_SL;
  constexpr int T_SL = Ro::T_SL, T_EP = Ro::T_EP, T_MMA = Ro::T_MMA;
  extern __shared__ __align__(1024) unsigned char sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t s0 = smem_u32(sm);
  double* s_ten = reinterpret_cast<double*>(sm + Lay::TEN);
  float2* s_ten2 = reinterpret_cast<float2*>(sm + Lay::TEN2);
  double* s_jxw = reinterpret_cast<double*>(sm + Lay::JXW);
  float* s_sig = reinterpret_cast<float*>(sm + Lay::SIG);
  int* s_tau = reinterpret_cast<int*>(sm + Lay::TAU);
  int* s_taust = reinterpret_cast<int*>(sm + Lay::TAUST);
  uint32_t* s_code = reinterpret_cast<uint32_t*>(sm + Lay::CODE);
  uint64_t* bar_sl = reinterpret_cast<uint64_t*>(sm + Lay::BAR);  // slices of a tile written
  uint64_t* bar_mma = bar_sl + 1;                                  // a tile's MMAs complete (and their issuer saw its slices)
  uint64_t* bar_tfree = bar_sl + 2;                                // the epilogue read a tile's accumulators
  float2* s_P = reinterpret_cast<float2*>(sm + Lay::P);
  float2* s_scr = reinterpret_cast<float2*>(sm + Lay::SCR);

  // ---- setup: A slices zero (padding rows and columns stay zero), W digits, tables ----
  for (int i = tid; i < ND * A_SLICE / 16; i += NTHR)
    reinterpret_cast<uint4*>(sm + Lay::A)[i] = make_uint4(0u, 0u, 0u, 0u);
  for (int i = tid; i < W_BYTES / 16; i += NTHR)
    reinterpret_cast<uint4*>(sm + Lay::W)[i] = __ldg(reinterpret_cast<const uint4*>(tab + T_W) + i);
  for (int i = tid; i < TEN_N; i += NTHR) {
    const double v = __ldg(reinterpret_cast<const double*>(tab + T_TEN) + i);
    s_ten[i] = v;
    if (i < 10) s_ten2[i] = df64_split(v);
  }
  if (tid < NQ) s_jxw[tid] = __ldg(reinterpret_cast<const double*>(tab + T_JXW) + tid);
  if (tid < NPAD) s_sig[tid] = pow2f(__ldg(reinterpret_cast<const int*>(tab + T_SIG) + tid) - 7);
  if (tid < 6 * 45) {
    // unique entry w = (r1, r2), r1 <= r2, r1 = 3i + J, r2 = 3k + L, of the j-th element
    // of a lane quarter: the operand positions (row 9j + 3i + k, column group 3J + L)
    // and (row 9j + 3k + i, column group 3L + J) as byte offsets, low and high half; the
    // quarter's start is 0 or 3: table 3 (quarter & 1) + j
    const int el = tid / 45, r0 = quarter_start(el / 3) + 9 * (el % 3);
    int m = tid % 45, r = 0;
    for (int c = 0; c < 9; ++c)
      if (m >= 9 - r) { m -= 9 - r; ++r; }
    const int r1 = r, r2 = r + m;
    const int i = r1 / 3, J = r1 % 3, k = r2 / 3, L = r2 % 3;
    s_code[el * 48 + tid % 45] = op_off(r0 + i * 3 + k, (J * 3 + L) * 8) | op_off(r0 + k * 3 + i, (L * 3 + J) * 8) << 16;
  }
  if (tid == 0) {
    mbar_init(bar_sl, NSL);
    mbar_init(bar_mma, 2);
    mbar_init(bar_tfree, 32 * EP_W);
    mbar_fence_init();
  }
  if (warp == T_EP / 32) tmem_alloc(reinterpret_cast<uint32_t*>(sm + Lay::TSLOT), TMEM_COLS);
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

  if (tid < T_SL) {
    // ---------------- producers: the group of tiles k = grp, grp + PG, ...; thread (el, q) ----------------
    const int grp = tid / NPT, pt = tid - grp * NPT, el = pt >> 3, q = pt & 7;
    const int sp = (NB == 1 ? 0 : grp) * NPT + pt;  // the staged point
    const int64_t G = gridDim.x;
    // the node of the group's next tile is fetched while it computes this one
    auto node_of = [&](int64_t tile) {
      const int64_t e = tile * EPT + el;
      return tile < ntiles && e < g.ne ? g.conn[e * 8 + corner_node(q)] : -1;
    };
    int node = node_of(blockIdx.x + grp * G);
    for (int k = grp;; k += PG) {
      const int64_t tile = blockIdx.x + k * G;
      if (tile >= ntiles) break;
      const int64_t e = tile * EPT + el;
      const bool live = e < g.ne;
      double uo[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) uo[d] = live ? __ldg(&g.U[int64_t(node) * 3 + d]) : 0.0;
      typename Model::Mid mid;
      if constexpr (Model::GENERAL) {
        double X[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) X[d] = live ? __ldg(&g.coords[int64_t(node) * 3 + d]) : 0.0;
        node = node_of(tile + PG * G);
        general_point(g, s_ten, s_jxw[q], q, live, X, uo, mid);
      } else {
        node = node_of(tile + PG * G);
        point_phase<Model>(g, s_ten, s_jxw, reinterpret_cast<const double*>(tab + T_G), e, q, live, uo, mid);
      }
      if (k >= NB) named_sync(Ro::EMPTY + grp, N_SL);  // the buffer's last tile has been read
      float bnd = 0.f;
      float2 P[9];
#pragma unroll
      for (int i = 0; i < 9; ++i) P[i] = make_float2(0.f, 0.f);
      if (live) {
        bnd = Model::stage(mid, P, s_scr + sp * SCR2) * 1.0001f;
        if (Model::TANGENT_P)
#pragma unroll
          for (int i = 0; i < 9; ++i) s_P[sp * 9 + i] = P[i];
      }
      // the element's scale 2^tau > |every tangent entry| (its eight points are
      // lanes 8j .. 8j+7 of this warp)
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) bnd = fmaxf(bnd, __shfl_xor_sync(0xffffffffu, bnd, o));
      if (q == 0) {
        int tau = 0;
        if (bnd > 0.f) frexpf(bnd, &tau);
        s_taust[(NB == 1 ? 0 : grp) * 16 + el] = tau < -119 ? -119 : (tau > 126 ? 126 : tau);
      }
      named_arrive(BAR_FULL + grp, N_SL);
      if (WANT_R) {  // while the slicers work on the staging
#pragma unroll 1
        for (int i = 0; i < 3; ++i) {
          const double r = residual_entry<Model>(s_ten, s_ten2, reinterpret_cast<const double*>(tab + T_G), q, P[0], P[1], P[2]);
          if (live) static_cast<double*>(g.Re)[e * 24 + corner_node(q) * 3 + i] = r;
#pragma unroll
          for (int j = 0; j < 6; ++j) P[j] = P[j + 3];
        }
      }
    }
  } else if (tid < T_EP) {
    // ---------------- slicers: three warps (96 points) per half of the entries; lane = point ----------------
    const int ts = tid - T_SL, half = ts / NPT, p = ts - half * NPT, el = p >> 3, q = p & 7;
    const int w0 = half ? N_HALF : 0, cnt = half ? 45 - N_HALF : N_HALF;
    // this warp's TMEM lanes (quarter warp % 4) and entry columns (every fourth slicer warp has the same lanes)
    const uint32_t ent = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(TM_ENT + ((ts >> 5) >> 2) * 48);
    const uint32_t* code = s_code + ((el / 3 & 1) * 3 + el % 3) * 48 + w0;
    unsigned char* As = sm + Lay::A + (el / 3) * 4 * SBO + q * 2;
    for (int k = 0;; ++k) {
      const int64_t tile = blockIdx.x + int64_t(k) * gridDim.x;
      if (tile >= ntiles) break;
      const int buf = k % NB;
      named_sync(BAR_FULL + k % PG, N_SL);
      const int tau = s_taust[buf * 16 + el];
      const float fs = tile * EPT + el < g.ne ? pow2f(7 - tau) : 0.f;  // entries scaled to |x| < 128
      // pass 1 (overlaps the previous tile's MMAs): the scaled entries into this
      // lane's TMEM columns ent + 2c (hi), + 2c + 1 (lo)
      const float2* scr = s_scr + (buf * NPT + p) * SCR2;
      const float2* P = s_P + (buf * NPT + p) * 9;
      if (half == 0)
        park_entries<Model, 0>(scr, P, fs, ent);
      else
        park_entries<Model, 1>(scr, P, fs, ent);
      tmem_wait_st();
      named_arrive(Ro::EMPTY + (k + NB) % PG, N_SL);  // the staging may be refilled (by tile k + NB's group)
      // pass 2: the digits, once tile k-1's MMAs have read the slices
      if (k >= 1) wait_or_report(bar_mma, uint32_t((k - 1) & 1));
      if (half == 0 && q == 0) s_tau[(k & 1) * 16 + el] = tau;
#pragma unroll 1
      for (int c = 0; c < cnt; ++c) {
        float xh, xl;
        tmem_ld2(ent + uint32_t(2 * c), xh, xl);
        const uint32_t at = code[c];
        unsigned char* p1 = As + (at & 0xffffu);
        unsigned char* p2 = As + (at >> 16);
        const bool twin = p1 != p2;
        // digit s: the part of x at or above 2^(-8s), by adding and subtracting
        // 1.5 2^(23-8s) (a rounding instruction issues at an eighth of the rate);
        // |xl| <= ulp(xh) / 2 <= 2^-18 has no digits before the third
#pragma unroll
        for (int s = 0; s < ND; ++s) {
          const float big = pow2f(23 - 8 * s) * 1.5f;
          float d = __fsub_rn(__fadd_rn(xh, big), big);
          xh = __fsub_rn(xh, d);
          if (s >= 3) {
            const float dl = __fsub_rn(__fadd_rn(xl, big), big);
            xl = __fsub_rn(xl, dl);
            d = __fadd_rn(d, dl);
          }
          const unsigned short bits = static_cast<unsigned short>(__float_as_uint(d) >> 16);
          *reinterpret_cast<unsigned short*>(p1 + s * A_SLICE) = bits;
          if (twin) *reinterpret_cast<unsigned short*>(p2 + s * A_SLICE) = bits;
        }
      }
      fence_async_smem();
      mbar_arrive(bar_sl);
    }
  } else if (tid < T_MMA) {
    // ---------------- epilogue: thread = TMEM lane = row (el, i, k) ----------------
    const int qw = warp & 3;
    const int row = lane - quarter_start(qw);  // of the quarter's 27
    const bool used = row >= 0 && row < 27;
    const int el = qw * 3 + (used ? row / 9 : 0), ik = used ? row % 9 : 0, i = ik / 3, kc = ik % 3;
    const uint32_t lane_addr = tmem + (uint32_t(qw * 32) << 16);
    for (int k = 0;; ++k) {
      const int64_t tile = blockIdx.x + int64_t(k) * gridDim.x;
      if (tile >= ntiles) break;
      const int64_t e0 = tile * EPT;
      const bool live = used && e0 + el < g.ne;
      // (bar_mma alone: its next phase needs this warp's arrival at bar_tfree.  The slicers'
      // barrier may complete another phase as soon as the MMAs are done, and a warp that
      // came that late would wait by parity for the phase after)
      wait_or_report(bar_mma, uint32_t(k & 1));
      tc_fence_after();
      const float f1 = pow2f(s_tau[(k & 1) * 16 + el] - 7);
#pragma unroll 1
      for (int n0 = 0; n0 < NPAIR; n0 += 4) {
        float v[NLEV][4];
        tmem_ld4x7<NPAD>(lane_addr + uint32_t(n0), v);
        if (g.ke_pairs) {
          // the symmetric half straight from the levels: pair n = (a, b) of row
          // (el, i, k) is K_(a,i),(b,k), entry 9n + 3i + k of the element's KE_PAIRS block
          float2* dst = static_cast<float2*>(g.Ke) + (e0 + el) * (NPAIR * 9) + ik + n0 * 9;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 hl = combine_levels(v, j);
            const float f = f1 * s_sig[n0 + j];
            if (live) dst[j * 9] = make_float2(hl.x * f, hl.y * f);
          }
        } else {
          // node rows of the whole K_e: pair n = (a, b) of row (el, i, k), K_(a,i),(b,k), is
          // entry b of node row (a, i, k) and, by symmetry, entry a of node row (b, k, i)
          float2* dst = static_cast<float2*>(g.Ke) + (e0 + el) * 576;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 hl = combine_levels(v, j);
            const float f = f1 * s_sig[n0 + j];
            const int ab = kPairNodes[n0 + j], a = ab >> 4, b = ab & 15;
            const float2 val = make_float2(hl.x * f, hl.y * f);
            if (live) {
              dst[((a * 3 + i) * 3 + kc) * 8 + b] = val;
              if (a != b) dst[((b * 3 + kc) * 3 + i) * 8 + a] = val;
            }
          }
        }
      }
      tc_fence_before();
      mbar_arrive(bar_tfree);  // the accumulators may be overwritten
    }
  } else {
    // ---------------- MMA warp: lane 0 issues, the warp waits together ----------------
    const uint32_t aB = s0 + Lay::A, wB = s0 + Lay::W;
    const uint64_t dA = smem_desc(aB, 128, SBO), dW = smem_desc(wB, 128, SBO);
    for (int k = 0;; ++k) {
      const int64_t tile = blockIdx.x + int64_t(k) * gridDim.x;
      if (tile >= ntiles) break;
      wait_or_report(bar_sl, uint32_t(k & 1));  // the tile's slices are written
      tc_fence_after();
      if (k >= 1) {
        wait_or_report(bar_tfree, uint32_t((k - 1) & 1));  // the accumulators are free
        tc_fence_after();
      }
      if (lane == 0) {
#pragma unroll 1
        for (int t = 0; t < ND; ++t)
#pragma unroll 1
          for (int s = 0; s < ND - t; s += MAXS) {
            const int ns = ND - t - s < MAXS ? ND - t - s : MAXS;
            const uint32_t idesc = tc::idesc_bf16(128, NPAD * ns);
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
  tc_fence_before();
  __syncthreads();
  if (warp == T_EP / 32) {
    tc_fence_after();
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

// Residual only (no tangent): the same point phase and residual arithmetic as
// the tensor-core kernel, so both give bitwise the same R and state.  16
// elements per CTA, one thread per point.
constexpr int R_EPB = 16;
template <class Model>
__global__ void __launch_bounds__(R_EPB * NQ) hex8_affine_r_kernel(ElemArgs g, const unsigned char* __restrict__ tab) {
  __shared__ double s_ten[TEN_N], s_jxw[NQ];
  __shared__ float2 s_ten2[10];
  const int tid = threadIdx.x, el = tid >> 3, q = tid & 7;
  for (int i = tid; i < TEN_N; i += blockDim.x) {
    const double v = __ldg(reinterpret_cast<const double*>(tab + T_TEN) + i);
    s_ten[i] = v;
    if (i < 10) s_ten2[i] = df64_split(v);
  }
  if (tid < NQ) s_jxw[tid] = __ldg(reinterpret_cast<const double*>(tab + T_JXW) + tid);
  __syncthreads();
  const int64_t e = int64_t(blockIdx.x) * R_EPB + el;
  const bool live = e < g.ne;
  double uo[3] = {0.0, 0.0, 0.0}, X[3] = {0.0, 0.0, 0.0};
  if (live) {
    const int64_t node = g.conn[e * 8 + corner_node(q)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      uo[d] = __ldg(&g.U[node * 3 + d]);
      if (Model::GENERAL) X[d] = __ldg(&g.coords[node * 3 + d]);
    }
  }
  typename Model::Mid mid;
  if constexpr (Model::GENERAL)
    general_point(g, s_ten, s_jxw[q], q, live, X, uo, mid);
  else
    point_phase<Model>(g, s_ten, s_jxw, reinterpret_cast<const double*>(tab + T_G), e, q, live, uo, mid);
  float2 P[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) P[i] = make_float2(0.f, 0.f);
  if (live) Model::stress(mid, P);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double r = residual_entry<Model>(s_ten, s_ten2, reinterpret_cast<const double*>(tab + T_G), q, P[i * 3], P[i * 3 + 1],
                                           P[i * 3 + 2]);
    if (live) static_cast<double*>(g.Re)[e * 24 + corner_node(q) * 3 + i] = r;
  }
}

// The transpose of tensor_gradient for one component in FP64: the value at node
// corner_node(q) from the row p of the lane's point q.
__device__ __forceinline__ double tensor_spread(const double* co, int q, double p0, double p1, double p2) {
  auto across = [](double v, int bit) { return __shfl_xor_sync(0xffffffffu, v, bit); };
  const double E = fma(co[8], p0, mul_rn(co[9], across(p0, 4)));
  const double D = fma(co[6], p1, mul_rn(co[7], across(p1, 4)));
  const double C = signed_by(p2 + across(p2, 4), q & 4);
  const double A = fma(co[4], C, fma(co[5], across(C, 2), signed_by(D + across(D, 2), q & 2)));
  const double B = fma(co[2], E, mul_rn(co[3], across(E, 2)));
  return fma(co[0], A, fma(co[1], across(A, 1), signed_by(B + across(B, 1), q & 1)));
}

// Matrix-free tangent action K_e v_e (see fec_action.cu) with the point phase and
// gradients of the kernels above, in FP64 throughout: the FP64 pipe bounds it, and
// the sum-factorised gradients and their transpose take 13 operations a component
// where the sums over nodes take 24 (about 300 a point instead of 500).  16
// elements per CTA, one thread per point.
template <class Model>
__global__ void __launch_bounds__(R_EPB * NQ) hex8_action_kernel(ElemArgs g, const unsigned char* __restrict__ tab,
                                                                 const double* __restrict__ V) {
  __shared__ double s_ten[TEN_N], s_jxw[NQ];
  const int tid = threadIdx.x, el = tid >> 3, q = tid & 7, lane = tid & 31;
  for (int i = tid; i < TEN_N; i += blockDim.x) s_ten[i] = __ldg(reinterpret_cast<const double*>(tab + T_TEN) + i);
  if (tid < NQ) s_jxw[tid] = __ldg(reinterpret_cast<const double*>(tab + T_JXW) + tid);
  __syncthreads();
  const int64_t e = int64_t(blockIdx.x) * R_EPB + el;
  const bool live = e < g.ne;
  double uo[3] = {0.0, 0.0, 0.0}, X[3] = {0.0, 0.0, 0.0}, v[3] = {0.0, 0.0, 0.0};
  if (live) {
    const int64_t node = g.conn[e * 8 + corner_node(q)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      uo[d] = __ldg(&g.U[node * 3 + d]);
      v[d] = __ldg(&V[node * 3 + d]);
      if (Model::GENERAL) X[d] = __ldg(&g.coords[node * 3 + d]);
    }
  }
  double D[3][3], out[3][3];
  std::conditional_t<Model::GENERAL, PointUpdate, typename Model::Mid> mid;
  if constexpr (Model::GENERAL) {
    double G[3][3];
    general_gradients(s_ten, q, X, uo, G, D);
    if (live) point_update(g.props, G, D, s_jxw[q], mid);
  } else {
    point_phase<Model>(g, s_ten, s_jxw, reinterpret_cast<const double*>(tab + T_G), e, q, live, uo, mid);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) v[d] -= __shfl_sync(0xffffffffu, v[d], lane & ~7);
  tensor_gradient(s_ten, q, v, D);
  const bool box = s_ten[10] != 0.0;
  const double* Ji = s_ten + 12 + q * 9;
  if (!box) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const double r0 = D[i][0], r1 = D[i][1], r2 = D[i][2];
#pragma unroll
      for (int j = 0; j < 3; ++j) D[i][j] = fma(r0, Ji[j], fma(r1, Ji[3 + j], mul_rn(r2, Ji[6 + j])));
    }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) out[i / 3][i % 3] = 0.0;
  if (live) Model::action(mid, D, out);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double p0 = out[i][0], p1 = out[i][1], p2 = out[i][2];
    if (!box) {
      const double x = fma(Ji[0], p0, fma(Ji[1], p1, mul_rn(Ji[2], p2))),
                   y = fma(Ji[3], p0, fma(Ji[4], p1, mul_rn(Ji[5], p2)));
      p2 = fma(Ji[6], p0, fma(Ji[7], p1, mul_rn(Ji[8], p2)));
      p0 = x;
      p1 = y;
    }
    const double r = tensor_spread(s_ten, q, p0, p1, p2);
    if (live) static_cast<double*>(g.Re)[e * 24 + corner_node(q) * 3 + i] = r;
  }
}

// Poisson on a block of translated elements (test/poisson/TestPoissonCommon.jl:75-107):
// its element matrix is the block's constant, read from the table; the residual is
// the transpose of the gradient applied to JxW grad u, less the source f(X_q) N_a JxW.
// A box's points have two coordinates per direction, so its eight lanes share six
// sines instead of forming 24.  FP64-pipe bound as before (about 70 instead of 460
// FP64 operations a point with the matrix): 36 x 32 x 34 elements element
// kernel 263 -> 48 us.
template <bool WANT_R, bool WANT_K>
__global__ void __launch_bounds__(R_EPB * NQ) hex8_poisson_kernel(ElemArgs g, const unsigned char* __restrict__ tab) {
  __shared__ double s_ten[TEN_N], s_jxw[NQ], s_off[NQ * 3], s_n[NQ * 8];
  __shared__ float2 s_k[64];
  const int tid = threadIdx.x, el = tid >> 3, q = tid & 7, lane = tid & 31, l0 = lane & ~7;
  const double* t = reinterpret_cast<const double*>(tab);
  for (int i = tid; i < TEN_N; i += blockDim.x) s_ten[i] = __ldg(t + T_TEN / 8 + i);
  if (tid < NQ) s_jxw[tid] = __ldg(t + T_JXW / 8 + tid);
  if (tid < NQ * 3) s_off[tid] = __ldg(t + T_OFF / 8 + tid);
  if (tid < NQ * 8) {
    s_n[tid] = __ldg(t + T_N / 8 + tid);
    s_k[tid] = df64_split(__ldg(t + T_K / 8 + tid));
  }
  __syncthreads();
  const int64_t e = int64_t(blockIdx.x) * R_EPB + el;
  const bool live = e < g.ne;
  if (WANT_K && live) {  // row q of K_e
    float4* dst = reinterpret_cast<float4*>(static_cast<float2*>(g.Ke) + (e * 8 + q) * 8);
#pragma unroll
    for (int b = 0; b < 8; b += 2)
      dst[b / 2] = make_float4(s_k[q * 8 + b].x, s_k[q * 8 + b].y, s_k[q * 8 + b + 1].x, s_k[q * 8 + b + 1].y);
  }
  if (!WANT_R) return;
  const int a = corner_node(q);
  double u = 0.0, X0[3] = {0.0, 0.0, 0.0};
  if (live) {
    u = __ldg(&g.U[g.conn[e * 8 + a]]);
    const int64_t n0 = g.conn[e * 8];
#pragma unroll
    for (int d = 0; d < 3; ++d) X0[d] = __ldg(&g.coords[n0 * 3 + d]);
  }
  // source at the lane's point
  double f = g.props[0] * s_jxw[q];
  if (s_ten[11] != 0.0) {
    const int d = q >> 1 < 3 ? q >> 1 : 2;  // lane 2d + side: the sine of that coordinate
    const double sn = sinpi((d == 0 ? X0[0] : d == 1 ? X0[1] : X0[2]) + s_off[((q & 1) ? 7 : 0) * 3 + d]);
#pragma unroll
    for (int k = 0; k < 3; ++k) f *= __shfl_sync(0xffffffffu, sn, l0 + 2 * k + (q >> k & 1));
  } else {
#pragma unroll
    for (int d = 0; d < 3; ++d) f *= sinpi(X0[d] + s_off[q * 3 + d]);
  }
  const double v = u - __shfl_sync(0xffffffffu, u, l0);
  double g0, g1, g2;
  tensor_gradient1(s_ten, q, v, g0, g1, g2);
  const double* Ji = s_ten + 12 + q * 9;
  const double w = s_jxw[q];
  if (s_ten[10] == 0.0) {  // (dxi/dX)(dxi/dX)^T of the reference gradient
    double p[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) p[j] = fma(g0, Ji[j], fma(g1, Ji[3 + j], mul_rn(g2, Ji[6 + j])));
    g0 = fma(Ji[0], p[0], fma(Ji[1], p[1], mul_rn(Ji[2], p[2])));
    g1 = fma(Ji[3], p[0], fma(Ji[4], p[1], mul_rn(Ji[5], p[2])));
    g2 = fma(Ji[6], p[0], fma(Ji[7], p[1], mul_rn(Ji[8], p[2])));
  }
  double R = tensor_spread(s_ten, q, mul_rn(w, g0), mul_rn(w, g1), mul_rn(w, g2));
#pragma unroll
  for (int k = 0; k < NQ; ++k) R = fma(-s_n[k * 8 + a], __shfl_sync(0xffffffffu, f, l0 + k), R);
  if (live) static_cast<double*>(g.Re)[e * 8 + a] = R;
}

template <class Model>
cudaError_t launch_act(const ElemArgs& a, const void* tab, const double* V, cudaStream_t s, int* launches) {
  const int64_t nb = (a.ne + R_EPB - 1) / R_EPB;
  if (nb == 0) return cudaSuccess;
  hex8_action_kernel<Model><<<unsigned(nb), R_EPB * NQ, 0, s>>>(a, static_cast<const unsigned char*>(tab), V);
  if (launches) ++*launches;
  return cudaGetLastError();
}

template <class Model, bool WANT_R>
cudaError_t launch1(const ElemArgs& a, cudaStream_t s, int* launches) {
  constexpr int SMEM = Layout<Model>::SMEM;
  const cudaError_t e = ensure_smem<hex8_affine_tc_kernel<Model, WANT_R>>(SMEM);
  if (e != cudaSuccess) return e;
  const int64_t ntiles = (a.ne + EPT - 1) / EPT;
  if (ntiles == 0) return cudaSuccess;
  const int grid = int(ntiles < num_sms() ? ntiles : num_sms());
  hex8_affine_tc_kernel<Model, WANT_R><<<grid, Roles<Model>::NTHR, SMEM, s>>>(a, static_cast<const unsigned char*>(a.affine));
  if (launches) ++*launches;
  return cudaGetLastError();
}

template <class Model>
cudaError_t launch_r(const ElemArgs& a, cudaStream_t s, int* launches) {
  const int64_t nb = (a.ne + R_EPB - 1) / R_EPB;
  if (nb == 0) return cudaSuccess;
  hex8_affine_r_kernel<Model><<<unsigned(nb), R_EPB * NQ, 0, s>>>(a, static_cast<const unsigned char*>(a.affine));
  if (launches) ++*launches;
  return cudaGetLastError();
}

}  // namespace aff

bool hex8_affine_enabled() {
  const char* v = std::getenv("FEC_HEX8_AFFINE");
  return !(v && v[0] == '0');
}

size_t hex8_affine_grad_offset() {
  static_assert(aff::T_JXW == aff::T_G + aff::NQ * 24 * 8, "gradients, then JxW");
  return size_t(aff::T_G);
}

bool hex8_pairs_enabled() {
  const char* v = std::getenv("FEC_HEX8_PAIRS");
  return !(v && v[0] == '0');
}

template <class Model>
static cudaError_t launch_affine(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (!want_k) return want_r ? aff::launch_r<Model>(a, s, launches) : cudaSuccess;
  return want_r ? aff::launch1<Model, true>(a, s, launches) : aff::launch1<Model, false>(a, s, launches);
}

cudaError_t launch_hex8_affine_tc(int physics, bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s,
                                  int* launches) {
  if (!a.affine || (want_k && !a.Ke) || (want_r && !a.Re)) return cudaErrorInvalidValue;
  if (physics == 2)
    return a.hex8_tensor ? launch_affine<aff::AffNeoHookean>(want_r, want_k, a, s, launches)
                         : launch_affine<aff::AnyRule<aff::AffNeoHookean>>(want_r, want_k, a, s, launches);
  if (physics == 3)
    return a.hex8_tensor ? launch_affine<aff::AffJ2>(want_r, want_k, a, s, launches)
                         : launch_affine<aff::AnyRule<aff::AffJ2>>(want_r, want_k, a, s, launches);
  return cudaErrorNotSupported;
}

// Whether the reference tables are trilinear gradients at points (-+t_0, -+t_1,
// -+t_2), x fastest (2 x 2 x 2 Gauss, Lobatto): c[d] = (1 + t_d) / 2 then.  (And the
// shape functions sum to one: Poisson's points are offsets from node 0.)
bool hex8_tensor_rule(const double* ref, double c[3]) {
  using L = RefLayout<1>;
  const double* dN = ref + L::DN_OFF;
  auto corner = [](int a) { return a ^ ((a >> 1) & 1); };  // bits x, y, z of node a
  for (int d = 0; d < 3; ++d) {
    // at the last point, the derivative along k summed over the direction that is neither k nor d
    const int k = (d + 1) % 3;
    double s = 0.0;
    for (int a = 0; a < 8; ++a)
      if ((corner(a) >> d & 1) && (corner(a) >> k & 1)) s += dN[(7 * 8 + a) * 3 + k];
    c[d] = 2.0 * s;
  }
  for (int q = 0; q < 8; ++q) {
    double sum = 0.0;
    for (int a = 0; a < 8; ++a) sum += ref[L::N_OFF + q * 8 + a];
    if (!(std::fabs(sum - 1.0) <= 1e-14)) return false;
  }
  for (int q = 0; q < 8; ++q)
    for (int a = 0; a < 8; ++a)
      for (int k = 0; k < 3; ++k) {
        double v = (corner(a) >> k & 1) ? 0.5 : -0.5;
        for (int d = 0; d < 3; ++d)
          if (d != k) v *= (corner(a) >> d & 1) == (q >> d & 1) ? c[d] : 1.0 - c[d];
        if (!(std::fabs(v - dN[(q * 8 + a) * 3 + k]) <= 1e-15)) return false;
      }
  return true;
}

// Half the inverse edge lengths of an axis-aligned box in node order; false for
// any other element (edges to 1e-13 of the largest, as in the congruence test).
static bool box_scales(const double* x0, double sc[3]) {
  double h = 0.0, len[3];
  for (int d = 0; d < 3; ++d) {
    len[d] = x0[6 * 3 + d] - x0[d];  // node 6 is opposite node 0
    h = std::fmax(h, std::fabs(len[d]));
  }
  for (int a = 0; a < 8; ++a)
    for (int d = 0; d < 3; ++d) {
      const int bit = (a ^ ((a >> 1) & 1)) >> d & 1;
      if (!(std::fabs(x0[a * 3 + d] - x0[d] - (bit ? len[d] : 0.0)) <= 1e-13 * h)) return false;
    }
  for (int d = 0; d < 3; ++d) {
    if (!(len[d] > 0.0)) return false;
    sc[d] = 1.0 / len[d];
  }
  return true;
}

// FEC_HEX8_GENERAL=0 keeps hex8 blocks of any shape on the per-element kernels.
bool hex8_general_enabled() {
  const char* v = std::getenv("FEC_HEX8_GENERAL");
  return !(v && v[0] == '0');
}

cudaError_t launch_hex8_general_tc(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (!a.general || (want_k && !a.Ke) || (want_r && !a.Re)) return cudaErrorInvalidValue;
  ElemArgs b = a;
  b.affine = a.general;
  if (!want_k) return want_r ? aff::launch_r<aff::GenNeoHookean>(b, s, launches) : cudaSuccess;
  return want_r ? aff::launch1<aff::GenNeoHookean, true>(b, s, launches)
                : aff::launch1<aff::GenNeoHookean, false>(b, s, launches);
}

cudaError_t launch_hex8_action(int physics, const ElemArgs& a, const double* V, cudaStream_t s, int* launches) {
  if (!a.Re) return cudaErrorInvalidValue;
  if (physics == 2 && a.affine) return aff::launch_act<aff::AffNeoHookean>(a, a.affine, V, s, launches);
  if (physics == 3 && a.affine) return aff::launch_act<aff::AffJ2>(a, a.affine, V, s, launches);
  if (physics == 2 && a.general) return aff::launch_act<aff::GenNeoHookean>(a, a.general, V, s, launches);
  return cudaErrorNotSupported;
}

cudaError_t launch_hex8_poisson(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  const int64_t nb = (a.ne + aff::R_EPB - 1) / aff::R_EPB;
  if (nb == 0 || (!want_r && !want_k)) return cudaSuccess;
  const unsigned char* tab = static_cast<const unsigned char*>(a.affine);
  constexpr int T = aff::R_EPB * aff::NQ;
  if (want_r && want_k)
    aff::hex8_poisson_kernel<true, true><<<unsigned(nb), T, 0, s>>>(a, tab);
  else if (want_r)
    aff::hex8_poisson_kernel<true, false><<<unsigned(nb), T, 0, s>>>(a, tab);
  else
    aff::hex8_poisson_kernel<false, true><<<unsigned(nb), T, 0, s>>>(a, tab);
  if (launches) ++*launches;
  return cudaGetLastError();
}

// The operand of the reference element itself (the cube [-1, 1]^3).
bool hex8_general_table(const double* ref, std::vector<unsigned char>& out) {
  double x[24];
  for (int a = 0; a < 8; ++a)
    for (int d = 0; d < 3; ++d) x[a * 3 + d] = (a ^ ((a >> 1) & 1)) >> d & 1 ? 1.0 : -1.0;
  return hex8_affine_table(x, ref, out);
}

// Host: sums of products and 2 x 2 determinants as if in twice the precision (Ogita, Rump and
// Oishi, SIAM J. Sci. Comput. 26 (2005) 1955-1988, Dot2).  The mapping of a block is a constant of
// all its elements, so its rounding would be a common factor of their matrices that no sum
// averages out: det J from rounded sums put 3 ulp on every entry.
namespace {
struct Dot2 {
  double s = 0.0, c = 0.0;
  void add(double a, double b) {
    const double p = a * b, e = std::fma(a, b, -p), t = s + p, z = t - s;
    c += e + ((s - (t - z)) + (p - z));
    s = t;
  }
  double value() const { return s + c; }
};
double det2(double a, double b, double c, double d) {  // a d - b c
  Dot2 t;
  t.add(a, d);
  t.add(-b, c);
  return t.value();
}
}  // namespace

// Host: the constant operand of a block whose elements are translates of its
// first one.  x0: the first element's node coordinates [8][3]; ref: the block's
// reference tables (RefLayout<1>: N, dN/dxi [q][a][3], weights).  Returns false
// for a degenerate element (det J <= 0 at a point) or gradient products outside
// the range the FP32 epilogue scales (2^-126 .. 2^127).
bool hex8_affine_table(const double* x0, const double* ref, std::vector<unsigned char>& out) {
  using L = RefLayout<1>;
  out.assign(aff::T_BYTES, 0);
  double dNX[8][8][3], jxw[8], ten[aff::TEN_N] = {0.0};
  double cI[3] = {1.0, 1.0, 1.0}, sc[3];
  const bool trilinear = hex8_tensor_rule(ref, cI), box = box_scales(x0, sc);
  auto corner = [](int bits) { return bits ^ (bits >> 1 & 1); };
  for (int q = 0; q < 8; ++q) {
    const double* dN = ref + L::DN_OFF + q * 24;
    double J[3][3], co[3][3], Ji[3][3];
    for (int d = 0; d < 3; ++d)
      for (int k = 0; k < 3; ++k) {
        if (trilinear) {
          // half the edges along k, interpolated: of a parallelepiped an edge, whatever the
          // tables' rounding (a box is taken as one to 1e-13, see box_scales)
          const int m = (k + 1) % 3, n = (k + 2) % 3;
          const double fm = q >> m & 1 ? cI[m] : 1.0 - cI[m], fn = q >> n & 1 ? cI[n] : 1.0 - cI[n];
          auto edge = [&](int bits) {
            return x0[corner(bits | 1 << k) * 3 + d] - x0[corner(bits) * 3 + d];
          };
          const double e = edge(0), em = edge(1 << m) - e, en = edge(1 << n) - e,
                       emn = edge(1 << m | 1 << n) - e - em - en;
          Dot2 s;
          s.add(e, 1.0);
          s.add(em, fm);
          s.add(en, fn);
          s.add(emn, fm * fn);
          J[d][k] = 0.5 * s.value();
          if (box) J[d][k] = d == k ? 0.5 * (x0[18 + d] - x0[d]) : 0.0;
        } else {
          Dot2 s;
          for (int a = 1; a < 8; ++a) s.add(x0[a * 3 + d] - x0[d], dN[a * 3 + k]);
          J[d][k] = s.value();
        }
      }
    for (int d = 0; d < 3; ++d)
      for (int k = 0; k < 3; ++k) {
        const int d1 = (d + 1) % 3, d2 = (d + 2) % 3, k1 = (k + 1) % 3, k2 = (k + 2) % 3;
        co[d][k] = det2(J[d1][k1], J[d1][k2], J[d2][k1], J[d2][k2]);
      }
    Dot2 sum;
    for (int k = 0; k < 3; ++k) sum.add(J[0][k], co[0][k]);
    const double det = sum.value();
    if (!(det > 0.0)) return false;
    for (int k = 0; k < 3; ++k)
      for (int d = 0; d < 3; ++d) Ji[k][d] = trilinear && box ? (d == k ? 2.0 * sc[d] : 0.0) : co[d][k] / det;
    for (int k = 0; k < 3; ++k)
      for (int d = 0; d < 3; ++d) ten[12 + q * 9 + k * 3 + d] = Ji[k][d];
    for (int a = 0; a < 8; ++a)
      for (int d = 0; d < 3; ++d) {
        double s = 0.0;
        for (int k = 0; k < 3; ++k) s = std::fma(dN[a * 3 + k], Ji[k][d], s);
        dNX[q][a][d] = s;
      }
    jxw[q] = det * ref[L::W_OFF + q];
  }
  int n = 0;
  int32_t sig[aff::NPAD] = {0};
  for (int a = 0; a < 8; ++a)
    for (int b = a; b < 8; ++b, ++n) {
      double w[aff::KR], mx = 0.0;
      for (int q = 0; q < 8; ++q)
        for (int J = 0; J < 3; ++J)
          for (int Lc = 0; Lc < 3; ++Lc) {
            w[q * 9 + J * 3 + Lc] = dNX[q][a][J] * dNX[q][b][Lc];
            mx = std::fmax(mx, std::fabs(w[q * 9 + J * 3 + Lc]));
          }
      int e = 0;
      if (mx > 0.0) std::frexp(mx, &e);  // |w| < 2^e
      if (e < -119 || e > 134) return false;  // the epilogue scales by 2^(e - 7) in FP32
      sig[n] = e;
      for (int r = 0; r < aff::KR; ++r) {
        uint16_t bits[aff::ND];
        aff::bf16_digits(w[r], e, bits);
        for (int s = 0; s < aff::ND; ++s)
          std::memcpy(out.data() + aff::T_W + s * aff::W_SLICE + aff::op_off(n, r % 9 * 8 + r / 9), &bits[s], 2);
      }
    }
  // tensor_gradient's coefficients, with the scales dxi/dX folded in for a box
  ten[10] = box ? 1.0 : 0.0;
  if (!box) sc[0] = sc[1] = sc[2] = 0.5;
  const double own[5] = {cI[0], cI[1], cI[1] * sc[2], cI[2] * sc[1], cI[2] * sc[0]};
  const double across[5] = {1.0 - cI[0], 1.0 - cI[1], (1.0 - cI[1]) * sc[2], (1.0 - cI[2]) * sc[1],
                            (1.0 - cI[2]) * sc[0]};
  for (int k = 0; k < 5; ++k) {
    ten[2 * k] = own[k];
    ten[2 * k + 1] = across[k];
  }
  // Poisson: the points' offsets from node 0, shape functions, element matrix
  double off[8][3], K[8][8] = {{0.0}};
  const double* N = ref + L::N_OFF;
  for (int q = 0; q < 8; ++q) {
    for (int d = 0; d < 3; ++d) {
      double s = 0.0;
      for (int a = 1; a < 8; ++a) s = std::fma(N[q * 8 + a], x0[a * 3 + d] - x0[d], s);
      off[q][d] = s;
    }
    for (int a = 0; a < 8; ++a)
      for (int b = 0; b < 8; ++b) {
        double s = 0.0;
        for (int d = 0; d < 3; ++d) s = std::fma(dNX[q][a][d] * jxw[q], dNX[q][b][d], s);
        K[a][b] += s;
      }
  }
  bool separable = true;  // coordinate d of a point only depends on its bit d
  for (int q = 0; q < 8; ++q) {
    for (int d = 0; d < 3; ++d) {
      const double h = std::fabs(off[7][d]) + std::fabs(off[0][d]);
      separable = separable && std::fabs(off[q][d] - off[(q >> d & 1) ? 7 : 0][d]) <= 4e-16 * h;
    }
  }
  ten[11] = separable ? 1.0 : 0.0;
  std::memcpy(out.data() + aff::T_OFF, off, sizeof off);
  std::memcpy(out.data() + aff::T_N, N, 64 * sizeof(double));
  std::memcpy(out.data() + aff::T_K, K, sizeof K);
  std::memcpy(out.data() + aff::T_TEN, ten, sizeof ten);
  std::memcpy(out.data() + aff::T_SIG, sig, sizeof sig);
  std::memcpy(out.data() + aff::T_G, dNX, sizeof dNX);
  std::memcpy(out.data() + aff::T_JXW, jxw, sizeof jxw);
  return true;
}

}  // namespace fec
