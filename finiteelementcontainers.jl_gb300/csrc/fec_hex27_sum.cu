// fec_hex27_sum.cu -- FP64 hex27 Neo-Hookean elements of any shape: the stiffness by sum
// factorisation, in reference coordinates and double-float.
//
// In reference coordinates (as GenNeoHookean, fec_digits.cuh) the gradients are the reference element's
// own, products of one-dimensional functions l_a at three points per direction:
//     K_(a,i),(b,k) = sum_q sum_(J,L) dN_qaJ dN_qbL A_q,iJkL,   dN_qaJ = prod_d x(d = J)_(a_d)(q_d),
// x = V (values l) or D (derivatives).  So q is summed one direction at a time: for a
// fixed (i, k), 9 (J, L) x 9 (a1 b1) x 9 (q2 q3) values after the first, the (J, L) with
// the same factors along the third direction added into one value during the second,
// four kinds x 81 (a1 b1 a2 b2) x 3 (q3), and the 729 (a, b) after the third: about 14,000
// double-float products instead of the 9 * 729 * 27 = 177,000 of the sum over points.
// With K = K^T, (i, k) runs over i <= k, and for i = k over half of the (a, b).
//
// One persistent CTA per SM:
//   8 producers   in turn an element each: lane = node and point, point phase in FP64,
//                 gradients and residual one direction at a time through shuffles (24
//                 operations a component instead of 81); the vectors of the tangent into
//                 one of eight staging buffers;
//   3 groups of   take the elements in turn: the 45 tangent entries of each point; then,
//   4 warps       thread = (i, k, a1 b1, q3), the first two directions (in registers);
//                 then, thread = (i, k, a1 b1, a2 b2), the third, whose 9 results go to K_e.
// The middle point's V = (0, 1, 0) and D = (-1/2, 0, 1/2) need no products.
// What bounds it: instruction issue, 31,100 warp instructions an element (2.2 a clock), so
// the groups are of four warps, one on each sub-partition (135 items of the first two
// directions on five warps of a CTA of their own: 0.93 ms), and enough producers keep
// them fed (4: 0.72 ms).  13,728 elements 0.65 ms, 3.60 with the per-element
// kernel's 826,000 products (fec_mech_hex27.cuh).
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
namespace h27 {

using namespace aff;

constexpr int NQ = 27, A = 27;
constexpr int T_V = 0, T_D = 9, T_W = 18, T_DOUBLES = 18 + NQ;  // table: V[m][q], D[m][q], weights
constexpr int NGRP = 3, GT = 128, NPROD = 8, NSLOT = 8;  // groups, their threads, producers, staging buffers
constexpr int NCON = NGRP * GT, NTHR = NCON + 32 * NPROD;
constexpr int BAR_GRP = 1;                               // + group: among its warps
constexpr int N_STAGE = 33;                              // H (9), Z (9), Y (9), c2 M (6) of a point
// (i, k): 0..2 are (0, 1), (0, 2), (1, 2), 3..5 are (0, 0), (1, 1), (2, 2)
constexpr int T2_OFF = 12 * 81, T2_DIAG = 12 * 54, N_T2 = 3 * (T2_OFF + T2_DIAG);

constexpr int N_FIRST = 135, N_THIRD = 378;              // items of the first two directions and of the third

struct Smem {
  float2 stage[NSLOT][N_STAGE][NQ];
  float2 ent[NGRP][54][NQ];     // (i, k) 6 x (J, L) 9
  float2 t2[NGRP][N_T2];        // per (i, k): [kind 4][q3][a2 b2][a1 b1] (a1 <= b1 only where i = k)
  double vd[18];                // V, D
  float2 vd2[18];               // split
  float2 prod[4][9][4];         // kind (VV, VD, DV, DD), (a, b), q: the products along the first direction
  uint64_t full[NSLOT], empty[NSLOT];
  uint32_t code[45];            // an entry's operands and places
  // of each item of the third direction: the places of its nine (a3, b3) in the symmetric
  // half (65535: the mirrored one's), then where its values start in t2 and, for a1 = b1,
  // a2 = b2 and i < k, k - i << 14: (i, k) of a node with itself has a second place
  unsigned short where[N_THIRD][10];
};
static_assert(sizeof(Smem) <= 232448 && 3 * (T2_OFF + T2_DIAG) < 8192, "shared memory");

__device__ __forceinline__ double shfl(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

struct Lane {
  int l, i, j, k;  // node / point and its place along each direction
};

// Gradient at the lane's point of the nodal values v (lane = node).
__device__ __forceinline__ void gradient(const double* vd, const Lane& n, double x, double (&g)[3]) {
  const double v = x - shfl(x, 0);
  const double *V = vd, *D = vd + 9;
  double a = 0.0, b = 0.0;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const double t = shfl(v, n.l + m - n.i);
    a = fma(V[m * 3 + n.i], t, a);
    b = fma(D[m * 3 + n.i], t, b);
  }
  double av = 0.0, ad = 0.0, bv = 0.0;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const int src = n.l + 3 * (m - n.j);
    const double s = shfl(a, src), t = shfl(b, src);
    av = fma(V[m * 3 + n.j], s, av);
    ad = fma(D[m * 3 + n.j], s, ad);
    bv = fma(V[m * 3 + n.j], t, bv);
  }
  g[0] = g[1] = g[2] = 0.0;
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const int src = n.l + 9 * (m - n.k);
    g[0] = fma(V[m * 3 + n.k], shfl(bv, src), g[0]);
    g[1] = fma(V[m * 3 + n.k], shfl(ad, src), g[1]);
    g[2] = fma(D[m * 3 + n.k], shfl(av, src), g[2]);
  }
}

// Its transpose: one component of the residual at the lane's node from the row p of JxW P
// at the points.
__device__ __forceinline__ double spread(const double* vd, const Lane& n, const double (&p)[3]) {
  const double *V = vd, *D = vd + 9;
  double x = 0.0, y = 0.0, z = 0.0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int src = n.l + 9 * (q - n.k);
    x = fma(V[n.k * 3 + q], shfl(p[0], src), x);
    y = fma(V[n.k * 3 + q], shfl(p[1], src), y);
    z = fma(D[n.k * 3 + q], shfl(p[2], src), z);
  }
  double s = 0.0, t = 0.0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int src = n.l + 3 * (q - n.j);
    s = fma(V[n.j * 3 + q], shfl(x, src), s);
    t = fma(D[n.j * 3 + q], shfl(y, src), fma(V[n.j * 3 + q], shfl(z, src), t));
  }
  double r = 0.0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int src = n.l + q - n.i;
    r = fma(D[n.i * 3 + q], shfl(s, src), fma(V[n.i * 3 + q], shfl(t, src), r));
  }
  return r;
}

__device__ __forceinline__ void point_phase(const ElemArgs& g, const double* vd, const Lane& n, double w, int node,
                                            RefPoint& m) {
  double G[3][3], D[3][3], uo[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double x = __ldg(&g.coords[int64_t(node) * 3 + d]);
    uo[d] = __ldg(&g.U[int64_t(node) * 3 + d]);
    gradient(vd, n, x, G[d]);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) gradient(vd, n, uo[d], D[d]);
  ref_point(g.props, G, D, w, m);
}

__device__ __forceinline__ Lane lane_place() {
  const int lane = threadIdx.x & 31, l = lane < A ? lane : A - 1;  // (the last lanes repeat node 26)
  return {l, l % 3, l / 3 % 3, l / 9};
}

// c + a b and c + a0 b0 + a1 b1 without renormalisation (df64_dot3_acc_lazy)
__device__ __forceinline__ float2 acc_sum(float2 c, float p) {
  const float t = __fadd_rn(c.x, p), v = __fsub_rn(t, c.x);
  return make_float2(t, __fadd_rn(c.y, __fadd_rn(__fsub_rn(c.x, __fsub_rn(t, v)), __fsub_rn(p, v))));
}
__device__ __forceinline__ float2 acc1(float2 c, float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = __fmaf_rn(a.x, b.x, -p);
  e = __fmaf_rn(a.x, b.y, e);
  e = __fmaf_rn(a.y, b.x, e);
  c.y = __fadd_rn(c.y, e);
  return acc_sum(c, p);
}
__device__ __forceinline__ float2 acc2(float2 c, float2 a0, float2 b0, float2 a1, float2 b1) {
  const float p0 = __fmul_rn(a0.x, b0.x), p1 = __fmul_rn(a1.x, b1.x);
  float e = __fmaf_rn(a0.x, b0.x, -p0);
  e = __fmaf_rn(a0.x, b0.y, e);
  e = __fmaf_rn(a0.y, b0.x, e);
  e = __fadd_rn(__fmaf_rn(a1.x, b1.x, -p1), e);
  e = __fmaf_rn(a1.x, b1.y, e);
  e = __fmaf_rn(a1.y, b1.x, e);
  c.y = __fadd_rn(c.y, e);
  return acc_sum(acc_sum(c, p0), p1);
}

// V_m, D_m at a point of one direction
struct Fn {
  float2 V[3], D[3];
  __device__ __forceinline__ Fn(const float2* vd2, int q) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      V[m] = vd2[m * 3 + q];
      D[m] = vd2[9 + m * 3 + q];
    }
  }
};

// c + p, 2 c, c / 2, c / 4 without renormalisation
__device__ __forceinline__ float2 acc0(float2 c, float2 p) {
  c.y = __fadd_rn(c.y, p.y);
  return acc_sum(c, p.x);
}
__device__ __forceinline__ float2 scaled(float2 p, float f) { return make_float2(p.x * f, p.y * f); }  // f a power of two

// out[a][b] += sum_(s,t) x(s)_a x(t)_b G[s][t]
__device__ __forceinline__ void expand(float2 (&out)[9], const Fn& f, float2 G00, float2 G01, float2 G10, float2 G11) {
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const float2 u0 = df64_dot2(f.V[b], G00, f.D[b], G01), u1 = df64_dot2(f.V[b], G10, f.D[b], G11);
#pragma unroll
    for (int a = 0; a < 3; ++a) out[a * 3 + b] = acc2(out[a * 3 + b], f.V[a], u0, f.D[a], u1);
  }
}

__device__ void place(int it, unsigned short* W) {
  const bool off = it < 243;
  const int d = off ? it : it - 243, per = off ? 81 : 45;
  const int f = d / per, r = d - f * per;
  int i = f, k = f, a1b1, a2b2, m1;
  if (off) {
    i = f == 2;
    k = f == 0 ? 1 : 2;
    m1 = a1b1 = r % 9;
    a2b2 = r / 9;
  } else if (r < 27) {  // a1 < b1
    m1 = r % 3 == 2 ? 4 : r % 3 + 1;
    a1b1 = r % 3 == 2 ? 5 : r % 3 + 1;
    a2b2 = r / 3;
  } else {              // a1 = b1, a2 <= b2
    const int s = r - 27, h = s / 3;
    m1 = s % 3 == 2 ? 5 : s % 3 * 3;
    a1b1 = s % 3 * 4;
    a2b2 = h < 3 ? h : h < 5 ? h + 1 : 8;
  }
  const bool self = a1b1 % 4 == 0 && a2b2 % 4 == 0;
  const int a0 = a1b1 / 3 + a2b2 / 3 * 3, b0 = a1b1 % 3 + a2b2 % 3 * 3;
  for (int m = 0; m < 9; ++m)  // i = k: a3 <= b3 where a1 = b1 and a2 = b2
    W[m] = !off && self && m / 3 > m % 3 ? 65535 : pair_entry(A, a0 + m / 3 * 9, i, b0 + m % 3 * 9, k);
  W[9] = (off ? f * T2_OFF + a2b2 * 9 : 3 * T2_OFF + f * T2_DIAG + a2b2 * 6) + m1 + (off && self ? (k - i) << 14 : 0);
}
// the nodes of pair n, a <= b
__device__ __forceinline__ void pair_nodes(int n, int& a, int& b) {
  a = 0;
  while (n >= A - a) n -= A - a++;
  b = a + n;
}

// An item of the first two directions.
struct First {
  int ent, out, n1, ab1;  // where its entries and results start, stride of the latter, (a1, b1)
  __device__ __forceinline__ explicit First(int t) {
    const bool off = t < 81;
    const int d = off ? t : t - 81, per = off ? 27 : 18, f = d / per, m1 = d % per / 3, q3 = d % 3;
    n1 = off ? 9 : 6;
    ab1 = off ? m1 : (m1 < 3 ? m1 : m1 < 5 ? m1 + 1 : 8);  // (00, 01, 02, 11, 12, 22)
    ent = (off ? f : f + 3) * 9 * NQ + q3 * 9;
    out = (off ? f * T2_OFF : 3 * T2_OFF + f * T2_DIAG) + q3 * 9 * n1 + m1;
  }
  // the entry (J, L) at (q2, q3), summed over q1
  __device__ __forceinline__ float2 sum(const Smem& S, const float2* ents, int J, int L, int q2) const {
    const float2* s = ents + ent + (J * 3 + L) * NQ + q2 * 3;
    const float2* p = S.prod[(J == 0 ? 2 : 0) + (L == 0 ? 1 : 0)][ab1];
    return df64_dot3(p[0], s[0], p[1], s[1], p[2], s[2]);
  }
  __device__ __forceinline__ void put(float2* t2, int kind, const float2 (&o)[9]) const {
#pragma unroll
    for (int m = 0; m < 9; ++m) t2[out + (kind * 27 + m) * n1] = df64_renorm(o[m]);
  }
};

// The same at the middle point, where V = (0, 1, 0) and D = (-1/2, 0, 1/2), as the
// first contribution.
__device__ __forceinline__ void centre(float2 (&o)[9], float2 G00, float2 G01, float2 G10, float2 G11) {
  const float2 r = scaled(G01, 0.5f), c = scaled(G10, 0.5f), d = scaled(G11, 0.25f);
  o[0] = o[8] = d;
  o[2] = o[6] = df64_neg(d);
  o[4] = G00;
  o[3] = df64_neg(r);
  o[5] = r;
  o[1] = df64_neg(c);
  o[7] = c;
}

template <bool WANT_R>
__global__ void __launch_bounds__(NTHR, 1) hex27_sum_kernel(ElemArgs g, const double* __restrict__ tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x;
  if (tid < 18) {
    const double v = __ldg(tab + tid);
    S.vd[tid] = v;
    S.vd2[tid] = df64_split(v);
  }
  if (tid < 108) {
    const int kind = tid / 27, ab = tid % 27 / 3, q = tid % 3;
    const double x = __ldg(tab + (kind & 2 ? T_D : T_V) + ab / 3 * 3 + q), y = __ldg(tab + (kind & 1 ? T_D : T_V) + ab % 3 * 3 + q);
    S.prod[kind][ab][q] = df64_split(mul_rn(x, y));
  }
  if (tid < 45) {
    // entry (r1, r2), r1 = 3i + J <= r2 = 3k + L: r1, r2, 3i + L, 3k + J, the index of c2 M
    // (7: none) and the entry's one or two places
    int r1 = 0, m = tid;
    for (int c = 0; c < 9; ++c)
      if (m >= 9 - r1) { m -= 9 - r1; ++r1; }
    const int r2 = r1 + m, i = r1 / 3, J = r1 % 3, k = r2 / 3, L = r2 % 3;
    const int f = i == k ? 3 + i : i + k - 1, M = i != k ? 7 : J == L ? J : 6 - J - L;
    const int d1 = f * 9 + J * 3 + L, d2 = i == k ? f * 9 + L * 3 + J : d1;
    S.code[tid] = uint32_t(r1 | r2 << 4 | (3 * i + L) << 8 | (3 * k + J) << 12 | M << 16 | d1 << 19 | d2 << 25);
  }
  if (tid < N_THIRD) place(tid, S.where[tid]);
  if (tid == 0) {
    for (int i = 0; i < NSLOT; ++i) {
      tc::mbar_init(S.full + i, 32);
      tc::mbar_init(S.empty + i, GT);
    }
    tc::mbar_fence_init();
  }
  __syncthreads();
  const int64_t G = gridDim.x;
  const long long budget = g.wait_budget > 0 ? g.wait_budget : WAIT_BUDGET;
  // a wait that gave up reports through the flag and waits again (the long budget)
  auto wait_or_report = [&](uint64_t* bar, int use) {
    if (!tc::mbar_wait(bar, uint32_t(use & 1), budget)) {
      if (g.wait_err) atomicExch(g.wait_err, 1);
      tc::mbar_wait(bar, uint32_t(use & 1), WAIT_BUDGET);
    }
  };

  if (tid >= NCON) {
    // ---------------- producer ----------------
    const Lane n = lane_place();
    const bool real = (tid & 31) < A;
    const double w = __ldg(tab + T_W + n.l);
    int64_t e = blockIdx.x + (tid - NCON) / 32 * G;
    int node = e < g.ne ? g.conn[e * A + n.l] : 0;
    for (int k = (tid - NCON) / 32; e < g.ne; e += NPROD * G, k += NPROD) {
      RefPoint m;
      const int at = node;
      if (e + NPROD * G < g.ne) node = g.conn[(e + NPROD * G) * A + n.l];
      point_phase(g, S.vd, n, w, at, m);
      const int slot = k % NSLOT, use = k / NSLOT;
      if (use) wait_or_report(S.empty + slot, use - 1);  // its last element's entries are formed
      if (real) {
        float2* st = &S.stage[slot][0][n.l];
        const float2 b = df64_split(m.b), a2 = df64_split(m.a2);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const float2 h = df64_split(m.H[i]);
          st[i * NQ] = h;
          st[(9 + i) * NQ] = tangent_z(b, h, m.P[i]);
          st[(18 + i) * NQ] = df64_mul(a2, h);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) st[(27 + i) * NQ] = df64_split(m.cM[i]);
      }
      mbar_arrive(S.full + slot);
      if (WANT_R)
#pragma unroll 1
        for (int i = 0; i < 3; ++i) {
          const double p[3] = {m.P[0], m.P[1], m.P[2]};
          const double r = spread(S.vd, n, p);
          if (real) static_cast<double*>(g.Re)[e * 81 + n.l * 3 + i] = r;
#pragma unroll
          for (int j = 0; j < 6; ++j) m.P[j] = m.P[j + 3];
        }
    }
    return;
  }

  // ---------------- contraction ----------------
  const int grp = tid / GT, gt = tid - grp * GT;
  // items (i, k), (a1, b1), q3 of the first two directions: this thread's, and of the last
  // ones a lane of the group's last warp takes one kind
  const int rest = gt - (GT - 32), kind0 = rest & 3;
  const First own(gt), last(GT + (rest >= 0 && rest < 4 * (N_FIRST - GT) ? rest >> 2 : 0));
  const float2 z = make_float2(0.f, 0.f);
  float2* t2 = S.t2[grp];
  const float2* ents = &S.ent[grp][0][0];
  int k = grp;
  for (int64_t e = blockIdx.x + grp * G; e < g.ne; e += NGRP * G, k += NGRP) {
    const int slot = k % NSLOT;
    wait_or_report(S.full + slot, k / NSLOT);
    // ---- tangent entries ----
    const float2* st = &S.stage[slot][0][0];
    for (int it = gt; it < 45 * NQ; it += GT) {
      const int w = it / NQ, q = it - w * NQ;
      const uint32_t c = S.code[w];
      const float2* H = st + q;
      const float2* Z = H + 9 * NQ;
      const float2* Y = H + 18 * NQ;
      const int r1 = int(c & 15u) * NQ, r2 = int(c >> 4 & 15u) * NQ, iL = int(c >> 8 & 15u) * NQ,
                kJ = int(c >> 12 & 15u) * NQ, M = int(c >> 16 & 7u);
      float2 v = df64_dot3(H[r1], Z[r2], Z[r1], H[r2], Y[iL], H[kJ]);
      if (M != 7) v = df64_add(v, st[(27 + M) * NQ + q]);
      S.ent[grp][c >> 19 & 63u][q] = v;
      S.ent[grp][c >> 25][q] = v;
    }
    mbar_arrive(S.empty + slot);
    named_sync(BAR_GRP + grp, GT);
    // ---- first and second direction ----
    {
      auto first = [&](int J, int L, int q2) { return own.sum(S, ents, J, L, q2); };
      auto put = [&](int kind, const float2 (&o)[9]) { own.put(t2, kind, o); };
      float2 o[9];
      // J, L along the first two directions
      centre(o, first(0, 0, 1), first(0, 1, 1), first(1, 0, 1), first(1, 1, 1));
#pragma unroll 1
      for (int q2 = 0; q2 < 3; q2 += 2)
        expand(o, Fn(S.vd2, q2), first(0, 0, q2), first(0, 1, q2), first(1, 0, q2), first(1, 1, q2));
      put(0, o);
      // L along the third
#pragma unroll
      for (int m = 0; m < 9; ++m) o[m] = z;
      {
        const float2 G1 = scaled(first(1, 2, 1), 0.5f);
        o[1] = df64_neg(G1);
        o[4] = first(0, 2, 1);
        o[7] = G1;
      }
#pragma unroll 1
      for (int q2 = 0; q2 < 3; q2 += 2) {
        const Fn f(S.vd2, q2);
        const float2 G0 = first(0, 2, q2), G1 = first(1, 2, q2);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float2 u = df64_dot2(f.V[a], G0, f.D[a], G1);
#pragma unroll
          for (int b = 0; b < 3; ++b) o[a * 3 + b] = acc1(o[a * 3 + b], f.V[b], u);
        }
      }
      put(1, o);
      // J along the third
#pragma unroll
      for (int m = 0; m < 9; ++m) o[m] = z;
      {
        const float2 G1 = scaled(first(2, 1, 1), 0.5f);
        o[3] = df64_neg(G1);
        o[4] = first(2, 0, 1);
        o[5] = G1;
      }
#pragma unroll 1
      for (int q2 = 0; q2 < 3; q2 += 2) {
        const Fn f(S.vd2, q2);
        const float2 G0 = first(2, 0, q2), G1 = first(2, 1, q2);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const float2 u = df64_dot2(f.V[b], G0, f.D[b], G1);
#pragma unroll
          for (int a = 0; a < 3; ++a) o[a * 3 + b] = acc1(o[a * 3 + b], f.V[a], u);
        }
      }
      put(2, o);
      // both
#pragma unroll
      for (int m = 0; m < 9; ++m) o[m] = z;
      o[4] = first(2, 2, 1);
#pragma unroll 1
      for (int q2 = 0; q2 < 3; q2 += 2) {
        const Fn f(S.vd2, q2);
        const float2 G0 = first(2, 2, q2);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const float2 u = df64_mul(f.V[b], G0);
#pragma unroll
          for (int a = 0; a < 3; ++a) o[a * 3 + b] = acc1(o[a * 3 + b], f.V[a], u);
        }
      }
      put(3, o);
    }
    if (rest >= 0 && rest < 4 * (N_FIRST - GT)) {
      // (J, L) for (s, t): 2 where the kind has it along the third direction, which leaves s
      // (or t) = 0
      auto G = [&](int s, int t, int q2) {
        return (kind0 & 2 && s) || (kind0 & 1 && t) ? z : last.sum(S, ents, kind0 & 2 ? 2 : s, kind0 & 1 ? 2 : t, q2);
      };
      float2 o[9];
      centre(o, G(0, 0, 1), G(0, 1, 1), G(1, 0, 1), G(1, 1, 1));
#pragma unroll 1
      for (int q2 = 0; q2 < 3; q2 += 2) expand(o, Fn(S.vd2, q2), G(0, 0, q2), G(0, 1, q2), G(1, 0, q2), G(1, 1, q2));
      last.put(t2, kind0, o);
    }
    named_sync(BAR_GRP + grp, GT);
    // ---- third direction ----
#pragma unroll 1
    for (int it = gt; it < N_THIRD; it += GT) {
      const unsigned short* W = S.where[it];
      const int w9 = W[9], n = it < 243 ? 9 : 6, twin = w9 >> 14;
      const float2* t = t2 + (w9 & 8191);
      float2 o[9];
      centre(o, t[9 * n], t[36 * n], t[63 * n], t[90 * n]);
#pragma unroll 1
      for (int q = 0; q < 3; q += 2, t += 18 * n)
        expand(o, Fn(S.vd2, q), t[0], t[27 * n], t[54 * n], t[81 * n]);
      if (g.ke_pairs) {
        float2* Kp = static_cast<float2*>(g.Ke) + e * (A * (A + 1) / 2 * 9);
#pragma unroll
        for (int m = 0; m < 9; ++m) {
          const float2 v = df64_renorm(o[m]);
          const int w = W[m];
          if (w != 65535) Kp[w] = v;
          if (m % 4 == 0 && twin) Kp[w + 2 * twin] = v;
        }
      } else {
        float2* Ke = static_cast<float2*>(g.Ke) + e * (81 * 81);
#pragma unroll
        for (int m = 0; m < 9; ++m) {
          const float2 v = df64_renorm(o[m]);
          const int w = W[m];
          if (w == 65535) continue;
          int a, b;
          pair_nodes(w / 9, a, b);
          const int r = a * 3 + w % 9 / 3, c = b * 3 + w % 3;
          Ke[r * 81 + c] = v;
          Ke[c * 81 + r] = v;
        }
      }
    }
  }
}

// Residual only: the same point phase and residual, one warp per element.
constexpr int R_WARPS = 4;
__global__ void __launch_bounds__(32 * R_WARPS) hex27_sum_r_kernel(ElemArgs g, const double* __restrict__ tab) {
  __shared__ double s_vd[18];
  if (threadIdx.x < 18) s_vd[threadIdx.x] = __ldg(tab + threadIdx.x);
  __syncthreads();
  const int64_t e = int64_t(blockIdx.x) * R_WARPS + (threadIdx.x >> 5);
  if (e >= g.ne) return;
  const Lane n = lane_place();
  RefPoint m;
  point_phase(g, s_vd, n, __ldg(tab + T_W + n.l), g.conn[e * A + n.l], m);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double p[3] = {m.P[i * 3], m.P[i * 3 + 1], m.P[i * 3 + 2]};
    const double r = spread(s_vd, n, p);
    if ((threadIdx.x & 31) < A) static_cast<double*>(g.Re)[e * 81 + n.l * 3 + i] = r;
  }
}

template <bool WANT_R>
cudaError_t launch(const ElemArgs& a, cudaStream_t s) {
  const cudaError_t e = ensure_smem<hex27_sum_kernel<WANT_R>>(sizeof(Smem));
  if (e != cudaSuccess) return e;
  const int64_t cap = int64_t(num_sms());
  const unsigned grid = unsigned(a.ne < cap ? a.ne : cap);
  hex27_sum_kernel<WANT_R><<<grid, NTHR, sizeof(Smem), s>>>(a, static_cast<const double*>(a.general));
  return cudaGetLastError();
}

}  // namespace h27

bool hex27_general_enabled() {
  const char* v = std::getenv("FEC_HEX27_GENERAL");
  return !(v && v[0] == '0');
}

cudaError_t launch_hex27_general(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (!a.general || (want_k && !a.Ke) || (want_r && !a.Re)) return cudaErrorInvalidValue;
  if (a.ne <= 0 || (!want_r && !want_k)) return cudaSuccess;
  ++*launches;
  if (want_k) return want_r ? h27::launch<true>(a, s) : h27::launch<false>(a, s);
  const int64_t nb = (a.ne + h27::R_WARPS - 1) / h27::R_WARPS;
  h27::hex27_sum_r_kernel<<<unsigned(nb), 32 * h27::R_WARPS, 0, s>>>(a, static_cast<const double*>(a.general));
  return cudaGetLastError();
}

bool hex27_general_table(const double* ref, std::vector<unsigned char>& out) {
  using namespace h27;
  const double* N = ref + RefLayout<8>::N_OFF;
  const double* dN = ref + RefLayout<8>::DN_OFF;
  double t[T_DOUBLES] = {0.0};
  for (int m = 0; m < 3; ++m)
    for (int q = 0; q < 3; ++q) {  // along the line through the middle of the other directions
      t[T_V + m * 3 + q] = N[(q + 12) * A + m + 12];
      t[T_D + m * 3 + q] = dN[((q + 12) * A + m + 12) * 3];
    }
  for (int m = 0; m < 3; ++m)
    if (t[T_V + m * 3 + 1] != (m == 1 ? 1.0 : 0.0) || t[T_D + m * 3 + 1] != 0.5 * (m - 1)) return false;
  for (int q = 0; q < NQ; ++q) {
    t[T_W + q] = ref[RefLayout<8>::W_OFF + q];
    for (int a = 0; a < A; ++a)
      for (int J = 0; J < 3; ++J) {
        double v = 1.0;
        for (int d = 0, aa = a, qq = q; d < 3; ++d, aa /= 3, qq /= 3) v *= t[(d == J ? T_D : T_V) + aa % 3 * 3 + qq % 3];
        if (!(std::fabs(v - dN[(q * A + a) * 3 + J]) <= 4e-15)) return false;
      }
  }
  out.resize(sizeof t);
  std::memcpy(out.data(), t, sizeof t);
  return true;
}

}  // namespace fec
