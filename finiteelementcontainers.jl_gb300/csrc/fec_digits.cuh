// fec_digits.cuh -- what the exact-digit tensor-core element kernels share
// (fec_hex8_affine_tc.cu, fec_tet10_tc.cu; the scheme is described in the former): the
// Neo-Hookean update and its tangent entries, the accumulators' levels, barriers.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

#include "fec_df64.cuh"
#include "fec_kernels.cuh"
#include "fec_tc.cuh"

namespace fec {
namespace aff {

constexpr int ND = 7;                // digits per operand
constexpr int NLEV = 7;              // accumulated levels s + t = 0..6
constexpr long long WAIT_BUDGET = 2000000000LL;

__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int n) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
// 2^k as a float for k in [-126, 127]
__device__ __forceinline__ float pow2f(int k) { return __uint_as_float(uint32_t(k + 127) << 23); }

// Host: the seven digits of w, |w| < 2^e, at their place values 2^(-8s), as BF16 (each
// exact).  Rounding by adding and subtracting 1.5 2^52: a table has 18,000 digits, whose
// nearbyint and ldexp calls took 0.2 ms of setting a mesh.
inline void bf16_digits(double w, int e, uint16_t (&out)[ND]) {
  double y = std::ldexp(w, 7 - e), place = 1.0;  // |y| < 128, exact
  for (int s = 0; s < ND; ++s, place *= 0x1p-8) {
    const double d = (y + 0x1.8p52) - 0x1.8p52;
    y = (y - d) * 256.0;
    const float f = float(d * place);
    uint32_t u;
    std::memcpy(&u, &f, 4);
    out[s] = uint16_t(u >> 16);
  }
}

// Seven 4-column loads (the seven levels of one column chunk) under one wait.
// NPAD: columns of a level.
template <int NPAD>
__device__ __forceinline__ void tmem_ld4x7(uint32_t taddr, float (*v)[4]) {
  uint32_t r[28];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%28];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4, %5, %6, %7}, [%29];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%8, %9, %10, %11}, [%30];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%12, %13, %14, %15}, [%31];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%16, %17, %18, %19}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%20, %21, %22, %23}, [%33];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%24, %25, %26, %27}, [%34];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27])
      : "r"(taddr), "r"(taddr + 1u * NPAD), "r"(taddr + 2u * NPAD), "r"(taddr + 3u * NPAD), "r"(taddr + 4u * NPAD),
        "r"(taddr + 5u * NPAD), "r"(taddr + 6u * NPAD)
      : "memory");
#pragma unroll
  for (int L = 0; L < NLEV; ++L)
#pragma unroll
    for (int j = 0; j < 4; ++j) v[L][j] = __uint_as_float(r[L * 4 + j]);
}

// The sum of the seven level accumulators of one pair: levels 6..4 in FP32 (their
// rounding is below 2^-55 of level 0), then 3..0 in double-float
__device__ __forceinline__ float2 combine_levels(const float (&v)[NLEV][4], int j) {
  float hi = (v[6][j] + v[5][j]) + v[4][j], lo = 0.f;
#pragma unroll
  for (int L = 3; L >= 0; --L) {
    const float a = v[L][j], b = hi;
    const float s = a + b, bb = s - a;
    lo += (a - (s - bb)) + (b - bb);
    hi = s + lo;
    lo = lo - (hi - s);
  }
  return make_float2(hi, lo);
}

// a0 b0 + a1 b1 in double-float
__device__ __forceinline__ float2 df64_dot2(float2 a0, float2 b0, float2 a1, float2 b1) {
  const float p0 = __fmul_rn(a0.x, b0.x), p1 = __fmul_rn(a1.x, b1.x);
  float e = __fmaf_rn(a0.x, b0.x, -p0);
  e = __fmaf_rn(a0.x, b0.y, e);
  e = __fmaf_rn(a0.y, b0.x, e);
  e = __fadd_rn(__fmaf_rn(a1.x, b1.x, -p1), e);
  e = __fmaf_rn(a1.x, b1.y, e);
  e = __fmaf_rn(a1.y, b1.x, e);
  const float t = __fadd_rn(p0, p1), v = __fsub_rn(t, p0);
  return df64_fast2sum(t, __fadd_rn(e, __fadd_rn(__fsub_rn(p0, __fsub_rn(t, v)), __fsub_rn(p1, v))));
}
// The Neo-Hookean update as the tensor-core kernel takes it.  With H = F^-T and the
// stress P = c2 F - a2 H (a1, a2, c2, P times JxW; see NeoHookean) the tangent entry
// is three products of per-point vectors,
//   A_iJkL = H_iJ Z_kL + Z_iJ H_kL + Y_iL H_kJ + c2 d_ik d_JL,
//   Z = a1/2 H - 2/3 c2 F = -2/3 P + b H,  b = a1/2 - 2/3 a2,   Y = a2 H,
// instead of four products of products, and a point hands on H, P (which the
// residual needs anyway) and three scalars.  Every product that feeds a sum is an
// explicit FMA or rounded on its own, so the residual-only kernel gives the same
// bits.
struct AffNeoHookean {
  static constexpr int NS = 0, SCR2 = 12;  // H, b, a2, c2
  static constexpr bool TANGENT_P = true;  // the slicers read the stress
  static constexpr bool GENERAL = false;
  static constexpr bool TENSOR = true;     // hex8: the tables of a symmetric rule (AnyRule: any others)
  static constexpr int PROD_GROUPS = 2, STAGES = 2;  // of the hex8 kernel
  struct Mid {
    double F[9], H[9], a1h, a2, c2, J, I13, r2;  // (r2 = J^(-2/3))
  };
  // J^(-1/3): CUDA's FP32 rcbrtf and one third-order step from the expansion of
  // (1 - e)^(-1/3), e = 1 - J r^3 (e is below 2^-20, the dropped term below
  // 2^-62); the library function outside FP32's range.
  __device__ static double inv_cbrt(double J) {
    if (!(J > 1e-30 && J < 1e30)) return rcbrt(J);
    const double r = double(rcbrtf(float(J)));
    const double e = fma(-J * r, r * r, 1.0);
    return fma(r * e, fma(e, 2.0 / 9.0, 1.0 / 3.0), r);
  }
  __device__ static void point(const double* props, const double (&gu)[3][3], double jxw, const double*, double*,
                               Mid& m) {
    const double Kj = props[0] * jxw, Gj = props[1] * jxw;
#pragma unroll
    for (int i = 0; i < 9; ++i) m.F[i] = gu[i / 3][i % 3] + (i % 4 == 0 ? 1.0 : 0.0);
    const double* F = m.F;
    double c[9];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {  // cofactors (cyclic indices: no signs)
        const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
        c[i * 3 + j] = fma(F[i1 * 3 + j1], F[i2 * 3 + j2], -mul_rn(F[i1 * 3 + j2], F[i2 * 3 + j1]));
      }
    const double J = fma(F[0], c[0], fma(F[1], c[1], mul_rn(F[2], c[2])));
    const double rJ = 1.0 / J;
    double I1 = mul_rn(F[0], F[0]);
#pragma unroll
    for (int i = 1; i < 9; ++i) I1 = fma(F[i], F[i], I1);
    const double r3 = inv_cbrt(J);
    const double I13 = mul_rn(I1, 1.0 / 3.0);
    const double JJ = mul_rn(J, J), d = JJ - J;
    m.J = J;
    m.I13 = I13;
    m.r2 = mul_rn(r3, r3);
    m.c2 = mul_rn(m.r2, Gj);
    m.a2 = fma(m.c2, I13, -mul_rn(0.5 * Kj, d - 1.0));
    m.a1h = fma(m.c2, mul_rn(I13, 1.0 / 3.0), mul_rn(0.25 * Kj, JJ + d));
#pragma unroll
    for (int i = 0; i < 9; ++i) m.H[i] = mul_rn(c[i], rJ);
  }
  __device__ static void stress(const Mid& m, float2* P) {
#pragma unroll
    for (int i = 0; i < 9; ++i) P[i] = df64_split(fma(m.c2, m.F[i], -mul_rn(m.a2, m.H[i])));
  }
  // (A : D)_iJ = (a1 h + m f) H + m h F + a2 H D^T H + c2 D, h = H : D, f = F : D, m = -2/3 c2
  __device__ static void action(const Mid& m, const double (&D)[3][3], double (&out)[3][3]) {
    const double m23 = mul_rn(-2.0 / 3.0, m.c2);
    action_terms(m.H, m.F, D, D, 2.0 * m.a1h, m.a2, m23, m.c2, out);
  }
  // (a1 h + m f) H + m h Q + a2 H D^T H + c E, h = H : D, f = Q : D
  __device__ static void action_terms(const double* H, const double* Q, const double (&D)[3][3],
                                      const double (&E)[3][3], double a1, double a2, double m, double c,
                                      double (&out)[3][3]) {
    double h = 0.0, f = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      h = fma(H[k], D[k / 3][k % 3], h);
      f = fma(Q[k], D[k / 3][k % 3], f);
    }
    const double s1 = fma(a1, h, mul_rn(m, f)), s2 = mul_rn(m, h);
    double M[3][3];  // a2 (D^T H)
#pragma unroll
    for (int l = 0; l < 3; ++l)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        M[l][j] = mul_rn(a2, fma(D[0][l], H[j], fma(D[1][l], H[3 + j], mul_rn(D[2][l], H[6 + j]))));
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        out[i][j] = fma(H[i * 3], M[0][j],
                        fma(H[i * 3 + 1], M[1][j],
                            fma(H[i * 3 + 2], M[2][j],
                                fma(c, E[i][j], fma(s2, Q[i * 3 + j], mul_rn(s1, H[i * 3 + j]))))));
  }
  // the point's split stress and tangent scratch; returns a bound of |A_iJkL|
  __device__ static float stage(const Mid& m, float2* P, float2* scr) {
    float hm = 0.f, pm = 0.f;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const float2 h = df64_split(m.H[i]), p = df64_split(fma(m.c2, m.F[i], -mul_rn(m.a2, m.H[i])));
      P[i] = p;
      scr[i] = h;
      hm = fmaxf(hm, fabsf(h.x));
      pm = fmaxf(pm, fabsf(p.x));
    }
    const float2 b = df64_split(fma(-2.0 / 3.0, m.a2, m.a1h)), a2 = df64_split(m.a2), c2 = df64_split(m.c2);
    scr[9] = b;
    scr[10] = a2;
    scr[11] = c2;
    return (2.f * (0.67f * pm + fabsf(b.x) * hm) + fabsf(a2.x) * hm) * hm + fabsf(c2.x);
  }
  // what a slicer thread keeps of its point (of these, the vectors its entries read)
  struct Tangent {
    float2 H[9], Z[9], Y[9], c2;
  };
  __device__ static void load(const float2* scr, const float2* P, Tangent& t) {
    const float2 m23 = make_float2(-0.666666686534881591796875f, 1.98682155172491e-08f);  // -2/3 to 2^-50
    const float2 b = scr[9], a2 = scr[10];
    t.c2 = scr[11];
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      t.H[i] = scr[i];
      t.Z[i] = df64_fma(b, t.H[i], df64_mul(m23, P[i]));
      t.Y[i] = df64_mul(a2, t.H[i]);
    }
  }
  __device__ static float2 entry(const Tangent& t, int i, int J, int k, int L) {
    float2 v = df64_dot3(t.H[i * 3 + J], t.Z[k * 3 + L], t.Z[i * 3 + J], t.H[k * 3 + L], t.Y[i * 3 + L],
                         t.H[k * 3 + J]);
    if (i == k && J == L) v = df64_add(v, t.c2);
    return v;
  }
};

// Neo-Hookean on an element of any shape: the same contraction in reference coordinates.  With
// G = dX/dxi, D = du/dxi and Gi = G^-1 at a point, F = I + D Gi, and the update of F pulled
// back to the reference element (indices J -> alpha through Gi) reads
//   H_ia = (F^-T Gi^T)_ia,   P_ia = (P Gi^T)_ia,   M = Gi Gi^T,
//   A_iakb = H_ia Z_kb + Z_ia H_kb + Y_ib H_ka + c2 d_ik M_ab,
// so the constant operand is that of the reference element's own gradients, whatever
// the element's shape.
// The update is formed in X and then pulled back: P is a difference of c2 F and a2 F^-T there,
// whose terms are of order one whatever the element.  Formed from dx/dxi and M det G^2
// (cofactor products) it is a difference of terms that grow with the square of the element's
// condition: errors of 6e-13 at an aspect ratio of 1000, where this has 4e-16.
struct PointUpdate {
  AffNeoHookean::Mid s;
  double Gi[3][3], jxw;
};
__device__ __forceinline__ void cofactors(const double (&F)[3][3], double (&c)[9]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
      c[i * 3 + j] = fma(F[i1][j1], F[i2][j2], -mul_rn(F[i1][j2], F[i2][j1]));
    }
}
// v Gi and v Gi^T
__device__ __forceinline__ void to_x(const double (&v)[3][3], const double (&Gi)[3][3], double (&out)[3][3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int j = 0; j < 3; ++j) out[d][j] = fma(v[d][0], Gi[0][j], fma(v[d][1], Gi[1][j], mul_rn(v[d][2], Gi[2][j])));
}
__device__ __forceinline__ double to_ref(const double* v, const double (&Gi)[3]) {
  return fma(v[0], Gi[0], fma(v[1], Gi[1], mul_rn(v[2], Gi[2])));
}
__device__ __forceinline__ void point_update(const double* props, const double (&G)[3][3], const double (&D)[3][3],
                                             double w, PointUpdate& m) {
  double gu[3][3], c[9];
  cofactors(G, c);
  const double detG = fma(G[0][0], c[0], fma(G[0][1], c[1], mul_rn(G[0][2], c[2]))), rG = 1.0 / detG;
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int j = 0; j < 3; ++j) m.Gi[j][d] = mul_rn(c[d * 3 + j], rG);
  to_x(D, m.Gi, gu);
  m.jxw = mul_rn(detG, w);
  AffNeoHookean::point(props, gu, m.jxw, nullptr, nullptr, m.s);
}
// The point's stress, H, c2 M, b and a2 (times JxW) in reference coordinates.  DEVIATOR: the
// stress as JxW (c1 H + G r2 (F - I1/3 H)), 20 operations more, which rounds a tenth less: where an
// element has one point, so that no sum averages that out.
struct RefPoint {
  double P[9], H[9], cM[6], b, a2;
};
template <bool DEVIATOR = false>
__device__ __forceinline__ void ref_point(const double* props, const double (&G)[3][3], const double (&D)[3][3],
                                          double w, RefPoint& m) {
  PointUpdate u;
  point_update(props, G, D, w, u);
  AffNeoHookean::Mid& s = u.s;
#pragma unroll
  for (int i = 0; i < 9; ++i) {  // the stress
    if (DEVIATOR) {
      const double c1 = mul_rn(0.5 * props[0], fma(s.J, s.J, -s.J) - 1.0), c2 = mul_rn(props[1], s.r2);
      s.F[i] = mul_rn(u.jxw, fma(c1, s.H[i], mul_rn(c2, fma(-s.I13, s.H[i], s.F[i]))));
    } else {
      s.F[i] = fma(s.c2, s.F[i], -mul_rn(s.a2, s.H[i]));
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      m.P[i * 3 + a] = to_ref(s.F + i * 3, u.Gi[a]);
      m.H[i * 3 + a] = to_ref(s.H + i * 3, u.Gi[a]);
    }
  constexpr int A[6] = {0, 1, 2, 1, 0, 0}, B[6] = {0, 1, 2, 2, 2, 1};
#pragma unroll
  for (int k = 0; k < 6; ++k) m.cM[k] = mul_rn(s.c2, to_ref(u.Gi[A[k]], u.Gi[B[k]]));
  m.b = fma(-2.0 / 3.0, s.a2, s.a1h);
  m.a2 = s.a2;
}

struct GenNeoHookean {
  static constexpr int NS = 0, SCR2 = 17;  // H, b, a2, c2 M (6)
  static constexpr bool GENERAL = true, TANGENT_P = true, TENSOR = true;
  static constexpr int PROD_GROUPS = 3, STAGES = 1;
  using Mid = RefPoint;
  __device__ static void stress(const Mid& m, float2* P) {
#pragma unroll
    for (int i = 0; i < 9; ++i) P[i] = df64_split(m.P[i]);
  }
  __device__ static void action(const PointUpdate& m, const double (&D)[3][3], double (&out)[3][3]) {
    double d[3][3], o[3][3];
    to_x(D, m.Gi, d);
    AffNeoHookean::action(m.s, d, o);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int a = 0; a < 3; ++a) out[i][a] = to_ref(o[i], m.Gi[a]);
  }
  __device__ static float stage(const Mid& m, float2* P, float2* scr) {
    float hm = 0.f, pm = 0.f, cm = 0.f;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const float2 h = df64_split(m.H[i]), p = df64_split(m.P[i]);
      P[i] = p;
      scr[i] = h;
      hm = fmaxf(hm, fabsf(h.x));
      pm = fmaxf(pm, fabsf(p.x));
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const float2 c = df64_split(m.cM[i]);
      scr[11 + i] = c;
      cm = fmaxf(cm, fabsf(c.x));
    }
    const float2 b = df64_split(m.b), a2 = df64_split(m.a2);
    scr[9] = b;
    scr[10] = a2;
    return (2.f * (0.67f * pm + fabsf(b.x) * hm) + fabsf(a2.x) * hm) * hm + cm;
  }
  struct Tangent {
    float2 H[9], Z[9], Y[9], cM[6];
  };
  __device__ static void load(const float2* scr, const float2* P, Tangent& t) {
    AffNeoHookean::Tangent u;
    AffNeoHookean::load(scr, P, u);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      t.H[i] = u.H[i];
      t.Z[i] = u.Z[i];
      t.Y[i] = u.Y[i];
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) t.cM[i] = scr[11 + i];
  }
  __device__ static float2 entry(const Tangent& t, int i, int J, int k, int L) {
    constexpr int S[9] = {0, 5, 4, 5, 1, 3, 4, 3, 2};
    float2 v = df64_dot3(t.H[i * 3 + J], t.Z[k * 3 + L], t.Z[i * 3 + J], t.H[k * 3 + L], t.Y[i * 3 + L],
                         t.H[k * 3 + J]);
    if (i == k) v = df64_add(v, t.cM[S[J * 3 + L]]);
    return v;
  }
};

// Z = -2/3 P + b H
__device__ __forceinline__ float2 tangent_z(float2 b, float2 h, double p) {
  const float2 m23 = make_float2(-0.666666686534881591796875f, 1.98682155172491e-08f);  // -2/3 to 2^-50
  return df64_fma(b, h, df64_mul(m23, df64_split(p)));
}

}  // namespace aff
}  // namespace fec
