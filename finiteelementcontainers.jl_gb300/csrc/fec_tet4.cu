// fec_tet4.cu -- FP64 tet4 Neo-Hookean elements (one point, constant gradients).
//
// In reference coordinates dN_0 = -(1, 1, 1), dN_j = e_j, so dX/dxi are coordinate
// differences and with h_a, z_a, y_a the columns of H, Z, Y and h_0 = -(h_1 + h_2 + h_3)
// and so on (GenNeoHookean, fec_digits.cuh)
//     K_(a,i),(b,k) = h_ai z_bk + z_ai h_bk + y_bi h_ak + d_ik (c2 M)_ab,   R_(a,i) = P_ia .
// First a thread per element: the update in FP64, the residual, the 46 values of the
// tangent split into shared memory; then a thread per entry of the symmetric half
// (KE_PAIRS, 90 entries an element), in double-float, consecutive threads consecutive
// entries.
//
// What bounds it: the FP64 operations of the update, about 320 an element.  82,368
// elements 0.077 ms (0.369 with the per-element kernel: a thread per matrix row, entries of A
// formed in FP64, then contracted in double-float over nine places each).
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "fec_digits.cuh"
#include "fec_kernels.cuh"
#include "fec_launch.h"

namespace fec {
namespace t4 {

using namespace aff;

constexpr int EPB = 64, NENT = 90, S_H = 0, S_Z = 12, S_Y = 24, S_M = 36, STRIDE = 47;  // (odd: no bank conflicts)

template <bool WANT_R, bool WANT_K>
__global__ void __launch_bounds__(EPB) tet4_kernel(ElemArgs g, const double* __restrict__ tab) {
  __shared__ float2 s_val[WANT_K ? EPB * STRIDE : 1];  // per element h, z, y [4][3], c2 M [10]
  __shared__ uint32_t s_code[WANT_K ? NENT : 1];       // of an entry: its factors' places
  const int tid = threadIdx.x;
  const int64_t e0 = int64_t(blockIdx.x) * EPB, e = e0 + tid;
  if (WANT_K)
    for (int t = tid; t < NENT; t += EPB) {
      int a = 0, m = t / 9;
      while (m >= 4 - a) m -= 4 - a++;
      const int b = a + m, i = t % 9 / 3, k = t % 3;
      s_code[t] = uint32_t(a * 3 + i) | uint32_t(b * 3 + k) << 4 | uint32_t(b * 3 + i) << 8 | uint32_t(a * 3 + k) << 12 |
                  uint32_t(i == k ? S_M + t / 9 : 63) << 16;
    }
  if (e < g.ne) {
    int node[4];  // (a block's connectivity starts at any multiple of 4 bytes)
#pragma unroll
    for (int a = 0; a < 4; ++a) node[a] = __ldg(g.conn + e * 4 + a);
    double G[3][3], D[3][3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double x0 = __ldg(&g.coords[int64_t(node[0]) * 3 + d]), u0 = __ldg(&g.U[int64_t(node[0]) * 3 + d]);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        G[d][j] = __ldg(&g.coords[int64_t(node[j + 1]) * 3 + d]) - x0;
        D[d][j] = __ldg(&g.U[int64_t(node[j + 1]) * 3 + d]) - u0;
      }
    }
    RefPoint m;
    ref_point<true>(g.props, G, D, __ldg(tab), m);
    double P0[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) P0[i] = -((m.P[i * 3] + m.P[i * 3 + 1]) + m.P[i * 3 + 2]);
    if (WANT_R) {
      double* R = static_cast<double*>(g.Re) + e * 12;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        R[i] = P0[i];
#pragma unroll
        for (int j = 0; j < 3; ++j) R[(j + 1) * 3 + i] = m.P[i * 3 + j];
      }
    }
    if (WANT_K) {
      float2* s = s_val + tid * STRIDE;
      const float2 b = df64_split(m.b), a2 = df64_split(m.a2);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float2 h = df64_split(a ? m.H[i * 3 + a - 1] : -((m.H[i * 3] + m.H[i * 3 + 1]) + m.H[i * 3 + 2]));
          s[S_H + a * 3 + i] = h;
          s[S_Z + a * 3 + i] = tangent_z(b, h, a ? m.P[i * 3 + a - 1] : P0[i]);
          s[S_Y + a * 3 + i] = df64_mul(a2, h);
        }
      const double* M = m.cM;  // xx, yy, zz, yz, xz, xy
      const double m0[3] = {-((M[0] + M[5]) + M[4]), -((M[5] + M[1]) + M[3]), -((M[4] + M[3]) + M[2])};
      const double v[10] = {-((m0[0] + m0[1]) + m0[2]), m0[0], m0[1], m0[2], M[0], M[5], M[4], M[1], M[3], M[2]};
#pragma unroll
      for (int n = 0; n < 10; ++n) s[S_M + n] = df64_split(v[n]);
    }
  }
  if (!WANT_K) return;
  __syncthreads();
  const int live = int(g.ne - e0 < EPB ? g.ne - e0 : EPB);
  float2* dst = static_cast<float2*>(g.Ke) + e0 * NENT;
  for (int t = tid; t < live * NENT; t += EPB) {
    const int el = t / NENT;
    const uint32_t c = s_code[t - el * NENT];
    const float2* s = s_val + el * STRIDE;
    const int ai = int(c & 15u), bk = int(c >> 4 & 15u), bi = int(c >> 8 & 15u), ak = int(c >> 12 & 15u), M = int(c >> 16);
    float2 v = df64_dot3(s[S_H + ai], s[S_Z + bk], s[S_Z + ai], s[S_H + bk], s[S_Y + bi], s[S_H + ak]);
    if (M != 63) v = df64_add(v, s[M]);
    dst[t] = v;
  }
}

}  // namespace t4

bool tet4_general_enabled() {
  const char* v = std::getenv("FEC_TET4_GENERAL");
  return !(v && v[0] == '0');
}

cudaError_t launch_tet4_general(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (!a.general || (want_k && !a.Ke) || (want_r && !a.Re)) return cudaErrorInvalidValue;
  if (a.ne <= 0 || (!want_r && !want_k)) return cudaSuccess;
  ++*launches;
  const unsigned nb = unsigned((a.ne + t4::EPB - 1) / t4::EPB);
  const double* tab = static_cast<const double*>(a.general);
  if (!want_k)
    t4::tet4_kernel<true, false><<<nb, t4::EPB, 0, s>>>(a, tab);
  else if (want_r)
    t4::tet4_kernel<true, true><<<nb, t4::EPB, 0, s>>>(a, tab);
  else
    t4::tet4_kernel<false, true><<<nb, t4::EPB, 0, s>>>(a, tab);
  return cudaGetLastError();
}

bool tet4_general_table(const double* ref, std::vector<unsigned char>& out) {
  for (int a = 0; a < 4; ++a)
    for (int j = 0; j < 3; ++j)
      if (ref[RefLayout<6>::DN_OFF + a * 3 + j] != (a == 0 ? -1.0 : (a == j + 1 ? 1.0 : 0.0))) return false;
  out.resize(sizeof(double));
  std::memcpy(out.data(), ref + RefLayout<6>::W_OFF, sizeof(double));
  return true;
}

}  // namespace fec
