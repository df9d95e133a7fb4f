// fec_poisson.cu -- instantiations of the Poisson element kernel.
#include <type_traits>
#include "fec_launch.h"

namespace fec {
namespace {

template <int ET, int EPB, typename Real>
cudaError_t go(bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  constexpr int TPE = Elem<ET>::NNPE;
  if (a.ne <= 0) return cudaSuccess;
  const dim3 block(TPE, EPB);
  const dim3 grid(unsigned((a.ne + EPB - 1) / EPB));
  if constexpr (ET == 1 && std::is_same<Real, double>::value) {
    if (a.affine && a.hex8_tensor) return launch_hex8_poisson(want_r, want_k, a, s, launches);
    if (a.affine) {  // a block of translated elements: its gradients and JxW from the affine table
      ElemArgs b = a;
      b.affine = static_cast<const unsigned char*>(a.affine) + hex8_affine_grad_offset();
      if (want_r && want_k)
        poisson_element_kernel<ET, Real, EPB, true, true, true><<<grid, block, 0, s>>>(b);
      else if (want_r)
        poisson_element_kernel<ET, Real, EPB, true, false, true><<<grid, block, 0, s>>>(b);
      else if (want_k)
        poisson_element_kernel<ET, Real, EPB, false, true, true><<<grid, block, 0, s>>>(b);
      else
        return cudaSuccess;
      ++*launches;
      return cudaGetLastError();
    }
  }
  if (want_r && want_k)
    poisson_element_kernel<ET, Real, EPB, true, true><<<grid, block, 0, s>>>(a);
  else if (want_r)
    poisson_element_kernel<ET, Real, EPB, true, false><<<grid, block, 0, s>>>(a);
  else if (want_k)
    poisson_element_kernel<ET, Real, EPB, false, true><<<grid, block, 0, s>>>(a);
  else
    return cudaSuccess;
  ++*launches;
  return cudaGetLastError();
}

template <int ET, int EPB>
cudaError_t by_prec(int precision, bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (precision == 0) return go<ET, EPB, double>(want_r, want_k, a, s, launches);
  if (precision == 1) return go<ET, EPB, float>(want_r, want_k, a, s, launches);
  return cudaErrorNotSupported;
}

// Elements per CTA: 128-256 threads, or one warp where that leaves most SMs without a
// CTA -- the point phase is a chain of FP64 instructions, 64 clocks a warp on its
// sub-partition, so a small mesh wants its warps on as many as there are (1,189
// quad4 elements, 19 CTAs: 14.8 us).
template <int ET, int EPB, int SMALL>
cudaError_t by_size(int precision, bool want_r, bool want_k, const ElemArgs& a, cudaStream_t s, int* launches) {
  if (a.ne < int64_t(EPB) * num_sms()) return by_prec<ET, SMALL>(precision, want_r, want_k, a, s, launches);
  return by_prec<ET, EPB>(precision, want_r, want_k, a, s, launches);
}

}  // namespace

cudaError_t launch_poisson(int elem_type, int precision, bool want_r, bool want_k, const ElemArgs& a,
                           cudaStream_t s, int* launches) {
  switch (elem_type) {
    case 1: return by_size<1, 16, 4>(precision, want_r, want_k, a, s, launches);
    case 2: return by_size<2, 64, 8>(precision, want_r, want_k, a, s, launches);
    case 6: return by_prec<6, 32>(precision, want_r, want_k, a, s, launches);
    case 7: return by_prec<7, 16>(precision, want_r, want_k, a, s, launches);
    case 8: return by_prec<8, 1>(precision, want_r, want_k, a, s, launches);
    default: return cudaErrorNotSupported;
  }
}

}  // namespace fec
