// fec_solver.h -- device linear algebra on the assembled CSC stiffness.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace fec {

// Symmetric matrix in CSC over the unknowns (0-based), values on the device.
struct CscSym {
  int64_t n, nnz;
  const int64_t* colptr;  // n + 1
  const int32_t* rowval;  // nnz
  const double* val;      // nnz
};

// Page-locked memory and events a solve reads its stopping test through; kept by
// the caller between solves (one solve at a time).
struct PcgHost {
  static constexpr size_t SLOT = 64;
  void* pinned = nullptr;
  cudaEvent_t done[2] = {nullptr, nullptr};
  cudaError_t ensure();
  void release();
};

size_t pcg_scratch_doubles(int64_t n);
// Conjugate gradients for A x = b from the x passed in (Jacobi-preconditioned if
// asked); stops when ||b - A x|| <= rtol ||b|| (tested every check_every
// iterations) or after max_iter.  wait_budget: clocks a barrier of the one-launch solve
// waits before the solve gives up with cudaErrorLaunchTimeout (0: the default, ~1 s).
// Synchronises the stream.
cudaError_t pcg(const CscSym& A, const double* b, double* x, double* scratch, int max_iter, double rtol,
                int check_every, bool jacobi, long long wait_budget, PcgHost& host, int* iterations,
                double* rel_residual, cudaStream_t s);

}  // namespace fec
