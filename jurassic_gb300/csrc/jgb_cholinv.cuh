// Batched blocked Cholesky inverse (jgb_cholinv.cu).
#pragma once

#include <cuda_runtime.h>

namespace jgb {

struct InvertDesc {
  int n;
  long long off;  // of the n x n row-major matrix in the concatenation
};

// Inverts the matrices with full[i] != 0 in place; status[i] = 1 marks those
// that are not positive definite, which keep their values.  L and W: scratch
// of the concatenation's size.
void matrix_invert_blocked(int nret, int nmax, const InvertDesc* d, const int* full, int* status,
                           double* A, double* L, double* W, cudaStream_t s);

}  // namespace jgb
