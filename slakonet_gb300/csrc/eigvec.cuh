// The eigenvector stage (eigvec.cu), shared by the entry points that solve with vectors.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace skn_vec {

constexpr int VNT = 128;                 // threads of a CTA of the inverse iteration

// CTAs of the inverse iteration: as many as fit on the GPU at once, but no more than the problems and no more than
// keep its scratch within 2 GB.  Each problem is solved by one CTA, so the results do not depend on the grid.
int grid(int n_prob, int max_n);
// Scratch bytes of one CTA of the inverse iteration.
int64_t cta_bytes(int max_n);
// Launches the stage: 2 kernels.  `counter` is one int32 that is zero at the launch; `real` (may be null) marks
// problems whose reflectors and L are real; `most` bounds n of the problems in `order`.
cudaError_t launch(int n_prob, const int32_t* n, const int64_t* hs_off, const int64_t* eig_off, const int32_t* order,
                   const int32_t* real, const double* H, const double* S, const double* eig, const double* tri,
                   const int32_t* status, double* vec, double* scratch, int n_cta, int32_t* counter, int most,
                   cudaStream_t stream);

}  // namespace skn_vec
