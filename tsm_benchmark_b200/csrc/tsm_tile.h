// tsm_tile.h -- host side of the any-layout tensor-core kernels (tsm_tile.cuh).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "../../include/tsm.h"
#include "tsm_plain.cuh"

namespace tsm {

struct Variant;

// Launches tile variant v (its capacities hold m x k, or k x m) on operands
// with element strides (a_row, a_col) and (b_row, b_col).  p carries A, B, C,
// the sizes, ldc, accumulate and the workspace; lda/ldb are set here.  At most
// max_ctas CTAs when max_ctas > 0.
template <typename T>
tsm_status launch_tile(const Variant* v, int sms, cudaStream_t stream, PlainArgs<T> p, int64_t a_row, int64_t a_col,
                       int64_t b_row, int64_t b_col, int64_t max_ctas);

// Whether row-major operands would be loaded as one (neighbouring column blocks of
// one matrix), and whether in phases rather than by bulk copies or whole boxes.
bool tile_joint(const void* A, int m, int64_t lda, const void* B, int k, int64_t ldb, size_t esize, bool* phases);

// launch_tile for the strided entry point: picks the variant, prepares it on the
// current device and checks the workspace.
tsm_status run_tile_f64(cudaStream_t stream, int64_t n, int m, int k, const double* A, int64_t a_row, int64_t a_col,
                        const double* B, int64_t b_row, int64_t b_col, double* C, int64_t ldc, int accumulate,
                        void* ws, size_t ws_bytes);

}  // namespace tsm
