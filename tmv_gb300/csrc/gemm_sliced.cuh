// gemm_sliced.cuh -- FP64 products on the tcgen05 tensor cores from exact
// 8-bit slices of the operands (gemm_sliced.cu).
#pragma once

#include "gemm.cuh"

namespace tmvg {

// One sliced operand: `rows` vectors of length K (the rows of A, or the
// columns of B), each scaled by its own power of two.
struct SlicedOperand {
    uint16_t* digits = nullptr;  // [kSlices][rows][Kp] bf16 integers, K contiguous
    int* exps = nullptr;         // per vector: every |entry| < 2^exps
    int* fill = nullptr;         // per group of vectors: fewest entries within 2^-4 of the largest
    int64_t rows = 0, Kp = 0;
    int group = 16;              // vectors per fill group
};

// Bytes of a sliced operand and its layout in a buffer of that size.
size_t sliced_bytes(int64_t rows, int64_t K);
SlicedOperand sliced_layout(void* buf, int64_t rows, int64_t K);

// Whether a product of this size is faster sliced than on the FP64 pipe.
bool sliced_wanted(Context* c, int64_t M, int64_t N, int64_t K);

// C (M x N, column-major) = alpha A B + beta C (beta 0 or 1).  `max_ctas` bounds
// the persistent grids (0: one CTA per SM).  TMVG_UNSUPPORTED (with nothing
// launched) where the workspace is not to be had, or a huge alpha meets a long K.
// The left operand may be a complex matrix in its real form (zleft): A.p is the
// complex data, A.si and A.sj its strides in complex elements, and the operand
// is the 2m x 2k real matrix of 2 x 2 blocks (re, -im; im, re).  With B and C
// the interleaved parts as they lie in memory (2k x n and 2m x n) the product
// is the complex one.
tmvg_status sliced_gemm(Context* c, int64_t M, int64_t N, int64_t K, double alpha, Mat<const double> A,
                        Mat<const double> B, double beta, double* C, int64_t ldc, int max_ctas = 0,
                        bool zleft = false);

// Stream-ordered scratch from the context's own pool (bounded: what a
// synchronisation finds unused above 1 GiB goes back to the device).
void* scratch_alloc(Context* c, size_t bytes, cudaStream_t s);
void scratch_free(void* p, cudaStream_t s);

}  // namespace tmvg
