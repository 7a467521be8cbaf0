// The encoder's training GEMM with what surrounds each product folded into it: how an operand's
// values are formed while it is packed, and what happens to a result before it is stored.  The layers
// are bound by memory; folding the im2col gather, the ReLU gradient, the biases, the residuals, the
// masks and the bias gradients took their passes over 67 to 201 MB out of a 2,048-pair step: 3.57 ->
// 2.77 ms with the attention kernels' wider reads (B200; sums keep the separate passes' order except
// the bias gradients').  Packing a matrix once for its product along the rows and the one along the
// columns, whose operands are read MN-major: 2.53 -> 2.06 ms.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"

namespace stb {

// Values of a row-major fp32 operand, formed as they are packed to bf16.
struct PackSrc {
    enum Kind { kPlain, kConv, kRelu };
    const float* x = nullptr;
    int ld = 0;
    int kind = kPlain;
    // kConv: x holds rows of 128 columns; value (r, c) of the 384-column im2col matrix is row r - 1, r or
    // r + 1 (c / 128) of x inside the 32-row sequence's first lens[r / 32] rows, 0 outside.
    const int32_t* lens = nullptr;
    // kRelu: x where y > 0 (y as x), else 0.
    const float* y = nullptr;
    // When set: the column sums of the matrix are added to it (pack_matrix).
    float* colsum = nullptr;
};

// What becomes of the product before it is stored.  Rows are positions of 32-row sequences; kinds
// with lens give 0 past a sequence's end.
struct GemmEpi {
    enum Kind { kNone, kBias, kResidual, kConv, kMaskAdd };
    int kind = kNone;
    const float* bias = nullptr;   // kBias, kResidual, kConv: per column
    const float* res = nullptr;    // kResidual, kConv: added, laid out as C
    float* out = nullptr;          // kResidual: res + C + bias here and C untouched;
                                   // kConv: C + bias to C, res + relu(C + bias) here
    const int32_t* lens = nullptr; // kResidual, kConv, kMaskAdd (C += product, 0 past the end)
};

// A matrix packed once for both of its products: as rows (op(A) = A) it is a K-major operand, and the
// same blocks, read along their rows, are the MN-major operand of A^T (cols a multiple of 128).
struct Packed {
    const uint8_t* op = nullptr;
    int rows = 0, cols = 0;
};
constexpr size_t packed_bytes(int64_t rows, int cols) { return size_t((rows + 127) / 128 * 128) * size_t(cols) * 2; }
Packed pack_matrix(const PackSrc& s, int rows, int cols, uint8_t* op, cudaStream_t st);  // op: packed_bytes

// Weights as B operands, all of a step's in one launch: rows x cols (multiples of 128 and 64) from x[r][c], or
// from x[c][r] when trans.  Each takes packed_bytes(rows, cols), one after another from op.
struct WeightSrc {
    const float* x = nullptr;
    int ld = 0, rows = 0, cols = 0;
    bool trans = false;
};
constexpr int kMaxWeights = 10;
void pack_weights(const WeightSrc* w, int n, uint8_t* op, Packed* out, cudaStream_t st);

// C (=, +=) A B^T, A [M x K] and B [N x K] packed.
void gemm_packed(const Packed& A, const Packed& B, float* C, int ldc, bool accumulate, const GemmEpi& epi,
                 cudaStream_t st, int sms);
// C += A^T B, both packed with the same rows.
void gemm_packed_tn(const Packed& A, const Packed& B, float* C, int ldc, cudaStream_t st, int sms);

}  // namespace stb
