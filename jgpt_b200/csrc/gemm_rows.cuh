// Products of few rows (decode steps, short prompts) with the weights as images in registers.  Host interface of gemm_rows.cu.
#pragma once

#include "common.cuh"

namespace jgpt {
namespace rows {

// The image of a weight matrix [K, N]: per 8 columns, per 16 k and per lane the 16 bytes that lane feeds to one m16n8k16
// product as B operand - two halves pairs of the high parts, two of the low parts - followed by one float per column.
// Element (k, n) is stored as fp16(w s) and fp16(w s - fp16(w s)), s the power of two that brings the column's largest element
// to [2^14, 2^15); the float is 1 / s.
inline int k_steps(int K) { return (K + 15) / 16; }
inline uint64_t image_bytes(int K, int N) {
    const uint64_t tiles = (uint64_t)(N + 7) / 8;
    return tiles * (uint64_t)k_steps(K) * 512u + tiles * 8u * sizeof(float);
}
// W [K, N] (row k times gamma[k] when given) -> image.  With W3 the columns alternate, W's and W3's (N = both).
int32_t pack(const float *W, const float *W3, const float *gamma, int K, int N, void *image, cudaStream_t st);

struct Batch {
    const void *image[3];
    float *C[3];
};
struct Fuse {
    const float *ss_in = nullptr;  // NORM: partial sums of squares of every row, parts_in per row
    float *ss_out = nullptr;       // RESIDUAL: the same of the result, one partial per 16 columns
    int parts_in = 0;
    float eps = 0.f;
    // bit 0: launched as a programmatic dependent (waits for the previous kernel itself); bit 1: lets the next one move in
    int pdl = 0;
#ifdef JGPT_B200_DECODE_TRACE
    Timeline timeline;
#endif
};
enum Kind { NORM, NORM_SWIGLU, RESIDUAL, NORM_PAGED };

// Whether the kernel is built for a product of this kind: every warp has a k slice, and its weights fit its registers.
bool shape_ok(Kind kind, int K);
inline int ss_parts(int D) { return (D + 15) / 16; }

// NORM: C_z[M, N] = rmsnorm(A) W_z (gamma is in the image), z < nb.  NORM_SWIGLU: C_0[M, N / 2] = h g sigmoid(g) over an
// alternating pair.  RESIDUAL: C_0 += A W_0, with the row sums of squares for the next norm.  NORM_PAGED: NORM for the Q, K, V products
// of a prefill at d_head 16 (N = heads * 16); products 1 and 2 go to the paged store as fp16, K with its RoPE, as the append kernel
// writes them.  Row r of A is rowsel[r] if given.
int32_t launch(Kind kind, Ctx *ctx, const float *A, const Batch &b, int nb, int M, int K, int N, const int *rowsel, const Fuse &fuse,
               const PagedAppendArgs &paged = PagedAppendArgs());

}  // namespace rows
}  // namespace jgpt
