// Large-M fp32 projections on the 5th-generation tensor cores (tcgen05.mma, accumulator in tensor memory).
// Host-side interface of gemm_umma.cu; operands are pre-tiled "images" (see the layout note there).
#pragma once

#include "common.cuh"

namespace jgpt {
namespace umma {

constexpr int BM = 128;  // rows of C per CTA (one TMEM lane per row)
constexpr int BK = 16;   // k extent of one pipeline stage (two K=8 tensor-core steps)

// Columns of C per CTA (one fp32 TMEM column per column): the widest tile that leaves no padded columns.
inline int tile_cols(int N) { return N % 256 == 0 ? 256 : (N % 192 == 0 ? 192 : 256); }

// Floats of the tiled hi/lo image of a [rows, K] operand whose rows are grouped in tiles of `tile_rows`.
inline uint64_t image_floats(int rows, int K, int tile_rows) {
    const uint64_t tiles = (uint64_t)(rows + tile_rows - 1) / tile_rows;
    return tiles * (uint64_t)tile_rows * (uint64_t)K * 2u;
}
inline uint64_t activation_image_floats(int M, int K) { return image_floats(M, K, BM); }
inline uint64_t weight_image_floats(int K, int N) { return image_floats(N, K, tile_cols(N)); }

// A[M, K] row major (row r taken from rowsel[r] when rowsel != nullptr) -> activation image.
int32_t pack_activations(const float *A, const int *rowsel, int M, int K, float *image, cudaStream_t st);
// RMSNorm of x[M, D] with gamma, written straight into an activation image (same arithmetic as the row-major
// RMSNorm kernel of the forward step).
int32_t rmsnorm_pack(const float *x, const float *gamma, int M, int D, float eps, float *image, cudaStream_t st);
// W[K, N] row major -> image of W^T (rows = output columns) in tiles of tile_cols(N) rows.
int32_t pack_weight(const float *W, int K, int N, float *image, cudaStream_t st);
// W1, W3 [K, F] -> one image of 2F rows in 256-row tiles: tile t = columns [128 t, 128 t + 128) of W1
// followed by the same columns of W3 (needs F % 128 == 0).
int32_t pack_weight_pair(const float *W1, const float *W3, int K, int F, float *image, cudaStream_t st);

struct Batch {
    const float *Wimg[3];
    float *C[3];
    const float *R[3];  // optional residual, may alias C
    const float *a_un = nullptr;  // fp16 images: one factor per row of A that undoes its power of two (nullptr: none)
    const float *r_up = nullptr, *c_up = nullptr;  // the SwiGLU form on fp16 images: the powers of two of the result's rows and columns
};
// C_z[M, N] = A . W_z (+ R_z) for z < nb; needs K % 16 == 0 and N % 4 == 0.
int32_t launch(const float *Aimg, const Batch &b, int nb, int M, int K, int N, int *d_status, cudaStream_t st);
// C[M, N] = A[M, K] . B[K, N], all row major: two launches, the operands' images in scratch.
uint64_t matmul_scratch_floats(int M, int K, int N);
int32_t matmul(const float *A, const float *B, float *C, int M, int K, int N, float *scratch, int *d_status, cudaStream_t st);
// act = (A . W1) * silu(A . W3), written as the activation image [M, F] of the next product.
int32_t launch_swiglu(const float *Aimg, const float *Wpair_img, int M, int K, int F, float *act_image, int *d_status,
                      cudaStream_t st);

// The Q, K, V products of a prefill (b.Wimg[0..2]; d_head 16, N = heads * 16): Q goes to b.C[0] row major, K gets its
// RoPE and both K and V are written as fp16 straight into the paged store - the arithmetic and the stores of the
// append kernel, without the fp32 round trip through memory.
int32_t launch_qkv_paged(const float *Aimg, const Batch &b, int M, int K, int N, const PagedAppendArgs &pa, int *d_status,
                         cudaStream_t st);

// The same products on fp16 images (kind::f16): a k tile holds 32 k in the bytes of 16 TF32 ones, so an image has half the bytes
// and a product half the tensor time.  See gemm_umma.cu for the scaling.
constexpr int HBK = 32;
inline bool half_ok(int D, int F) { return D % HBK == 0 && F % 128 == 0; }
inline uint64_t half_activation_floats(int M, int K) { return image_floats(M, K, BM) / 2; }
// W [K, N], row k times gamma[k] or divided by k_scale[k] if given -> image, then one float per image row that undoes that row's (column of W's) power
// of two, then work space of the same size.
inline uint64_t half_weight_floats(int K, int N) {
    const uint64_t rows = (uint64_t)((N + tile_cols(N) - 1) / tile_cols(N)) * (uint64_t)tile_cols(N);
    return rows * (uint64_t)K + 2 * rows;
}
inline uint64_t half_pair_floats(int K, int F) { return (uint64_t)2 * F * (uint64_t)K + 4 * (uint64_t)F; }
// Where the attention leaves its output for the next product: the image and its columns' powers of two (none: a TF32 image; no image:
// row major).
struct ImageOut {
    float *image = nullptr;
    const float *scale = nullptr;
};
int32_t pack_weight_half(const float *W, const float *gamma, const float *k_scale, int K, int N, float *image, cudaStream_t st);
int32_t pack_weight_pair_half(const float *W1, const float *W3, const float *gamma, int K, int F, float *image, cudaStream_t st);
// scale[n] = the power of two that keeps column n of rmsnorm(x) W (gamma applied) below 2^15.
int32_t column_scales(const float *W, const float *gamma, int K, int N, float *scale, cudaStream_t st);
// The same for h g sigmoid(g) of the pair, times a power of two of the row (see gemm_umma.cu): F column scales, then the K weights of the
// elements that the row's is taken with, then work space.
inline uint64_t pair_scale_floats(int K, int F) { return (uint64_t)F + 3 * (uint64_t)K; }
int32_t pair_scales(const float *W1, const float *W3, const float *gamma, int K, int F, float *scale, cudaStream_t st);
// RMSNorm into an fp16 image, its weights being in the next product's; a_un[M] receives the rows' factors.  With the weights r of a pair's
// elements a_un[M .. 2 M) and [2 M .. 3 M) receive the power of two of the row's SwiGLU result and its inverse.
int32_t rmsnorm_pack_half(const float *x, const float *r, int M, int D, float eps, float *image, float *a_un, cudaStream_t st, int pdl = 0);
// pdl, of the fp16 forms: bit 0 = the launch may start early and waits itself; bit 1 = it lets the next launch in.
int32_t launch_half(const float *Aimg, const Batch &b, int nb, int M, int K, int N, int *d_status, cudaStream_t st, int pdl = 0);
// a_un: the rows' factors as rmsnorm_pack_half leaves them; c_up[F]: the powers of two of the result's columns in its image.
int32_t launch_swiglu_half(const float *Aimg, const float *Wpair_img, const float *a_un, const float *c_up, int M, int K, int F, float *act_image,
                           int *d_status, cudaStream_t st, int pdl = 0);
int32_t launch_qkv_paged_half(const float *Aimg, const Batch &b, int M, int K, int N, const PagedAppendArgs &pa, int *d_status, cudaStream_t st, int pdl = 0);

inline bool shape_ok(int K, int N) { return K >= BK && K % BK == 0 && N % 4 == 0; }
inline bool swiglu_shape_ok(int K, int F) { return K >= BK && K % BK == 0 && F % 128 == 0; }

}  // namespace umma
}  // namespace jgpt
