// fp32 projections for prefill-sized M on the Blackwell tensor cores: tcgen05.mma (kind::tf32) issued by one
// thread per CTA, operands staged in shared memory by bulk async copies (TMA engine, non-multicast), the
// 128 x BN fp32 accumulator double-buffered in tensor memory and read back with tcgen05.ld by epilogue warps
// that overlap the next tile's MMAs.
//
// Accuracy: every fp32 operand is split into a TF32 high part and a TF32 low part and
// C += Ah.Wh + Al.Wh + Ah.Wl with fp32 accumulation, the same "3xTF32" scheme as the mma.sync kernel the
// small-M path uses (the reference runs these GEMMs through cuBLAS under plain TF32 math,
// src/main/cpp/jgpt_cuda_jni_init_matmul.inl:67, 794, 892).  The tensor core truncates when it adds into the
// fp32 accumulator; with all three products in one accumulator (3K / 8 additions) the result sits about
// 8e-9 * K of the largest element away from a float64 product (plain TF32: ~1e-3).
//
// Operand images.  Both operands are stored K-major in the tensor core's canonical no-swizzle layout so that
// one stage of one operand is ONE contiguous bulk copy: for a tile of TR rows and 16 k,
//     byte offset(r, k) = (r / 8) * 512 + (k / 4) * 128 + (r % 8) * 16 + (k % 4) * 4
// i.e. 8-row x 16-byte core matrices, 128 bytes each; the four core matrices of a row group along k are
// adjacent (leading-dimension byte offset 128), row groups follow each other (stride byte offset 512).
// A tile holds the high-part image followed by the low-part image; tiles are ordered [row tile][k tile].
// Weights are static, so their images are built once (transposed: image rows are output columns).
// Activation images are written by whatever produces the activation: the RMSNorm packer, the SwiGLU epilogue
// of the W1/W3 product, or the plain packer (attention output).
//
// fp16 images (kind::f16, the forward step of models with d_head 16).  An operand as an fp16 high and an fp16 low part, 11 + 11 bits
// like the TF32 parts: two bytes each instead of four, and the tensor cores take 16 k per step instead of 8 at the same rate, so a
// product costs half the time and half the operand traffic.  A 16-byte chunk holds eight k, a k tile 32, everything else lies
// where the TF32 layout has it.  What fp16's exponent lacks is made up by powers of two, which change no bit:
//   weights: per column of W, from its largest element; undone in the epilogue (the factors stand behind the image).  The norm weights
//   gamma are in the rows of the W that follows the norm, so their spread is not the normalised row's;
//   RMSNorm rows: per row, from the row's largest element; undone in the epilogue;
//   attention results, whose rows no single CTA sees: per column, from what the column can reach at all.  A normalised row is at most
//   sqrt(D) long, so |v_n| <= sqrt(D) |gamma o Wv_n|, and an attention output is a weighted mean of such values.  The next weight's rows
//   are divided by the same powers.  (However far below that bound they lie, a value that comes from an fp16 cache has 2^-12 of itself as
//   error anyway.)
//   SwiGLU results, likewise: per column and per row.  For any weights r > 0 of the elements, |x . w_n| <= |x o r| |w_n / r|, so
//   |h g sigmoid(g)| <= |x o r|^2 . |gamma o W1_n / r| |gamma o W3_n / r|: the first factor is the row's, taken by the norm in front,
//   the others the column's.  r_k is the size of row k of both weights, which makes all terms of a sum alike: without it a row
//   whose large elements meet small weights lies as far below the bound as the spread of its elements, squared.
// An element down to 2^-16 of the largest its scale allows for is within 2^-23 of itself, like a TF32 pair at any size; below that an
// absolute error of at most 2^-39 of that largest remains.  So the 22 bits are those of the largest in the row (column), and a row whose
// elements spread further along k, with weights the other way round, loses bits that TF32 pairs keep.  Typical results of a SwiGLU lie
// about 2^10 below their bound at any such spread.  Error of a block's feed-forward part against float64 (2-norm, 384 / 768, 2000 rows): TF32 4.8e-6, fp16
// 2.5e-6, of its Wo product 9.5e-7 and 5.2e-7 (half as many steps of accumulation).
// The attention output of a prefill is such a mean because every key it sees was produced by the same call's Q,K,V product.
// Measured for 32 x 1024 tokens, 24 heads of 16 (ncu, us per launch, TF32 -> fp16 images): Q,K,V 139 -> 91, W1/W3 + SwiGLU 164 -> 116,
// Wo / W2 87 -> 73, RMSNorm 26.8 -> 21.5; the prefill of 12 layers 9.9 -> 7.8 ms.
//
// Roles in the 320-thread CTA: warp 0 lane 0 issues the bulk copies, warp 1 allocates tensor memory and its
// lane 0 issues the MMAs, warps 2-9 are the epilogue (TMEM lane quarter = warp % 4, two warps per quarter).  Stages are handed over
// with mbarriers: full[s] by the copies' complete_tx, empty[s] and "accumulator buffer ready" by
// tcgen05.commit, "accumulator buffer drained" by the epilogue warps.  Every wait is bounded; on expiry the status word gets DEV_STATUS_WAIT_TIMEOUT and the CTA
// winds down through the common exit (tensor memory is always released).
#include "gemm_umma.cuh"

#include <type_traits>

#include "ptx.cuh"
#include "tcgen05.cuh"

namespace jgpt {
namespace umma {

constexpr int A_TILE_FLOATS = BM * BK * 2;
constexpr uint32_t A_TILE_BYTES = A_TILE_FLOATS * 4;
constexpr uint32_t TMEM_COLS = 512;  // two accumulator buffers of 256 columns
constexpr uint32_t LBO = 128, SBO = 512;
constexpr int EPI_WARPS = 8;  // two per TMEM lane quarter, each draining half of the tile's columns
constexpr int THREADS = 64 + 32 * EPI_WARPS;

// ------------------------------------------------------------------------------------------------
// Packing
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void split_hi_lo(float x, float &hi, float &lo) {
    uint32_t h, l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
    hi = __uint_as_float(h);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(x - hi));
    lo = __uint_as_float(l);
}
__device__ __forceinline__ void split4(const float4 v, float4 &hi, float4 &lo) {
    split_hi_lo(v.x, hi.x, lo.x), split_hi_lo(v.y, hi.y, lo.y), split_hi_lo(v.z, hi.z, lo.z), split_hi_lo(v.w, hi.w, lo.w);
}
// Float offset of the 16-byte chunk (row rr of the tile, k chunk k4) inside one half (hi or lo) of a tile.
__device__ __forceinline__ int chunk_offset(int rr, int k4) { return (rr >> 3) * 128 + k4 * 32 + (rr & 7) * 4; }

// One CTA per (k tile, row tile).  TRANSPOSED: the source is [K, rows] (a weight matrix), element (r, k) is
// src[k * rows + r]; otherwise the source is [rows, K].  Rows past `rows` are zero.
template <int TR, bool TRANSPOSED>
__global__ void __launch_bounds__(256) pack_kernel(const float *__restrict__ src, const int *__restrict__ rowsel, int rows, int K,
                                                   float *__restrict__ image) {
    const int kt = blockIdx.x, rt = blockIdx.y, nkt = K / BK;
    float *tile = image + ((size_t)rt * nkt + kt) * (size_t)(TR * BK * 2);
    for (int e = threadIdx.x; e < TR * (BK / 4); e += 256) {
        const int rr = e % TR, k4 = e / TR;  // consecutive threads: consecutive rows = consecutive 16-byte chunks
        const int r = rt * TR + rr, k = kt * BK + k4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) {
            if (TRANSPOSED) {
                v.x = src[(size_t)(k + 0) * rows + r], v.y = src[(size_t)(k + 1) * rows + r];
                v.z = src[(size_t)(k + 2) * rows + r], v.w = src[(size_t)(k + 3) * rows + r];
            } else {
                const int sr = rowsel ? rowsel[r] : r;
                v = *reinterpret_cast<const float4 *>(src + (size_t)sr * K + k);
            }
        }
        float4 hi, lo;
        split4(v, hi, lo);
        const int off = chunk_offset(rr, k4);
        *reinterpret_cast<float4 *>(tile + off) = hi;
        *reinterpret_cast<float4 *>(tile + TR * BK + off) = lo;
    }
}

// Both operands of a product in one launch: the row tiles of A [M, K], then the column tiles of B [K, N], TR columns each.
template <int TR>
__global__ void __launch_bounds__(256) pack_both_kernel(const float *__restrict__ A, int M, const float *__restrict__ B, int N, int K,
                                                        float *__restrict__ a_image, float *__restrict__ b_image, int a_tiles) {
    const int nkt = K / BK, t = blockIdx.x / nkt, kt = blockIdx.x - t * nkt;
    const bool second = t >= a_tiles;
    const int rt = second ? t - a_tiles : t, rows = second ? TR : BM, lg = second ? (TR == 192 ? 0 : TR == 64 ? 6 : TR == 128 ? 7 : 8) : 7;
    float *tile = (second ? b_image : a_image) + ((size_t)rt * nkt + kt) * (size_t)(rows * BK * 2);
    griddep_launch_dependents();
    for (int e = threadIdx.x; e < rows * (BK / 4); e += 256) {
        const int k4 = lg ? e >> lg : e / TR, rr = e - k4 * rows, r = rt * rows + rr, k = kt * BK + k4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (second) {
            if (r < N) v = make_float4(B[(size_t)k * N + r], B[(size_t)(k + 1) * N + r], B[(size_t)(k + 2) * N + r], B[(size_t)(k + 3) * N + r]);
        } else if (r < M) {
            v = *reinterpret_cast<const float4 *>(A + (size_t)r * K + k);
        }
        float4 hi, lo;
        split4(v, hi, lo);
        const int off = chunk_offset(rr, k4);
        *reinterpret_cast<float4 *>(tile + off) = hi;
        *reinterpret_cast<float4 *>(tile + rows * BK + off) = lo;
    }
}

// 256-row tiles of the W1 / W3 pair: rows 0..127 = columns [128 t, +128) of W1, rows 128..255 = the same of W3.
__global__ void __launch_bounds__(256) pack_pair_kernel(const float *__restrict__ W1, const float *__restrict__ W3, int K, int F,
                                                        float *__restrict__ image) {
    constexpr int TR = 256;
    const int kt = blockIdx.x, rt = blockIdx.y, nkt = K / BK;
    float *tile = image + ((size_t)rt * nkt + kt) * (size_t)(TR * BK * 2);
    for (int e = threadIdx.x; e < TR * (BK / 4); e += 256) {
        const int rr = e % TR, k4 = e / TR;
        const float *__restrict__ src = rr < 128 ? W1 : W3;
        const int col = rt * 128 + (rr & 127), k = kt * BK + k4 * 4;
        float4 v;
        v.x = src[(size_t)(k + 0) * F + col], v.y = src[(size_t)(k + 1) * F + col];
        v.z = src[(size_t)(k + 2) * F + col], v.w = src[(size_t)(k + 3) * F + col];
        float4 hi, lo;
        split4(v, hi, lo);
        const int off = chunk_offset(rr, k4);
        *reinterpret_cast<float4 *>(tile + off) = hi;
        *reinterpret_cast<float4 *>(tile + TR * BK + off) = lo;
    }
}

// RMSNorm of 8 rows (one row group of the image) per CTA with exactly the reduction order of the row-major
// RMSNorm kernel and its 128 threads per row (strided partial sums, warp shuffle, four partials added in order;
// rms_norm_fwd_block_kernel, src/main/cpp/jgpt_cuda_extra_kernels_launches.inl:694-713), so both produce the
// same bits.  The normalised rows go through shared memory so that the image is written in contiguous
// 512-byte runs.
//
// One warp per row: lane l plays the row-major kernel's threads l, l + 32, l + 64, l + 96 (one partial sum
// each, elements taken in the same ascending order), the four butterflies run over the same lanes as that
// kernel's four warps, and the four results are added left to right.
__global__ void __launch_bounds__(256) rmsnorm_pack_kernel(const float *__restrict__ x, const float *__restrict__ gamma, int M, int D,
                                                           float eps, float *__restrict__ image) {
    extern __shared__ __align__(16) float rp_rows[];  // [8][D + 4]
    const int tid = threadIdx.x, rr = tid >> 5, lane = tid & 31;
    const int row = blockIdx.x * 8 + rr;
    const int stride = D + 4;
    const float *xr = x + (size_t)(row < M ? row : 0) * D;
    float ss[4] = {0.f, 0.f, 0.f, 0.f};
    if (row < M) {
        for (int j0 = 0; j0 < D; j0 += 128) {
#pragma unroll
            for (int w = 0; w < 4; w++) {
                const int j = j0 + 32 * w + lane;
                if (j < D) ss[w] += xr[j] * xr[j];
            }
        }
    }
#pragma unroll
    for (int w = 0; w < 4; w++)
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) ss[w] += __shfl_xor_sync(0xffffffffu, ss[w], off);
    const float tot = ss[0] + ss[1] + ss[2] + ss[3];
    const float rms = sqrtf(tot / (float)D + eps);
    const float inv = (rms > 0.f && isfinite(rms)) ? (1.f / rms) : 0.f;
    for (int j = lane; j < D; j += 32) rp_rows[rr * stride + j] = row < M ? xr[j] * inv * gamma[j] : 0.f;
    __syncthreads();
    const int nkt = D / BK, mt = (blockIdx.x * 8) / BM, rg = ((blockIdx.x * 8) % BM) >> 3;
    float *base = image + (size_t)mt * nkt * A_TILE_FLOATS + rg * 128;
    for (int e = tid; e < nkt * 32; e += 256) {
        const int kt = e >> 5, k4 = (e >> 3) & 3, r8 = e & 7;
        const float4 v = *reinterpret_cast<const float4 *>(&rp_rows[r8 * stride + kt * BK + k4 * 4]);
        float4 hi, lo;
        split4(v, hi, lo);
        float *dst = base + (size_t)kt * A_TILE_FLOATS + k4 * 32 + r8 * 4;
        *reinterpret_cast<float4 *>(dst) = hi;
        *reinterpret_cast<float4 *>(dst + BM * BK) = lo;
    }
}

// ---- fp16 images ----
// Byte offset of the 16-byte chunk (row rr, eight k) inside one half (high or low) of a tile.
__device__ __forceinline__ int half_chunk(int rr, int k8) { return (rr >> 3) * 512 + k8 * 128 + (rr & 7) * 16; }
__device__ __forceinline__ void split8(const float (&v)[8], uint4 &hi, uint4 &lo) {
    split_pair(v[0], v[1], hi.x, lo.x), split_pair(v[2], v[3], hi.y, lo.y);
    split_pair(v[4], v[5], hi.z, lo.z), split_pair(v[6], v[7], hi.w, lo.w);
}
// The exponent e <= limit that brings values up to mx into [2^14, 2^15) as mx 2^e; 0 for a column that is all zeros or not finite (its
// results are zeros, or not finite, at any scale).
__device__ __forceinline__ int half_exponent(double mx, int limit) {
    if (!(mx > 0.) || isinf(mx)) return 0;
    int e;
    frexp(mx, &e);  // mx in [2^(e - 1), 2^e)
    return max(-126, min(limit, 15 - e));  // 2^e and 2^-e are normal numbers
}
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }
// One thread per column: up[n] brings the column's largest element (row k times the norm weight gamma[k] in front of it, or divided by
// k_scale[k]) to [2^14, 2^15), un[n] undoes it.
// Image row r is column r of W, or, for a pair, column (r / 256) * 128 + r % 128 of W1 (first 128 rows of a 256-row tile) or W3.
// In fp64: a weight over a power of two may lie outside fp32 where the product of the two does not.
__device__ __forceinline__ const float *half_source(const float *W, const float *W3, int r, int &col) {
    if (!W3) return col = r, W;
    col = (r >> 8) * 128 + (r & 127);
    return r & 128 ? W3 : W;
}
__device__ __forceinline__ double half_element(float w, const float *gamma, const float *k_scale, int k) {
    return gamma ? (double)w * gamma[k] : k_scale ? (double)w / k_scale[k] : (double)w;
}
__global__ void __launch_bounds__(256) half_scale_kernel(const float *W, const float *W3, const float *gamma, const float *k_scale, int K, int N, int rows,
                                                         float *un, float *up) {
    const int r = blockIdx.x * 256 + threadIdx.x;
    if (r >= rows) return;
    int col;
    const float *src = half_source(W, W3, r, col);
    double mx = 0.;
    if (col < N)
        for (int k = 0; k < K; k++) mx = fmax(mx, fabs(half_element(src[(size_t)k * N + col], gamma, k_scale, k)));
    const int e = half_exponent(mx, 126);
    up[r] = pow2(e), un[r] = pow2(-e);
}
template <int TR>
__global__ void __launch_bounds__(256) half_pack_kernel(const float *W, const float *W3, const float *gamma, const float *k_scale, const float *up, int K,
                                                        int N, uint8_t *image) {
    const int kt = blockIdx.x, rt = blockIdx.y, nkt = K / HBK;
    uint8_t *tile = image + ((size_t)rt * nkt + kt) * (size_t)(TR * HBK * 4);
    for (int e = threadIdx.x; e < TR * 4; e += 256) {
        const int rr = e % TR, k8 = e / TR, r = rt * TR + rr;
        int col;
        const float *src = half_source(W, W3, r, col);
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int k = kt * HBK + k8 * 8 + q;
            v[q] = col < N ? (float)(half_element(src[(size_t)k * N + col], gamma, k_scale, k) * up[r]) : 0.f;
        }
        uint4 hi, lo;
        split8(v, hi, lo);
        *reinterpret_cast<uint4 *>(tile + half_chunk(rr, k8)) = hi;
        *reinterpret_cast<uint4 *>(tile + TR * HBK * 2 + half_chunk(rr, k8)) = lo;
    }
}
// In fp64, where no square of an fp32 weight leaves the range: a column of 1e-24 has a reach that is not 0, one of 1e20 a finite one.
// The limit leaves room for the factors that undo the powers.
__global__ void __launch_bounds__(256) column_scale_kernel(const float *W, const float *gamma, int K, int N, float *scale) {
    const int n = blockIdx.x * 256 + threadIdx.x;
    if (n >= N) return;
    double a = 0.;
    for (int k = 0; k < K; k++) {
        const double x = (double)gamma[k] * W[(size_t)k * N + n];
        a += x * x;
    }
    scale[n] = pow2(half_exponent(sqrt((double)K * a), 113));
}
// The weights r of the elements in front of the pair W1, W3: the 2-norm of row k of both over the largest of all, at least 2^-60 (any
// positive r makes a bound).
constexpr double kLeastWeight = 0x1p-60;
__global__ void __launch_bounds__(256) pair_row_size_kernel(const float *W1, const float *W3, const float *gamma, int K, int N, double *size) {
    __shared__ double red[8];
    const int k = blockIdx.x;
    double a = 0.;
    for (int n = threadIdx.x; n < N; n += 256) {
        const double g = gamma[k], x = g * W1[(size_t)k * N + n], y = g * W3[(size_t)k * N + n];
        a += x * x + y * y;
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) a += red[w];
        size[k] = sqrt(a);
    }
}
__global__ void __launch_bounds__(256) pair_weight_kernel(const double *size, int K, float *r) {
    double mx = 0.;  // every block finds the largest by itself
    for (int k = 0; k < K; k++) mx = fmax(mx, size[k]);
    const int k = blockIdx.x * 256 + threadIdx.x;
    if (k < K) r[k] = (mx > 0. && isfinite(mx)) ? (float)fmax(size[k] / mx, kLeastWeight) : 1.f;
}
__global__ void __launch_bounds__(256) pair_scale_kernel(const float *W1, const float *W3, const float *gamma, const float *r, int K, int N, float *scale) {
    const int n = blockIdx.x * 256 + threadIdx.x;
    if (n >= N) return;
    double a = 0., b = 0.;
    for (int k = 0; k < K; k++) {
        const double g = (double)gamma[k] / r[k], x = g * W1[(size_t)k * N + n], y = g * W3[(size_t)k * N + n];
        a += x * x, b += y * y;
    }
    scale[n] = pow2(half_exponent(sqrt(a) * sqrt(b), 113));
}
// RMSNorm, without its weights, of 8 rows per CTA like rmsnorm_pack_kernel, a warp per row; up to kKept elements per lane stay in registers
// between the sum of squares and the product.  x is a plain pointer: the launch in front still writes it while this one is resident, and
// const __restrict__ would promise that nobody does.
constexpr int kKept = 16;
__global__ void __launch_bounds__(256) rmsnorm_pack_half_kernel(const float *x, const float *__restrict__ r, int M, int D, float eps,
                                                                uint8_t *__restrict__ image, float *__restrict__ a_un, int pdl) {
    extern __shared__ __align__(16) float rp_rows[];  // [8][D + 4]
    if (pdl & 2) griddep_launch_dependents();
    if (pdl & 1) griddep_wait();
    const int tid = threadIdx.x, rr = tid >> 5, lane = tid & 31;
    const int row = blockIdx.x * 8 + rr;
    const int stride = D + 4;
    const float *xr = x + (size_t)(row < M ? row : 0) * D;
    float *mine = rp_rows + rr * stride;
    const bool kept = D <= 32 * kKept;
    float v[kKept], ss[4] = {0.f, 0.f, 0.f, 0.f};
    if (kept) {
#pragma unroll
        for (int i = 0; i < kKept; i++) v[i] = (32 * i + lane < D && row < M) ? xr[32 * i + lane] : 0.f;
#pragma unroll
        for (int i = 0; i < kKept; i++) ss[i & 3] += v[i] * v[i];
    } else if (row < M) {
        for (int j0 = 0; j0 < D; j0 += 128) {
#pragma unroll
            for (int w = 0; w < 4; w++) {
                const int j = j0 + 32 * w + lane;
                if (j < D) ss[w] += xr[j] * xr[j];
            }
        }
    }
#pragma unroll
    for (int w = 0; w < 4; w++)
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) ss[w] += __shfl_xor_sync(0xffffffffu, ss[w], off);
    const float tot = ss[0] + ss[1] + ss[2] + ss[3];
    const float rms = sqrtf(tot / (float)D + eps);
    const float inv = (rms > 0.f && isfinite(rms)) ? (1.f / rms) : 0.f;
    float mx = 0.f, size = 0.f;  // size: |x o r|^2 of the normalised row
    if (kept) {
#pragma unroll
        for (int i = 0; i < kKept; i++)
            if (32 * i + lane < D) {
                v[i] *= inv;
                mx = fmaxf(mx, fabsf(v[i]));
                if (r) {
                    const float t = v[i] * r[32 * i + lane];
                    size = fmaf(t, t, size);
                }
            }
    } else {
        for (int j = lane; j < D; j += 32) {
            const float y = row < M ? xr[j] * inv : 0.f;
            mine[j] = y;
            mx = fmaxf(mx, fabsf(y));
            if (r) size = fmaf(y * r[j], y * r[j], size);
        }
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off)), size += __shfl_xor_sync(0xffffffffu, size, off);
    if (r && lane == 0 && row < M) {
        // the result's power of two: |x o r|^2 up to [1/2, 1); a sum that underflows is below 2^-100 in any case
        const int e = isfinite(size) ? -ilogbf(fmaxf(size, 0x1p-100f)) - 1 : 0;
        a_un[M + row] = pow2(e), a_un[2 * (size_t)M + row] = pow2(-e);
    }
    float up, un;
    pow2_scale(mx, up, un);
    if (lane == 0 && row < M) a_un[row] = un;
    if (kept) {
#pragma unroll
        for (int i = 0; i < kKept; i++)
            if (32 * i + lane < D) mine[32 * i + lane] = v[i] * up;
    } else {
        for (int j = lane; j < D; j += 32) mine[j] *= up;
    }
    __syncthreads();
    const int nkt = D / HBK, mt = (blockIdx.x * 8) / BM, rg = ((blockIdx.x * 8) % BM) >> 3;
    uint8_t *base = image + (size_t)mt * nkt * A_TILE_BYTES + rg * 512;
    for (int e = tid; e < nkt * 32; e += 256) {
        const int kt = e >> 5, k8 = (e >> 3) & 3, r8 = e & 7;
        const float4 a = *reinterpret_cast<const float4 *>(&rp_rows[r8 * stride + kt * HBK + k8 * 8]);
        const float4 b = *reinterpret_cast<const float4 *>(&rp_rows[r8 * stride + kt * HBK + k8 * 8 + 4]);
        const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint4 hi, lo;
        split8(w, hi, lo);
        uint8_t *dst = base + (size_t)kt * A_TILE_BYTES + k8 * 128 + r8 * 16;
        *reinterpret_cast<uint4 *>(dst) = hi;
        *reinterpret_cast<uint4 *>(dst + BM * HBK * 2) = lo;
    }
}

int32_t pack_weight_half(const float *W, const float *gamma, const float *k_scale, int K, int N, float *image, cudaStream_t st) {
    const int bn = tile_cols(N), tiles = (N + bn - 1) / bn, rows = tiles * bn;
    float *un = image + (size_t)rows * K, *up = un + rows;
    half_scale_kernel<<<(rows + 255) / 256, 256, 0, st>>>(W, nullptr, gamma, k_scale, K, N, rows, un, up);
    dim3 grid(K / HBK, tiles);
    uint8_t *im = reinterpret_cast<uint8_t *>(image);
    if (bn == 256) half_pack_kernel<256><<<grid, 256, 0, st>>>(W, nullptr, gamma, k_scale, up, K, N, im);
    else half_pack_kernel<192><<<grid, 256, 0, st>>>(W, nullptr, gamma, k_scale, up, K, N, im);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t pack_weight_pair_half(const float *W1, const float *W3, const float *gamma, int K, int F, float *image, cudaStream_t st) {
    JGPT_REQUIRE(half_ok(K, F), JGPT_ERR_UNSUPPORTED, "pack_weight_pair_half: K=%d F=%d", K, F);
    float *un = image + (size_t)2 * F * K, *up = un + 2 * F;
    half_scale_kernel<<<(2 * F + 255) / 256, 256, 0, st>>>(W1, W3, gamma, nullptr, K, F, 2 * F, un, up);
    half_pack_kernel<256><<<dim3(K / HBK, F / 128), 256, 0, st>>>(W1, W3, gamma, nullptr, up, K, F, reinterpret_cast<uint8_t *>(image));
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t column_scales(const float *W, const float *gamma, int K, int N, float *scale, cudaStream_t st) {
    column_scale_kernel<<<(N + 255) / 256, 256, 0, st>>>(W, gamma, K, N, scale);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t pair_scales(const float *W1, const float *W3, const float *gamma, int K, int F, float *scale, cudaStream_t st) {
    float *r = scale + F;
    double *size = reinterpret_cast<double *>(r + K);  // F and K are even: 8-byte aligned
    pair_row_size_kernel<<<K, 256, 0, st>>>(W1, W3, gamma, K, F, size);
    pair_weight_kernel<<<(K + 255) / 256, 256, 0, st>>>(size, K, r);
    pair_scale_kernel<<<(F + 255) / 256, 256, 0, st>>>(W1, W3, gamma, r, K, F, scale);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t rmsnorm_pack_half(const float *x, const float *r, int M, int D, float eps, float *image, float *a_un, cudaStream_t st, int pdl) {
    const size_t smem = sizeof(float) * 8 * (size_t)(D + 4);
    JGPT_REQUIRE(D % HBK == 0 && smem <= 48 * 1024, JGPT_ERR_UNSUPPORTED, "rmsnorm_pack_half: d_model %d", D);
    const int padded_rows = (M + BM - 1) / BM * BM;  // rows past M are written as zeros
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(padded_rows / 8)), cfg.blockDim = dim3(256), cfg.dynamicSmemBytes = smem, cfg.stream = st, cfg.attrs = attr, cfg.numAttrs = pdl & 1;
    JGPT_CUDA_TRY(cudaLaunchKernelEx(&cfg, rmsnorm_pack_half_kernel, x, r, M, D, eps, reinterpret_cast<uint8_t *>(image), a_un, pdl));
    return JGPT_OK;
}

int32_t pack_activations(const float *A, const int *rowsel, int M, int K, float *image, cudaStream_t st) {
    dim3 grid(K / BK, (M + BM - 1) / BM);
    pack_kernel<BM, false><<<grid, 256, 0, st>>>(A, rowsel, M, K, image);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t rmsnorm_pack(const float *x, const float *gamma, int M, int D, float eps, float *image, cudaStream_t st) {
    const size_t smem = sizeof(float) * 8 * (size_t)(D + 4);
    JGPT_REQUIRE(D % BK == 0 && smem <= 48 * 1024, JGPT_ERR_UNSUPPORTED, "rmsnorm_pack: d_model %d", D);
    const int padded_rows = (M + BM - 1) / BM * BM;  // rows past M are written as zeros
    rmsnorm_pack_kernel<<<padded_rows / 8, 256, smem, st>>>(x, gamma, M, D, eps, image);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t pack_weight(const float *W, int K, int N, float *image, cudaStream_t st) {
    const int bn = tile_cols(N);
    dim3 grid(K / BK, (N + bn - 1) / bn);
    if (bn == 256) pack_kernel<256, true><<<grid, 256, 0, st>>>(W, nullptr, N, K, image);
    else pack_kernel<192, true><<<grid, 256, 0, st>>>(W, nullptr, N, K, image);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}
int32_t pack_weight_pair(const float *W1, const float *W3, int K, int F, float *image, cudaStream_t st) {
    JGPT_REQUIRE(swiglu_shape_ok(K, F), JGPT_ERR_UNSUPPORTED, "pack_weight_pair: K=%d F=%d", K, F);
    dim3 grid(K / BK, F / 128);
    pack_pair_kernel<<<grid, 256, 0, st>>>(W1, W3, K, F, image);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}

// ------------------------------------------------------------------------------------------------
// tcgen05: descriptors and the TF32 instruction (the wrappers that do not depend on the operand type: tcgen05.cuh)
// ------------------------------------------------------------------------------------------------
// Shared-memory matrix descriptor, no swizzle: start address, leading / stride byte offsets in 16-byte units,
// descriptor version 1 (bits 46-47), base offset 0, layout type 0.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(LBO >> 4) << 16) | ((uint64_t)(SBO >> 4) << 32) | (1ull << 46);
}
// Instruction descriptor: D fp32 (bits 4-5 = 1), A and B TF32 or both f16 (bits 7-9, 10-12 = 2 or 0), both K-major, N / 8 at
// bit 17, M / 16 at bit 24.
template <int BN, bool HALF>
__host__ __device__ constexpr uint32_t instr_desc() {
    return (1u << 4) | ((HALF ? 0u : 2u) << 7) | ((HALF ? 0u : 2u) << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_f16_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// ------------------------------------------------------------------------------------------------
// The GEMM: a persistent CTA per SM walks the output tiles (n fastest, so CTAs running side by side share the
// A tile through L2).  The accumulator is double-buffered in tensor memory (2 x 256 columns): while the
// epilogue warps drain tile j, the MMA thread is already accumulating tile j + 1, and the bulk copies run
// ahead of both through the stage ring.
//
// MODE 0: C row major.  MODE 2: C = R + product.  MODE 1 (BN = 256 over a W1/W3 pair image): columns [0,128) of the tile are h1,
// columns [128,256) are g for the same 128 outputs; the epilogue writes h1 * g * sigmoid(g) (sigmoid clamped
// to 1 / 0 at |g| >= 20: sigmoid_kernel, mul_kernel, src/main/cpp/jgpt_cuda_extra_kernels_launches.inl:799-832)
// as the activation image of the next product.
// ------------------------------------------------------------------------------------------------
template <int BN, int STAGES>
constexpr uint32_t smem_bytes() { return (uint32_t)STAGES * (A_TILE_BYTES + (uint32_t)BN * BK * 8u) + 128u; }

struct TileWalk {
    int n_tiles_n, nb, total;  // tiles along N, products in the batch, total tiles
    int image_cols;            // rows of a tile of the weight image; BN or a multiple of it
};

template <int BN, int STAGES, int MODE, bool HALF>
__global__ void __launch_bounds__(THREADS, 1) gemm_umma_kernel(const float *__restrict__ Aimg, const Batch B, const TileWalk walk,
                                                               int M, int K, int N, int *__restrict__ status, const PagedAppendArgs pa, int pdl) {
    constexpr int W_TILE_FLOATS = BN * BK * 2;
    constexpr uint32_t W_TILE_BYTES = W_TILE_FLOATS * 4, STAGE_BYTES = A_TILE_BYTES + W_TILE_BYTES;
    constexpr uint32_t IDESC = instr_desc<BN, HALF>();
    constexpr int KT = HALF ? HBK : BK;  // k of a stage; the tile's bytes are the same
    static_assert(BN % 64 == 0 && BN <= 256 && (MODE != 1 || BN == 256), "bad tile width");
    static_assert(MODE >= 0 && MODE <= 3, "MODE 3: products 1 and 2 of the batch are K and V rows for the paged store");
    extern __shared__ uint8_t umma_smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t s_tmem_base;
    __shared__ int s_abort_mem;
    volatile int *s_abort = &s_abort_mem;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nkt = K / KT;
    if (pdl & 2) griddep_launch_dependents();
    uint8_t *tiles = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(umma_smem_raw) + 127) & ~(uintptr_t)127);

    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) mbar_init(&full_bar[s], 1), mbar_init(&empty_bar[s], 1);
        for (int b = 0; b < 2; b++) mbar_init(&acc_full[b], 1), mbar_init(&acc_empty[b], EPI_WARPS);  // one arrival per epilogue warp
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&s_tmem_base, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem_base;
    if (pdl & 1) griddep_wait();  // what lies above runs beside the launch in front

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;  // k steps issued so far, over all tiles: stage = it % STAGES
            for (int t = blockIdx.x; t < walk.total && !*s_abort; t += gridDim.x) {
                const int n_idx = t % walk.n_tiles_n, z = (t / walk.n_tiles_n) % walk.nb, m_idx = t / (walk.n_tiles_n * walk.nb);
                const float *__restrict__ a_src = Aimg + (size_t)m_idx * nkt * A_TILE_FLOATS;
                // BN rows of an image tile: its row groups of eight lie one after the other, in the high and in the low half
                const int wt = walk.image_cols, w_tile = n_idx * BN / wt, w_floats = wt * BK * 2;
                const float *__restrict__ w_src = (z == 0 ? B.Wimg[0] : (z == 1 ? B.Wimg[1] : B.Wimg[2])) + (size_t)w_tile * nkt * w_floats +
                                                  (n_idx * BN - w_tile * wt) / 8 * 128;
                for (int kt = 0; kt < nkt; kt++, it++) {
                    const uint32_t s = it % STAGES, use = it / STAGES;
                    if (use > 0 && !mbar_wait_bounded(&empty_bar[s], (use - 1) & 1u, status, s_abort)) break;
                    uint8_t *dst = tiles + (size_t)s * STAGE_BYTES;
                    mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                    bulk_g2s(dst, a_src + (size_t)kt * A_TILE_FLOATS, A_TILE_BYTES, &full_bar[s]);
                    if (wt == BN) {
                        bulk_g2s(dst + A_TILE_BYTES, w_src + (size_t)kt * W_TILE_FLOATS, W_TILE_BYTES, &full_bar[s]);
                    } else {
                        bulk_g2s(dst + A_TILE_BYTES, w_src + (size_t)kt * w_floats, W_TILE_BYTES / 2, &full_bar[s]);
                        bulk_g2s(dst + A_TILE_BYTES + W_TILE_BYTES / 2, w_src + (size_t)kt * w_floats + w_floats / 2, W_TILE_BYTES / 2, &full_bar[s]);
                    }
                }
            }
            if (*s_abort) {
                // Copies already issued still target this CTA's shared memory: give each a bounded chance to land.
                for (uint32_t k = it > (uint32_t)STAGES ? it - STAGES : 0; k < it; k++) {
                    const uint32_t s = k % STAGES, ph = (k / STAGES) & 1u;
                    for (uint32_t i = 0; i < (1u << 16) && !mbar_try_wait(&full_bar[s], ph); i++) {
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t it = 0, j = 0;  // k steps consumed; tiles started
            bool ok = true;
            for (int t = blockIdx.x; t < walk.total && ok; t += gridDim.x, j++) {
                const uint32_t buf = j & 1u, round = j >> 1;
                if (round > 0 && !mbar_wait_bounded(&acc_empty[buf], (round - 1) & 1u, status, s_abort)) break;
                tc_fence_after();
                const uint32_t acc = tmem + buf * 256u;
                for (int kt = 0; kt < nkt; kt++, it++) {
                    const uint32_t s = it % STAGES, use = it / STAGES;
                    if (!mbar_wait_bounded(&full_bar[s], use & 1u, status, s_abort)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_hi = smem_u32(tiles + (size_t)s * STAGE_BYTES), a_lo = a_hi + A_TILE_BYTES / 2;
                    const uint32_t w_hi = a_hi + A_TILE_BYTES, w_lo = w_hi + W_TILE_BYTES / 2;
#pragma unroll
                    for (int ks = 0; ks < 2; ks++) {
                        const uint32_t adv = ks * 2 * LBO;  // two 16-byte core-matrix columns per K = 8 (f16: 16) step
                        const uint64_t ah = smem_desc(a_hi + adv), al = smem_desc(a_lo + adv);
                        const uint64_t wh = smem_desc(w_hi + adv), wl = smem_desc(w_lo + adv);
                        if constexpr (HALF) {
                            mma_f16_ss(acc, ah, wh, IDESC, (kt | ks) != 0);
                            mma_f16_ss(acc, al, wh, IDESC, 1);
                            mma_f16_ss(acc, ah, wl, IDESC, 1);
                        } else {
                            mma_tf32_ss(acc, ah, wh, IDESC, (kt | ks) != 0);
                            mma_tf32_ss(acc, al, wh, IDESC, 1);
                            mma_tf32_ss(acc, ah, wl, IDESC, 1);
                        }
                    }
                    mma_commit(&empty_bar[s]);  // the stage is free once these MMAs have read it
                }
                if (ok) mma_commit(&acc_full[buf]);
            }
        }
    } else {
        const int quarter = warp & 3;  // a warp reads TMEM lanes [32 * (warp % 4), +32)
        const int half = (warp - 2) >> 2;  // which half of the tile's columns
        const int rloc = quarter * 32 + lane;
        uint32_t j = 0;
        for (int t = blockIdx.x; t < walk.total; t += gridDim.x, j++) {
            const uint32_t buf = j & 1u, round = j >> 1;
            const uint32_t acc = tmem + buf * 256u;
            const int n_idx = t % walk.n_tiles_n, z = (t / walk.n_tiles_n) % walk.nb, m_idx = t / (walk.n_tiles_n * walk.nb);
            const int m = m_idx * BM + rloc, n0 = n_idx * BN;
            constexpr int SLABS = BN / 2 / 32;  // 32-column slabs per warp
            float4 res[MODE == 2 ? SLABS : 1][8];
            if (MODE == 2) {
                // The residual rows of this tile are requested before the accumulator is ready: their latency hides
                // behind the MMAs.  (R may be C itself: every element is read, then written, by this one thread.)
                const float *R = z == 0 ? B.R[0] : (z == 1 ? B.R[1] : B.R[2]);
#pragma unroll
                for (int sl = 0; sl < SLABS; sl++)
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const int n = n0 + half * (BN / 2) + sl * 32 + q * 4;
                        res[sl][q] = (m < M && n < N) ? *reinterpret_cast<const float4 *>(R + (size_t)m * N + n)
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
            }
            // fp16 images: the factors that undo the operands' powers of two
            const float a_un = (HALF && B.a_un && m < M) ? B.a_un[m] : 1.f;
            const float *w_un = HALF ? (z == 0 ? B.Wimg[0] : (z == 1 ? B.Wimg[1] : B.Wimg[2])) +
                                           (size_t)((walk.n_tiles_n * BN + walk.image_cols - 1) / walk.image_cols) * nkt * (walk.image_cols * BK * 2) + (size_t)n_idx * BN
                                     : nullptr;
            auto unscale = [&](float (&v)[32], int c) {  // 32 columns of the tile from c on
                if constexpr (HALF) {
#pragma unroll
                    for (int q = 0; q < 32; q += 4) {
                        const float4 u = __ldg(reinterpret_cast<const float4 *>(w_un + c + q));
                        v[q] *= a_un * u.x, v[q + 1] *= a_un * u.y, v[q + 2] *= a_un * u.z, v[q + 3] *= a_un * u.w;
                    }
                }
            };
            int ok = 0;
            if (lane == 0) ok = mbar_wait_bounded(&acc_full[buf], round & 1u, status, s_abort) ? 1 : 0;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            tc_fence_after();
            if (MODE == 3 && z != 0) {
                // K (z == 1) or V (z == 2) rows of a prefill: row m is slot m - row0 of its sequence.  Same arithmetic
                // and store shape as kv_append_rows_kernel (RoPE from the table with separately rounded products, fp16
                // round-to-nearest-even, 16-byte stores; the last prompt row zero-fills the rest of its block).
                bool row_ok = m < M;
                int slot = 0, tail = 0;
                size_t blk = 0;
                float2 cs[8];
                if (row_ok) {
                    int lo = 0, hi = pa.n_seqs - 1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (pa.seqs[mid].row0 <= m) lo = mid; else hi = mid - 1;
                    }
                    const PrefillSeq sd = pa.seqs[lo];
                    slot = m - sd.row0;
                    const int rp = sd.rope_off + slot;
                    if (slot < 0 || slot >= sd.S || rp < 0 || rp >= pa.max_positions) {
                        atomicOr(pa.status, DEV_STATUS_BAD_POSITION);
                        row_ok = false;
                    } else {
                        const int phys = pa.table[(size_t)sd.seq_id * pa.mbs + slot / kBlockTokens];
                        if (phys < 0 || phys >= pa.n_blocks) {
                            atomicOr(pa.status, DEV_STATUS_BAD_BLOCK);
                            row_ok = false;
                        } else {
                            blk = ((size_t)pa.layer * pa.n_blocks + phys) * pa.H;
                            tail = slot == sd.S - 1 ? kBlockTokens - 1 - slot % kBlockTokens : 0;
                            if (z == 1) {
#pragma unroll
                                for (int q = 0; q < 8; q++) cs[q] = pa.rope[(size_t)rp * 8 + q];
                            }
                        }
                    }
                }
#pragma unroll
                for (int sl = 0; sl < SLABS; sl++) {
                    const int c0 = half * (BN / 2) + sl * 32;
                    if (n0 + c0 >= N) break;  // uniform across the warp
                    float v[32];
                    load_acc32(acc, quarter, c0, v);
                    unscale(v, c0);
                    if (row_ok) {
#pragma unroll
                        for (int hh = 0; hh < 2; hh++) {
                            const int head = (n0 + c0) / 16 + hh;
                            if (head < pa.H) {
                                __align__(16) __half hv[16];
#pragma unroll
                                for (int q = 0; q < 8; q++) {
                                    const float x1 = v[hh * 16 + 2 * q], x2 = v[hh * 16 + 2 * q + 1];
                                    if (z == 1) {
                                        hv[2 * q] = __float2half_rn(__fsub_rn(__fmul_rn(x1, cs[q].x), __fmul_rn(x2, cs[q].y)));
                                        hv[2 * q + 1] = __float2half_rn(__fadd_rn(__fmul_rn(x1, cs[q].y), __fmul_rn(x2, cs[q].x)));
                                    } else {
                                        hv[2 * q] = __float2half_rn(x1), hv[2 * q + 1] = __float2half_rn(x2);
                                    }
                                }
                                __half *dst = pa.kv + (blk + head) * (size_t)(2 * kBlockTokens * 16) + (size_t)(slot % kBlockTokens) * 16 +
                                              (z == 2 ? kBlockTokens * 16 : 0);
                                *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(hv);
                                *reinterpret_cast<uint4 *>(dst + 8) = *reinterpret_cast<const uint4 *>(hv + 8);
                                for (int t2 = 1; t2 <= tail; t2++) {
                                    *reinterpret_cast<uint4 *>(dst + t2 * 16) = make_uint4(0, 0, 0, 0);
                                    *reinterpret_cast<uint4 *>(dst + t2 * 16 + 8) = make_uint4(0, 0, 0, 0);
                                }
                            }
                        }
                    }
                }
            } else if (MODE != 1) {
                float *C = z == 0 ? B.C[0] : (z == 1 ? B.C[1] : B.C[2]);  // selects, not an indexed copy of B
#pragma unroll
                for (int sl = 0; sl < SLABS; sl++) {
                    const int c0 = half * (BN / 2) + sl * 32;
                    if (n0 + c0 >= N) break;  // uniform across the warp
                    float v[32];
                    load_acc32(acc, quarter, c0, v);
                    unscale(v, c0);
                    if (m < M) {
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            const int n = n0 + c0 + q * 4;
                            if (n < N) {
                                float4 o = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                                if (MODE == 2) {
                                    const float4 r4 = res[sl][q];
                                    o.x += r4.x, o.y += r4.y, o.z += r4.z, o.w += r4.w;
                                }
                                *reinterpret_cast<float4 *>(C + (size_t)m * N + n) = o;
                            }
                        }
                    }
                }
            } else {
                // N is F here; the activation image has F / 16 (fp16: F / 32) k tiles per row tile.  Rows past M are zero in A,
                // so h1 = g = 0 and zeros are written: the image stays fully defined.
                const int out_nkt = N / KT;
                float *__restrict__ out = B.C[0] + (size_t)m_idx * out_nkt * A_TILE_FLOATS + chunk_offset(rloc, 0);
#pragma unroll 1
                for (int c0 = half * 64; c0 < half * 64 + 64; c0 += 32) {
                    float h[32], g[32];
                    load_acc32(acc, quarter, c0, h);
                    load_acc32(acc, quarter, 128 + c0, g);
                    unscale(h, c0), unscale(g, 128 + c0);
#pragma unroll
                    for (int q = 0; q < 32; q++) {
                        const float gv = g[q];
                        float s;
                        if (gv >= 20.f) s = 1.f;
                        else if (gv <= -20.f) s = 0.f;
                        else s = 1.f / (1.f + expf(-gv));
                        h[q] = h[q] * (gv * s);
                    }
                    if constexpr (HALF) {  // these 32 columns are one k tile of the next product
                        // (the finished value times the powers of two of its row and column: h alone may exceed what h g sigmoid(g) can reach)
                        const float r_up = m < M ? B.r_up[m] : 1.f;
#pragma unroll
                        for (int q = 0; q < 32; q += 4) {
                            const float4 u = __ldg(reinterpret_cast<const float4 *>(B.c_up + n_idx * 128 + c0 + q));
                            h[q] = h[q] * r_up * u.x, h[q + 1] = h[q + 1] * r_up * u.y, h[q + 2] = h[q + 2] * r_up * u.z, h[q + 3] = h[q + 3] * r_up * u.w;
                        }
                        uint8_t *tile = reinterpret_cast<uint8_t *>(B.C[0] + ((size_t)m_idx * out_nkt + (n_idx * 128 + c0) / HBK) * A_TILE_FLOATS);
#pragma unroll
                        for (int k8 = 0; k8 < 4; k8++) {
                            const float w[8] = {h[k8 * 8], h[k8 * 8 + 1], h[k8 * 8 + 2], h[k8 * 8 + 3], h[k8 * 8 + 4], h[k8 * 8 + 5], h[k8 * 8 + 6], h[k8 * 8 + 7]};
                            uint4 hi, lo;
                            split8(w, hi, lo);
                            *reinterpret_cast<uint4 *>(tile + half_chunk(rloc, k8)) = hi;
                            *reinterpret_cast<uint4 *>(tile + BM * HBK * 2 + half_chunk(rloc, k8)) = lo;
                        }
                    } else {
#pragma unroll
                    for (int q = 0; q < 32; q += 4) {
                        const int k = n_idx * 128 + c0 + q;  // column of the activation = k of the next product
                        float4 hi, lo;
                        split4(make_float4(h[q], h[q + 1], h[q + 2], h[q + 3]), hi, lo);
                        float *dst = out + (size_t)(k / BK) * A_TILE_FLOATS + ((k % BK) >> 2) * 32;
                        *reinterpret_cast<float4 *>(dst) = hi;
                        *reinterpret_cast<float4 *>(dst + BM * BK) = lo;
                    }
                    }
                }
            }
            // this warp has read everything it needs from the buffer: hand it back to the MMA thread
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

static int sm_count_of_current_device() {
    static int cached[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    int &c = cached[dev & 63];
    if (c == 0 && cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) c = 1;
    return c > 0 ? c : 1;
}

template <int BN, int STAGES, int MODE, bool HALF = false>
static int32_t launch_t(const TileWalk &walk, const float *Aimg, const Batch &b, int M, int K, int N, int *d_status, cudaStream_t st,
                        const PagedAppendArgs &pa = PagedAppendArgs(), int pdl = 0) {
    constexpr uint32_t smem = smem_bytes<BN, STAGES>();
    static thread_local int set_for = -1;  // the opt-in to more than 48 KiB, once per device
    int dev = 0;
    JGPT_CUDA_TRY(cudaGetDevice(&dev));
    if (set_for != dev) {
        JGPT_CUDA_TRY(cudaFuncSetAttribute(gemm_umma_kernel<BN, STAGES, MODE, HALF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        set_for = dev;
    }
    const int grid = walk.total < sm_count_of_current_device() ? walk.total : sm_count_of_current_device();
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)grid), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = smem, cfg.stream = st, cfg.attrs = attr, cfg.numAttrs = pdl & 1;
    JGPT_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_umma_kernel<BN, STAGES, MODE, HALF>, Aimg, b, walk, M, K, N, d_status, pa, pdl));
    return JGPT_OK;
}

// Columns per CTA of a product on its own: the fewest rounds of CTAs times what a tile takes, its columns and about 64 more for its
// share of A and its start; the widest of equals.  Calls in a row with 64, 128, 192 and 256 columns, us, the choice of this rule first:
// 3000 x 384 x 768 128: 24.6 (30.9, 26.7, 30.8), 1000 x 384 x 768 64: 20.5 (22.6, 24.6, 28.7), 6000 x 1024 x 1024 192: 77 (169, 100, 86),
// 20000 x 384 x 768 256: 84 (149, 96, 84).  Against three launches (an image each, then tiles of 192 or 256), in a row and alone on operands that
// have left L2: 3000 x 384 x 768 36.4 -> 24.6 and 54 -> 40, 1500 x 2048 x 2048 88 -> 76 and 107 -> 95.  Replayed from a graph, its launches
// one behind the other, the first takes 16.2 -> 15.8: more bytes leave L2 (eight per element and tile, 110 MB in 144 tiles, 83 MB in 72).
static int matmul_cols(int M, int N, int sms) {
    const long long rows = (M + BM - 1) / BM;
    int best = 0;
    long long least = 0;
    for (int bn : {256, 192, 128, 64}) {
        const long long cost = (rows * ((N + bn - 1) / bn) + sms - 1) / sms * (bn + 64);
        if (!best || cost < least) best = bn, least = cost;
    }
    return best;
}
uint64_t matmul_scratch_floats(int M, int K, int N) {
    return activation_image_floats(M, K) + image_floats(N, K, matmul_cols(M, N, sm_count_of_current_device()));
}
int32_t matmul(const float *A, const float *B, float *C, int M, int K, int N, float *scratch, int *d_status, cudaStream_t st) {
    JGPT_REQUIRE(shape_ok(K, N) && M > 0, JGPT_ERR_INVALID_ARGUMENT, "matmul: unsupported shape M=%d K=%d N=%d", M, K, N);
    float *wimg = scratch + activation_image_floats(M, K);
    Batch b{};
    b.Wimg[0] = wimg, b.C[0] = C, b.R[0] = nullptr;
    auto run = [&](auto cols, auto stages) -> int32_t {
        constexpr int BN = decltype(cols)::value, ST = decltype(stages)::value;
        const int a_tiles = (M + BM - 1) / BM;
        TileWalk walk{(N + BN - 1) / BN, 1, 0, BN};
        walk.total = walk.n_tiles_n * a_tiles;
        pack_both_kernel<BN><<<(unsigned)(K / BK * (a_tiles + walk.n_tiles_n)), 256, 0, st>>>(A, M, B, N, K, scratch, wimg, a_tiles);
        JGPT_CUDA_TRY(cudaGetLastError());
        return launch_t<BN, ST, 0, false>(walk, scratch, b, M, K, N, d_status, st, PagedAppendArgs(), 1);
    };
    switch (matmul_cols(M, N, sm_count_of_current_device())) {
        case 64: return run(std::integral_constant<int, 64>(), std::integral_constant<int, 8>());
        case 128: return run(std::integral_constant<int, 128>(), std::integral_constant<int, 6>());
        case 192: return run(std::integral_constant<int, 192>(), std::integral_constant<int, 5>());
        default: return run(std::integral_constant<int, 256>(), std::integral_constant<int, 4>());
    }
}

// Fewer rows than the image's tiles fill SMs with: 64 columns per CTA where that takes fewer rounds of CTAs times what a tile takes, its columns and
// what goes with its 128 rows: as much as 128 columns, since both come out of L2, and less where k is short and the epilogue of a wide tile
// counts.  At width 384 on 148 SMs that is up to 3072 rows for Wo and W2 and up to 1024 for Q,K,V.  (1130 rows are 18 tiles of Wo and of W2, three times as many of
// 64: 23.9 -> 15.8 us a launch.  With the early launches three prompts of 848 rows take 1339 -> 969 us, three of 1130 1366 -> 1045.)
// Four layers of other widths, d_ff twice as wide, all wide and with the weight of the rows at 64 and as it is, us: 1300 rows of 1024 796, 862, 796,
// 1550 of 832 748, 853, 749, 4200 of 640 875, 972, 872; 5000 rows of 256 530, 490, 495, 3000 of 448 600, 578, 583, 8000 of 320 786, 812, 783.
static bool narrow_tiles(TileWalk &walk, int N, int M, int K) {
    const int sms = sm_count_of_current_device(), tiles = (N + 63) / 64 * walk.nb * ((M + BM - 1) / BM), rows = K <= 512 ? 96 : 128;
    if ((tiles + sms - 1) / sms * (64 + rows) >= (walk.total + sms - 1) / sms * (walk.image_cols + rows)) return false;
    walk.n_tiles_n = (N + 63) / 64, walk.total = tiles;
    return true;
}

template <bool HALF>
static int32_t launch_rows(const float *Aimg, const Batch &b, int nb, int M, int K, int N, int *d_status, cudaStream_t st, int pdl = 0) {
    JGPT_REQUIRE(shape_ok(K, N) && (!HALF || K % HBK == 0) && M > 0 && nb >= 1 && nb <= 3, JGPT_ERR_INVALID_ARGUMENT,
                 "gemm_umma: unsupported shape M=%d K=%d N=%d", M, K, N);
    const int bn = tile_cols(N);
    TileWalk walk{(N + bn - 1) / bn, nb, 0, bn};
    walk.total = walk.n_tiles_n * nb * ((M + BM - 1) / BM);
    bool residual = b.R[0] != nullptr;
    for (int z = 0; z < nb; z++)
        JGPT_REQUIRE((b.R[z] != nullptr) == residual, JGPT_ERR_INVALID_ARGUMENT, "gemm_umma: residuals for all products of a batch or for none");
    const PagedAppendArgs none{};
    if constexpr (HALF) {
        if (residual && narrow_tiles(walk, N, M, K)) return launch_t<64, 8, 2, HALF>(walk, Aimg, b, M, K, N, d_status, st, none, pdl);
    }
    if (bn == 256)
        return residual ? launch_t<256, 4, 2, HALF>(walk, Aimg, b, M, K, N, d_status, st, none, pdl) : launch_t<256, 4, 0, HALF>(walk, Aimg, b, M, K, N, d_status, st, none, pdl);
    return residual ? launch_t<192, 5, 2, HALF>(walk, Aimg, b, M, K, N, d_status, st, none, pdl) : launch_t<192, 5, 0, HALF>(walk, Aimg, b, M, K, N, d_status, st, none, pdl);
}
int32_t launch(const float *Aimg, const Batch &b, int nb, int M, int K, int N, int *d_status, cudaStream_t st) {
    return launch_rows<false>(Aimg, b, nb, M, K, N, d_status, st);
}
int32_t launch_half(const float *Aimg, const Batch &b, int nb, int M, int K, int N, int *d_status, cudaStream_t st, int pdl) {
    return launch_rows<true>(Aimg, b, nb, M, K, N, d_status, st, pdl);
}

template <bool HALF>
static int32_t launch_qkv(const float *Aimg, const Batch &b, int M, int K, int N, const PagedAppendArgs &pa, int *d_status, cudaStream_t st, int pdl = 0) {
    JGPT_REQUIRE(shape_ok(K, N) && (!HALF || K % HBK == 0) && M > 0 && N == pa.H * 16, JGPT_ERR_INVALID_ARGUMENT,
                 "gemm_umma qkv: unsupported shape M=%d K=%d N=%d (heads %d, d_head 16)", M, K, N, pa.H);
    const int bn = tile_cols(N);
    TileWalk walk{(N + bn - 1) / bn, 3, 0, bn};
    walk.total = walk.n_tiles_n * 3 * ((M + BM - 1) / BM);
    if constexpr (HALF) {
        if (narrow_tiles(walk, N, M, K)) return launch_t<64, 8, 3, HALF>(walk, Aimg, b, M, K, N, d_status, st, pa, pdl);
    }
    if (bn == 256) return launch_t<256, 4, 3, HALF>(walk, Aimg, b, M, K, N, d_status, st, pa, pdl);
    return launch_t<192, 5, 3, HALF>(walk, Aimg, b, M, K, N, d_status, st, pa, pdl);
}
int32_t launch_qkv_paged(const float *Aimg, const Batch &b, int M, int K, int N, const PagedAppendArgs &pa, int *d_status, cudaStream_t st) {
    return launch_qkv<false>(Aimg, b, M, K, N, pa, d_status, st);
}
int32_t launch_qkv_paged_half(const float *Aimg, const Batch &b, int M, int K, int N, const PagedAppendArgs &pa, int *d_status, cudaStream_t st, int pdl) {
    return launch_qkv<true>(Aimg, b, M, K, N, pa, d_status, st, pdl);
}

template <bool HALF>
static int32_t launch_pair(const float *Aimg, const float *Wpair_img, const float *a_un, const float *c_up, int M, int K, int F, float *act_image,
                           int *d_status, cudaStream_t st, int pdl = 0) {
    JGPT_REQUIRE(swiglu_shape_ok(K, F) && (!HALF || K % HBK == 0) && M > 0, JGPT_ERR_INVALID_ARGUMENT,
                 "gemm_umma swiglu: unsupported shape M=%d K=%d F=%d", M, K, F);
    Batch b{};
    b.Wimg[0] = Wpair_img, b.C[0] = act_image, b.a_un = a_un, b.r_up = a_un + M, b.c_up = c_up;
    TileWalk walk{F / 128, 1, 0, 256};
    walk.total = walk.n_tiles_n * ((M + BM - 1) / BM);
    return launch_t<256, 4, 1, HALF>(walk, Aimg, b, M, K, F, d_status, st, PagedAppendArgs(), pdl);
}
int32_t launch_swiglu(const float *Aimg, const float *Wpair_img, int M, int K, int F, float *act_image, int *d_status, cudaStream_t st) {
    return launch_pair<false>(Aimg, Wpair_img, nullptr, nullptr, M, K, F, act_image, d_status, st);
}
int32_t launch_swiglu_half(const float *Aimg, const float *Wpair_img, const float *a_un, const float *c_up, int M, int K, int F, float *act_image,
                           int *d_status, cudaStream_t st, int pdl) {
    return launch_pair<true>(Aimg, Wpair_img, a_un, c_up, M, K, F, act_image, d_status, st, pdl);
}

}  // namespace umma
}  // namespace jgpt
