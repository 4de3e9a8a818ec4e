// Products of few rows with fp32-level accuracy: the projections of a decode step and of a short prompt.
//
// At these sizes a product is not bound by bytes or by the tensor cores but by its longest chain: wait for the previous kernel, fetch
// the rows, multiply, add the k slices, store.  So everything that does not depend on the previous kernel is done before the wait and
// nothing in the loop meets at a barrier.  A CTA owns 16 or 32 columns; its eight warps split k, and a warp holds the weights of
// its k slice in registers, in the order the tensor core reads them (one 16-byte load per 8 columns, 16 k and lane, out of an image
// built once per weight set): requested before the wait, used for every row tile the CTA walks.  A lane loads the rows it multiplies
// itself, the next tile's while this one is summed and stored; the only barrier of a row tile is the one in front of the sum over the
// eight slices.  (Rows through a cp.async ring in shared memory: a prompt of 201 tokens 0.52 ms, against 0.45.)
//
// Accuracy: an fp32 operand is an fp16 high and an fp16 low part, 11 + 11 bits as the TF32 pair has, at half the tensor time (m16n8k16
// instead of two m16n8k8) and, for the weights, in the four bytes of the original.  fp16's narrow exponent is dealt with by powers of
// two, which change no bit: weights are scaled per column (image), rows per warp and row tile from the largest element of the slice,
// and the partial sums are scaled back before they are added.  The low parts carry 2^11 more and have an accumulator of their own (the two
// mixed products), so that they stay clear of fp16's subnormals as long as the high parts do: an element down to 2^-28 of the largest of
// its slice (column) is within 2^-23 of itself, like a TF32 pair at any size, below that an absolute error of 2^-50 of that
// largest remains.  Without the factor, one multiplication per row element less, the two were 2^-16 and 2^-39 (same times: 250 rows
// of 1000 9.42 ms, a prompt of 201 tokens 458 and 461 us).
//
// Against the form with shared-memory k tiles, TF32 pairs split in the loop and a barrier per 64 k (12 layers of 384, per launch inside
// a decode step of 64 rows, from the previous kernel's end to its own): Q,K,V 5.2 -> 3.2, Wo 4.1 -> 3.1, W1/W3 7.0 -> 3.7, W2 6.6 -> 2.8 us;
// per step: 8 rows 0.32 -> 0.23, 64 rows 0.45 -> 0.37, 250 rows 1.37 -> 1.18 ms with the attention of the same time; a prompt of 201
// tokens 0.72 -> 0.45 ms.  Error against float64 of the LM head's 384 x 8000 product: 1.5e-7 of the result (2-norm), 1.8e-7 with TF32
// pairs.
#include "gemm_rows.cuh"

#include <algorithm>

#include "ptx.cuh"

namespace jgpt {
namespace rows {

constexpr int kWarps = 8, kThreads = 256, kRows = 16;

// One CTA per 8 columns: a warp per column finds its largest element, then every lane writes its 16 bytes per 16 k.  Inside 16 k the
// tensor core's positions 2 t, 2 t + 1, 2 t + 8, 2 t + 9 of lane t hold k = 4 t .. 4 t + 3, so that a row's four elements are one load.
__global__ void __launch_bounds__(256) pack_kernel(const float *W, const float *W3, const float *gamma, int K, int N, uint4 *image, float *unscale) {
    __shared__ float s_scale[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto element = [&](int k, int n) {
        if (k >= K || n >= N) return 0.f;
        float w;
        if (W3) {
            w = (n & 1 ? W3 : W)[(size_t)k * (N / 2) + (n >> 1)];
        } else {
            w = W[(size_t)k * N + n];
        }
        return gamma ? gamma[k] * w : w;
    };
    const int n0 = blockIdx.x * 8;
    float mx = 0.f;
    for (int k = lane; k < K; k += 32) mx = fmaxf(mx, fabsf(element(k, n0 + warp)));
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (lane == 0) {
        float s, inv;
        pow2_scale(mx, s, inv);
        s_scale[warp] = s;
        unscale[n0 + warp] = inv;
    }
    __syncthreads();
    const int steps = (K + 15) / 16, g = lane >> 2, t = lane & 3;
    const float s = s_scale[g];
    for (int step = warp; step < steps; step += kWarps) {
        const int k = step * 16 + 4 * t;
        uint4 o;
        split_pair_wide(element(k, n0 + g) * s, element(k + 1, n0 + g) * s, o.x, o.z);
        split_pair_wide(element(k + 2, n0 + g) * s, element(k + 3, n0 + g) * s, o.y, o.w);
        image[((size_t)blockIdx.x * steps + step) * 32 + lane] = o;
    }
}

int32_t pack(const float *W, const float *W3, const float *gamma, int K, int N, void *image, cudaStream_t st) {
    const unsigned tiles = (unsigned)((N + 7) / 8);
    uint4 *im = static_cast<uint4 *>(image);
    pack_kernel<<<tiles, 256, 0, st>>>(W, W3, gamma, K, N, im, reinterpret_cast<float *>(im + (size_t)tiles * k_steps(K) * 32));
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}

// S: steps of 16 k per warp.  NT: column groups of 8 per CTA.
// CTAs of a kernel on an SM: two while 128 registers hold the weights, the rows and the sums.
template <int S, int NT>
constexpr int per_sm() { return S * NT <= 12 && S <= 4 ? 2 : 1; }

template <int S, int NT, int KIND>
__global__ void __launch_bounds__(kThreads, per_sm<S, NT>()) gemm_rows_kernel(const float *A, const Batch B, int M, int K, int N, const int *rowsel,
                                                                             const Fuse F, const PagedAppendArgs pa) {
    constexpr int BN = NT * 8, RS = BN + 8;
    constexpr bool PAIR = KIND != RESIDUAL;  // a thread sums two neighbouring columns: two results, h and g, or a pair to be turned
    constexpr int OUT = KIND == NORM_SWIGLU ? BN / 2 : BN;  // columns of the result per CTA
    static_assert(BN == (PAIR ? 32 : 16), "sixteen threads per row of the tile");
    __shared__ __align__(16) float red[2][kWarps][kRows][RS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int z = blockIdx.z;
#ifdef JGPT_B200_DECODE_TRACE
    timeline_in(F.timeline);
#endif
    const int steps = (K + 15) / 16, tiles = (N + 7) / 8;
    const uint4 *image = static_cast<const uint4 *>(z == 0 ? B.image[0] : (z == 1 ? B.image[1] : B.image[2]));
    float *C = z == 0 ? B.C[0] : (z == 1 ? B.C[1] : B.C[2]);
    const float *unscale = reinterpret_cast<const float *>(image + (size_t)tiles * steps * 32);
    const int step0 = warp * S, k0 = step0 * 16;
    uint4 w[S][NT];
#pragma unroll
    for (int j = 0; j < NT; j++)
#pragma unroll
        for (int s = 0; s < S; s++) {
            const int tile = blockIdx.x * NT + j;
            w[s][j] = (tile < tiles && step0 + s < steps) ? __ldg(image + ((size_t)tile * steps + step0 + s) * 32 + lane) : make_uint4(0, 0, 0, 0);
        }
    // the epilogue's share: row tid / 16 of the tile, column(s) c of it
    const int orow = tid >> 4, oj = tid & 15, c = PAIR ? 2 * oj : oj;
    const int Nout = KIND == NORM_SWIGLU ? N / 2 : N, col = blockIdx.x * OUT + (KIND == NORM_SWIGLU ? oj : c);
    const bool col_ok = col < Nout;  // N % 4 == 0: a pair is inside or outside as a whole
    float2 un = make_float2(0.f, 0.f);
    if (col_ok) un = PAIR ? __ldg(reinterpret_cast<const float2 *>(unscale + blockIdx.x * BN + c)) : make_float2(__ldg(unscale + col), 0.f);

    if (F.pdl & 1) griddep_wait();
#ifdef JGPT_B200_DECODE_TRACE
    timeline_at(F.timeline, 1);
#endif
    if (F.pdl & 2) griddep_launch_dependents();

    // This warp's k slice of 16 rows, straight into the registers of the lanes that multiply it: rows g and g + 8, four k per step of
    // 16.  Rows and k past the end become zeros.  Read through L2: an SM's L1 may hold the row of an earlier layer.
    float4 lo_row[S], hi_row[S];
    auto fetch = [&](int rt) {
        const int ma = rt * kRows + g, mb = ma + 8;
        const float *pa_ = A + (size_t)(ma < M ? (rowsel ? rowsel[ma] : ma) : 0) * K + k0 + 4 * t;
        const float *pb_ = A + (size_t)(mb < M ? (rowsel ? rowsel[mb] : mb) : 0) * K + k0 + 4 * t;
#pragma unroll
        for (int s = 0; s < S; s++) {
            const bool in = k0 + s * 16 + 4 * t < K;
            lo_row[s] = in && ma < M ? __ldcg(reinterpret_cast<const float4 *>(pa_ + s * 16)) : make_float4(0.f, 0.f, 0.f, 0.f);
            hi_row[s] = in && mb < M ? __ldcg(reinterpret_cast<const float4 *>(pb_ + s * 16)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    const int row_tiles = (M + kRows - 1) / kRows;
    int rb = 0;
    fetch(blockIdx.y);
    for (int rt = blockIdx.y; rt < row_tiles; rt += gridDim.y) {
        // what the epilogue adds or multiplies, and where its row goes, requested now
        const int m = rt * kRows + orow;
        const bool ok = m < M && col_ok;
        float *out = C + (size_t)m * Nout + col;
        float extra = 0.f;
        if (KIND == RESIDUAL) {
            if (ok) extra = __ldcg(out);
        } else if (m < M) {  // the sixteen lanes that share a row add its partial sums of squares, always in the same order
            const float *pp = F.ss_in + (size_t)(rowsel ? rowsel[m] : m) * F.parts_in;
            for (int p = oj; p < F.parts_in; p += 16) extra += __ldcg(pp + p);
        }
        __half *kv_at = nullptr;
        float2 turn = make_float2(1.f, 0.f);
        int dead = 0;  // slots of the block behind the prompt's last row
        if (KIND == NORM_PAGED && z > 0 && ok) {
            int lo = 0, hi = pa.n_seqs - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (pa.seqs[mid].row0 <= m) lo = mid; else hi = mid - 1;
            }
            const PrefillSeq sd = pa.seqs[lo];
            const int slot = m - sd.row0, rp = sd.rope_off + slot;
            const bool pos_ok = slot >= 0 && slot < sd.S && rp >= 0 && rp < pa.max_positions;
            const int phys = pos_ok ? pa.table[(size_t)sd.seq_id * pa.mbs + slot / kBlockTokens] : 0;
            if (!pos_ok) {
                atomicOr(pa.status, DEV_STATUS_BAD_POSITION);
            } else if (phys < 0 || phys >= pa.n_blocks) {
                atomicOr(pa.status, DEV_STATUS_BAD_BLOCK);
            } else {
                kv_at = pa.kv + (((size_t)pa.layer * pa.n_blocks + phys) * pa.H + col / 16) * (size_t)(2 * kBlockTokens * 16) +
                        (z == 2 ? kBlockTokens * 16 : 0) + (slot % kBlockTokens) * 16 + (col & 15);
                dead = slot == sd.S - 1 ? kBlockTokens - 1 - slot % kBlockTokens : 0;
                if (z == 1) turn = pa.rope[(size_t)rp * 8 + (col & 15) / 2];
            }
        }
        float m0 = 0.f, m1 = 0.f;
#pragma unroll
        for (int s = 0; s < S; s++) {
            m0 = fmaxf(m0, fmaxf(fmaxf(fabsf(lo_row[s].x), fabsf(lo_row[s].y)), fmaxf(fabsf(lo_row[s].z), fabsf(lo_row[s].w))));
            m1 = fmaxf(m1, fmaxf(fmaxf(fabsf(hi_row[s].x), fabsf(hi_row[s].y)), fmaxf(fabsf(hi_row[s].z), fabsf(hi_row[s].w))));
        }
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 1)), m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 1));
        m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, 2)), m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, 2));
        float s0, s1, u0, u1;
        pow2_scale(m0, s0, u0), pow2_scale(m1, s1, u1);
        float acc[NT][4], cor[NT][4];
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[j][e] = 0.f, cor[j][e] = 0.f;
#pragma unroll
        for (int s = 0; s < S; s++) {
            uint32_t ah[4], al[4];
            split_pair_wide(lo_row[s].x * s0, lo_row[s].y * s0, ah[0], al[0]);
            split_pair_wide(hi_row[s].x * s1, hi_row[s].y * s1, ah[1], al[1]);
            split_pair_wide(lo_row[s].z * s0, lo_row[s].w * s0, ah[2], al[2]);
            split_pair_wide(hi_row[s].z * s1, hi_row[s].w * s1, ah[3], al[3]);
            // the rows are in the parts: the next tile's are on their way during the last products, the sums and the stores
            if (s == S - 1 && rt + (int)gridDim.y < row_tiles) fetch(rt + gridDim.y);
#pragma unroll
            for (int j = 0; j < NT; j++) mma_16816(acc[j], ah, w[s][j].x, w[s][j].y);
#pragma unroll
            for (int j = 0; j < NT; j++) mma_16816(cor[j], al, w[s][j].x, w[s][j].y);
#pragma unroll
            for (int j = 0; j < NT; j++) mma_16816(cor[j], ah, w[s][j].z, w[s][j].w);
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            *reinterpret_cast<float2 *>(&red[rb][warp][g][j * 8 + 2 * t]) = make_float2(fmaf(cor[j][0], 1.f / kLowScale, acc[j][0]) * u0, fmaf(cor[j][1], 1.f / kLowScale, acc[j][1]) * u0);
            *reinterpret_cast<float2 *>(&red[rb][warp][g + 8][j * 8 + 2 * t]) = make_float2(fmaf(cor[j][2], 1.f / kLowScale, acc[j][2]) * u1, fmaf(cor[j][3], 1.f / kLowScale, acc[j][3]) * u1);
        }
        float inv = 0.f;
        if (KIND != RESIDUAL) {
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) extra += __shfl_xor_sync(0xffffffffu, extra, off);
            const float rms = sqrtf(extra / (float)K + F.eps);
            inv = (rms > 0.f && isfinite(rms)) ? (1.f / rms) : 0.f;
        }
        // the buffer of slices written here is rewritten two tiles later, behind the next tile's barrier
        __syncthreads();
        float2 v = make_float2(0.f, 0.f);
#pragma unroll
        for (int q = kWarps - 1; q >= 0; q--) {
            if (PAIR) {
                const float2 p = *reinterpret_cast<const float2 *>(&red[rb][q][orow][c]);
                v.x += p.x, v.y += p.y;
            } else {
                v.x += red[rb][q][orow][c];
            }
        }
        v.x *= un.x, v.y *= un.y;
        if (KIND == RESIDUAL) {
            const float x = extra + v.x;
            if (ok) *out = x;
            float sq = ok ? x * x : 0.f;
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
            if (oj == 0 && m < M) F.ss_out[(size_t)m * gridDim.x + blockIdx.x] = sq;
        } else {
            v.x *= inv, v.y *= inv;
            if (KIND == NORM_SWIGLU) {
                float sg;
                if (v.y >= 20.f) sg = 1.f;
                else if (v.y <= -20.f) sg = 0.f;
                else sg = 1.f / (1.f + expf(-v.y));
                if (ok) *out = v.x * (v.y * sg);
            } else if (KIND == NORM_PAGED && z > 0) {
                if (kv_at) {
                    const __half2 p = z == 1 ? __floats2half2_rn(__fsub_rn(__fmul_rn(v.x, turn.x), __fmul_rn(v.y, turn.y)),
                                                                 __fadd_rn(__fmul_rn(v.x, turn.y), __fmul_rn(v.y, turn.x)))
                                             : __floats2half2_rn(v.x, v.y);
                    *reinterpret_cast<__half2 *>(kv_at) = p;
                    for (int s = 1; s <= dead; s++) *reinterpret_cast<__half2 *>(kv_at + s * 16) = __floats2half2_rn(0.f, 0.f);
                }
            } else if (ok) {
                *reinterpret_cast<float2 *>(out) = v;
            }
        }
        rb ^= 1;
    }
#ifdef JGPT_B200_DECODE_TRACE
    timeline_at(F.timeline, 2);
#endif
}

constexpr int kMaxSteps32 = 4, kMaxSteps16 = 8;  // steps of 16 k per warp whose weights fit: 64 registers either way
constexpr size_t kSoloBytes = 115 * 1024;        // static and dynamic: more than half an SM, no two CTAs of the launch share one

bool shape_ok(Kind kind, int K) {
    const int s = (k_steps(K) + kWarps - 1) / kWarps;
    return K % 4 == 0 && k_steps(K) >= kWarps && s <= (kind == RESIDUAL ? kMaxSteps16 : kMaxSteps32);
}

template <int S, int NT, int KIND>
static int32_t launch_t(Ctx *ctx, const float *A, const Batch &b, int nb, int M, int K, int N, const int *rowsel, const Fuse &fuse, const PagedAppendArgs &pa) {
    auto *kernel = gemm_rows_kernel<S, NT, KIND>;
    constexpr size_t fixed = sizeof(float) * 2 * kWarps * kRows * (NT * 8 + 8), solo = kSoloBytes - fixed;
    static bool opted[64] = {};
    if (!opted[ctx->device & 63]) {
        JGPT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solo));
        opted[ctx->device & 63] = true;
    }
    // As many row groups as stay resident at once, every one with the same number of row tiles where that goes: a CTA keeps its weights
    // over its row tiles, and a second round of CTAs would fetch theirs behind the wait.
    const int cols = (N + NT * 8 - 1) / (NT * 8) * nb, row_tiles = (M + kRows - 1) / kRows;
    int groups = std::min(row_tiles, std::max(1, per_sm<S, NT>() * ctx->sm_count / cols));
    const int per_group = (row_tiles + groups - 1) / groups;
    groups = (row_tiles + per_group - 1) / per_group;
    // A launch of at most one CTA per SM that moves in early, while the previous kernel holds most SMs, would be packed onto the few
    // with room.  More than this and the attention's CTAs could not move in beside it in turn.
    const size_t smem = (fuse.pdl & 1) && cols * groups <= ctx->sm_count ? solo : 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(cols / nb), (unsigned)groups, (unsigned)nb), cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem, cfg.stream = ctx->stream, cfg.attrs = attr, cfg.numAttrs = fuse.pdl & 1;
    JGPT_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, A, b, M, K, N, rowsel, fuse, pa));
    return JGPT_OK;
}

template <int NT, int KIND, int MAX>
static int32_t launch_s(int s, Ctx *ctx, const float *A, const Batch &b, int nb, int M, int K, int N, const int *rowsel, const Fuse &fuse, const PagedAppendArgs &pa) {
    if (s <= 1) return launch_t<1, NT, KIND>(ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    if (s <= 2) return launch_t<2, NT, KIND>(ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    if (s <= 3) return launch_t<3, NT, KIND>(ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    if (s <= 4) return launch_t<4, NT, KIND>(ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    if constexpr (MAX > 4) {
        if (s <= 6) return launch_t<6, NT, KIND>(ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
        return launch_t<8, NT, KIND>(ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    }
    return fail(JGPT_ERR_UNSUPPORTED, "gemm_rows: K=%d", K);
}

int32_t launch(Kind kind, Ctx *ctx, const float *A, const Batch &b, int nb, int M, int K, int N, const int *rowsel, const Fuse &fuse_in,
               const PagedAppendArgs &pa) {
    JGPT_REQUIRE(shape_ok(kind, K) && M > 0 && nb >= 1 && nb <= 3 && (kind != NORM_SWIGLU || N % 32 == 0), JGPT_ERR_UNSUPPORTED,
                 "gemm_rows: unsupported shape M=%d K=%d N=%d", M, K, N);
    Fuse fuse = fuse_in;
#ifdef JGPT_B200_DECODE_TRACE
    fuse.timeline = timeline_next();
#endif
    const int s = (k_steps(K) + kWarps - 1) / kWarps;
    if (kind == NORM) return launch_s<4, NORM, kMaxSteps32>(s, ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    if (kind == NORM_SWIGLU) return launch_s<4, NORM_SWIGLU, kMaxSteps32>(s, ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    if (kind == NORM_PAGED) {
        JGPT_REQUIRE(nb == 3 && N == pa.H * 16, JGPT_ERR_UNSUPPORTED, "gemm_rows: paged products of %d columns, %d heads", N, pa.H);
        return launch_s<4, NORM_PAGED, kMaxSteps32>(s, ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
    }
    return launch_s<2, RESIDUAL, kMaxSteps16>(s, ctx, A, b, nb, M, K, N, rowsel, fuse, pa);
}

}  // namespace rows
}  // namespace jgpt
