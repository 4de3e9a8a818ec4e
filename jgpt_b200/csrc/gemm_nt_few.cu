// C[M, N] = A[M, K] . W[N, K]^T in bf16 for at most 32 rows and weights that the SMs' shared memory holds at once: most products of a
// decode step, links of a chain of launches.
//
// What bounds them is the time from the end of the launch in front to their own end.  A CTA's whole weight slice (8, 16 or 32 columns)
// is requested before the wait, its rows at once behind it, so that what is left is one trip to L2, the products and one reduction over
// the eight warps; no cluster, and a barrier per group of rows instead of one per k tile.
//
// The sums are those of gemm_nt.cu, bit for bit, so that a model's tokens do not depend on which kernel ran: a warp has the same 16 of
// every 128 k, the parts into which that kernel would cut k are summed for themselves, warps are added in order, then parts.
//
// Against the ring of gemm_nt.cu (128-wide k tiles, a barrier each, parts of k in clusters of up to eight CTAs), layered model of width 1024,
// prompts of 200 tokens and 24 steps: one row 6.71 -> 5.95 ms, 16 rows 8.47 -> 7.60, 30 rows 10.34 -> 9.55.
#include "gemm_nt.cuh"

#include <algorithm>

#include "ptx.cuh"

namespace jgpt {
namespace nt {

constexpr int kWarps = 8, kTile = 128;  // k of a tile, 16 of them a warp's
__host__ __device__ constexpr int few_pitch(int NT) { return NT == 1 ? 8 : 8 * NT + 8; }  // floats of a row of partial sums: no bank conflicts

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Bytes of a k tile of n rows of 256 bytes, 16-byte chunk c of row r at c ^ (r & 7): a line of memory stays a line of shared memory, and the
// eight rows of an ldmatrix do not meet in a bank.
__host__ __device__ constexpr int few_tile_bytes(int n) { return n * kTile * 2; }
__device__ __forceinline__ int few_chunk(int r, int c) { return r * kTile * 2 + (c ^ (r & 7)) * 16; }

// MT: row tiles of 16, NT: column tiles of 8.  The code is kept short, rolled loops and every part of it once.  A form of the same sums with
// the loops unrolled, rows in registers and cursors over the parts took 2.6 us longer per launch inside a decode step, where a
// dozen different kernels follow one another, all of it between the rows' arrival and the reduction.
template <int MT, int NT, int EPI>
__global__ void __launch_bounds__(32 * kWarps, 2) gemm_nt_few_kernel(const Problem P, int per_seg, int log_parts, int group, int pdl) {
    constexpr int BM = 16 * MT, BN = 8 * NT, PITCH = few_pitch(NT);
    extern __shared__ __align__(128) uint8_t few_smem[];  // weight tiles of all k; two groups of row tiles; the partial sums (over both with one part)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, c16 = tid & 15, r16 = tid >> 4;
    const int parts = 1 << log_parts, K = P.K, nk = (K + kTile - 1) / kTile;
    const int seg = P.seg_n < P.N ? blockIdx.x / per_seg : 0, n0 = seg * P.seg_n + (blockIdx.x - seg * per_seg) * BN, n_end = min(P.N, (seg + 1) * P.seg_n), cn = seg * P.c_seg;
    uint8_t *rows_smem = few_smem + nk * few_tile_bytes(BN);
    float *partials = reinterpret_cast<float *>(parts > 1 ? rows_smem + min(nk, 2 * group) * few_tile_bytes(BM) : few_smem);  // [parts][kWarps][BM][PITCH]
    if (pdl & 2) griddep_launch_dependents();
    {
        const int r0 = r16 % BN;  // with eight columns the upper half of the threads has the next k tile
        const __nv_bfloat16 *W = reinterpret_cast<const __nv_bfloat16 *>(P.W), *from = W + (size_t)(n0 + r0) * P.ldw + c16 * 8;
#pragma unroll 1
        for (int kt = r16 / BN; kt < nk; kt += BN < 16 ? 2 : 1) {
#pragma unroll
            for (int i = 0; i < (BN + 15) / 16; i++) {
                const int r = r0 + 16 * i;
                const bool ok = n0 + r < n_end && kt * kTile + c16 * 8 < K;
                cp_async16(few_smem + kt * few_tile_bytes(BN) + few_chunk(r, c16), ok ? from + (size_t)(16 * i) * P.ldw + kt * kTile : W, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int own_n = n0 + tid % BN;  // the column of all of this thread's results
    const float bias = P.bias && own_n < n_end ? __ldg(P.bias + own_n) : 0.f;
    const int M = P.M, m0 = blockIdx.y * BM;
    if (pdl & 1) griddep_wait();

    // the rows that this thread brings pieces of; what lies past M is computed on zeros and dropped
    const __nv_bfloat16 *A = reinterpret_cast<const __nv_bfloat16 *>(P.A) + min(seg, P.a_cap) * P.a_seg + c16 * 8, *row[MT];
#pragma unroll
    for (int i = 0; i < MT; i++) {
        const int m = m0 + 16 * i + r16;
        row[i] = m < M ? A + (size_t)(P.rowsel ? P.rowsel[m] : m) * P.lda : nullptr;
    }
    float acc[MT][NT][4] = {};
    int part = 0, part_end = nk >> log_parts, filled = 0, ahead = 0, left = 0;  // k tiles whose rows are on their way; the group they go to; tiles left in the present one
    const uint8_t *x = rows_smem;
#pragma unroll 1
    for (int kt = -1; kt < nk; kt++) {
        if (left == 0) {  // a group of rows is through, or both are empty
            if (kt > 0) __syncthreads();
            const int end = min(nk, filled + group);
#pragma unroll 1
            for (uint8_t *to = rows_smem + ahead * group * few_tile_bytes(BM); filled < end; filled++, to += few_tile_bytes(BM)) {
#pragma unroll
                for (int i = 0; i < MT; i++) {
                    const bool ok = row[i] && filled * kTile + c16 * 8 < K;
                    cp_async16(to + few_chunk(16 * i + r16, c16), ok ? row[i] + filled * kTile : A, ok);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            ahead ^= 1;
            if (kt < 0) continue;
            left = group, x = rows_smem + ahead * group * few_tile_bytes(BM);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
        }
        const uint8_t *w = few_smem + kt * few_tile_bytes(BN);
        uint32_t a[MT][4], b[(NT + 1) / 2][4];
#pragma unroll
        for (int i = 0; i < MT; i++) ldmatrix_x4(a[i], x + few_chunk(16 * i + (((lane >> 3) & 1) << 3) + (lane & 7), 2 * warp + (lane >> 4)));
#pragma unroll
        for (int j = 0; j < (NT + 1) / 2; j++)
            ldmatrix_x4(b[j], w + few_chunk((16 * j + ((lane >> 4) << 3) + (lane & 7)) % BN, 2 * warp + ((lane >> 3) & 1)));
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int j = 0; j < NT; j++) mma_bf16_16816(acc[i][j], a[i][0], a[i][1], a[i][2], a[i][3], b[j >> 1][(j & 1) * 2], b[j >> 1][(j & 1) * 2 + 1]);
        left--, x += few_tile_bytes(BM);
        if (kt + 1 < part_end) continue;
        if (parts == 1) __syncthreads();  // the partial sums lie over the tiles
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int j = 0; j < NT; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    *reinterpret_cast<float2 *>(partials + ((part * kWarps + warp) * BM + 16 * i + 8 * h + g) * PITCH + 8 * j + 2 * t) = make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
                    acc[i][j][2 * h] = acc[i][j][2 * h + 1] = 0.f;
                }
        part++, part_end = (part + 1) * nk >> log_parts;
    }
    __syncthreads();
    auto total = [&](int r, int c) {
        float sum = 0.f;
#pragma unroll 1
        for (int p = 0; p < parts; p++) {
            float s = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; w++) s += partials[((p * kWarps + w) * BM + r) * PITCH + c];
            sum = p ? sum + s : s;
        }
        return sum;
    };
    if constexpr (EPI == EPI_GATE) {  // 16 columns of the gate, the linear part's behind them
        for (int e = tid; e < BM * 16; e += 32 * kWarps) {
            const int r = e >> 4, c = e & 15, n = n0 + c;
            if (m0 + r < M && n + 16 < P.N)
                reinterpret_cast<__nv_bfloat16 *>(P.C)[(size_t)(m0 + r) * P.ldc + n / 32 * 16 + c] = __float2bfloat16(activate<true>(P.act, 0.f, 0.f, total(r, c)) * total(r, c + 16));
        }
    } else {
#pragma unroll 1
        for (int e = tid; e < BM * BN; e += 32 * kWarps) {
            const int r = e / BN;
            if (m0 + r < M && own_n < n_end) store_sum<EPI>(P, (size_t)(m0 + r) * P.ldc + own_n + cn, own_n, total(r, e % BN), bias);
        }
    }
}

static int few_tiles(const Problem &p) { return (p.K + kTile - 1) / kTile; }
static size_t few_smem_bytes(int MT, int nt, int nk, int parts, int group) {
    const size_t tiles = (size_t)nk * few_tile_bytes(8 * nt) + (size_t)std::min(nk, 2 * group) * few_tile_bytes(16 * MT), partials = sizeof(float) * parts * kWarps * 16 * MT * few_pitch(nt);
    return parts > 1 ? tiles + partials : std::max(tiles, partials);
}

template <int MT, int NT, int EPI>
static int32_t few_launch(const Problem &p, int parts, int pdl, cudaStream_t st) {
    auto kern = gemm_nt_few_kernel<MT, NT, EPI>;
    const int nk = few_tiles(p);
    int group = nk;  // all rows at once, or in groups of which two fit
    if (few_smem_bytes(MT, NT, nk, parts, group) > kFewSmem)
        for (group = (nk + 1) / 2; group > 1 && few_smem_bytes(MT, NT, nk, parts, group) > kFewSmem;) group--;
    const size_t smem = few_smem_bytes(MT, NT, nk, parts, group);
    static thread_local int set_for = -1;  // the opt-in to more than 48 KiB, once per device
    int dev = 0;
    JGPT_CUDA_TRY(cudaGetDevice(&dev));
    if (set_for != dev) {
        JGPT_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFewSmem));
        set_for = dev;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)p.column_tiles(8 * NT), (unsigned)((p.M + 16 * MT - 1) / (16 * MT)));
    cfg.blockDim = dim3(32 * kWarps), cfg.dynamicSmemBytes = smem, cfg.stream = st, cfg.attrs = attr, cfg.numAttrs = pdl & 1 ? 1u : 0u;
    JGPT_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p, (p.segment_cols() + 8 * NT - 1) / (8 * NT), parts == 8 ? 3 : parts >> 1, group, pdl));
    return JGPT_OK;
}

// Column tiles of 8 per CTA, 0: not for this kernel.  Tiles as wide as three SMs in four stay busy: every CTA reads all rows.  What a CTA's
// memory does not hold (two of 112 KB share an SM) streams through the ring, and so do products of many CTAs with long slices: a CTA that
// finds no room requests its slice when another leaves, and multiplies nothing until all of it is there, where the ring begins with its
// first k tile.  Launches by themselves, four rows, us here and in the ring: k 1024, 264 CTAs 5.9 and 7.5; k 1536, 240 CTAs 7.1 and 7.9, 580 CTAs
// 11.5 and 9.6, 2000 CTAs 29 and 22; k 512, 1000 CTAs (slices of 32 KB, four on an SM) 9.9 and 12.1.  It is not the bytes of the rows that
// are there: 528 CTAs of k 2048 take 13.7 and 10.6 with four rows, 17.1 and 12.4 with 24.
// The line itself is tuned, CTAs times k times row tiles.  Prompts of 16 tokens and 24 steps, ms, with it, with two CTAs per SM for a line, with none,
// all in the ring: width 512, 4 rows 4.72, 5.08, 4.75, 5.53; width 1536, 4 rows 7.40, 7.54, 7.62, 7.76, 17 rows 9.16, 9.14, 9.76, 9.21; width 2048,
// 4 rows 8.91, 8.92, 9.55, 8.99, 24 rows 11.44, 11.45, 12.94, 11.48; width 1024, 1 to 32 rows, the first three within 1.5 %, the ring 8-14 % more.
static int few_columns(const Ctx *ctx, const Problem &p, Epilogue epi, int parts) {
    if (p.M > kFewRows || p.grp.tiles) return 0;
    const int nk = few_tiles(p), MT = p.M <= 16 ? 1 : 2;
    auto fits = [&](int nt) { return few_smem_bytes(MT, nt, nk, parts, std::min((nk + 1) / 2, 4 / MT)) <= kFewSmem; };
    int nt = 1;
    if (epi == EPI_GATE) nt = 4;
    else
        for (int w : {2, 4})
            if (4 * p.column_tiles(8 * w) >= 3 * ctx->sm_count && fits(w)) nt = w;
    return fits(nt) && (long long)MT * p.column_tiles(8 * nt) * p.K <= 625000 ? nt : 0;
}

template <int EPI>
static int32_t few_dispatch(const Problem &p, int nt, int parts, int pdl, cudaStream_t st) {
    if constexpr (EPI != EPI_GATE) {
        if (nt == 1) return p.M <= 16 ? few_launch<1, 1, EPI>(p, parts, pdl, st) : few_launch<2, 1, EPI>(p, parts, pdl, st);
        if (nt == 2) return p.M <= 16 ? few_launch<1, 2, EPI>(p, parts, pdl, st) : few_launch<2, 2, EPI>(p, parts, pdl, st);
    }
    return p.M <= 16 ? few_launch<1, 4, EPI>(p, parts, pdl, st) : few_launch<2, 4, EPI>(p, parts, pdl, st);
}

bool launch_bf16_few(const Ctx *ctx, const Problem &p, Epilogue epi, int parts, int pdl, cudaStream_t st, int32_t *rc) {
    const int nt = few_columns(ctx, p, epi, parts);
    if (!nt) return false;
    switch (epi) {
        case EPI_STORE: *rc = few_dispatch<EPI_STORE>(p, nt, parts, pdl, st); return true;
        case EPI_ADD_F32: *rc = few_dispatch<EPI_ADD_F32>(p, nt, parts, pdl, st); return true;
        case EPI_SCALE_F32: *rc = few_dispatch<EPI_SCALE_F32>(p, nt, parts, pdl, st); return true;
        case EPI_GATE: *rc = few_dispatch<EPI_GATE>(p, nt, parts, pdl, st); return true;
        case EPI_ACT: *rc = few_dispatch<EPI_ACT>(p, nt, parts, pdl, st); return true;
        case EPI_ACT_SOME: *rc = few_dispatch<EPI_ACT_SOME>(p, nt, parts, pdl, st); return true;
    }
    return false;
}

}  // namespace nt
}  // namespace jgpt
