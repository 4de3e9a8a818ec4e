// sampleNextToken on the device (src/main/java/com/veles/llm/jgpt/model/GptAutoregressiveGenerator.java:208-286), one CTA per
// row, the arithmetic of the reference in its own order so that the token is the one the host routine picks: logits /
// temperature; keep the top_k by (logit descending, index ascending), the rest -inf; maximum; e = (float)exp((double)(z - max));
// sum and running CDF accumulated in fp32 in INDEX order by one thread (a float sum is not associative: a parallel reduction
// would move CDF boundaries); first index with u <= cdf, else the last one.  The uniform draw u is supplied per row (the
// reference draws from an unseeded ThreadLocalRandom).
//
// The serial chain bounds it, so the chain is made short and everything else runs beside it.  The top_k-th element is found by a
// radix selection over order-preserving keys (three passes of 11, 11 and 10 bits); up to kListMax kept elements are then
// compacted in index order - a dropped element is a zero in either sum and changes neither - which leaves top_k additions out of
// shared memory, twice.  A search over the row per kept element and both sums over the whole vocabulary out of global memory
// took 1471 us for 8 rows of 8000 logits at top_k 40; a decode step of 8 sampled rows (12 layers of 384) went from 1.71 to
// 0.32 ms with this form.
#include "decoder.cuh"

namespace jgpt {

constexpr int kThreads = 1024, kWarps = kThreads / 32;
constexpr int kBins = 2048;
constexpr int kListMax = 1024;                 // more kept elements: the chain runs over the whole row
constexpr size_t kRowBytesMax = 192 * 1024;    // longer rows stay in the global work area
constexpr int kBatch = 16;

// A larger key comes earlier in (value descending); the two zeros share a key, as they compare equal.
__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t b = __float_as_uint(v + 0.f);
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}

// s = ((e[0] + e[1]) + e[2]) + ...; the loads of the next batch are in flight during the additions of this one.
// FIND: the first index whose running sum reaches u, n when none does (e >= 0: the sums never fall).
template <bool FIND>
__device__ __forceinline__ float chain(const float *e, int n, float u, int *at) {
    float s = 0.f, cur[kBatch];
    const int full = n / kBatch * kBatch;
#pragma unroll
    for (int q = 0; q < kBatch; q++) cur[q] = q < full ? e[q] : 0.f;
    for (int i = 0; i < full; i += kBatch) {
        float nxt[kBatch];
        const int ahead = i + kBatch < full ? i + kBatch : 0;
#pragma unroll
        for (int q = 0; q < kBatch; q++) nxt[q] = e[ahead + q];
#pragma unroll
        for (int q = 0; q < kBatch; q++) s += cur[q], cur[q] = s;
        if (FIND && u <= s) {
            int first = 0;
#pragma unroll
            for (int q = kBatch - 1; q >= 0; q--) first = u <= cur[q] ? q : first;
            *at = i + first;
            return s;
        }
#pragma unroll
        for (int q = 0; q < kBatch; q++) cur[q] = nxt[q];
    }
    for (int i = full; i < n; i++) {
        s += e[i];
        if (FIND && u <= s) {
            *at = i;
            return s;
        }
    }
    if (FIND) *at = n;
    return s;
}

__global__ void __launch_bounds__(kThreads) sample_kernel(const float *__restrict__ logits, float *__restrict__ work, int V, float temperature,
                                                          int top_k, const float *u01, int *__restrict__ out, const HostMirror host, int row_in_smem) {
    extern __shared__ float smem_row[];
    __shared__ int hist[kBins];
    __shared__ int list_i[kListMax];
    __shared__ float list_e[kListMax];
    __shared__ int w_gt[kWarps], w_eq[kWarps];
    __shared__ float w_mx[kWarps];
    __shared__ int s_bin, s_above;
    __shared__ float s_sum;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *row = logits + (size_t)blockIdx.x * V;
    float *z = row_in_smem ? smem_row : work + (size_t)blockIdx.x * V;
    float mx = -INFINITY;
    bool bad = false;
    const float u = tid == 0 ? u01[blockIdx.x] : 0.f;  // perhaps from the host's memory: requested first, used last
    auto leave = [&](int tok) {
        out[blockIdx.x] = tok;
        if (host.next) host.next[blockIdx.x] = tok;
        if (host.next && blockIdx.x == 0) *host.status = *host.status_dev;
    };
    for (int i0 = tid; i0 < V; i0 += 8 * kThreads) {
        float v[8];
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = i0 + q * kThreads < V ? row[i0 + q * kThreads] : -INFINITY;
#pragma unroll
        for (int q = 0; q < 8; q++) {
            if (temperature != 1.0f) v[q] = v[q] / temperature;
            bad |= isnan(v[q]);
            mx = fmaxf(mx, v[q]);
            if (i0 + q * kThreads < V) z[i0 + q * kThreads] = v[q];
        }
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (lane == 0) w_mx[warp] = mx;
    bad = __syncthreads_or(bad);  // z and w_mx are visible behind it
    mx = w_mx[0];
#pragma unroll
    for (int w = 1; w < kWarps; w++) mx = fmaxf(mx, w_mx[w]);
    // a NaN, or a maximum that is not finite, makes every sum a NaN: no index is reached and the last one is taken
    if (bad || !isfinite(mx)) {
        if (tid == 0) leave(V - 1);
        return;
    }
    const bool some = top_k > 0 && top_k < V;
    uint32_t thr = 0;  // key of the top_k-th element
    int need = 0;      // how many elements with that key are kept, the first ones by index
    if (some) {
        uint32_t mask = 0;
        need = top_k;
#pragma unroll 1
        for (int pass = 0; pass < 3; pass++) {
            const int shift = pass == 0 ? 21 : (pass == 1 ? 10 : 0), bins = pass == 2 ? 1024 : 2048;
            hist[tid] = 0, hist[tid + kThreads] = 0;
            __syncthreads();
            for (int i = tid; i < V; i += kThreads) {
                const uint32_t k = order_key(z[i]);
                if ((k & mask) == thr) atomicAdd(&hist[(k >> shift) & (bins - 1)], 1);
            }
            __syncthreads();
            // thread t stands for the bins bins - 1 - 2 t and the one below: a running count from the top finds the place
            const int hi = bins - 1 - 2 * tid;
            const int c0 = hi >= 0 ? hist[hi] : 0, c = c0 + (hi >= 1 ? hist[hi - 1] : 0);
            int upto = c;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(0xffffffffu, upto, off);
                if (lane >= off) upto += o;
            }
            if (lane == 31) w_gt[warp] = upto;
            __syncthreads();
            int before = lane < warp ? w_gt[lane] : 0;
            before = __reduce_add_sync(0xffffffffu, before) + upto - c;
            if (before < need && need <= before + c) {
                const bool first = need <= before + c0;
                s_bin = first ? hi : hi - 1, s_above = first ? before : before + c0;
            }
            __syncthreads();
            thr |= (uint32_t)s_bin << shift, mask |= (uint32_t)(bins - 1) << shift;
            need -= s_above;
        }
    }
    // Two sweeps in index order, a contiguous part per warp: counts of the elements above and at the threshold, then every kept
    // element's place.
    const bool list = some && top_k <= kListMax;
    const int per = (V + kWarps * 32 - 1) / (kWarps * 32) * 32, i_first = warp * per, i_end = min(V, i_first + per);
    int gt = 0, eq = 0;
    if (some) {
        for (int i = i_first + lane; i - lane < i_end; i += 32) {
            const uint32_t k = i < i_end ? order_key(z[i]) : 0u;
            gt += __popc(__ballot_sync(0xffffffffu, i < i_end && k > thr));
            eq += __popc(__ballot_sync(0xffffffffu, i < i_end && k == thr));
        }
        __syncthreads();  // w_gt was read above
        if (lane == 0) w_gt[warp] = gt, w_eq[warp] = eq;
        __syncthreads();
        gt = __reduce_add_sync(0xffffffffu, lane < warp ? w_gt[lane] : 0);
        eq = __reduce_add_sync(0xffffffffu, lane < warp ? w_eq[lane] : 0);
    }
    const unsigned below = (1u << lane) - 1u;
    for (int i = i_first + lane; i - lane < i_end; i += 32) {
        const bool in = i < i_end;
        const float v = in ? z[i] : 0.f;
        bool keep = in;
        int at = 0;
        if (some) {
            const uint32_t k = order_key(v);
            const bool above = in && k > thr, level = in && k == thr;
            const unsigned b_gt = __ballot_sync(0xffffffffu, above), b_eq = __ballot_sync(0xffffffffu, level);
            const int my_eq = eq + __popc(b_eq & below);
            at = gt + __popc(b_gt & below) + min(my_eq, need);
            keep = above || (level && my_eq < need);
            gt += __popc(b_gt), eq += __popc(b_eq);
        }
        const float e = keep ? (float)exp((double)(v - mx)) : 0.f;
        if (list) {
            if (keep) list_i[at] = i, list_e[at] = e;
        } else if (in) {
            z[i] = e;
        }
    }
    __syncthreads();
    float *e = list ? list_e : z;
    const int n = list ? top_k : V;
    if (tid == 0) s_sum = chain<false>(e, n, 0.f, nullptr);
    __syncthreads();
    const float sum = s_sum;
    for (int i = tid; i < n; i += kThreads) e[i] = e[i] / sum;
    __syncthreads();
    if (tid == 0) {
        int at;
        chain<true>(e, n, u, &at);
        int tok = at == n ? V - 1 : (list ? list_i[at] : at);
        if (list && list_i[0] != 0 && u <= 0.f) tok = 0;  // index 0, dropped: its running sum is 0
        leave(tok);
    }
}

// work: [rows, vocab], used by rows that do not fit shared memory.
int32_t launch_sample(const float *logits, float *work, int rows, int vocab, const SampleSpec &spec, const float *u01_dev, int *next_dev,
                      const HostMirror &host, cudaStream_t st) {
    const size_t row = sizeof(float) * (size_t)vocab;
    const bool in_smem = row <= kRowBytesMax;
    static bool opted[64] = {};
    int dev = 0;
    JGPT_CUDA_TRY(cudaGetDevice(&dev));
    if (!opted[dev & 63]) {
        JGPT_CUDA_TRY(cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowBytesMax));
        opted[dev & 63] = true;
    }
    sample_kernel<<<rows, kThreads, in_smem ? row : 0, st>>>(logits, work, vocab, spec.temperature, spec.top_k, u01_dev, next_dev, host, in_smem);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}

}  // namespace jgpt
