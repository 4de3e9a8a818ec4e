// Single-query decode attention over the paged fp16 K/V store, optionally fused with the append
// of the step's new token.
//
// Work item = (layer, sequence, head group, chunk of `chunk_blocks` KV blocks).  A CTA owns a
// ring of shared-memory stages; one producer warp walks the block table and fetches, per KV
// block, the contiguous [head group][K tile | V tile] slab with ONE bulk async copy (TMA engine,
// cp.async.bulk + mbarrier complete_tx).  At dhead 16 and a multiple of four heads a consumer warp owns four
// of them and runs their products on the tensor cores with high + low operands; at other head sizes and counts, and for
// small launches of several layers, consumer threads are (head, token-in-block) pairs: a thread scores its token against q (fp32 FMA), keeps a private
// online-softmax state (m, l, o[DH]) and, at the end of the chunk, the 16 lanes of a head merge their
// states with warp shuffles.  Chunks of one sequence are merged by the last CTA to arrive (atomic ticket, no
// waiting), through a small fp32 scratch buffer.
//
// The kernel is HBM-bound (about 1 FLOP per byte at dhead 16): what matters is bytes in flight
// per SM (stages x slab bytes x resident CTAs) and few, large, 16-byte-aligned transactions.
#include "common.cuh"
#include "ptx.cuh"

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <map>
#include <mutex>
#include <tuple>

namespace jgpt {

struct DecodeParams {
    __half *kv;
    const int *table;
    const float2 *rope;
    const float *q, *k_new, *v_new;
    float *out;
    const int *seq_ids, *rope_pos, *lens;
    float *partials;
    int *tickets;
    int *status;
    int n, H, HG, n_hg, layer0, n_layers, mbs, n_blocks, max_seqs, max_positions;
    int chunk_blocks, max_chunks, n_items, stages, max_len;
    float scale_log2e;
    // Launch overlap (programmatic dependent launch).  0: ordinary launch.  1: the launch may start while the previous
    // kernel on the stream drains; everything that reads memory waits for that kernel first (only the barrier set-up
    // runs ahead).  2: additionally the producer warp runs ahead -- lengths, block-table entries and the first K/V
    // slabs are fetched before the previous kernel has finished -- which is only legal when that kernel does not
    // write the K/V store of these layers, the block tables or the index arrays (the caller's promise).
    int overlap;
    int stream_hint;  // 1: K/V slabs are fetched with an evict-first L2 policy
    // 1: the launch is made of clusters of max_chunks CTAs, the chunks of one (layer, sequence, head group); their
    // partial softmax states are merged through distributed shared memory by the CTA of chunk 0 instead of through
    // global scratch and an arrival counter.  Every thread of the cluster passes two cluster barriers, whatever its path.
    int cluster;
    int dynamic;    // 1: CTAs claim work items from counters[0]; 0: item = blockIdx.x + k * gridDim.x
    int *counters;  // [0] next item, [1] CTAs that have finished (the last one resets both)
#ifdef JGPT_B200_DECODE_TRACE
    long long *trace;  // experiments only: 8 timestamps per CTA (never compiled into the shipped library)
    Timeline timeline;
#endif
};

constexpr int kMaxStages = 8;
constexpr int kItemRing = 4;

// Loads one token row of DH halfs from a shared-memory tile into fp32 registers.  For DH = 16
// (two 16-byte halves per row) the order of the two loads alternates with bit 2 of the token
// index so the 8 lanes of a quarter-warp hit 8 distinct 16-byte bank groups; a lane with that bit
// set therefore receives the row with its two halves exchanged (dims 8..15 first).  Callers keep q
// and the accumulator in the same exchanged order (see swap_halves) instead of selecting per load.
template <int DH>
__device__ __forceinline__ void load_row(const unsigned char *tile, int t, float (&r)[DH]) {
    if constexpr (DH == 16) {
        const int sw = (t >> 2) & 1;
        const uint4 lo = *reinterpret_cast<const uint4 *>(tile + t * 32 + sw * 16);
        const uint4 hi = *reinterpret_cast<const uint4 *>(tile + t * 32 + (sw ^ 1) * 16);
        const __half2 *pl = reinterpret_cast<const __half2 *>(&lo), *ph = reinterpret_cast<const __half2 *>(&hi);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 f = __half22float2(pl[i]), g = __half22float2(ph[i]);
            r[2 * i] = f.x, r[2 * i + 1] = f.y, r[8 + 2 * i] = g.x, r[8 + 2 * i + 1] = g.y;
        }
    } else if constexpr (DH >= 8) {
#pragma unroll
        for (int c = 0; c < DH / 8; c++) {
            const uint4 a = *reinterpret_cast<const uint4 *>(tile + t * (DH * 2) + c * 16);
            const __half2 *pa = reinterpret_cast<const __half2 *>(&a);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 f = __half22float2(pa[i]);
                r[c * 8 + 2 * i] = f.x, r[c * 8 + 2 * i + 1] = f.y;
            }
        }
    } else {
        const uint2 a = *reinterpret_cast<const uint2 *>(tile + t * (DH * 2));
        const __half2 *pa = reinterpret_cast<const __half2 *>(&a);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float2 f = __half22float2(pa[i]);
            r[2 * i] = f.x, r[2 * i + 1] = f.y;
        }
    }
}

// Exchanges the two 8-element halves of a 16-element register row on lanes whose rows arrive exchanged.
template <int DH>
__device__ __forceinline__ void swap_halves(float (&r)[DH], int t) {
    if constexpr (DH == 16) {
        if ((t >> 2) & 1) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float x = r[j];
                r[j] = r[8 + j];
                r[8 + j] = x;
            }
        }
    }
}

// Sum v[0..DH) over the 16 lanes of a half-warp.  On return lane t holds, in v[i], the total of
// dimension (i*16 + t) for DH >= 16, or in v[0] the total of dimension (t % DH) for DH < 16.
template <int DH>
__device__ __forceinline__ void halfwarp_reduce_scatter(float (&v)[DH], int t) {
    if constexpr (DH >= 16) {
#pragma unroll
        for (int g = 0; g < DH / 16; g++) {
            float a8[8], a4[4], a2[2];
            const bool b8 = t & 8, b4 = t & 4, b2 = t & 2, b1 = t & 1;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float keep = b8 ? v[g * 16 + 8 + j] : v[g * 16 + j];
                const float send = b8 ? v[g * 16 + j] : v[g * 16 + 8 + j];
                a8[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float keep = b4 ? a8[4 + j] : a8[j];
                const float send = b4 ? a8[j] : a8[4 + j];
                a4[j] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float keep = b2 ? a4[2 + j] : a4[j];
                const float send = b2 ? a4[j] : a4[2 + j];
                a2[j] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
            }
            const float keep = b1 ? a2[1] : a2[0];
            const float send = b1 ? a2[0] : a2[1];
            v[g] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        }
    } else {
        float mine = 0.f;
#pragma unroll
        for (int d = 0; d < DH; d++) {
            float x = v[d];
#pragma unroll
            for (int off = 8; off >= 1; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if (d == (t % DH)) mine = x;
        }
        v[0] = mine;
    }
}

// Head-group cap: slab <= 24 KiB and at most 30 heads (480 consumer threads + the producer warp).
template <int DH>
constexpr int max_head_group() { return (384 / DH) < 30 ? (384 / DH) : 30; }

// Consumer threads of a CTA: (head, token) pairs, or a warp per four heads with the products of dhead 16 on the tensor cores.
template <bool MMA>
__host__ __device__ constexpr int consumer_threads(int HG) {
    return MMA ? HG / 4 * 32 : (kBlockTokens * HG + 31) / 32 * 32;
}

template <int DH, bool FUSED, bool MMA = DH == 16>
__global__ void __launch_bounds__(consumer_threads<MMA>(max_head_group<DH>()) + 32, MMA ? 3 : 2) attn_decode_kernel(const DecodeParams P) {
    constexpr int BT = kBlockTokens;
    constexpr int TILE = BT * DH * 2;    // bytes of one K (or V) tile
    constexpr int HEAD_BYTES = 2 * TILE; // K tile | V tile
    constexpr int OPL = DH >= 16 ? DH / 16 : 1;  // output dims held per lane after the merge
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages];
    __shared__ int s_last;
    __shared__ int s_abort_mem;
    constexpr int kMaxHG = (384 / DH) < 30 ? (384 / DH) : 30;  // == max_head_group<DH>()
    __shared__ float cl_part[kMaxHG * (DH + 2)];  // this CTA's partial (m, l, o[DH]) per head, cluster mode
    // Dynamic mode: the producer warp claims work items from a global counter and hands their ids to the
    // consumers through this small ring, so a resident CTA keeps its copy pipeline full across items and the
    // launch has no wave quantisation (items are a few KV blocks each, claimed as CTAs become free).
    __shared__ int item_ring[kItemRing];
    __shared__ uint64_t item_full[kItemRing], item_empty[kItemRing];
    volatile int *s_abort = &s_abort_mem;

    const int tid = threadIdx.x;
#ifdef JGPT_B200_DECODE_TRACE
    long long tr_gt0 = 0, tr_c0 = clock64(), tr_c1 = 0, tr_c2 = 0, tr_c3 = 0, tr_c4 = 0;
    timeline_in(P.timeline);
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(tr_gt0));
#endif
    const int n_cons = consumer_threads<MMA>(P.HG);  // padded to whole warps
    const int n_cons_warps = n_cons / 32;
    const int stage_bytes = P.HG * HEAD_BYTES;
    const int NS = P.stages;

    if (tid == 0) {
        for (int s = 0; s < NS; s++) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], (uint32_t)n_cons_warps);
        }
        for (int s = 0; s < kItemRing; s++) {
            mbar_init(&item_full[s], 1);
            mbar_init(&item_empty[s], (uint32_t)n_cons_warps);
        }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

#ifdef JGPT_B200_DECODE_TRACE
    tr_c1 = clock64();
#endif
    const bool is_producer = tid >= n_cons;
    // q / k_new / v_new come from the previous kernel on the stream, and the split-K scratch and counters are shared
    // with it: the consumers always wait for it.  The producer touches neither; it waits unless the caller has
    // promised that what it reads (lengths, tables, cached K/V) is not written by that kernel.
    // With overlap 2 the consumers wait later still: right before they read q (see below).
    const bool late_wait = P.overlap == 2;
    if (P.overlap && !(P.overlap == 2 && is_producer) && !(late_wait && !is_producer)) griddep_wait();
#ifdef JGPT_B200_DECODE_TRACE
    if (!late_wait) timeline_at(P.timeline, 1);
#endif
    bool waited = !late_wait || is_producer;
    uint32_t it = 0;  // KV blocks processed so far by this CTA (producer and consumers count alike)
    int stage = 0;    // it % NS, kept incrementally (no integer division in the block loop)
    uint32_t phase = 0;  // (it / NS) & 1
    int next_static = blockIdx.x;
    int rslot = 0, rcount = 0;  // item ring position (each side keeps its own)
    uint32_t rphase = 0;

    if (is_producer) {
        // ---------------- producer warp ----------------
        // Walks its work items, publishes each item id to the consumers and issues one bulk copy per KV block.
        // The next item is prepared while the current one is being copied (claim -> lengths -> block-table
        // entries are three dependent global-memory round trips): the steps are spread over the first copy
        // issues of the current item so their latency never leaves the copy ring empty.
        const int lane = tid & 31;
        const uint64_t l2_stream = l2_policy_evict_first();
        int raw = 0;                 // pending claim (lane 0 holds the atomic's result in dynamic mode)
        int nid = -1, n_i = 0, n_z = 0, n_hg = 0, n_c = 0, n_len = 0, n_seq = 0;  // next item, partly resolved
        int cur_nb = 0, cur_entry = 0, nxt_nb = 0, nxt_entry = 0;
        size_t cur_base = 0, nxt_base = 0;
        auto step_claim = [&]() {
            if (P.dynamic) {
                raw = -1;
                if (lane == 0) raw = atomicAdd(P.counters, 1);
            } else {
                raw = next_static;
                next_static += gridDim.x;
            }
        };
        auto step_resolve = [&]() {  // item id known: publish it, start loading its length and sequence id
            nid = P.dynamic ? __shfl_sync(0xffffffffu, raw, 0) : raw;
            if (nid >= P.n_items) nid = -1;
            if (P.dynamic) {
                if (lane == 0) {
                    if (rcount >= kItemRing && !*s_abort) mbar_wait_bounded(&item_empty[rslot], rphase ^ 1u, P.status, s_abort);
                    item_ring[rslot] = nid;
                    mbar_arrive(&item_full[rslot]);
                }
                rcount++;
                if (++rslot == kItemRing) rslot = 0, rphase ^= 1u;
            }
            if (nid >= 0) {
                int r = nid;
                n_c = r % P.max_chunks, r /= P.max_chunks;
                n_hg = r % P.n_hg, r /= P.n_hg;
                n_i = r % P.n, n_z = r / P.n;
                n_len = P.lens[n_i];
                n_seq = P.seq_ids[n_i];
            }
        };
        auto step_table = [&]() {  // length known: block range of the chunk, start loading its table entries
            nxt_nb = 0, nxt_entry = 0;
            if (nid < 0) return;
            const int len = min(n_len, P.max_len);
            const int nblk = len > 0 ? (len + BT - 1) / BT : 0;
            const int nsplit = (nblk + P.chunk_blocks - 1) / P.chunk_blocks;  // balanced chunks, see the consumers
            const int b0 = n_c < nsplit ? (int)((long long)n_c * nblk / nsplit) : nblk;
            const int b1 = n_c < nsplit ? (int)((long long)(n_c + 1) * nblk / nsplit) : nblk;
            if (b0 >= b1 || n_seq < 0 || n_seq >= P.max_seqs) return;  // empty chunk: the consumers skip it too
            nxt_nb = b1 - b0;
            if (lane < nxt_nb) nxt_entry = P.table[(size_t)n_seq * P.mbs + b0 + lane];
            nxt_base = (((size_t)(P.layer0 + n_z) * P.n_blocks) * P.H + (size_t)n_hg * P.HG) * (size_t)HEAD_BYTES;
        };
        step_claim(), step_resolve(), step_table();
        bool triggered = false;
        while (nid >= 0 && !*s_abort) {
            cur_nb = nxt_nb, cur_entry = nxt_entry, cur_base = nxt_base;
            step_claim();
            // static grids know at once whether another item follows; the work queue only after the claim resolves
            const int nid_after_this = P.dynamic ? 0 : (raw < P.n_items ? raw : -1);
            int pending = 2;  // step_resolve, step_table still to run for the next item
            for (int j = 0; j < cur_nb; j++, it++) {
                // Overlapped launches: once most of this CTA's copies are out -- and no further item is coming -- the next
                // launch on the stream may move in, so that ITS first slabs arrive as this launch's last ones are consumed.
                if (P.overlap && !triggered && nid_after_this < 0 && 5 * j >= 3 * cur_nb) {
                    griddep_launch_dependents();
                    triggered = true;
                }
                int phys = __shfl_sync(0xffffffffu, cur_entry, j);
                if (lane == 0) {
                    if (phys < 0 || phys >= P.n_blocks) {
                        atomicOr(P.status, DEV_STATUS_BAD_BLOCK);
                        phys = 0;
                    }
                    const int s = stage;
                    if (it >= (uint32_t)NS && !*s_abort) mbar_wait_bounded(&empty_bar[s], phase ^ 1u, P.status, s_abort);
                    if (!*s_abort) {
                        mbar_expect_tx(&full_bar[s], (uint32_t)stage_bytes);
                        const unsigned char *src = reinterpret_cast<const unsigned char *>(P.kv) + cur_base +
                                                   (size_t)phys * P.H * (size_t)HEAD_BYTES;
                        if (P.stream_hint) bulk_g2s_hint(smem + (size_t)s * stage_bytes, src, (uint32_t)stage_bytes, &full_bar[s], l2_stream);
                        else bulk_g2s(smem + (size_t)s * stage_bytes, src, (uint32_t)stage_bytes, &full_bar[s]);
                    }
                }
                if (++stage == NS) stage = 0, phase ^= 1u;
                if (pending == 2 && j >= 1) step_resolve(), pending = 1;
                else if (pending == 1 && j >= 3) step_table(), pending = 0;
            }
            if (pending == 2) step_resolve(), pending = 1;
            if (pending == 1) step_table();
        }
        // every copy of this CTA has been issued: at the latest now the next launch on the stream may move in
        if (P.overlap && !triggered) griddep_launch_dependents();
        if (P.cluster) cluster_sync(), cluster_sync();  // the two barriers of the consumers' merge
    } else
    for (;;) {
        // a bounded wait ran out: stop taking work (status word says why).  In cluster mode every warp must still walk
        // through its one item to the cluster barriers; with the abort flag up its waits return at once.
        if (*s_abort && !P.cluster) break;
        int item;
        if (!P.dynamic) {
            item = next_static;
            next_static += gridDim.x;
            if (item >= P.n_items) break;
        } else {
            if (!mbar_wait_bounded(&item_full[rslot], rphase, P.status, s_abort)) break;
            item = item_ring[rslot];
            __syncwarp();
            if ((tid & 31) == 0) mbar_arrive(&item_empty[rslot]);
            if (++rslot == kItemRing) rslot = 0, rphase ^= 1u;
            if (item < 0) break;
        }
        // item -> (z = layer slab, i = sequence row, hg = head group, c = chunk); chunk is fastest.
        int r = item;
        const int c = r % P.max_chunks;
        r /= P.max_chunks;
        const int hg = r % P.n_hg;
        r /= P.n_hg;
        const int i = r % P.n;
        const int z = r / P.n;
        int len = P.lens[i];
        if (len > P.max_len) {
            if (tid == 0) atomicOr(P.status, DEV_STATUS_LEN_OVER_BOUND);
            len = P.max_len;
        }
        const int nblk = len > 0 ? (len + BT - 1) / BT : 0;
        // The sequence's blocks are cut into nsplit chunks of equal size (+-1), none longer than chunk_blocks.
        const int nsplit = (nblk + P.chunk_blocks - 1) / P.chunk_blocks;
        const int b0 = c < nsplit ? (int)((long long)c * nblk / nsplit) : nblk;
        const int b1 = c < nsplit ? (int)((long long)(c + 1) * nblk / nsplit) : nblk;
        const int seq = P.seq_ids[i];
        const bool seq_ok = seq >= 0 && seq < P.max_seqs;
        if (!seq_ok && tid == 0) atomicOr(P.status, DEV_STATUS_BAD_SEQ);
        const size_t row = ((size_t)z * P.n + i) * (size_t)(P.H * DH);  // fp32 row of q / k / v / out
        const int head0 = hg * P.HG;
        const int rp_raw = P.rope_pos[i];
        if (!waited) {
            // Late wait (overlap 2): everything the previous kernel on the stream cannot have written -- lengths, ids,
            // RoPE position -- has been fetched above; q, k_new, v_new and every store come after the wait.
            griddep_wait();
            waited = true;
#ifdef JGPT_B200_DECODE_TRACE
            timeline_at(P.timeline, 1);
#endif
        }

        if (b0 >= b1 || !seq_ok) {
            // Empty chunk.  A sequence without any key (len <= 0) gets a zero output row.
            if ((nblk == 0 || !seq_ok) && c == 0)
                for (int e = tid; e < P.HG * DH; e += n_cons) P.out[row + (size_t)head0 * DH + e] = 0.f;
            if (P.cluster) cluster_sync(), cluster_sync();
            continue;
        }
        const int nb = b1 - b0;
        const size_t layer_base = (size_t)(P.layer0 + z) * P.n_blocks;

        if constexpr (MMA) {
            // ---------------- consumers, tensor-core form (dhead 16) ----------------
            // A warp owns four heads.  Per KV block and head one m16n8k16 product K [16 tok x 16] . Q^T [16 x 8] and one
            // V^T [16 dh x 16 tok] . P^T [16 x 8], K and V^T straight from the staged fp16 tile (ldmatrix: no conversions).  Columns
            // 2 c and 2 c + 1 of Q^T and P^T hold the fp16 high and low part of head c's q and p, so the four products share their B
            // operand and the sum over a column pair keeps fp32-level accuracy; of head i's product only the pair i is used, which
            // sits in the lanes with lane % 4 == i.  Lane (g, t) thus carries the scores of tokens g and g + 8 and the sums of
            // dims g and g + 8 of head t: every lane has work, and maximum, exponentials and rescaling serve four heads at once.
            // A product's unused columns stay unused, so an infinity in one head does not reach another.
            // q is scaled by a power of two per head and p by 2^14, both to keep the low parts clear of fp16's subnormals; the factor
            // cancels in o / l.  p is scaled behind its exponential: a reference 14 below the maximum gives the same factor for one
            // instruction less, but rounds s - m at 14 instead of near 0, 2e-7 of every p.
            // Error against float64 over 64 x 1024 keys (2-norm, fp16-exact K and V), fp32 consumers -> these, for q of 0.2, 1 and 4:
            // 1.5e-7 -> 1.6e-7, 2.3e-7 -> 2.0e-7, 5.0e-7 -> 3.4e-7 (with the reference below the maximum 2.5e-7, 2.9e-7, 3.4e-7).
            // About 95 instructions per 4 heads x 16 tokens where fp32 FMAs on converted rows took 380: one CTA alone was
            // issue-bound at 43 GB/s.
            constexpr float kLift = 16384.f;
            const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
            int rp = rp_raw;
            if (rp < 0 || rp >= P.max_positions) {
                if (tid == 0) atomicOr(P.status, DEV_STATUS_BAD_POSITION);
                rp = 0;
            }
            const float2 *cs = P.rope + (size_t)rp * (DH / 2);
            const int hl = 4 * warp + t4, h = head0 + hl;  // HG is a multiple of four
            auto turned = [](float2 x, float2 w) {  // RoPE with separate roundings
                return make_float2(__fsub_rn(__fmul_rn(x.x, w.x), __fmul_rn(x.y, w.y)), __fadd_rn(__fmul_rn(x.x, w.y), __fmul_rn(x.y, w.x)));
            };
            // column g of the B operand: dims 2 t, 2 t + 1, 2 t + 8, 2 t + 9 of head g / 2, high parts for even g, low parts for odd g
            auto column = [&](float x, float y) {
                const __half2 hi = __floats2half2_rn(x, y);
                const float2 f = __half22float2(hi);
                const __half2 v = g & 1 ? __floats2half2_rn(x - f.x, y - f.y) : hi;
                return *reinterpret_cast<const uint32_t *>(&v);
            };
            uint32_t qb0, qb1;
            float q_un;  // undoes head t's power of two
            {
                const float *qp = P.q + row + (size_t)(head0 + 4 * warp + (g >> 1)) * DH;
                const float2 x0 = turned(*reinterpret_cast<const float2 *>(qp + 2 * t4), cs[t4]);
                const float2 x1 = turned(*reinterpret_cast<const float2 *>(qp + 2 * t4 + 8), cs[t4 + 4]);
                float mx = fmaxf(fmaxf(fabsf(x0.x), fabsf(x0.y)), fmaxf(fabsf(x1.x), fabsf(x1.y)));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                float up, down;
                pow2_scale(mx * P.scale_log2e, up, down);
                const float f = P.scale_log2e;
                qb0 = column(x0.x * f * up, x0.y * f * up), qb1 = column(x1.x * f * up, x1.y * f * up);
                q_un = __shfl_sync(0xffffffffu, down, 8 * t4);
            }
            float m = -FLT_MAX, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};  // (finite: a block of scores of -inf is 0)  o: dim g (high, low column), dim g + 8; l: this lane's tokens
            const int len_cached = FUSED ? len - 1 : len;
            if (FUSED && len_cached / BT >= b0 && len_cached / BT < b1) {
                // Fused append: the eight lanes of a head compute the stored payload (RoPE'd K, raw V, both rounded to fp16), write
                // it to the cache and start the softmax state from it; the loop below covers the tokens already cached.
                const size_t at = row + (size_t)h * DH + 2 * g;
                const float2 w = cs[g];
                const float2 qr = turned(*reinterpret_cast<const float2 *>(P.q + at), w);
                const float2 kr = turned(*reinterpret_cast<const float2 *>(P.k_new + at), w);
                const float2 vr = *reinterpret_cast<const float2 *>(P.v_new + at);
                const float va = P.v_new[row + (size_t)h * DH + g], vb = P.v_new[row + (size_t)h * DH + g + 8];
                const __half2 kh = __floats2half2_rn(kr.x, kr.y), vh = __floats2half2_rn(vr.x, vr.y);
                const float2 kf = __half22float2(kh);
                float sc = (qr.x * P.scale_log2e) * kf.x + (qr.y * P.scale_log2e) * kf.y;
                sc += __shfl_xor_sync(0xffffffffu, sc, 4);
                sc += __shfl_xor_sync(0xffffffffu, sc, 8);
                sc += __shfl_xor_sync(0xffffffffu, sc, 16);
                m = sc;
                l = g == 0 ? kLift : 0.f;
                o[0] = kLift * __half2float(__float2half_rn(va)), o[2] = kLift * __half2float(__float2half_rn(vb));
                const int phys = P.table[(size_t)seq * P.mbs + len_cached / BT];
                if (phys < 0 || phys >= P.n_blocks) {
                    if (lane == 0) atomicOr(P.status, DEV_STATUS_BAD_BLOCK);
                } else {
                    __half *dst = P.kv + ((layer_base + phys) * P.H + h) * (size_t)(2 * BT * DH) + (size_t)(len_cached % BT) * DH + 2 * g;
                    *reinterpret_cast<__half2 *>(dst) = kh;
                    *reinterpret_cast<__half2 *>(dst + BT * DH) = vh;
                }
            }
            const int mi = lane >> 3, rr = lane & 7;
            const int k_off = ((mi & 1) * 8 + rr) * 32 + (mi >> 1) * 16;          // K tile as the A operand (rows = tokens)
            const int v_off = TILE + ((mi >> 1) * 8 + rr) * 32 + (mi & 1) * 16;   // V tile, transposed load (rows = dims)
            auto of_head_t = [&](float a0, float a1, float a2, float a3) {
                const float e = t4 & 1 ? a1 : a0, f = t4 & 1 ? a3 : a2;
                return t4 & 2 ? f : e;
            };
            // A key that fp16 holds as an infinity: the high part has the score, the low part the same infinity at either sign.
            auto both = [](float hi, float lo) { return isinf(hi) ? hi : hi + lo; };
            const int src0 = 8 * t4 + (g >> 1), src1 = src0 + 4;  // the lanes with p of tokens 2 t and 2 t + 1 of head g / 2

            bool aborted = false;
            for (int j = 0; j < nb; j++, it++) {
                const int s = stage;
                const uint32_t ph = phase;
                if (++stage == NS) stage = 0, phase ^= 1u;
                if (!aborted && !mbar_wait_bounded(&full_bar[s], ph, P.status, s_abort)) aborted = true;
                if (aborted) continue;  // keep counting blocks, touch nothing
#ifdef JGPT_B200_DECODE_TRACE
                if (j == 0 && tr_c2 == 0) tr_c2 = clock64();
#endif
                const int left = len_cached - (b0 + j) * BT;  // tokens of this block that are cached
                if (left > 0) {  // else the block holds the appended token alone
                    const unsigned char *base = smem + (size_t)s * stage_bytes;
                    float d[4][4];
                    uint32_t va[4][4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const unsigned char *tile = base + (size_t)(4 * warp + i) * HEAD_BYTES;
                        uint32_t ka[4];
                        ldmatrix_x4(ka, tile + k_off);
                        ldmatrix_x4_trans(va[i], tile + v_off);
#pragma unroll
                        for (int e = 0; e < 4; e++) d[i][e] = 0.f;
                        mma_16816(d[i], ka, qb0, qb1);
                    }
                    float s0 = both(of_head_t(d[0][0], d[1][0], d[2][0], d[3][0]), of_head_t(d[0][1], d[1][1], d[2][1], d[3][1])) * q_un;
                    float s1 = both(of_head_t(d[0][2], d[1][2], d[2][2], d[3][2]), of_head_t(d[0][3], d[1][3], d[2][3], d[3][3])) * q_un;
                    if (left < BT) {
                        // The slots beyond the last cached token hold whatever they held before: no score, and zeros in place of V
                        // (their probabilities are 0, but 0 x Inf or NaN is NaN inside the product).
                        if (g >= left) s0 = -INFINITY;
                        if (g + 8 >= left) s1 = -INFINITY;
                        const uint32_t lo = (2 * t4 < left ? 0xffffu : 0u) | (2 * t4 + 1 < left ? 0xffff0000u : 0u);
                        const uint32_t hi = (2 * t4 + 8 < left ? 0xffffu : 0u) | (2 * t4 + 9 < left ? 0xffff0000u : 0u);
#pragma unroll
                        for (int i = 0; i < 4; i++) va[i][0] &= lo, va[i][1] &= lo, va[i][2] &= hi, va[i][3] &= hi;
                    }
                    float bm = fmaxf(s0, s1);
                    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 4));
                    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 8));
                    bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, 16));
                    const float mn = fmaxf(m, bm);
                    const float corr = fast_exp2(m - mn);
                    const float p0 = fast_exp2(s0 - mn) * kLift, p1 = fast_exp2(s1 - mn) * kLift;
                    m = mn;
                    l = l * corr + (p0 + p1);
                    const uint32_t pb0 = column(__shfl_sync(0xffffffffu, p0, src0), __shfl_sync(0xffffffffu, p0, src1));
                    const uint32_t pb1 = column(__shfl_sync(0xffffffffu, p1, src0), __shfl_sync(0xffffffffu, p1, src1));
#pragma unroll
                    for (int i = 0; i < 4; i++) {
#pragma unroll
                        for (int e = 0; e < 4; e++) d[i][e] = 0.f;
                        mma_16816(d[i], va[i], pb0, pb1);
                    }
#pragma unroll
                    for (int e = 0; e < 4; e++) o[e] = fmaf(o[e], corr, of_head_t(d[0][e], d[1][e], d[2][e], d[3][e]));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty_bar[s]);
            }
#ifdef JGPT_B200_DECODE_TRACE
            tr_c3 = clock64();
#endif
            // After a timed-out wait the thread keeps walking the barriers below (so nobody is left waiting for it) but stores
            // nothing; the item loop ends at its next iteration.
            l += __shfl_xor_sync(0xffffffffu, l, 4);
            l += __shfl_xor_sync(0xffffffffu, l, 8);
            l += __shfl_xor_sync(0xffffffffu, l, 16);
            const float o0 = o[0] + o[1], o1 = o[2] + o[3];  // dims g, g + 8 of head h
            const bool writer = !aborted;
            float *op = P.out + row + (size_t)h * DH + g;
            if (nsplit == 1) {
                if (writer) {
                    const float inv = 1.f / fmaxf(l, 1e-12f);
                    op[0] = o0 * inv, op[8] = o1 * inv;
                }
                if (P.cluster) cluster_sync(), cluster_sync();
                continue;
            }
            constexpr int PS = DH + 2;
            if (P.cluster) {
                // ---- split-K inside a cluster: partials stay in shared memory, the CTA of chunk 0 merges them ----
                float *pp = cl_part + hl * PS;
                if (writer) {
                    pp[2 + g] = o0, pp[10 + g] = o1;
                    if (g == 0) pp[0] = m, pp[1] = l;
                } else if (g == 0) {
                    pp[0] = -INFINITY, pp[1] = 0.f;  // a chunk that gave up contributes nothing
                }
                cluster_sync();
                if (c == 0 && writer) {
                    float mc[8], lc[8], a0[8], a1[8];  // at most eight chunks: all of them requested before the first is used
#pragma unroll
                    for (int cc = 0; cc < 8; cc++) {
                        const bool in = cc < nsplit;
                        mc[cc] = in ? ld_cluster_f32(pp, (uint32_t)cc) : -INFINITY;
                        lc[cc] = in ? ld_cluster_f32(pp + 1, (uint32_t)cc) : 0.f;
                        a0[cc] = in ? ld_cluster_f32(pp + 2 + g, (uint32_t)cc) : 0.f;
                        a1[cc] = in ? ld_cluster_f32(pp + 10 + g, (uint32_t)cc) : 0.f;
                    }
                    float Mx = -INFINITY, L = 0.f, r0 = 0.f, r1 = 0.f;
#pragma unroll
                    for (int cc = 0; cc < 8; cc++) Mx = fmaxf(Mx, mc[cc]);
#pragma unroll
                    for (int cc = 0; cc < 8; cc++)
                        if (cc < nsplit) {
                            const float w = mc[cc] == -INFINITY ? 0.f : exp2f(mc[cc] - Mx);
                            L = fmaf(lc[cc], w, L), r0 = fmaf(a0[cc], w, r0), r1 = fmaf(a1[cc], w, r1);
                        }
                    const float inv = 1.f / fmaxf(L, 1e-12f);
                    op[0] = r0 * inv, op[8] = r1 * inv;
                }
                cluster_sync();  // nobody leaves (and frees its shared memory) before chunk 0 has read it
                continue;
            }
            // ---- split-K: publish the partial, last CTA of the sequence row merges ----
            const size_t prow = (((size_t)z * P.n + i) * P.max_chunks) * (size_t)P.H;  // + c*H + head
            if (writer) {
                float *pp = P.partials + (prow + (size_t)c * P.H + h) * PS;
                pp[2 + g] = o0, pp[10 + g] = o1;
                if (g == 0) pp[0] = m, pp[1] = l;
            }
#ifdef JGPT_B200_TRACE_NOMERGE
            if (P.n > 0) continue;  // timing experiment only: partials written, nobody merges
#endif
            __threadfence();
            named_bar_sync(1, n_cons);
            int *ticket = P.tickets + ((size_t)z * P.n + i) * P.n_hg + hg;
            if (tid == 0) {
                const int prev = atomicAdd(ticket, 1);
                s_last = (prev == nsplit - 1);
                if (prev == nsplit - 1) *ticket = 0;  // self-reset for the next launch
            }
            named_bar_sync(1, n_cons);
            if (s_last) {
                __threadfence();
                if (writer) {
                    float Mx = -INFINITY, L = 0.f, r0 = 0.f, r1 = 0.f;
                    for (int cc = 0; cc < nsplit; cc++) Mx = fmaxf(Mx, __ldcg(P.partials + (prow + (size_t)cc * P.H + h) * PS));
                    for (int cc = 0; cc < nsplit; cc++) {
                        const float *pp = P.partials + (prow + (size_t)cc * P.H + h) * PS;
                        const float w = exp2f(__ldcg(pp) - Mx);
                        L = fmaf(__ldcg(pp + 1), w, L);
                        r0 = fmaf(__ldcg(pp + 2 + g), w, r0), r1 = fmaf(__ldcg(pp + 10 + g), w, r1);
                    }
                    const float inv = 1.f / fmaxf(L, 1e-12f);
                    op[0] = r0 * inv, op[8] = r1 * inv;
                }
            }
            continue;
        }

        // ---------------- consumers, scalar form ----------------
        const int hl = tid / BT, t = tid % BT;
        const bool active = hl < P.HG;
        const int h = head0 + (active ? hl : 0);
        int rp = rp_raw;
        if (rp < 0 || rp >= P.max_positions) {
            if (tid == 0) atomicOr(P.status, DEV_STATUS_BAD_POSITION);
            rp = 0;
        }
        // q row: RoPE at rope_pos, then scaled by (1/sqrt(DH)) * log2(e) so that exp2f can be used.
        float q[DH];
        {
            const float *qp = P.q + row + (size_t)h * DH;
            const float2 *cs = P.rope + (size_t)rp * (DH / 2);
#pragma unroll
            for (int j = 0; j < DH / 2; j++) {
                const float2 x = *reinterpret_cast<const float2 *>(qp + 2 * j);
                const float2 w = cs[j];
                q[2 * j] = __fsub_rn(__fmul_rn(x.x, w.x), __fmul_rn(x.y, w.y)) * P.scale_log2e;
                q[2 * j + 1] = __fadd_rn(__fmul_rn(x.x, w.y), __fmul_rn(x.y, w.x)) * P.scale_log2e;
            }
        }
        // Fused append: the thread whose token is the new one computes the stored payload (RoPE'd K,
        // raw V, both rounded to fp16), writes it to the cache and scores it from registers.
        // Private online-softmax state of this (head, token lane).  The maximum starts finite: a first score of -inf has no weight.
        float m = -FLT_MAX, l = 0.f, o[DH];
#pragma unroll
        for (int d = 0; d < DH; d++) o[d] = 0.f;
        // Fused append: the new token sits at slot len-1.  The lane that owns that slot computes the
        // stored payload (RoPE'd K, raw V, both rounded to fp16), writes it to the cache and starts its
        // softmax state from it; the block loop below then covers the len-1 tokens already cached.
        const int len_cached = FUSED ? len - 1 : len;
        if constexpr (FUSED) {
            const int new_tok = len - 1;
            if (active && (new_tok / BT >= b0) && (new_tok / BT < b1) && (t == new_tok % BT)) {
                const float *kp = P.k_new + row + (size_t)h * DH, *vp = P.v_new + row + (size_t)h * DH;
                const float2 *cs = P.rope + (size_t)rp * (DH / 2);
                __align__(16) __half kh[DH], vh[DH];
                float sc = 0.f;
#pragma unroll
                for (int j = 0; j < DH / 2; j++) {
                    const float2 x = *reinterpret_cast<const float2 *>(kp + 2 * j);
                    const float2 y = *reinterpret_cast<const float2 *>(vp + 2 * j);
                    const float2 w = cs[j];
                    kh[2 * j] = __float2half_rn(__fsub_rn(__fmul_rn(x.x, w.x), __fmul_rn(x.y, w.y)));
                    kh[2 * j + 1] = __float2half_rn(__fadd_rn(__fmul_rn(x.x, w.y), __fmul_rn(x.y, w.x)));
                    vh[2 * j] = __float2half_rn(y.x);
                    vh[2 * j + 1] = __float2half_rn(y.y);
                    sc = fmaf(q[2 * j], __half2float(kh[2 * j]), sc);
                    sc = fmaf(q[2 * j + 1], __half2float(kh[2 * j + 1]), sc);
                    o[2 * j] = __half2float(vh[2 * j]);
                    o[2 * j + 1] = __half2float(vh[2 * j + 1]);
                }
                m = sc, l = 1.f;
                const int phys = P.table[(size_t)seq * P.mbs + new_tok / BT];
                if (phys < 0 || phys >= P.n_blocks) {
                    atomicOr(P.status, DEV_STATUS_BAD_BLOCK);
                } else {
                    __half *dst = P.kv + ((layer_base + phys) * P.H + h) * (size_t)(2 * BT * DH) + (size_t)t * DH;
                    if constexpr (DH >= 8) {
#pragma unroll
                        for (int cc = 0; cc < DH / 8; cc++) {
                            reinterpret_cast<uint4 *>(dst)[cc] = reinterpret_cast<const uint4 *>(kh)[cc];
                            reinterpret_cast<uint4 *>(dst + BT * DH)[cc] = reinterpret_cast<const uint4 *>(vh)[cc];
                        }
                    } else {
                        *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(kh);
                        *reinterpret_cast<uint2 *>(dst + BT * DH) = *reinterpret_cast<const uint2 *>(vh);
                    }
                }
            }
        }

        swap_halves<DH>(q, t);  // match the order in which load_row delivers rows on this lane
        swap_halves<DH>(o, t);
        bool aborted = false;
        for (int j = 0; j < nb; j++, it++) {
            const int s = stage;
            const uint32_t ph = phase;
            if (++stage == NS) stage = 0, phase ^= 1u;
            if (!aborted && !mbar_wait_bounded(&full_bar[s], ph, P.status, s_abort)) aborted = true;
            if (aborted) continue;  // keep counting blocks, touch nothing
#ifdef JGPT_B200_DECODE_TRACE
            if (j == 0 && tr_c2 == 0) tr_c2 = clock64();
#endif
            const int tok = (b0 + j) * BT + t;
            if (active && tok < len_cached) {
                const unsigned char *ktile = smem + (size_t)s * stage_bytes + (size_t)hl * HEAD_BYTES;
                float kr[DH], vr[DH];
                load_row<DH>(ktile, t, kr);
                float sc = 0.f;
#pragma unroll
                for (int d = 0; d < DH; d++) sc = fmaf(q[d], kr[d], sc);
                if (sc > m) {  // new running maximum: rescale the private state
                    const float corr = fast_exp2(m - sc);  // 0 on the first token
                    l *= corr;
#pragma unroll
                    for (int d = 0; d < DH; d++) o[d] *= corr;
                    m = sc;
                }
                load_row<DH>(ktile + TILE, t, vr);
                const float pexp = fast_exp2(sc - m);
                l += pexp;
#pragma unroll
                for (int d = 0; d < DH; d++) o[d] = fmaf(pexp, vr[d], o[d]);
            }
            __syncwarp();
            if ((tid & 31) == 0) mbar_arrive(&empty_bar[s]);
        }
        // After a timed-out wait the thread keeps walking the barriers below (so nobody is left
        // waiting for it) but stores nothing; the item loop ends at its next iteration.

#ifdef JGPT_B200_DECODE_TRACE
        tr_c3 = clock64();
#endif
        // ---- merge the 16 token lanes of each head (warp shuffles) ----
        swap_halves<DH>(o, t);  // back to natural dimension order
        float M = m;
#pragma unroll
        for (int off = 8; off >= 1; off >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, off));
        const float f = exp2f(m - M);  // 0 for a lane without a token
        l *= f;
#pragma unroll
        for (int d = 0; d < DH; d++) o[d] *= f;
#pragma unroll
        for (int off = 8; off >= 1; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
        halfwarp_reduce_scatter<DH>(o, t);
        // lane t now holds dims {g*16 + t} (DH >= 16) or dim t % DH (DH < 16) in o[0..OPL)
        const bool writer = active && !aborted && (DH >= 16 || t < DH);

        if (nsplit == 1) {
            if (writer) {
                const float inv = 1.f / fmaxf(l, 1e-12f);
#pragma unroll
                for (int g = 0; g < OPL; g++) P.out[row + (size_t)h * DH + g * 16 + (DH >= 16 ? t : t % DH)] = o[g] * inv;
            }
            if (P.cluster) cluster_sync(), cluster_sync();
            continue;
        }
        if (P.cluster) {
            // ---- split-K inside a cluster: partials stay in shared memory, the CTA of chunk 0 merges them ----
            constexpr int PS = DH + 2;
            if (writer) {
                float *pp = cl_part + hl * PS;
#pragma unroll
                for (int g = 0; g < OPL; g++) pp[2 + g * 16 + (DH >= 16 ? t : t % DH)] = o[g];
                if (t == 0) pp[0] = M, pp[1] = l;
            } else if (active && aborted && t == 0) {
                cl_part[hl * PS] = -INFINITY, cl_part[hl * PS + 1] = 0.f;  // a chunk that gave up contributes nothing
            }
            cluster_sync();
            if (c == 0 && writer) {
                const float *pp = cl_part + hl * PS;
                float Mx = -INFINITY;
                for (int cc = 0; cc < nsplit; cc++) Mx = fmaxf(Mx, ld_cluster_f32(pp, (uint32_t)cc));
                float L = 0.f, acc[OPL];
#pragma unroll
                for (int g = 0; g < OPL; g++) acc[g] = 0.f;
                for (int cc = 0; cc < nsplit; cc++) {
                    const float mc = ld_cluster_f32(pp, (uint32_t)cc);
                    const float w = mc == -INFINITY ? 0.f : exp2f(mc - Mx);
                    L = fmaf(ld_cluster_f32(pp + 1, (uint32_t)cc), w, L);
#pragma unroll
                    for (int g = 0; g < OPL; g++)
                        acc[g] = fmaf(ld_cluster_f32(pp + 2 + g * 16 + (DH >= 16 ? t : t % DH), (uint32_t)cc), w, acc[g]);
                }
                const float inv = 1.f / fmaxf(L, 1e-12f);
#pragma unroll
                for (int g = 0; g < OPL; g++) P.out[row + (size_t)h * DH + g * 16 + (DH >= 16 ? t : t % DH)] = acc[g] * inv;
            }
            cluster_sync();  // nobody leaves (and frees its shared memory) before chunk 0 has read it
            continue;
        }

        // ---- split-K: publish the partial, last CTA of the sequence row merges ----
        constexpr int PSTRIDE = DH + 2;
        const size_t prow = (((size_t)z * P.n + i) * P.max_chunks) * (size_t)P.H;  // + c*H + head
        if (writer) {
            float *pp = P.partials + (prow + (size_t)c * P.H + h) * PSTRIDE;
#pragma unroll
            for (int g = 0; g < OPL; g++) pp[2 + g * 16 + (DH >= 16 ? t : t % DH)] = o[g];
            if (t == 0) pp[0] = M, pp[1] = l;
        }
#ifdef JGPT_B200_TRACE_NOMERGE
        if (P.n > 0) continue;  // timing experiment only: partials written, nobody merges
#endif
        __threadfence();
        named_bar_sync(1, n_cons);
        int *ticket = P.tickets + ((size_t)z * P.n + i) * P.n_hg + hg;
        if (tid == 0) {
            const int prev = atomicAdd(ticket, 1);
            s_last = (prev == nsplit - 1);
            if (prev == nsplit - 1) *ticket = 0;  // self-reset for the next launch
        }
        named_bar_sync(1, n_cons);
        if (s_last) {
            __threadfence();
            if (writer) {
                float Mx = -INFINITY;
                for (int cc = 0; cc < nsplit; cc++)
                    Mx = fmaxf(Mx, __ldcg(P.partials + (prow + (size_t)cc * P.H + h) * PSTRIDE));
                float L = 0.f, acc[OPL];
#pragma unroll
                for (int g = 0; g < OPL; g++) acc[g] = 0.f;
                for (int cc = 0; cc < nsplit; cc++) {
                    const float *pp = P.partials + (prow + (size_t)cc * P.H + h) * PSTRIDE;
                    const float w = exp2f(__ldcg(pp) - Mx);
                    L = fmaf(__ldcg(pp + 1), w, L);
#pragma unroll
                    for (int g = 0; g < OPL; g++) acc[g] = fmaf(__ldcg(pp + 2 + g * 16 + (DH >= 16 ? t : t % DH)), w, acc[g]);
                }
                const float inv = 1.f / fmaxf(L, 1e-12f);
#pragma unroll
                for (int g = 0; g < OPL; g++) P.out[row + (size_t)h * DH + g * 16 + (DH >= 16 ? t : t % DH)] = acc[g] * inv;
            }
        }
    }
    // Abort path only: before the CTA (and its shared memory) goes away, give the bulk copies that
    // were already issued a bounded chance to land.
    __syncthreads();
#ifdef JGPT_B200_DECODE_TRACE
    tr_c4 = clock64();
    timeline_at(P.timeline, 2);
    if (tid == 0 && P.trace) {
        long long gt1;
        unsigned smid;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(gt1));
        asm volatile("mov.u32 %0, %smid;" : "=r"(smid));
        long long *tp = P.trace + (size_t)blockIdx.x * 8;
        tp[0] = tr_gt0, tp[1] = gt1, tp[2] = tr_c1 - tr_c0, tp[3] = tr_c2 - tr_c0, tp[4] = tr_c3 - tr_c0, tp[5] = tr_c4 - tr_c0, tp[6] = smid, tp[7] = 0;
    }
#endif
    if (*s_abort && tid == n_cons) {
        const uint32_t first = it > (uint32_t)NS ? it - NS : 0;
        for (uint32_t idx = first; idx < it; idx++)
            for (uint32_t spin = 0; spin < (1u << 16); spin++)
                if (mbar_try_wait(&full_bar[idx % NS], (idx / NS) & 1)) break;
    }
    // Dynamic mode: the last CTA to leave puts both counters back to zero for the next launch (by then every
    // CTA has drawn its sentinel, so nobody touches the item counter any more).
    if (P.dynamic && tid == 0) {
        __threadfence();
        if (atomicAdd(P.counters + 1, 1) == (int)gridDim.x - 1) {
            P.counters[0] = 0;
            P.counters[1] = 0;
            __threadfence();
        }
    }
}

// Raises a decode kernel's dynamic shared-memory limit to the largest request any launch makes, once per
// (kernel variant, device).  Guarded: contexts of different devices may launch from different host threads.
static cudaError_t decode_opt_in_smem(void (*kern)(const DecodeParams), int variant, int device) {
    static std::mutex mu;
    static bool done[16][64] = {};
    std::lock_guard<std::mutex> lock(mu);
    const bool tracked = variant >= 0 && variant < 16 && device >= 0 && device < 64;
    if (tracked && done[variant][device]) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxStages * 24 * 1024);
    if (e == cudaSuccess && tracked) done[variant][device] = true;
    return e;
}

// Largest divisor of H whose slab (HG * 64 * DH bytes) stays within 24 KiB and 480 consumer threads.
// A launch with few (layer, sequence) pairs - the model's per-layer decode step at small batch - takes the smallest
// group of at least 6 heads that still gives no more CTAs than fit at once (two per SM): more, lighter CTAs
// (measured on the decode step at batch 64: 0.638 ms with 24 heads per CTA, 0.613 ms with 6 or 8).
static int pick_head_group(int H, int DH, int forced, long long pairs = 0, long long slots = 0) {
    const int cap = std::min(30, std::max(1, 384 / DH));  // == max_head_group<DH>()
    if (forced > 0 && forced <= cap && H % forced == 0) return forced;
    int best = 1;
    for (int g = 1; g <= std::min(H, cap); g++)
        if (H % g == 0) best = g;
    if (pairs > 0 && slots > 0 && pairs * (H / best) < slots)
        for (int g = 6; g < best; g++)
            if (H % g == 0 && pairs * (H / g) <= slots) return g;
    return best;
}

// d_head 16: the tensor-core consumers for the per-layer launches of a decode loop and for launches of more (layer, sequence) pairs than
// fit at once, in CTAs of a multiple of four heads.  A smaller launch is latency, and a block is a longer chain on the tensor cores (two
// products, three shuffles for the maximum, two for p) than for a thread with its own token: 12 layers of a few sequences in one launch
// took 39.9 and 8.7 us with the fp32 consumers, 43.6 and 10.9 us with these; 64 x 1024 takes 190 and 188 us.  A warp with fewer than four
// heads does the same work for less: a launch per layer for 200 sequences of 1000, 1 / 2 / 6 heads, 13.3 / 13.5 / 20.1 us with the fp32
// consumers, 18.5 / 18.5 / 21.0 with a ragged last warp.
static bool tensor_consumers(const Pool *p, int HG, bool per_layer, long long pairs) {
    if (HG % 4 != 0) return false;
    return per_layer || pairs * (p->heads / pick_head_group(p->heads, 16, p->head_group)) >= 2ll * p->ctx->sm_count;
}

template <int DH>
static int32_t launch_decode_t(Pool *p, const DecodeParams &P, bool fused, bool mma, int threads, size_t smem, int grid) {
    void (*kern)(const DecodeParams) = fused ? attn_decode_kernel<DH, true, false> : attn_decode_kernel<DH, false, false>;
    if constexpr (DH == 16)
        if (mma) kern = fused ? attn_decode_kernel<DH, true, true> : attn_decode_kernel<DH, false, true>;
    // Opt in to > 48 KiB of dynamic shared memory once per kernel and device: the most a launch can ask for
    // (kMaxStages stages of a 24 KiB slab), so that no later, smaller request ever lowers the limit again.
    JGPT_CUDA_TRY(decode_opt_in_smem(kern, (fused ? 1 : 0) + (DH == 16 && mma ? 2 : 0) + 4 * (DH == 4 ? 0 : DH == 8 ? 1 : DH == 16 ? 2 : 3), p->ctx->device));
    if (P.overlap || P.cluster) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid), cfg.blockDim = dim3((unsigned)threads), cfg.dynamicSmemBytes = smem, cfg.stream = p->ctx->stream;
        cudaLaunchAttribute attr[2];
        int na = 0;
        if (P.overlap) {
            attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[na].val.programmaticStreamSerializationAllowed = 1;
            na++;
        }
        if (P.cluster) {
            attr[na].id = cudaLaunchAttributeClusterDimension;
            attr[na].val.clusterDim.x = (unsigned)P.max_chunks, attr[na].val.clusterDim.y = 1, attr[na].val.clusterDim.z = 1;
            na++;
        }
        cfg.attrs = attr, cfg.numAttrs = (unsigned)na;
        JGPT_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, P));
    } else {
        kern<<<grid, threads, smem, p->ctx->stream>>>(P);
    }
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}

#ifdef JGPT_B200_DECODE_TRACE
static long long *g_decode_trace = nullptr;
static int g_decode_trace_items = 0;
extern "C" __attribute__((visibility("default"))) int jgpt_debug_decode_trace(long long *host_out, int cap_items) {
    const int n = g_decode_trace_items < cap_items ? g_decode_trace_items : cap_items;
    cudaDeviceSynchronize();
    if (g_decode_trace && n > 0) cudaMemcpy(host_out, g_decode_trace, sizeof(long long) * 8 * 65536, cudaMemcpyDeviceToHost);
    return n;
}
#endif

// Clusters of `c` CTAs of the decode kernel with these consumers, block size and ring that the device holds at once, as
// cudaOccupancyMaxActiveClusters reports it; cached per shape.  On B200 with 416 threads (fp32 consumers of 24 heads) and a 72 KiB ring:
// 296 single CTAs, but 93 / 71 / 56 / 45 / 37 / 33 clusters of 3 / 4 / 5 / 6 / 7 / 8 (a cluster stays inside one GPC).
// 0 when the query fails (the caller then plans without clusters).
static int cluster_capacity(Pool *p, bool fused, bool mma, int threads, size_t smem, int c) {
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, int, size_t, int, int>, int> cache;
    const auto key = std::make_tuple(p->ctx->device, p->dhead, (int)fused, (int)mma, smem, threads, c);
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find(key);
        if (it != cache.end()) return it->second;
    }
    void (*kern)(const DecodeParams) = nullptr;
    int variant = -1;
    switch (p->dhead) {
        case 4: kern = fused ? attn_decode_kernel<4, true> : attn_decode_kernel<4, false>, variant = 0; break;
        case 8: kern = fused ? attn_decode_kernel<8, true> : attn_decode_kernel<8, false>, variant = 4; break;
        case 16:
            if (mma) kern = fused ? attn_decode_kernel<16, true, true> : attn_decode_kernel<16, false, true>, variant = 10;
            else kern = fused ? attn_decode_kernel<16, true, false> : attn_decode_kernel<16, false, false>, variant = 8;
            break;
        case 32: kern = fused ? attn_decode_kernel<32, true> : attn_decode_kernel<32, false>, variant = 12; break;
        default: return 0;
    }
    int n = 0;
    if (decode_opt_in_smem(kern, variant + (fused ? 1 : 0), p->ctx->device) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)c, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)c * 64), cfg.blockDim = dim3((unsigned)threads), cfg.dynamicSmemBytes = smem;
        cfg.attrs = attr, cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            n = 0;
        }
    }
    std::lock_guard<std::mutex> lock(mu);
    cache[key] = n;
    return n;
}

// Split-K chunk length of a launch with `base` (layer, sequence, head group) triples of up to max_blocks KV blocks.
// Two CTAs fit on an SM.  When the triples alone fill those slots the launch runs in several waves anyway and
// 32-block chunks keep the per-item set-up small.  Otherwise every sequence is cut into as many chunks as still
// fit in ONE wave (a few CTAs spilling into a second wave would double the launch time), at least 4 blocks each.
static int pick_chunk_blocks(const Pool *p, long long base, int max_blocks) {
    const long long slots = 2ll * p->ctx->sm_count;
    if (base >= slots) return 32;
    const long long nsplit = std::max(1ll, std::min(slots / base, (long long)(max_blocks + 3) / 4));
    const int cb = (int)((max_blocks + nsplit - 1) / nsplit);
    return std::min(32, std::max(4, cb));
}

int32_t launch_attn_decode(Pool *p, int layer0, int n_layers, const float *q, const float *k_new, const float *v_new,
                           const int *seq_ids, const int *rope_pos, const int *lens, int n, int max_len, float *out, int overlap, int of_layers) {
    DecodeParams P;
    memset(&P, 0, sizeof(P));
    const int DH = p->dhead;
    P.kv = p->kv, P.table = p->d_table, P.rope = p->d_rope;
    P.q = q, P.k_new = k_new, P.v_new = v_new, P.out = out;
    P.seq_ids = seq_ids, P.rope_pos = rope_pos, P.lens = lens;
    P.status = p->ctx->d_status;
    P.n = n, P.H = p->heads, P.layer0 = layer0, P.n_layers = n_layers, P.mbs = p->max_blocks_per_seq;
    P.n_blocks = p->n_blocks, P.max_seqs = p->max_seqs, P.max_positions = p->max_positions;
    const int ov = overlap >= 0 ? overlap : p->launch_overlap;
    // Head group and ring depth.  An overlapped single-layer launch (the per-layer decode loop) runs best with all
    // heads in one CTA (one 24 KiB slab per copy) and a three-stage ring, so that three CTAs fit on an SM and the next
    // launch's CTAs can move in beside the ones still draining: 20.7 us per layer at batch 64 / context 1024 against
    // 22.7 us for the ordinary launch (6-8 heads per CTA, four stages).
    const bool overlapped_single = ov >= 1 && n_layers == 1 && p->persistent <= 0;
    P.HG = overlapped_single ? pick_head_group(p->heads, DH, p->head_group)
                             : pick_head_group(p->heads, DH, p->head_group, (long long)n_layers * n, 2ll * p->ctx->sm_count);
    // (a launch that is one of several over a call's layers chooses its consumers by all of them, like the launch of the whole call)
    const int rule_layers = of_layers > 0 ? of_layers : n_layers;
    const bool mma = DH == 16 && tensor_consumers(p, P.HG, overlapped_single && rule_layers == 1, (long long)rule_layers * n);
    // With up to a row per SM and sequences of up to 1024 tokens the heads go to two CTAs: smaller CTAs spread more evenly, and the last one
    // is done sooner.  Tensor-core consumers, JGPT-35M step of context 512 at 8 / 32 / 64 / 128 / 160 / 200 rows, us: one CTA
    // 208 / 278 / 351 / 524 / 582 / 697, two 203 / 270 / 344 / 508 / 550 / 742, three 201 / 286 / 358 / 524 / 568 / 755 (160 rows would gain
    // as well; between them and 200 it turns).  fp32 consumers, host calls of 3 to 11 layers in stages, 1 to 8 rows of 1000: 0-4 % of the call.
    // Long sequences stream, and whole slabs do that better (48 of 1024 to 8192 tokens, 12 layers: 567 us, 596 in halves).
    const bool halves = overlapped_single && DH == 16 && p->head_group <= 0 && P.HG >= 12 && P.HG % (mma ? 8 : 2) == 0 && max_len <= 1024 &&
                        (long long)n * (p->heads / P.HG) <= p->ctx->sm_count;
    if (halves) P.HG /= 2;
    P.n_hg = p->heads / P.HG;
    const int max_blocks = std::min(p->max_blocks_per_seq, (max_len + kBlockTokens - 1) / kBlockTokens);
    // Work distribution.  Default (persistent <= 0): one CTA per work item, the hardware block scheduler hands
    // items to SMs as CTAs retire.  persistent = k > 0: k CTAs per SM claim items from a global counter (kept
    // for experiments: on B200 it measured 4-15 % slower than the plain grid at every chunk length).
    const int per_sm = p->persistent > 0 ? p->persistent : 2;
    const long long slots = (long long)per_sm * p->ctx->sm_count;
    const bool dynamic = p->persistent > 0;
    P.stages = p->stages > 0 ? p->stages : (overlapped_single ? 3 : 4);
    const int n_cons = mma ? consumer_threads<true>(P.HG) : consumer_threads<false>(P.HG);
    const int threads = n_cons + 32;
    const size_t stage_bytes = (size_t)P.HG * 2 * kBlockTokens * DH * 2;
    const bool may_cluster = p->cluster_merge && !dynamic, fused = k_new != nullptr;
    // The chunks of one sequence as one thread-block cluster (up to the portable size of 8): merge in shared memory.
    // Not for the work queue (its CTAs take several items).
    // Only for launches of a wave or two: there the merge's global round trips are a visible part of the launch (per-layer
    // launch at batch 64 / context 1024: 24.1 -> 22.7 us).  A launch of many waves hides them behind other CTAs' copies,
    // and co-scheduling pairs of CTAs costs it more than it saves (12-layer launch: 198 us without, 202 us with).
    auto cluster_launch = [&](int chunks, long long items) { return may_cluster && chunks >= 2 && chunks <= 8 && items <= 4ll * p->ctx->sm_count; };
    // How a launch whose CTAs take `ring` bytes of shared memory is cut, and how many rounds of CTAs that makes (where it is asked below).
    struct Cut {
        int chunk_blocks, max_chunks;
        long long items, slots;
        long long rounds() const { return (items + slots - 1) / slots; }
    };
    auto cut = [&](size_t ring) {
        Cut o{};
        if (p->chunk_blocks > 0) {
            o.chunk_blocks = p->chunk_blocks;
        } else if (overlapped_single && may_cluster) {
            // The per-layer launch of the model's decode step: the chunks of a sequence are one cluster, so the launch is one
            // wave only while the device holds `base` clusters of that size at once -- fewer CTAs than two per SM (see
            // cluster_capacity; clusters beyond it wait for a whole CTA time).  Most chunks of at least 4 blocks that stay
            // 1/16 under that number (a launch at the exact limit measured slower than the next smaller cluster).  JGPT-35M
            // step, ms per step before / after: 40 rows 0.591 / 0.509, 48 rows 0.614 / 0.512, 96 rows 0.775 / 0.672;
            // up to 29 rows ten chunks merged through global scratch became eight in a cluster (16 rows: 0.430 / 0.413).
            const long long base = (long long)n * P.n_hg;
            int c = 1;
            for (int t = std::min(8, (max_blocks + 3) / 4); t >= 2; t--)
                if (16 * base <= 15ll * cluster_capacity(p, fused, mma, threads, ring, t)) {
                    c = t;
                    break;
                }
            const int c_min = (max_blocks + 31) / 32;  // a chunk holds at most 32 blocks
            if (c == 1 && (c_min > 1 || base > 2ll * p->ctx->sm_count)) {
                // No split fits one wave: take the one with the least rounds x (chunk length + ~6 blocks' worth of per-CTA
                // start-up and merge).  160 rows of 40 blocks: 3 chunks in 2 rounds (0.925 ms per step) against 2 chunks in
                // 2 rounds (0.985); 224 rows: 2 chunks in 2 rounds (1.217) against 3 chunks in 3 (1.264).
                long long best_cost = -1;
                for (int t = c_min; t <= std::min(8, (max_blocks + 3) / 4); t++) {
                    const long long cap = t == 1 ? 2ll * p->ctx->sm_count : (long long)cluster_capacity(p, fused, mma, threads, ring, t);
                    if (cap <= 0) continue;
                    // (clusters of three and more: a round counts as full at 15/16 of the capacity, like the one-wave rule above --
                    // 186 rows are two rounds of 93 three-CTA clusters on paper and measured 0.98 ms against 0.92 ms with pairs)
                    const long long full = t >= 3 ? 15 * cap : 16 * cap;
                    const long long rounds = (16 * base + full - 1) / full, cost = rounds * ((max_blocks + t - 1) / t + 6);
                    if (best_cost < 0 || cost < best_cost) best_cost = cost, c = t;
                }
            }
            c = std::max(c, c_min);
            o.chunk_blocks = std::min(32, std::max(4, (max_blocks + c - 1) / c));
        } else {
            o.chunk_blocks = pick_chunk_blocks(p, (long long)n_layers * n * P.n_hg, max_blocks);
        }
        o.max_chunks = std::max(1, (max_blocks + o.chunk_blocks - 1) / o.chunk_blocks);
        o.items = (long long)n_layers * n * P.n_hg * o.max_chunks, o.slots = 1;
        if (mma && overlapped_single) {
            const int size = cluster_launch(o.max_chunks, o.items) ? o.max_chunks : 1;
            o.slots = std::max(1ll, (long long)size * cluster_capacity(p, fused, mma, threads, ring, size));
        }
        return o;
    };
    // The tensor-core consumers need few registers, so shared memory decides how many CTAs of a per-layer launch share an SM: three with
    // all 24 heads, where the fp32 consumers stand two at a time.  Three are one round less for some launches (36 sequences of 4096: 43 us
    // a layer, 61 with two).  Otherwise the third only lets CTAs that move in early pile up on the SMs that are free first and makes a last,
    // short round as long as a full one (28 of 1024 to 4096 tokens 38 us with three, 32 with two; 64 of 4096 83 and 73), so the ring is
    // padded by half unless it saves a round.  A launch of at most half the slots spreads by itself where it runs back to back with
    // its like (48 of 2000 with 8 heads 16 us, 18 padded), and halves of the heads (96 of 1000: 30 and 33) and CTAs of four (200 of 4000: 42
    // and 57) always.
    size_t smem = stage_bytes * P.stages;
    Cut plan = cut(smem);
    if (mma && overlapped_single && !halves && P.HG >= 8 && p->stages <= 0 && (ov >= 2 || 2 * plan.items > plan.slots)) {
        const Cut two = cut(smem * 3 / 2);
        if (two.rounds() <= plan.rounds()) plan = two, smem = smem * 3 / 2;
    }
    P.chunk_blocks = plan.chunk_blocks, P.max_chunks = plan.max_chunks;
    P.max_len = max_blocks * kBlockTokens;
    P.overlap = ov;
    P.stream_hint = p->stream_hint;
    P.scale_log2e = (1.0f / sqrtf((float)DH)) * 1.4426950408889634f;
    JGPT_REQUIRE(plan.items < (1ll << 31), JGPT_ERR_INVALID_ARGUMENT, "too many work items (%lld)", plan.items);
    P.n_items = (int)plan.items;
    P.cluster = cluster_launch(P.max_chunks, plan.items) ? 1 : 0;
    if (P.max_chunks > 1 && !P.cluster) {
        int32_t rc = pool_ensure_split_scratch(p, (uint64_t)n_layers * n * P.max_chunks * p->heads * (DH + 2),
                                               (uint64_t)n_layers * n * P.n_hg);
        if (rc) return rc;
    }
    P.partials = p->d_partials, P.tickets = p->d_tickets;
#ifdef JGPT_B200_DECODE_TRACE
    {
        static long long *d_trace = nullptr;
        static int launch_no = 0;
        if (!d_trace) cudaMalloc(&d_trace, sizeof(long long) * 8 * 65536);
        // two halves used in turn: the last two launches can be compared (where did the second start / the first end)
        if (n_layers == 1) P.timeline = timeline_next();
        P.trace = P.n_items <= 32768 ? d_trace + (size_t)(launch_no & 1) * 8 * 32768 : nullptr;
        launch_no++;
        g_decode_trace = d_trace, g_decode_trace_items = P.n_items;
    }
#endif
    int grid = P.n_items;
    if (dynamic && (long long)P.n_items > slots) {
        grid = (int)slots;
        P.dynamic = 1;
        P.counters = p->d_item_counters;
    }
    if (P.dynamic && P.overlap > 1) P.overlap = 1;  // the work-queue counters are reset by the previous launch's last CTA
    switch (DH) {
        case 4: return launch_decode_t<4>(p, P, fused, mma, threads, smem, grid);
        case 8: return launch_decode_t<8>(p, P, fused, mma, threads, smem, grid);
        case 16: return launch_decode_t<16>(p, P, fused, mma, threads, smem, grid);
        case 32: return launch_decode_t<32>(p, P, fused, mma, threads, smem, grid);
        default: return fail(JGPT_ERR_UNSUPPORTED, "dhead %d not supported", DH);
    }
}

}  // namespace jgpt

using namespace jgpt;

static int32_t decode_common(jgpt_kvpool h, int32_t layer0, int32_t n_layers, const float *q, const float *k, const float *v,
                             const int32_t *seq_ids, const int32_t *rope_pos, const int32_t *lens, int32_t n, int32_t max_len,
                             float *out, bool fused) {
    Pool *p = pool_registry().get(h);
    JGPT_REQUIRE(p, JGPT_ERR_BAD_HANDLE, "bad kvpool handle");
    JGPT_REQUIRE(!p->layered, JGPT_ERR_UNSUPPORTED, "not available on a layered decoder's pool");
    JGPT_CUDA_TRY(make_current(p->ctx));
    JGPT_REQUIRE(n_layers >= 1 && layer0 >= 0 && layer0 + n_layers <= p->layers, JGPT_ERR_OUT_OF_RANGE,
                 "layers [%d, %d) outside [0,%d)", layer0, layer0 + n_layers, p->layers);
    if (n == 0) return JGPT_OK;
    JGPT_REQUIRE(n > 0 && q && seq_ids && rope_pos && lens && out && (!fused || (k && v)), JGPT_ERR_INVALID_ARGUMENT,
                 "null pointer or negative count");
    JGPT_REQUIRE(max_len >= 1, JGPT_ERR_INVALID_ARGUMENT, "max_len must be >= 1");
    return launch_attn_decode(p, layer0, n_layers, q, fused ? k : nullptr, fused ? v : nullptr, seq_ids, rope_pos, lens, n,
                              max_len, out);
}

extern "C" {

int32_t jgpt_attn_decode(jgpt_kvpool pool, int32_t layer0, int32_t n_layers, const float *q_dev, const int32_t *seq_ids_dev,
                         const int32_t *rope_pos_dev, const int32_t *lens_dev, int32_t n, int32_t max_len, float *out_dev) {
    return decode_common(pool, layer0, n_layers, q_dev, nullptr, nullptr, seq_ids_dev, rope_pos_dev, lens_dev, n, max_len,
                         out_dev, false);
}

int32_t jgpt_attn_decode_append(jgpt_kvpool pool, int32_t layer0, int32_t n_layers, const float *q_dev, const float *k_dev,
                                const float *v_dev, const int32_t *seq_ids_dev, const int32_t *rope_pos_dev,
                                const int32_t *lens_dev, int32_t n, int32_t max_len, float *out_dev) {
    return decode_common(pool, layer0, n_layers, q_dev, k_dev, v_dev, seq_ids_dev, rope_pos_dev, lens_dev, n, max_len,
                         out_dev, true);
}

int32_t jgpt_attn_decode_append_host(jgpt_kvpool pool, int32_t layer0, int32_t n_layers, const float *q_host,
                                     const float *k_host, const float *v_host, const int32_t *seq_ids_host,
                                     const int32_t *rope_pos_host, const int32_t *lens_host, int32_t n, float *out_host) {
    Pool *p = pool_registry().get(pool);
    JGPT_REQUIRE(p, JGPT_ERR_BAD_HANDLE, "bad kvpool handle");
    JGPT_REQUIRE(!p->layered, JGPT_ERR_UNSUPPORTED, "not available on a layered decoder's pool");
    JGPT_CUDA_TRY(make_current(p->ctx));
    if (n == 0) return JGPT_OK;
    JGPT_REQUIRE(n > 0 && n_layers >= 1 && q_host && k_host && v_host && seq_ids_host && rope_pos_host && lens_host && out_host,
                 JGPT_ERR_INVALID_ARGUMENT, "null pointer or bad count");
    const size_t slab = (size_t)n_layers * n * p->heads * p->dhead;
    int32_t rc = pool_ensure_staging(p, 4 * slab, 3 * (size_t)n);
    if (rc) return rc;
    int max_len = 1;
    for (int i = 0; i < n; i++) {
        JGPT_REQUIRE(seq_ids_host[i] >= 0 && seq_ids_host[i] < p->max_seqs && p->seqs[(size_t)seq_ids_host[i]].used,
                     JGPT_ERR_OUT_OF_RANGE, "seq_ids[%d] = %d is not an allocated sequence", i, seq_ids_host[i]);
        JGPT_REQUIRE(lens_host[i] >= 1 && lens_host[i] <= (int)p->seqs[(size_t)seq_ids_host[i]].blocks.size() * kBlockTokens,
                     JGPT_ERR_ILLEGAL_STATE, "lens[%d] = %d is beyond the blocks reserved for sequence %d", i, lens_host[i],
                     seq_ids_host[i]);
        JGPT_REQUIRE(rope_pos_host[i] >= 0 && rope_pos_host[i] < p->max_positions, JGPT_ERR_INVALID_ARGUMENT,
                     "rope_pos[%d] = %d outside [0,%d)", i, rope_pos_host[i], p->max_positions);
        max_len = std::max(max_len, lens_host[i]);
    }
    cudaStream_t st = p->ctx->stream;
    float *dq = p->d_stage_f, *dk = dq + slab, *dv = dk + slab, *dout = dv + slab;
    int *dseq = p->d_stage_i, *drp = dseq + n, *dlen = drp + n;
    // Three ways to move the bytes.  STAGED: copies in and out around the kernel, pipelined over groups of layers
    // (works for any host memory).  ZEROCOPY (page-locked, device-mapped buffers): nothing is staged, the kernel
    // reads q / k / v and writes the result through the buffers' device addresses inside the one launch; fastest
    // when this process has the host fabric to itself (0.25 ms per 12-layer step against 0.30), slower when eight
    // processes do it at once (0.46 against 0.33: many small PCIe reads).  HYBRID: inputs by one copy each, the
    // result written in place.  Which one wins is a property of the machine at that moment, so the first calls
    // on a pool take turns (three samples each, same results whatever the way) and the fastest is kept;
    // JGPT_B200_HOST_ZEROCOPY = 0 / 1 / 2 pins STAGED / ZEROCOPY / HYBRID.
    enum { STAGED = 0, ZEROCOPY = 1, HYBRID = 2 };
    void *dp[4] = {};
    bool mapped = true;
    {
        const void *hp[4] = {q_host, k_host, v_host, out_host};
        for (int i = 0; i < 4 && mapped; i++) {
            cudaPointerAttributes a;
            if (cudaPointerGetAttributes(&a, hp[i]) != cudaSuccess) {
                cudaGetLastError();
                mapped = false;
            } else if (a.type != cudaMemoryTypeHost || !a.devicePointer) {
                mapped = false;
            } else {
                dp[i] = a.devicePointer;
            }
        }
    }
    int mode = STAGED;
    bool tuning = false;
    if (mapped) {
        const int pinned_mode = env_int("JGPT_B200_HOST_ZEROCOPY", -1);
        if (pinned_mode >= 0 && pinned_mode <= 2) {
            mode = pinned_mode;
        } else {
            if (p->host_tune_n != n || p->host_tune_layers != n_layers) {  // another shape: measure again
                p->host_tune_n = n, p->host_tune_layers = n_layers, p->host_tune_calls = 0, p->host_mode = -1;
                for (double &b : p->host_tune_best) b = 1e30;
            }
            // Which way wins is a property of the machine AT THAT MOMENT (other ranks load the same host fabric), so
            // the choice is kept under review: the first nine calls take turns (three samples each), and afterwards
            // two calls in every 128 go to the ways not in use; each way keeps a running average of what it cost.
            static const int order[3] = {ZEROCOPY, HYBRID, STAGED};
            const int c = p->host_tune_calls;
            if (c < 9) {
                mode = order[c % 3];
            } else {
                mode = p->host_mode;
                const int phase = (c - 9) % 128;
                if (phase == 126 || phase == 127) {
                    int others[2], k = 0;
                    for (int mth = 0; mth < 3; mth++)
                        if (mth != p->host_mode) others[k++] = mth;
                    mode = others[phase - 126];
                }
            }
            tuning = true;
        }
    }
    // The three index arrays travel as ONE copy out of the pool's page-locked staging area (three copies from
    // pageable memory cost ~15 us of driver staging per call; the previous call has synchronised, so the area is free).
    auto upload_indices = [&]() -> cudaError_t {
        memcpy(p->h_stage_i, seq_ids_host, sizeof(int) * (size_t)n);
        memcpy(p->h_stage_i + n, rope_pos_host, sizeof(int) * (size_t)n);
        memcpy(p->h_stage_i + 2 * (size_t)n, lens_host, sizeof(int) * (size_t)n);
        return cudaMemcpyAsync(dseq, p->h_stage_i, sizeof(int) * 3 * (size_t)n, cudaMemcpyHostToDevice, st);
    };
    const auto t_begin = std::chrono::steady_clock::now();
    auto finish = [&]() {
        if (!tuning) return;
        const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t_begin).count();
        double &avg = p->host_tune_best[mode];
        // first nine calls: the best of a way's three samples (the very first call of a way pays one-off set-up);
        // later: a running average that follows the machine's load
        if (p->host_tune_calls < 9) avg = std::min(avg, us);
        else avg = avg > 1e29 ? us : 0.75 * avg + 0.25 * us;
        p->host_tune_calls++;
        if (p->host_tune_calls >= 9) {
            int best = STAGED;
            for (int mth = 0; mth < 3; mth++)
                if (p->host_tune_best[mth] < p->host_tune_best[best]) best = mth;
            // change horses only for a clear gain: the samples are single wall-clock readings
            if (p->host_mode < 0 || p->host_tune_best[best] < 0.93 * p->host_tune_best[p->host_mode]) p->host_mode = best;
        }
    };
    if (mode == ZEROCOPY || mode == HYBRID) {
        JGPT_CUDA_TRY(upload_indices());
        const float *qi = static_cast<const float *>(dp[0]), *ki = static_cast<const float *>(dp[1]), *vi = static_cast<const float *>(dp[2]);
        if (mode == HYBRID) {
            JGPT_CUDA_TRY(cudaMemcpyAsync(dq, q_host, sizeof(float) * slab, cudaMemcpyHostToDevice, st));
            JGPT_CUDA_TRY(cudaMemcpyAsync(dk, k_host, sizeof(float) * slab, cudaMemcpyHostToDevice, st));
            JGPT_CUDA_TRY(cudaMemcpyAsync(dv, v_host, sizeof(float) * slab, cudaMemcpyHostToDevice, st));
            qi = dq, ki = dk, vi = dv;
        }
        rc = launch_attn_decode(p, layer0, n_layers, qi, ki, vi, dseq, drp, dlen, n, max_len, static_cast<float *>(dp[3]));
        if (rc) return rc;
        JGPT_CUDA_TRY(status_enqueue_read(p->ctx));
        JGPT_CUDA_TRY(cudaStreamSynchronize(st));
        finish();
        return status_check_after_sync(p->ctx, p, "jgpt_attn_decode_append_host");
    }
    JGPT_CUDA_TRY(upload_indices());
    // The layers of one call are independent, so the call is pipelined in groups of layers: while group g is
    // in the kernel, the inputs of group g+1 cross PCIe on the inbound copy engine and the outputs of group g-1
    // leave on the outbound one (three streams ordered by events).  One group = the plain path.
    constexpr int kMaxGroups = 4;  // events are allocated for up to four groups
    // Only the first group's inbound copy and the last group's outbound copy are exposed, but every launch costs
    // a fixed ~20 us.  Measured on the 12-layer step (us per step): one group 333, 4-4-4 301, 2-8-2 298,
    // 1-10-1 318, 1-5-5-1 325.  Default: a sixth of the layers first and last, the rest in between.
    // JGPT_B200_HOST_SPLIT = "a-b-c" (layers per group) overrides it, JGPT_B200_HOST_GROUPS = 1 selects the
    // unpipelined path.
    int sizes[kMaxGroups] = {n_layers, 0, 0, 0};
    int groups = 1;
    if (n_layers >= 3 && env_int("JGPT_B200_HOST_GROUPS", 3) > 1) {
        const int edge = std::max(1, n_layers / 6);
        groups = 3, sizes[0] = edge, sizes[1] = n_layers - 2 * edge, sizes[2] = edge;
    }
    if (const char *spec = getenv("JGPT_B200_HOST_SPLIT")) {
        int tmp[kMaxGroups] = {}, cnt = 0, sum = 0;
        for (const char *c = spec; *c && cnt < kMaxGroups;) {
            const int v = atoi(c);
            if (v <= 0) break;
            tmp[cnt++] = v, sum += v;
            while (*c && *c != '-') c++;
            if (*c == '-') c++;
        }
        if (cnt >= 1 && sum == n_layers) {
            groups = cnt;
            for (int g = 0; g < kMaxGroups; g++) sizes[g] = tmp[g];
        }
    }
    if (groups == 1) {
        JGPT_CUDA_TRY(cudaMemcpyAsync(dq, q_host, sizeof(float) * slab, cudaMemcpyHostToDevice, st));
        JGPT_CUDA_TRY(cudaMemcpyAsync(dk, k_host, sizeof(float) * slab, cudaMemcpyHostToDevice, st));
        JGPT_CUDA_TRY(cudaMemcpyAsync(dv, v_host, sizeof(float) * slab, cudaMemcpyHostToDevice, st));
        rc = launch_attn_decode(p, layer0, n_layers, dq, dk, dv, dseq, drp, dlen, n, max_len, dout);
        if (rc) return rc;
        JGPT_CUDA_TRY(cudaMemcpyAsync(out_host, dout, sizeof(float) * slab, cudaMemcpyDeviceToHost, st));
        JGPT_CUDA_TRY(status_enqueue_read(p->ctx));
        JGPT_CUDA_TRY(cudaStreamSynchronize(st));
        finish();
        return status_check_after_sync(p->ctx, p, "jgpt_attn_decode_append_host");
    }
    if (!p->s_in) {
        JGPT_CUDA_TRY(cudaStreamCreateWithFlags(&p->s_in, cudaStreamNonBlocking));
        JGPT_CUDA_TRY(cudaStreamCreateWithFlags(&p->s_out, cudaStreamNonBlocking));
        for (int g = 0; g < kMaxGroups; g++) {
            JGPT_CUDA_TRY(cudaEventCreateWithFlags(&p->ev_in[g], cudaEventDisableTiming));
            JGPT_CUDA_TRY(cudaEventCreateWithFlags(&p->ev_done[g], cudaEventDisableTiming));
        }
        JGPT_CUDA_TRY(cudaEventCreateWithFlags(&p->ev_start, cudaEventDisableTiming));
    }
    // the staging buffers may still be in use by earlier work on the main stream
    JGPT_CUDA_TRY(cudaEventRecord(p->ev_start, st));
    JGPT_CUDA_TRY(cudaStreamWaitEvent(p->s_in, p->ev_start, 0));
    const size_t per_layer = (size_t)n * p->heads * p->dhead;
    int l0 = 0;
    for (int g = 0; g < groups; g++) {
        const int nl = sizes[g];
        const size_t off = (size_t)l0 * per_layer, cnt = (size_t)nl * per_layer;
        JGPT_CUDA_TRY(cudaMemcpyAsync(dq + off, q_host + off, sizeof(float) * cnt, cudaMemcpyHostToDevice, p->s_in));
        JGPT_CUDA_TRY(cudaMemcpyAsync(dk + off, k_host + off, sizeof(float) * cnt, cudaMemcpyHostToDevice, p->s_in));
        JGPT_CUDA_TRY(cudaMemcpyAsync(dv + off, v_host + off, sizeof(float) * cnt, cudaMemcpyHostToDevice, p->s_in));
        JGPT_CUDA_TRY(cudaEventRecord(p->ev_in[g], p->s_in));
        JGPT_CUDA_TRY(cudaStreamWaitEvent(st, p->ev_in[g], 0));
        rc = launch_attn_decode(p, layer0 + l0, nl, dq + off, dk + off, dv + off, dseq, drp, dlen, n, max_len, dout + off, -1, n_layers);
        if (rc) return rc;
        JGPT_CUDA_TRY(cudaEventRecord(p->ev_done[g], st));
        JGPT_CUDA_TRY(cudaStreamWaitEvent(p->s_out, p->ev_done[g], 0));
        JGPT_CUDA_TRY(cudaMemcpyAsync(out_host + off, dout + off, sizeof(float) * cnt, cudaMemcpyDeviceToHost, p->s_out));
        l0 += nl;
    }
    JGPT_CUDA_TRY(status_enqueue_read(p->ctx));
    JGPT_CUDA_TRY(cudaStreamSynchronize(p->s_out));
    JGPT_CUDA_TRY(cudaStreamSynchronize(st));
    finish();
    return status_check_after_sync(p->ctx, p, "jgpt_attn_decode_append_host");
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------
// Decode attention with its split-K scratch in a fixed, library-owned device array.
//
// jgpt_attn_decode sizes its split-K scratch (partial softmax states + arrival counters) with
// cudaMalloc the first time a launch needs more than it has.  Some hosts cannot tolerate that on the
// generation path: a process that has already handed the whole GPU to its own buffers (a trainer
// that samples text between optimizer steps with the device full, a server that sizes its KV pool to
// whatever memory is left) can see that late cudaMalloc fail, and any cudaMalloc/cudaFree stalls the
// device while it runs.  This variant never calls an allocator: its scratch is the array below.
//
// When the memory is taken: CUDA loads a module lazily, so the device memory of the array is
// reserved (and the kernel's code loaded) the first time this translation unit is used on a device --
// the set-up below -- not when the shared library is opened.  A call with n == 0 runs only that
// set-up, so a host can do it before it commits the rest of the GPU.  From then on every GPU that ran
// the set-up holds the array until the process exits.
//
// Limits, stated: kStaticPartialFloats fp32 partial words (4 MiB) and kStaticTickets counters
// (16 KiB) per device.  One layer per call.  Requests that need more are rejected.
// ------------------------------------------------------------------------------------------------
namespace jgpt {

constexpr size_t kStaticPartialFloats = size_t(1) << 20;  // 4 MiB of (m, l, o[dhead]) partials
constexpr size_t kStaticTickets = 4096;                   // arrival counters, one per (sequence row, head group)

// In host code this name is only a handle for cudaGetSymbolAddress, never an address to pass to a kernel.
static __device__ __align__(256) float g_decode_static_scratch[kStaticPartialFloats + kStaticTickets];

constexpr int kStaticMaxDevices = 64;
static float *g_static_scratch_addr[kStaticMaxDevices] = {};  // per device, resolved by the set-up
static std::mutex g_static_scratch_mu;                        // the table above and the opt-in below

// Once per device, with that device current: resolves the array's device address and loads the kernel
// (both trigger the lazy module load that reserves the array's memory).
static int32_t static_scratch_setup(const Pool *p, float **partials, int **tickets) {
    const Ctx *c = p->ctx;
    JGPT_REQUIRE(c->device >= 0 && c->device < kStaticMaxDevices, JGPT_ERR_UNSUPPORTED,
                 "device index %d is beyond the %d devices the static scratch table covers", c->device, kStaticMaxDevices);
    std::lock_guard<std::mutex> lock(g_static_scratch_mu);
    if (!g_static_scratch_addr[c->device]) {
        void *addr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&addr, g_decode_static_scratch);
        if (e != cudaSuccess || !addr)
            return fail(e == cudaErrorMemoryAllocation ? JGPT_ERR_OUT_OF_MEMORY : JGPT_ERR_CUDA,
                        "cudaGetSymbolAddress(static decode scratch) on device %d: %s", c->device, cudaGetErrorString(e));
        cudaError_t a = cudaSuccess;
        switch (p->dhead) {
            case 4: a = decode_opt_in_smem(attn_decode_kernel<4, false>, 0, c->device); break;
            case 8: a = decode_opt_in_smem(attn_decode_kernel<8, false>, 4, c->device); break;
            case 16:
                a = decode_opt_in_smem(attn_decode_kernel<16, false, false>, 8, c->device);
                if (a == cudaSuccess) a = decode_opt_in_smem(attn_decode_kernel<16, false, true>, 10, c->device);
                break;
            case 32: a = decode_opt_in_smem(attn_decode_kernel<32, false>, 12, c->device); break;
            default: break;
        }
        if (a != cudaSuccess) return fail(JGPT_ERR_CUDA, "static decode scratch set-up on device %d: %s", c->device, cudaGetErrorString(a));
        g_static_scratch_addr[c->device] = static_cast<float *>(addr);
    }
    *partials = g_static_scratch_addr[c->device];
    *tickets = reinterpret_cast<int *>(g_static_scratch_addr[c->device] + kStaticPartialFloats);
    return JGPT_OK;
}

static int32_t launch_attn_decode_static(Pool *p, int layer, const float *q, const int *seq_ids, const int *rope_pos,
                                         const int *lens, int n, int max_len, float *out) {
    DecodeParams P;
    memset(&P, 0, sizeof(P));
    const int DH = p->dhead;
    P.kv = p->kv, P.table = p->d_table, P.rope = p->d_rope;
    P.q = q, P.k_new = nullptr, P.v_new = nullptr, P.out = out;
    P.seq_ids = seq_ids, P.rope_pos = rope_pos, P.lens = lens;
    P.status = p->ctx->d_status;
    P.n = n, P.H = p->heads, P.layer0 = layer, P.n_layers = 1, P.mbs = p->max_blocks_per_seq;
    P.n_blocks = p->n_blocks, P.max_seqs = p->max_seqs, P.max_positions = p->max_positions;
    // the launch shape of a one-layer jgpt_attn_decode whose launches do not overlap (small batches get lighter CTAs)
    P.stream_hint = p->stream_hint;
    P.HG = pick_head_group(p->heads, DH, p->head_group, (long long)n, 2ll * p->ctx->sm_count);
    P.n_hg = p->heads / P.HG;
    const int max_blocks = std::min(p->max_blocks_per_seq, (max_len + kBlockTokens - 1) / kBlockTokens);
    P.chunk_blocks = p->chunk_blocks > 0 ? p->chunk_blocks : pick_chunk_blocks(p, (long long)n * P.n_hg, max_blocks);
    P.max_len = max_blocks * kBlockTokens;
    P.max_chunks = std::max(1, (max_blocks + P.chunk_blocks - 1) / P.chunk_blocks);
    P.stages = p->stages > 0 ? p->stages : 4;
    P.scale_log2e = (1.0f / sqrtf((float)DH)) * 1.4426950408889634f;
    const long long items = (long long)n * P.n_hg * P.max_chunks;
    JGPT_REQUIRE(items < (1ll << 31), JGPT_ERR_INVALID_ARGUMENT, "too many work items (%lld)", items);
    P.n_items = (int)items;
    int32_t rc = static_scratch_setup(p, &P.partials, &P.tickets);
    if (rc) return rc;
    if (P.max_chunks > 1) {
        // Only a split sequence touches the scratch; an unsplit launch needs none of it and has no size limit.
        const unsigned long long need_partials = (unsigned long long)n * P.max_chunks * p->heads * (DH + 2);
        const unsigned long long need_tickets = (unsigned long long)n * P.n_hg;
        JGPT_REQUIRE(need_partials <= kStaticPartialFloats && need_tickets <= kStaticTickets, JGPT_ERR_INVALID_ARGUMENT,
                     "request needs %llu partial words and %llu counters; the static scratch holds %llu and %llu "
                     "(lower n or max_len, or use jgpt_attn_decode)",
                     need_partials, need_tickets, (unsigned long long)kStaticPartialFloats,
                     (unsigned long long)kStaticTickets);
        // The array keeps whatever the previous call left.  Partials are always written before they are read;
        // the counters must start at zero (they reset themselves, but not if an earlier launch gave up half way).
        JGPT_CUDA_TRY(cudaMemsetAsync(P.tickets, 0, sizeof(int) * need_tickets, p->ctx->stream));
    }
    const bool mma = DH == 16 && tensor_consumers(p, P.HG, false, n);
    const int n_cons = mma ? consumer_threads<true>(P.HG) : consumer_threads<false>(P.HG);
    const int threads = n_cons + 32;
    const size_t smem = (size_t)P.HG * 2 * kBlockTokens * DH * 2 * P.stages;
    void (*kern)(const DecodeParams) = nullptr;
    switch (DH) {
        case 4: kern = attn_decode_kernel<4, false>; break;
        case 8: kern = attn_decode_kernel<8, false>; break;
        case 16: kern = mma ? attn_decode_kernel<16, false, true> : attn_decode_kernel<16, false, false>; break;
        case 32: kern = attn_decode_kernel<32, false>; break;
        default: return fail(JGPT_ERR_UNSUPPORTED, "dhead %d not supported", DH);
    }
    kern<<<P.n_items, threads, smem, p->ctx->stream>>>(P);
    JGPT_CUDA_TRY(cudaGetLastError());
    return JGPT_OK;
}

}  // namespace jgpt

extern "C" int32_t jgpt_attn_decode_static_scratch(jgpt_kvpool pool, int32_t layer, const float *q_dev,
                                                   const int32_t *seq_ids_dev, const int32_t *rope_pos_dev,
                                                   const int32_t *lens_dev, int32_t n, int32_t max_len, float *out_dev) {
    Pool *p = pool_registry().get(pool);
    JGPT_REQUIRE(p, JGPT_ERR_BAD_HANDLE, "bad kvpool handle");
    JGPT_REQUIRE(!p->layered, JGPT_ERR_UNSUPPORTED, "not available on a layered decoder's pool");
    JGPT_CUDA_TRY(make_current(p->ctx));
    JGPT_REQUIRE(layer >= 0 && layer < p->layers, JGPT_ERR_OUT_OF_RANGE, "layer %d outside [0,%d)", layer, p->layers);
    JGPT_REQUIRE(p->dhead == 4 || p->dhead == 8 || p->dhead == 16 || p->dhead == 32, JGPT_ERR_UNSUPPORTED,
                 "dhead %d not supported", p->dhead);
    if (n == 0) {  // set-up only: take the array's memory and load the kernel now, launch nothing
        float *partials;
        int *tickets;
        return static_scratch_setup(p, &partials, &tickets);
    }
    JGPT_REQUIRE(n > 0 && q_dev && seq_ids_dev && rope_pos_dev && lens_dev && out_dev, JGPT_ERR_INVALID_ARGUMENT,
                 "null pointer or negative count");
    JGPT_REQUIRE(max_len >= 1, JGPT_ERR_INVALID_ARGUMENT, "max_len must be >= 1");
    return launch_attn_decode_static(p, layer, q_dev, seq_ids_dev, rope_pos_dev, lens_dev, n, max_len, out_dev);
}
