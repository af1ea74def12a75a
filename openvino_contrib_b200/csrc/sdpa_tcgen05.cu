// Fused attention for prefill on the 5th-generation tensor core: S = Q K^T and O = P V as tcgen05.mma with
// accumulators in tensor memory, online softmax in registers.  f16 / bf16, grouped-query heads, D = Dv = 128 (dense
// tensors also 64).
// Three front ends share one kernel body (template parameter kMode):
//   0 dense  (ScaledDotProductAttention): Q, K, V are [B, H, S, 128] tensors, causal or unmasked; K/V tiles are
//     staged by TMA;
//   1 paged, de-quantising in the kernel (PagedAttentionExtension, sequences with two or more new tokens): Q rows
//     come from the step's [tokens, Hq*128] matrix, K/V from the u8 block pool through the block table - a producer
//     warpgroup de-quantises 128-token tiles ((code - zp) * scale in float32, rounded once to f16: queries, keys,
//     values and P are all f16 in the paged modes) straight into the swizzled shared-memory layout the tensor core
//     reads;
//   2 paged, gathered: paged_gather_kernel has de-quantised the contexts of the step's multi-token sequences once
//     into an f16 scratch (a row range per sequence), and K/V tiles are staged from there by TMA like dense ones.
//     Taken when the caller passes the scheduler's bound on those contexts (b2a_paged_desc.prefill_kv_tokens).
//   In the paged modes query token i of a sequence sees cache positions 0 .. past_len + i, or only the last
//   `sliding_window` of them: an item then starts at the first key tile that any of its rows still sees, and key
//   tiles that begin below the window of a tile's last row are masked at their low edge like diagonal tiles at
//   their high edge.
//
// Work is cut into items: TWO 128-row query tiles of one KV head, walked over the keys 128 at a time.  CTAs are
// persistent (one per SM; mode 1 keeps one item per CTA): the items, heaviest first, are dealt in snake order.
//   warps 0-3   softmax of tile A: thread = query row = TMEM lane.  Reads S (tcgen05.ld) and gives its place up, keeps the
//               running max and sum, writes P_A = exp2(S*c - m) as 16-bit pairs into P_A's columns (tcgen05.st) and
//               signals the PV issuer; rescales O_A in TMEM when the maximum moved; finally normalises O_A and stores
//               it, a thread its row (heads sharded over several ranks: through a staging slab per warp, [32 x 64] and
//               one TMA tensor store per slab and rank).
//   warps 4-7   the same for tile B.
//   warp  8     TMA producer (one lane): the Q tiles of an item as soon as the previous item's last QK^T has
//               completed, and (modes 0, 2) K_j and V_j into two-stage rings that run on across items, K a step ahead.
//   warp  9     issues S = Q_X K_j^T (A and B from shared memory, K-major, 128-byte swizzle), in turn A(0) B(0) A(1) B(1)
//               ..  S has ONE place of 128 columns: a turn's QK is issued as soon as the turn before has its scores in
//               registers, which is long before its own softmax warps come for them.
//   warp 10     issues O_X += P_X(j) V_j (A from TMEM, B from shared memory, MN-major) when P_X is ready.
//   warp 11     completes the service warpgroup; in mode 2 with bf16 queries it and the producer's warp convert the Q
//               tiles to f16 in shared memory, a tile each.
//   warps 12-15 mode 1 only: the de-quantising K/V producers, which convert the Q tiles there.
// TMEM: S 128 columns, P_A and P_B 64 each, O_A and O_B 128 each: all 512 (allocated by warp 9).
// Why S is shared and QK and PV have issuers of their own: with S and P of a tile in one place a step is the chain softmax ->
// PV -> QK -> softmax (1750 + 256 + 512 cycles and three trips over barriers), and one issuer, which stands still while the
// tensor core's short queue is full and pays about 130 cycles for every barrier it looks at, leaves the tensor core idle
// for a third of a step.  Causal prefill of 4 x 4096 tokens, 32/8 heads, bf16: 785 thousand cycles a launch before, 695 now; in
// a loop of passes, where the power limit lowers the clock, 542 us before and 509 now.  Three prompts of 400 to 1100 tokens
// behind caches of up to 3000: 92.2 -> 86.9 us a step.  (Issued by one warp on a shared S: 785 thousand cycles.  P's first half
// sent ahead of the second, P kept in registers until PV(j-1) has read the columns, the maximum of half a row while the
// other half is loaded, two PV issuers: no gain.  The special-function unit, where the exponentials of both tiles go,
// is busy 70 % of the launch's cycles now, the tensor pipe 67 %.)
// Where that does not pay, S_X has a place per tile, P lies over it, and one lane of warp 9 issues PV_A(j), QK_A(j+1), PV_B(j),
// QK_B(j+1), PV in two halves as those of P arrive: calls that hold P in several pieces (kSplitP: no columns left for a P of its
// own), in-kernel de-quantisation (mode 1, bound by its producers) and items of one key step (kOwnS).
// The two tiles are consecutive entries of the list (row block, query head of the group), query heads fastest, so
// with an even group size both tiles cover the same rows of two heads that share K/V, and the causal structure of
// the pair is identical.
//
// The maximum used for P is allowed to lag: O and the sum are rescaled only when some row's maximum grew by more
// than 2^8, so P stays below 256 and the result is exact after the final division.
//
// Every mbarrier wait is bounded (tcgen05.cuh); on a timeout the CTA raises an abort flag, all roles leave their
// loops, outstanding copies and MMAs are drained with bounded waits, TMEM is freed and the status word gets
// B2A_DEV_TIMEOUT.  All barrier phases are derived from running counts (K/V ring position, steps of a tile, Q tiles
// loaded) so that they carry over from one item to the next.
#include <algorithm>

#include "launch.cuh"
#include "tcgen05.cuh"

namespace b2a {
namespace {

using namespace tc;

constexpr int kBM = 128;             // query rows per tile = TMEM lanes
constexpr int kBN = 128;             // keys per step
constexpr int kHeadDim = 128;
constexpr int kPanel = 128 * 128;    // bytes of one [128 rows x 64 elements] swizzled panel
constexpr int kThreadsDense = 384;   // 3 warpgroups: softmax A, softmax B, {producer, QK issuer, PV issuer, one more}
constexpr int kThreadsPaged = 512;   // plus the de-quantising producer warpgroup
constexpr int kNumBars = 28;
constexpr int kStageOut = 8 * 4096;  // epilogue staging: one [32 rows x 64 elements] slab per softmax warp
constexpr int smem_bytes(int tile) { return 6 * tile + kStageOut + 1024 /* alignment slack */ + 256 /* barriers, TMEM slot, abort flag */; }
constexpr float kLazyThreshold = 8.0f;  // log2 units
constexpr int kCacheChunk = 16 * (kHeadDim + 4);  // bytes of one (block, KV head) chunk of the u8 pool

enum Bar { Q_FULL = 0, K_FULL = 2, K_EMPTY = 4, V_FULL = 6, V_EMPTY = 8, S_FULL = 10, P_READY = 12, O_DONE = 14, DRAIN = 16, P_HALF = 17, Q_CONV = 19, Q_EMPTY = 21,
           HALVES = 23, S_FREE = 27 };

// n / d for 0 <= n < 2^31 by one multiplication: mul = ceil(2^(31 + shift) / d) with shift = ceil(log2 d) errs by less than
// n / 2^(31 + shift) < 1 / d (Granlund and Montgomery's division by an invariant).  A role works out its place from the
// item's number at every item, and the run-time divisions took 1500 cycles of the issuing thread's.
struct FastDiv {
    uint32_t mul, shift, d;
};
FastDiv fast_div(int d) {
    FastDiv f{0, 0, static_cast<uint32_t>(d)};
    while ((1u << f.shift) < f.d) ++f.shift;
    if (f.d > 1) f.mul = static_cast<uint32_t>(((1ull << (31 + f.shift)) + f.d - 1) / f.d);
    return f;
}
__device__ __forceinline__ int div_by(int n, const FastDiv& f) {
    return f.d == 1 ? n : static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * f.mul) >> (31 + f.shift));
}

struct TcParams {
    int B, Hq, Hkv, G, Sq, Skv;
    FastDiv div_g, div_hkv, div_streams;  // by G, Hkv, B * Hkv
    int64_t out_strides[3];  // dense output: batch, head, row, in elements
    int out_wide;            // every output row starts on a 32-byte boundary
    int causal;
    int window;  // paged modes: a query at position p sees keys p - window + 1 .. p (0: all of them)
    float scale_log2;
    // dense mode with an attention mask (u8, non-zero keeps; or additive, the tensors' 16-bit type): logical
    // [B, Hq, Sq, Skv] with element strides mask_strides (0 on broadcast dimensions)
    const uint8_t* mask;
    int mask_kind;
    int64_t mask_strides[4];
    int32_t* status;
    // paged mode
    const uint8_t* k_cache;
    const uint8_t* v_cache;
    PagedTables t;
    void* out;        // [tokens, Hq*128]
    const int* plan;  // work list built by paged_tc_plan_kernel: header, then entries of kPlanEntryInts
};

// Output side of a head-sharded launch (world == 0: single GPU, TcParams::out is the output).
struct TcPeers {
    CUtensorMap out_map[kMaxShardWorld];  // [rank]: that rank's [B, Hq_total, Sq, 128] output buffer
    int32_t* flags[kMaxShardWorld];
    int32_t* done_counter;
    int world, rank, head_offset;
    int32_t step;
    int light_first;  // a CTA takes its items lightest first: their output tiles are on the wire while the heavy ones compute
};

// Work list of the paged front end.  Lengths live on the device, so a one-CTA kernel turns them into the list of
// (sequence, tile pair) items that have work; the attention grid is then sized by a host-side bound on the item
// count (exact when the caller passes the scheduler's hint) instead of max_q_len x num_seqs, which for a step with
// a few long prefills and many decode sequences would be almost all empty CTAs.
constexpr int kPlanHeaderInts = 4;  // [0] items in the list (per KV head), [1] CTAs of the attention kernel that take items
// An entry carries all that the attention kernel's warps have to know about the item, so that starting one costs them one
// trip to memory instead of a chain of table lookups: {sequence, first token, new tokens (0: tables inconsistent), past
// length}, {tile pair, first scratch row of the sequence, 0, 0}.
constexpr int kPlanEntryInts = 8;
// A mixed step runs its prefill rows (tensor-bound) and its decode rows (HBM-bound) at the same time: the attention
// kernel keeps only as many SMs as its share of the step's work needs and the decode kernel, launched as soon as
// those CTAs are seated, takes the rest (and the others as they come free).  The share is worked out here from the
// tables: item-steps of the work list against cached bytes of the one-token sequences, each divided by what one SM
// gets through per microsecond (measured on a step of eight 1024-token prefills beside 120 decode sequences: about
// 2.8 us per item-step of two 128 x 128 tiles over 128 keys at the efficiency of short items; about 52 bytes per
// nanosecond of u8 cache per SM while the SMs that decode are a minority - a sweep of the share on that step was
// flat within 5 % between 0.59 and 0.70 and best at 0.59).
constexpr float kUsPerItemStep = 2.8f;
constexpr float kDecodeBytesPerNsPerSm = 52.f;
constexpr float kHbmBytesPerNs = 6500.f;
// With `owner` given the kernel also lays out the gathered K/V scratch: every multi-token sequence gets a row range
// of roundup(context, 128) rows (kv_base[seq]; allocation order is whatever the atomics make it), and owner[g] names
// the sequence that 128-row group g belongs to (-1: nobody), which is how paged_gather_kernel finds its work.
__global__ void __launch_bounds__(256) paged_tc_plan_kernel(const PagedTables t, const int G, const int Hkv,
                                                            const int capacity, int* plan, int32_t* status,
                                                            int* kv_base, int* owner, const int owner_groups,
                                                            const int attention_ctas, const int share_with_decode) {
    // The list is sorted by weight (key steps of the pair's later tile, clamped to 255), heaviest first: a counting
    // sort in three passes over the sequences - histogram, bucket offsets, scatter.  Sequences are looked at 256 at a time,
    // a thread each, and the tile pairs of those with several new tokens are spread over the lanes of a warp.
    constexpr int kBuckets = 256;
    __shared__ int s_hist[kBuckets], s_count, s_groups, s_steps;
    __shared__ int c_tok[256], c_qlen[256], c_past[256];
    __shared__ unsigned char c_ok[256];
    __shared__ unsigned long long s_decode_blocks;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Everything that only reads the step's tables - the histogram of the weights, the counts, the bucket offsets -
    // is done while the kernel in front (the step's store) drains; what this kernel WRITES (list, scratch layout)
    // may still be read by earlier kernels, so the writes come after the wait.  (The tables of a step exist before
    // its kernels are launched.)
    for (int i = threadIdx.x; i < kBuckets; i += blockDim.x) s_hist[i] = 0;
    if (threadIdx.x == 0) {
        s_count = s_groups = s_steps = 0;
        s_decode_blocks = 0ull;
    }
    auto weight = [&](int past, int qlen, int pair) {
        const int tiles = ((qlen + 127) / 128) * G;
        const int tile = min(2 * pair + 1, tiles - 1);  // the pair's later tile
        const int keys = min(past + qlen, past + (tile / G) * 128 + 128);
        return min(kBuckets - 1, max(0, (keys + 127) / 128));
    };
    auto pairs_of = [&](int qlen) { return (((qlen + 127) / 128) * G + 1) / 2; };
    // this thread's sequence of the 256 from s0; returns the blocks of its context if it is a one-token sequence
    auto load_chunk = [&](int s0) -> int {
        const int s = s0 + threadIdx.x;
        int tok0 = 0, qlen = 0, past = 0, ok = 0;
        if (s < t.num_seqs) {
            tok0 = t.subsequence_begins[s];
            qlen = t.subsequence_begins[s + 1] - tok0;
            past = t.past_lens[s];
            const int have = t.block_indices_begins[s + 1] - t.block_indices_begins[s];
            ok = past >= 0 && tok0 >= 0 && tok0 + qlen <= t.num_tokens && (past + qlen + 15) / 16 <= have;
        }
        c_tok[threadIdx.x] = tok0;
        c_qlen[threadIdx.x] = qlen >= 2 ? qlen : 0;
        c_past[threadIdx.x] = past;
        c_ok[threadIdx.x] = static_cast<unsigned char>(ok);
        return qlen == 1 && past >= 0 ? past / t.block_size + 1 : 0;
    };
    int steps = 0;
    long long decode_blocks = 0;
    for (int s0 = 0; s0 < t.num_seqs; s0 += 256) {
        if (s0 > 0) __syncthreads();  // the chunk before has been read
        decode_blocks += load_chunk(s0);
        __syncthreads();
        for (int i = warp; i < min(256, t.num_seqs - s0); i += 8) {
            const int qlen = c_qlen[i];
            if (qlen == 0) continue;
            const int past = max(0, c_past[i]), pairs = pairs_of(qlen);
            if (lane == 0) atomicAdd(&s_count, pairs);
            for (int k = lane; k < pairs; k += 32) {
                const int w = weight(past, qlen, k);
                atomicAdd(&s_hist[w], 1);
                steps += w;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        steps += __shfl_xor_sync(0xffffffffu, steps, o);
        decode_blocks += __shfl_xor_sync(0xffffffffu, decode_blocks, o);
    }
    if (lane == 0 && steps > 0) atomicAdd(&s_steps, steps);
    if (lane == 0 && decode_blocks > 0) atomicAdd(&s_decode_blocks, static_cast<unsigned long long>(decode_blocks));
    __syncthreads();
    {  // bucket w starts after all heavier buckets: one bucket per thread, lightest in the last
        static_assert(kBuckets == 256, "a bucket per thread");
        __shared__ int s_warp[kBuckets / 32];
        const int n = s_hist[kBuckets - 1 - threadIdx.x];
        int upto = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += x;
        }
        if (lane == 31) s_warp[warp] = upto;
        __syncthreads();
        for (int w = 0; w < warp; ++w) upto += s_warp[w];
        s_hist[kBuckets - 1 - threadIdx.x] = upto - n;
    }
    grid_dependency_wait();
    grid_launch_dependents();
    if (owner != nullptr)
        for (int g = threadIdx.x; g < owner_groups; g += blockDim.x) owner[g] = -1;
    __syncthreads();
    for (int s0 = 0; s0 < t.num_seqs; s0 += 256) {
        if (t.num_seqs > 256) {  // (a single chunk is still there)
            __syncthreads();
            load_chunk(s0);
            __syncthreads();
        }
        for (int i = warp; i < min(256, t.num_seqs - s0); i += 8) {
            const int s = s0 + i, qlen = c_qlen[i];
            if (qlen == 0) continue;
            const int past = max(0, c_past[i]), pairs = pairs_of(qlen);
            int base = 0;
            if (owner != nullptr) {  // the sequence's rows of the scratch
                const int groups = c_past[i] < 0 ? 0 : (past + qlen + 127) / 128;
                if (lane == 0) base = atomicAdd(&s_groups, groups);
                base = __shfl_sync(0xffffffffu, base, 0);
                for (int g = lane; g < groups; g += 32)
                    if (base + g < owner_groups) owner[base + g] = s;
                base *= 128;
                if (lane == 0) kv_base[s] = base;
            }
            // inconsistent tables (reported): the sequence's items are empty
            const bool ok = c_ok[i] != 0;
            if (!ok && lane == 0) report(status, B2A_DEV_BAD_LEN);
            const int4 rec0 = make_int4(s, c_tok[i], ok ? qlen : 0, past);
            for (int k = lane; k < pairs; k += 32) {
                const int at = atomicAdd(&s_hist[weight(past, qlen, k)], 1);
                if (at < capacity) {
                    int4* rec = reinterpret_cast<int4*>(plan + kPlanHeaderInts) + 2 * at;
                    rec[0] = rec0;
                    rec[1] = make_int4(k, base, 0, 0);
                }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        plan[0] = min(s_count, capacity);
        if (s_count > capacity) {  // the caller's prefill_row_blocks was too small
            report(status, B2A_DEV_BAD_LEN);
            plan[0] = 0;  // a truncated sorted list would drop arbitrary pairs: compute nothing instead
        }
        if (owner != nullptr && s_groups > owner_groups) {        // the caller's prefill_kv_tokens was too small
            report(status, B2A_DEV_BAD_LEN);
            plan[0] = 0;  // nothing is computed from a scratch that does not hold every sequence
        }
        // how many of the attention kernel's CTAs take items (the others leave at once and free their SMs)
        int ctas = attention_ctas;
        if (share_with_decode && s_decode_blocks > 0ull && attention_ctas > 1) {
            const float prefill_sm_us = static_cast<float>(s_steps) * Hkv * kUsPerItemStep;
            const float decode_bytes = static_cast<float>(s_decode_blocks) * Hkv * 2.f * kCacheChunk;
            const float decode_sm_us = decode_bytes / (kDecodeBytesPerNsPerSm * 1000.f);
            const float share = prefill_sm_us / (prefill_sm_us + decode_sm_us);
            ctas = static_cast<int>(ceilf(share * attention_ctas));
            // the decode rows cannot use more SMs than it takes to saturate the memory system
            const int decode_max = static_cast<int>(kHbmBytesPerNs / kDecodeBytesPerNsPerSm);
            ctas = max(ctas, attention_ctas - decode_max);
            ctas = min(max(ctas, 1), attention_ctas);
        }
        plan[1] = ctas;
    }
}

__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// two float32 lanes in one 64-bit register pair, for the packed f32x2 arithmetic of sm_100
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    if constexpr (kBf16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&v);
    } else {
        const __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&v);
    }
}
// 64 bytes of an output row, in 32-byte stores where the row starts on such a boundary (else 16)
__device__ __forceinline__ void store_64_bytes(uint16_t* dst, const uint32_t (&w)[16], bool wide) {
    if (wide) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + 16 * h), "r"(w[8 * h]), "r"(w[8 * h + 1]),
                         "r"(w[8 * h + 2]), "r"(w[8 * h + 3]), "r"(w[8 * h + 4]), "r"(w[8 * h + 5]), "r"(w[8 * h + 6]), "r"(w[8 * h + 7])
                         : "memory");
    } else {
#pragma unroll
        for (int h = 0; h < 4; ++h) reinterpret_cast<uint4*>(dst)[h] = make_uint4(w[4 * h], w[4 * h + 1], w[4 * h + 2], w[4 * h + 3]);
    }
}
// two values rounded to f16, magnitudes beyond its range to the largest finite one
__device__ __forceinline__ uint32_t pack_f16_finite(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
template <bool kBf16>
__device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi) {
    if constexpr (kBf16) {
        lo = __uint_as_float(w << 16);
        hi = __uint_as_float(w & 0xffff0000u);
    } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
        lo = f.x;
        hi = f.y;
    }
}
// One value of an additive mask, in log2 units.  Finite values end at kMaskFloor (the lowest bf16 times log2(e) would
// overflow): a row whose keys all carry the type's lowest value stays uniform over them, as in attn_generic_kernel.
constexpr float kMaskFloor = -1.0e30f;
__device__ __forceinline__ float mask_log2(float f) {
    const float v = f * kLog2e;
    return v < kMaskFloor && f != -INFINITY ? kMaskFloor : v;
}
template <bool kBf16>
__device__ __forceinline__ float mask_log2(const uint8_t* row, int64_t at) {
    const uint16_t bits = reinterpret_cast<const uint16_t*>(row)[at];
    return mask_log2(kBf16 ? __uint_as_float(static_cast<uint32_t>(bits) << 16) : __half2float(__ushort_as_half(bits)));
}
// time-bounded wait that ignores the abort flag: used only to drain work already in flight
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > kWaitTicks) return;
    }
}

// De-quantise the 16 codes of one 16-byte piece: (code - zp) * scale in float32, as the decode kernel and the CPU
// restatement compute it - the difference is exact in float32 (an integer below 256 minus an f16 value), the product
// rounds once - and then one rounding to f16, the operand format of the tensor core.  0x4B0000XX is 2^23 + XX as a
// float, so a byte permute and one exact subtraction turn a code into its float value.  scale and zp arrive as the
// raw f16 bits the cache stores; a zero scale with zero codes (positions past the context) gives exact zeros.
__device__ __forceinline__ void dequant16_f16(uint4 w, unsigned short scale_bits, unsigned short zp_bits, uint32_t (&outw)[8]) {
    const uint32_t words[4] = {w.x, w.y, w.z, w.w};
    const float sc = __half2float(__ushort_as_half(scale_bits));
    const float zp = __half2float(__ushort_as_half(zp_bits));
    constexpr float k2p23 = 8388608.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float c0 = __uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7650)) - k2p23;
        const float c1 = __uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7651)) - k2p23;
        const float c2 = __uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7652)) - k2p23;
        const float c3 = __uint_as_float(__byte_perm(words[i], 0x4B000000u, 0x7653)) - k2p23;
        outw[2 * i] = pack2<false>((c0 - zp) * sc, (c1 - zp) * sc);
        outw[2 * i + 1] = pack2<false>((c2 - zp) * sc, (c3 - zp) * sc);
    }
}
// ... and store them as two 16-byte chunks of a swizzled shared-memory tile row
__device__ __forceinline__ void dequant_piece_f16(uint4 w, unsigned short scale_bits, unsigned short zp_bits,
                                                  uint8_t* row, int c16, int token) {
    uint32_t outw[8];
    dequant16_f16(w, scale_bits, zp_bits, outw);
    // the piece covers d = 16*c16 .. +15: chunks 2*c16 and 2*c16+1 of the 128-wide row, 8 chunks per 64-wide panel
    uint8_t* panel = row + (c16 >> 2) * kPanel;
    const int cp = (2 * c16) & 7;
    *reinterpret_cast<uint4*>(panel + ((cp ^ (token & 7)) << 4)) = make_uint4(outw[0], outw[1], outw[2], outw[3]);
    *reinterpret_cast<uint4*>(panel + (((cp + 1) ^ (token & 7)) << 4)) = make_uint4(outw[4], outw[5], outw[6], outw[7]);
}

// De-quantise the contexts of the step's multi-token sequences into the f16 scratch [Hkv][rows][128] (K and V each):
// one CTA per (kGatherRows scratch rows, KV head), thread = (token, 16-byte piece) of K and of V in every block of sixteen.
// A chain of dependent loads (owner, tables, block ids, cache), so a thread carries several blocks along it at once.  Rows
// past a sequence's context (its range is rounded up to 128 rows) become zeros, so a tile that reaches past the context
// holds nothing that could turn 0 * x into NaN.
constexpr int kGatherRows = 64;
__global__ void __launch_bounds__(128) paged_gather_kernel(const PagedTables t, const uint8_t* k_cache, const uint8_t* v_cache,
                                                           const int Hkv, const int* kv_base, const int* owner,
                                                           const int scratch_rows, uint16_t* k_out, uint16_t* v_out,
                                                           int32_t* status) {
    constexpr int kBlocks = kGatherRows / 16;
    const int row0 = blockIdx.x * kGatherRows, hk = blockIdx.y;
    grid_dependency_wait();  // the scratch layout (plan kernel) and this step's cache rows (store kernel)
    grid_launch_dependents();
    const int seq = owner[row0 / 128];
    if (seq < 0) return;
    const int tok = threadIdx.x >> 3, c16 = threadIdx.x & 7;
    const int pos0 = row0 - kv_base[seq] + tok;  // position inside the sequence
    const int qlen = t.subsequence_begins[seq + 1] - t.subsequence_begins[seq];
    const int ctx = t.past_lens[seq] + qlen;
    const int bib0 = t.block_indices_begins[seq], have = t.block_indices_begins[seq + 1] - bib0;
    int phys[kBlocks];
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {
        const int pos = pos0 + 16 * i, lb = pos >> 4;
        phys[i] = -1;
        if (pos < ctx) {
            if (lb < have) phys[i] = t.block_indices[bib0 + lb];
            if (phys[i] < 0 || phys[i] >= t.num_blocks_total) {
                report(status, B2A_DEV_BAD_BLOCK);
                phys[i] = -1;
            }
        }
    }
    uint4 wk[kBlocks], wv[kBlocks];
    unsigned short sck[kBlocks], zpk[kBlocks], scv[kBlocks], zpv[kBlocks];
    const int tb = pos0 & 15;  // (the same in every block)
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {
        wk[i] = wv[i] = make_uint4(0u, 0u, 0u, 0u);
        sck[i] = zpk[i] = scv[i] = zpv[i] = 0;
        if (phys[i] >= 0) {
            const size_t chunk = (static_cast<size_t>(phys[i]) * Hkv + hk) * kCacheChunk;
            wk[i] = *reinterpret_cast<const uint4*>(k_cache + chunk + tb * 128 + c16 * 16);
            wv[i] = *reinterpret_cast<const uint4*>(v_cache + chunk + tb * 128 + c16 * 16);
            const unsigned short* mk = reinterpret_cast<const unsigned short*>(k_cache + chunk + 2048);
            const unsigned short* mv = reinterpret_cast<const unsigned short*>(v_cache + chunk + 2048);
            sck[i] = mk[tb];
            zpk[i] = mk[16 + tb];
            scv[i] = mv[tb];
            zpv[i] = mv[16 + tb];
        }
    }
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {
        const size_t at = (static_cast<size_t>(hk) * scratch_rows + row0 + 16 * i + tok) * kHeadDim + c16 * 16;
        uint32_t o[8];
        dequant16_f16(wk[i], sck[i], zpk[i], o);
        *reinterpret_cast<uint4*>(k_out + at) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(k_out + at + 8) = make_uint4(o[4], o[5], o[6], o[7]);
        dequant16_f16(wv[i], scv[i], zpv[i], o);
        *reinterpret_cast<uint4*>(v_out + at) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(v_out + at + 8) = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

// kMode: 0 dense tensors; 1 paged, K/V de-quantised by producer warps inside the kernel; 2 paged, K/V de-quantised
// beforehand into per-sequence row ranges of an f16 scratch (paged_gather_kernel) and staged by TMA like dense ones
// kMask: 0 no mask; 1 boolean and 2 additive, every row read by its thread in 16-byte pieces (unit stride, aligned);
//   3 boolean and 4 additive, the same for all rows (row stride 0: a padding mask), read once per warp, any key stride
//   and alignment; 5 either kind with any strides, element by element.
// kDim: head size, 64 or 128.
// kSplitP: P enters the second product as several 16-bit values (ProbPieces in common.cuh), so that these calls keep the
//   precision of attn_generic_kernel's float32 probabilities: 22 bits in f16, 24 in bf16.  Two pieces lie in the two halves of S's
//   columns; the second product of f16's low one has an accumulator of its own, bf16's third piece columns of its own, both
//   `kDim` columns behind O_X.  With a head size of 128 that is tile B's place: an item is then ONE tile.  It costs one or two
//   times as many second products again (the tensor pipe idles behind the exponentials anyway) and six to eight instructions
//   per pair of probabilities.  Bound: the special-function unit, 128 exponentials per row and step; the f16 encoder batch
//   of 8 x 16 heads x 512 tokens, head size 64, boolean padding mask: 1167 us in attn_generic_kernel, 26.3 us here (5.1 us
//   of memory traffic at the copy rate).  With 509 keys: f16 26.2 us, bf16 33.9 us; head size 128 46.9 and 60.8 us.
// kKeySplit (dense): a small problem - fewer pairs of tiles than SMs - is bound by its longest chain of key steps, one tile's
//   softmax after the other's.  Then an item is ONE tile whose keys are shared out: "tile A" takes the first half of its key
//   tiles, "tile B" the second, each with its own maximum, sum and accumulator, which are merged in the epilogue (the two
//   warps of the same 32 rows exchange maximum and sum through shared memory and read both accumulators: a warp reaches
//   the tensor-memory lanes of its number modulo four).  One item per CTA; the launcher's rule compares the two chains.
//   Causal prompts, 32/8 heads, D = 128, graph replay: 512 tokens 12.9 -> 9.4 us, 777 tokens 17.6 -> 15.7 us; 8 heads x 2048
//   tokens, D = 64, no mask: 36.9 -> 22.2 us.
// kOwnS (dense, no mask, at most 128 keys): a place of S per tile although P is not in pieces.
template <bool kBf16, int kMode, int kMask = 0, int kDim = kHeadDim, bool kSplitP = false, bool kKeySplit = false, bool kOwnS = false>
__global__ void __launch_bounds__(kMode == 1 ? kThreadsPaged : kThreadsDense, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
               const __grid_constant__ CUtensorMap tmV, const TcParams p, const __grid_constant__ TcPeers peers) {
    static_assert(kDim == kHeadDim || kMode == 0, "the paged modes are built for a head size of 128");
    static_assert(!kKeySplit || kMode == 0, "the keys of a tile are shared out in dense mode only");
    static_assert(!kSplitP || kMode == 0, "the paged modes hold P in 16 bits");
    constexpr bool kSingle = kSplitP && kDim == kHeadDim;  // an item is one tile: the pieces of P need tile B's columns
    static_assert(!(kSingle && kKeySplit), "no columns for the other half of the keys");
    // One place for S, which the tiles take in turn; P has columns of its own.  (Not with in-kernel de-quantisation, which is bound
    // by its producers: a step of three prompts behind caches takes 209 us in f16 and 216 in bf16 that way, 202 and 208 with a
    // place per tile - two more warps that issue and wait beside them.)
    constexpr bool kSharedS = !kSplitP && kMode != 1 && !kOwnS;
    constexpr int kTile = 128 * kDim * 2;  // bytes of a [128 x kDim] 16-bit tile: kDim / 64 panels
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // 128-byte swizzle atoms want 1024-byte aligned tiles
    uint8_t* gbase = smem_raw + (base - raw);
    const uint32_t sQ = base, sK = base + 2 * kTile, sV = base + 4 * kTile;
    const uint32_t sOut = base + 6 * kTile;
    const uint32_t bars = base + 6 * kTile + kStageOut;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + 6 * kTile + kStageOut + kNumBars * 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(gbase + 6 * kTile + kStageOut + kNumBars * 8 + 8);
    auto BAR = [&](int i) { return bars + 8u * static_cast<uint32_t>(i); };
    constexpr bool kPaged = kMode != 0, kDequant = kMode == 1, kGathered = kMode == 2;
    constexpr bool kKvBf16 = kPaged ? false : kBf16;  // element format of the K/V tiles and of P
    using Pieces = ProbPieces<std::conditional_t<kKvBf16, __nv_bfloat16, __half>>;
    constexpr bool kLowAcc = kSplitP && Pieces::kAccs == 2;      // O = O_X + kLowScale * (what lies kDim columns on)
    constexpr bool kThirdPiece = kSplitP && Pieces::kCount == 3;  // kDim columns behind O_X

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if constexpr (kDequant) {  // the grid is only a bound on the number of items: CTAs without one set nothing up
        grid_dependency_wait();
        if (static_cast<int>(blockIdx.x * gridDim.y + blockIdx.y) >= p.plan[0] * p.Hkv) return;
    }

    // ---- work items.  An item is a pair of tiles of one KV head.  Rows are numbered inside the sequence (paged) or
    // the tensor (dense); `pos_base` is the key position the first row of the problem may see up to, `kv_limit` the
    // number of keys that exist.  The CTA is persistent (except with in-kernel de-quantisation: one item per CTA):
    // the items, heaviest first - late row blocks in dense mode, the weight-sorted device-built list in paged mode -
    // are dealt to the CTAs in snake order (round k forwards, round k+1 backwards), which evens out the causal
    // imbalance without any shared counter.  Every role calls get_item for itself, so the per-sequence values
    // below are private to the calling thread and follow its own progress through the items.
    // nkvA, nkvB, nmax count key steps from the item's first key tile kv_tile0 (0 unless a sliding window lets the
    // item skip the tiles that all its rows have left behind)
    struct Item {
        int b, hk, row0A, row0B, headA, headB, nkvA, nkvB, nmax, kv_tile0;
    };
    int seq = 0, tok_base = 0, nrows_total = 0, pos_base = 0, kv_limit = 0, kv_row_base = 0;
    bool causal = true;
    int nrb = 0, tiles = 0, pairs = 0, total_items = 0;
    int active_ctas = static_cast<int>(gridDim.x);  // CTAs that take items
    auto get_item = [&](int k, Item& it) -> bool {  // the k-th item of this CTA
        int pair;
        if constexpr (kPaged) {
            int idx;
            if constexpr (kDequant) {
                if (k > 0) return false;
                idx = static_cast<int>(blockIdx.x * gridDim.y + blockIdx.y);
            } else {
                const int ctas = active_ctas, me = static_cast<int>(blockIdx.x);
                idx = k * ctas + ((k & 1) ? ctas - 1 - me : me);
            }
            if (idx >= total_items) return false;
            const int e = div_by(idx, p.div_hkv);
            it.b = 0;
            it.hk = idx - e * p.Hkv;
            const int4* rec = reinterpret_cast<const int4*>(p.plan + kPlanHeaderInts) + 2 * e;
            const int4 r0 = rec[0], r1 = rec[1];
            seq = r0.x;
            tok_base = r0.y;
            nrows_total = r0.z;
            pos_base = r0.w;
            pair = r1.x;
            kv_row_base = r1.y;
            kv_limit = pos_base + nrows_total;
            nrb = (nrows_total + kBM - 1) / kBM;
            tiles = nrb * p.G;
            pairs = (tiles + 1) / 2;
            if (nrows_total < 2 || pair >= pairs) {  // inconsistent tables (reported by the plan kernel): an empty item
                it.hk = 0;
                it.row0A = it.row0B = it.headA = it.headB = it.nkvA = it.nkvB = it.nmax = it.kv_tile0 = 0;
                return true;
            }
        } else {
            if constexpr (kKeySplit) {  // one tile, both halves of its keys; heaviest row blocks first
                if (k > 0) return false;
                const int idx = static_cast<int>(blockIdx.x), round = div_by(idx, p.div_streams), y = idx - round * p.B * p.Hkv;
                const int t = tiles - 1 - round, rb = div_by(t, p.div_g);
                it.b = div_by(y, p.div_hkv);
                it.hk = y - it.b * p.Hkv;
                it.row0A = it.row0B = rb * kBM;
                it.headA = it.headB = it.hk * p.G + (t - rb * p.G);
                const int n = ((causal ? min(kv_limit, it.row0A + kBM) : kv_limit) + kBN - 1) / kBN;
                it.nkvA = (n + 1) / 2;
                it.nkvB = n / 2;
                it.kv_tile0 = 0;
                it.nmax = it.nkvA;
                return true;
            }
            const int ctas = static_cast<int>(gridDim.x), me = static_cast<int>(blockIdx.x);
            // With four or more ranks the step is bound by the exchange of the output tiles, which can only start
            // when the first items end: then a CTA walks the SAME items (the deal below is what balances the CTAs)
            // from its lightest to its heaviest, and the epilogue's stores to the other ranks are on the wire from
            // the first microseconds on.  Measured with four ranks: 0.200 ms a step, against 0.231 ms heaviest
            // first.  (Storing a tile once locally and letting the CTA's two spare warps forward it to the other
            // ranks - so that no softmax warp ever waits for the links - was built and measured as well: 0.207-0.211
            // ms at best, the forwarding stores queue up in the SM's path to memory in front of the K/V loads.)
            if (peers.light_first) {
                const int rounds = total_items / ctas, rem = total_items - rounds * ctas;
                const int mine = rounds + ((((rounds & 1) ? ctas - 1 - me : me) < rem) ? 1 : 0);
                if (k >= mine) return false;
                k = mine - 1 - k;
            }
            const int idx = k * ctas + ((k & 1) ? ctas - 1 - me : me);
            if (idx >= total_items) return false;
            // heaviest row blocks of ALL (batch, KV head) streams first (measured faster than walking one stream
            // after the other, although that keeps fewer K/V streams in flight)
            const int bh = p.B * p.Hkv;
            const int round = div_by(idx, p.div_streams), y = idx - round * bh;
            pair = pairs - 1 - round;
            it.b = div_by(y, p.div_hkv);
            it.hk = y - it.b * p.Hkv;
        }
        // a tile's rows, its head, the end of its keys (in tiles) and the first key tile any of its rows still sees
        auto tile_of = [&](int t, int& row0, int& head, int& nkv, int& first) {
            const bool present = t < tiles;
            const int rb = present ? div_by(t, p.div_g) : 0, g = present ? t - rb * p.G : 0;
            row0 = rb * kBM;
            head = it.hk * p.G + g;
            const int kv_end = causal ? min(kv_limit, pos_base + row0 + kBM) : kv_limit;
            nkv = present ? (kv_end + kBN - 1) / kBN : 0;
            if constexpr (kPaged) {
                first = (p.window > 0 && present) ? max(0, pos_base + row0 - p.window + 1) / kBN : 0;
                if (!present) first = 1 << 30;
            } else {
                first = 0;
            }
        };
        int firstA, firstB;
        tile_of(kSingle ? pair : 2 * pair, it.row0A, it.headA, it.nkvA, firstA);
        tile_of(kSingle ? tiles : 2 * pair + 1, it.row0B, it.headB, it.nkvB, firstB);
        it.kv_tile0 = 0;
        if constexpr (kPaged) {
            // the two tiles walk the same key tiles: both start at the earlier of their first ones (a tile that starts
            // before its window only meets keys its mask removes)
            it.kv_tile0 = min(min(firstA, firstB), max(it.nkvA, it.nkvB));
            it.nkvA = max(0, it.nkvA - it.kv_tile0);
            it.nkvB = max(0, it.nkvB - it.kv_tile0);
        }
        it.nmax = max(it.nkvA, it.nkvB);
        return true;
    };

    // ---- set-up: barriers, TMEM
    if (threadIdx.x == 0) {
        for (int i = 0; i < kNumBars; ++i) {
            uint32_t count = 1;
            if (i == P_READY || i == P_READY + 1 || i == P_HALF || i == P_HALF + 1) count = 128;
            if (i == Q_CONV || i == Q_CONV + 1) count = 128;
            if (i == Q_EMPTY || i == Q_EMPTY + 1) count = 1;
            if (i >= HALVES && i < HALVES + 4) count = 64;  // the two warps of the same rows
            if (i == S_FREE) count = 128;
            if (kDequant && (i == K_FULL || i == K_FULL + 1 || i == V_FULL || i == V_FULL + 1)) count = 128;
            if (kGathered && (i == Q_CONV || i == Q_CONV + 1)) count = 32;  // a warp each
            if (i == DRAIN && kSharedS) count = 2;
            mbar_init(BAR(i), count);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 9) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = kSharedS ? 0u : *tmem_slot;  // (an allocation of all 512 columns starts at the first one)

    // Launched programmatically dependent: what is above overlaps the kernel before this one, everything that touches
    // memory comes after it.  Then a kernel that depends on this one (the decode kernel of a mixed step) may take the SMs
    // that this grid leaves free.
    grid_dependency_wait();
    grid_launch_dependents();
    if constexpr (kPaged) {
        total_items = p.plan[0] * p.Hkv;  // the grid is only a bound on the number of items
        if constexpr (kGathered) {
            // the plan kernel decides how many CTAs the prefill rows keep; the others give their SM to the decode rows
            active_ctas = min(max(p.plan[1], 1), static_cast<int>(gridDim.x));
            if (static_cast<int>(blockIdx.x) >= active_ctas) total_items = 0;
        }
    } else {
        nrows_total = p.Sq;
        kv_limit = p.Skv;
        causal = p.causal != 0;
        nrb = (nrows_total + kBM - 1) / kBM;
        tiles = nrb * p.G;
        pairs = kSingle ? tiles : (tiles + 1) / 2;
        total_items = pairs * p.B * p.Hkv;  // the launcher keeps this below 2^31
    }

    // Gathered K/V and bf16 queries: one warp turns Q tile X into f16 where it lies (the swizzle only permutes 16-byte chunks, so
    // an element-wise pass keeps the layout).  `n`: Q tiles of this kind before it.
    constexpr bool kConvertQ = kGathered && kBf16;
    auto convert_q = [&](int X, int n) {
        if (!__all_sync(0xffffffffu, mbar_wait(BAR(Q_FULL + X), n & 1, abort_flag))) return false;
        uint4* tile = reinterpret_cast<uint4*>(gbase + X * kTile);
        // (eight pieces in flight: the warp has nothing else to hide shared memory's latency behind)
        for (int i = lane; i < kTile / 16; i += 32 * 8) {
            uint4 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = tile[i + 32 * u];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                uint32_t* w = reinterpret_cast<uint32_t*>(&v[u]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[e]));
                    w[e] = pack_f16_finite(f.x, f.y);
                }
                tile[i + 32 * u] = v[u];
            }
        }
        fence_proxy_async_smem();
        mbar_arrive(BAR(Q_CONV + X));
        return true;
    };

    // Registers follow the work: the service warpgroup keeps 72 (56) per thread, the softmax groups take what is left
    // (2*128*216 + 128*72 = 384*168; a place of S per tile: 224 and 56; in-kernel de-quantisation: 2*128*168 + 128*56 + 128*112
    // <= 512*128).  A sum above what the launch has would wait forever.  (88 and 208: the masked and the bf16 gathered forms spill
    // 8 bytes more, three steps of 384 keys without a mask take 33.6 us instead of 32.8.)  With P in three pieces the issuing lane
    // wants 72 as well (us, 56 and 72 registers: 8 x 16 heads x 512 tokens, D = 64, bf16, causal 28.7 and 27.3, unmasked 33.1
    // and 31.5; two pieces 21.9 and 23.2, 23.6 and 24.9), but for the forms that have the most to keep in the softmax warps.
    constexpr bool kWideService = kSharedS || (kSplitP && kBf16 && kMask != 5 && !kKeySplit);
    constexpr int kServiceRegs = kWideService ? 72 : 56, kSoftmaxRegs = kDequant ? 168 : kWideService ? 216 : 224, kDequantRegs = kDequant ? 112 : 0;
    static_assert(256 * kSoftmaxRegs + 128 * kServiceRegs + 128 * kDequantRegs <= (kDequant ? 512 * 128 : 384 * 168), "register split");
    if (warp >= 8 && warp < 12) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kServiceRegs));
    if (warp >= 12) {
        // =============================== de-quantising K/V producers (paged) ===============================
        if constexpr (kDequant) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kDequantRegs));
            Item item;
            get_item(0, item);  // paged mode: exactly one item per CTA
            const int nkvA = item.nkvA, nkvB = item.nkvB, nmax = item.nmax, hk = item.hk;
            const int tp = static_cast<int>(threadIdx.x) - 384;
            const int tok_in_blk = tp >> 3, c16 = tp & 7;
            const int32_t* btab = p.t.block_indices + p.t.block_indices_begins[seq];
            const int nblk = (kv_limit + 15) / 16;
            bool ok = true;
            if constexpr (kBf16) {
                // bf16 queries: convert the Q tiles to f16 where they lie (the swizzle only permutes 16-byte
                // chunks, so an element-wise pass keeps the layout); magnitudes beyond the f16 range saturate
#pragma unroll
                for (int X = 0; X < 2; ++X) {
                    if ((X ? nkvB : nkvA) > 0) {
                        ok = ok && __all_sync(0xffffffffu, mbar_wait(BAR(Q_FULL + X), 0, abort_flag));
                        if (ok) {
                            uint4* tile = reinterpret_cast<uint4*>(gbase + X * kTile);
                            for (int i = tp; i < kTile / 16; i += 128) {
                                uint4 v = tile[i];
                                uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[k]));
                                    w[k] = pack_f16_finite(f.x, f.y);
                                }
                                tile[i] = v;
                            }
                            fence_proxy_async_smem();
                            mbar_arrive(BAR(Q_CONV + X));
                        }
                    }
                }
            }
            // One tile = 8 logical blocks; per block the 128 threads cover 16 tokens x 8 sixteen-byte pieces, so a
            // block's 2048 code bytes are read with fully coalesced 128-bit loads.  Everything a tile needs is
            // requested before anything is converted (one memory latency per tile, not one per block), and the
            // block ids of the next step are fetched while this step is converted.
            int phys[8], phys_next[8];
            const int kv_tile0 = item.kv_tile0;
            auto load_ids = [&](int j, int (&ids)[8]) {
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int lb = (kv_tile0 + j) * 8 + it;
                    int id = -1;
                    if (lb < nblk && lb * 16 + tok_in_blk < kv_limit) {
                        id = btab[lb];
                        if (id < 0 || id >= p.t.num_blocks_total) {
                            report(p.status, B2A_DEV_BAD_BLOCK);
                            id = -1;
                        }
                    }
                    ids[it] = id;
                }
            };
            uint4 w[8];
            unsigned short sc[8], zp[8];  // raw f16 bits: converting here would wait for each load in turn
            auto load_tile = [&](const uint8_t* cache) {
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    // positions past the context (and unusable blocks) become exact zeros: 0 * anything finite
                    w[it] = make_uint4(0u, 0u, 0u, 0u);
                    sc[it] = 0;
                    zp[it] = 0;
                    if (phys[it] >= 0) {
                        const uint8_t* chunk = cache + (static_cast<size_t>(phys[it]) * p.Hkv + hk) * kCacheChunk;
                        w[it] = *reinterpret_cast<const uint4*>(chunk + tok_in_blk * 128 + c16 * 16);
                        const unsigned short* meta = reinterpret_cast<const unsigned short*>(chunk + 2048);
                        sc[it] = meta[tok_in_blk];
                        zp[it] = meta[16 + tok_in_blk];
                    }
                }
            };
            auto convert_tile = [&](uint8_t* tile) {
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int token = it * 16 + tok_in_blk;
                    dequant_piece_f16(w[it], sc[it], zp[it], tile + token * 128, c16, token);
                }
            };
            load_ids(0, phys_next);
            for (int j = 0; j < nmax; ++j) {
                const int st = j & 1, n = j >> 1;
#pragma unroll
                for (int it = 0; it < 8; ++it) phys[it] = phys_next[it];
                load_tile(p.k_cache);
                if (j + 1 < nmax) load_ids(j + 1, phys_next);
                if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(BAR(K_EMPTY + st), (n - 1) & 1, abort_flag));
                if (!ok) break;
                convert_tile(gbase + 2 * kTile + st * kTile);
                fence_proxy_async_smem();  // generic-proxy writes must be visible to the tensor core's reads
                mbar_arrive(BAR(K_FULL + st));
                load_tile(p.v_cache);
                if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(BAR(V_EMPTY + st), (n - 1) & 1, abort_flag));
                if (!ok) break;
                convert_tile(gbase + 4 * kTile + st * kTile);
                fence_proxy_async_smem();
                mbar_arrive(BAR(V_FULL + st));
            }
        }
    } else if (warp >= (kSharedS ? 11 : 10)) {
        // idle warps of the service warpgroup; with gathered K/V and bf16 queries warp 11 turns the Q tiles A into f16
        if constexpr (kConvertQ) {
            Item item;
            bool ok = true;
            int qn = 0;
            for (int k = 0; ok && get_item(k, item); ++k)
                if (item.nkvA > 0) ok = convert_q(0, qn++);
        }
    } else if (warp == 8) {
        // =============================== TMA producer ===============================
        const bool lead = lane == 0;  // (with bf16 queries the whole warp goes along and converts the Q tiles B)
        if (lead || kConvertQ) {
            if (lead) {
                prefetch_tensormap(&tmQ);
                if constexpr (!kDequant) {
                    prefetch_tensormap(&tmK);
                    prefetch_tensormap(&tmV);
                }
            }
            // running counts over the items of this CTA: K/V tiles issued (ring position) and Q tiles loaded
            int g = 0, issued_k = 0, issued_v = 0, qn[2] = {0, 0};
            bool ok = true;
            const uint64_t once_policy = l2_evict_first_policy();  // Q tiles are read once
            Item it;
            for (int k = 0; ok && get_item(k, it); ++k) {
                auto load_q = [&](int X) {
                    const int nkvX = X ? it.nkvB : it.nkvA;
                    if (nkvX == 0) return;
                    if (!lead) { ++qn[X]; return; }
                    // the tile's previous occupant is free once its last QK^T has completed
                    if (qn[X] > 0 && !mbar_wait(BAR(Q_EMPTY + X), (qn[X] - 1) & 1, abort_flag)) { ok = false; return; }
                    mbar_expect_tx(BAR(Q_FULL + X), kTile);
                    const int row = tok_base + (X ? it.row0B : it.row0A), head = X ? it.headB : it.headA;
                    tma_load_4d_hint(sQ + X * kTile, &tmQ, BAR(Q_FULL + X), 0, row, head, it.b, once_policy);
                    if constexpr (kDim > 64)
                        tma_load_4d_hint(sQ + X * kTile + kPanel, &tmQ, BAR(Q_FULL + X), 64, row, head, it.b, once_policy);
                    ++qn[X];
                };
                if constexpr (kDequant) {
                    load_q(0);
                    if (ok) load_q(1);
                }
                if constexpr (kKeySplit) {
                    // tiles in the order A0 B0 A1 B1 ..: stage 0 of the rings is A's, stage 1 is B's; both use A's queries
                    const int total = it.nkvA + it.nkvB;
                    auto load = [&](int n, bool is_v) {
                        if (!ok || n >= total) return;
                        const int st = n & 1, j = n >> 1, row = (st ? it.nkvA + j : j) * kBN;
                        const int full = (is_v ? V_FULL : K_FULL) + st, empty = (is_v ? V_EMPTY : K_EMPTY) + st;
                        const uint32_t dst = (is_v ? sV : sK) + st * kTile;
                        const CUtensorMap* map = is_v ? &tmV : &tmK;
                        if (j > 0 && !mbar_wait(BAR(empty), (j - 1) & 1, abort_flag)) { ok = false; return; }
                        mbar_expect_tx(BAR(full), kTile);
                        tma_load_4d(dst, map, BAR(full), 0, row, it.hk, it.b);
                        if constexpr (kDim > 64) tma_load_4d(dst + kPanel, map, BAR(full), 64, row, it.hk, it.b);
                        ++(is_v ? issued_v : issued_k);
                    };
                    load(0, false);
                    load_q(0);
                    load(1, false);
                    load(0, true);
                    load(1, true);
                    load(2, false);
                    for (int n = 2; ok && n < total; ++n) {  // (QK runs ahead of PV)
                        load(n + 1, false);
                        load(n, true);
                    }
                } else if constexpr (!kDequant) {
                    // gathered mode: the sequence's keys start at row kv_row0 of the scratch, which is one [1, Hkv, rows, 128] tensor
                    const int kv_row0 = kGathered ? kv_row_base + it.kv_tile0 * kBN : 0;
                    auto load_k = [&](int j) {
                        if (!lead) return;
                        const int st = (g + j) & 1, n = (g + j) >> 1;
                        if (n > 0 && !mbar_wait(BAR(K_EMPTY + st), (n - 1) & 1, abort_flag)) { ok = false; return; }
                        mbar_expect_tx(BAR(K_FULL + st), kTile);
                        tma_load_4d(sK + st * kTile, &tmK, BAR(K_FULL + st), 0, kv_row0 + j * kBN, it.hk, it.b);
                        if constexpr (kDim > 64)
                            tma_load_4d(sK + st * kTile + kPanel, &tmK, BAR(K_FULL + st), 64, kv_row0 + j * kBN, it.hk, it.b);
                        ++issued_k;
                    };
                    if (it.nmax > 0) load_k(0);
                    for (int j = 0; j < it.nmax; ++j) {
                        if (j == 0) {  // (the first K tile has room before the previous item's last QK^T gives up the Q tiles)
                            if (ok) load_q(0);
                            if (ok) load_q(1);
                        }
                        if (kSharedS && ok && j + 1 < it.nmax) load_k(j + 1);  // (QK runs ahead of PV)
                        const int st = (g + j) & 1, n = (g + j) >> 1;
                        if (lead && ok && n > 0 && !mbar_wait(BAR(V_EMPTY + st), (n - 1) & 1, abort_flag)) ok = false;
                        if (kConvertQ) ok = __shfl_sync(0xffffffffu, ok, 0);  // (the only place where the warp's lanes part)
                        if (!ok) break;
                        if (lead) {
                            mbar_expect_tx(BAR(V_FULL + st), kTile);
                            tma_load_4d(sV + st * kTile, &tmV, BAR(V_FULL + st), 0, kv_row0 + j * kBN, it.hk, it.b);
                            if constexpr (kDim > 64)
                                tma_load_4d(sV + st * kTile + kPanel, &tmV, BAR(V_FULL + st), 64, kv_row0 + j * kBN, it.hk, it.b);
                            ++issued_v;
                        }
                        if (!kSharedS && j + 1 < it.nmax) load_k(j + 1);
                        if constexpr (kConvertQ)
                            if (j == 0 && it.nkvB > 0) ok = convert_q(1, qn[1] - 1);
                    }
                    g += it.nmax;
                }
            }
            if (lead && *abort_flag) {  // let copies already in flight land before the CTA goes away
                for (int X = 0; X < 2; ++X)
                    if (qn[X] > 0) mbar_drain(BAR(Q_FULL + X), (qn[X] - 1) & 1);
                for (int jj = max(0, issued_k - 2); jj < issued_k; ++jj) mbar_drain(BAR(K_FULL + (jj & 1)), (jj >> 1) & 1);
                for (int jj = max(0, issued_v - 2); jj < issued_v; ++jj) mbar_drain(BAR(V_FULL + (jj & 1)), (jj >> 1) & 1);
            }
        }
    } else if (kSharedS && (warp == 9 || warp == 10)) {
        // =============================== MMA issuers: QK and PV ===============================
        if constexpr (kSharedS) {  // whole warps, converged (tcgen05.cuh)
            auto wait_for = [&](int bar, int parity) { return __all_sync(0xffffffffu, mbar_wait(BAR(bar), parity, abort_flag)) != 0; };
            // operand formats (A and B of one MMA must agree): dense mode as given; paged mode f16 throughout - the
            // de-quantised values keep 11 significant bits and bf16 queries are converted in shared memory first
            constexpr uint32_t idesc_qk = instr_desc_f16(kKvBf16, false, kBM, kBN);
            constexpr uint32_t idesc_pv = instr_desc_f16(kKvBf16, true, kBM, kDim);
            const uint64_t q_desc = smem_desc_sw128(sQ, 16, 1024), k_desc = smem_desc_sw128(sK, 16, 1024);  // K-major: Q and K tiles
            const uint64_t v_desc = smem_desc_sw128(sV, kPanel, 1024);                                      // MN-major: V tiles
            auto issue_qk = [&](int X, int st) {  // S_X = Q_X K^T : steps of 16 along D
                constexpr uint32_t d = 0;
                const uint64_t qa = q_desc + static_cast<uint32_t>((kKeySplit ? 0 : X) * (kTile >> 4)), ka = k_desc + static_cast<uint32_t>(st * (kTile >> 4));
                mma_ss_x4<2, 2, idesc_qk>(d, qa, ka, 0u);
                if constexpr (kDim > 64) mma_ss_x4<2, 2, idesc_qk>(d, qa + kPanel / 16, ka + kPanel / 16, 1u);
            };
            // O_X += P_X V : 8 steps of 16 along the keys, in two halves
            auto issue_pv = [&](int X, int st, bool acc, int half) {
                const uint32_t d = static_cast<uint32_t>(256 + X * 128);
                const uint32_t pa = static_cast<uint32_t>(128 + X * 64 + half * 32);
                const uint64_t va = v_desc + static_cast<uint32_t>(st * (kTile >> 4) + half * (4 * 2048 / 16));
                mma_ts_x4<8, 2048 / 16, idesc_pv>(d, pa, va, acc ? 1u : 0u);
            };
            bool ok = true;
            constexpr int kQReady = (kPaged && kBf16) ? Q_CONV : Q_FULL;
            // running counts over the items of this CTA: K/V ring position, steps of each tile, Q tiles consumed
            int g0 = 0, sx[2] = {0, 0}, qn[2] = {0, 0};
            Item it;
            if (warp == 9) {
                // S has one place, which the tiles' turns A(0) B(0) A(1) B(1) .. share: QK of a turn is issued as soon as the
                // turn before has its scores in registers, long before its own softmax warps are there.
                int turns = 0;
                for (int k = 0; ok && get_item(k, it); ++k) {
#pragma unroll 1
                    for (int j = 0; ok && j < it.nmax; ++j) {
                        const int g = g0 + j;
#pragma unroll
                        for (int X = 0; X < 2; ++X) {
                            const int nkvX = X ? it.nkvB : it.nkvA, st = kKeySplit ? X : g & 1;
                            if (ok && j < nkvX) {
                                if (kKeySplit || X == 0 || it.nkvA <= j) ok = wait_for(K_FULL + st, (kKeySplit ? j : g >> 1) & 1);
                                if (j == 0 && !(kKeySplit && X)) ok = ok && wait_for(kQReady + X, qn[X]++ & 1);
                                if (turns > 0) ok = ok && wait_for(S_FREE, (turns - 1) & 1);
                                if (!ok) break;
                                ++turns;
                                tc_fence_after();
                                issue_qk(X, st);
                                mma_commit<true>(BAR(S_FULL + X));
                                if (j + 1 == nkvX) mma_commit<true>(BAR(Q_EMPTY + X));  // last use of this Q tile: the producer may refill it
                                if (kKeySplit) mma_commit<true>(BAR(K_EMPTY + st));
                            }
                        }
                        if (!kKeySplit) mma_commit<true>(BAR(K_EMPTY + (g & 1)));
                    }
                    g0 += it.nmax;
                }
            } else {
                // warp 10: PV of every turn when its P is ready
                for (int k = 0; ok && get_item(k, it); ++k) {
#pragma unroll 1
                    for (int j = 0; ok && j < it.nmax; ++j) {
                        const int g = g0 + j;
#pragma unroll
                        for (int X = 0; X < 2; ++X) {
                            const int st = kKeySplit ? X : g & 1;
                            if (ok && j < (X ? it.nkvB : it.nkvA)) {
                                if (kKeySplit || X == 0 || it.nkvA <= j) ok = wait_for(V_FULL + st, (kKeySplit ? j : g >> 1) & 1);
                                ok = ok && wait_for(P_READY + X, sx[X]++ & 1);
                                if (!ok) break;
                                tc_fence_after();
                                issue_pv(X, st, j > 0, 0);
                                issue_pv(X, st, true, 1);
                                mma_commit<true>(BAR(O_DONE + X));
                                if (kKeySplit) mma_commit<true>(BAR(V_EMPTY + st));
                            }
                        }
                        if (!kKeySplit) mma_commit<true>(BAR(V_EMPTY + (g & 1)));
                    }
                    g0 += it.nmax;
                }
            }
            mma_commit<true>(BAR(DRAIN));  // everything issued has completed before TMEM and shared memory are given up
            mbar_drain(BAR(DRAIN), 0);
        }
    } else if (warp == 9) {
        // =============================== MMA issuer, a place of S per tile ===============================
        // One lane: a step is a chain of waits here, and a vote of the warp behind each costs more than the faster issue gives
        // (encoder batch of 8 x 16 heads x 512 tokens: by the whole warp 2 % slower).
        if (!kSharedS && lane == 0) {
            // operand formats (A and B of one MMA must agree): dense mode as given; paged mode f16 throughout - the
            // de-quantised values keep 11 significant bits and bf16 queries are converted in shared memory first
            constexpr uint32_t idesc_qk = instr_desc_f16(kKvBf16, false, kBM, kBN);
            constexpr uint32_t idesc_pv = instr_desc_f16(kKvBf16, true, kBM, kDim);
            // descriptors are assembled at the point of issue from (tile address >> 4) plus compile-time parts
            constexpr uint32_t kLoK = desc_lo_sw128(16), kHiK = desc_hi_sw128(1024);        // K-major: Q and K tiles
            constexpr uint32_t kLoV = desc_lo_sw128(kPanel), kHiV = desc_hi_sw128(1024);    // MN-major: V tiles
            const uint32_t q16 = (sQ >> 4) & 0x3FFFu, k16 = (sK >> 4) & 0x3FFFu, v16 = (sV >> 4) & 0x3FFFu;
            auto issue_qk = [&](int X, int st) {  // S_X = Q_X K^T : steps of 16 along D
                const uint32_t d = tmem + static_cast<uint32_t>(X * 128);
                const uint32_t qa = q16 + static_cast<uint32_t>((kKeySplit ? 0 : X) * (kTile >> 4)), ka = k16 + static_cast<uint32_t>(st * (kTile >> 4));
#define B2A_QK(ks) \
    mma_ss_c<((((ks) / 4) * kPanel + ((ks) & 3) * 32) / 16), ((((ks) / 4) * kPanel + ((ks) & 3) * 32) / 16), kLoK, kLoK, kHiK, kHiK, \
             idesc_qk>(d, qa, ka, (ks) > 0 ? 1u : 0u)
                B2A_QK(0); B2A_QK(1); B2A_QK(2); B2A_QK(3);
                if constexpr (kDim > 64) { B2A_QK(4); B2A_QK(5); B2A_QK(6); B2A_QK(7); }
#undef B2A_QK
            };
            // O_X += P_X V : 8 steps of 16 along the keys, issued in two halves as the halves of P arrive
            auto issue_pv = [&](int X, int st, bool acc, int half) {
                const uint32_t d = tmem + static_cast<uint32_t>(256 + X * 128);
                const uint32_t pa = tmem + static_cast<uint32_t>(X * 128 + half * 32);
                const uint32_t va = v16 + static_cast<uint32_t>(st * (kTile >> 4) + half * (4 * 2048 / 16));
#define B2A_PV(ks, accv) mma_ts_c<(ks) * 8, ((ks) * 2048) / 16, kLoV, kHiV, idesc_pv>(d, pa, va, accv)
                B2A_PV(0, acc ? 1u : 0u); B2A_PV(1, 1u); B2A_PV(2, 1u); B2A_PV(3, 1u);
#undef B2A_PV
                if constexpr (kSplitP) {  // the second pieces of the same probabilities, 64 columns on
                    const uint32_t dl = kLowAcc ? d + kDim : d;
#define B2A_PVLO(ks, accv) mma_ts_c<64 + (ks) * 8, ((ks) * 2048) / 16, kLoV, kHiV, idesc_pv>(dl, pa, va, accv)
                    B2A_PVLO(0, acc || !kLowAcc ? 1u : 0u); B2A_PVLO(1, 1u); B2A_PVLO(2, 1u); B2A_PVLO(3, 1u);
#undef B2A_PVLO
                }
                if constexpr (kThirdPiece) {
                    const uint32_t pt = d + kDim + static_cast<uint32_t>(half * 32);
#define B2A_PV3(ks) mma_ts_c<(ks) * 8, ((ks) * 2048) / 16, kLoV, kHiV, idesc_pv>(d, pt, va, 1u)
                    B2A_PV3(0); B2A_PV3(1); B2A_PV3(2); B2A_PV3(3);
#undef B2A_PV3
                }
            };
            bool ok = true;
            constexpr int kQReady = (kPaged && kBf16) ? Q_CONV : Q_FULL;
            // running counts over the items of this CTA: K/V ring position, steps of each tile, Q tiles consumed
            int g0 = 0, sx[2] = {0, 0}, qn[2] = {0, 0};
            Item it;
            for (int k = 0; ok && get_item(k, it); ++k) {
                const int nkvA = it.nkvA, nkvB = it.nkvB, nmax = it.nmax;
                if (nmax == 0) continue;  // an item that was refused (inconsistent tables)
                if constexpr (kKeySplit) {
                    const int n = nkvA + nkvB;
                    ok = mbar_wait(BAR(Q_FULL), 0, abort_flag);
                    for (int X = 0; ok && X < min(n, 2); ++X) {
                        ok = mbar_wait(BAR(K_FULL + X), 0, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        issue_qk(X, X);
                        mma_commit<false>(BAR(S_FULL + X));
                        mma_commit<false>(BAR(K_EMPTY + X));
                    }
                    for (int i = 0; ok && i < n; ++i) {
                        const int X = i & 1, j = i >> 1;
                        ok = mbar_wait(BAR(V_FULL + X), j & 1, abort_flag) && mbar_wait(BAR(P_HALF + X), j & 1, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        issue_pv(X, X, j > 0, 0);
                        ok = mbar_wait(BAR(P_READY + X), j & 1, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        issue_pv(X, X, true, 1);
                        mma_commit<false>(BAR(O_DONE + X));
                        mma_commit<false>(BAR(V_EMPTY + X));
                        if (i + 2 < n) {
                            ok = mbar_wait(BAR(K_FULL + X), (j + 1) & 1, abort_flag);
                            if (!ok) break;
                            tc_fence_after();
                            issue_qk(X, X);
                            mma_commit<false>(BAR(S_FULL + X));
                            mma_commit<false>(BAR(K_EMPTY + X));
                        }
                    }
                    break;  // one item per CTA
                }
                ok = ok && mbar_wait(BAR(K_FULL + (g0 & 1)), (g0 >> 1) & 1, abort_flag);
                if (nkvA > 0) ok = ok && mbar_wait(BAR(kQReady + 0), qn[0] & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                if (nkvA > 0) {  // (tile A starts as soon as its own operands are there)
                    issue_qk(0, g0 & 1);
                    mma_commit<false>(BAR(S_FULL + 0));
                    if (nkvA == 1) mma_commit<false>(BAR(Q_EMPTY + 0));  // last use of this Q tile: the producer may refill it
                }
                if (nkvB > 0) {
                    ok = mbar_wait(BAR(kQReady + 1), qn[1] & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    issue_qk(1, g0 & 1);
                    mma_commit<false>(BAR(S_FULL + 1));
                    if (nkvB == 1) mma_commit<false>(BAR(Q_EMPTY + 1));
                }
                mma_commit<false>(BAR(K_EMPTY + (g0 & 1)));
                for (int j = 0; ok && j < nmax; ++j) {
                    const int g = g0 + j, stv = g & 1;
                    if (!mbar_wait(BAR(V_FULL + stv), (g >> 1) & 1, abort_flag)) { ok = false; break; }
                    bool k_next_ready = false;
#pragma unroll
                    for (int X = 0; X < 2; ++X) {
                        const int nkvX = X ? nkvB : nkvA;
                        if (ok && j < nkvX) {
                            const int par = (sx[X] + j) & 1;
                            if (!mbar_wait(BAR(P_HALF + X), par, abort_flag)) { ok = false; break; }
                            tc_fence_after();
                            issue_pv(X, stv, j > 0, 0);
                            if (!mbar_wait(BAR(P_READY + X), par, abort_flag)) { ok = false; break; }
                            tc_fence_after();
                            issue_pv(X, stv, true, 1);
                            mma_commit<false>(BAR(O_DONE + X));
                        }
                        if (ok && j + 1 < nkvX) {
                            if (!k_next_ready) {
                                if (!mbar_wait(BAR(K_FULL + ((g + 1) & 1)), ((g + 1) >> 1) & 1, abort_flag)) { ok = false; break; }
                                k_next_ready = true;
                                tc_fence_after();
                            }
                            issue_qk(X, (g + 1) & 1);
                            mma_commit<false>(BAR(S_FULL + X));
                            if (j + 2 == nkvX) mma_commit<false>(BAR(Q_EMPTY + X));
                        }
                    }
                    if (!ok) break;
                    mma_commit<false>(BAR(V_EMPTY + stv));
                    if (j + 1 < nmax) mma_commit<false>(BAR(K_EMPTY + ((g + 1) & 1)));
                }
                g0 += nmax;
                sx[0] += nkvA;
                sx[1] += nkvB;
                qn[0] += nkvA > 0;
                qn[1] += nkvB > 0;
            }
            mma_commit<false>(BAR(DRAIN));  // everything issued has completed before TMEM and shared memory are given up
            mbar_drain(BAR(DRAIN), 0);
        }
    } else {
        // =============================== softmax + epilogue of tile X ===============================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        const int X = warp >> 2;
        const int r = static_cast<int>(threadIdx.x) - X * 128;
        const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tS = tmem + lane_base + static_cast<uint32_t>(kSharedS ? 0 : X * 128);
        const uint32_t tP = tmem + lane_base + static_cast<uint32_t>(kSharedS ? 128 + X * 64 : X * 128);
        const uint32_t tO = tmem + lane_base + static_cast<uint32_t>(256 + X * 128);
        // 32 columns of an accumulator
        auto load_o = [&](uint32_t t, int q, uint32_t (&o)[32]) {
            tmem_ld32(t + 32 * q, o);
            if constexpr (kLowAcc) {
                uint32_t low[32];
                tmem_ld32(t + kDim + 32 * q, low);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(fmaf(__uint_as_float(low[i]), Pieces::kLowScale, __uint_as_float(o[i])));
            }
        };
        int sxb = 0;  // steps of this tile in the CTA's earlier items: every per-step barrier is at phase (sxb + j)
        bool ok = true;
        Item item;
        for (int k = 0; ok && get_item(k, item); ++k) {
            const int nkv = X ? item.nkvB : item.nkvA;
            if (nkv == 0) continue;
            const int row_pos0 = pos_base + (X ? item.row0B : item.row0A);
            // first step whose tile touches the end of the keys or the causal diagonal (both conditions only
            // become true as j grows): steps before it need no masking
            int jb;
            {
                const int j_end = kv_limit / kBN;
                const int dgl = row_pos0 - (kBN - 1);
                const int j_diag = dgl < 0 ? 0 : dgl / kBN + 1;
                jb = (causal ? min(j_end, j_diag) : j_end) - (kPaged ? item.kv_tile0 : kKeySplit && X ? item.nkvA : 0);
            }
            // with a sliding window, key tiles that begin below the window of the tile's LAST row need the mask too
            const int tile0 = kPaged ? item.kv_tile0 : kKeySplit && X ? item.nkvA : 0;
            const int window = kPaged ? p.window : 0;
            const int low_limit = window > 0 ? row_pos0 + kBM - window : -(1 << 30);  // mask while key0 < low_limit
            // (additive masks: the blocks below have scaled the scores)
            const float c = kMask == 2 || kMask == 4 || (kMask == 5 && p.mask_kind == B2A_MASK_ADD) ? 1.0f : p.scale_log2;
            float m_used = -1.0e30f, l = 0.f;
            // rows past the end of the tensor read the last row's mask: their results are dropped
            const uint8_t* mrow = nullptr;
            if constexpr (kMask != 0)
                mrow = p.mask + (item.b * p.mask_strides[0] + (X ? item.headB : item.headA) * p.mask_strides[1] +
                                 min(row_pos0 + r, nrows_total - 1) * p.mask_strides[2]) *
                                    (kMask == 1 || kMask == 3 || (kMask == 5 && p.mask_kind == B2A_MASK_BOOL) ? 1 : 2);
            // kMask 4: this warp's 128 mask values of a step, as floats, at the start of its staging slab
            float* mslab = reinterpret_cast<float*>(gbase + 6 * kTile + warp * 4096);
            for (int j = 0; j < nkv; ++j) {
                uint32_t mword[4];  // kMask 3: bit i of word q keeps key 32 q + i of the step
                if constexpr (kMask == 3) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int key = (tile0 + j) * kBN + 32 * q + lane;
                        mword[q] = key < kv_limit ? mrow[key * p.mask_strides[3]] : 0u;
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) mword[q] = __ballot_sync(0xffffffffu, mword[q] != 0u);
                }
                if constexpr (kMask == 4) {
                    float mv[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int key = (tile0 + j) * kBN + 32 * q + lane;
                        mv[q] = key < kv_limit ? mask_log2<kBf16>(mrow, key * p.mask_strides[3]) : -INFINITY;
                    }
                    __syncwarp();  // the last step's values have been read
#pragma unroll
                    for (int q = 0; q < 4; ++q) mslab[32 * q + lane] = mv[q];
                    __syncwarp();
                }
                // every lane takes the same decision, so the warp-collective TMEM instructions stay converged
                ok = __all_sync(0xffffffffu, mbar_wait(BAR(S_FULL + X), (sxb + j) & 1, abort_flag));
                if (!ok) break;
                tc_fence_after();
                uint32_t s[4][32];
#pragma unroll
                for (int q = 0; q < 4; ++q) tmem_ld32(tS + 32 * q, s[q]);
                tmem_wait_ld();
                if constexpr (kSharedS) {  // the other tile's scores may come
                    tc_fence_before();
                    mbar_arrive(BAR(S_FREE));
                }
                const int key0 = (tile0 + j) * kBN;
                if constexpr (kMask == 3) {
                    if ((mword[0] & mword[1] & mword[2] & mword[3]) != 0xffffffffu) {
#pragma unroll
                        for (int q = 0; q < 4; ++q)
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (((mword[q] >> i) & 1u) == 0u) s[q][i] = 0xff800000u;  // -inf
                    }
                }
                if constexpr (kMask == 4) {
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int i = 0; i < 32; i += 4) {
                            const float4 m4 = *reinterpret_cast<const float4*>(mslab + 32 * q + i);
                            s[q][i] = __float_as_uint(fmaf(__uint_as_float(s[q][i]), p.scale_log2, m4.x));
                            s[q][i + 1] = __float_as_uint(fmaf(__uint_as_float(s[q][i + 1]), p.scale_log2, m4.y));
                            s[q][i + 2] = __float_as_uint(fmaf(__uint_as_float(s[q][i + 2]), p.scale_log2, m4.z));
                            s[q][i + 3] = __float_as_uint(fmaf(__uint_as_float(s[q][i + 3]), p.scale_log2, m4.w));
                        }
                }
                if constexpr (kMask == 5) {
                    const bool keeps = p.mask_kind == B2A_MASK_BOOL;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int key = key0 + 32 * q + i;
                            if (key < kv_limit) {
                                if (keeps) {
                                    if (mrow[key * p.mask_strides[3]] == 0) s[q][i] = 0xff800000u;
                                } else {
                                    s[q][i] = __float_as_uint(fmaf(__uint_as_float(s[q][i]), p.scale_log2,
                                                                   mask_log2<kBf16>(mrow, key * p.mask_strides[3])));
                                }
                            }
                        }
                }
                if constexpr (kMask == 1 || kMask == 2) {
                    // this row's 128 mask values of the step, 32 keys at a time (keys past the end are removed below)
                    const uint8_t* mbase = mrow + key0 * (kMask == 1 ? 1 : 2);
                    const bool whole = key0 + kBN <= kv_limit;  // else only whole 16-byte pieces inside the row are read
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if constexpr (kMask == 1) {
                            uint4 m0 = make_uint4(0u, 0u, 0u, 0u), m1 = m0;
                            if (whole || key0 + 32 * q + 16 <= kv_limit) m0 = *reinterpret_cast<const uint4*>(mbase + 32 * q);
                            if (whole || key0 + 32 * q + 32 <= kv_limit) m1 = *reinterpret_cast<const uint4*>(mbase + 32 * q + 16);
                            const uint32_t w[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (((w[i >> 2] >> (8 * (i & 3))) & 0xffu) == 0u) s[q][i] = 0xff800000u;  // -inf
                        } else {
                            // additive: the scores leave this block as S * scale * log2(e) + mask * log2(e)
                            const float c = p.scale_log2;
#pragma unroll
                            for (int h = 0; h < 4; ++h) {
                                uint4 m = make_uint4(0u, 0u, 0u, 0u);
                                if (whole || key0 + 32 * q + 8 * h + 8 <= kv_limit) m = *reinterpret_cast<const uint4*>(mbase + 64 * q + 16 * h);
                                const uint32_t w[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    float lo, hi;
                                    unpack2<kBf16>(w[i], lo, hi);
                                    const int e = 8 * h + 2 * i;
                                    s[q][e] = __float_as_uint(fmaf(__uint_as_float(s[q][e]), c, mask_log2(lo)));
                                    s[q][e + 1] = __float_as_uint(fmaf(__uint_as_float(s[q][e + 1]), c, mask_log2(hi)));
                                }
                            }
                        }
                    }
                }
                if (kMask != 3 && kMask != 4 && (j >= jb || (kPaged && key0 < low_limit))) {
                    // the row keeps the tile's keys [low, lim): one comparison with a constant per key, and only in the
                    // groups of 32 that some row of the warp does not keep whole (the diagonal crosses one of four)
                    const int row_pos = row_pos0 + r;  // last key position this row may see (causal)
                    const int lim = (causal ? min(kv_limit, row_pos + 1) : kv_limit) - key0;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (__any_sync(0xffffffffu, lim < 32 * q + 32)) {
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (32 * q + i >= lim) s[q][i] = 0xff800000u;  // -inf
                        }
                    if (kPaged && key0 < low_limit) {
                        const int low = row_pos - window + 1 - key0;
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (__any_sync(0xffffffffu, low > 32 * q)) {
#pragma unroll
                                for (int i = 0; i < 32; ++i)
                                    if (32 * q + i < low) s[q][i] = 0xff800000u;
                            }
                    }
                }
                // row maximum: four independent chains of 3-input max (a single chain of 128 would be latency-bound)
                float mq[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    mq[q] = -INFINITY;
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        mq[q] = max3f(mq[q], __uint_as_float(s[q][i]), __uint_as_float(s[q][i + 1]));
                }
                const float mx = fmaxf(fmaxf(mq[0], mq[1]), fmaxf(mq[2], mq[3]));
                const float m_cand = mx * c;
                const bool need = (j == 0) || (m_cand > m_used + kLazyThreshold);
                const bool need_any = __any_sync(0xffffffffu, need);
                float alpha = 1.f;
                if (need_any) {
                    const float m_new = fmaxf(m_used, m_cand);
                    alpha = ex2f(m_used - m_new);
                    m_used = m_new;
                    l *= alpha;
                }
                if (kSharedS && j > 0) {  // PV(j-1) has read P's columns.  (Waited for in the middle of the exponentials it cost 7 %.)
                    ok = __all_sync(0xffffffffu, mbar_wait(BAR(O_DONE + X), (sxb + j - 1) & 1, abort_flag));
                    tc_fence_after();
                }
                // P = exp2(S*c - m): the scale-and-shift and the row sum run two elements per instruction (f32x2).  (f16 in
                // pieces: 2^7 P, at most 2^15, so that the pieces reach as far down as they can; the sum carries the factor too)
                const float shift = kLowAcc ? 7.f - m_used : -m_used;
                const uint64_t c2 = f2_pack(c, c), nm2 = f2_pack(shift, shift);
                uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t pk[16], pk_lo[16], pk_third[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const uint64_t x2 = f2_fma(f2_pack(__uint_as_float(s[q][2 * i]), __uint_as_float(s[q][2 * i + 1])), c2, nm2);
                        float x0, x1;
                        f2_unpack(x2, x0, x1);
                        const float p0 = ex2f(x0), p1 = ex2f(x1);
                        sum2[i & 3] = f2_add(sum2[i & 3], f2_pack(p0, p1));
                        if constexpr (kSplitP) {
                            uint32_t w[Pieces::kCount];
                            Pieces::split(p0, p1, w);
                            pk[i] = w[0];
                            pk_lo[i] = w[1];
                            if constexpr (kThirdPiece) pk_third[i] = w[2];
                        } else {
                            pk[i] = pack2<kKvBf16>(p0, p1);
                        }
                    }
                    tmem_st16(tP + 16 * q, pk);  // (pieces of P: over S's columns, all of which have been read)
                    if constexpr (kSplitP) tmem_st16(tS + 64 + 16 * q, pk_lo);  // (all of S is in registers by now)
                    if constexpr (kThirdPiece) tmem_st16(tO + kDim + 16 * q, pk_third);
                    // first 64 keys of P are in TMEM: PV can start on them, unless O still has to be rescaled
                    if (!kSharedS && q == 1 && !(need_any && j > 0)) {
                        tmem_wait_st();
                        tc_fence_before();
                        mbar_arrive(BAR(P_HALF + X));
                    }
                }
                {
                    float a0, a1;
                    f2_unpack(f2_add(f2_add(sum2[0], sum2[1]), f2_add(sum2[2], sum2[3])), a0, a1);
                    l += a0 + a1;
                }
                if (need_any && j > 0) {
                    // O_X still holds the old scale; PV_X(j-1) must have landed before it is touched
                    if constexpr (!kSharedS) {
                        ok = __all_sync(0xffffffffu, mbar_wait(BAR(O_DONE + X), (sxb + j - 1) & 1, abort_flag));
                        tc_fence_after();
                    }
                    if (!ok) break;
#pragma unroll
                    for (int q = 0; q < (kLowAcc ? 2 : 1) * kDim / 32; ++q) {
                        uint32_t o[32];
                        tmem_ld32(tO + 32 * q, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st32(tO + 32 * q, o);
                    }
                    if constexpr (!kSharedS) {
                        tmem_wait_st();
                        tc_fence_before();
                        mbar_arrive(BAR(P_HALF + X));
                    }
                }
                if (kSharedS && !ok) break;
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(BAR(P_READY + X));
            }
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(BAR(O_DONE + X), (sxb + nkv - 1) & 1, abort_flag));
            sxb += nkv;
            if (ok) {
                tc_fence_after();
                const float inv = l > 0.f ? 1.f / l : 0.f;
                // Where the tile goes is kept across the key loop.  (Worked out again here it is 192 bytes of spill loads instead of
                // 24 in the unmasked form of head size 128, and 300 cycles an item: 8 x 32 heads x 300 tokens 27.3 us instead of 25.1,
                // 2048 tokens 33.6 instead of 32.4.)  Only three pieces of P beside a mask read element by element leave no
                // room for it (4 x 16 heads x 509 tokens, a boolean mask row per query: 99 us kept, 90 this way).
                if constexpr (kSplitP && kBf16 && kMask == 5) {
                    int k_again = k;
                    asm volatile("" : "+r"(k_again));
                    get_item(k_again, item);
                }
                const int row0 = X ? item.row0B : item.row0A, head = X ? item.headB : item.headA, b = item.b;
                if constexpr (kKeySplit) {
                    // (maximum, sum) of this row's other half of the keys, from the warp that has it; a tile of one key
                    // step has no other half
                    const bool both = item.nkvB > 0;
                    float inv_own = inv, inv_other = 0.f;
                    if (both) {
                        float2* mine = reinterpret_cast<float2*>(gbase + kTile) + warp * 32;  // (Q tile B's place, not used here)
                        const float2* theirs = reinterpret_cast<const float2*>(gbase + kTile) + (warp ^ 4) * 32;
                        mine[lane] = make_float2(m_used, l);
                        tc_fence_before();
                        mbar_arrive(BAR(HALVES + (warp & 3)));
                        ok = __all_sync(0xffffffffu, mbar_wait(BAR(HALVES + (warp & 3)), 0, abort_flag));
                        if (!ok) break;
                        tc_fence_after();  // (the other warp has waited for its accumulator: it may be read here too)
                        const float2 o = theirs[lane];
                        const float m = fmaxf(m_used, o.x);
                        const float f_own = ex2f(m_used - m), f_other = ex2f(o.x - m);
                        const float sum = l * f_own + o.y * f_other;
                        const float inv_sum = sum > 0.f ? 1.f / sum : 0.f;
                        inv_own = f_own * inv_sum;
                        inv_other = f_other * inv_sum;
                    }
                    uint16_t* orow = static_cast<uint16_t*>(p.out) + b * p.out_strides[0] + head * p.out_strides[1] +
                                     (row0 + r) * p.out_strides[2];
                    const bool valid = row0 + r < nrows_total;
                    const uint32_t tOther = tmem + lane_base + static_cast<uint32_t>(256 + (X ^ 1) * 128);
#pragma unroll
                    for (int q = 0; q < kDim / 32; ++q) {
                        if (both && (q / (kDim / 64)) != X) continue;  // the other warp's columns
                        uint32_t o[32], w[16];
                        load_o(tO, q, o);
                        if (both) {
                            uint32_t o2[32];
                            load_o(tOther, q, o2);
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                o[i] = __float_as_uint(__uint_as_float(o[i]) * inv_own + __uint_as_float(o2[i]) * inv_other);
                        } else {
                            tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * inv_own);
                        }
#pragma unroll
                        for (int i = 0; i < 16; ++i) w[i] = pack2<kBf16>(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
                        if (peers.world == 0) {
                            if (valid) store_64_bytes(orow + 32 * q, w, p.out_wide != 0);
                            continue;
                        }
                        // sharded heads: 64 columns through this warp's slab into every rank's buffer, as below
                        if ((q & 1) == 0) {
                            if (lane == 0) tma_store_wait_read();
                            __syncwarp();
                        }
#pragma unroll
                        for (int ch = 0; ch < 4; ++ch)
                            *reinterpret_cast<uint4*>(gbase + 6 * kTile + warp * 4096 + lane * 128 + ((((q & 1) * 4 + ch) ^ (lane & 7)) << 4)) =
                                make_uint4(w[4 * ch], w[4 * ch + 1], w[4 * ch + 2], w[4 * ch + 3]);
                        if ((q & 1) == 1) {
                            fence_proxy_async_smem();
                            __syncwarp();
                            if (lane == 0) {
                                for (int i = 1; i <= peers.world; ++i) {
                                    const int dst = (peers.rank + i) % peers.world;
                                    tma_store_4d(&peers.out_map[dst], sOut + static_cast<uint32_t>(warp) * 4096u, 32 * (q - 1),
                                                 row0 + 32 * (warp & 3), peers.head_offset + head, b);
                                }
                                tma_store_commit();
                            }
                        }
                    }
                } else if (kPaged || peers.world == 0) {
                    // A thread's row straight from its registers, whole 32-byte sectors: nothing to wait for, and the
                    // warp goes on to the next item while the stores drain.  (Through the slab and TMA stores, the second
                    // half waited for the first to be read, behind the next item's loads in the TMA unit's queue: 5000
                    // cycles an item, longer than a key step.)  Rows past the end belong to nobody, or to another sequence.
                    uint16_t* orow = static_cast<uint16_t*>(p.out);
                    if constexpr (kPaged) orow += (static_cast<int64_t>(tok_base + row0 + r) * p.Hq + head) * kDim;
                    else orow += b * p.out_strides[0] + head * p.out_strides[1] + (row0 + r) * p.out_strides[2];
                    const bool valid = row0 + r < nrows_total;
#pragma unroll
                    for (int q = 0; q < kDim / 32; ++q) {
                        uint32_t o[32], w[16];
                        load_o(tO, q, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            w[i] = pack2<kBf16>(__uint_as_float(o[2 * i]) * inv, __uint_as_float(o[2 * i + 1]) * inv);
                        if (valid) store_64_bytes(orow + 32 * q, w, p.out_wide != 0);
                    }
                } else {
                    // passes of 64 columns through this warp's [32 rows x 128 bytes] staging slab
                    const uint32_t slab = sOut + static_cast<uint32_t>(warp) * 4096u;
                    uint8_t* prow = gbase + 6 * kTile + warp * 4096 + (r & 31) * 128;
#pragma unroll
                    for (int half = 0; half < kDim / 64; ++half) {
                        if (lane == 0) tma_store_wait_read();  // the slab's previous store has read it
                        __syncwarp();
#pragma unroll
                        for (int qq = 0; qq < 2; ++qq) {
                            const int q = 2 * half + qq;
                            uint32_t o[32];
                            tmem_ld32(tO + 32 * q, o);
                            tmem_wait_ld();
#pragma unroll
                            for (int ch = 0; ch < 4; ++ch) {
                                uint4 v;
                                v.x = pack2<kBf16>(__uint_as_float(o[8 * ch + 0]) * inv, __uint_as_float(o[8 * ch + 1]) * inv);
                                v.y = pack2<kBf16>(__uint_as_float(o[8 * ch + 2]) * inv, __uint_as_float(o[8 * ch + 3]) * inv);
                                v.z = pack2<kBf16>(__uint_as_float(o[8 * ch + 4]) * inv, __uint_as_float(o[8 * ch + 5]) * inv);
                                v.w = pack2<kBf16>(__uint_as_float(o[8 * ch + 6]) * inv, __uint_as_float(o[8 * ch + 7]) * inv);
                                const int chunk = qq * 4 + ch;  // 16-byte chunk of the 128-byte row, swizzled like TMA's
                                *reinterpret_cast<uint4*>(prow + ((chunk ^ (r & 7)) << 4)) = v;
                            }
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            // the slab into every rank's buffer, the next rank first so that the ranks do not all write to
                            // the same peer at the same time; local copy last
                            for (int i = 1; i <= peers.world; ++i) {
                                const int dst = (peers.rank + i) % peers.world;
                                tma_store_4d(&peers.out_map[dst], slab, 64 * half, row0 + 32 * (warp & 3), peers.head_offset + head, b);
                            }
                            tma_store_commit();
                        }
                    }
                }
            }
        }
        // stores still in flight: their completion (not only the read of shared memory) before the CTA ends
        if (lane == 0) tma_store_wait_all();
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && *abort_flag) report(p.status, B2A_DEV_TIMEOUT);
    if constexpr (!kPaged) {
        if (peers.world > 0 && threadIdx.x == 0) {
            // every storing lane has waited for its writes and passed the barrier above: order them before the
            // arrival, and let the last CTA of the grid publish the step to every rank
            __threadfence_system();
            const int total = static_cast<int>(gridDim.x * gridDim.y);
            if (atomicAdd(peers.done_counter, 1) == total - 1) {
                *peers.done_counter = 0;
                __threadfence_system();
                for (int r = 0; r < peers.world; ++r)
                    asm volatile("st.release.sys.global.s32 [%0], %1;" ::"l"(peers.flags[r] + peers.rank), "r"(peers.step)
                                 : "memory");
            }
        }
    }
}

// Stream-ordered wait for the other ranks of a head-sharded prefill step: returns when every flag shows `step`.
// Bounded in wall-clock time: a peer that never arrives turns into B2A_DEV_TIMEOUT in the status word.
__global__ void __launch_bounds__(32) sdpa_peer_wait_kernel(const int32_t* flags, const int world, const int32_t step,
                                                            const long long wait_ns, int32_t* status) {
    grid_dependency_wait();  // launched while the attention kernel is still running: first let that one finish
    if (static_cast<int>(threadIdx.x) < world) {
        const int32_t* flag = flags + threadIdx.x;
        long long t0;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (;;) {
            int32_t v;
            asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
            if (v - step >= 0) break;
            long long t1;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
            if (t1 - t0 > wait_ns) {
                report(status, B2A_DEV_TIMEOUT);
                break;
            }
        }
    }
}

// ---- host side ---------------------------------------------------------------------------------------------

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return reinterpret_cast<EncodeTiledFn>(ptr);
    }();
    return fn;
}

// [B, H, S, head_dim] view with element strides st[0..3] (st[3] == 1) as a 4-D map, box = [64 x box_rows x 1 x 1],
// 128-byte swizzle
bool make_map(CUtensorMap* map, const void* ptr, bool bf16, int B, int H, int S, const int64_t (&st)[4], int box_rows,
              int head_dim = kHeadDim) {
    EncodeTiledFn enc = encode_fn();
    if (enc == nullptr) return false;
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(head_dim), static_cast<cuuint64_t>(S),
                                static_cast<cuuint64_t>(H), static_cast<cuuint64_t>(B)};
    // a stride of an extent-1 dimension is never used for addressing but is still validated: give it a legal value
    auto bytes = [](int64_t elems, int extent) { return static_cast<cuuint64_t>(extent == 1 || elems <= 0 ? 256 : elems * 2); };
    const cuuint64_t strides[3] = {bytes(st[2], S), bytes(st[1], H), bytes(st[0], B)};
    const cuuint32_t box[4] = {64, static_cast<cuuint32_t>(box_rows), 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
               const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int kMask, int kDim, bool kSplitP, bool kKeySplit = false, bool kOwnS = false>
int launch_dense(bool bf16, dim3 grid, cudaStream_t stream, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                 const TcParams& p, const TcPeers& peers) {
    constexpr int smem = smem_bytes(128 * kDim * 2);
    static OncePerDevice configured[2];
    auto kern = bf16 ? attn_tc_kernel<true, 0, kMask, kDim, kSplitP, kKeySplit, kOwnS> : attn_tc_kernel<false, 0, kMask, kDim, kSplitP, kKeySplit, kOwnS>;
    const int rc = configure_once(kern, configured[bf16], smem);
    if (rc != B2A_OK) return rc;
    return launch_overlapped(kern, grid, dim3(kThreadsDense), smem, stream, mq, mk, mv, p, peers) == cudaSuccess ? B2A_OK : B2A_ERR_CUDA;
}

bool strides_ok(const int64_t (&st)[4], int B, int H, int S) {
    if (st[3] != 1) return false;
    const int ext[3] = {B, H, S};
    for (int i = 0; i < 3; ++i)
        if (ext[i] > 1 && (st[i] <= 0 || st[i] % 8 != 0)) return false;  // 16-byte multiples
    return true;
}

}  // namespace

static bool tc_tensors_ok(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                          const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* o) {
    if (d.dtype != B2A_F16 && d.dtype != B2A_BF16) return false;
    if (static_cast<long long>(d.B) * d.Hkv > 65535) return false;
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (!al(q) || !al(k) || !al(v) || !al(o)) return false;
    if (!strides_ok(qs, d.B, d.Hq, d.Sq) || !strides_ok(ks, d.B, d.Hkv, d.Skv) || !strides_ok(vs, d.B, d.Hkv, d.Skv) ||
        !strides_ok(os, d.B, d.Hq, d.Sq))
        return false;
    return encode_fn() != nullptr;
}

bool sdpa_tc_supported(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                       const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* o) {
    return d.D == kHeadDim && d.Dv == kHeadDim && tc_tensors_ok(d, qs, ks, vs, os, q, k, v, o);
}

bool sdpa_tc_split_supported(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                             const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* o) {
    return (d.D == 64 || d.D == kHeadDim) && d.D == d.Dv && tc_tensors_ok(d, qs, ks, vs, os, q, k, v, o);
}

bool sdpa_tc_mask_supported(const b2a_sdpa_desc& d, const void* mask) {
    // the mask is read in 16-byte pieces along the keys: unit stride there, every row start 16-byte aligned, and a
    // key count that is a whole number of pieces
    if (d.mask_kind != B2A_MASK_BOOL && d.mask_kind != B2A_MASK_ADD) return false;
    const int es = d.mask_kind == B2A_MASK_BOOL ? 1 : 2;
    const int per_piece = 16 / es;
    if (d.mask_strides[3] != 1 || d.Skv % per_piece != 0) return false;
    if ((reinterpret_cast<uintptr_t>(mask) & 15) != 0) return false;
    for (int i = 0; i < 3; ++i)
        if (d.mask_strides[i] < 0 || (d.mask_strides[i] * es) % 16 != 0) return false;
    return true;
}

int sdpa_tc_launch(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                   const int64_t (&os)[4], const void* q, const void* k, const void* v, void* o, int32_t* status,
                   cudaStream_t stream, const TcPeerOut* peer_out, const void* mask, bool split_p, int parts) {
    const bool bf16 = d.dtype == B2A_BF16;
    CUtensorMap mq, mk, mv;
    // A causal row sees at most Sq keys: what lies behind (a cache's unfilled rows, which may hold NaN) comes in as zeros, like
    // everything outside a map.
    const int keys = d.causal ? std::min(d.Skv, d.Sq) : d.Skv;
    if (!make_map(&mq, q, bf16, d.B, d.Hq, d.Sq, qs, 128, d.D) || !make_map(&mk, k, bf16, d.B, d.Hkv, keys, ks, 128, d.D) ||
        !make_map(&mv, v, bf16, d.B, d.Hkv, keys, vs, 128, d.D))
        return B2A_ERR_CUDA;
    TcPeers peers{};
    if (peer_out != nullptr) {
        const int64_t fs[4] = {static_cast<int64_t>(peer_out->hq_total) * d.Sq * kHeadDim,
                               static_cast<int64_t>(d.Sq) * kHeadDim, kHeadDim, 1};
        for (int r = 0; r < peer_out->world; ++r) {
            if (!make_map(&peers.out_map[r], peer_out->out_base[r], bf16, d.B, peer_out->hq_total, d.Sq, fs, 32))
                return B2A_ERR_CUDA;
            peers.flags[r] = peer_out->flags[r];
        }
        peers.done_counter = peer_out->done_counter;
        peers.world = peer_out->world;
        peers.rank = peer_out->rank;
        peers.head_offset = peer_out->head_offset;
        peers.step = peer_out->step;
        peers.light_first = peer_out->world >= 4 ? 1 : 0;
    }
    TcParams p{};
    p.B = d.B; p.Hq = d.Hq; p.Hkv = d.Hkv; p.G = d.Hq / d.Hkv; p.Sq = d.Sq; p.Skv = keys;
    p.div_g = fast_div(p.G);
    p.div_hkv = fast_div(p.Hkv);
    p.div_streams = fast_div(p.B * p.Hkv);
    p.out = o;
    const int extents[3] = {d.B, d.Hq, d.Sq};
    p.out_wide = (reinterpret_cast<uintptr_t>(o) & 31) == 0;
    for (int i = 0; i < 3; ++i) {
        p.out_strides[i] = os[i];
        if (extents[i] > 1 && os[i] % 16 != 0) p.out_wide = 0;
    }
    p.causal = d.causal;
    p.scale_log2 = d.scale * kLog2e;
    p.status = status;
    const int nrb = (d.Sq + kBM - 1) / kBM;
    const bool single = split_p && d.D == kHeadDim;  // (kSingle)
    const int pairs = single ? nrb * p.G : (nrb * p.G + 1) / 2;
    const long long items = static_cast<long long>(pairs) * d.B * d.Hkv;
    if (items >= (1LL << 30)) return B2A_ERR_UNSUPPORTED;
    const int sms = device_sm_count();
    if (sms <= 0) return B2A_ERR_CUDA;
    dim3 grid(static_cast<unsigned>(items < sms ? items : sms));  // persistent CTAs, one per SM
    const int mask_kind = (mask != nullptr && !d.causal) ? d.mask_kind : B2A_MASK_NONE;
    if (mask_kind != B2A_MASK_NONE) {
        p.mask = static_cast<const uint8_t*>(mask);
        p.mask_kind = mask_kind;
        for (int i = 0; i < 4; ++i) p.mask_strides[i] = d.mask_strides[i];
    }
    // Pairs of tiles, or single tiles with their keys shared out (kKeySplit)?  With fewer pairs than SMs the former takes the
    // longest pair's key steps, n.  The latter takes the longest half per round of CTAs (tiles of equal length) or, if
    // more, the halves' steps over the SMs (causal), plus a CTA's start (about one and a half steps) for a second round.
    // It reads K and V twice as fast.  On more than half of the SMs that is more than the pairs ever ask of L2, and copies
    // running beside it starve: host tensors in pieces of 8 heads x 4096 tokens (256 tiles) took 5.05 ms a step instead of
    // 4.53, although the kernel itself went from 61 to 37 us.  So such grids share the keys out up to sixteen steps only.
    // A sharded launch, or one that is a part of a problem, asks the rule for ALL heads: its output is that of one launch over
    // them, bit for bit.
    bool key_split = false;
    const long long shares = peer_out != nullptr ? peer_out->hq_total / d.Hq : parts;
    const long long streams = static_cast<long long>(d.B) * d.Hkv * shares, all_tiles = streams * nrb * p.G;
    const int n = (keys + kBN - 1) / kBN, half = (n + 1) / 2;
    if (items * shares <= sms && (n <= 16 || 2 * all_tiles <= sms)) {
        const long long rounds = (all_tiles + sms - 1) / sms;
        double steps = static_cast<double>(rounds * half);
        if (d.causal) {
            long long halves = 0;
            for (int rb = 0; rb < nrb; ++rb) halves += ((std::min(keys, (rb + 1) * kBM) + kBN - 1) / kBN + 1) / 2;
            steps = std::max<double>(half, static_cast<double>(halves * p.G * streams) / sms);
        }
        key_split = steps + (rounds > 1 ? 1.5 : 0.0) < n;
    }
    const dim3 tile_grid(static_cast<unsigned>(key_split ? all_tiles / shares : 0));
    if (split_p) {
        // a mask that is one row for all queries is read once per warp; anything else row by row
        const int form = mask_kind == B2A_MASK_NONE                    ? 0
                         : d.mask_strides[2] != 0 && d.Sq > 1          ? 5
                         : mask_kind == B2A_MASK_BOOL                  ? 3
                                                                       : 4;
        if (d.D == 64 && key_split && form != 5) {
            if (form == 0) return launch_dense<0, 64, true, true>(bf16, tile_grid, stream, mq, mk, mv, p, peers);
            if (form == 3) return launch_dense<3, 64, true, true>(bf16, tile_grid, stream, mq, mk, mv, p, peers);
            return launch_dense<4, 64, true, true>(bf16, tile_grid, stream, mq, mk, mv, p, peers);
        }
        if (d.D == 64) {
            if (form == 0) return launch_dense<0, 64, true>(bf16, grid, stream, mq, mk, mv, p, peers);
            if (form == 3) return launch_dense<3, 64, true>(bf16, grid, stream, mq, mk, mv, p, peers);
            if (form == 4) return launch_dense<4, 64, true>(bf16, grid, stream, mq, mk, mv, p, peers);
            return launch_dense<5, 64, true>(bf16, grid, stream, mq, mk, mv, p, peers);
        }
        if (form == 3) return launch_dense<3, kHeadDim, true>(bf16, grid, stream, mq, mk, mv, p, peers);
        if (form == 4) return launch_dense<4, kHeadDim, true>(bf16, grid, stream, mq, mk, mv, p, peers);
        if (form == 5) return launch_dense<5, kHeadDim, true>(bf16, grid, stream, mq, mk, mv, p, peers);
    }
    if (mask_kind == B2A_MASK_BOOL) return launch_dense<1, kHeadDim, false>(bf16, grid, stream, mq, mk, mv, p, peers);
    if (mask_kind == B2A_MASK_ADD) return launch_dense<2, kHeadDim, false>(bf16, grid, stream, mq, mk, mv, p, peers);
    if (key_split) return launch_dense<0, kHeadDim, false, true>(bf16, tile_grid, stream, mq, mk, mv, p, peers);
    // One key step an item: there is no next step whose QK^T could run beside the softmax, and PV starts on the first half of P where
    // S has a place per tile (us, shared and per tile: 4 x 200 heads x 100 tokens 23.6 and 21.2, 32 heads x 128 6.15 and
    // 5.8, 8 x 32/8 heads x 128 without the causal mask 8.2 and 7.6).  From two steps on it is even (4 x 32/8 heads x 256: 9.8
    // both) or the other way round (16 x 32/8 heads x 129: 21.7 and 22.8).
    if (n == 1) return launch_dense<0, kHeadDim, false, false, true>(bf16, grid, stream, mq, mk, mv, p, peers);
    return launch_dense<0, kHeadDim, false>(bf16, grid, stream, mq, mk, mv, p, peers);
}

int sdpa_peer_wait_launch(const int32_t* local_flags, int world, int32_t step, long long wait_ns, int32_t* status,
                          cudaStream_t stream) {
    return launch_overlapped(sdpa_peer_wait_kernel, dim3(1), dim3(32), 0, stream, local_flags, world, step, wait_ns, status) ==
                   cudaSuccess
               ? B2A_OK
               : B2A_ERR_CUDA;
}

bool paged_tc_supported(const b2a_paged_desc& d, const void* query, const void* out) {
    const int g = d.Hkv > 0 ? d.Hq / d.Hkv : 0;
    auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return d.kv_dtype == B2A_U8 && (d.q_dtype == B2A_F16 || d.q_dtype == B2A_BF16) && d.D == kHeadDim &&
           d.Dv == kHeadDim && d.block_size == 16 && d.max_q_len >= 2 && g >= 1 &&
           d.Hkv <= 65535 && al(query) && al(out) && encode_fn() != nullptr;
}

// upper bound on the (sequence, tile pair) items of a step
static int paged_tc_capacity(const b2a_paged_desc& d) {
    const long long g = d.Hq / d.Hkv;
    const long long rb = d.prefill_row_blocks > 0 ? d.prefill_row_blocks
                                                  : static_cast<long long>(d.num_tokens) / 128 + d.num_seqs;
    const long long cap = (rb * g + 1) / 2 + (rb < d.num_seqs ? rb : d.num_seqs);  // + one round-up per sequence
    return static_cast<int>(cap < 1 ? 1 : cap);
}

// Layout of the prefill kernel's part of the workspace: [work list][kv_base per sequence][owner per 128-row group]
// [K scratch][V scratch]; the last three only when the caller gave prefill_kv_tokens.
namespace {
struct TcWorkspace {
    size_t kv_base_at, owner_at, k_at, v_at, total;
    int rows, groups;
};
TcWorkspace tc_workspace(const b2a_paged_desc& d) {
    auto up = [](size_t x, size_t a) { return (x + a - 1) / a * a; };
    TcWorkspace w{};
    size_t at = up(sizeof(int) * (kPlanHeaderInts + kPlanEntryInts * static_cast<size_t>(paged_tc_capacity(d))), 16);
    if (d.prefill_kv_tokens > 0) {
        w.rows = (d.prefill_kv_tokens + 127) / 128 * 128;
        w.groups = w.rows / 128;
        w.kv_base_at = at;
        at = up(at + sizeof(int) * static_cast<size_t>(d.num_seqs), 16);
        w.owner_at = at;
        at = up(at + sizeof(int) * static_cast<size_t>(w.groups), 256);
        const size_t scratch = static_cast<size_t>(d.Hkv) * w.rows * kHeadDim * 2;
        w.k_at = at;
        w.v_at = at + scratch;
        at += 2 * scratch;
    }
    w.total = at;
    return w;
}
}  // namespace

size_t paged_tc_plan_bytes(const b2a_paged_desc& d) { return tc_workspace(d).total; }

int paged_tc_launch(const b2a_paged_desc& d, const void* query, const void* k_cache, const void* v_cache,
                    const PagedTables& t, void* out, void* plan_ws, int32_t* status, cudaStream_t stream,
                    bool* decode_may_overlap) {
    const bool bf16 = d.q_dtype == B2A_BF16;
    const int capacity = paged_tc_capacity(d);
    const TcWorkspace w = tc_workspace(d);
    const bool gathered = w.rows > 0;
    char* ws = static_cast<char*>(plan_ws);
    int* kv_base = gathered ? reinterpret_cast<int*>(ws + w.kv_base_at) : nullptr;
    int* owner = gathered ? reinterpret_cast<int*>(ws + w.owner_at) : nullptr;
    const int sms = device_sm_count();
    if (sms <= 0) return B2A_ERR_CUDA;
    const long long bound = static_cast<long long>(capacity) * d.Hkv;
    const int attention_ctas = static_cast<int>(bound < sms ? bound : sms);  // persistent CTAs over the sorted list
    // The decode rows may run beside the prefill rows when the attention kernel is the persistent one (one CTA per SM
    // at most, so what it leaves free is whole SMs) and the caller launches the decode kernel right behind it.
    const bool share = gathered && decode_may_overlap != nullptr;
    if (decode_may_overlap != nullptr) *decode_may_overlap = share;
    if (launch_overlapped(paged_tc_plan_kernel, dim3(1), dim3(256), 0, stream, t, d.Hq / d.Hkv, d.Hkv, capacity,
                          static_cast<int*>(plan_ws), status, kv_base, owner, w.groups, attention_ctas,
                          share ? 1 : 0) != cudaSuccess)
        return B2A_ERR_CUDA;
    // the step's query matrix [tokens, Hq*128] as a [1, Hq, tokens, 128] view
    const int64_t qs[4] = {static_cast<int64_t>(d.num_tokens) * d.Hq * kHeadDim, kHeadDim,
                           static_cast<int64_t>(d.Hq) * kHeadDim, 1};
    CUtensorMap mq, mk, mv;
    if (!make_map(&mq, query, bf16, 1, d.Hq, d.num_tokens, qs, 128)) return B2A_ERR_CUDA;
    mk = mv = mq;  // not read unless K/V are gathered
    if (gathered) {
        uint16_t* ks = reinterpret_cast<uint16_t*>(ws + w.k_at);
        uint16_t* vs = reinterpret_cast<uint16_t*>(ws + w.v_at);
        if (launch_overlapped(paged_gather_kernel, dim3(w.rows / kGatherRows, d.Hkv), dim3(128), 0, stream, t,
                              static_cast<const uint8_t*>(k_cache), static_cast<const uint8_t*>(v_cache), d.Hkv,
                              static_cast<const int*>(kv_base), static_cast<const int*>(owner), w.rows, ks, vs,
                              status) != cudaSuccess)
            return B2A_ERR_CUDA;
        // the scratch as a [1, Hkv, rows, 128] f16 tensor
        const int64_t ss[4] = {static_cast<int64_t>(d.Hkv) * w.rows * kHeadDim, static_cast<int64_t>(w.rows) * kHeadDim,
                               kHeadDim, 1};
        if (!make_map(&mk, ks, false, 1, d.Hkv, w.rows, ss, 128) || !make_map(&mv, vs, false, 1, d.Hkv, w.rows, ss, 128))
            return B2A_ERR_CUDA;
    }
    TcParams p{};
    p.B = 1; p.Hq = d.Hq; p.Hkv = d.Hkv; p.G = d.Hq / d.Hkv; p.Sq = 0; p.Skv = 0;
    p.div_g = fast_div(p.G);
    p.div_hkv = p.div_streams = fast_div(p.Hkv);
    p.out_wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
    p.causal = 1;
    p.window = d.sliding_window;
    p.scale_log2 = d.scale * kLog2e;
    p.status = status;
    p.k_cache = static_cast<const uint8_t*>(k_cache);
    p.v_cache = static_cast<const uint8_t*>(v_cache);
    p.t = t;
    p.out = out;
    p.plan = static_cast<const int*>(plan_ws);
    dim3 grid(capacity, d.Hkv, 1);
    TcPeers peers{};
    constexpr int kSmemPaged = smem_bytes(128 * kHeadDim * 2);
    if (gathered) {
        grid = dim3(static_cast<unsigned>(attention_ctas));
        static OncePerDevice configured[2];
        auto kern = bf16 ? attn_tc_kernel<true, 2> : attn_tc_kernel<false, 2>;
        const int rc = configure_once(kern, configured[bf16], kSmemPaged);
        if (rc != B2A_OK) return rc;
        if (launch_overlapped(kern, grid, dim3(kThreadsDense), kSmemPaged, stream, mq, mk, mv, p, peers) != cudaSuccess) return B2A_ERR_CUDA;
    } else {
        static OncePerDevice configured[2];
        auto kern = bf16 ? attn_tc_kernel<true, 1> : attn_tc_kernel<false, 1>;
        const int rc = configure_once(kern, configured[bf16], kSmemPaged);
        if (rc != B2A_OK) return rc;
        // (only the Q map is read)
        if (launch_overlapped(kern, grid, dim3(kThreadsPaged), kSmemPaged, stream, mq, mq, mq, p, peers) != cudaSuccess) return B2A_ERR_CUDA;
    }
    return B2A_OK;
}

}  // namespace b2a
