// Append this step's K/V rows to the block pools through the block table.
//
// One warp per (token, KV head, K-or-V): it finds the token's sequence by bisection of subsequence_begins, its
// cache position past_lens[s] + offset, the physical block from the block table, and writes the row.  For a u8
// cache the row is quantised per token, asymmetrically, with the scale and zero-point rounded to f16 BEFORE the
// values are quantised, every step a single round-to-nearest-even binary32 operation:
//     s  = f16((max - min) / 255)  (1.0 when that is 0 or not finite)
//     zp = f16(-min / s)
//     q  = clamp(rint(x / s + zp), 0, 255)
// so the bytes and the two f16 values are reproducible bit for bit on a CPU.
//
// Rotary position embedding can be applied to the key rows on the way (b2a_paged_kv_store_rope): the first
// rotary_dim values of a key row, at cache position p, are rotated in pairs (i, i + rotary_dim/2) -
//     x'[i]         = x[i] * cos[p][i] - x[i + r/2] * sin[p][i]
//     x'[i + r/2]   = x[i + r/2] * cos[p][i] + x[i] * sin[p][i]            (r = rotary_dim, i < r/2)
// each product and the sum single round-to-nearest binary32 operations (no fused multiply-add), and the rotated
// float32 values are what is quantised (or rounded to the cache's 16-bit type).  A model then feeds the un-rotated
// key projection to the store and saves the pass that rotates K in memory; queries are rotated by their producer.
#include "launch.cuh"

namespace b2a {
namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kFewPasses = 148 * 32;  // warps that the GPU holds at once, at the kernel's registers

struct StoreParams {
    const void* key;
    const void* value;
    uint8_t* k_cache;
    uint8_t* v_cache;
    PagedTables t;
    int Hkv, D, Dv, kv_dtype;
    int32_t* status;
    // rotary embedding of the key rows (rotary_dim == 0: none): f32 tables [positions][rotary_dim / 2]
    const float* rope_cos;
    const float* rope_sin;
    int rotary_dim, rope_positions;
};

// x[d] of a key row at cache position `pos`, rotated; `own` is x[d], `partner` is x[d +- rotary_dim/2]
__device__ __forceinline__ float rope_value(const StoreParams& p, int pos, int d, float own, float partner) {
    const int half = p.rotary_dim >> 1;
    const int i = d < half ? d : d - half;
    const float c = p.rope_cos[static_cast<size_t>(pos) * half + i], s = p.rope_sin[static_cast<size_t>(pos) * half + i];
    return d < half ? __fsub_rn(__fmul_rn(own, c), __fmul_rn(partner, s)) : __fadd_rn(__fmul_rn(own, c), __fmul_rn(partner, s));
}

// Sequence of token `tok`: the last s with subsequence_begins[s] <= tok, found by the whole warp - every round the 32
// lanes probe 32 evenly spaced entries of the remaining range and a ballot picks the segment, so 65535 sequences take
// four dependent loads instead of sixteen.  Returns -1 for a token outside the scheduled range.
__device__ __forceinline__ int find_sequence(const PagedTables& t, int tok, int lane) {
    if (tok >= t.subsequence_begins[t.num_seqs] || tok < t.subsequence_begins[0]) return -1;
    int lo = 0, hi = t.num_seqs;  // invariant: begins[lo] <= tok < begins[hi]
    while (hi - lo > 1) {
        const int step = (hi - lo + 31) / 32;
        const int probe = lo + lane * step;  // lane 0 probes lo itself
        const bool le = probe < hi && t.subsequence_begins[probe] <= tok;
        const unsigned m = __ballot_sync(0xffffffffu, le);  // a prefix of the lanes (begins are non-decreasing)
        const int last = 31 - __clz(static_cast<int>(m));
        const int nlo = lo + last * step;
        hi = min(hi, nlo + step);
        lo = nlo;
    }
    return lo;
}

template <typename T>
__global__ void __launch_bounds__(kWarpsPerCta * 32) paged_kv_store_kernel(const StoreParams p) {
    const int lane = threadIdx.x & 31;
    const long long item = static_cast<long long>(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
    const long long total = 2LL * p.t.num_tokens * p.Hkv;
    grid_dependency_wait();  // the new key/value rows (and the pool's previous readers) belong to earlier kernels
    grid_launch_dependents();
    if (item >= total) return;
    const int which = static_cast<int>(item % 2);  // 0 = key, 1 = value
    const int hk = static_cast<int>((item / 2) % p.Hkv);
    const int tok = static_cast<int>(item / (2LL * p.Hkv));
    const int D = which ? p.Dv : p.D;

    const int seq = find_sequence(p.t, tok, lane);
    if (seq < 0) return;  // not scheduled
    const int pos = p.t.past_lens[seq] + (tok - p.t.subsequence_begins[seq]);
    const int bs = p.t.block_size;
    const int nblk_seq = p.t.block_indices_begins[seq + 1] - p.t.block_indices_begins[seq];
    if (pos < 0 || pos / bs >= nblk_seq) {
        if (lane == 0) report(p.status, B2A_DEV_BAD_LEN);
        return;
    }
    const int blk = p.t.block_indices[p.t.block_indices_begins[seq] + pos / bs];
    if (blk < 0 || blk >= p.t.num_blocks_total) {
        if (lane == 0) report(p.status, B2A_DEV_BAD_BLOCK);
        return;
    }
    const int slot = pos % bs;
    const T* src = reinterpret_cast<const T*>(which ? p.value : p.key) + (static_cast<size_t>(tok) * p.Hkv + hk) * D;
    uint8_t* cache = which ? p.v_cache : p.k_cache;
    const bool rope = which == 0 && p.rotary_dim > 0;
    if (rope && pos >= p.rope_positions) {  // no table row for this position
        if (lane == 0) report(p.status, B2A_DEV_BAD_LEN);
        return;
    }
    auto value_at = [&](int d) {
        const float x = to_f32<T>(src[d]);
        if (!rope || d >= p.rotary_dim) return x;
        const int half = p.rotary_dim >> 1;
        return rope_value(p, pos, d, x, to_f32<T>(src[d < half ? d + half : d - half]));
    };

    if (p.kv_dtype != B2A_U8) {
        // plain [block_size, D] chunk of f16 / bf16
        uint16_t* dst = reinterpret_cast<uint16_t*>(cache) +
                        ((static_cast<size_t>(blk) * p.Hkv + hk) * bs + slot) * D;
        for (int d = lane; d < D; d += 32) {
            const float x = value_at(d);
            dst[d] = p.kv_dtype == B2A_F16 ? __half_as_ushort(__float2half_rn(x))
                                           : __bfloat16_as_ushort(__float2bfloat16_rn(x));
        }
        return;
    }

    uint8_t* chunk = cache + (static_cast<size_t>(blk) * p.Hkv + hk) * u8_chunk_bytes(bs, D);
    uint8_t* row = chunk + slot * D;
    // D == 128 with 16-bit inputs: each lane keeps its 4 consecutive values in registers (one 8-byte load, one
    // 4-byte store); other sizes take the strided loops below.  Same arithmetic either way.
    const bool vec = !rope && (D == 128) && sizeof(T) == 2 && ((reinterpret_cast<uintptr_t>(src) & 7) == 0);
    float xv[4];
    float mn = INFINITY, mx = -INFINITY;
    if (vec) {
        const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint16_t*>(src) + 4 * lane);
        const T* h = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xv[i] = to_f32<T>(h[i]);
            mn = fminf(mn, xv[i]);
            mx = fmaxf(mx, xv[i]);
        }
    } else {
        for (int d = lane; d < D; d += 32) {
            const float x = value_at(d);
            mn = fminf(mn, x);
            mx = fmaxf(mx, x);
        }
    }
    mx = warp_max(mx);
    mn = -warp_max(-mn);
    __half s16 = __float2half_rn(__fdiv_rn(__fsub_rn(mx, mn), 255.0f));
    float sf = __half2float(s16);
    if (sf == 0.f || isinf(sf) || isnan(sf)) {
        s16 = __float2half_rn(1.0f);
        sf = 1.0f;
    }
    const __half z16 = __float2half_rn(__fdiv_rn(-mn, sf));
    const float zf = __half2float(z16);
    if (vec) {
        uint32_t packed = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float t = rintf(__fadd_rn(__fdiv_rn(xv[i], sf), zf));
            packed |= static_cast<uint32_t>(fminf(fmaxf(t, 0.f), 255.f)) << (8 * i);
        }
        reinterpret_cast<uint32_t*>(row)[lane] = packed;
    } else {
        for (int d = lane; d < D; d += 32) {
            const float x = value_at(d);
            const float t = rintf(__fadd_rn(__fdiv_rn(x, sf), zf));
            row[d] = static_cast<uint8_t>(fminf(fmaxf(t, 0.f), 255.f));
        }
    }
    if (lane == 0) {
        __half* meta = reinterpret_cast<__half*>(chunk + bs * D);
        meta[slot] = s16;
        meta[bs + slot] = z16;
    }
}

// The common geometry (u8 cache, D = Dv = 128, 16-bit rows): a row is handled by EIGHT lanes (16 values each: two
// 16-byte loads, one 16-byte store of codes), so one pass of a warp quantises four rows - the per-row work (min/max
// reduction, now three shuffle steps, the two scalar divisions, addressing) is issued once for four rows.  Same
// arithmetic as above, operation for operation, except that x / s for the row's values uses one reciprocal (see below).
// A large step gives a warp all 2*Hkv rows of a token, so that the walk through the step's tables is paid once for
// them, and reads the next four rows while it quantises these; bound there by instruction issue.  A small step (fewer
// than kFewPasses passes in all: they fit the GPU at once) is a chain of latencies instead, so it gives a warp one pass, and
// the table entries are requested in one go on the guess that the token is its sequence's only one.
// Measured cold, 8 KV heads (before: a warp per token, conversions per value): 2 and 64 f16 tokens 11 -> 4.5 us, 8312 bf16
// tokens 25.6 -> 17.8 us.
template <typename T>
__device__ __forceinline__ float bits_to_f32(uint32_t h16);
template <>
__device__ __forceinline__ float bits_to_f32<__half>(uint32_t h16) {
    return __half2float(__ushort_as_half(static_cast<unsigned short>(h16)));
}
template <>
__device__ __forceinline__ float bits_to_f32<__nv_bfloat16>(uint32_t h16) {
    return __uint_as_float(h16 << 16);
}

// kRope: the key rows are rotated over all 128 values (rotary_dim == 128): a value's partner, 64 further on or back,
// sits at the same place in the registers of the lane four lanes away; rotated values are arbitrary float32
// numbers, for which the reciprocal shortcut below is not proved, so those rows take the division itself.
template <typename T, bool kRope>
__global__ void __launch_bounds__(kWarpsPerCta * 32, kRope ? 2 : 4) paged_kv_store_rows128_kernel(const StoreParams p, const int passes_per_warp) {
    constexpr int D = 128;
    const int lane = threadIdx.x & 31, l8 = lane & 7, rg = lane >> 3;
    const int rows = 2 * p.Hkv;  // row r: head r >> 1, key (0) or value (1)
    const int passes = (rows + 3) / 4, warps_per_token = (passes + passes_per_warp - 1) / passes_per_warp;
    const long long item = static_cast<long long>(blockIdx.x) * kWarpsPerCta + (threadIdx.x >> 5);
    const int tok = static_cast<int>(item / warps_per_token);
    const int first = static_cast<int>(item - static_cast<long long>(tok) * warps_per_token) * passes_per_warp * 4;
    const int last = min(rows, first + passes_per_warp * 4);
    grid_dependency_wait();  // the new key/value rows (and the pool's previous readers) belong to earlier kernels
    grid_launch_dependents();
    if (tok >= p.t.num_tokens) return;
    uint4 next0 = make_uint4(0u, 0u, 0u, 0u), next1 = next0;
    auto fetch = [&](int r) {  // this lane's 16 values of row r
        if (r < last) {
            const uint4* src = reinterpret_cast<const uint4*>(
                reinterpret_cast<const T*>((r & 1) ? p.value : p.key) + (static_cast<size_t>(tok) * p.Hkv + (r >> 1)) * D);
            next0 = src[2 * l8];
            next1 = src[2 * l8 + 1];
        }
    };
    fetch(first + rg);
    // the token's sequence: itself in a step of one-token sequences, else by search; the entries of the guess are
    // requested together with the two that confirm it
    int seq = -1, past = 0, begin = 0, bib0 = 0, bib1 = 0;
    if (tok < p.t.num_seqs) {
        const int b0 = p.t.subsequence_begins[0], bn = p.t.subsequence_begins[p.t.num_seqs];
        const int mine = p.t.subsequence_begins[tok], after = p.t.subsequence_begins[tok + 1];
        past = p.t.past_lens[tok];
        bib0 = p.t.block_indices_begins[tok];
        bib1 = p.t.block_indices_begins[tok + 1];
        begin = mine;
        if (mine <= tok && tok < after && b0 <= tok && tok < bn) seq = tok;
    }
    if (seq < 0) {
        seq = find_sequence(p.t, tok, lane);
        if (seq < 0) return;  // not scheduled
        past = p.t.past_lens[seq];
        begin = p.t.subsequence_begins[seq];
        bib0 = p.t.block_indices_begins[seq];
        bib1 = p.t.block_indices_begins[seq + 1];
    }
    const int pos = past + (tok - begin);
    const int bs = p.t.block_size;
    if (pos < 0 || pos / bs >= bib1 - bib0) {
        if (lane == 0) report(p.status, B2A_DEV_BAD_LEN);
        return;
    }
    const int blk = p.t.block_indices[bib0 + pos / bs];
    if (blk < 0 || blk >= p.t.num_blocks_total) {
        if (lane == 0) report(p.status, B2A_DEV_BAD_BLOCK);
        return;
    }
    const int slot = pos % bs;
    if (kRope && pos >= p.rope_positions) {  // no table row for this position
        if (lane == 0) report(p.status, B2A_DEV_BAD_LEN);
        return;
    }
    const size_t chunk_bytes = u8_chunk_bytes(bs, D);
    for (int r0 = first; r0 < last; r0 += 4) {
        const int r = r0 + rg;
        const bool live = r < last;  // whole 8-lane groups are live or not: the shuffles below stay inside a group
        const uint32_t w[8] = {next0.x, next0.y, next0.z, next0.w, next1.x, next1.y, next1.z, next1.w};
        fetch(r + 4);
        float xv[16];
        float mn = INFINITY, mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            xv[2 * i] = bits_to_f32<T>(w[i] & 0xffffu);
            xv[2 * i + 1] = bits_to_f32<T>(w[i] >> 16);
        }
        const bool rotated = kRope && (r & 1) == 0;  // key rows
        if constexpr (kRope) {
            // lane l8 holds values 16*l8 .. +15: partners are in lane l8 ^ 4 (every lane takes part in the exchange)
#pragma unroll
            for (int e = 0; e < 16; ++e) {
                const float partner = __shfl_xor_sync(0xffffffffu, xv[e], 4);
                if (rotated) xv[e] = rope_value(p, pos, 16 * l8 + e, xv[e], partner);
            }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            mn = fminf(mn, xv[e]);
            mx = fmaxf(mx, xv[e]);
        }
#pragma unroll
        for (int o = 1; o <= 4; o <<= 1) {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        }
        __half s16 = __float2half_rn(__fdiv_rn(__fsub_rn(mx, mn), 255.0f));
        float sf = __half2float(s16);
        if (sf == 0.f || isinf(sf) || isnan(sf)) {
            s16 = __float2half_rn(1.0f);
            sf = 1.0f;
        }
        const __half z16 = __float2half_rn(__fdiv_rn(-mn, sf));
        const float zf = __half2float(z16);
        // x / s for the row's values with ONE reciprocal: q0 = x * r, then one Newton step in fused arithmetic.
        // For a scale that is an f16 value and x an f16 or bf16 value this equals the correctly rounded quotient in
        // every case except |x| below 2^-116 (checked exhaustively on the CPU by oracle/div_by_scale_check.c) - and
        // such a quotient, below 2^-92 whichever way it is rounded (s is at least 2^-24), is lost in the sum with zp,
        // zero or at least 2^-24: the code is the same.  A row with an infinity (or without a number) has s = 1:
        // x / s is x, where the Newton step would make a NaN of it.
        // rint and clamp commute (the bounds are integers), and adding 2^23 to a value in 0..255 rounds it to an
        // integer, ties to even, in the low byte: no conversion instruction, whose rate is a quarter of the adder's.
        const bool finite = mn > -INFINITY && mx < INFINITY && mn <= mx;
        const float rs = __frcp_rn(sf);
        uint32_t packed[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t code[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float x = xv[4 * i + u];
                float q;
                if (kRope && rotated) {
                    q = __fdiv_rn(x, sf);
                } else {
                    const float q0 = __fmul_rn(x, rs);
                    const float q1 = __fmaf_rn(__fmaf_rn(-sf, q0, x), rs, q0);
                    q = finite ? q1 : x;
                }
                code[u] = __float_as_uint(__fadd_rn(fminf(fmaxf(__fadd_rn(q, zf), 0.f), 255.f), 8388608.f));
            }
            packed[i] = __byte_perm(__byte_perm(code[0], code[1], 0x0040), __byte_perm(code[2], code[3], 0x0040), 0x5410);
        }
        if (live) {
            uint8_t* chunk = ((r & 1) ? p.v_cache : p.k_cache) + (static_cast<size_t>(blk) * p.Hkv + (r >> 1)) * chunk_bytes;
            reinterpret_cast<uint4*>(chunk + slot * D)[l8] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            if (l8 == 0) {
                __half* meta = reinterpret_cast<__half*>(chunk + bs * D);
                meta[slot] = s16;
                meta[bs + slot] = z16;
            }
        }
    }
}

// A pool of the rows' own 16-bit type: the rows are copied, a thread per 16 bytes of a token's key or value rows, K first.  Bound by
// its chain of loads: rows and tables in one trip (the entries on the guess that the token is its sequence's only one, as
// above), the block id in a second, where a warp per row with the search in front took seven.  (Through float32 and back, as
// every 16-bit row is stored: only a NaN's bits change.)  8 KV heads x 128, us, a warp per row and now: 8 tokens 3.1 and 1.9, 812
// tokens of two sequences 7.4 and 3.4, 4096 tokens 24.9 and 8.7.
template <typename T>
__global__ void __launch_bounds__(256) paged_kv_copy_rows_kernel(const StoreParams p, const int pieces_per_token) {
    const int lane = threadIdx.x & 31;
    const long long piece = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
    const int tok = static_cast<int>(piece / pieces_per_token);  // (a multiple of 32 pieces a token: the same in all of a warp)
    const int at = static_cast<int>(piece - static_cast<long long>(tok) * pieces_per_token);
    grid_dependency_wait();  // the new key/value rows (and the pool's previous readers) belong to earlier kernels
    grid_launch_dependents();
    if (tok >= p.t.num_tokens) return;
    const int half = pieces_per_token / 2, which = at >= half, e = at - which * half;  // 0 = key, 1 = value
    uint4 row = reinterpret_cast<const uint4*>(which ? p.value : p.key)[static_cast<size_t>(tok) * half + e];
    int seq = -1, past = 0, begin = 0, bib0 = 0, bib1 = 0;
    if (tok < p.t.num_seqs) {
        const int b0 = p.t.subsequence_begins[0], bn = p.t.subsequence_begins[p.t.num_seqs];
        const int mine = p.t.subsequence_begins[tok], after = p.t.subsequence_begins[tok + 1];
        past = p.t.past_lens[tok];
        bib0 = p.t.block_indices_begins[tok];
        bib1 = p.t.block_indices_begins[tok + 1];
        begin = mine;
        if (mine <= tok && tok < after && b0 <= tok && tok < bn) seq = tok;
    }
    if (seq < 0) {
        seq = find_sequence(p.t, tok, lane);
        if (seq < 0) return;  // not scheduled
        past = p.t.past_lens[seq];
        begin = p.t.subsequence_begins[seq];
        bib0 = p.t.block_indices_begins[seq];
        bib1 = p.t.block_indices_begins[seq + 1];
    }
    const int pos = past + (tok - begin), bs = p.t.block_size;
    if (pos < 0 || pos / bs >= bib1 - bib0) {
        if (lane == 0) report(p.status, B2A_DEV_BAD_LEN);
        return;
    }
    const int blk = p.t.block_indices[bib0 + pos / bs];
    if (blk < 0 || blk >= p.t.num_blocks_total) {
        if (lane == 0) report(p.status, B2A_DEV_BAD_BLOCK);
        return;
    }
    const int row_pieces = p.D / 8, hk = e / row_pieces;
    uint4* dst = reinterpret_cast<uint4*>(which ? p.v_cache : p.k_cache) +
                 ((static_cast<size_t>(blk) * p.Hkv + hk) * bs + pos % bs) * row_pieces + (e - hk * row_pieces);
    T* h = reinterpret_cast<T*>(&row);
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = from_f32<T>(to_f32<T>(h[i]));
    *dst = row;
}

}  // namespace

int paged_kv_store_launch(const b2a_paged_desc& d, const void* key, const void* value, void* k_cache, void* v_cache,
                          const PagedTables& t, int32_t* status, cudaStream_t stream, const RopeTables* rope) {
    if (d.num_tokens == 0) return B2A_OK;
    StoreParams p{key, value, static_cast<uint8_t*>(k_cache), static_cast<uint8_t*>(v_cache), t,
                  d.Hkv, d.D, d.Dv, d.kv_dtype, status, nullptr, nullptr, 0, 0};
    if (rope != nullptr && rope->rotary_dim > 0) {
        p.rope_cos = rope->cos;
        p.rope_sin = rope->sin;
        p.rotary_dim = rope->rotary_dim;
        p.rope_positions = rope->positions;
    }
    const bool rope_all = p.rotary_dim == 128;
    auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    if (d.kv_dtype == B2A_U8 && d.D == 128 && d.Dv == 128 && (d.q_dtype == B2A_F16 || d.q_dtype == B2A_BF16) &&
        al16(key) && al16(value) && (p.rotary_dim == 0 || rope_all)) {
        const int passes = (2 * d.Hkv + 3) / 4;
        const int per_warp = static_cast<long long>(d.num_tokens) * passes <= kFewPasses ? 1 : passes;
        const long long warps = static_cast<long long>(d.num_tokens) * ((passes + per_warp - 1) / per_warp);
        const unsigned grid_t = static_cast<unsigned>((warps + kWarpsPerCta - 1) / kWarpsPerCta);
        const dim3 block(kWarpsPerCta * 32);
        cudaError_t e;
        if (d.q_dtype == B2A_F16)
            e = rope_all ? launch_overlapped(paged_kv_store_rows128_kernel<__half, true>, dim3(grid_t), block, 0, stream, p, per_warp)
                         : launch_overlapped(paged_kv_store_rows128_kernel<__half, false>, dim3(grid_t), block, 0, stream, p, per_warp);
        else
            e = rope_all ? launch_overlapped(paged_kv_store_rows128_kernel<__nv_bfloat16, true>, dim3(grid_t), block, 0, stream, p, per_warp)
                         : launch_overlapped(paged_kv_store_rows128_kernel<__nv_bfloat16, false>, dim3(grid_t), block, 0, stream, p, per_warp);
        return e == cudaSuccess ? B2A_OK : B2A_ERR_CUDA;
    }
    // (equal head sizes, and whole warps per token)
    const long long pieces = 2LL * d.Hkv * d.D / 8;
    if (d.kv_dtype != B2A_U8 && d.kv_dtype == d.q_dtype && d.D == d.Dv && d.D % 8 == 0 && pieces % 32 == 0 && pieces < (1 << 20) &&
        p.rotary_dim == 0 && al16(key) && al16(value) && al16(k_cache) && al16(v_cache)) {
        const unsigned grid_c = static_cast<unsigned>((pieces * d.num_tokens + 255) / 256);
        return launch_overlapped(d.kv_dtype == B2A_F16 ? paged_kv_copy_rows_kernel<__half> : paged_kv_copy_rows_kernel<__nv_bfloat16>, dim3(grid_c), dim3(256), 0, stream, p, static_cast<int>(pieces)) == cudaSuccess
                   ? B2A_OK
                   : B2A_ERR_CUDA;
    }
    const long long total = 2LL * d.num_tokens * d.Hkv;
    const unsigned grid = static_cast<unsigned>((total + kWarpsPerCta - 1) / kWarpsPerCta);
    void (*kern)(StoreParams) = nullptr;
    switch (d.q_dtype) {
        case B2A_F32: kern = paged_kv_store_kernel<float>; break;
        case B2A_F16: kern = paged_kv_store_kernel<__half>; break;
        case B2A_BF16: kern = paged_kv_store_kernel<__nv_bfloat16>; break;
        default: return B2A_ERR_DTYPE;
    }
    return launch_overlapped(kern, dim3(grid), dim3(kWarpsPerCta * 32), 0, stream, p) == cudaSuccess ? B2A_OK : B2A_ERR_CUDA;
}

}  // namespace b2a
