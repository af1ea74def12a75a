// Few query rows over 16-bit keys and values: token generation on a dense K/V cache (ScaledDotProductAttention with one
// or a few query rows) and decode rows over an f16 / bf16 block pool (PagedAttentionExtension).  D = Dv = 64 or 128,
// at most sixteen query rows per KV head (its query heads times the query positions).
//
// Bound by HBM: every cached token is 2 * D * 2 bytes per KV head, read once for all the query heads that share it.
// Both contractions run on the warp-level MMA (m16n8k16) with the keys / the value columns as the M side, so a KV
// head's rows fill the N side and the instruction count follows the bytes (sixteen keys: 8 KB and 24 to 32 MMAs at D = 128).
//
// One launch, no workspace: a CLUSTER of up to eight CTAs owns one (sequence, KV head).  The sequence's 16-key tiles
// are cut evenly over the cluster whatever its length, each of a CTA's four warps walks its share with its own cp.async
// pipeline and online softmax, and the partial results (maximum, sum, O) are merged in the CTA's shared memory and then
// across the cluster through distributed shared memory, every CTA finishing its slice of the output columns.
// (A workspace would have to be asked of callers that never needed one, and a merge kernel costs a launch.)
//
// The probabilities keep float32's precision and, as far as a row can tell, its range: they enter the second product as two
// f16 or three bf16 values (ProbPieces), which costs eight or sixteen more MMAs per tile where the tensor pipe idles anyway.
//
// Measured on a B200 (graph replay): bf16, 8 sequences x 3003 keys x 8 KV heads, additive mask (98 MB): 2049 us on
// attn_generic_kernel before, 21.2 us now (4.6 TB/s; 15.1 us at the copy rate); 32 bf16 sequences of 256..4096 tokens in
// a pool (293 MB, with the store of the step): 8149 us before, 52.3 us now (5.6 TB/s; 44.8 us at the copy rate).
// On another box and before a cheaper floor for the mask: two bf16 pieces, which keep 2^-16 of a probability, 22.8 and 55.3 us,
// three 23.3 and 56.5, two tf32 pieces beside V widened to tf32 24.0 and 59.5.
#include <algorithm>

#include "launch.cuh"

namespace b2a {
namespace {

constexpr int kWarps = 4;
constexpr int kTileKeys = 16;
constexpr int kMaxCluster = 8;          // the portable limit
constexpr unsigned kSeats = 148 * 2;    // CTAs that the GPU holds at once
constexpr float kNegBig = -1.0e30f;     // finite "minus infinity": start of the running maximum, floor of finite masks

struct Dec16Params {
    const uint8_t* q;
    const uint8_t* k;
    const uint8_t* v;
    uint8_t* o;
    const uint8_t* mask;
    int mask_kind;
    int Hq, G, rows, Sq, Skv, causal;
    float scale_log2;
    // byte strides: batch, head, position
    int64_t q_b, q_h, q_s, k_b, k_h, k_s, v_b, v_h, v_s, o_b, o_h, o_s;
    int64_t m_b, m_h, m_s, m_k;  // element strides of the mask
    // paged pools: k_h / v_h are the chunk sizes, k_b / v_b the block sizes, k_s / v_s the rows
    PagedTables t;
    int sliding_window;
    int32_t* status;
};

__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(pol));
    return pol;
}
// 16 bytes, or 16 zero bytes when `bytes` is 0
__device__ __forceinline__ void cp_async16z(uint32_t dst, const void* src, int bytes, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;\n" ::"r"(dst), "l"(src), "r"(bytes), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma16816<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma16816<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Factor on the probabilities before they are cut into pieces (ProbPieces), carried by the row sum: f16's pieces reach down to
// 2^-49 of the row's maximum with it.
template <typename T>
constexpr float kPieceScale = 1.f;
template <>
constexpr float kPieceScale<__half> = 16384.f;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 ld_cluster2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

template <int D>
constexpr int tile_bytes() { return 2 * kTileKeys * D * 2; }  // K and V of sixteen keys
// Copy stages of a warp: 24 KB per warp at either head size, two CTAs (eight warps, 192 KB) per SM
template <int D>
constexpr int stages() { return D == 128 ? 3 : 6; }
template <int D, int NT>
constexpr int part_floats() { return NT * 8 * D + 2 * NT * 8; }  // O, then maximum and sum of every row
template <int D, int NT>
constexpr int smem_bytes() { return kWarps * stages<D>() * tile_bytes<D>() + part_floats<D, NT>() * 4; }

// One mask value in base-2 score units.  A finite additive value stays finite (a row whose every key carries the
// type's lowest value averages its values, as softmax of equal scores does); -inf and a false boolean remove the key.
template <typename T>
__device__ __forceinline__ float mask_value(const Dec16Params& p, int64_t at) {
    if (p.mask_kind == B2A_MASK_BOOL) return p.mask[at] != 0 ? 0.f : -INFINITY;
    const float m = to_f32<T>(reinterpret_cast<const T*>(p.mask)[at]), v = m * kLog2e;
    return v < kNegBig && m != -INFINITY ? kNegBig : v;  // (a NaN stays one)
}

// Grid (cluster size, KV heads, sequences); cluster (size, 1, 1).  NT: groups of eight query rows.
template <typename T, int NT, int D, bool kPaged>
__global__ void __launch_bounds__(kWarps * 32, 2) attn_decode16_kernel(const Dec16Params p) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int kStages = stages<D>();
    constexpr int kRowBytes = D * 2, kChunks = kRowBytes / 16;  // 16-byte pieces of a row
    constexpr int kHalfTile = kTileKeys * kRowBytes;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gid = lane >> 2, tid4 = lane & 3;
    const int csize = static_cast<int>(gridDim.x), split = static_cast<int>(cluster_rank());
    const int hk = blockIdx.y, seq = blockIdx.z;

    // ---- the keys of this (sequence, KV head), in 16-key tiles
    int kv_end = 0, first_pos = 0, tok = 0, bib0 = 0;
    bool bad = false, decode_row = true;
    if constexpr (kPaged) {
        tok = __ldcg(p.t.subsequence_begins + seq);
        const int tok_end = __ldcg(p.t.subsequence_begins + seq + 1);
        const int past = __ldcg(p.t.past_lens + seq);
        bib0 = __ldcg(p.t.block_indices_begins + seq);
        const int bib1 = __ldcg(p.t.block_indices_begins + seq + 1);
        kv_end = past + 1;
        first_pos = p.sliding_window > 0 ? max(0, kv_end - p.sliding_window) : 0;
        decode_row = tok_end - tok == 1;  // the others belong to the multi-token kernel
        bad = decode_row && (past < 0 || tok < 0 || tok >= p.t.num_tokens ||
                             (kv_end + p.t.block_size - 1) / p.t.block_size > bib1 - bib0);
    } else {
        kv_end = p.causal ? min(p.Skv, p.Sq) : p.Skv;
        grid_dependency_wait();
        grid_launch_dependents();
    }
    const int tile_lo = first_pos / kTileKeys;
    const int tiles = (kv_end + kTileKeys - 1) / kTileKeys - tile_lo;
    const int per_cta = (tiles + csize - 1) / csize;
    const int my_lo = tile_lo + min(tiles, split * per_cta), my_hi = tile_lo + min(tiles, (split + 1) * per_cta);
    const int n_w = decode_row && !bad ? max(0, (my_hi - my_lo - warp + kWarps - 1) / kWarps) : 0;  // tiles my_lo + warp + kWarps * i

    const uint32_t smem_warp = static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + warp * (kStages * tile_bytes<D>());
    const uint64_t policy = evict_first_policy();
    // paged: lanes hold the block ids of a window of 32 tiles; the copies run ahead of the arithmetic, so the window
    // follows the copies and a stage remembers in a bit whether its block was usable
    int window_ids = -1;
    uint32_t stage_ok = 0;
    bool bad_block = false;
    auto load_window = [&](int i0) {
        window_ids = -1;
        if (i0 + lane < n_w) {
            const int key = (my_lo + warp + kWarps * (i0 + lane)) * kTileKeys;
            window_ids = __ldcg(p.t.block_indices + bib0 + key / p.t.block_size);
            if (window_ids < 0 || window_ids >= p.t.num_blocks_total) {
                bad_block = true;
                window_ids = -1;
            }
        }
    };
    const uint8_t *kb, *vb;  // dense: this (batch entry, KV head); paged: this KV head of block 0
    if constexpr (kPaged) {
        kb = p.k + hk * p.k_h;
        vb = p.v + hk * p.v_h;
    } else {
        kb = p.k + seq * p.k_b + hk * p.k_h;
        vb = p.v + seq * p.v_b + hk * p.v_h;
    }
    constexpr int kRowsPerCopy = 32 / kChunks;  // rows that one warp-wide copy covers: 2 or 4
    const int c_row = lane / kChunks, c_col = lane % kChunks;
    auto issue = [&](int i) {
        const int key0 = (my_lo + warp + kWarps * i) * kTileKeys;
        const uint8_t *ks, *vs;
        bool usable = true;
        if constexpr (kPaged) {
            if ((i & 31) == 0 && i > 0) load_window(i);
            const int phys = __shfl_sync(0xffffffffu, window_ids, i & 31);
            usable = phys >= 0;
            const int slot = key0 % p.t.block_size;
            ks = kb + static_cast<int64_t>(max(phys, 0)) * p.k_b + slot * kRowBytes;
            vs = vb + static_cast<int64_t>(max(phys, 0)) * p.v_b + slot * kRowBytes;
        } else {
            ks = kb + key0 * p.k_s;
            vs = vb + key0 * p.v_s;
        }
        const int st_i = i % kStages;
        stage_ok = (stage_ok & ~(1u << st_i)) | (usable ? 1u << st_i : 0u);
        const uint32_t st = smem_warp + st_i * tile_bytes<D>();
#pragma unroll
        for (int r = 0; r < kTileKeys / kRowsPerCopy; ++r) {
            const int row = r * kRowsPerCopy + c_row;
            const uint32_t off = row * kRowBytes + ((c_col ^ (row & 7)) << 4);
            // rows past the last key become zeros: 0 * whatever an unused cache slot holds could be NaN
            const bool in = usable && key0 + row < kv_end;
            const int64_t at_k = in ? (kPaged ? static_cast<int64_t>(row) * kRowBytes : row * p.k_s) + c_col * 16 : 0;
            const int64_t at_v = in ? (kPaged ? static_cast<int64_t>(row) * kRowBytes : row * p.v_s) + c_col * 16 : 0;
            cp_async16z(st + off, in ? ks + at_k : kb, in ? 16 : 0, policy);
            cp_async16z(st + kHalfTile + off, in ? vs + at_v : vb, in ? 16 : 0, policy);
        }
    };
    auto fill = [&]() {
#pragma unroll
        for (int s = 0; s < kStages - 1; ++s) {
            if (s < n_w) issue(s);
            cp_async_commit();
        }
    };
    if constexpr (kPaged) {
        // The step's tables exist before its kernels are launched, so the block ids are read while the kernel in front, as a rule
        // the step's store, drains, and the first wave's CTAs ask their first tiles into L2.  Not into shared memory: a block that this sequence
        // holds as cached may be one that another sequence's new token goes into (prefixes shared within a step), and only
        // what is read behind the wait is sure to show that row.  Cold pools, f16, 8 KV heads, us a step with the store, without
        // the prefetch and with it: 2 sequences of 300..900 tokens 7.9 and 7.5, 8 of 2000 21.4 and 20.3, 32 of 256..4096 53.7
        // and 51.7.  (Copies into shared memory here, of the tiles before a sequence's last: 7.2, 21.1 and 53.1.)
        load_window(0);
        if (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z) < kSeats) {
#pragma unroll
            for (int s = 0; s < kStages - 1; ++s) {
                const int phys = __shfl_sync(0xffffffffu, window_ids, s);
                if (s < n_w && phys >= 0 && lane < 2) {
                    const int key0 = (my_lo + warp + kWarps * s) * kTileKeys;
                    const int64_t at = static_cast<int64_t>(phys) * p.k_b + key0 % p.t.block_size * kRowBytes;
                    prefetch_l2((lane == 0 ? kb : vb) + at, kHalfTile);
                }
            }
        }
        grid_dependency_wait();
        grid_launch_dependents();
        if (bad && split == 0 && tid == 0) report(p.status, B2A_DEV_BAD_LEN);
        if (!decode_row || bad) return;  // the same decision in every CTA of the cluster
    }
    fill();

    // ---- query rows as the B operand of S^T = K Q^T: row r = g * Sq + i is query position i of the group's head g
    auto row_base = [&](const uint8_t* base, int64_t sb, int64_t sh, int64_t ss, int r) {
        const int g = r / p.Sq, i = r - g * p.Sq;
        return base + (kPaged ? static_cast<int64_t>(tok) * sb : seq * sb) + (hk * p.G + g) * sh + i * ss;
    };
    uint32_t qf[NT][D / 16][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int r = nt * 8 + gid;
        const uint8_t* qrow = row_base(p.q, p.q_b, p.q_h, p.q_s, min(r, p.rows - 1));
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {
            qf[nt][j][0] = r < p.rows ? *reinterpret_cast<const uint32_t*>(qrow + (j * 16 + 2 * tid4) * 2) : 0u;
            qf[nt][j][1] = r < p.rows ? *reinterpret_cast<const uint32_t*>(qrow + (j * 16 + 8 + 2 * tid4) * 2) : 0u;
        }
    }
    // of this thread's two rows per group of eight (2 * tid4, + 1): where their keys end, and their mask rows
    int row_end[NT][2];
    int64_t mrow[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = min(nt * 8 + 2 * tid4 + e, p.rows - 1);
            const int g = r / p.Sq, i = r - g * p.Sq;
            row_end[nt][e] = !kPaged && p.causal ? min(kv_end, i + 1) : kv_end;
            mrow[nt][e] = kPaged ? 0 : seq * p.m_b + (hk * p.G + g) * p.m_h + i * p.m_s;
        }
    const bool masked = !kPaged && p.mask_kind != B2A_MASK_NONE;
    float mv[NT][4];
    auto load_mask = [&](int i) {  // token gid: rows a, b; token gid + 8: rows a, b
        const int key0 = (my_lo + warp + kWarps * i) * kTileKeys + gid;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int key = key0 + (e >> 1) * 8;
                mv[nt][e] = key < kv_end ? mask_value<T>(p, mrow[nt][e & 1] + key * p.m_k) : 0.f;
            }
    };
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) mv[nt][0] = mv[nt][1] = mv[nt][2] = mv[nt][3] = 0.f;
    if (masked && n_w > 0) load_mask(0);

    using P = ProbPieces<T>;
    float acc[NT][P::kAccs][D / 16][4];
    float m_a[NT], m_b[NT], l_a[NT], l_b[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        m_a[nt] = m_b[nt] = kNegBig;
        l_a[nt] = l_b[nt] = 0.f;
#pragma unroll
        for (int a = 0; a < P::kAccs; ++a)
#pragma unroll
            for (int j = 0; j < D / 16; ++j) acc[nt][a][j][0] = acc[nt][a][j][1] = acc[nt][a][j][2] = acc[nt][a][j][3] = 0.f;
    }

    const int mat = lane >> 3, mrow8 = lane & 7;  // ldmatrix: matrix and row whose address this lane supplies
    for (int i = 0; i < n_w; ++i) {
        const bool blk_ok = (stage_ok >> (i % kStages)) & 1u;  // before the copy below reuses the bit of stage i - 1
        if (i + kStages - 1 < n_w) issue(i + kStages - 1);
        cp_async_commit();
        cp_async_wait<kStages - 1>();
        __syncwarp();
        const uint32_t sK = smem_warp + (i % kStages) * tile_bytes<D>(), sV = sK + kHalfTile;
        const int pos0 = (my_lo + warp + kWarps * i) * kTileKeys + gid, pos1 = pos0 + 8;

        float sc[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) sc[nt][0] = sc[nt][1] = sc[nt][2] = sc[nt][3] = 0.f;
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {
            // A = K: matrices (keys 0-7, d 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15) of the 16 x 16 piece
            const int row = (mat & 1) * 8 + mrow8, col = 2 * j + (mat >> 1);
            uint32_t a[4];
            ldmatrix4(sK + row * kRowBytes + ((col ^ (row & 7)) << 4), a);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) mma16816<T>(sc[nt], a, qf[nt][j][0], qf[nt][j][1]);
        }
        uint32_t pp[NT][P::kCount][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            float s0 = fmaf(sc[nt][0], p.scale_log2, mv[nt][0]), s1 = fmaf(sc[nt][1], p.scale_log2, mv[nt][1]);
            float s2 = fmaf(sc[nt][2], p.scale_log2, mv[nt][2]), s3 = fmaf(sc[nt][3], p.scale_log2, mv[nt][3]);
            if (!(blk_ok && pos0 < row_end[nt][0] && pos0 >= first_pos)) s0 = -INFINITY;
            if (!(blk_ok && pos0 < row_end[nt][1] && pos0 >= first_pos)) s1 = -INFINITY;
            if (!(blk_ok && pos1 < row_end[nt][0] && pos1 >= first_pos)) s2 = -INFINITY;
            if (!(blk_ok && pos1 < row_end[nt][1] && pos1 >= first_pos)) s3 = -INFINITY;
            float ta = fmaxf(s0, s2), tb = fmaxf(s1, s3);
#pragma unroll
            for (int o = 4; o <= 16; o <<= 1) {
                ta = fmaxf(ta, __shfl_xor_sync(0xffffffffu, ta, o));
                tb = fmaxf(tb, __shfl_xor_sync(0xffffffffu, tb, o));
            }
            const float na = fmaxf(m_a[nt], ta), nb = fmaxf(m_b[nt], tb);
            const float alpha_a = ex2(m_a[nt] - na), alpha_b = ex2(m_b[nt] - nb);
            m_a[nt] = na;
            m_b[nt] = nb;
            const float p0 = ex2(s0 - na), p1 = ex2(s1 - nb), p2 = ex2(s2 - na), p3 = ex2(s3 - nb);
            l_a[nt] = l_a[nt] * alpha_a + p0 + p2;
            l_b[nt] = l_b[nt] * alpha_b + p1 + p3;
            uint32_t w0[P::kCount], w1[P::kCount];
            P::split(p0 * kPieceScale<T>, p1 * kPieceScale<T>, w0);
            P::split(p2 * kPieceScale<T>, p3 * kPieceScale<T>, w1);
#pragma unroll
            for (int e = 0; e < P::kCount; ++e) {
                pp[nt][e][0] = movmatrix_trans(w0[e]);
                pp[nt][e][1] = movmatrix_trans(w1[e]);
            }
            if (__any_sync(0xffffffffu, alpha_a != 1.f || alpha_b != 1.f)) {
#pragma unroll
                for (int a = 0; a < P::kAccs; ++a)
#pragma unroll
                    for (int j = 0; j < D / 16; ++j) {
                        acc[nt][a][j][0] *= alpha_a;
                        acc[nt][a][j][1] *= alpha_b;
                        acc[nt][a][j][2] *= alpha_a;
                        acc[nt][a][j][3] *= alpha_b;
                    }
            }
        }
        if (masked && i + 1 < n_w) load_mask(i + 1);
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {
            // A = V^T: matrices (d 0-7, keys 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15), stored [key][d]
            const int row = (mat >> 1) * 8 + mrow8, col = 2 * j + (mat & 1);
            uint32_t a[4];
            ldmatrix4_trans(sV + row * kRowBytes + ((col ^ (row & 7)) << 4), a);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < P::kCount; ++e) mma16816<T>(acc[nt][e < P::kAccs ? e : P::kAccs - 1][j], a, pp[nt][e][0], pp[nt][e][1]);
        }
        __syncwarp();  // every lane is done with this stage before it is refilled
    }
    cp_async_wait<0>();
    __syncwarp();
    if (bad_block) report(p.status, B2A_DEV_BAD_BLOCK);

    // ---- the warp's partial into its own stage memory
    constexpr int GP = NT * 8;
    float* wbuf = reinterpret_cast<float*>(smem + warp * (kStages * tile_bytes<D>()));
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
        for (int o = 4; o <= 16; o <<= 1) {
            l_a[nt] += __shfl_xor_sync(0xffffffffu, l_a[nt], o);
            l_b[nt] += __shfl_xor_sync(0xffffffffu, l_b[nt], o);
        }
        const int ra = nt * 8 + 2 * tid4, rb = ra + 1;
#pragma unroll
        for (int j = 0; j < D / 16; ++j) {  // accumulator rows: d = 16 j + gid, + 8; columns: rows a, b
            float o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                o[i] = acc[nt][0][j][i];
                if constexpr (P::kAccs == 2) o[i] = fmaf(acc[nt][1][j][i], P::kLowScale, o[i]);
            }
            wbuf[ra * D + 16 * j + gid] = o[0];
            wbuf[rb * D + 16 * j + gid] = o[1];
            wbuf[ra * D + 16 * j + gid + 8] = o[2];
            wbuf[rb * D + 16 * j + gid + 8] = o[3];
        }
        if (gid == 0) {  // (f16: O carries the pieces' factor, so the sums do too)
            wbuf[GP * D + ra] = m_a[nt];
            wbuf[GP * D + rb] = m_b[nt];
            wbuf[GP * D + GP + ra] = l_a[nt] * kPieceScale<T>;
            wbuf[GP * D + GP + rb] = l_b[nt] * kPieceScale<T>;
        }
    }
    __syncthreads();

    // ---- the CTA's partial: merge of its warps
    float* part = reinterpret_cast<float*>(smem + kWarps * kStages * tile_bytes<D>());
    constexpr int kWarpFloats = kStages * tile_bytes<D>() / 4;
    const float* w0 = reinterpret_cast<const float*>(smem);
    for (int e = tid; e < p.rows * D; e += kWarps * 32) {
        const int r = e / D;
        float mc = kNegBig;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) mc = fmaxf(mc, w0[w * kWarpFloats + GP * D + r]);
        float o = 0.f, l = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float f = ex2(w0[w * kWarpFloats + GP * D + r] - mc);
            o += w0[w * kWarpFloats + e] * f;
            l += w0[w * kWarpFloats + GP * D + GP + r] * f;
        }
        part[e] = o;
        if (e % D == 0) {
            part[GP * D + r] = mc;
            part[GP * D + GP + r] = l;
        }
    }
    cluster_sync();  // every CTA's partial is complete and visible to its peers

    // ---- the output: this CTA finishes every csize-th run of 32 column pairs
    const uint32_t part_addr = static_cast<uint32_t>(__cvta_generic_to_shared(part));
    for (int e2 = split * (kWarps * 32) + tid; e2 < p.rows * D / 2; e2 += csize * (kWarps * 32)) {
        const int r = 2 * e2 / D, d = 2 * e2 - r * D;
        float ml[kMaxCluster], ll[kMaxCluster];
        float2 ov[kMaxCluster];
#pragma unroll
        for (int s = 0; s < kMaxCluster; ++s) {
            ml[s] = kNegBig;
            ll[s] = 0.f;
            ov[s] = make_float2(0.f, 0.f);
            if (s < csize) {
                const uint32_t peer = map_to_rank(part_addr, s);
                ml[s] = ld_cluster(peer + (GP * D + r) * 4);
                ll[s] = ld_cluster(peer + (GP * D + GP + r) * 4);
                ov[s] = ld_cluster2(peer + (r * D + d) * 4);
            }
        }
        float mc = kNegBig;
#pragma unroll
        for (int s = 0; s < kMaxCluster; ++s) mc = fmaxf(mc, ml[s]);
        float x = 0.f, y = 0.f, l = 0.f;
#pragma unroll
        for (int s = 0; s < kMaxCluster; ++s) {
            const float f = ex2(ml[s] - mc);
            x += ov[s].x * f;
            y += ov[s].y * f;
            l += ll[s] * f;
        }
        const float inv = l > 0.f ? 1.f / l : 0.f;
        uint8_t* orow = const_cast<uint8_t*>(row_base(p.o, p.o_b, p.o_h, p.o_s, r));
        *reinterpret_cast<uint32_t*>(orow + d * 2) = pack_pair<T>(x * inv, y * inv);
    }
    cluster_sync();  // nobody leaves while a peer still reads its shared memory
}

template <typename T, int NT, int D, bool kPaged>
int launch_variant(const Dec16Params& p, int csize, int hkv, int batch, cudaStream_t stream) {
    auto kern = attn_decode16_kernel<T, NT, D, kPaged>;
    constexpr int kSmem = smem_bytes<D, NT>();
    static OncePerDevice configured;
    const int rc = configure_once(kern, configured, kSmem);
    if (rc != B2A_OK) return rc;
    return launch_overlapped_cluster(kern, dim3(csize, hkv, batch), dim3(kWarps * 32), csize, kSmem, stream, p) == cudaSuccess
               ? B2A_OK
               : B2A_ERR_CUDA;
}

template <typename T, int NT>
int launch_d(const Dec16Params& p, int D, bool paged, int csize, int hkv, int batch, cudaStream_t stream) {
    if (paged) return D == 128 ? launch_variant<T, NT, 128, true>(p, csize, hkv, batch, stream)
                               : launch_variant<T, NT, 64, true>(p, csize, hkv, batch, stream);
    return D == 128 ? launch_variant<T, NT, 128, false>(p, csize, hkv, batch, stream)
                    : launch_variant<T, NT, 64, false>(p, csize, hkv, batch, stream);
}

int launch_any(int dtype, const Dec16Params& p, int D, bool paged, int keys, int hkv, int batch, cudaStream_t stream, int parts = 1) {
    // CTAs per (sequence, KV head), as long as every warp keeps two tiles or more.  Dense tensors: equal lengths, so at
    // least three quarters of one wave of two CTAs per SM and no second wave (8 x 3003 keys x 8 KV heads, with the
    // additive mask: two CTAs 32.3 us, four 20.9, eight 25.6).  A pool: lengths differ, and shorter pieces even them out
    // (32 sequences of 256..4096 tokens x 8 KV heads, bf16, cold, with the store kernel: one CTA 61.5 us, two 57.5, four 52.7,
    // eight 71.5 - then the start and the merge of a CTA outweigh its tiles), so about three waves.  The line is the ragged
    // step's: equal lengths would have fewer (8 sequences of 2000 tokens: four CTAs 14.9 us, the rule's eight 20.7), and
    // so would contexts far below the capacity that the rule goes by (8 of 64 tokens, built for 8192: two 6.3, eight 12.0).
    const int sms = device_sm_count();
    if (sms <= 0) return B2A_ERR_CUDA;
    const int tiles = std::max(1, (keys + kTileKeys - 1) / kTileKeys);
    const long long want = paged ? 6LL * sms : 3LL * sms / 2;
    int csize = 1;
    while (csize < kMaxCluster && static_cast<long long>(csize) * hkv * batch * parts < want && tiles >= 4 * csize * kWarps) csize *= 2;
    if (dtype == B2A_F16)
        return p.rows > 8 ? launch_d<__half, 2>(p, D, paged, csize, hkv, batch, stream)
                          : launch_d<__half, 1>(p, D, paged, csize, hkv, batch, stream);
    return p.rows > 8 ? launch_d<__nv_bfloat16, 2>(p, D, paged, csize, hkv, batch, stream)
                      : launch_d<__nv_bfloat16, 1>(p, D, paged, csize, hkv, batch, stream);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

bool sdpa_decode16_supported(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                             const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* o) {
    if (d.dtype != B2A_F16 && d.dtype != B2A_BF16) return false;
    if (d.D != d.Dv || (d.D != 64 && d.D != 128)) return false;
    if (static_cast<long long>(d.Hq / d.Hkv) * d.Sq > 16 || d.Hkv > 65535) return false;
    // K and V rows are copied in 16-byte pieces, Q and O rows in pairs
    if (!aligned16(k) || !aligned16(v) || (reinterpret_cast<uintptr_t>(q) & 3) != 0 || (reinterpret_cast<uintptr_t>(o) & 3) != 0)
        return false;
    const int ext_q[3] = {d.B, d.Hq, d.Sq}, ext_k[3] = {d.B, d.Hkv, d.Skv};
    for (int i = 0; i < 3; ++i) {
        if (ext_q[i] > 1 && (qs[i] % 2 != 0 || os[i] % 2 != 0)) return false;
        if (ext_k[i] > 1 && (ks[i] % 8 != 0 || vs[i] % 8 != 0)) return false;
    }
    return true;
}

int sdpa_decode16_launch(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                         const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* mask, void* o,
                         int32_t* status, cudaStream_t stream, int parts) {
    Dec16Params p{};
    p.q = static_cast<const uint8_t*>(q);
    p.k = static_cast<const uint8_t*>(k);
    p.v = static_cast<const uint8_t*>(v);
    p.o = static_cast<uint8_t*>(o);
    p.mask = static_cast<const uint8_t*>(mask);
    p.mask_kind = mask != nullptr && !d.causal ? d.mask_kind : B2A_MASK_NONE;
    p.Hq = d.Hq;
    p.G = d.Hq / d.Hkv;
    p.Sq = d.Sq;
    p.Skv = d.Skv;
    p.rows = p.G * d.Sq;
    p.causal = d.causal;
    p.scale_log2 = d.scale * kLog2e;
    p.q_b = 2 * qs[0]; p.q_h = 2 * qs[1]; p.q_s = 2 * qs[2];
    p.k_b = 2 * ks[0]; p.k_h = 2 * ks[1]; p.k_s = 2 * ks[2];
    p.v_b = 2 * vs[0]; p.v_h = 2 * vs[1]; p.v_s = 2 * vs[2];
    p.o_b = 2 * os[0]; p.o_h = 2 * os[1]; p.o_s = 2 * os[2];
    p.m_b = d.mask_strides[0]; p.m_h = d.mask_strides[1]; p.m_s = d.mask_strides[2]; p.m_k = d.mask_strides[3];
    p.status = status;
    return launch_any(d.dtype, p, d.D, false, d.causal ? std::min(d.Sq, d.Skv) : d.Skv, d.Hkv, d.B, stream, parts);
}

bool paged_decode16_supported(const b2a_paged_desc& d) {
    return (d.kv_dtype == B2A_F16 || d.kv_dtype == B2A_BF16) && d.q_dtype == d.kv_dtype && d.D == d.Dv &&
           (d.D == 64 || d.D == 128) && d.block_size % kTileKeys == 0 && d.Hq / d.Hkv <= 16 && d.Hkv <= 65535;
}

int paged_decode16_launch(const b2a_paged_desc& d, const void* query, const void* k_cache, const void* v_cache,
                          const PagedTables& t, void* out, int32_t* status, cudaStream_t stream) {
    Dec16Params p{};
    p.q = static_cast<const uint8_t*>(query);
    p.k = static_cast<const uint8_t*>(k_cache);
    p.v = static_cast<const uint8_t*>(v_cache);
    p.o = static_cast<uint8_t*>(out);
    p.mask_kind = B2A_MASK_NONE;
    p.Hq = d.Hq;
    p.G = d.Hq / d.Hkv;
    p.Sq = 1;
    p.rows = p.G;
    p.scale_log2 = d.scale * kLog2e;
    p.q_b = p.o_b = static_cast<int64_t>(d.Hq) * d.D * 2;  // a token's row
    p.q_h = p.o_h = d.D * 2;
    p.k_h = p.v_h = static_cast<int64_t>(d.block_size) * d.D * 2;
    p.k_b = p.v_b = d.Hkv * p.k_h;
    p.t = t;
    p.sliding_window = d.sliding_window;
    p.status = status;
    const int keys = d.sliding_window > 0 ? std::min(d.sliding_window, d.max_context_len) : d.max_context_len;
    return launch_any(d.kv_dtype, p, d.D, true, keys, d.Hkv, d.num_seqs, stream);
}

}  // namespace b2a
