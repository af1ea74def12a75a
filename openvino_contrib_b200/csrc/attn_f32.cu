// ScaledDotProductAttention on float32 tensors: D = Dv up to 128, a multiple of four; causal, any mask, any outer
// strides.  All arithmetic in float32 on the FMA pipe (a tensor-core split of the operands would not keep the precision).
//
// Bound: FMA issue.  A warp owns eight query rows; a thread computes 4 rows x (its share of the keys) of S and 4 rows x 4
// (or 8) columns of O, so that four shared-memory vectors of Q (two distinct ones per warp) and the keys' vectors feed 16
// FMAs per key vector; the scores add up as two lanes (even and odd d) of packed fma.f32x2.  K and V tiles are staged by
// cp.async, two buffers.  Rows of Q and K are padded by four floats: eight lanes' 128-bit reads then fall into different
// banks for every D that is a multiple of eight.
//
// A CTA has eight warps, as kSplit key ranges x 8 / kSplit row groups.  kSplit 1 is the efficient form; where its 64-row
// tiles would leave SMs without work (small batches, the single operator of a functional test), the CTA takes 32 or 16
// rows and its warps share out the keys of a tile, each with its own running maximum, merged once at the end.  The
// launcher takes the smallest kSplit that gives a CTA to every SM, else 4.
//
// Measured on a B200: 8 heads x 256 tokens, D = 64, causal (kSplit 4): 82.6 us in attn_generic_kernel, 12.5 us here;
// 16 heads x 912 tokens, D = 64 (kSplit 1): 164 us, 21 TFLOP/s, where the shared-memory reads of 4 x 4 register tiles cost
// about as much as the FMAs they feed.
#include "launch.cuh"

namespace b2a {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kRowsPerWarp = 8;

struct F32Params {
    int B, Hq, G, Sq, Skv, D, causal;
    float scale;
    const float* q;
    const float* k;
    const float* v;
    float* o;
    int64_t qs[3], ks[3], vs[3], os[3];
    const void* mask;
    int mask_kind;
    int64_t ms[4];
};

__device__ __forceinline__ void cp_async16z(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float f2_sum(uint64_t a) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a));
    return lo + hi;
}
__host__ __device__ constexpr int row_groups(int split) { return kWarps / split; }
// keys of a staged tile: two buffers of K and V, Q and P in at most 227 KB (NC: 64-column chunks of the head size)
__host__ __device__ constexpr int tile_keys(int nc, int split) { return nc == 1 && split > 1 ? 128 : 64; }
template <int NC, int kSplit>
size_t smem_floats(int D) {
    constexpr int BM = kRowsPerWarp * row_groups(kSplit), BN = tile_keys(NC, kSplit);
    return static_cast<size_t>(BM) * (D + 4) + 2 * (static_cast<size_t>(BN) * (D + 4) + static_cast<size_t>(BN) * D) +
           static_cast<size_t>(kWarps) * kRowsPerWarp * (BN / kSplit + 4);
}

template <int NC, int kSplit>
__global__ void __launch_bounds__(kThreads) attn_f32_kernel(const F32Params p) {
    constexpr int BM = kRowsPerWarp * row_groups(kSplit), BN = tile_keys(NC, kSplit);
    constexpr int kKeysW = BN / kSplit;   // keys of a tile that one warp takes
    constexpr int NK = kKeysW / 16;       // ... and one thread
    extern __shared__ __align__(16) float smem[];
    const int D = p.D, LD = D + 4, D4 = D / 4;
    float* sQ = smem;                          // [BM][D + 4]
    float* sK = sQ + BM * LD;                  // 2 x [BN][D + 4]
    float* sV = sK + 2 * BN * LD;              // 2 x [BN][D]
    float* sP = sV + 2 * BN * D;               // [warp][8][kKeysW + 4]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rg = lane >> 4, kg = lane & 15;  // rows 4 rg .. +3 of the warp's eight; keys kg + 16 n, columns 4 kg + 64 c
    const int part = warp % kSplit, wrow = (warp / kSplit) * kRowsPerWarp;

    const int h = blockIdx.y, b = blockIdx.z, hk = h / p.G;
    const int row0 = (p.causal ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x)) * BM;  // longest first
    const int nrows = min(BM, p.Sq - row0);
    const int k_end = p.causal ? min(p.Skv, row0 + nrows) : p.Skv;
    const float* qb = p.q + b * p.qs[0] + h * p.qs[1];
    const float* kb = p.k + b * p.ks[0] + hk * p.ks[1];
    const float* vb = p.v + b * p.vs[0] + hk * p.vs[1];

    // A thread's 16-byte pieces of a tile are kThreads apart: their row and column follow from the ones before (with a
    // division by the run-time row length for each piece, 16 heads x 912 tokens took 170 us instead of 164).
    const int r_first = tid / D4, c_first = tid - r_first * D4, r_step = kThreads / D4, c_step = kThreads - r_step * D4;
    auto pieces = [&](int rows, auto&& piece) {
        int r = r_first, c = c_first;
        while (r < rows) {
            piece(r, 4 * c);
            r += r_step;
            c += c_step;
            if (c >= D4) {
                c -= D4;
                ++r;
            }
        }
    };
    auto stage = [&](int j0, int buf) {  // keys past the end become zeros
        float* dk = sK + buf * BN * LD;
        float* dv = sV + buf * BN * D;
        pieces(BN, [&](int r, int c) {
            const bool in = j0 + r < k_end;
            const int64_t row = in ? j0 + r : 0;
            cp_async16z(dk + r * LD + c, kb + row * p.ks[2] + c, in ? 16 : 0);
            cp_async16z(dv + r * D + c, vb + row * p.vs[2] + c, in ? 16 : 0);
        });
    };
    pieces(BM, [&](int r, int c) {
        const bool in = r < nrows;
        cp_async16z(sQ + r * LD + c, qb + (in ? row0 + r : 0) * p.qs[2] + c, in ? 16 : 0);
    });
    stage(0, 0);
    cp_async_commit();

    float m[4], l[4], acc[4][4 * NC];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * NC; ++c) acc[i][c] = 0.f;
    }
    const float* qrow = sQ + (wrow + 4 * rg) * LD;
    float* pw = sP + warp * kRowsPerWarp * (kKeysW + 4);
    const int wlast = row0 + wrow + kRowsPerWarp - 1;  // last row of the warp (causal horizon)

    const int tiles = (k_end + BN - 1) / BN;
    for (int t = 0; t < tiles; ++t) {
        const int buf = t & 1, key0 = t * BN + part * kKeysW;
        if (t + 1 < tiles) stage((t + 1) * BN, buf ^ 1);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        // (warp-uniform) nothing to do for a warp whose keys all lie past the end or past its rows' horizon
        if (key0 < k_end && (!p.causal || key0 <= wlast)) {
            const float* kt = sK + buf * BN * LD + (part * kKeysW + kg) * LD;
            uint64_t s2[4][NK];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int n = 0; n < NK; ++n) s2[i][n] = 0ull;
#pragma unroll 4
            for (int d = 0; d < D; d += 4) {
                ulonglong2 qv[4], kv[NK];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(qrow + i * LD + d);
#pragma unroll
                for (int n = 0; n < NK; ++n) kv[n] = *reinterpret_cast<const ulonglong2*>(kt + 16 * n * LD + d);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int n = 0; n < NK; ++n) {
                        s2[i][n] = f2_fma(qv[i].x, kv[n].x, s2[i][n]);
                        s2[i][n] = f2_fma(qv[i].y, kv[n].y, s2[i][n]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = row0 + wrow + 4 * rg + i;
                float s[NK], mx = -INFINITY;
#pragma unroll
                for (int n = 0; n < NK; ++n) {
                    const int key = key0 + kg + 16 * n;
                    s[n] = f2_sum(s2[i][n]) * p.scale;
                    bool keep = key < k_end && row < p.Sq && (!p.causal || key <= row);
                    if (p.mask_kind != B2A_MASK_NONE && keep) {
                        const int64_t at = b * p.ms[0] + h * p.ms[1] + row * p.ms[2] + key * p.ms[3];
                        if (p.mask_kind == B2A_MASK_BOOL) keep = static_cast<const uint8_t*>(p.mask)[at] != 0;
                        else s[n] += static_cast<const float*>(p.mask)[at];
                    }
                    if (!keep) s[n] = -INFINITY;
                    mx = fmaxf(mx, s[n]);
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m[i], mx);
                const bool none = m_new == -INFINITY;  // nothing kept so far
                const float alpha = none ? 1.f : expf(m[i] - m_new);
                float sum = 0.f;
#pragma unroll
                for (int n = 0; n < NK; ++n) {
                    const float e = none ? 0.f : expf(s[n] - m_new);
                    sum += e;
                    pw[(4 * rg + i) * (kKeysW + 4) + kg + 16 * n] = e;
                }
                l[i] = l[i] * alpha + sum;  // this thread's keys; the 16 lanes are added up at the end
                m[i] = m_new;
#pragma unroll
                for (int c = 0; c < 4 * NC; ++c) acc[i][c] *= alpha;
            }
            __syncwarp();
            const float* vt = sV + buf * BN * D + part * kKeysW * D;
            const float* pr = pw + 4 * rg * (kKeysW + 4);
#pragma unroll 4
            for (int j = 0; j < kKeysW; j += 4) {
                float pv[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 x = *reinterpret_cast<const float4*>(pr + i * (kKeysW + 4) + j);
                    pv[i][0] = x.x;
                    pv[i][1] = x.y;
                    pv[i][2] = x.z;
                    pv[i][3] = x.w;
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const int col = 4 * kg + 64 * c;
                        if (col < D) {
                            const float4 x = *reinterpret_cast<const float4*>(vt + (j + u) * D + col);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                acc[i][4 * c] = fmaf(pv[i][u], x.x, acc[i][4 * c]);
                                acc[i][4 * c + 1] = fmaf(pv[i][u], x.y, acc[i][4 * c + 1]);
                                acc[i][4 * c + 2] = fmaf(pv[i][u], x.z, acc[i][4 * c + 2]);
                                acc[i][4 * c + 3] = fmaf(pv[i][u], x.w, acc[i][4 * c + 3]);
                            }
                        }
                    }
            }
        }
        __syncthreads();  // the buffer is refilled in the next step
    }
    cp_async_wait<0>();

#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], o);

    if constexpr (kSplit == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = wrow + 4 * rg + i;
            if (r >= nrows) continue;
            const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
            float* orow = p.o + b * p.os[0] + h * p.os[1] + (row0 + r) * p.os[2];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int col = 4 * kg + 64 * c;
                if (col < D)
                    *reinterpret_cast<float4*>(orow + col) =
                        make_float4(acc[i][4 * c] * inv, acc[i][4 * c + 1] * inv, acc[i][4 * c + 2] * inv, acc[i][4 * c + 3] * inv);
            }
        }
    } else {
        // the key ranges of a row: [BM][kSplit] maxima and sums, [BM][kSplit][D] weighted sums, over the K and V buffers
        float* sm = sK;
        float* sl = sm + BM * kSplit;
        float* sa = sl + BM * kSplit;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int at = (wrow + 4 * rg + i) * kSplit + part;
            if (kg == 0) {
                sm[at] = m[i];
                sl[at] = l[i];
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const int col = 4 * kg + 64 * c;
                if (col < D)
                    *reinterpret_cast<float4*>(sa + at * D + col) =
                        make_float4(acc[i][4 * c], acc[i][4 * c + 1], acc[i][4 * c + 2], acc[i][4 * c + 3]);
            }
        }
        __syncthreads();
        pieces(nrows, [&](int r, int c) {
            float mx = -INFINITY, sum = 0.f;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int w = 0; w < kSplit; ++w) mx = fmaxf(mx, sm[r * kSplit + w]);
#pragma unroll
            for (int w = 0; w < kSplit; ++w) {
                const float mw = sm[r * kSplit + w];
                const float f = mw == -INFINITY ? 0.f : expf(mw - mx);
                const float4 x = *reinterpret_cast<const float4*>(sa + (r * kSplit + w) * D + c);
                sum = fmaf(sl[r * kSplit + w], f, sum);
                o.x = fmaf(x.x, f, o.x);
                o.y = fmaf(x.y, f, o.y);
                o.z = fmaf(x.z, f, o.z);
                o.w = fmaf(x.w, f, o.w);
            }
            const float inv = sum > 0.f ? 1.f / sum : 0.f;
            *reinterpret_cast<float4*>(p.o + b * p.os[0] + h * p.os[1] + (row0 + r) * p.os[2] + c) =
                make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
        });
    }
}

template <int NC, int kSplit>
int launch(const F32Params& p, cudaStream_t stream) {
    constexpr int BM = kRowsPerWarp * row_groups(kSplit);
    const size_t smem = smem_floats<NC, kSplit>(p.D) * sizeof(float);
    auto kern = attn_f32_kernel<NC, kSplit>;
    static OncePerDevice configured;
    const int rc = configure_once(kern, configured, static_cast<int>(smem_floats<NC, kSplit>(64 * NC) * sizeof(float)));
    if (rc != B2A_OK) return rc;
    kern<<<dim3((p.Sq + BM - 1) / BM, p.Hq, p.B), kThreads, smem, stream>>>(p);
    return cudaGetLastError() == cudaSuccess ? B2A_OK : B2A_ERR_CUDA;
}

}  // namespace

bool sdpa_f32_supported(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                        const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* o) {
    if (d.dtype != B2A_F32 || d.D != d.Dv || d.D > 128 || d.D % 4 != 0) return false;
    auto al = [](const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
    if (!al(q) || !al(k) || !al(v) || !al(o)) return false;
    for (int i = 0; i < 3; ++i)  // 16-byte rows
        if (qs[i] % 4 != 0 || ks[i] % 4 != 0 || vs[i] % 4 != 0 || os[i] % 4 != 0) return false;
    return true;
}

int sdpa_f32_launch(const b2a_sdpa_desc& d, const int64_t (&qs)[4], const int64_t (&ks)[4], const int64_t (&vs)[4],
                    const int64_t (&os)[4], const void* q, const void* k, const void* v, const void* mask, void* o,
                    cudaStream_t stream, int parts) {
    F32Params p{};
    p.B = d.B; p.Hq = d.Hq; p.G = d.Hq / d.Hkv; p.Sq = d.Sq; p.Skv = d.Skv; p.D = d.D;
    p.causal = d.causal;
    p.scale = d.scale;
    p.q = static_cast<const float*>(q);
    p.k = static_cast<const float*>(k);
    p.v = static_cast<const float*>(v);
    p.o = static_cast<float*>(o);
    for (int i = 0; i < 3; ++i) {
        p.qs[i] = qs[i]; p.ks[i] = ks[i]; p.vs[i] = vs[i]; p.os[i] = os[i];
    }
    p.mask_kind = d.causal || mask == nullptr ? B2A_MASK_NONE : d.mask_kind;
    p.mask = mask;
    for (int i = 0; i < 4; ++i) p.ms[i] = d.mask_strides[i];
    const int sms = device_sm_count();
    if (sms <= 0) return B2A_ERR_CUDA;
    const long long heads = static_cast<long long>(d.B) * d.Hq * parts;
    const int split = heads * ((d.Sq + 63) / 64) >= sms ? 1 : heads * ((d.Sq + 31) / 32) >= sms ? 2 : 4;
    if (d.D <= 64) return split == 1 ? launch<1, 1>(p, stream) : split == 2 ? launch<1, 2>(p, stream) : launch<1, 4>(p, stream);
    return split == 1 ? launch<2, 1>(p, stream) : split == 2 ? launch<2, 2>(p, stream) : launch<2, 4>(p, stream);
}

}  // namespace b2a
