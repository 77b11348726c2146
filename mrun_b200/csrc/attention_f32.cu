// Paged grouped-query attention in 32-bit arithmetic for heads of 64 and 128 features: the attention of the
// 32-bit path, prompts and single tokens alike.
//
// A block takes one kv head and a tile of tokens of one request; the query heads of the group are rows
// side by side, RT rows a block, so the keys and values that it brings to shared memory serve all of
// them (32 heads over 8 of 128, prompts of 207 and 310 tokens: 102 us; a block a token and head, which reads
// the keys again for every row: 1,184).  Bound by the shared-memory reads that feed the FMA pipe, for
// single tokens by the latency of one tile after the other (4.5 us a tile, so 590 us at a context of 8,000, whether
// one request decodes or sixteen: a token and kv head's keys are not dealt to several blocks).
//
// Keys come in tiles of KT counted from position 0.  A thread owns RPT rows x 4 keys of the scores (keys tx,
// tx + 16, ...) and the same rows x D / 16 columns of the output.  A score is one chain of fused
// multiply-adds over the features, a row's sum of a tile is added in an order fixed by the keys'
// places, an output element is one chain over the keys; a tile in which a row sees nothing changes none
// of the row's numbers.  So a token's result depends on its own keys only: it is bit-identical however
// the request was cut into steps, and whichever RT runs.  A key that a row does not see does not
// enter its sums at all, whatever lies there.
//
// Math: s = scale * q·k, p = softmax(s), o = p·v; query head h reads kv head h / (heads/kv_heads)
// (crates/mrun-engine/src/models/common.rs:129,199-205; causal alignment to the end of the keys,
// crates/mrun-engine/src/tensor/nuvec.rs:866-872).
#include <type_traits>

#include "common.cuh"

using namespace mrun;

namespace {

constexpr int KT = 64;               // keys of a tile
constexpr int THREADS = 256;         // RT / RPT * 16 of them compute, all of them copy

__device__ __forceinline__ void copy_16_or_zero(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int D, int RT> constexpr int f32_smem_floats() { return (RT + KT) * (D + 4) + KT * D + RT * (KT + 4); }

// first / count: the tiles' first token rows and token counts, or null for a tile a token.
template <int D, int RT, int RPT>
__global__ void __launch_bounds__(THREADS)
attention_f32_kernel(const float* __restrict__ q, long q_stride, float* __restrict__ out, const float* __restrict__ k_cache,
                     const float* __restrict__ v_cache, const int* __restrict__ block_tables, int max_blocks,
                     const int* __restrict__ token_slot, const int* __restrict__ positions, const int* __restrict__ first,
                     const int* __restrict__ count, int heads, int kv_heads, int page_size, float scale, int window) {
    constexpr int PITCH = D + 4, PP = KT + 4, CC = D / 64;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                     // [RT][PITCH]
    float* ks = qs + RT * PITCH;          // [KT][PITCH]
    float* vs = ks + KT * PITCH;          // [KT][D]
    float* ps = vs + KT * D;              // [RT][PP]
    __shared__ int key_rows[2][KT];       // where a tile's keys lie in the cache, in rows (negative: none)

    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int kvh = blockIdx.y, group = heads / kv_heads;
    const int t0 = first ? first[blockIdx.x] : blockIdx.x;
    const int tokens = count ? count[blockIdx.x] : 1;
    const int rows = tokens * group;
    const int pos0 = positions[t0];
    if (pos0 < 0) {                       // padding
        for (int e = tid; e < rows * D; e += THREADS)
            out[((size_t)(t0 + e / D / group) * heads + (size_t)kvh * group + e / D % group) * D + e % D] = 0.f;
        return;
    }
    const int last = pos0 + tokens - 1;   // positions of a tile's tokens follow one another
    const int* table = block_tables + (size_t)token_slot[t0] * max_blocks;
    const int begin = first_visible(pos0, window) / KT * KT;
    const bool computes = ty < RT / RPT;

    auto look_up = [&](int tile, int which) {
        const int j = tid - (THREADS - KT);               // the last warps, which have no rows of a single token
        if (j >= 0) {
            const int key = tile + j;
            key_rows[which][j] = -1;
            if (key <= last && key >= first_visible(pos0, window))
                key_rows[which][j] = (table[key / page_size] * kv_heads + kvh) * page_size + key % page_size;
        }
    };
    auto bring = [&](const float* cache, float* dst, int pitch, int which) {
        for (int e = tid; e < KT * (D / 4); e += THREADS) {
            const int j = e / (D / 4), c = e % (D / 4) * 4, row = key_rows[which][j];
            copy_16_or_zero(dst + j * pitch + c, cache + (size_t)max(row, 0) * D + c, row >= 0 ? 16 : 0);
        }
    };
    for (int e = tid; e < RT * (D / 4); e += THREADS) {
        const int r = e / (D / 4), c = e % (D / 4) * 4;
        const bool in = r < rows;
        const float* src = q + (size_t)(t0 + (in ? r / group : 0)) * q_stride + ((size_t)kvh * group + (in ? r % group : 0)) * D + c;
        copy_16_or_zero(qs + r * PITCH + c, src, in ? 16 : 0);
    }
    look_up(begin, 0);
    __syncthreads();
    bring(k_cache, ks, PITCH, 0);
    copies_commit();
    bring(v_cache, vs, D, 0);
    copies_commit();

    int pos[RPT], lo[RPT];
    float m[RPT], l[RPT], acc[RPT][4 * CC];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = ty * RPT + i;
        pos[i] = r < rows ? pos0 + r / group : -1;
        lo[i] = first_visible(pos[i], window);
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 4 * CC; ++c) acc[i][c] = 0.f;
    }
    int which = 0;
    for (int tile = begin; tile <= last; tile += KT, which ^= 1) {
        copies_wait<1>();                 // the keys are here
        __syncthreads();
        if (tile + KT <= last) look_up(tile + KT, which ^ 1);
        float s[RPT][4];
#pragma unroll
        for (int i = 0; i < RPT; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
        const int here = min(KT, last + 1 - tile);        // keys of the tile that there are
        auto score = [&](auto columns) {
#pragma unroll 4
            for (int d = 0; d < D; d += 4) {
                float4 a[RPT], b[columns];
#pragma unroll
                for (int i = 0; i < RPT; ++i) a[i] = *reinterpret_cast<const float4*>(qs + (ty * RPT + i) * PITCH + d);
#pragma unroll
                for (int j = 0; j < columns; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * PITCH + d);
#pragma unroll
                for (int i = 0; i < RPT; ++i)
#pragma unroll
                    for (int j = 0; j < columns; ++j) {
                        s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
                        s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
                        s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
                        s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
                    }
            }
        };
        // the first tokens of a request see a quarter of a tile
        if (computes && here > 16) score(std::integral_constant<int, 4>());
        else if (computes) score(std::integral_constant<int, 1>());
        __syncthreads();                  // the keys have been read, the next ones looked up
        if (tile + KT <= last) bring(k_cache, ks, PITCH, which ^ 1);
        copies_commit();
        // whether every row of the block sees every key of the tile
        const bool whole = tile >= first_visible(last, window) && tile + KT - 1 <= pos0 && rows == RT;
        if (computes)
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = tile + tx + 16 * j;
                s[i][j] = key <= pos[i] && key >= lo[i] ? s[i][j] * scale : -INFINITY;
                top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const float next = fmaxf(m[i], top);
            const float base = next == -INFINITY ? 0.f : next;
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                s[i][j] = expf(s[i][j] - base);
                sum += s[i][j];
                ps[(ty * RPT + i) * PP + tx + 16 * j] = s[i][j];
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float shrink = m[i] == -INFINITY ? 0.f : expf(m[i] - base);
            l[i] = l[i] * shrink + sum;
            m[i] = next;
#pragma unroll
            for (int c = 0; c < 4 * CC; ++c) acc[i][c] *= shrink;
        }
        copies_wait<1>();                 // the values are here
        __syncthreads();
        if (computes)
#pragma unroll 2
        for (int j = 0; j < here; j += 4) {
            float p[RPT][4];
#pragma unroll
            for (int i = 0; i < RPT; ++i)
                *reinterpret_cast<float4*>(p[i]) = *reinterpret_cast<const float4*>(ps + (ty * RPT + i) * PP + j);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float v[4 * CC];
#pragma unroll
                for (int c = 0; c < CC; ++c)
                    *reinterpret_cast<float4*>(v + 4 * c) = *reinterpret_cast<const float4*>(vs + (j + k) * D + c * 64 + tx * 4);
                if (whole) {
#pragma unroll
                    for (int i = 0; i < RPT; ++i)
#pragma unroll
                        for (int c = 0; c < 4 * CC; ++c) acc[i][c] = fmaf(p[i][k], v[c], acc[i][c]);
                } else {
#pragma unroll
                    for (int i = 0; i < RPT; ++i)
                        if (tile + j + k <= pos[i] && tile + j + k >= lo[i])
#pragma unroll
                            for (int c = 0; c < 4 * CC; ++c) acc[i][c] = fmaf(p[i][k], v[c], acc[i][c]);
                }
            }
        }
        __syncthreads();                  // the values and the weights have been read
        if (tile + KT <= last) bring(v_cache, vs, D, which ^ 1);
        copies_commit();
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = ty * RPT + i;
        if (!computes || r >= rows) continue;
        const float inv = 1.f / l[i];
        float* dst = out + ((size_t)(t0 + r / group) * heads + (size_t)kvh * group + r % group) * D + tx * 4;
#pragma unroll
        for (int c = 0; c < CC; ++c)
            *reinterpret_cast<float4*>(dst + c * 64) =
                make_float4(acc[i][4 * c] * inv, acc[i][4 * c + 1] * inv, acc[i][4 * c + 2] * inv, acc[i][4 * c + 3] * inv);
    }
}

template <int D, int RT, int RPT>
int launch_f32(dim3 grid, const float* q, long q_stride, float* out, const float* k_cache, const float* v_cache, const int* block_tables,
               int max_blocks, const int* token_slot, const int* positions, const int* first, const int* count, int heads, int kv_heads,
               int page_size, float scale, int window, cudaStream_t stream) {
    constexpr int bytes = f32_smem_floats<D, RT>() * (int)sizeof(float);
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(attention_f32_kernel<D, RT, RPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
                    "paged_attention_f32");
    attention_f32_kernel<D, RT, RPT><<<grid, THREADS, bytes, stream>>>(q, q_stride, out, k_cache, v_cache, block_tables, max_blocks,
                                                                           token_slot, positions, first, count, heads, kv_heads,
                                                                           page_size, scale, window);
    return 0;
}

}  // namespace

// q: row t starts at q + t * q_stride (16-byte rows), heads contiguous [heads, head_dim]; out: dense [tokens,
// heads * head_dim]; key and value pages [pages, kv_heads, page_size, head_dim].  block_tables: [slots,
// max_blocks]; token_slot[t] picks the row; positions[t] < 0 = padding.  first / count (int32 [tiles]): a tile's
// first token row and its tokens, which are consecutive tokens of one request, at most `tile_tokens` of
// them (64 rows of query heads a tile); null: `tiles` single tokens.
MRUN_API int mrun_paged_attention_f32(const float* q, long q_stride, float* out, const float* k_cache, const float* v_cache,
                                      const int* block_tables, int max_blocks, const int* token_slot, const int* positions,
                                      const int* first, const int* count, int tiles, int tile_tokens, int heads, int kv_heads,
                                      int head_dim, int page_size, long cache_rows, float scale, int window, cudaStream_t stream) {
    MRUN_REQUIRE(tiles >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && page_size > 0 && max_blocks > 0,
                 "paged_attention_f32: bad sizes");
    MRUN_REQUIRE(head_dim == 64 || head_dim == 128, "paged_attention_f32: heads of %d features, the kernel takes 64 and 128", head_dim);
    MRUN_REQUIRE((first == nullptr) == (count == nullptr), "paged_attention_f32: first and count come together");
    const int rows = tile_tokens * (heads / kv_heads);
    MRUN_REQUIRE(tile_tokens > 0 && (first != nullptr || tile_tokens == 1) && rows <= 64,
                 "paged_attention_f32: tiles of %d tokens x %d heads, the kernel takes 64 rows", tile_tokens, heads / kv_heads);
    MRUN_REQUIRE(kv_heads <= 65535, "paged_attention_f32: kv_heads=%d exceeds 65535", kv_heads);
    MRUN_REQUIRE(cache_rows < (1L << 31), "paged_attention_f32: the cache has %ld rows, the limit is 2^31", cache_rows);
    MRUN_REQUIRE(q_stride % 4 == 0 && ((((uintptr_t)q) | ((uintptr_t)out) | ((uintptr_t)k_cache) | ((uintptr_t)v_cache)) & 15) == 0,
                 "paged_attention_f32: rows that do not start on 16 bytes");
    if (tiles == 0) return 0;
    const dim3 grid(tiles, kv_heads);
#define MRUN_F32(D, RT, RPT)                                                                                                      \
    failed = launch_f32<D, RT, RPT>(grid, q, q_stride, out, k_cache, v_cache, block_tables, max_blocks, token_slot, positions, first,  \
                                    count, heads, kv_heads, page_size, scale, window, stream)
    int failed = 0;
    // the rows of one token: fewer threads a block, more blocks a multiprocessor
    if (head_dim == 64) {
        if (rows > 16) MRUN_F32(64, 64, 4);
        else if (rows > 4) MRUN_F32(64, 16, 1);
        else MRUN_F32(64, 4, 1);
    } else {
        if (rows > 16) MRUN_F32(128, 64, 4);
        else if (rows > 4) MRUN_F32(128, 16, 1);
        else MRUN_F32(128, 4, 1);
    }
#undef MRUN_F32
    if (failed) return failed;
    MRUN_CHECK_LAUNCH("paged_attention_f32");
    return 0;
}
