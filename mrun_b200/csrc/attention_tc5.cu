// Paged grouped-query attention for prompt portions on the fifth-generation tensor cores
// (tcgen05, accumulators in tensor memory), compiled for one head size that is a multiple of 64
// and at most 128: -DMRUN_HEAD_DIM=<64 | 128> (values of another of these sizes: -DMRUN_VALUE_DIM;
// worked-on scores and gated outputs, attention_score.cuh: -DMRUN_SCORED=1).  Keys may have 192 features
// where the values have 64 or 128 and the scores are plain: Q and two stages of K and V then take 209 KB.
//
// One thread block per (tile of query tokens, kv head).  A row is a (token, query head of the kv head's group) pair, so a
// key/value tile read once serves the whole group.  Rows come in streams of 128; keys are consumed 128 at a time in position order
// with an online softmax.  A long tile is a pair of streams that take turns: while the tensor cores work for one, the softmax of the other runs, and both
// take every key tile.  A short tile (and all with keys of 192 features, where a second Q has no place) is a single stream, half a
// row a thread.  Both ways do the same arithmetic in the same order on a row, so its bits do not depend on how the step is cut:
//
//   warps 0..7   softmax.  Of a pair four warps a stream, a thread a row (tensor-memory lane r is row r).  A thread reads its row of
//                S = Q·Kᵀ (tcgen05.ld), masks it, keeps the running maximum and the sums of either half of the keys in 32-bit, and writes P =
//                exp2(s - max) as packed bf16 (tcgen05.st), the first half of the keys as soon as it is there.
//                Of a single stream warp w and warp w + 4 share the lanes 32 (w % 4) .., the first takes keys 0..63 of a tile, the
//                second keys 64..127; they meet for the row's maximum through shared memory and a barrier of the two warps, and for the sum at the end.
//                A row of O is rescaled when the
//                maximum has grown by more than 2^8 since the last rescale (until then P is
//                taken against the older maximum, which is exact: the final division uses the
//                same maximum);
//   warp 8       issues the products.  Of a pair: O += P[j]·V[j] in halves as P is written, then the stream's next S = Q·Kᵀ.  Of a
//                single stream: O += P[j]·V[j] as P is there, S up to two tiles ahead of the softmax.  P is
//                read from tensor memory, Q, K and V from shared memory, V as the MN-major
//                operand (its rows are keys, as the cache stores them);
//   warp 9       brings K tiles from the pages into a ring of two stages by TMA: a lane per page
//                of the tile looks the page up in the block table, a tile ahead, and copies its rows as
//                [rows x 64] boxes with the 128-byte swizzle; warp 10 the V tiles likewise.
//
// Bound by the chain of a stream's row (scores out of tensor memory, maximum, exponentials, P back, two products), of which two
// run side by side in a pair: a tile of 128 keys for 256 rows of 128 features takes 2.25 us (2,048 cycles of MMAs and as many of the
// special-function units would be 1.1), for a single stream's 128 rows 1.32.  1,531 tokens behind 9,000, 32 heads over 8, B200:
// 270 us, 0.91 PFLOP/s; single streams alone 299.
// What the parts of a pair gave, us a tile, back to back (the figures above are after a pause: 2.05 for 1.9), before the next scores waited
// for the product that reads P: a warp of products for both streams in place of one each 2.9 -> 2.1 (two fall into
// step); one elected lane and every wait but P's taken before 2.1 -> 1.9; P in halves 2.3 -> 2.25.  A quarter of the exponentials as polynomials on the multiply-add pipe 1.92 -> 1.96, a third stage of K or V nothing.
//
// The roles hand tiles to one another through mbarriers; every wait is bounded by a cycle budget.
// When a wait runs out the block records a code in the status word, every role stops, the block
// frees its tensor memory and returns; the host reads the status word after the step and raises.
//
// A token at position p sees keys lo..p, lo = 0, p - window + 1, or the start of p's chunk for a
// window of minus the chunk's size (first_visible()).  Pages that lie wholly
// outside the tile's range, or that were given back, are never dereferenced; their rows of a
// stage keep what an earlier tile left there (the V stages start as zeros), and every key outside
// a row's range is masked.  The page size must be a power of two (pages of 1 .. 128 keys divide
// a tile, larger pages hold whole tiles).
// Math as in the other attention kernels: s = scale * q·k, softmax in 32-bit, o = p·v
// (crates/mrun-engine/src/models/common.rs:129,199-205); P is rounded to bf16 for the second
// product, as the tensor cores take bf16 operands.
#include <cstdio>

#include "attention_paging.cuh"
#include "attention_score.cuh"
#include "common.cuh"
#include "tcgen05.cuh"

#ifndef MRUN_HEAD_DIM
#error "compile with -DMRUN_HEAD_DIM=<head size>"
#endif

#ifndef MRUN_VALUE_DIM
#define MRUN_VALUE_DIM MRUN_HEAD_DIM
#endif
#ifndef MRUN_SCORED
#define MRUN_SCORED 0
#endif

#if MRUN_HEAD_DIM % 64 == 0 && MRUN_HEAD_DIM <= (MRUN_SCORED ? 128 : 192) && MRUN_VALUE_DIM % 64 == 0 && MRUN_VALUE_DIM <= 128
#define MRUN_ATTN_TC5 1
#else
#define MRUN_ATTN_TC5 0
#endif

#if MRUN_ATTN_TC5

namespace {

using bf16 = __nv_bfloat16;
using namespace tc5;

constexpr int D = MRUN_HEAD_DIM, DV = MRUN_VALUE_DIM;
constexpr bool SCORED = MRUN_SCORED;
constexpr int ROWS = 128;                    // query rows per stream = MMA M
constexpr int KEYS = 128, HALF = 64;         // keys per tile = N of the first product, K of the second
constexpr int SPANS_D = D / 64, SPANS_V = DV / 64;      // 64-wide spans of the head dimensions
constexpr int SPAN_BYTES = 128 * 128;        // one swizzled tile of 128 rows x 64 bf16
constexpr int K_BYTES = SPANS_D * SPAN_BYTES;           // one stage of K: 128 keys x D
constexpr int V_BYTES = SPANS_V * SPAN_BYTES;           // one stage of V: 128 keys x DV
constexpr int Q_BYTES = SPANS_D * SPAN_BYTES;           // the rows of one stream
constexpr int MAX_Q = D <= 128 ? 2 : 1;      // streams with rows of their own that fit beside the stages
constexpr int SMEM_BYTES = MAX_Q * Q_BYTES + 2 * K_BYTES + 2 * V_BYTES + 1024;        // Q, two stages of K and of V
constexpr int SOFTMAX_WARPS = 8, SOFTMAX_THREADS = SOFTMAX_WARPS * 32, STREAM_WARPS = 4;
constexpr int MMA_WARP = 8, K_WARP = 9, V_WARP = 10;
constexpr int THREADS = SOFTMAX_THREADS + 4 * 32;                        // 384: registers are dealt to four warps together
constexpr int SOFTMAX_REGISTERS = 216, OTHER_REGISTERS = 72, LAUNCH_REGISTERS = 168;
static_assert(SOFTMAX_THREADS * SOFTMAX_REGISTERS + 128 * OTHER_REGISTERS <= THREADS * LAUNCH_REGISTERS, "more registers than the block has");
constexpr unsigned TMEM_COLS = 512;          // S0 [0,128) S1 [128,256), then of a pair O0 [256, 256 + DV) O1 [384, 384 + DV);
                                             // of a single stream P0 [256,320) P1 [320,384) O [384, 384 + DV)
constexpr unsigned O_COL = 256, P_COL = 256, SINGLE_O_COL = 384;
constexpr bool P_ON_S = DV > 64;             // a pair's P: over the scores it was made of, or beside its O where that is narrow
constexpr unsigned PAIR_P_COL = P_ON_S ? 0 : O_COL + 64;              // of stream 0; stream 1's 128 further
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_STEP = 8.f;          // log2 of the growth of a row maximum that forces a rescale
constexpr long long WAIT_CYCLES = 3000000000LL;         // about 1.5 s at 2 GHz

enum : int { STATUS_OK = 0, STATUS_LOADER = 1, STATUS_MMA = 2, STATUS_SOFTMAX = 3 };


__device__ __forceinline__ void cp_async_16(void* dst, const void* src, bool valid) {
    const int bytes = valid ? 16 : 0;        // 0: the destination is zero-filled, the source not read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
// 2^x by the special-function unit (two units in the last place; P is rounded to bf16 after it).
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// The two warps that share a quarter of the lanes meet here (barrier 1 + quarter, 64 threads).
__device__ __forceinline__ void pair_sync(int quarter) {
    asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory");
}

struct Barriers {
    unsigned long long q_full;
    unsigned long long k_full[2], k_empty[2], v_full[2], v_empty[2];
    unsigned long long s_full[2], s_empty[2];                        // of a pair's streams, of a single stream's two accumulators
    unsigned long long p_full[2][2];                                 // [stream or buffer][half of the keys, of a pair]
    unsigned long long pv_done, p_read[2], o_full;                   // of a single stream's tile, of a pair's [stream]; of all
};

// ------------------------------------------------------------------------------------------ a row's keys, half a tile at a time
// Both ways of taking a tile use these on the same 64 keys, in the same order, so a row has the same bits in a pair and alone.

// Worked-on scores, in base-2 units: two a step where the polynomial serves (every row of the warp alike), then the bias, an entry
// a distance only near the query.  first_pos: the position of the stream's first row.
__device__ __forceinline__ void work_on(float (&sc)[HALF], const mrun_score_form& form, const mrun::ScoreRow& form_row, int key_base,
                                        int first_pos, int row_pos) {
    if constexpr (SCORED) {
        if (__all_sync(0xffffffffu, form_row.small)) {
            const float2 factor2 = make_float2(form_row.factor, form_row.factor);
            const float2 cap2 = make_float2(form_row.cap2, form_row.cap2);
            const float2 far2 = make_float2(form_row.far_bias, form_row.far_bias);
#pragma unroll
            for (int i = 0; i < HALF; i += 2) {
                const float2 th = mrun::tanh_small2(__fmul2_rn(make_float2(sc[i], sc[i + 1]), factor2));
                const float2 v = __ffma2_rn(th, cap2, far2);
                sc[i] = v.x; sc[i + 1] = v.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < HALF; ++i) sc[i] = mrun::capped_score(form_row, sc[i]) + form_row.far_bias;
        }
        if (form.bias != nullptr && first_pos - (key_base + HALF - 1) < form.bias_len - 1) {
            // every entry as its difference from the far one, which the scores hold already
            const float* table = form_row.bias;
            const int distance = row_pos - key_base;
#pragma unroll
            for (int i = 0; i < HALF; ++i)
                sc[i] += fmaf(__ldg(table + min(max(distance - i, 0), form_row.bias_last)), LOG2E, -form_row.far_bias);
        }
    }
}

// Keys outside lo..hi, counted from the first of these, become -inf and later give p = 0.
__device__ __forceinline__ void mask_out(float (&sc)[HALF], int lo, int hi) {
#pragma unroll
    for (int i = 0; i < HALF; ++i)
        if (i > hi || i < lo) sc[i] = -INFINITY;
}

__device__ __forceinline__ float largest(const float (&sc)[HALF]) {
    float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int i = 0; i < HALF; i += 8)
#pragma unroll
        for (int c = 0; c < 4; ++c) mx4[c] = fmaxf(fmaxf(mx4[c], sc[i + 2 * c]), sc[i + 2 * c + 1]);
    return fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
}

// The maximum the probabilities are taken against moves only by large steps.  mx: the largest raw score (the scale is positive,
// so it scales the maximum alike).
__device__ __forceinline__ float next_max(float mx, float m_used, float scale_log2) {
    if constexpr (!SCORED) mx *= scale_log2;
    return mx > m_used + RESCALE_STEP || (m_used == -INFINITY && mx > -INFINITY) ? mx : m_used;
}

// A row's columns of O times corr.
__device__ __forceinline__ void rescale(unsigned address, int columns, float corr) {
#pragma unroll 1
    for (int c = 0; c < columns; c += 16) {
        float v[16];
        tmem_load16(address + c, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] *= corr;
        tmem_store16_start(address + c, v);
    }
}

// P = 2^(s * unit - m): one fused multiply-add and one special-function call a score, two scores an instruction where the hardware
// has one (fma.f32x2, add.f32x2), stored as packed bf16 from `address` on.  Masked scores are -inf and give 0; a row that has
// seen nothing yet keeps m = -inf.  Returns the sum.
__device__ __forceinline__ float probabilities(const float (&sc)[HALF], float unit, float m, unsigned address) {
    const float m_sub = m == -INFINITY ? 0.f : -m;
    const float2 scale2 = make_float2(unit, unit), m_sub2 = make_float2(m_sub, m_sub);
    float2 sums = make_float2(0.f, 0.f);
#pragma unroll
    for (int c = 0; c < HALF; c += 32) {
        float packed[16];                                             // two bf16 a word, even key low
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
            const float2 x = __ffma2_rn(make_float2(sc[c + i], sc[c + i + 1]), scale2, m_sub2);
            const float2 p = make_float2(fast_exp2(x.x), fast_exp2(x.y));
            sums = __fadd2_rn(sums, p);
            packed[i >> 1] = __uint_as_float(pack_bf16(p.x, p.y));
        }
        tmem_store16_start(address + c / 2, packed);
    }
    return sums.x + sums.y;
}

__global__ void __launch_bounds__(THREADS, 1)
prefill_tc5_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const bf16* __restrict__ q, long q_stride, bf16* __restrict__ out,
                   const int* __restrict__ block_tables, int max_blocks, const int* __restrict__ token_slot,
                   const int* __restrict__ positions, const int* __restrict__ tile_tok0,
                   const int* __restrict__ tile_ntok, int heads, int kv_heads, int page_size, int page_shift,
                   float scale_log2, int window, const float* __restrict__ sinks, const mrun_score_form form, int* __restrict__ status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* q_tile = base;
    unsigned char* k_stages = q_tile + MAX_Q * Q_BYTES;
    unsigned char* v_stages = k_stages + 2 * K_BYTES;

    __shared__ Barriers bars;
    __shared__ unsigned tmem_base_slot;
    __shared__ int aborted;
    __shared__ float half_max[2][2][ROWS];               // of a single stream: [tile parity][half of the keys][row]
    __shared__ float half_sum[2][ROWS];                  // [half][row], at the end

    // Blocks start in the order of their index, x first: all kv heads of the first tile of the
    // list, which the host sorted by falling work, then all of the second, ...
    const int tile = blockIdx.y, kvh = blockIdx.x;
    const int group = heads / kv_heads;
    const int tok0 = tile_tok0[tile], ntok = tile_ntok[tile];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per_stream = ROWS / group;                 // tokens
    const bool pair = MAX_Q == 2 && ntok > per_stream;   // two streams of rows
    // tokens of a tile are consecutive positions of one request
    const int pos_first = positions[tok0], pos_last = pos_first + ntok - 1;
    const int lo_tile = mrun::first_visible(pos_first, window);
    const int first_block = lo_tile / KEYS, last_block = pos_last / KEYS;
    const int n_tiles = last_block - first_block + 1;

    if (threadIdx.x == 0) {
        mbar_init(&bars.q_full, SOFTMAX_WARPS);                     // one arrival per softmax warp
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars.k_full[s], 32);                         // every lane of the loader warp arrives
            mbar_init(&bars.v_full[s], 32);
            mbar_init(&bars.k_empty[s], 1);
            mbar_init(&bars.v_empty[s], 1);
            mbar_init(&bars.s_full[s], 1);
            mbar_init(&bars.s_empty[s], SOFTMAX_WARPS);
            mbar_init(&bars.p_read[s], 1);
            mbar_init(&bars.p_full[s][0], pair ? STREAM_WARPS : SOFTMAX_WARPS);
            mbar_init(&bars.p_full[s][1], STREAM_WARPS);
        }
        mbar_init(&bars.pv_done, 1);
        mbar_init(&bars.o_full, 1);
        aborted = 0;
        mbar_init_fence();
    }
    // rows of a V stage that no copy ever fills must not hold NaN patterns: 0 * NaN is NaN
    for (int i = threadIdx.x; i < 2 * V_BYTES / 16; i += THREADS)
        reinterpret_cast<uint4*>(v_stages)[i] = make_uint4(0, 0, 0, 0);
    fence_async_smem();
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmem_base_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = tmem_base_slot;

    if (warp < SOFTMAX_WARPS) {
        // ------------------------------------------------------------------------------- softmax
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SOFTMAX_REGISTERS));
        const int quarter = warp & 3, side = warp >> 2;               // a pair: the stream; a single stream: the half of the keys
        const int row = quarter * 32 + lane;                          // 0..127
        const unsigned lane_base = tmem_base + ((unsigned)(quarter * 32) << 16);
        // q rows: row r = (token r / group, head kvh * group + r % group); rows past the stream's are zero
        for (int c = threadIdx.x; c < (pair ? 2 : 1) * ROWS * (D / 8); c += SOFTMAX_THREADS) {
            const int part = c / (ROWS * (D / 8)), in = c - part * (ROWS * (D / 8));
            const int r = in / (D / 8), chunk = in - r * (D / 8), token = part * per_stream + r / group;
            const bool valid = r < per_stream * group && token < ntok;
            const bf16* src = q;
            if (valid) src = q + (size_t)(tok0 + token) * q_stride + (size_t)(kvh * group + r % group) * D + chunk * 8;
            cp_async_16(q_tile + part * Q_BYTES + (chunk >> 3) * SPAN_BYTES + swizzled_offset(r, chunk & 7), src, valid);
        }
        cp_async_commit();
        cp_async_wait<0>();
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars.q_full);

        const int token0 = pair ? side * per_stream : 0;                          // the stream's tokens within the tile
        const int tokens = min(ntok - token0, per_stream);
        const int n_rows = tokens * group;
        const int first_pos = pos_first + token0, last_pos = first_pos + tokens - 1;
        const int row_pos = row < n_rows ? first_pos + row / group : -1;      // -1: padding row
        const int row_lo = mrun::first_visible(row_pos, window);
        // the stream's last row sees the most recent keys, its first row the oldest
        const int lo_last = mrun::first_visible(last_pos, window);
        const int head = kvh * group + row % group;
        mrun::ScoreRow form_row = {};
        if constexpr (SCORED) form_row = mrun::score_row(form, scale_log2 / LOG2E, row_pos, kvh * group + min(row, n_rows - 1) % group);
        const float unit = SCORED ? 1.f : scale_log2;
        float m_used = -INFINITY;
        float sum[2] = {0.f, 0.f};                    // of the row's keys 0..63 and 64..127 of every tile; a half's thread: its own first
        bool alive = true;
        // every row of the stream sees every key of the tile: no comparisons
        auto needs_mask = [&](int key0) { return key0 + KEYS - 1 > first_pos || key0 < lo_last || n_rows < ROWS; };
        if (pair) {
            for (int it = 0; it < n_tiles; ++it) {
                if (!__all_sync(0xffffffffu, mbar_wait(&bars.s_full[side], it & 1, WAIT_CYCLES, &aborted))) { alive = false; break; }
                const int key0 = (first_block + it) * KEYS;
                float sc[2][HALF];
                tc_fence_after();
                {
                    unsigned raw[KEYS];
#pragma unroll
                    for (int c = 0; c < KEYS; c += 32)
                        tmem_load32_start(lane_base + side * KEYS + c, *reinterpret_cast<unsigned (*)[32]>(&raw[c]));
                    tmem_load_wait();
#pragma unroll
                    for (int i = 0; i < KEYS; ++i) {
                        pin(raw[i]);
                        sc[i / HALF][i % HALF] = __uint_as_float(raw[i]);
                    }
                }
                const bool mask = needs_mask(key0);
                float mx = -INFINITY;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    work_on(sc[h], form, form_row, key0 + h * HALF, first_pos, row_pos);
                    if (mask) mask_out(sc[h], row_lo - key0 - h * HALF, row_pos - key0 - h * HALF);
                    mx = fmaxf(mx, largest(sc[h]));
                }
                const float m_new = next_max(mx, m_used, scale_log2);
                const bool moved = m_new != m_used && m_used != -INFINITY;       // O holds something to rescale
                if (__any_sync(0xffffffffu, moved)) {
                    // the second product of this stream's item before was issued before this one's first, so it has finished
                    const float corr = moved ? exp2f(m_used - m_new) : 1.f;
                    rescale(lane_base + O_COL + side * 128, DV, corr);
                    sum[0] *= corr;
                    sum[1] *= corr;
                }
                m_used = m_new;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    sum[h] += probabilities(sc[h], unit, m_used, lane_base + PAIR_P_COL + side * 128 + h * (HALF / 2));
                    tmem_store_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars.p_full[side][h]);           // half of the second product may begin
                }
            }
        } else {
            // A warp that gave up on a wait still walks through the remaining tiles, doing nothing but meeting its partner at
            // every barrier, so that no warp is left waiting at one.
            for (int j = 0; j < n_tiles; ++j) {
                const int buf = j & 1;
                if (alive && !__all_sync(0xffffffffu, mbar_wait(&bars.s_full[buf], (j >> 1) & 1, WAIT_CYCLES, &aborted))) alive = false;
                const int key0 = (first_block + j) * KEYS, half0 = key0 + side * HALF;
                float sc[HALF];
                float mx = -INFINITY;
                if (alive) {
                    tc_fence_after();
                    unsigned raw[HALF];
#pragma unroll
                    for (int c = 0; c < HALF; c += 32)
                        tmem_load32_start(lane_base + buf * KEYS + side * HALF + c, *reinterpret_cast<unsigned (*)[32]>(&raw[c]));
                    tmem_load_wait();
                    // the scores are in registers: the product after next may overwrite the accumulator
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars.s_empty[buf]);
#pragma unroll
                    for (int i = 0; i < HALF; ++i) {
                        pin(raw[i]);
                        sc[i] = __uint_as_float(raw[i]);
                    }
                    work_on(sc, form, form_row, half0, first_pos, row_pos);
                    if (needs_mask(key0)) mask_out(sc, row_lo - half0, row_pos - half0);
                    mx = largest(sc);
                }
                half_max[buf][side][row] = mx;
                pair_sync(quarter);
                if (!alive) continue;
                // both halves of a row decide alike, from the same numbers
                const float m_new = next_max(fmaxf(mx, half_max[buf][side ^ 1][row]), m_used, scale_log2);
                const bool moved = m_new != m_used && m_used != -INFINITY;
                if (__any_sync(0xffffffffu, moved)) {
                    // O belongs to the second product of the tile before until that has finished (the one before it has: its
                    // scores' barrier came behind it)
                    if (j > 0 && !__all_sync(0xffffffffu, mbar_wait(&bars.pv_done, (j - 1) & 1, WAIT_CYCLES, &aborted))) {
                        alive = false;
                        continue;
                    }
                    tc_fence_after();
                    const float corr = moved ? exp2f(m_used - m_new) : 1.f;
                    rescale(lane_base + SINGLE_O_COL + side * (DV / 2), DV / 2, corr);
                    sum[0] *= corr;
                }
                m_used = m_new;
                // the P buffer of this tile was read by the second product of the tile before last
                if (j >= 2 && !__all_sync(0xffffffffu, mbar_wait(&bars.v_empty[buf], ((j >> 1) - 1) & 1, WAIT_CYCLES, &aborted))) {
                    alive = false;
                    continue;
                }
                sum[0] += probabilities(sc, unit, m_used, lane_base + P_COL + buf * (KEYS / 2) + side * (HALF / 2));
                tmem_store_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars.p_full[buf][0]);
            }
        }
        // A warp leaves the loop as a whole, so every lane takes part in what follows.  o_full has one phase: of pv_done's, any of
        // the last three may be open when a warp comes here, and a parity tells a phase from its neighbours only.
        if (alive && !__all_sync(0xffffffffu, mbar_wait(&bars.o_full, 0, WAIT_CYCLES, &aborted))) alive = false;
        if (!alive) {
            if (!*(volatile int*)&aborted) atomicExch(status, STATUS_SOFTMAX);
            atomicExch(&aborted, 1);
        }
        if (!pair) {                                  // the other half's sum (its warp may have given up: it still comes here)
            half_sum[side][row] = sum[0];
            pair_sync(quarter);
            sum[1] = half_sum[side ^ 1][row];
        }
        if (alive) {
            tc_fence_after();
            const float total = with_sink(sum[0] + sum[1], m_used, sinks, head);
            const float inv = total > 0.f ? 1.f / total : 0.f;
            const int token = tok0 + token0 + row / group;
            // a pair's thread writes its row, a half's thread half of the columns
            const unsigned src = lane_base + (pair ? O_COL + side * 128 : SINGLE_O_COL);
            const int col0 = pair ? 0 : side * (DV / 2), col1 = pair ? DV : col0 + DV / 2;
            bf16* dst = out + (size_t)token * (SCORED ? form.out_stride : (long)heads * DV) + head * DV;
#pragma unroll 1
            for (int c = col0; c < col1; c += 32) {
                float v[32];
                tmem_load32(src + c, v);              // every lane of the warp takes part
                if (row < n_rows) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] *= inv;
                    if constexpr (SCORED) mrun::gate_outputs<32>(form, token, head * DV + c, v);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        *reinterpret_cast<uint4*>(dst + c + 8 * k) =
                            make_uint4(pack_bf16(v[8 * k], v[8 * k + 1]), pack_bf16(v[8 * k + 2], v[8 * k + 3]),
                                       pack_bf16(v[8 * k + 4], v[8 * k + 5]), pack_bf16(v[8 * k + 6], v[8 * k + 7]));
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OTHER_REGISTERS));
        if (warp == MMA_WARP) {
            // ------------------------------------------------------------------------ MMA issuer
            constexpr unsigned idesc_qk = instruction_descriptor(ROWS, KEYS);
            constexpr unsigned idesc_pv = instruction_descriptor(ROWS, DV, true);
            const unsigned long long q_desc = smem_descriptor(q_tile), k_desc = smem_descriptor(k_stages);
            const unsigned long long v_desc = smem_descriptor(v_stages, SPAN_BYTES, 1024);
            auto wait = [&](unsigned long long* bar, unsigned parity) {
                return (bool)__all_sync(0xffffffffu, mbar_wait(bar, parity, WAIT_CYCLES, &aborted));
            };
            // Descriptors further on differ in their address field, which counts 16-byte units.
            auto issue_qk = [&](int acc, int q_part, int s) {             // by the elected lane; s: K's stage
                const unsigned long long qd = q_desc + q_part * (Q_BYTES >> 4), kd = k_desc + s * (K_BYTES >> 4);
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {                     // 32 bytes further along d per step
                    const int off = ((kk >> 2) * SPAN_BYTES + (kk & 3) * 32) >> 4;
                    umma_bf16(tmem_base + acc * KEYS, qd + off, kd + off, idesc_qk, kk > 0 ? 1u : 0u);
                }
                umma_commit(&bars.s_full[acc]);
                if (!pair || acc == 1) umma_commit(&bars.k_empty[s]);
            };
            // P: eight columns (16 keys) further per step; V: sixteen rows.  Steps [from, to) of the tile's eight.
            auto issue_pv = [&](unsigned o, unsigned p, int s, int from, int to, bool first) {
                const unsigned long long vd = v_desc + s * (V_BYTES >> 4);
#pragma unroll
                for (int kk = 0; kk < KEYS / 16; ++kk)
                    if (kk >= from && kk < to)
                        umma_bf16_a_tmem(tmem_base + o, tmem_base + p + kk * 8, vd + kk * (2048 >> 4), idesc_pv, (!first || kk > 0) ? 1u : 0u);
            };
            bool alive = wait(&bars.q_full, 0);
            // Item i of a pair is stream i & 1's, key tile i / 2; a single stream's is key tile i.
            const int n_items = pair ? 2 * n_tiles : n_tiles;
            for (int i = 0; alive && i < 2 && i < n_items; ++i) {
                const int s = pair ? 0 : i;
                alive = wait(&bars.k_full[s], 0);
                if (!alive) break;
                if (elect_one()) issue_qk(i, pair ? i : 0, s);
                __syncwarp();
            }
            for (int i = 0; alive && i < n_items; ++i) {
                const int acc = i & 1, j = pair ? i >> 1 : i, s = j & 1;
                const int next = pair ? j + 1 : j + 2, next_s = next & 1;         // the key tile of the accumulator's next item
                const bool more = i + 2 < n_items;
                // what is waited for comes in the order of its arrival, P last, so that it goes on at once then
                if (!wait(&bars.v_full[s], (j >> 1) & 1) || (more && !wait(&bars.k_full[next_s], (next >> 1) & 1)) ||
                    !wait(&bars.p_full[acc][0], (i >> 1) & 1)) {
                    alive = false;
                    break;
                }
                tc_fence_after();
                if (pair) {
                    const unsigned o = O_COL + acc * 128, p = PAIR_P_COL + acc * 128;
                    if (elect_one()) issue_pv(o, p, s, 0, KEYS / 32, i < 2);
                    __syncwarp();
                    if (!wait(&bars.p_full[acc][1], (i >> 1) & 1)) { alive = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
                        issue_pv(o, p, s, KEYS / 32, KEYS / 16, i < 2);
                        if (acc == 1) umma_commit(&bars.v_empty[s]);
                        if (P_ON_S) umma_commit(&bars.p_read[acc]);
                        if (i + 1 == n_items) umma_commit(&bars.o_full);
                    }
                    __syncwarp();
                    // The stream's next scores go where its P lies.  Products into different accumulators have no promised order, so
                    // the ones that read P end first: 2.25 us a tile in place of 2.05.  (Held back behind the other stream's product
                    // where that could go on 2.37; the upper 64 keys' scores, which lie beside P, at once 2.4.)
                    if (P_ON_S && more && !wait(&bars.p_read[acc], (i >> 1) & 1)) { alive = false; break; }
                    tc_fence_after();
                    if (more && elect_one()) issue_qk(acc, acc, next_s);
                    __syncwarp();
                } else {
                    if (elect_one()) {
                        issue_pv(SINGLE_O_COL, P_COL + acc * (KEYS / 2), s, 0, KEYS / 16, i == 0);
                        umma_commit(&bars.v_empty[s]);
                        umma_commit(&bars.pv_done);
                        if (i + 1 == n_items) umma_commit(&bars.o_full);
                    }
                    __syncwarp();
                    // the scores before are in registers
                    if (more && !wait(&bars.s_empty[acc], (i >> 1) & 1)) { alive = false; break; }
                    if (more && elect_one()) issue_qk(acc, 0, next_s);
                    __syncwarp();
                }
            }
            if (!alive) {
                if (!*(volatile int*)&aborted) atomicExch(status, STATUS_MMA);
                atomicExch(&aborted, 1);
            }
        } else if (warp <= V_WARP) {
            // --------------------------------------------------------------------------- loaders
            const bool keys_role = warp == K_WARP;                        // one warp for K, one for V
            const CUtensorMap* map = keys_role ? &map_k : &map_v;
            unsigned char* stages = keys_role ? k_stages : v_stages;
            unsigned long long* full = keys_role ? bars.k_full : bars.v_full;
            unsigned long long* empty = keys_role ? bars.k_empty : bars.v_empty;
            const int* table = block_tables + (size_t)token_slot[tok0] * max_blocks;
            // pages of up to 128 keys: 128 / page_size boxes of page_size rows; larger pages: one box
            const int box_rows = page_size < KEYS ? page_size : KEYS;
            const int boxes = KEYS / box_rows;
            // The pages of a lane's boxes (lane, lane + 32, ...), looked up a tile ahead: -1 where nothing is to be copied.
            constexpr int MAX_BOXES = KEYS / 32;
            int pages[MAX_BOXES];
            auto look_up = [&](int j) {
#pragma unroll
                for (int u = 0; u < MAX_BOXES; ++u) {
                    const int b = lane + 32 * u, first_key = (first_block + j) * KEYS + b * box_rows;
                    const bool wanted = j < n_tiles && b < boxes && first_key <= pos_last && first_key + box_rows - 1 >= lo_tile;
                    pages[u] = wanted ? table[first_key >> page_shift] : -1;
                }
            };
            look_up(0);
            bool alive = true;
            for (int j = 0; j < n_tiles; ++j) {
                const int s = j & 1;
                const bool free_now = j < 2 || mbar_wait(&empty[s], ((j >> 1) - 1) & 1, WAIT_CYCLES, &aborted);
                if (!__all_sync(0xffffffffu, free_now)) { alive = false; break; }
                unsigned char* stage = stages + s * (keys_role ? K_BYTES : V_BYTES);
                unsigned bytes = 0;                               // a lane announces its boxes' bytes, then copies them
#pragma unroll
                for (int u = 0; u < MAX_BOXES; ++u) bytes += pages[u] >= 0 ? (unsigned)(box_rows * (keys_role ? D : DV) * 2) : 0u;
                if (bytes) mbar_expect_tx(&full[s], bytes);
                else mbar_arrive(&full[s]);
#pragma unroll
                for (int u = 0; u < MAX_BOXES; ++u) {
                    if (pages[u] < 0) continue;
                    const int b = lane + 32 * u, first_key = (first_block + j) * KEYS + b * box_rows;
#pragma unroll
                    for (int h = 0; h < (SPANS_D > SPANS_V ? SPANS_D : SPANS_V); ++h)
                        if (h < (keys_role ? SPANS_D : SPANS_V))
                            tma_load_4d(stage + h * SPAN_BYTES + b * box_rows * 128, map, h * 64,
                                        first_key & (page_size - 1), kvh, pages[u], &full[s]);
                }
                look_up(j + 1);
            }
            if (!alive) {
                if (!*(volatile int*)&aborted) atomicExch(status, STATUS_LOADER);
                atomicExch(&aborted, 1);
            }
        }
    }

    // ---------------------------------------------------------------------------------- teardown
    tc_fence_before();
    __syncthreads();
    if (*(volatile int*)&aborted) {
        // copies that were requested may still be landing in this block's shared memory
        const long long start = clock64();
        while (clock64() - start < 4000000LL) __nanosleep(1000);
    }
    if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace

#endif  // MRUN_ATTN_TC5

// Rows per block of the tcgen05 kernel (head sizes 64 and 128, and keys of 192): a tile of the list holds at most this
// divided by heads / kv_heads tokens, cut into streams of 128 / (heads / kv_heads).  0: not in this library.
MRUN_API int mrun_attn_prefill_tc5_rows() {
#if MRUN_ATTN_TC5
    return MAX_Q * ROWS;
#else
    return 0;
#endif
}

// As mrun_attn_prefill, with tiles of as many tokens as mrun_attn_prefill_tc5_rows() says, a page size that is
// a power of two, and `pages` the number of pages of the two cache tensors.  `status` is one
// int on the device, zero before the first call; a non-zero value afterwards names the role whose
// wait ran out (1 loader, 2 products, 3 softmax) and the outputs of that launch are void.
MRUN_API int mrun_attn_prefill_tc5(const void* q, long q_stride, void* out, const void* k_cache,
                                   const void* v_cache, const int* block_tables, int max_blocks,
                                   const int* token_slot, const int* positions, const int* tile_tok0,
                                   const int* tile_ntok, int n_tiles, int heads, int kv_heads, int head_dim,
                                   int page_size, float scale, int window, const float* sinks, long pages,
                                   const mrun_score_form* form, int* status, cudaStream_t stream) {
#if MRUN_ATTN_TC5
    MRUN_REQUIRE(head_dim == D, "attn_prefill_tc5: this library was built for head_dim=%d, got %d", D, head_dim);
    MRUN_REQUIRE(heads > 0 && kv_heads > 0 && heads % kv_heads == 0,
                 "attn_prefill_tc5: heads=%d must be a positive multiple of kv_heads=%d", heads, kv_heads);
    MRUN_REQUIRE(heads / kv_heads <= ROWS, "attn_prefill_tc5: %d query heads per kv head exceed the supported %d",
                 heads / kv_heads, ROWS);
    MRUN_REQUIRE(page_size > 0 && max_blocks > 0, "attn_prefill_tc5: bad page_size/max_blocks");
    MRUN_REQUIRE(n_tiles >= 0, "attn_prefill_tc5: n_tiles=%d", n_tiles);
    MRUN_REQUIRE(q_stride % 8 == 0 && ((uintptr_t)q & 15) == 0 && ((uintptr_t)out & 15) == 0 &&
                 ((uintptr_t)k_cache & 15) == 0 && ((uintptr_t)v_cache & 15) == 0,
                 "attn_prefill_tc5: q, out and the caches must be 16-byte aligned, q_stride a multiple of 8");
    MRUN_REQUIRE(SCORED == (form != nullptr), "attn_prefill_tc5: this library was built %s a score form",
                 SCORED ? "for" : "without");
    if (form)
        MRUN_REQUIRE(form->out_stride >= (long)heads * DV && form->out_stride % 8 == 0 &&
                     (form->gate == nullptr || (form->gate_stride >= (long)heads * DV && form->gate_stride % 8 == 0 &&
                                                ((uintptr_t)form->gate & 15) == 0)),
                     "attn_prefill_tc5: the output's and the gate's rows must start on 16 bytes and hold %d features", heads * DV);
    MRUN_REQUIRE(status != nullptr, "attn_prefill_tc5: the status word is missing");
    MRUN_REQUIRE(page_shift_of(page_size) >= 0, "attn_prefill_tc5: page_size=%d is not a power of two", page_size);
    MRUN_REQUIRE(pages > 0 && pages < (1L << 31), "attn_prefill_tc5: pages=%ld", pages);
    if (n_tiles == 0) return 0;
    CUtensorMap map_k, map_v;
    const int box_rows = page_size < KEYS ? page_size : KEYS;
    if (int rc = paged_cache_map(&map_k, k_cache, pages, kv_heads, page_size, D, box_rows, "attn_prefill_tc5")) return rc;
    if (int rc = paged_cache_map(&map_v, v_cache, pages, kv_heads, page_size, DV, box_rows, "attn_prefill_tc5")) return rc;
    static bool configured = false;
    if (!configured) {
        MRUN_CHECK_CUDA(cudaFuncSetAttribute(prefill_tc5_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             SMEM_BYTES), "attn_prefill_tc5");
        cudaFuncAttributes has;
        MRUN_CHECK_CUDA(cudaFuncGetAttributes(&has, prefill_tc5_kernel), "attn_prefill_tc5");
        MRUN_REQUIRE(has.numRegs == LAUNCH_REGISTERS, "attn_prefill_tc5: built with %d registers a thread, %d are dealt out", has.numRegs,
                     LAUNCH_REGISTERS);
        configured = true;
    }
    for (int done = 0; done < n_tiles; done += 65535) {          // the grid's second dimension ends at 65535
        const int now = n_tiles - done < 65535 ? n_tiles - done : 65535;
        prefill_tc5_kernel<<<dim3(kv_heads, now), THREADS, SMEM_BYTES, stream>>>(
            map_k, map_v, (const bf16*)q, q_stride, (bf16*)out, block_tables, max_blocks,
            token_slot, positions, tile_tok0 + done, tile_ntok + done, heads, kv_heads, page_size, page_shift_of(page_size),
            scale * LOG2E, window, sinks, form ? *form : mrun_score_form{}, status);
        MRUN_CHECK_LAUNCH("attn_prefill_tc5");
    }
    return 0;
#else
    return mrun_set_error("attn_prefill_tc5: not built for head_dim=%d (head sizes 64 and 128, keys of 192 with smaller values)", MRUN_HEAD_DIM);
#endif
}
