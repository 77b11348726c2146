// 32-bit linear layer on the bfloat16 tensor cores (tcgen05): y[M, N] = x[M, K] · w[N, K]^T where every 32-bit
// operand is taken as the exact sum of three bfloat16 values, 2^24 a = a1 + a2 + a3 (8 significant bits each, rounded to
// nearest, so |a2| <= 2^-8 |a1| and |a3| <= 2^-16 |a1|), and the six products
//     a1 b1,  a1 b2 + a2 b1,  a1 b3 + a2 b2 + a3 b1
// are added up; what is left out is below 2^-24 of |a b|, and of either sign.  Without the factor, which a sum loses again, the third
// part of an operand below 2^-109 would have fallen under bfloat16's least value; with it the split is exact down to the least 32-bit
// value.  Products of two bfloat16 values are exact in 32 bits.  The tensor core adds up 64 values of k at a time from zero; these sums are added by 32-bit
// additions in order, and where a row of w is cut into `split` ranges of k (chosen from N and K alone), the ranges' sums in order of
// range.  So a row of x has the same bits whatever M is and wherever it sits in the batch.  A result that is not
// finite (an operand that is not or is beyond 2^103, or a sum beyond 2^79) is computed again as a chain of fused multiply-adds.
//
//   split   (a kernel in front) writes the three parts of x, [3][M][K], so that TMA brings them
//   product a block a tile of 128 rows of w (the MMA's M) x TOK tokens (its N) and a range of k; a cluster's
//           blocks have the ranges of one tile and meet in shared memory at the end, or (many tokens) a block takes the ranges
//           one after the other and adds each range's sum to y.  The raw 32-bit w comes by TMA; two groups of four warps, a
//           thread a row, take 32 k of it in turn to three bfloat16 parts in tensor memory (the MMA's A operand: shared
//           memory's bandwidth is left to B, and w is read from HBM once, 4 bytes a weight); two warps issue twelve
//           MMAs for 32 k, each for every second sum, so that one's waits pass while the other's MMAs run; eight warps add every
//           64-k sum of the tensor core to their registers.
//
// Few rows are bound by reading w, many by the MMAs (six products).  us, B200, this / the chain of multiply-adds of
// gemm_f32.cu: N = 24,576, K = 4,096, four rows 78 / 92 (5.1 TB/s), 24 rows 80 / 231, 100 rows 173 / 592, 517 rows 429 / 2,233
// (1.46 PFLOP/s of MMAs, 243 TFLOP/s of the product; 74 is the multiply-add pipe's peak); N = 4,096, K = 12,288, four rows 38 / 57,
// 517 rows 310 / 1,246.  Error against 64 bits over results (2-norms): K = 4,096 3.4e-7 / 1.14e-6, K = 1,028 3.3e-7 / 5.7e-7.
// What the parts of the design gave (N = 4,096, K = 4,096, one range, four rows): an elected lane in place of lane 0 80 -> 50 us (the
// descriptors of an MMA then lie in uniform registers: 22 cycles an instruction instead of 57); four stages of w's parts in place of
// two 112 -> 105 (N = 24,576, 64 tokens); a second warp of MMAs 442 -> 428 (N = 24,576, 517 rows).
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

using namespace tc5;

typedef __nv_bfloat16 bf16;

constexpr int ROWS = 128;                 // rows of w a tile
constexpr int BK = 64, HALF = 32;         // k of a sum of the tensor core (and of a box of x), of a box of w
constexpr int PARTS = 3;
constexpr int CONVERT_WARPS = 8;          // two groups, each every second box of w: a group's waits hide behind the other
constexpr int MAX_SPLIT = 8;              // the portable cluster size
constexpr int W_BYTES = ROWS * HALF * 4;
constexpr int A_COLUMNS = PARTS * HALF / 2;
constexpr float SCALE = 16777216.f, UNSCALE = 1.f / SCALE / SCALE;      // 2^24 of either operand, 2^-48 of a sum
constexpr long long WAIT_CYCLES = 3000000000LL;   // about 1.5 s at 2 GHz

enum : int { STATUS_W = 1, STATUS_X = 2, STATUS_CONVERT = 3, STATUS_MMA = 4, STATUS_SUM = 5 };

template <int TOK> struct Shape {
    static constexpr int BLOCKS = TOK <= 32 ? 2 : 1;              // on a multiprocessor
    static constexpr bool FOLDS = TOK > 32;                       // whether a block may take the ranges one after the other
    static constexpr int X_BYTES = PARTS * TOK * BK * 2;
    static constexpr int X_STAGES = TOK <= 96 ? 3 : 2;
    static constexpr int BUDGET = (BLOCKS == 2 ? 112 : 225) * 1024 - 1024;
    static constexpr int W_FIT = (BUDGET - X_STAGES * X_BYTES) / W_BYTES;
    // an even number: a stage is read by one group of converting warps, which meets every phase of its barriers
    static constexpr int W_STAGES = (W_FIT < 10 ? W_FIT : 10) / 2 * 2;
    static constexpr int SMEM = 1024 + X_STAGES * X_BYTES + W_STAGES * W_BYTES;
    static constexpr int A_STAGES = TOK <= 160 ? 4 : 2;           // of w's parts, for the groups in turn
    static constexpr int COLUMNS_USED = 2 * TOK + A_STAGES * A_COLUMNS;
    static constexpr unsigned COLUMNS = COLUMNS_USED <= 128 ? 128 : COLUMNS_USED <= 256 ? 256 : 512;
    static constexpr int SUM_WARPS = TOK <= 32 ? 4 : 8, EACH = TOK * 4 / SUM_WARPS;      // EACH: tokens of a summing thread
    static constexpr int W_WARP = CONVERT_WARPS + SUM_WARPS, MMA_WARP = W_WARP + 1, X_WARP = W_WARP + 3;
    // The summing warps of the widest tiles take registers from the others (setmaxnreg works on four warps together, and waits
    // for good where the block was launched with fewer than are dealt out: launch() looks).
    static constexpr bool UNEVEN = TOK >= 112;
    static constexpr int THREADS = 32 * (X_WARP + 1), LAUNCH_REGISTERS = 96;
    static_assert(!UNEVEN || CONVERT_WARPS * 72 + SUM_WARPS * 144 + 4 * 40 <= THREADS / 32 * LAUNCH_REGISTERS, "more registers than the block has");
    static_assert(COLUMNS_USED <= 512 && W_STAGES >= 4 && TOK % 16 == 0, "the tile does not fit");
    static_assert(X_STAGES * X_BYTES >= TOK * ROWS * 4, "the ranges' sums take the place of x");
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void tmem_store8(unsigned address, const unsigned (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(address), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_load8(unsigned address, float (&v)[8]) {
    unsigned r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(address) : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// The three parts of 2^24 times two values, packed as the tensor core wants them (the first in the low half).
__device__ __forceinline__ void three_parts(float x, float y, unsigned (&part)[PARTS]) {
    const float2 scaled = __fmul2_rn(make_float2(x, y), make_float2(SCALE, SCALE));
    x = scaled.x;
    y = scaled.y;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
        const __nv_bfloat162 both = __floats2bfloat162_rn(x, y);
        part[p] = *reinterpret_cast<const unsigned*>(&both);
        x -= __uint_as_float(part[p] << 16);
        y -= __uint_as_float(part[p] & 0xffff0000u);
    }
}

// ------------------------------------------------------------------------------------------ split
constexpr int SPLIT_THREADS = 256;

// parts[p][row][k], `plane` values a part, four values of k a thread.
template <bool ALIGNED>
__global__ void __launch_bounds__(SPLIT_THREADS)
split_rows_kernel(const float* __restrict__ x, long ldx, bf16* __restrict__ parts, long plane, int pitch, long quads, int quads_a_row) {
    mrun::wait_for_kernel_before();
    mrun::dependents_may_start();
    const long i = (long)blockIdx.x * SPLIT_THREADS + threadIdx.x;
    if (i >= quads) return;
    const long row = i / quads_a_row;
    const int k = (int)(i - row * quads_a_row) * 4;
    const float* src = x + row * ldx + k;
    float4 v;
    if constexpr (ALIGNED) v = *reinterpret_cast<const float4*>(src);
    else v = make_float4(src[0], src[1], src[2], src[3]);
    unsigned lo[PARTS], hi[PARTS];
    three_parts(v.x, v.y, lo);
    three_parts(v.z, v.w, hi);
    bf16* dst = parts + row * pitch + k;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) *reinterpret_cast<uint2*>(dst + p * plane) = make_uint2(lo[p], hi[p]);
}

// ------------------------------------------------------------------------------------------ product
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// What block `rank` of the cluster has at an own shared address.
__device__ __forceinline__ float cluster_load(unsigned own_shared, unsigned rank) {
    unsigned remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote) : "r"(own_shared), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }

struct ProductArgs {
    const float *x, *w;
    float* y;
    long ldx, ldy;
    int M, N, K, blocks;                  // blocks: of BK, in K
    int ranges;                           // of k: a block of the cluster each, or (clusters of one) one after the other
    int* status;
};

template <int TOK>
__global__ void __launch_bounds__(Shape<TOK>::THREADS, Shape<TOK>::BLOCKS)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const ProductArgs a) {
    using S = Shape<TOK>;
    constexpr int WS = S::W_STAGES, XS = S::X_STAGES, A_STAGES = S::A_STAGES, SUM_WARPS = S::SUM_WARPS;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* x_ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* w_ring = x_ring + XS * S::X_BYTES;
    __shared__ unsigned long long w_full[WS], w_empty[WS], x_full[XS], x_empty[XS], a_full[4], a_empty[A_STAGES], sum_full[2],
        sum_empty[2];
    __shared__ unsigned tmem_slot;
    __shared__ int aborted;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = (int)gridDim.x, rank = (int)blockIdx.x;     // a cluster is a row of the grid
    const int tok0 = blockIdx.y * TOK, row0 = blockIdx.z * ROWS;
    const int b0 = (int)((long)rank * a.blocks / split), n = (int)((long)(rank + 1) * a.blocks / split) - b0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < WS; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], CONVERT_WARPS / 2); }
        for (int s = 0; s < XS; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
        for (int s = 0; s < 4; ++s) mbar_init(&a_full[s], CONVERT_WARPS / 2);      // of each half of the sums of either accumulator
        for (int s = 0; s < A_STAGES; ++s) mbar_init(&a_empty[s], 1);
        for (int s = 0; s < 2; ++s) { mbar_init(&sum_full[s], 1); mbar_init(&sum_empty[s], SUM_WARPS); }
        aborted = 0;
        mbar_init_fence();
    }
    __syncwarp();
    if (warp == S::MMA_WARP) tmem_alloc(&tmem_slot, S::COLUMNS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_slot, a_tmem = tmem + 2 * TOK;
    auto wait = [&](unsigned long long* bar, int parity, int role) {
        if (mbar_wait(bar, (unsigned)parity, WAIT_CYCLES, &aborted)) return true;
        if (!*(volatile int*)&aborted) atomicExch(a.status, role);
        atomicExch(&aborted, 1);
        return false;
    };
    int out_of_range = 0;
    if (warp >= S::W_WARP) {
        if constexpr (S::UNEVEN) asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == S::W_WARP) {
            // Before the kernel in front has ended: it writes x's parts only, and began when what was before it had ended.
            for (int j = 0; j < 2 * n; ++j) {
                const int s = j % WS;
                if (j >= WS && !__all_sync(0xffffffffu, wait(&w_empty[s], (j / WS - 1) & 1, STATUS_W))) break;
                if (elect_one()) {
                    mbar_expect_tx(&w_full[s], W_BYTES);
                    tma_load_2d(w_ring + s * W_BYTES, &map_w, b0 * BK + j * HALF, row0, &w_full[s]);
                }
                __syncwarp();
            }
        } else if (warp == S::X_WARP) {
            mrun::wait_for_kernel_before();
            for (int j = 0; j < n; ++j) {
                const int s = j % XS;
                if (j >= XS && !__all_sync(0xffffffffu, wait(&x_empty[s], (j / XS - 1) & 1, STATUS_X))) break;
                if (elect_one()) {
                    mbar_expect_tx(&x_full[s], S::X_BYTES);
                    tma_load_3d(x_ring + s * S::X_BYTES, &map_x, (b0 + j) * BK, tok0, 0, &x_full[s]);
                }
                __syncwarp();
            }
        } else {
            // Two warps, each every second sum: the waits of one pass while the other's products run.
            constexpr unsigned idesc = instruction_descriptor(ROWS, TOK);
            const int buf = warp - S::MMA_WARP;
            const unsigned d = tmem + buf * TOK;
            bool alive = true;
            for (int j = buf; j < n && alive; j += 2) {
                const int xs = j % XS;
                if (j >= 2 && !__all_sync(0xffffffffu, wait(&sum_empty[buf], ((j >> 1) - 1) & 1, STATUS_MMA))) break;
                // The sum before the last one has been read, so the other warp's products before it are done: with three stages of x
                // this warp meets every second phase of a stage's barrier, and the one between has passed.
                if (!__all_sync(0xffffffffu, wait(&x_full[xs], (j / XS) & 1, STATUS_MMA))) break;
                const unsigned long long b = smem_descriptor(x_ring + xs * S::X_BYTES);
                constexpr unsigned long long b_part = TOK * BK * 2 >> 4, b_step = 32 >> 4;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int as = (2 * buf + h) % A_STAGES;  // a sum takes two boxes of w
                    if (!__all_sync(0xffffffffu, wait(&a_full[2 * buf + h], (j >> 1) & 1, STATUS_MMA))) { alive = false; break; }
                    tc_fence_after();
                    if (elect_one()) {
                        // the smallest first, so that few additions are rounded at the size of the whole sum
                        constexpr int order[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
#pragma unroll
                        for (int o = 0; o < 6; ++o)
#pragma unroll
                            for (int k = 0; k < 2; ++k)
                                umma_bf16_a_tmem(d, a_tmem + as * A_COLUMNS + order[o][0] * (HALF / 2) + k * 8,
                                                 b + order[o][1] * b_part + (2 * h + k) * b_step, idesc, (h | o | k) ? 1u : 0u);
                        umma_commit(&a_empty[as]);
                        if (h == 1) {
                            umma_commit(&x_empty[xs]);
                            umma_commit(&sum_full[buf]);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < CONVERT_WARPS) {
        if constexpr (S::UNEVEN) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        const int r = threadIdx.x % ROWS;
        for (int j = warp / 4; j < 2 * n; j += 2) {
            const int s = j % WS, as = j % A_STAGES;
            if (!__all_sync(0xffffffffu, wait(&w_full[s], (j / WS) & 1, STATUS_CONVERT))) break;
            if (j >= A_STAGES && !__all_sync(0xffffffffu, wait(&a_empty[as], (j / A_STAGES - 1) & 1, STATUS_CONVERT))) break;
            tc_fence_after();
            const unsigned char* src = w_ring + s * W_BYTES + r * 128;
            const unsigned dst = a_tmem + as * A_COLUMNS + ((unsigned)((warp & 3) * 32) << 16);
#pragma unroll
            for (int half = 0; half < 2; ++half) {        // 16 k each
                unsigned part[PARTS][8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = *reinterpret_cast<const float4*>(src + (((half * 4 + c) ^ (r & 7)) << 4));
                    unsigned lo[PARTS], hi[PARTS];
                    three_parts(v.x, v.y, lo);
                    three_parts(v.z, v.w, hi);
#pragma unroll
                    for (int p = 0; p < PARTS; ++p) { part[p][2 * c] = lo[p]; part[p][2 * c + 1] = hi[p]; }
                }
#pragma unroll
                for (int p = 0; p < PARTS; ++p) tmem_store8(dst + p * (HALF / 2) + half * 8, part[p]);
            }
            tmem_store_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&w_empty[s]);
                mbar_arrive(&a_full[j & 3]);
            }
        }
    } else {
        if constexpr (S::UNEVEN) asm volatile("setmaxnreg.inc.sync.aligned.u32 144;");
        float acc[S::EACH];
        const int quarter = warp & 3, part = (warp - CONVERT_WARPS) >> 2;      // lanes of tensor memory, half of the tokens
        const unsigned src = tmem + part * S::EACH + ((unsigned)(quarter * 32) << 16);
        const int in = quarter * 32 + lane, row = row0 + in;
        int range = 0, range_end = a.blocks / a.ranges;
        mrun::wait_for_kernel_before();
#pragma unroll
        for (int i = 0; i < S::EACH; ++i) acc[i] = 0.f;
        for (int j = 0; j < n; ++j) {
            const int buf = j & 1;
            if (!__all_sync(0xffffffffu, wait(&sum_full[buf], (j >> 1) & 1, STATUS_SUM))) break;
            tc_fence_after();
#pragma unroll
            for (int c = 0; c + 16 <= S::EACH; c += 16) {
                float v[16];
                tmem_load16(src + buf * TOK + c, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[c + i] += v[i];
            }
            if constexpr (S::EACH % 16 != 0) {
                float v[8];
                tmem_load8(src + buf * TOK + S::EACH / 16 * 16, v);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[S::EACH / 16 * 16 + i] += v[i];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[buf]);
            if (split == 1 && j + 1 == range_end) {       // y takes the ranges' sums one after the other
                const int first = tok0 + part * S::EACH;
                float* dst = a.y + (long)min(first, a.M - 1) * a.ldy + min(row, a.N - 1);
                asm volatile("" : "+l"(dst));             // or all the addresses are kept through the loop
                constexpr int RUN = 8;
#pragma unroll
                for (int c = 0; c < S::EACH; c += RUN) {
                    float before[RUN];
                    if (S::FOLDS && range > 0) {          // no branch a load: they are on their way together
                        const float* src_y = dst;
#pragma unroll
                        for (int i = 0; i < RUN; ++i) {
                            before[i] = *src_y;
                            src_y += first + c + i + 1 < a.M ? a.ldy : 0;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < RUN; ++i) {
                        const float sum = acc[c + i] * UNSCALE, v = S::FOLDS && range > 0 ? before[i] + sum : sum;
                        if (first + c + i < a.M && row < a.N) {
                            *dst = v;
                            if (j + 1 == n) out_of_range |= !finite(v);
                        }
                        dst += first + c + i + 1 < a.M ? a.ldy : 0;
                    }
                    asm volatile("" ::: "memory");
                }
#pragma unroll
                for (int i = 0; i < S::EACH; ++i) acc[i] = 0.f;
                range += 1;
                range_end = (int)((long)(range + 1) * a.blocks / a.ranges);
            }
        }
        // Every MMA has ended and every copy has landed: x's place takes the sums, [TOK][ROWS].
        if (split > 1) {
            float* sums = reinterpret_cast<float*>(x_ring);
            if (!*(volatile int*)&aborted)
#pragma unroll
                for (int i = 0; i < S::EACH; ++i) sums[(part * S::EACH + i) * ROWS + in] = acc[i] * UNSCALE;
        }
    }

    tc_fence_before();
    out_of_range = __syncthreads_or(out_of_range);
    if (*(volatile int*)&aborted) {
        // copies that were requested may still be landing in this block's shared memory
        const long long start = clock64();
        while (clock64() - start < 4000000LL) __nanosleep(1000);
    }
    __syncwarp();
    if (warp == S::MMA_WARP) tmem_dealloc(tmem, S::COLUMNS);
    __syncwarp();
    if (split > 1) {
        cluster_sync_all();
        // a block finishes every split-th token
        const unsigned sums = smem_u32(x_ring);
        for (int e = threadIdx.x; e < TOK * ROWS; e += S::THREADS) {
            const int t = e / ROWS, in = e % ROWS, tok = tok0 + t, row = row0 + in;
            if (t % split != rank || tok >= a.M || row >= a.N) continue;
            float v = cluster_load(sums + e * 4, 0);
            for (int r = 1; r < split; ++r) v += cluster_load(sums + e * 4, r);
            a.y[(long)tok * a.ldy + row] = v;
            out_of_range |= !finite(v);
        }
        __syncwarp();
        cluster_sync_all();                               // nobody leaves while another block still reads here
        out_of_range = __syncthreads_or(out_of_range);
    }
    if (!out_of_range) return;
    for (int e = threadIdx.x; e < TOK * ROWS; e += S::THREADS) {
        const int t = e / ROWS, tok = tok0 + t, row = row0 + e % ROWS;
        if (t % split != rank || tok >= a.M || row >= a.N || finite(a.y[(long)tok * a.ldy + row])) continue;
        float v = 0.f;
        for (int k = 0; k < a.K; ++k) v = fmaf(a.x[(long)tok * a.ldx + k], a.w[(long)row * a.K + k], v);
        a.y[(long)tok * a.ldy + row] = v;
    }
}

// ------------------------------------------------------------------------------------------ host
int encode_map(CUtensorMap* map, CUtensorMapDataType type, int rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides,
               const cuuint32_t* box) {
    EncodeTiled encode = encode_tiled();
    MRUN_REQUIRE(encode != nullptr, "gemm_f32_tc: the driver does not offer cuTensorMapEncodeTiled");
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult rc = encode(map, type, rank, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    MRUN_REQUIRE(rc == CUDA_SUCCESS, "gemm_f32_tc: cuTensorMapEncodeTiled failed with code %d", (int)rc);
    return 0;
}

template <int TOK>
void configure(cudaLaunchConfig_t* config, cudaLaunchAttribute* attributes, dim3 grid, cudaStream_t stream) {
    *config = cudaLaunchConfig_t{};
    config->gridDim = grid;
    config->blockDim = dim3(Shape<TOK>::THREADS);
    config->dynamicSmemBytes = Shape<TOK>::SMEM;
    config->stream = stream;
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = grid.x;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[1].val.programmaticStreamSerializationAllowed = 1;
    config->attrs = attributes;
    config->numAttrs = 2;
}

int registers_of(const void* kernel) {
    cudaFuncAttributes has;
    return cudaFuncGetAttributes(&has, kernel) == cudaSuccess ? has.numRegs : -1;
}

template <int TOK>
int launch(const CUtensorMap& map_w, const void* parts, int pitch, const ProductArgs& a, int cluster, cudaStream_t stream) {
    CUtensorMap map_x;
    const cuuint64_t dims[3] = {(cuuint64_t)a.K, (cuuint64_t)a.M, PARTS};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)a.M * pitch * 2};
    const cuuint32_t box[3] = {BK, TOK, PARTS};
    if (int rc = encode_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, parts, dims, strides, box)) return rc;
    const dim3 grid(cluster, (a.M + TOK - 1) / TOK, (a.N + ROWS - 1) / ROWS);
    MRUN_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "gemm_f32_tc: M=%d N=%d exceed the grid", a.M, a.N);
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(gemm_f32_tc_kernel<TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<TOK>::SMEM),
                    "gemm_f32_tc");
    if constexpr (Shape<TOK>::UNEVEN) {
        static const int registers = registers_of((const void*)gemm_f32_tc_kernel<TOK>);
        MRUN_REQUIRE(registers == Shape<TOK>::LAUNCH_REGISTERS, "gemm_f32_tc: tiles of %d tokens were built with %d registers a thread, %d are dealt out",
                     TOK, registers, Shape<TOK>::LAUNCH_REGISTERS);
    }
    cudaLaunchConfig_t config;
    cudaLaunchAttribute attributes[2];
    configure<TOK>(&config, attributes, grid, stream);
    MRUN_CHECK_CUDA(cudaLaunchKernelEx(&config, gemm_f32_tc_kernel<TOK>, map_w, map_x, a), "gemm_f32_tc");
    return 0;
}

constexpr int MULTIPROCESSORS = 148;      // of a B200: the ranges, and with them a result's bits, are the same everywhere
constexpr int TILES[] = {16, 32, 64, 96, 112, 128, 144, 160, 176, 192};

// Ranges of k for N rows of w: as many, by doubling, as give each multiprocessor a block in a product of few rows.
// Four rows, us with 1 / 2 / 4 / 8 ranges: N = 4,096, K = 4,096 51 / 30 / 20 / 20, K = 12,288 141 / 75 / 44 / 39; N = 6,144
// 50 / 30 / 26 / 31; N = 24,576 79 / 81 / 80 / 93.
int ranges_of(int N, int K) {
    const long tiles = (N + ROWS - 1) / ROWS;
    const int blocks = (K + BK - 1) / BK;
    int ranges = 1;
    while (ranges < MAX_SPLIT && tiles * ranges < MULTIPROCESSORS && blocks / (2 * ranges) >= 4) ranges *= 2;
    return ranges;
}

// What a product takes in tiles of `tile` tokens, in blocks of 64 k of a tile of one token: rounds of tiles over the
// multiprocessors (clusters fill fewer of them), each with a start and an end.
float cost_of(int tile, int cluster, int M, int N, const ProductArgs& a) {
    const long tiles = (long)((M + tile - 1) / tile) * ((N + ROWS - 1) / ROWS);
    const long room = cluster == 1 ? MULTIPROCESSORS : cluster == 2 ? MULTIPROCESSORS / 2 : 136 / cluster;
    const long rounds = (tiles + room - 1) / room;
    // a block of k takes 0.35 + 0.0075 us a token, the start and the end of a tile 4 us and 2 us more in a cluster
    return (float)rounds * ((0.35f + 0.0075f * (float)tile) * (float)((a.blocks + cluster - 1) / cluster) + (cluster == 1 ? 4.f : 6.f));
}

}  // namespace

// parts: scratch of 3 * M * pitch bfloat16 values, pitch = K rounded up to 8.  0 stands for chosen: ranges (of k), tile (of tokens),
// cluster (1, or as many blocks as there are ranges).
MRUN_API int mrun_gemm_f32_tc(const float* x, const float* w, float* y, void* parts, int M, int N, int K, long ldx, long ldy, int ranges,
                              int tile, int cluster, int* status, cudaStream_t stream) {
    MRUN_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_tc: bad sizes M=%d N=%d K=%d", M, N, K);
    MRUN_REQUIRE(ldx >= K && ldy >= N, "gemm_f32_tc: row strides ldx=%ld ldy=%ld below K=%d N=%d", ldx, ldy, K, N);
    MRUN_REQUIRE((((uintptr_t)w | (uintptr_t)parts) & 15) == 0, "gemm_f32_tc: w and the scratch must be 16-byte aligned");
    MRUN_REQUIRE(status != nullptr, "gemm_f32_tc: a status word is required");
    if (M == 0) return 0;
    if (ranges == 0) ranges = ranges_of(N, K);
    ProductArgs a = {x, w, y, ldx, ldy, M, N, K, (K + BK - 1) / BK, ranges, status};
    MRUN_REQUIRE(ranges >= 1 && ranges <= MAX_SPLIT && ranges <= a.blocks, "gemm_f32_tc: %d ranges of %d blocks of k", ranges, a.blocks);
    MRUN_REQUIRE(cluster == 0 || cluster == ranges || (cluster == 1 && (tile == 0 || tile > 32)),
                 "gemm_f32_tc: a cluster of %d for %d ranges", cluster, ranges);
    const int pitch = (K + 7) / 8 * 8;
    const bool aligned = ((uintptr_t)x & 15) == 0 && (ldx % 4 == 0 || M == 1);
    // Up to 32 rows: w's bytes count, and two blocks on a multiprocessor read it in all the ranges at once.  (A block of the
    // small tiles has one range: only the larger ones take several one after the other.)
    if (tile == 0 && M <= 32 && (cluster == 0 || cluster == ranges)) {
        tile = M <= 16 ? 16 : 32;
        cluster = ranges;
    } else if (tile == 0 || cluster == 0) {
        const int asked_tile = tile, asked_cluster = cluster;
        float least = 0.f;
        for (int t : TILES) {
            if (asked_tile ? t != asked_tile : t <= 32) continue;
            for (int c : {ranges, 1}) {
                if ((asked_cluster && c != asked_cluster) || (t <= 32 && c != ranges)) continue;
                const float cost = cost_of(t, c, M, N, a);
                if (least == 0.f || cost < least) { least = cost; tile = t; cluster = c; }
            }
        }
    }
    const long quads = (long)M * (K / 4), blocks = (quads + SPLIT_THREADS - 1) / SPLIT_THREADS;
    MRUN_REQUIRE(blocks <= 0x7fffffffL, "gemm_f32_tc: M=%d K=%d exceed the grid", M, K);
    auto kernel = aligned ? split_rows_kernel<true> : split_rows_kernel<false>;
    MRUN_CHECK_CUDA(mrun::launch_kernel_overlapped(kernel, dim3((unsigned)blocks), dim3(SPLIT_THREADS), 0, stream, x, ldx, (bf16*)parts,
                                                   (long)M * pitch, pitch, quads, K / 4), "gemm_f32_tc");
    CUtensorMap map_w;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {HALF, ROWS};
    if (int rc = encode_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, w, dims, strides, box)) return rc;
    switch (tile) {
#define MRUN_TILE(T) case T: return launch<T>(map_w, parts, pitch, a, cluster, stream)
        MRUN_TILE(16); MRUN_TILE(32); MRUN_TILE(64); MRUN_TILE(96); MRUN_TILE(112); MRUN_TILE(128); MRUN_TILE(144); MRUN_TILE(160);
        MRUN_TILE(176); MRUN_TILE(192);
#undef MRUN_TILE
    }
    return mrun_set_error("gemm_f32_tc: no tile of %d tokens", tile);
}
