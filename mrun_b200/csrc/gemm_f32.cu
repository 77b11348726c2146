// True 32-bit linear layer: y[M, N] = x[M, K] · w[N, K]^T (+ nothing), IEEE fp32 fused
// multiply-adds, no tensor cores, no TF32.
//
// Every output element is the sum over k = 0 .. K-1 in that order, in one chain of fused multiply-adds,
// whatever M is, wherever the row sits in the batch and whichever of the kernels below runs, so a
// token's result is bit-identical under every way of cutting the work.
// Weights of 64 rows and more with a multiple of 4 and at least 2,048 k that start on 16 bytes go to gemm_f32_tc.cu (kernels/ops.py, f32_tc_ok).
// Reference call site: crates/mrun-engine/src/load.rs:294-306 (`x · Wᵀ`, weights [out, in]).
//
//   stream  up to 16 rows whose operands lie on 16-byte boundaries: bound by reading w once, and by the
//           chain itself (four cycles a k, and the waits of its stages).  A lane takes one row of w and MT
//           rows of x; both come through a ring of asynchronous 16-byte copies.  K = 4,096: one row, N =
//           4,096 23 us (64 x 64 tiles: 323), N = 24,576 75 us (509), 5.4 TB/s; four rows, N = 24,576 95 us (513).
//   tile    everything else: bound by the FMA pipe and by the shared-memory reads that feed it, which take as
//           long.  BM x BN outputs a block, TM x TN a thread as pairs of columns (packed fused multiply-adds,
//           two a lane and instruction, which leaves issue slots for the loads), k slices of 16 brought
//           k-major by asynchronous 4-byte copies, so no operand needs an alignment of its own.  517 rows, K =
//           4,096: N = 24,576 2,241 us (64 x 64 tiles of one slice at a time: 3,676), 46 TFLOP/s of 74; N = 6,144
//           594 us (1,132).  Thread tiles of 8 x 16, which read less, leave too few warps: 2,865 us.
#include "common.cuh"

namespace {

// `bytes` = 0 writes zeros and reads nothing.
__device__ __forceinline__ void copy_16_or_zero(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copy_4_or_zero(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------ stream
constexpr int STREAM_ROWS = 16;      // rows of x at most
constexpr int STREAM_K = 128;        // k of a stage: a warp's lanes bring one row's 512 bytes with one instruction
constexpr int STREAM_PITCH = STREAM_K + 4;      // eight lanes' 16-byte reads of eight rows meet no bank twice
constexpr int STREAM_STAGES = 6;
constexpr int STREAM_WARPS = 4;

// COLS rows of w a block (32 or 16), a lane one of them; MT rows of x a lane.
template <int MT, int COLS>
__global__ void __launch_bounds__(STREAM_WARPS * 32)
gemm_f32_stream_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, long ldx,
                       long ldy, long batch_x, long batch_w, long batch_y) {
    constexpr int W_EACH = COLS / STREAM_WARPS, X_EACH = STREAM_ROWS / STREAM_WARPS;     // rows of w and of x a warp brings
    constexpr int QUADS = 4;                              // 16-byte pieces of k held in registers ahead of the arithmetic
    extern __shared__ __align__(16) float smem[];
    x += blockIdx.z * batch_x;
    w += blockIdx.z * batch_w;
    y += blockIdx.z * batch_y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col0 = blockIdx.x * COLS, col = col0 + lane % COLS;
    const int row0 = (warp * (32 / COLS) + lane / COLS) * MT;
    const bool walks = warp * (32 / COLS) * MT < M;       // whether the warp has rows
    const int stage_floats = (COLS + M) * STREAM_PITCH;
    const int steps = (K + STREAM_K - 1) / STREAM_K;

    const float* w_src[W_EACH];
#pragma unroll
    for (int i = 0; i < W_EACH; ++i) w_src[i] = w + (size_t)min(col0 + warp * W_EACH + i, N - 1) * K + lane * 4;
    const float* x_src = x + (size_t)min(warp, M - 1) * ldx + lane * 4;
    auto fetch = [&](int step) {
        float* dst = smem + (step % STREAM_STAGES) * stage_floats + lane * 4;
        const int k0 = step * STREAM_K;
        const int bytes = k0 + lane * 4 < K ? 16 : 0;     // K is a multiple of 4
        const int at = bytes ? k0 : -lane * 4;            // a row's start where nothing is read
#pragma unroll
        for (int i = 0; i < W_EACH; ++i) copy_16_or_zero(dst + (warp * W_EACH + i) * STREAM_PITCH, w_src[i] + at, bytes);
#pragma unroll
        for (int i = 0; i < X_EACH; ++i)
            if (warp + STREAM_WARPS * i < M)
                copy_16_or_zero(dst + (COLS + warp + STREAM_WARPS * i) * STREAM_PITCH, x_src + i * STREAM_WARPS * ldx + at, bytes);
    };
#pragma unroll
    for (int s = 0; s < STREAM_STAGES - 1; ++s) {
        if (s < steps) fetch(s);
        copies_commit();
    }
    float acc[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[i] = 0.f;
    const float* rows[MT];                                // rows beyond the last read the last and are not written
#pragma unroll
    for (int i = 0; i < MT; ++i) rows[i] = smem + (COLS + min(row0 + i, M - 1)) * STREAM_PITCH;
    const float* ws = smem + (lane % COLS) * STREAM_PITCH;
    for (int step = 0; step < steps; ++step) {
        copies_wait<STREAM_STAGES - 2>();
        __syncthreads();                                  // this stage is here, and the one before has been read
        const int base = (step % STREAM_STAGES) * stage_floats;
        float4 b[2][QUADS], a[2][QUADS][MT];
        auto load = [&](int half, int k) {
#pragma unroll
            for (int q = 0; q < QUADS; ++q) {
                b[half][q] = *reinterpret_cast<const float4*>(ws + base + k + 4 * q);
#pragma unroll
                for (int i = 0; i < MT; ++i) a[half][q][i] = *reinterpret_cast<const float4*>(rows[i] + base + k + 4 * q);
            }
        };
        if (walks) load(0, 0);                            // under way while the next copies are asked for
        if (step + STREAM_STAGES - 1 < steps) fetch(step + STREAM_STAGES - 1);
        copies_commit();
        if (!walks) continue;
#pragma unroll
        for (int k = 0; k < STREAM_K; k += 4 * QUADS) {
            const int half = (k / (4 * QUADS)) & 1;
            if (k + 4 * QUADS < STREAM_K) load(half ^ 1, k + 4 * QUADS);
#pragma unroll
            for (int q = 0; q < QUADS; ++q) {
                const float4 bb = b[half][q];
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(a[half][q][i].x, bb.x, acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(a[half][q][i].y, bb.y, acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(a[half][q][i].z, bb.z, acc[i]);
#pragma unroll
                for (int i = 0; i < MT; ++i) acc[i] = fmaf(a[half][q][i].w, bb.w, acc[i]);
            }
        }
    }
    if (col < N) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
            if (row0 + i < M) y[(size_t)(row0 + i) * ldy + col] = acc[i];
    }
}

// ------------------------------------------------------------------------------------------ tile
constexpr int TILE_K = 16;
constexpr int TILE_STAGES = 4;

template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), 3)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, long ldx,
                     long ldy, long batch_x, long batch_w, long batch_y) {
    constexpr int THREADS = (BM / TM) * (BN / TN), WARPS_X = BN / TN / 8;
    // k slices 4 banks apart; from the ninth on the pairs of each run of four stand swapped, so that the
    // copies of a warp (sixteen k of two rows) meet no bank twice
    constexpr int PM = BM + 4, PN = BN + 4;
    constexpr int STAGE = TILE_K * (PM + PN);
    constexpr int RC = TM / 4, CC = TN / 4;               // a thread's rows and columns come in runs of four
    extern __shared__ __align__(16) float smem[];
    x += blockIdx.z * batch_x;
    w += blockIdx.z * batch_w;
    y += blockIdx.z * batch_y;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a warp is 4 x 8 threads: its reads of a row run are 64 bytes, of a column run 128
    const int ty = (warp / WARPS_X) * 4 + lane / 8, tx = (warp % WARPS_X) * 8 + lane % 8;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int steps = (K + TILE_K - 1) / TILE_K;

    // copies: a thread keeps its k within the slice and walks over rows
    constexpr int PER = THREADS / TILE_K;
    const int ck = tid % TILE_K, row_of = tid / TILE_K, place = row_of ^ (ck & 8 ? 2 : 0);
    // The FMAs share their issue slots with this arithmetic: a thread's rows by an addition each from its first, held on
    // the last row there is, instead of a clamped index times the pitch (517 rows, K = 4,096, N = 24,576, B200:
    // 2,306 -> 2,241 us; 100 rows, K = 12,288: 464 -> 433).
    const float* x_first = x + (size_t)min(row0 + row_of, M - 1) * ldx;
    const float* w_first = w + (size_t)min(col0 + row_of, N - 1) * K;
    const long x_step = (long)PER * ldx, w_step = (long)PER * K;
    const int x_rows = M - row0 - row_of, w_rows = N - col0 - row_of;      // of this thread's rows on
    auto fetch = [&](int step) {
        float* as = smem + (step % TILE_STAGES) * STAGE + ck * PM + place;
        float* bs = smem + (step % TILE_STAGES) * STAGE + TILE_K * PM + ck * PN + place;
        const int k = step * TILE_K + ck;
        const int bytes = k < K ? 4 : 0, at = k < K ? k : 0;
        const float *x_at = x_first + at, *w_at = w_first + at;
#pragma unroll
        for (int r = 0; r < BM; r += PER) {
            copy_4_or_zero(as + r, x_at, bytes);
            x_at += r + PER < x_rows ? x_step : 0;
        }
#pragma unroll
        for (int r = 0; r < BN; r += PER) {
            copy_4_or_zero(bs + r, w_at, bytes);
            w_at += r + PER < w_rows ? w_step : 0;
        }
    };
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; ++s) {
        if (s < steps) fetch(s);
        copies_commit();
    }
    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.f, 0.f);

    for (int step = 0; step < steps; ++step) {
        copies_wait<TILE_STAGES - 2>();
        __syncthreads();                                  // this slice is here, and the one before has been read
        if (step + TILE_STAGES - 1 < steps) fetch(step + TILE_STAGES - 1);
        copies_commit();
        const float* as = smem + (step % TILE_STAGES) * STAGE + ty * 4;
        const float* bs = smem + (step % TILE_STAGES) * STAGE + TILE_K * PM + tx * 4;
#pragma unroll
        for (int k = 0; k < TILE_K; ++k) {
            float a[TM];
            float2 b[TN / 2];
#pragma unroll
            for (int c = 0; c < RC; ++c)
                *reinterpret_cast<float4*>(a + 4 * c) = *reinterpret_cast<const float4*>(as + k * PM + c * (BM / RC));
#pragma unroll
            for (int c = 0; c < CC; ++c)
                *reinterpret_cast<float4*>(b + 2 * c) = *reinterpret_cast<const float4*>(bs + k * PN + c * (BN / CC));
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float v = a[k & 8 ? i ^ 2 : i];
                const float2 aa = make_float2(v, v);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = __ffma2_rn(aa, b[k & 8 ? j ^ 1 : j], acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int row = row0 + (i / 4) * (BM / RC) + ty * 4 + i % 4;
        if (row >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) {
            const int col = col0 + (j / 2) * (BN / CC) + tx * 4 + (j % 2) * 2;
            if (col < N) y[(size_t)row * ldy + col] = acc[i][j].x;
            if (col + 1 < N) y[(size_t)row * ldy + col + 1] = acc[i][j].y;
        }
    }
}

template <int BM, int BN, int TM, int TN>
int launch_tile(const float* x, const float* w, float* y, int batch, int M, int N, int K, long ldx, long ldy, long batch_x, long batch_w,
                long batch_y, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    MRUN_REQUIRE(grid.y <= 65535, "gemm_f32_nt: M=%d exceeds the supported %d rows", M, 65535 * BM);
    constexpr int bytes = TILE_STAGES * TILE_K * (BM + 4 + BN + 4) * (int)sizeof(float);
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(gemm_f32_tile_kernel<BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
                    "gemm_f32_nt");
    gemm_f32_tile_kernel<BM, BN, TM, TN><<<grid, (BM / TM) * (BN / TN), bytes, stream>>>(x, w, y, M, N, K, ldx, ldy, batch_x, batch_w,
                                                                                        batch_y);
    return 0;
}

template <int MT, int COLS>
int launch_stream(const float* x, const float* w, float* y, int batch, int M, int N, int K, long ldx, long ldy, long batch_x, long batch_w,
                  long batch_y, cudaStream_t stream) {
    const int bytes = STREAM_STAGES * (COLS + M) * STREAM_PITCH * (int)sizeof(float);
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(gemm_f32_stream_kernel<MT, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
                    "gemm_f32_nt");
    const dim3 grid((N + COLS - 1) / COLS, 1, batch);
    gemm_f32_stream_kernel<MT, COLS><<<grid, 32 * STREAM_WARPS, bytes, stream>>>(x, w, y, M, N, K, ldx, ldy, batch_x, batch_w, batch_y);
    return 0;
}

// What a launch of BM x BN tiles takes, in microseconds for K = 4,096 (measured on B200; all forms grow with K
// alike): a multiprocessor's tiles one after the other at `each`, and at least `alone`, what a tile takes
// that has the multiprocessor to itself.
struct TileCost { int bm, bn; float each, alone; };
constexpr TileCost TILE_COSTS[] = {{64, 128, 205.f, 250.f}, {64, 64, 120.f, 165.f}, {32, 32, 45.f, 88.f}};

int multiprocessors() {
    int device = 0, count = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
        return 148;
    return count;
}

int launch_product(const float* x, const float* w, float* y, int batch, int M, int N, int K, long ldx, long ldy, long batch_x,
                   long batch_w, long batch_y, cudaStream_t stream) {
    const bool aligned = ((((uintptr_t)x) | ((uintptr_t)w)) & 15) == 0 && K % 4 == 0 && (ldx % 4 == 0 || M == 1) && batch_x % 4 == 0 &&
                         batch_w % 4 == 0;
#define MRUN_PRODUCT(LAUNCH) return LAUNCH(x, w, y, batch, M, N, K, ldx, ldy, batch_x, batch_w, batch_y, stream)
    if (aligned && M <= STREAM_ROWS) {
        // Many blocks (wide): shared memory's bandwidth counts, so a lane takes as many rows as there are.
        // Few: a block's own time counts, so the rows are spread over its warps.  M = 4, K = 4,096, us a
        // product with 1 / 2 / 4 rows a lane: N = 4,096 26.0 / 23.5 / 29.6, N = 24,576 122 / 105 / 95.  Sixteen
        // columns a block give M = 8 at N = 24,576 123 where thirty-two give 155.
        const bool wide = (long)N * batch >= 16384;
        if (M <= 2) MRUN_PRODUCT((launch_stream<1, 32>));
        if (M <= 4 && !wide) MRUN_PRODUCT((launch_stream<2, 32>));
        if (M > 4 && M <= 8 && wide) MRUN_PRODUCT((launch_stream<4, 16>));
        MRUN_PRODUCT((launch_stream<4, 32>));
    }
    const int sms = multiprocessors();
    int best = 0;
    float least = 0.f;
    for (int i = 0; i < 3; ++i) {
        const TileCost& c = TILE_COSTS[i];
        if (i > 0 && (M + c.bm - 1) / c.bm > 65535) continue;         // more rows of tiles than a grid has
        const long tiles = (long)((M + c.bm - 1) / c.bm) * ((N + c.bn - 1) / c.bn) * batch;
        const float cost = fmaxf(c.alone, c.each * (float)((tiles + sms - 1) / sms));
        if (i == 0 || cost < least) { best = i; least = cost; }
    }
    if (best == 0) MRUN_PRODUCT((launch_tile<64, 128, 8, 8>));
    if (best == 1) MRUN_PRODUCT((launch_tile<64, 64, 8, 4>));
    MRUN_PRODUCT((launch_tile<32, 32, 4, 4>));
#undef MRUN_PRODUCT
}

}  // namespace

// x rows are ldx floats apart, y rows ldy floats apart; w is dense [N, K].
MRUN_API int mrun_gemm_f32_nt(const float* x, const float* w, float* y, int M, int N, int K, long ldx,
                              long ldy, cudaStream_t stream) {
    MRUN_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32_nt: bad sizes M=%d N=%d K=%d", M, N, K);
    MRUN_REQUIRE(ldx >= K && ldy >= N, "gemm_f32_nt: row strides ldx=%ld ldy=%ld below K=%d N=%d", ldx, ldy,
                 K, N);
    if (M == 0) return 0;
    if (const int failed = launch_product(x, w, y, 1, M, N, K, ldx, ldy, 0, 0, 0, stream)) return failed;
    MRUN_CHECK_LAUNCH("gemm_f32_nt");
    return 0;
}

// The same product for `batch` independent problems (the heads of a per-head projection): problem b
// reads x + b * batch_x (rows ldx apart) and the dense w + b * batch_w [N, K], and writes
// y + b * batch_y (rows ldy apart).  The sum over k keeps its fixed order.
MRUN_API int mrun_gemm_f32_nt_batched(const float* x, const float* w, float* y, int batch, int M, int N, int K,
                                      long ldx, long ldy, long batch_x, long batch_w, long batch_y,
                                      cudaStream_t stream) {
    MRUN_REQUIRE(batch > 0 && batch <= 65535 && M >= 0 && N > 0 && K > 0,
                 "gemm_f32_nt_batched: bad sizes batch=%d M=%d N=%d K=%d", batch, M, N, K);
    MRUN_REQUIRE(ldx >= K && ldy >= N, "gemm_f32_nt_batched: row strides ldx=%ld ldy=%ld below K=%d N=%d", ldx,
                 ldy, K, N);
    if (M == 0) return 0;
    if (const int failed = launch_product(x, w, y, batch, M, N, K, ldx, ldy, batch_x, batch_w, batch_y, stream)) return failed;
    MRUN_CHECK_LAUNCH("gemm_f32_nt_batched");
    return 0;
}
