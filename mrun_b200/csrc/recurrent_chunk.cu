// The scans of long segments in chunks of CHUNK tokens (see recurrent.cu for the formulas), for bfloat16
// inputs and key and value sizes of 64 and 128.  All arithmetic is 32-bit on the FMA pipe.
//
// With the tokens of a chunk numbered from 0, the state S at its start, and G(i, j) the product of the
// decays of tokens i + 1 .. j, channel by channel:
//     o_i  = (q_i G(-1, i)) S + sum over j <= i of (q_i . G(j, i) k_j) v_j
//     S'   = G(-1, last) S + sum over j of (G(j, last) k_j) v_j^T
// so a segment is a chain over its chunks, not over its tokens, and everything but one multiply-add a
// chunk and state element is a matrix product:
//   prepare  (a block a chunk and head) the read vectors q_i G(-1, i), the weights q_i . G(j, i) k_j and
//            the chunk's own share of S'
//   carry    (a thread four state elements of a head) walks over a segment's chunks, leaves each the state
//            at its start and the request the state at the end
//   finish   (a block a chunk and head) o as one product: [read vectors | weights] times [state; values]
// Products of decays that differ are formed by multiplication inside runs of SUB tokens and from run to run, never as
// a quotient or a difference of logarithms: none overflows, and what underflows is as small as it says.
// Pairs of tokens within a run multiply their decays one after the other as the walk does.
//
// Bound by the FMA pipe, the shared-memory reads that feed it (thread tiles of 8 x 8) and, in prepare, by the
// exponentials.  2,048 tokens, 16 heads of 128 x 128, walked / in chunks, us: decay 521 / 118 (prepare 64, carry
// 13, finish 41), gated 561 / 133; 32 heads 621 / 229 and 677 / 258 (prepare 145, carry 53, finish 60: its 117
// MB of scratch leave the L2 cache).  finish leaves out the values that come after a row's token, runs of them as a whole
// (decay 44 -> 41, delta 36 -> 34).
#include "common.cuh"

using namespace mrun;

namespace {

constexpr int CHUNK = 64, SUB = 16, SUBS = CHUNK / SUB;
constexpr int THREADS = 256;
typedef __nv_bfloat16 bf16;

enum : int { CHUNK_DECAY = 0, CHUNK_GATED = 1, CHUNK_DELTA = 2 };

struct ChunkArgs {
    const void *q, *k, *v;           // bfloat16, row t at + t * ld: [H, D], [H, D], [H, V]
    long ld;
    const float* a;                  // gated, delta: [tokens, H * D], the decay projection's output
    const float* bias;               // gated, delta: [H * D]
    const float* decay;              // decay: [H]
    const float* a_log;              // delta: [H]
    const bf16* b;                   // delta: [H], row t at + t * ldb
    long ldb;
    int group;                       // delta: heads that share a q and a k
    float tau;
    int silu_inputs;
    float* state;                    // [slots, H, D, V]
    float* out;                      // [tokens, H * V]
    float* scratch;
    const int *seg_q_start, *seg_slot;
    int segments, chunks, H, D, V;   // chunks: at least as many as the segments have
};

__device__ __forceinline__ float softplus_f(float x) { return x > 20.f ? x : log1pf(expf(x)); }
__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 widen4(uint2 raw) {
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 silu4(float4 v) { return make_float4(silu(v.x), silu(v.y), silu(v.z), silu(v.w)); }
__device__ __forceinline__ void copy_async_16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Scratch of one (chunk, head) in a decay or gated scan, in floats: [D + CHUNK][CHUNK] read vectors and weights, both with the token
// last; [D][V] the chunk's share of the state, then the state at its start; [D] the chunk's whole decay.
__host__ __device__ constexpr long left_floats(int D) { return (long)(D + CHUNK) * CHUNK; }
__host__ __device__ constexpr long unit_floats(int D, int V) { return left_floats(D) + (long)D * V + D; }
// In a delta scan three more follow: [D][CHUNK] what the state at the chunk's start takes from the tokens' writes,
// [CHUNK][D] k with the decays up to the chunk's end, [CHUNK][V] the tokens' writes without and then with the state.
__host__ __device__ constexpr long delta_floats(int D, int V) { return unit_floats(D, V) + (long)CHUNK * (2 * D + V); }
template <int MODE> __host__ __device__ constexpr long unit_of(int D, int V) { return MODE == CHUNK_DELTA ? delta_floats(D, V) : unit_floats(D, V); }

// The segment a chunk belongs to: its first row in the batch and its tokens (0: beyond the last chunk).  All
// lanes of a warp ask together: a lane counts one segment's chunks.
struct ChunkPlace { int row, tokens; };
__device__ __forceinline__ ChunkPlace place_of(const ChunkArgs& w, int chunk) {
    const int lane = threadIdx.x & 31;
    for (int base = 0, before = 0; base < w.segments; base += 32) {
        const int s = base + lane;
        const int q0 = s < w.segments ? w.seg_q_start[s] : 0, n = s < w.segments ? w.seg_q_start[s + 1] - q0 : 0;
        const int mine = (n + CHUNK - 1) / CHUNK;
        int upto = mine;                  // chunks of the segments up to this one
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += other;
        }
        const unsigned past = __ballot_sync(0xffffffffu, before + upto > chunk);
        if (past) {
            const int from = __ffs(past) - 1;
            const int t = (chunk - before - __shfl_sync(0xffffffffu, upto - mine, from)) * CHUNK;
            return {__shfl_sync(0xffffffffu, q0, from) + t, min(CHUNK, __shfl_sync(0xffffffffu, n, from) - t)};
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return {0, 0};
}

// 8 x 8 outputs a thread, one k: rows a[0..3], a[BM/2 ..], columns likewise.
template <int BM, int BN>
__device__ __forceinline__ void outer8(const float* as, const float* bs, float2 (&acc)[8][4]) {
    float a[8];
    float2 b[4];
    *reinterpret_cast<float4*>(a) = load4(as);
    *reinterpret_cast<float4*>(a + 4) = load4(as + BM / 2);
    *reinterpret_cast<float4*>(b) = load4(bs);
    *reinterpret_cast<float4*>(b + 2) = load4(bs + BN / 2);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float2 aa = make_float2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __ffma2_rn(aa, b[j], acc[i][j]);
    }
}
__device__ __forceinline__ void clear8(float2 (&acc)[8][4]) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
}

template <int D, int V> constexpr int third_floats() { return CHUNK * (D + 4 > V ? D + 4 : V); }     // decays, then values
template <int D, int V> constexpr int prepare_smem() { return (2 * CHUNK * (D + 4) + third_floats<D, V>() + SUBS * D) * (int)sizeof(float); }

template <int MODE, int D, int V>
__global__ void __launch_bounds__(THREADS)
chunk_prepare_kernel(const ChunkArgs w) {
    constexpr int P = D + 4;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                     // [CHUNK][P]
    float* ks = qs + CHUNK * P;
    float* gs = ks + CHUNK * P;           // the decays, then the values ([CHUNK][V])
    float* es = gs + third_floats<D, V>();           // [SUBS][D] a run's whole decay
    __shared__ float powers[CHUNK + 1];   // of a head's one decay
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = blockIdx.x, h = blockIdx.y;
    const ChunkPlace at = place_of(w, chunk);
    const int n = at.tokens;
    if (n == 0) return;
    float* left = w.scratch + ((long)chunk * w.H + h) * unit_floats(D, V);
    float* share = left + left_floats(D);
    float* whole = share + (long)D * V;

    // Rows of q, k and the decays, four features a thread and row, and this thread's pieces of the values, kept until
    // the decays' place is free: everything is asked for before anything is looked at.  Tokens that are not there
    // decay nothing and bring nothing.
    constexpr int LANES = D / 4, ROWS = THREADS / LANES, PASSES = CHUNK / ROWS, PIECES = CHUNK * V / 4 / THREADS;
    const int d0 = (tid % LANES) * 4, r0 = tid / LANES;
    uint2 rq[PASSES], rk[PASSES], values[PIECES];
    float4 ra[MODE == CHUNK_GATED ? PASSES : 1], bias = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
        const long row = at.row + min(r0 + p * ROWS, n - 1);
        rq[p] = *reinterpret_cast<const uint2*>((const bf16*)w.q + row * w.ld + (long)h * D + d0);
        rk[p] = *reinterpret_cast<const uint2*>((const bf16*)w.k + row * w.ld + (long)h * D + d0);
        if constexpr (MODE == CHUNK_GATED) ra[p] = load4(w.a + (row * w.H + h) * D + d0);
    }
    if constexpr (MODE == CHUNK_GATED) bias = load4(w.bias + (long)h * D + d0);
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int e = tid + i * THREADS, r = e / (V / 4), c = e % (V / 4) * 4;
        values[i] = *reinterpret_cast<const uint2*>((const bf16*)w.v + (long)(at.row + min(r, n - 1)) * w.ld + (long)h * V + c);
        if (r >= n) values[i] = make_uint2(0, 0);
    }
#pragma unroll
    for (int p = 0; p < PASSES; ++p) {
        const int r = r0 + p * ROWS;
        float4 q = widen4(rq[p]), k = widen4(rk[p]), g = make_float4(1.f, 1.f, 1.f, 1.f);
        if constexpr (MODE == CHUNK_GATED) {
            const float4 a = ra[p];
            const float size = 1.f / sqrtf((float)D);
            q = make_float4(q.x * size, q.y * size, q.z * size, q.w * size);
            if (r < n)
                g = make_float4(expf(-softplus_f(-(a.x + bias.x)) / w.tau), expf(-softplus_f(-(a.y + bias.y)) / w.tau),
                                expf(-softplus_f(-(a.z + bias.z)) / w.tau), expf(-softplus_f(-(a.w + bias.w)) / w.tau));
        } else if (w.silu_inputs) {
            q = silu4(q);
            k = silu4(k);
        }
        if (r >= n) q = k = make_float4(0.f, 0.f, 0.f, 0.f);
        store4(qs + r * P + d0, q);
        store4(ks + r * P + d0, k);
        if constexpr (MODE == CHUNK_GATED) store4(gs + r * P + d0, g);
    }
    // The powers of one decay, each rounded once: a power multiplied up in 32 bits would be off the same way in
    // every chunk.
    if (MODE == CHUNK_DECAY && tid <= CHUNK) {
        double f = 1.0, base = (double)w.decay[h];
        for (int e = tid; e; e >>= 1, base *= base)
            if (e & 1) f *= base;
        powers[tid] = (float)f;
    }
    __syncthreads();

    if constexpr (MODE == CHUNK_GATED) {
        // Weights of token pairs within a run: two warps a run, eight lanes a pair of tokens j (a lane every
        // eighth group of four features), the decays multiplied on from token to token.
        {
            const int sub = warp >> 1, slice = lane & 7, j0 = (warp & 1) * 8 + (lane >> 3) * 2;
            const float* q0 = qs + sub * SUB * P + slice * 4;
            const float* g0 = gs + sub * SUB * P + slice * 4;
            const float* k0 = ks + (sub * SUB + j0) * P + slice * 4;
            float4 x[D / 32], y[D / 32];      // k of tokens j0 and j0 + 1, decayed up to token i
#pragma unroll
            for (int m = 0; m < D / 32; ++m) { x[m] = load4(k0 + 32 * m); y[m] = load4(k0 + P + 32 * m); }
            float* dst = left + (long)(D + sub * SUB + j0) * CHUNK + sub * SUB;
            for (int i = (warp & 1) * 8; i < SUB; ++i) {
                float sx = 0.f, sy = 0.f;
#pragma unroll
                for (int m = 0; m < D / 32; ++m) {
                    const float4 q = load4(q0 + i * P + 32 * m), g = load4(g0 + i * P + 32 * m);
                    if (i > j0) { x[m].x *= g.x; x[m].y *= g.y; x[m].z *= g.z; x[m].w *= g.w; }
                    if (i > j0 + 1) { y[m].x *= g.x; y[m].y *= g.y; y[m].z *= g.z; y[m].w *= g.w; }
                    sx = fmaf(q.x, x[m].x, sx); sx = fmaf(q.y, x[m].y, sx); sx = fmaf(q.z, x[m].z, sx); sx = fmaf(q.w, x[m].w, sx);
                    sy = fmaf(q.x, y[m].x, sy); sy = fmaf(q.y, y[m].y, sy); sy = fmaf(q.z, y[m].z, sy); sy = fmaf(q.w, y[m].w, sy);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) {
                    sx += __shfl_xor_sync(0xffffffffu, sx, o);
                    sy += __shfl_xor_sync(0xffffffffu, sy, o);
                }
                if (slice == 0) {
                    dst[i] = i >= j0 ? sx : 0.f;
                    dst[CHUNK + i] = i > j0 ? sy : 0.f;
                }
            }
            // the second warp's tokens do not see the run's first half
            if (warp & 1)
                for (int e = lane; e < 64; e += 32) left[(long)(D + sub * SUB + 8 + e / 8) * CHUNK + sub * SUB + e % 8] = 0.f;
        }
        __syncthreads();
        // q and k with the decays of their own run: q from the run's start, k up to its end
        for (int e = tid; e < SUBS * D; e += THREADS) {
            const int sub = e / D, d = e % D;
            float* q = qs + sub * SUB * P + d;
            float* k = ks + sub * SUB * P + d;
            const float* g = gs + sub * SUB * P + d;
            float f = 1.f;
#pragma unroll
            for (int i = 0; i < SUB; ++i) { f *= g[i * P]; q[i * P] *= f; }
            es[e] = f;
            f = 1.f;
#pragma unroll
            for (int i = SUB - 1; i >= 0; --i) { k[i * P] *= f; f *= g[i * P]; }
        }
        __syncthreads();
    }

    // the values take the decays' place
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        float4 v = widen4(values[i]);
        if (MODE == CHUNK_DECAY && w.silu_inputs) v = silu4(v);
        store4(gs + (tid + i * THREADS) * 4, v);
    }
    // Weights of token pairs of different runs (one decay a head: of all runs): a warp a pair of runs, its halves
    // one half of the features each, 4 x 4 pairs a lane.
    for (int pair = warp; pair < (MODE == CHUNK_DECAY ? 10 : 6); pair += THREADS / 32) {
        const int run_i = pair < 3 ? 3 : pair < 5 ? 2 : pair < 6 ? 1 : pair - 6;
        const int run_j = pair < 3 ? pair : pair < 5 ? pair - 3 : pair < 6 ? 0 : pair - 6;
        const int half = lane >> 4, ti = (lane >> 2) & 3, tj = lane & 3;
        const float* q0 = qs + (run_i * SUB + ti) * P + half * (D / 2);         // rows ti + 4 r
        const float* k0 = ks + (run_j * SUB + tj) * P + half * (D / 2);
        float s[4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[r][c] = 0.f;
#pragma unroll 2
        for (int d = 0; d < D / 2; d += 4) {
            float4 q[4], k[4];
            float4 f = make_float4(1.f, 1.f, 1.f, 1.f);           // the decays of the runs in between
            if constexpr (MODE == CHUNK_GATED) {
                for (int m = run_j + 1; m < run_i; ++m) {
                    const float4 e = load4(es + m * D + half * (D / 2) + d);
                    f.x *= e.x; f.y *= e.y; f.z *= e.z; f.w *= e.w;
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                q[r] = load4(q0 + 4 * r * P + d);
                k[r] = load4(k0 + 4 * r * P + d);
                k[r].x *= f.x; k[r].y *= f.y; k[r].z *= f.z; k[r].w *= f.w;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    s[r][c] = fmaf(q[r].x, k[c].x, s[r][c]);
                    s[r][c] = fmaf(q[r].y, k[c].y, s[r][c]);
                    s[r][c] = fmaf(q[r].z, k[c].z, s[r][c]);
                    s[r][c] = fmaf(q[r].w, k[c].w, s[r][c]);
                }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                s[r][c] += __shfl_xor_sync(0xffffffffu, s[r][c], 16);
                const int i = run_i * SUB + ti + 4 * r, j = run_j * SUB + tj + 4 * c;
                if (MODE == CHUNK_DECAY) s[r][c] = i >= j ? s[r][c] * powers[i - j] : 0.f;
                if (half == 0) left[(long)(D + j) * CHUNK + i] = s[r][c];
            }
        // the mirrored pairs: a token does not see later ones
        for (int e = lane; e < (run_i == run_j ? 0 : SUB * SUB); e += 32)
            left[(long)(D + run_i * SUB + e / SUB) * CHUNK + run_j * SUB + e % SUB] = 0.f;
    }
    __syncthreads();

    // the read vectors leave with the decays since the chunk's start; k gets those up to its end
    for (int e = tid; e < SUBS * D; e += THREADS) {
        const int sub = e / D, d = e % D;
        const float* q = qs + sub * SUB * P + d;
        float* k = ks + sub * SUB * P + d;
        float* dst = left + (long)d * CHUNK + sub * SUB;
        if constexpr (MODE == CHUNK_DECAY) {
            const float* f = powers + sub * SUB + 1;
#pragma unroll
            for (int i = 0; i < SUB; i += 4)
                store4(dst + i, make_float4(q[i * P] * f[i], q[(i + 1) * P] * f[i + 1], q[(i + 2) * P] * f[i + 2], q[(i + 3) * P] * f[i + 3]));
            if (sub == SUBS - 1) whole[d] = powers[n];
#pragma unroll
            for (int i = 0; i < SUB; ++i) k[i * P] *= powers[max(n - 1 - sub * SUB - i, 0)];
        } else {
            float f = 1.f;
            for (int m = 0; m < sub; ++m) f *= es[m * D + d];
#pragma unroll
            for (int i = 0; i < SUB; i += 4)
                store4(dst + i, make_float4(q[i * P] * f, q[(i + 1) * P] * f, q[(i + 2) * P] * f, q[(i + 3) * P] * f));
            if (sub == SUBS - 1) whole[d] = f * es[e];
            f = 1.f;
            for (int m = sub + 1; m < SUBS; ++m) f *= es[m * D + d];
#pragma unroll
            for (int i = 0; i < SUB; ++i) k[i * P] *= f;
        }
    }
    __syncthreads();

    // the chunk's share of the state: k^T v
    constexpr int TX = V / 8, TY = D / 8;
    for (int t = tid; t < TX * TY; t += THREADS) {
        // a warp is 4 x 8 threads
        const int wt = t >> 5, ty = (wt / (TX / 8)) * 4 + (t & 31) / 8, tx = (wt % (TX / 8)) * 8 + (t & 7);
        float2 acc[8][4];
        clear8(acc);
#pragma unroll 4
        for (int r = 0; r < CHUNK; ++r) outer8<D, V>(ks + r * P + ty * 4, gs + r * V + tx * 4, acc);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float* dst = share + (long)((i / 4) * (D / 2) + ty * 4 + i % 4) * V + tx * 4;
            store4(dst, make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y));
            store4(dst + V / 2, make_float4(acc[i][2].x, acc[i][2].y, acc[i][3].x, acc[i][3].y));
        }
    }
}

// grid (H * D * V / 4 / THREADS, segments)
template <int D, int V>
__global__ void __launch_bounds__(THREADS)
chunk_carry_kernel(const ChunkArgs w) {
    const long e = ((long)blockIdx.x * THREADS + threadIdx.x) * 4;
    const int h = (int)(e / (D * V)), in = (int)(e % (D * V)), d = in / V;
    int before = 0;                       // chunks of the segments before this one
    for (int s = threadIdx.x & 31; s < (int)blockIdx.y; s += 32) before += (w.seg_q_start[s + 1] - w.seg_q_start[s] + CHUNK - 1) / CHUNK;
    before = __reduce_add_sync(0xffffffffu, before);
    const int n = w.seg_q_start[blockIdx.y + 1] - w.seg_q_start[blockIdx.y], chunks = (n + CHUNK - 1) / CHUNK;
    if (chunks == 0) return;
    float* st = w.state + ((long)w.seg_slot[blockIdx.y] * w.H + h) * D * V + in;
    const long unit = unit_floats(D, V), step = unit * w.H;
    float* base = w.scratch + ((long)before * w.H + h) * unit + left_floats(D);
    float4 s = load4(st);
    constexpr int AHEAD = 4;
    for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
        float4 share[AHEAD];
        float whole[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < chunks) {
                const float* p = base + (c0 + i) * step;
                share[i] = load4(p + in);
                whole[i] = p[(long)D * V + d];
            }
#pragma unroll
        for (int i = 0; i < AHEAD; ++i)
            if (c0 + i < chunks) {
                store4(base + (c0 + i) * step + in, s);
                s.x = fmaf(whole[i], s.x, share[i].x);
                s.y = fmaf(whole[i], s.y, share[i].y);
                s.z = fmaf(whole[i], s.z, share[i].z);
                s.w = fmaf(whole[i], s.w, share[i].w);
            }
    }
    store4(st, s);
}

constexpr int SLICE = SUB, STAGES = 3;       // k of a slice, slices in flight
template <int V> constexpr int finish_smem() { return STAGES * SLICE * (CHUNK + V) * (int)sizeof(float); }

// Four rows of a thread's outputs over one slice of values; with SEEN, row i takes the values up to its own, the slice's
// (row + i)-th.
template <int V, bool SEEN>
__device__ __forceinline__ void quad_rows(const float* as, const float* bs, int row, float2 (&x0)[4], float2 (&x1)[4], float2 (&x2)[4],
                                          float2 (&x3)[4]) {
#pragma unroll 4
    for (int k = 0; k < SLICE; ++k) {
        const float4 a = load4(as + k * CHUNK);
        float2 b[4];
        *reinterpret_cast<float4*>(b) = load4(bs + k * V);
        *reinterpret_cast<float4*>(b + 2) = load4(bs + k * V + V / 2);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!SEEN || k <= row) x0[j] = __ffma2_rn(make_float2(a.x, a.x), b[j], x0[j]);
            if (!SEEN || k <= row + 1) x1[j] = __ffma2_rn(make_float2(a.y, a.y), b[j], x1[j]);
            if (!SEEN || k <= row + 2) x2[j] = __ffma2_rn(make_float2(a.z, a.z), b[j], x2[j]);
            if (!SEEN || k <= row + 3) x3[j] = __ffma2_rn(make_float2(a.w, a.w), b[j], x3[j]);
        }
    }
}

template <int MODE, int D, int V>
__global__ void __launch_bounds__(V, 512 / V)
chunk_finish_kernel(const ChunkArgs w) {
    constexpr int NT = V;                 // CHUNK / 8 rows x V / 8 columns of threads
    extern __shared__ __align__(16) float smem[];        // [STAGES][SLICE][CHUNK + V]
    const int tid = threadIdx.x;
    const int chunk = blockIdx.x, h = blockIdx.y;
    const ChunkPlace at = place_of(w, chunk);
    if (at.tokens == 0) return;
    const float* left = w.scratch + ((long)chunk * w.H + h) * unit_of<MODE>(D, V);
    const float* state = left + left_floats(D);
    const float* writes = left + unit_floats(D, V) + 2 * CHUNK * D;       // delta: in place of the values
    constexpr int STEPS = (D + CHUNK) / SLICE, STATE_STEPS = D / SLICE, PIECES = SLICE * V / 4 / NT;
    // slices of values come through registers: asked for a step before they go to the ring
    uint2 values[PIECES];
    auto ask = [&](int step) {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int e = tid + i * NT, r = (step - STATE_STEPS) * SLICE + e / (V / 4), c = e % (V / 4) * 4;
            values[i] = *reinterpret_cast<const uint2*>((const bf16*)w.v + (long)(at.row + min(r, at.tokens - 1)) * w.ld + (long)h * V + c);
            if (r >= at.tokens) values[i] = make_uint2(0, 0);
        }
    };
    auto fetch = [&](int step) {
        float* as = smem + (step % STAGES) * SLICE * (CHUNK + V);
        float* bs = as + SLICE * CHUNK;
#pragma unroll
        for (int e = 0; e < SLICE * CHUNK; e += NT * 4) copy_async_16(as + e + tid * 4, left + (long)step * SLICE * CHUNK + e + tid * 4);
        if (MODE == CHUNK_DELTA || step < STATE_STEPS) {
            const float* src = step < STATE_STEPS ? state + (long)step * SLICE * V : writes + (long)(step - STATE_STEPS) * SLICE * V;
#pragma unroll
            for (int e = 0; e < SLICE * V; e += NT * 4) copy_async_16(bs + e + tid * 4, src + e + tid * 4);
        } else {
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                float4 v = widen4(values[i]);
                if (MODE == CHUNK_DECAY && w.silu_inputs) v = silu4(v);
                store4(bs + (tid + i * NT) * 4, v);
            }
        }
        if (MODE != CHUNK_DELTA && step + 1 >= STATE_STEPS && step + 1 < STEPS) ask(step + 1);
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    constexpr int TX = V / 8;
    const int wt = tid >> 5, ty = (wt / (TX / 8)) * 4 + (tid & 31) / 8, tx = (wt % (TX / 8)) * 8 + (tid & 7);
    float2 acc[8][4];
    clear8(acc);
    for (int step = 0; step < STEPS; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        if (step + STAGES - 1 < STEPS) fetch(step + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = smem + (step % STAGES) * SLICE * (CHUNK + V);
        const float* bs = as + SLICE * CHUNK;
        if (step < STATE_STEPS) {
#pragma unroll
            for (int k = 0; k < SLICE; ++k) outer8<CHUNK, V>(as + k * CHUNK + ty * 4, bs + k * V + tx * 4, acc);
            continue;
        }
        // A value enters the sums of its own token and of later ones only (zero times an infinity is no number): a
        // slice is one run's values, a warp's quads of rows lie in one run of the chunk's first half and one of its second.
        const int run = step - STATE_STEPS;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int ahead = half * (SUBS / 2) + ty / 4 - run;           // the rows' run before (negative), at or after the values'
            const float* a = as + half * (CHUNK / 2) + ty * 4;
            if (ahead > 0) quad_rows<V, false>(a, bs + tx * 4, 0, acc[half * 4], acc[half * 4 + 1], acc[half * 4 + 2], acc[half * 4 + 3]);
            if (ahead == 0)
                quad_rows<V, true>(a, bs + tx * 4, ty % 4 * 4, acc[half * 4], acc[half * 4 + 1], acc[half * 4 + 2], acc[half * 4 + 3]);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = (i / 4) * (CHUNK / 2) + ty * 4 + i % 4;
        if (r >= at.tokens) continue;
        float* dst = w.out + ((long)(at.row + r) * w.H + h) * V + tx * 4;
        store4(dst, make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y));
        store4(dst + V / 2, make_float4(acc[i][2].x, acc[i][2].y, acc[i][3].x, acc[i][3].y));
    }
}

// ------------------------------------------------------------------------------------------
// The delta rule: u_i = beta_i (v_i - S_i^T k_i) with S_i the decayed state, S_(i) = S_i + k_i u_i^T, o_i = S_(i)^T q_i.
// With L_ij = beta_i (k_i . G(j, i) k_j) for j < i the writes of a chunk solve (I + L) U = beta (V - (k G(-1, .)) S), so
//   U = U0 - W S,   U0 = (I + L)^-1 beta V,   W = (I + L)^-1 beta (k G(-1, .))
// and the chunk goes on as above with U in the place of V.  prepare makes U0 and W by forward substitution, two
// columns a thread; the carry is a chain of two products a chunk, U = U0 - W S and S' = G S + k^T U, for a slice of
// value columns a block; finish is the same.  The carry is bound by the shared-memory reads of its two products and,
// with one block a multiprocessor, by their latency (3.9 us a chunk).  16 heads of 128 x 128, walked / in chunks, us:
// 2,048 tokens 642 / 257 (prepare 99, carry 124, finish 34), segments of 396, 592 and 789 tokens 346 / 239 (96, 108,
// 34; the segments in the order they come instead of the longest first, and reads that met banks twice: 174).
// ------------------------------------------------------------------------------------------
constexpr int PAIR_FLOATS = SUBS * (SUBS + 1) / 2 * SUB * SUB;     // L below and on its diagonal blocks, [block][j][i]
__host__ __device__ constexpr int pair_block(int run_i, int run_j) { return (run_i * (run_i + 1) / 2 + run_j) * SUB * SUB; }
template <int D, int V> constexpr int delta_smem() {
    return (3 * third_floats<D, V>() + SUBS * D + PAIR_FLOATS + CHUNK) * (int)sizeof(float);
}

template <int D, int V>
__global__ void __launch_bounds__(THREADS, 2)
chunk_delta_prepare_kernel(const ChunkArgs w) {
    constexpr int P = D + 4;
    extern __shared__ __align__(16) float smem[];
    float* qs = smem;                                 // q, then beta v and U0 ([CHUNK][V])
    float* ks = qs + third_floats<D, V>();            // k, then with the decays up to its run's end
    float* gs = ks + third_floats<D, V>();            // the decays, then k with those from its run's start, then W
    float* es = gs + third_floats<D, V>();            // [SUBS][D] a run's whole decay
    float* lower = es + SUBS * D;                     // L
    float* beta = lower + PAIR_FLOATS;                // [CHUNK]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int chunk = blockIdx.x, h = blockIdx.y, kh = h / w.group;
    const ChunkPlace at = place_of(w, chunk);
    const int n = at.tokens;
    if (n == 0) return;
    float* left = w.scratch + ((long)chunk * w.H + h) * delta_floats(D, V);
    float* whole = left + left_floats(D) + (long)D * V;
    float* takes = whole + D;                         // W, tokens last
    float* ends = takes + CHUNK * D;
    float* writes = ends + CHUNK * D;

    constexpr int LANES = D / 4, ROWS = THREADS / LANES, PASSES = CHUNK / ROWS, PIECES = CHUNK * V / 4 / THREADS;
    const int d0 = (tid % LANES) * 4, r0 = tid / LANES;
    uint2 values[PIECES];
    {
        uint2 rq[PASSES], rk[PASSES];
        float4 ra[PASSES];
        const float4 bias = load4(w.bias + (long)h * D + d0);
        const float rate = expf(w.a_log[h]);
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            const long row = at.row + min(r0 + p * ROWS, n - 1);
            rq[p] = *reinterpret_cast<const uint2*>((const bf16*)w.q + row * w.ld + (long)kh * D + d0);
            rk[p] = *reinterpret_cast<const uint2*>((const bf16*)w.k + row * w.ld + (long)kh * D + d0);
            ra[p] = load4(w.a + (row * w.H + h) * D + d0);
        }
        if (tid < CHUNK) beta[tid] = tid < n ? 1.f / (1.f + expf(-to_float(w.b[(at.row + tid) * w.ldb + h]))) : 0.f;
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            const int r = r0 + p * ROWS;
            float4 q = widen4(rq[p]), k = widen4(rk[p]), g = make_float4(1.f, 1.f, 1.f, 1.f);
            float sq = q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w, sk = k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w;
#pragma unroll
            for (int o = LANES / 2; o > 0; o >>= 1) {             // a row's lanes lie side by side
                sq += __shfl_xor_sync(0xffffffffu, sq, o);
                sk += __shfl_xor_sync(0xffffffffu, sk, o);
            }
            const bool in = r < n;
            const float fq = in ? (1.f / sqrtf((float)D)) / sqrtf(sq + 1e-6f) : 0.f, fk = in ? 1.f / sqrtf(sk + 1e-6f) : 0.f;
            q = make_float4(q.x * fq, q.y * fq, q.z * fq, q.w * fq);
            k = make_float4(k.x * fk, k.y * fk, k.z * fk, k.w * fk);
            if (in)
                g = make_float4(expf(-rate * softplus_f(ra[p].x + bias.x)), expf(-rate * softplus_f(ra[p].y + bias.y)),
                                expf(-rate * softplus_f(ra[p].z + bias.z)), expf(-rate * softplus_f(ra[p].w + bias.w)));
            else
                q = k = make_float4(0.f, 0.f, 0.f, 0.f);
            store4(qs + r * P + d0, q);
            store4(ks + r * P + d0, k);
            store4(gs + r * P + d0, g);
        }
    }
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int e = tid + i * THREADS, r = e / (V / 4), c = e % (V / 4) * 4;
        values[i] = *reinterpret_cast<const uint2*>((const bf16*)w.v + (long)(at.row + min(r, n - 1)) * w.ld + (long)h * V + c);
        if (r >= n) values[i] = make_uint2(0, 0);
    }
    __syncthreads();

    // token pairs within a run, as in the gated scan; k meets k as q does
    {
        const int sub = warp >> 1, slice = lane & 7, j0 = (warp & 1) * 8 + (lane >> 3) * 2;
        const float* q0 = qs + sub * SUB * P + slice * 4;
        const float* g0 = gs + sub * SUB * P + slice * 4;
        const float* i0 = ks + sub * SUB * P + slice * 4;
        const float* k0 = i0 + j0 * P;
        float4 x[D / 32], y[D / 32];
#pragma unroll
        for (int m = 0; m < D / 32; ++m) { x[m] = load4(k0 + 32 * m); y[m] = load4(k0 + P + 32 * m); }
        float* dst = left + (long)(D + sub * SUB + j0) * CHUNK + sub * SUB;
        float* low = lower + pair_block(sub, sub) + j0 * SUB;
        for (int i = (warp & 1) * 8; i < SUB; ++i) {
            float s[4] = {0.f, 0.f, 0.f, 0.f};        // q with j0, j0 + 1; k likewise
#pragma unroll
            for (int m = 0; m < D / 32; ++m) {
                const float4 q = load4(q0 + i * P + 32 * m), g = load4(g0 + i * P + 32 * m), k = load4(i0 + i * P + 32 * m);
                if (i > j0) { x[m].x *= g.x; x[m].y *= g.y; x[m].z *= g.z; x[m].w *= g.w; }
                if (i > j0 + 1) { y[m].x *= g.x; y[m].y *= g.y; y[m].z *= g.z; y[m].w *= g.w; }
                s[0] = fmaf(q.x, x[m].x, s[0]); s[0] = fmaf(q.y, x[m].y, s[0]); s[0] = fmaf(q.z, x[m].z, s[0]); s[0] = fmaf(q.w, x[m].w, s[0]);
                s[1] = fmaf(q.x, y[m].x, s[1]); s[1] = fmaf(q.y, y[m].y, s[1]); s[1] = fmaf(q.z, y[m].z, s[1]); s[1] = fmaf(q.w, y[m].w, s[1]);
                s[2] = fmaf(k.x, x[m].x, s[2]); s[2] = fmaf(k.y, x[m].y, s[2]); s[2] = fmaf(k.z, x[m].z, s[2]); s[2] = fmaf(k.w, x[m].w, s[2]);
                s[3] = fmaf(k.x, y[m].x, s[3]); s[3] = fmaf(k.y, y[m].y, s[3]); s[3] = fmaf(k.z, y[m].z, s[3]); s[3] = fmaf(k.w, y[m].w, s[3]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                for (int c = 0; c < 4; ++c) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
            if (slice == 0) {
                const float f = beta[sub * SUB + i];
                dst[i] = i >= j0 ? s[0] : 0.f;
                dst[CHUNK + i] = i > j0 ? s[1] : 0.f;
                low[i] = i > j0 ? f * s[2] : 0.f;
                low[SUB + i] = i > j0 + 1 ? f * s[3] : 0.f;
            }
        }
        if (warp & 1)
            for (int e = lane; e < 64; e += 32) {
                left[(long)(D + sub * SUB + 8 + e / 8) * CHUNK + sub * SUB + e % 8] = 0.f;
                lower[pair_block(sub, sub) + (8 + e / 8) * SUB + e % 8] = 0.f;
            }
    }
    __syncthreads();

    for (int e = tid; e < SUBS * D; e += THREADS) {
        const int sub = e / D, d = e % D;
        float* q = qs + sub * SUB * P + d;
        float* k = ks + sub * SUB * P + d;
        float* g = gs + sub * SUB * P + d;
        float decay[SUB];
        float f = 1.f;
#pragma unroll
        for (int i = 0; i < SUB; ++i) {
            decay[i] = g[i * P];
            f *= decay[i];
            q[i * P] *= f;
            g[i * P] = k[i * P] * f;
        }
        es[e] = f;
        f = 1.f;
#pragma unroll
        for (int i = SUB - 1; i >= 0; --i) { k[i * P] *= f; f *= decay[i]; }
    }
    __syncthreads();

    // token pairs of different runs
    if (warp < 6) {
        const int run_i = warp < 3 ? 3 : warp < 5 ? 2 : 1, run_j = warp < 3 ? warp : warp < 5 ? warp - 3 : 0;
        const int half = lane >> 4, ti = (lane >> 2) & 3, tj = lane & 3;
        const float* q0 = qs + (run_i * SUB + ti) * P + half * (D / 2);
        const float* i0 = gs + (run_i * SUB + ti) * P + half * (D / 2);
        const float* k0 = ks + (run_j * SUB + tj) * P + half * (D / 2);
        float s[2][4][4];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) s[0][r][c] = s[1][r][c] = 0.f;
        for (int d = 0; d < D / 2; d += 4) {
            float4 k[4];
            float4 f = make_float4(1.f, 1.f, 1.f, 1.f);
            for (int m = run_j + 1; m < run_i; ++m) {
                const float4 e = load4(es + m * D + half * (D / 2) + d);
                f.x *= e.x; f.y *= e.y; f.z *= e.z; f.w *= e.w;
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                k[r] = load4(k0 + 4 * r * P + d);
                k[r].x *= f.x; k[r].y *= f.y; k[r].z *= f.z; k[r].w *= f.w;
            }
#pragma unroll
            for (int which = 0; which < 2; ++which)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float4 x = load4((which ? i0 : q0) + 4 * r * P + d);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        float& t = s[which][r][c];
                        t = fmaf(x.x, k[c].x, t);
                        t = fmaf(x.y, k[c].y, t);
                        t = fmaf(x.z, k[c].z, t);
                        t = fmaf(x.w, k[c].w, t);
                    }
                }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int i = ti + 4 * r, j = tj + 4 * c;
                const float wq = s[0][r][c] + __shfl_xor_sync(0xffffffffu, s[0][r][c], 16);
                const float wk = s[1][r][c] + __shfl_xor_sync(0xffffffffu, s[1][r][c], 16);
                if (half == 0) left[(long)(D + run_j * SUB + j) * CHUNK + run_i * SUB + i] = wq;
                else lower[pair_block(run_i, run_j) + j * SUB + i] = beta[run_i * SUB + i] * wk;
            }
        for (int e = lane; e < SUB * SUB; e += 32)
            left[(long)(D + run_i * SUB + e / SUB) * CHUNK + run_j * SUB + e % SUB] = 0.f;
    }
    __syncthreads();

    // the read vectors and the chunk's k leave; k from the chunk's start, times beta, is one half of what is solved for
    for (int e = tid; e < SUBS * D; e += THREADS) {
        const int sub = e / D, d = e % D;
        const float* q = qs + sub * SUB * P + d;
        const float* k = ks + sub * SUB * P + d;
        float* g = gs + sub * SUB * P + d;
        float* dst = left + (long)d * CHUNK + sub * SUB;
        float f = 1.f;
        for (int m = 0; m < sub; ++m) f *= es[m * D + d];
#pragma unroll
        for (int i = 0; i < SUB; i += 4)
            store4(dst + i, make_float4(q[i * P] * f, q[(i + 1) * P] * f, q[(i + 2) * P] * f, q[(i + 3) * P] * f));
#pragma unroll
        for (int i = 0; i < SUB; ++i) g[i * P] *= f * beta[sub * SUB + i];
        if (sub == SUBS - 1) whole[d] = f * es[e];
        f = 1.f;
        for (int m = sub + 1; m < SUBS; ++m) f *= es[m * D + d];
#pragma unroll
        for (int i = 0; i < SUB; ++i) ends[(sub * SUB + i) * D + d] = k[i * P] * f;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PIECES; ++i) {
        const int e = tid + i * THREADS;
        const float f = beta[e / (V / 4)];
        const float4 v = widen4(values[i]);
        store4(qs + e * 4, make_float4(v.x * f, v.y * f, v.z * f, v.w * f));
    }
    __syncthreads();

    // forward substitution, in place, two columns a thread
    if (tid < (D + V) / 2) {
        const bool key = tid < D / 2;
        float* x0 = key ? gs + 2 * tid : qs + 2 * (tid - D / 2);
        const int pitch = key ? P : V;
#pragma unroll
        for (int run = 0; run < SUBS; ++run) {
            float2 x[SUB];
#pragma unroll
            for (int i = 0; i < SUB; ++i) x[i] = *reinterpret_cast<const float2*>(x0 + (run * SUB + i) * pitch);
#pragma unroll
            for (int before = 0; before < run; ++before) {
                const float* low = lower + pair_block(run, before);
#pragma unroll 2
                for (int j = 0; j < SUB; ++j) {
                    float2 t = *reinterpret_cast<const float2*>(x0 + (before * SUB + j) * pitch);
                    t.x = -t.x; t.y = -t.y;
#pragma unroll
                    for (int i = 0; i < SUB; i += 4) {
                        const float4 f = load4(low + j * SUB + i);
                        x[i] = __ffma2_rn(make_float2(f.x, f.x), t, x[i]);
                        x[i + 1] = __ffma2_rn(make_float2(f.y, f.y), t, x[i + 1]);
                        x[i + 2] = __ffma2_rn(make_float2(f.z, f.z), t, x[i + 2]);
                        x[i + 3] = __ffma2_rn(make_float2(f.w, f.w), t, x[i + 3]);
                    }
                }
            }
            const float* low = lower + pair_block(run, run);
#pragma unroll
            for (int j = 0; j < SUB - 1; ++j) {
                const float2 t = make_float2(-x[j].x, -x[j].y);
#pragma unroll
                for (int i = j / 4 * 4; i < SUB; i += 4) {            // L is zero up to its diagonal
                    const float4 f = load4(low + j * SUB + i);
                    if (i > j) x[i] = __ffma2_rn(make_float2(f.x, f.x), t, x[i]);
                    if (i + 1 > j) x[i + 1] = __ffma2_rn(make_float2(f.y, f.y), t, x[i + 1]);
                    if (i + 2 > j) x[i + 2] = __ffma2_rn(make_float2(f.z, f.z), t, x[i + 2]);
                    if (i + 3 > j) x[i + 3] = __ffma2_rn(make_float2(f.w, f.w), t, x[i + 3]);
                }
            }
#pragma unroll
            for (int i = 0; i < SUB; ++i) *reinterpret_cast<float2*>(x0 + (run * SUB + i) * pitch) = x[i];
        }
    }
    __syncthreads();
    for (int e = tid; e < SUBS * D; e += THREADS) {
        const int sub = e / D, d = e % D;
        const float* g = gs + sub * SUB * P + d;
#pragma unroll
        for (int i = 0; i < SUB; i += 4)
            store4(takes + (long)d * CHUNK + sub * SUB + i, make_float4(g[i * P], g[(i + 1) * P], g[(i + 2) * P], g[(i + 3) * P]));
    }
#pragma unroll
    for (int i = 0; i < PIECES; ++i) store4(writes + (tid + i * THREADS) * 4, load4(qs + (tid + i * THREADS) * 4));
}

// grid (V / COLS, H, segments): a block carries COLS value columns of a head's state over a segment's chunks.  W and
// the chunk's k have one buffer each, filled again while the other is read.
constexpr int COLS = 16, TAKES_P = CHUNK + 4, STATE_P = COLS + 8;       // the lanes of a read meet no bank twice
template <int D> constexpr int delta_carry_smem() {
    return (D * TAKES_P + CHUNK * (D + 4) + 3 * CHUNK * COLS + D * STATE_P + 2 * D) * (int)sizeof(float);
}

template <int D, int V>
__global__ void __launch_bounds__(THREADS)
chunk_delta_carry_kernel(const ChunkArgs w) {
    extern __shared__ __align__(16) float smem[];
    float* ts = smem;                                 // [D][TAKES_P] W, tokens last
    float* es = ts + D * TAKES_P;                     // [CHUNK][D + 4] k
    float* us = es + CHUNK * (D + 4);                       // [2][CHUNK][COLS] U0 of this chunk and the next
    float* ws = us + 2 * CHUNK * COLS;                // [CHUNK][COLS] U
    float* st = ws + CHUNK * COLS;                 // [D][STATE_P] the state
    float* fs = st + D * STATE_P;                     // [2][D] the chunk's whole decay
    const int tid = threadIdx.x;
    const int h = blockIdx.y, col0 = blockIdx.x * COLS;
    int seg = blockIdx.z;
    if (w.segments <= 32) {               // blocks start in the order of their index: the longest segments first
        const int lane = tid & 31;
        const int mine = lane < w.segments ? w.seg_q_start[lane + 1] - w.seg_q_start[lane] : -1;
        int rank = 0;
        for (int s = 0; s < w.segments; ++s) {
            const int other = __shfl_sync(0xffffffffu, mine, s);
            rank += other > mine || (other == mine && s < lane);
        }
        seg = __ffs(__ballot_sync(0xffffffffu, lane < w.segments && rank == (int)blockIdx.z)) - 1;
    }
    int before = 0;
    for (int s = tid & 31; s < seg; s += 32) before += (w.seg_q_start[s + 1] - w.seg_q_start[s] + CHUNK - 1) / CHUNK;
    before = __reduce_add_sync(0xffffffffu, before);
    const int n = w.seg_q_start[seg + 1] - w.seg_q_start[seg], chunks = (n + CHUNK - 1) / CHUNK;
    if (chunks <= 0) return;
    const long step = delta_floats(D, V) * w.H;
    float* unit = w.scratch + ((long)before * w.H + h) * delta_floats(D, V);
    constexpr long STATE = left_floats(D), WHOLE = STATE + (long)D * V, TAKES = WHOLE + D, ENDS = TAKES + CHUNK * D, WRITES = ENDS + CHUNK * D;
    float* home = w.state + ((long)w.seg_slot[seg] * w.H + h) * D * V + col0;

    auto bring_takes = [&](int c) {
        const float* src = unit + c * step;
        for (int e = tid * 4; e < D * CHUNK; e += THREADS * 4) copy_async_16(ts + e / CHUNK * TAKES_P + e % CHUNK, src + TAKES + e);
        for (int e = tid * 4; e < CHUNK * COLS; e += THREADS * 4)
            copy_async_16(us + (c & 1) * CHUNK * COLS + e, src + WRITES + (long)(e / COLS) * V + col0 + e % COLS);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto bring_ends = [&](int c) {
        const float* src = unit + c * step;
        for (int e = tid * 4; e < CHUNK * D; e += THREADS * 4) copy_async_16(es + e / D * (D + 4) + e % D, src + ENDS + e);
        for (int e = tid * 4; e < D; e += THREADS * 4) copy_async_16(fs + (c & 1) * D + e, src + WHOLE + e);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    bring_takes(0);
    bring_ends(0);
    for (int e = tid * 4; e < D * COLS; e += THREADS * 4) store4(st + e / COLS * STATE_P + e % COLS, load4(home + (long)(e / COLS) * V + e % COLS));

    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");          // W and U0 are here
        __syncthreads();
        float* old = unit + c * step + STATE + col0;                  // the state at the chunk's start, for finish
        for (int e = tid * 4; e < D * COLS; e += THREADS * 4) store4(old + (long)(e / COLS) * V + e % COLS, load4(st + e / COLS * STATE_P + e % COLS));
        {
            // U = U0 - W S: 4 x 4 outputs a group of four lanes, a quarter of the features a lane
            const int part = tid & 3, tile = tid >> 2, row = (tile >> 2) * 4, col = (tile & 3) * 4;
            float2 acc[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
#pragma unroll 8
            for (int d = part; d < D; d += 4) {
                const float4 a = load4(ts + d * TAKES_P + row), b = load4(st + d * STATE_P + col);
                const float2 b0 = make_float2(b.x, b.y), b1 = make_float2(b.z, b.w);
                acc[0][0] = __ffma2_rn(make_float2(a.x, a.x), b0, acc[0][0]); acc[0][1] = __ffma2_rn(make_float2(a.x, a.x), b1, acc[0][1]);
                acc[1][0] = __ffma2_rn(make_float2(a.y, a.y), b0, acc[1][0]); acc[1][1] = __ffma2_rn(make_float2(a.y, a.y), b1, acc[1][1]);
                acc[2][0] = __ffma2_rn(make_float2(a.z, a.z), b0, acc[2][0]); acc[2][1] = __ffma2_rn(make_float2(a.z, a.z), b1, acc[2][1]);
                acc[3][0] = __ffma2_rn(make_float2(a.w, a.w), b0, acc[3][0]); acc[3][1] = __ffma2_rn(make_float2(a.w, a.w), b1, acc[3][1]);
            }
            // the four lanes' sums meet: each keeps half of the rows, then one
            float2 two[2][2], one[2];
            const bool upper = part & 2, odd = part & 1;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float2 keep = upper ? acc[2 + i][j] : acc[i][j], give = upper ? acc[i][j] : acc[2 + i][j];
                    two[i][j] = make_float2(keep.x + __shfl_xor_sync(0xffffffffu, give.x, 2), keep.y + __shfl_xor_sync(0xffffffffu, give.y, 2));
                }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float2 keep = odd ? two[1][j] : two[0][j], give = odd ? two[0][j] : two[1][j];
                one[j] = make_float2(keep.x + __shfl_xor_sync(0xffffffffu, give.x, 1), keep.y + __shfl_xor_sync(0xffffffffu, give.y, 1));
            }
            const int r = row + part;
            const float4 u0 = load4(us + (c & 1) * CHUNK * COLS + r * COLS + col);
            const float4 u = make_float4(u0.x - one[0].x, u0.y - one[0].y, u0.z - one[1].x, u0.w - one[1].y);
            store4(ws + r * COLS + col, u);
            store4(unit + c * step + WRITES + (long)r * V + col0 + col, u);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");          // the chunk's k is here
        __syncthreads();
        if (c + 1 < chunks) bring_takes(c + 1);
        {
            // S' = G S + k^T U: tiles of 4 x 4, a part of the tokens a lane of two (D = 128) or four (D = 64)
            constexpr int PARTS = THREADS * 16 / (D * COLS);
            const int part = tid % PARTS, tile = tid / PARTS, row = (tile >> 2) * 4, col = (tile & 3) * 4;
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 8
            for (int r = part; r < CHUNK; r += PARTS) {
                const float4 a = load4(es + r * (D + 4) + row), b = load4(ws + r * COLS + col);
                const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
            }
#pragma unroll
            for (int o = 1; o < PARTS; o <<= 1)
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] += __shfl_xor_sync(0xffffffffu, acc[i][j], o);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i % PARTS == part) {
                    float* s = st + (row + i) * STATE_P + col;
                    const float f = fs[(c & 1) * D + row + i];
                    const float4 v = load4(s);
                    store4(s, make_float4(fmaf(f, v.x, acc[i][0]), fmaf(f, v.y, acc[i][1]), fmaf(f, v.z, acc[i][2]), fmaf(f, v.w, acc[i][3])));
                }
        }
        __syncthreads();
        if (c + 1 < chunks) bring_ends(c + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    for (int e = tid * 4; e < D * COLS; e += THREADS * 4) store4(home + (long)(e / COLS) * V + e % COLS, load4(st + e / COLS * STATE_P + e % COLS));
}

template <int MODE, int D, int V>
int launch(const ChunkArgs& w, cudaStream_t stream) {
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(chunk_prepare_kernel<MODE, D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, prepare_smem<D, V>()),
                    "chunked scan");
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(chunk_finish_kernel<MODE, D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, finish_smem<V>()),
                    "chunked scan");
    const dim3 grid(w.chunks, w.H);
    chunk_prepare_kernel<MODE, D, V><<<grid, THREADS, prepare_smem<D, V>(), stream>>>(w);
    chunk_carry_kernel<D, V><<<dim3(w.H * (D * V / 4 / THREADS), w.segments), THREADS, 0, stream>>>(w);
    chunk_finish_kernel<MODE, D, V><<<grid, V, finish_smem<V>(), stream>>>(w);
    MRUN_CHECK_LAUNCH("chunked scan");
    return 0;
}

template <int D, int V>
int launch_delta(const ChunkArgs& w, cudaStream_t stream) {
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(chunk_delta_prepare_kernel<D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, delta_smem<D, V>()),
                    "chunked delta scan");
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(chunk_delta_carry_kernel<D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, delta_carry_smem<D>()),
                    "chunked delta scan");
    MRUN_CHECK_CUDA(cudaFuncSetAttribute(chunk_finish_kernel<CHUNK_DELTA, D, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, finish_smem<V>()),
                    "chunked delta scan");
    const dim3 grid(w.chunks, w.H);
    chunk_delta_prepare_kernel<D, V><<<grid, THREADS, delta_smem<D, V>(), stream>>>(w);
    chunk_delta_carry_kernel<D, V><<<dim3(V / COLS, w.H, w.segments), THREADS, delta_carry_smem<D>(), stream>>>(w);
    chunk_finish_kernel<CHUNK_DELTA, D, V><<<grid, V, finish_smem<V>(), stream>>>(w);
    MRUN_CHECK_LAUNCH("chunked delta scan");
    return 0;
}

template <int MODE, int D, int V>
int launch_mode(const ChunkArgs& w, cudaStream_t stream) {
    if constexpr (MODE == CHUNK_DELTA) return launch_delta<D, V>(w, stream);
    else return launch<MODE, D, V>(w, stream);
}

template <int MODE>
int launch_sizes(const ChunkArgs& w, cudaStream_t stream) {
    if (w.D == 128) return w.V == 128 ? launch_mode<MODE, 128, 128>(w, stream) : launch_mode<MODE, 128, 64>(w, stream);
    return w.V == 128 ? launch_mode<MODE, 64, 128>(w, stream) : launch_mode<MODE, 64, 64>(w, stream);
}

}  // namespace

// Floats of scratch that the chunked form of a decay, gated or (delta = 1) delta scan over `chunks` chunks takes, or
// 0 where it does not take these rows (q, k, v, ld, state and out as for the scan itself; a and bias, dt_bias in
// a delta scan, null for a decay scan).
MRUN_API long mrun_chunked_scan_floats(int delta, const void* q, const void* k, const void* v, long ld, int act_dtype, const float* a,
                                       const float* bias, const float* state, const float* out, int chunks, int H, int D, int V) {
    const bool takes = act_dtype == MRUN_BF16 && (D == 64 || D == 128) && (V == 64 || V == 128) && ld % 4 == 0 && chunks > 0 && H <= 65535 &&
                       ((((uintptr_t)q) | ((uintptr_t)k) | ((uintptr_t)v)) & 7) == 0 &&
                       ((((uintptr_t)a) | ((uintptr_t)bias) | ((uintptr_t)state) | ((uintptr_t)out)) & 15) == 0;
    return takes ? (long)chunks * H * (delta ? delta_floats(D, V) : unit_floats(D, V)) : 0;
}

// A decay scan (decay given: float32 [H], q, k, v through SiLU where silu_inputs) or a gated scan (a, bias, tau)
// as mrun_decay_scan() and mrun_gated_scan() compute them, bfloat16 rows.  chunks: at least the sum of ceil(tokens /
// 64) over the segments; scratch: mrun_chunked_scan_floats() floats on a 16-byte boundary.
MRUN_API int mrun_chunked_scan(const void* q, const void* k, const void* v, long ld, const float* decay, int silu_inputs, const float* a,
                               const float* bias, float tau, float* state, float* out, float* scratch, const int* seg_q_start,
                               const int* seg_slot, int segments, int chunks, int H, int D, int V, cudaStream_t stream) {
    MRUN_REQUIRE(segments >= 0 && segments <= 65535 && (decay != nullptr || tau > 0.f), "chunked_scan: bad sizes");
    MRUN_REQUIRE(mrun_chunked_scan_floats(0, q, k, v, ld, MRUN_BF16, a, bias, state, out, chunks, H, D, V) > 0 &&
                     (((uintptr_t)scratch) & 15) == 0,
                 "chunked_scan: these sizes or rows have no chunked form");
    if (segments == 0) return 0;
    const ChunkArgs w = {q, k, v, ld, a, bias, decay, nullptr, nullptr, 0, 1, tau, silu_inputs, state, out, scratch, seg_q_start, seg_slot,
                         segments, chunks, H, D, V};
    return decay ? launch_sizes<CHUNK_DECAY>(w, stream) : launch_sizes<CHUNK_GATED>(w, stream);
}

// A delta scan as mrun_delta_scan() computes it, bfloat16 rows; chunks and scratch as above.
MRUN_API int mrun_chunked_delta_scan(const void* q, const void* k, const void* v, long ld, int group, const float* a, const void* b,
                                     long ldb, const float* a_log, const float* dt_bias, float* state, float* out, float* scratch,
                                     const int* seg_q_start, const int* seg_slot, int segments, int chunks, int H, int D, int V,
                                     cudaStream_t stream) {
    MRUN_REQUIRE(segments >= 0 && segments <= 65535 && group > 0 && H % group == 0, "chunked_delta_scan: bad sizes");
    MRUN_REQUIRE(mrun_chunked_scan_floats(1, q, k, v, ld, MRUN_BF16, a, dt_bias, state, out, chunks, H, D, V) > 0 &&
                     (((uintptr_t)scratch) & 15) == 0,
                 "chunked_delta_scan: these sizes or rows have no chunked form");
    if (segments == 0) return 0;
    const ChunkArgs w = {q, k, v, ld, a, dt_bias, nullptr, a_log, (const bf16*)b, ldb, group, 1.f, 0, state, out, scratch, seg_q_start,
                         seg_slot, segments, chunks, H, D, V};
    return launch_sizes<CHUNK_DELTA>(w, stream);
}
