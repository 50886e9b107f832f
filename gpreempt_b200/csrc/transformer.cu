// Memory-bound transformer layers: embedding + LayerNorm, LayerNorm, multi-head attention.
//
// They stand in for the fused take/add/layer_norm, layer_norm and batch_matmul + softmax +
// batch_matmul kernels TVM generates for the reference's BERT workload
// (scripts/compile/compile-bert.py:33-91 traces the encoder; src/executor.cpp:157-162 replays
// the kernels).  Activations are [token][channel] matrices in the split-plane format of
// act_layout.h; all arithmetic is fp32 with a fixed reduction order, every kernel walks its
// tiles through the block-level preemption loop (scripts/compile/convert_to_blp.py:39-70), so a
// preempted and resumed run is bit-identical to an uninterrupted one.
#include "layers.cuh"

#include <algorithm>
#include <type_traits>

namespace gpx {

constexpr int kTfThreads = 256;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int sh = 16; sh >= 1; sh >>= 1) v += __shfl_xor_sync(0xffffffffu, v, sh);
    return v;
}

// Eight channels of a row as four pairs (the packed instructions halve the arithmetic of a row).
struct Vec8 {
    float2 v[4];
};
template <bool TWO>
__device__ __forceinline__ Vec8 vec8_decode(const uint4 &a, const uint4 &b, int fmt) {
    float x[8];
    planes_decode8(a, b, TWO ? (int)PF_SPLIT : fmt, x);
    return {{{x[0], x[1]}, {x[2], x[3]}, {x[4], x[5]}, {x[6], x[7]}}};
}
__device__ __forceinline__ Vec8 vec8_load(const float *p) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    return {{{a.x, a.y}, {a.z, a.w}, {b.x, b.y}, {b.z, b.w}}};
}
__device__ __forceinline__ Vec8 vec8_zero() { return {}; }
__device__ __forceinline__ void vec8_add(Vec8 &a, const Vec8 &b) {
#pragma unroll
    for (int j = 0; j < 4; ++j) a.v[j] = add2(a.v[j], b.v[j]);
}
__device__ __forceinline__ float vec8_sum(const Vec8 &a) {
    const float2 s = add2(add2(a.v[0], a.v[1]), add2(a.v[2], a.v[3]));
    return s.x + s.y;
}
// a - mean, and the sum of its squares
__device__ __forceinline__ float vec8_centre(Vec8 &a, float mean) {
    const float2 m = make_float2(-mean, -mean);
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        a.v[j] = add2(a.v[j], m);
        s = fma2(a.v[j], a.v[j], s);
    }
    return s.x + s.y;
}
// a * rstd * gamma + beta, stored
template <bool TWO>
__device__ __forceinline__ void vec8_finish(const LayerNormParams &p, Vec8 &a, float rstd, const Vec8 &gamma, const Vec8 &beta, size_t off) {
    float x[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 y = fma2(mul2(a.v[j], make_float2(rstd, rstd)), gamma.v[j], beta.v[j]);
        x[2 * j] = y.x, x[2 * j + 1] = y.y;
    }
    if (p.out_f32) {
        float4 *o = reinterpret_cast<float4 *>(p.out_f32 + off);
        o[0] = make_float4(x[0], x[1], x[2], x[3]);
        o[1] = make_float4(x[4], x[5], x[6], x[7]);
    } else {
        planes_store8(p.out_hi, p.out_lo, off, TWO ? (int)PF_SPLIT : p.fmt, x);
    }
}

// What a lane fetches of a row before it is worked on: eight channels in planes, or of the word's embedding.
template <bool TWO, bool EMB>
struct RawVec {
    uint4 a, b;
};
template <bool TWO, bool EMB>
__device__ __forceinline__ void raw_fetch(const LayerNormParams &p, int row, int v, RawVec<TWO, EMB> &r) {
    if (EMB) {
        const uint4 *w = reinterpret_cast<const uint4 *>(p.word + (size_t)p.ids[row] * p.H + v * 8);
        r.a = w[0], r.b = w[1];
    } else {
        planes_fetch8(p.in_hi, p.in_lo, (size_t)row * p.H + v * 8, TWO ? (int)PF_SPLIT : p.fmt, r.a, r.b);
    }
}
// word + position (+ token type 0 where the model has that table), or the row as it is
template <bool TWO, bool EMB>
__device__ __forceinline__ Vec8 raw_decode(const LayerNormParams &p, int row, int v, const RawVec<TWO, EMB> &r) {
    if (!EMB) return vec8_decode<TWO>(r.a, r.b, p.fmt);
    auto f = [](unsigned u) { return __uint_as_float(u); };
    Vec8 x = {{{f(r.a.x), f(r.a.y)}, {f(r.a.z), f(r.a.w)}, {f(r.b.x), f(r.b.y)}, {f(r.b.z), f(r.b.w)}}};
    vec8_add(x, vec8_load(p.pos + (size_t)(row % p.S) * p.H + v * 8));
    if (p.type) vec8_add(x, vec8_load(p.type + v * 8));
    return x;
}

// Many rows: one row a warp (NV 8-channel vectors a lane), eight rows a tile.  Bound by memory in principle
// (a row is read and written once); what it waits for in practice is latency, so the next tile's rows are on
// their way while this tile's are worked on, the claim after that is in flight beside them, gamma and
// beta lie in shared memory, and the arithmetic is packed.  16 384 rows of 768 bf16: 18.9 us with a claim and a
// load per tile and scalar arithmetic, 15.2 like this (14.5 to 16.1 over the layers of BERT).  When the word goes up a CTA has up to three tiles to run (this one,
// the next and the one just claimed): 6.0 us in the middle and 6.8 at most from the word being seen to the end.
template <int NV, bool TWO, bool EMB>
__global__ void __launch_bounds__(kTfThreads, NV <= 3 && !EMB ? 3 : 2)
layernorm_kernel(const __grid_constant__ LayerNormParams p, BlpArgs blp) {
    __shared__ __align__(16) float s_gamma[256 * NV], s_beta[256 * NV];
    __shared__ int s_tile[kClaimSlots];
    // (parameters: no kernel writes them, so they are fetched while the predecessor drains)
    for (int i = threadIdx.x; i < p.H / 4; i += kTfThreads) {
        reinterpret_cast<float4 *>(s_gamma)[i] = __ldg(reinterpret_cast<const float4 *>(p.gamma) + i);
        reinterpret_cast<float4 *>(s_beta)[i] = __ldg(reinterpret_cast<const float4 *>(p.beta) + i);
    }
    pdl_enter();
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int V = p.H / 8;
    int iter = 0, tile, next;
    if (dynamic) {
        if (threadIdx.x == 0) {
            const int first = blp_claim(blp, 0);
            s_tile[claim_slot(0)] = first;
            s_tile[claim_slot(1)] = first >= 0 ? blp_claim(blp, 1) : -1;
        }
        __syncthreads();
        tile = s_tile[claim_slot(0)], next = s_tile[claim_slot(1)];
    } else {
        __syncthreads();
        tile = blp_claim(blp, 0), next = blp_claim(blp, 1);
    }
    RawVec<TWO, EMB> now[NV], ahead[NV];
    auto fetch = [&](int t, RawVec<TWO, EMB> (&raw)[NV]) {
        const int row = t * (kTfThreads / 32) + wid;
#pragma unroll
        for (int i = 0; i < NV; ++i)
            if (t >= 0 && row < p.rows && lane + 32 * i < V) raw_fetch<TWO, EMB>(p, row, lane + 32 * i, raw[i]);
    };
    fetch(tile, now);
    while (tile >= 0) {
        fetch(next, ahead);
        int after = -1;
        if (next >= 0 && (!dynamic || threadIdx.x == 0)) after = blp_claim(blp, iter + 2);
        const int row = tile * (kTfThreads / 32) + wid;
        if (row < p.rows) {
            Vec8 x[NV];
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                x[i] = lane + 32 * i < V ? raw_decode<TWO, EMB>(p, row, lane + 32 * i, now[i]) : vec8_zero();
                s += vec8_sum(x[i]);
            }
            const float mean = warp_sum(s) / (float)p.H;
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if (lane + 32 * i < V) ss += vec8_centre(x[i], mean);
            const float rstd = rsqrtf(warp_sum(ss) / (float)p.H + p.eps);
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const int v = lane + 32 * i;
                if (v < V) vec8_finish<TWO>(p, x[i], rstd, vec8_load(s_gamma + v * 8), vec8_load(s_beta + v * 8), (size_t)row * p.H + v * 8);
            }
        }
        ++iter;
        if (dynamic && next >= 0) {  // (next is the same for the whole CTA)
            if (threadIdx.x == 0) s_tile[claim_slot(iter + 1)] = after;
            __syncthreads();
            after = s_tile[claim_slot(iter + 1)];
        }
        tile = next, next = after;
#pragma unroll
        for (int i = 0; i < NV; ++i) now[i] = ahead[i];
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

// Few rows (a latency-critical request): a row is a chain of loads, sums and roundings, so it is cut over NV
// warps with one vector a lane, and its scale and shift are in registers before the predecessor ends.
// 128 rows of 768 fp16: 3.3 us with a warp to a row, 1.2 like this.
template <int NV>
constexpr int ln_few_rows() { return NV == 1 ? 8 : (NV == 2 ? 4 : 2); }
template <int NV, bool TWO, bool EMB>
__global__ void __launch_bounds__(32 * NV * ln_few_rows<NV>())
layernorm_few_kernel(const __grid_constant__ LayerNormParams p, BlpArgs blp) {
    constexpr int kRows = ln_few_rows<NV>();
    __shared__ float s_sum[kRows * NV], s_sq[kRows * NV];
    __shared__ int s_tile;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int V = p.H / 8;
    const int r = wid / NV, v = (wid - r * NV) * 32 + lane;
    Vec8 gamma = vec8_zero(), beta = vec8_zero();
    if (v < V) gamma = vec8_load(p.gamma + v * 8), beta = vec8_load(p.beta + v * 8);
    pdl_enter();
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    auto row_sum = [&](float s, float *part) {
        s = warp_sum(s);
        if (NV == 1) return s;
        if (lane == 0) part[wid] = s;
        __syncthreads();
        float all = part[r * NV];
#pragma unroll
        for (int i = 1; i < NV; ++i) all += part[r * NV + i];
        return all;
    };
    int iter = 0;
    for (;; ++iter) {
        int tile;
        if (dynamic) {
            if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        const int row = tile * kRows + r;
        const bool live = row < p.rows && v < V;
        Vec8 x = vec8_zero();
        if (live) {
            RawVec<TWO, EMB> raw;
            raw_fetch<TWO, EMB>(p, row, v, raw);
            x = raw_decode<TWO, EMB>(p, row, v, raw);
        }
        const float mean = row_sum(vec8_sum(x), s_sum) / (float)p.H;
        float ss = 0.f;
        if (live) ss = vec8_centre(x, mean);
        const float rstd = rsqrtf(row_sum(ss, s_sq) / (float)p.H + p.eps);
        if (live) vec8_finish<TWO>(p, x, rstd, gamma, beta, (size_t)row * p.H + v * 8);
        if (dynamic) __syncthreads();  // s_tile
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

static int layernorm_vectors(int H) { return (H + 255) / 256; }

// The instance for a width, format and kind of input, as f(kernel, threads).
template <typename F>
static auto layernorm_instance(const LayerNormParams &p, F &&f) {
    auto width = [&](auto two, auto emb) {
        constexpr bool T = decltype(two)::value, E = decltype(emb)::value;
        const bool few = p.few_rows != 0;
        switch (layernorm_vectors(p.H)) {
            case 1: return few ? f(layernorm_few_kernel<1, T, E>, 32 * ln_few_rows<1>()) : f(layernorm_kernel<1, T, E>, kTfThreads);
            case 2: return few ? f(layernorm_few_kernel<2, T, E>, 64 * ln_few_rows<2>()) : f(layernorm_kernel<2, T, E>, kTfThreads);
            case 3: return few ? f(layernorm_few_kernel<3, T, E>, 96 * ln_few_rows<3>()) : f(layernorm_kernel<3, T, E>, kTfThreads);
            default: return few ? f(layernorm_few_kernel<4, T, E>, 128 * ln_few_rows<4>()) : f(layernorm_kernel<4, T, E>, kTfThreads);
        }
    };
    if (p.ids) return p.fmt == PF_SPLIT ? width(std::true_type(), std::true_type()) : width(std::false_type(), std::true_type());
    return p.fmt == PF_SPLIT ? width(std::true_type(), std::false_type()) : width(std::false_type(), std::false_type());
}

// A row over several warps up to 32 rows an SM: with fewer the chain is what counts, with more the loads under
// way are.  One warp a row against several, 768 channels: 2 048 rows bf16 4.3 / 4.0 us, 4 096 rows 6.5 / 5.7 and
// float32 8.4 / 6.6, 16 384 rows 15.2 / 16.6.
void layernorm_plan(LayerNormParams &p, int sm_count, int &grid, int &threads) {
    p.few_rows = p.rows <= 32 * sm_count;
    const int nv = layernorm_vectors(p.H);
    const int rows = !p.few_rows ? kTfThreads / 32 : (nv == 1 ? ln_few_rows<1>() : (nv == 2 ? ln_few_rows<2>() : ln_few_rows<3>()));
    p.total_tiles = (p.rows + rows - 1) / rows;
    int per_sm = 1;
    threads = layernorm_instance(p, [&](auto kernel, int t) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, t, 0);
        return t;
    });
    grid = (int)std::min<long long>((long long)sm_count * std::max(per_sm, 1), p.total_tiles);
}

cudaError_t layernorm_launch(const LayerNormParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    return layernorm_instance(p, [&](auto kernel, int threads) { return launch_layer(kernel, grid, threads, 0, s, p, blp); });
}

// ---- multi-head attention ---------------------------------------------------------------------

constexpr int kAttnThreads = 128;  // 32 queries x 4 key partitions
constexpr int kAttnKeys = 64;      // keys per shared-memory block
constexpr int kAttnDh = 64;        // head dimension
constexpr int kAttnLd = kAttnDh + 4;

// softmax(Q K^T / sqrt(d)) V for one (batch, head, block of 32 queries) per tile.  Four lanes
// share a query: lane `part` walks keys part, part+4, ... of every 64-key block with an online
// softmax (running maximum m, normaliser l, weighted sum o), the four partial results are merged
// in a fixed order by shuffles.
__global__ void __launch_bounds__(kAttnThreads)
attention_kernel(const __grid_constant__ AttnParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    __shared__ __align__(16) float Ks[kAttnKeys][kAttnLd];
    __shared__ __align__(16) float Vs[kAttnKeys][kAttnLd];
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int tid = threadIdx.x;
    const int qi = tid >> 2, part = tid & 3;
    const int qblocks = (p.S + 31) / 32;
    int iter = 0;
    for (;;) {
        int tile;
        if (dynamic) {
            if (tid == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        const int qb = tile % qblocks;
        const int head = (tile / qblocks) % p.heads;
        const int b = tile / (qblocks * p.heads);
        const int qrow = qb * 32 + qi;
        const bool qvalid = qrow < p.S;
        const size_t col = (size_t)head * kAttnDh;
        float q[kAttnDh], o[kAttnDh];
#pragma unroll
        for (int d = 0; d < kAttnDh; ++d) o[d] = 0.f;
        {
            const size_t off = ((size_t)b * p.S + (qvalid ? qrow : 0)) * p.ld + col;
#pragma unroll
            for (int v = 0; v < kAttnDh / 8; ++v) {
                float x[8];
                planes_load8(p.q_hi, p.q_lo, off + v * 8, p.fmt, x);
#pragma unroll
                for (int j = 0; j < 8; ++j) q[v * 8 + j] = x[j] * p.scale;
            }
        }
        float m = -INFINITY, l = 0.f;
        for (int k0 = 0; k0 < p.S; k0 += kAttnKeys) {
            // stage 64 keys and values of this head as fp32
            for (int e = tid; e < kAttnKeys * (kAttnDh / 8); e += kAttnThreads) {
                const int kr = e / (kAttnDh / 8), v = e % (kAttnDh / 8);
                float kx[8], vx[8];
                if (k0 + kr < p.S) {
                    const size_t off = ((size_t)b * p.S + k0 + kr) * p.ld + col + v * 8;
                    planes_load8(p.k_hi, p.k_lo, off, p.fmt, kx);
                    planes_load8(p.v_hi, p.v_lo, off, p.fmt, vx);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) kx[j] = vx[j] = 0.f;
                }
                *reinterpret_cast<float4 *>(&Ks[kr][v * 8]) = make_float4(kx[0], kx[1], kx[2], kx[3]);
                *reinterpret_cast<float4 *>(&Ks[kr][v * 8 + 4]) = make_float4(kx[4], kx[5], kx[6], kx[7]);
                *reinterpret_cast<float4 *>(&Vs[kr][v * 8]) = make_float4(vx[0], vx[1], vx[2], vx[3]);
                *reinterpret_cast<float4 *>(&Vs[kr][v * 8 + 4]) = make_float4(vx[4], vx[5], vx[6], vx[7]);
            }
            __syncthreads();
            for (int j = part; j < kAttnKeys; j += 4) {
                if (k0 + j >= p.S) break;
                float sc = 0.f;
#pragma unroll
                for (int d = 0; d < kAttnDh; d += 4) {
                    float4 kv = *reinterpret_cast<const float4 *>(&Ks[j][d]);
                    sc = fmaf(q[d], kv.x, sc);
                    sc = fmaf(q[d + 1], kv.y, sc);
                    sc = fmaf(q[d + 2], kv.z, sc);
                    sc = fmaf(q[d + 3], kv.w, sc);
                }
                if (sc > m) {
                    const float corr = __expf(m - sc);  // 0 on the first key (m = -inf)
                    l *= corr;
#pragma unroll
                    for (int d = 0; d < kAttnDh; ++d) o[d] *= corr;
                    m = sc;
                }
                const float w = __expf(sc - m);
                l += w;
#pragma unroll
                for (int d = 0; d < kAttnDh; d += 4) {
                    float4 vv = *reinterpret_cast<const float4 *>(&Vs[j][d]);
                    o[d] = fmaf(w, vv.x, o[d]);
                    o[d + 1] = fmaf(w, vv.y, o[d + 1]);
                    o[d + 2] = fmaf(w, vv.z, o[d + 2]);
                    o[d + 3] = fmaf(w, vv.w, o[d + 3]);
                }
            }
            __syncthreads();
        }
        // merge the four partitions of a query (lanes 4q .. 4q+3)
        float mm = m;
        mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, 1));
        mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, 2));
        const float corr = m == -INFINITY ? 0.f : __expf(m - mm);
        l *= corr;
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        const float inv = 1.0f / l;
        float mine[16];
#pragma unroll
        for (int d = 0; d < kAttnDh; ++d) {
            float v = o[d] * corr;
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if ((d >> 4) == part) mine[d & 15] = v * inv;
        }
        if (qvalid) {
            const size_t off = ((size_t)b * p.S + qrow) * p.ld_out + col + part * 16;
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = mine[v * 8 + j];
                planes_store8(p.out_hi, p.out_lo, off + v * 8, p.fmt, x);
            }
        }
        ++iter;
    }
    if (tid == 0) trace_end(blp, iter);
}

// The same for sequences of at most 64 tokens, where a request is a chain of latencies: eight queries of a head per
// tile, a warp to a query.  Keys and values are staged once, a lane scores the keys `lane` and `lane` + 32, the
// softmax is two warp reductions, and for the weighted sum a lane owns two of the 64 channels.
// Six tokens, 12 heads: 5.7 us with four lanes to a query walking the keys one by one, 2.0 like this.
constexpr int kShortKeys = 64, kShortQueries = 8;
__global__ void __launch_bounds__(32 * kShortQueries)
attention_short_kernel(const __grid_constant__ AttnParams p, BlpArgs blp) {
    __shared__ int s_tile;
    __shared__ __align__(16) float s_k[kShortKeys][kAttnLd], s_v[kShortKeys][kAttnDh], s_q[kShortQueries][kAttnDh];
    pdl_enter();
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int qblocks = (p.S + kShortQueries - 1) / kShortQueries;
    const int vecs = p.S * (kAttnDh / 8);  // of the keys, and of the values
    constexpr int kLoads = kShortKeys * (kAttnDh / 8) / (32 * kShortQueries);
    int iter = 0;
    for (;; ++iter) {
        int tile;
        if (dynamic) {
            if (tid == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        const int qb = tile % qblocks;
        const int head = (tile / qblocks) % p.heads;
        const int b = tile / (qblocks * p.heads);
        const int qrow = qb * kShortQueries + wid;
        const size_t col = (size_t)head * kAttnDh, row0 = (size_t)b * p.S;
        // every load of the tile is requested before any is converted
        uint4 kh[kLoads], kl[kLoads], vh[kLoads], vl[kLoads];
        unsigned qh = 0, ql = 0;
        const size_t q_at = (row0 + (qrow < p.S ? qrow : 0)) * p.ld + col + 2 * lane;
        qh = *reinterpret_cast<const unsigned *>(p.q_hi + q_at);
        if (p.fmt == PF_SPLIT) ql = *reinterpret_cast<const unsigned *>(p.q_lo + q_at);
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int e = tid + i * 32 * kShortQueries;
            if (e < vecs) {
                const size_t off = (row0 + e / (kAttnDh / 8)) * p.ld + col + e % (kAttnDh / 8) * 8;
                planes_fetch8(p.k_hi, p.k_lo, off, p.fmt, kh[i], kl[i]);
                planes_fetch8(p.v_hi, p.v_lo, off, p.fmt, vh[i], vl[i]);
            }
        }
        float2 q2 = pf_unpack2(qh, p.fmt);
        if (p.fmt == PF_SPLIT) q2.x += __uint_as_float(ql << 16), q2.y += __uint_as_float(ql & 0xffff0000u);
        *reinterpret_cast<float2 *>(&s_q[wid][2 * lane]) = make_float2(q2.x * p.scale, q2.y * p.scale);
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
            const int e = tid + i * 32 * kShortQueries;
            if (e < vecs) {
                const int kr = e / (kAttnDh / 8), c = e % (kAttnDh / 8) * 8;
                float x[8];
                planes_decode8(kh[i], kl[i], p.fmt, x);
                *reinterpret_cast<float4 *>(&s_k[kr][c]) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4 *>(&s_k[kr][c + 4]) = make_float4(x[4], x[5], x[6], x[7]);
                planes_decode8(vh[i], vl[i], p.fmt, x);
                *reinterpret_cast<float4 *>(&s_v[kr][c]) = make_float4(x[0], x[1], x[2], x[3]);
                *reinterpret_cast<float4 *>(&s_v[kr][c + 4]) = make_float4(x[4], x[5], x[6], x[7]);
            }
        }
        __syncthreads();
        if (qrow < p.S) {
            float sc[2];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int key = lane + 32 * half;
                sc[half] = -INFINITY;
                if (key >= p.S) continue;
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int d = 0; d < kAttnDh; d += 4) {
                    const float4 kv = *reinterpret_cast<const float4 *>(&s_k[key][d]);
                    const float4 qv = *reinterpret_cast<const float4 *>(&s_q[wid][d]);
                    a.x = fmaf(qv.x, kv.x, a.x), a.y = fmaf(qv.y, kv.y, a.y);
                    a.z = fmaf(qv.z, kv.z, a.z), a.w = fmaf(qv.w, kv.w, a.w);
                }
                sc[half] = (a.x + a.y) + (a.z + a.w);
            }
            float m = fmaxf(sc[0], sc[1]);
#pragma unroll
            for (int sh = 16; sh >= 1; sh >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, sh));
            const float w0 = __expf(sc[0] - m), w1 = __expf(sc[1] - m);  // (0 for keys past the sequence)
            const float inv = 1.0f / warp_sum(w0 + w1);
            float2 o = make_float2(0.f, 0.f);
            for (int j = 0; j < p.S; ++j) {
                const float w = __shfl_sync(0xffffffffu, j < 32 ? w0 : w1, j & 31);
                o = fma2(make_float2(w, w), *reinterpret_cast<const float2 *>(&s_v[j][2 * lane]), o);
            }
            o.x *= inv, o.y *= inv;
            const size_t off = (row0 + qrow) * p.ld_out + col + 2 * lane;
            const unsigned hi = pf_pack2(o.x, o.y, p.fmt);
            *reinterpret_cast<unsigned *>(p.out_hi + off) = hi;
            if (p.fmt == PF_SPLIT)
                *reinterpret_cast<unsigned *>(p.out_lo + off) =
                    pf_pack2(o.x - __uint_as_float(hi << 16), o.y - __uint_as_float(hi & 0xffff0000u), PF_SPLIT);
        }
        __syncthreads();  // the staging area and the tile number are rewritten
    }
    if (tid == 0) trace_end(blp, iter);
}

// Tiles, form and threads of a launch.  The short form wherever it applies, except for many sequences of more
// than 48 tokens, whose keys it stages four times as often (12 heads, us a layer, walking the keys / short: 32
// sequences of 6 tokens 12.3 / 4.0, 32 of 33 36 / 25, 1 of 40 11.6 / 3.4, 48 of 64 71 / 79).  The line at six tiles an SM:
// DistilBERT float32, us a latency-critical request of 8, 10 and 12 sequences, 64 tokens 451 / 428, 482 / 484 and 495 / 533, 58 tokens
// 437 / 417, 468 / 469 and 487 / 536, 52 tokens (a tile fewer of eight) 426 / 413, 453 / 444 and 469 / 474.
void attention_plan(AttnParams &p, int sm_count, int &threads) {
    const int short_tiles = p.B * p.heads * ((p.S + kShortQueries - 1) / kShortQueries);
    p.few_keys = p.S <= 48 || (p.S <= kShortKeys && short_tiles <= 6 * sm_count);
    p.total_tiles = p.few_keys ? short_tiles : p.B * p.heads * ((p.S + 31) / 32);
    threads = p.few_keys ? 32 * kShortQueries : kAttnThreads;
}

cudaError_t attention_launch(const AttnParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    if (p.few_keys) return launch_layer(attention_short_kernel, grid, 32 * kShortQueries, 0, s, p, blp);
    return launch_layer(attention_kernel, grid, kAttnThreads, 0, s, p, blp);
}

}  // namespace gpx
