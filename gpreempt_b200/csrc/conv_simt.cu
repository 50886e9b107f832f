// Convolution / dense layer as an implicit GEMM on the CUDA cores (fp32 FFMA), pooling and
// sub-sampling; block-level preemption at output-tile granularity.
//
// These kernels cover what the tensor-core convolution does not: the stem (fp32 NCHW input with
// three channels), dense layers with a handful of rows, and the memory-bound layers.  They stand
// in for TVM-generated fused kernels the reference replays (src/executor.cpp:157-162); the
// preemption loop is the native form of scripts/compile/convert_to_blp.py:39-70.
//
// One FFMA per multiply-add with K walked in increasing order inside one thread, so the result
// does not depend on which CTA runs a tile: preempt + resume is bit-identical.
#include "layers.cuh"

#include <algorithm>

namespace gpx {

constexpr int kConvThreads = 256;
constexpr int kConvBK = 16;

__device__ __forceinline__ float bf16_bits_to_f32(bf16_bits v) {
    return __uint_as_float((unsigned)v << 16);
}
__device__ __forceinline__ bf16_bits f32_to_bf16_bits(float f) {
    unsigned u = __float_as_uint(f);
    u += 0x7fffu + ((u >> 16) & 1u);  // round to nearest even (finite inputs)
    return (bf16_bits)(u >> 16);
}

__device__ __forceinline__ float view_load(const ActView &v, int n, int h, int w, int c) {
    if (v.f32) return v.f32[(((size_t)n * v.l.C + c) * v.l.H + h) * v.l.W + w];
    size_t off = (size_t)layout_row(v.l, n, h, w) * v.l.C + c;
    return planes_load1(v.hi, v.lo, off, v.l.fmt);
}

template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(kConvThreads)
conv_simt_kernel(const __grid_constant__ ConvParams p, BlpArgs blp) {
    pdl_enter();
    constexpr int BK = kConvBK;
    static_assert((BM / TM) * (BN / TN) == kConvThreads, "thread layout");
    constexpr int SB = (BN * 4 + kConvThreads - 1) / kConvThreads;  // float4 slots of B per thread
    constexpr int EA = BM / 16;                                      // A elements per thread

    __shared__ __align__(16) float As[2][BK][BM + 4];
    __shared__ __align__(16) float Bs[2][BK][BN + 4];
    __shared__ int s_tile;

    const int tid = threadIdx.x;
    const int tx = tid % (BN / TN);
    const int ty = tid / (BN / TN);
    const int nchunks = (p.K + BK - 1) / BK;
    const bool dynamic = blp.preempted != nullptr;
    const int H = p.in.l.H, W = p.in.l.W;

    if (tid == 0) trace_begin(blp);
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
        const int m0 = (tile % p.tiles_m) * BM;
        const int n0 = (tile / p.tiles_m) * BN;

        // Output pixel of the A row this thread stages; fixed for the whole tile.
        int row_n, row_h, row_w;
        {
            int m = m0 + tid % BM;
            bool ok = m < p.M;
            int mm = ok ? m : 0;
            int wo = mm % p.Wo;
            int t = mm / p.Wo;
            int ho = t % p.Ho;
            row_n = ok ? t / p.Ho : -1;
            row_h = ho * p.stride - p.pad;
            row_w = wo * p.stride - p.pad_w;
        }

        float ra[EA];
        float4 rb[SB];

        auto load_chunk = [&](int c) {
            const int k0 = c * BK;
#pragma unroll
            for (int e = 0; e < EA; ++e) {
                int kk = tid / BM + e * (kConvThreads / BM);
                int k = k0 + kk;
                float v = 0.f;
                if (k < p.K && row_n >= 0) {
                    int tap = k / p.Cin;
                    int ci = k - tap * p.Cin;
                    int fh = tap / p.kw;
                    int fw = tap - fh * p.kw;
                    int hi = row_h + fh, wi = row_w + fw;
                    if (hi >= 0 && hi < H && wi >= 0 && wi < W) v = view_load(p.in, row_n, hi, wi, ci);
                }
                ra[e] = v;
            }
#pragma unroll
            for (int j = 0; j < SB; ++j) {
                int i = tid + j * kConvThreads;
                int kk = i / (BN / 4);
                int c4 = i - kk * (BN / 4);
                int k = k0 + kk;
                int n = n0 + c4 * 4;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < BN * 4 && k < p.K && n < p.Cout)
                    v = *reinterpret_cast<const float4 *>(p.w + (size_t)k * p.Cout + n);
                rb[j] = v;
            }
        };

        auto store_chunk = [&](int buf) {
#pragma unroll
            for (int e = 0; e < EA; ++e) {
                int kk = tid / BM + e * (kConvThreads / BM);
                As[buf][kk][tid % BM] = ra[e];
            }
#pragma unroll
            for (int j = 0; j < SB; ++j) {
                int i = tid + j * kConvThreads;
                if (i < BN * 4) {
                    int kk = i / (BN / 4);
                    int c4 = i - kk * (BN / 4);
                    *reinterpret_cast<float4 *>(&Bs[buf][kk][c4 * 4]) = rb[j];
                }
            }
        };

        float acc[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

        load_chunk(0);
        store_chunk(0);
        __syncthreads();
        for (int c = 0; c < nchunks; ++c) {
            const int buf = c & 1;
            if (c + 1 < nchunks) load_chunk(c + 1);
#pragma unroll
            for (int k = 0; k < BK; ++k) {
                float a[TM], b[TN];
#pragma unroll
                for (int i = 0; i < TM; ++i) a[i] = As[buf][k][ty * TM + i];
#pragma unroll
                for (int j = 0; j < TN; ++j) b[j] = Bs[buf][k][tx * TN + j];
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            }
            if (c + 1 < nchunks) store_chunk(buf ^ 1);
            __syncthreads();
        }

        // Epilogue: + bias, + residual, ReLU; rows go to the consumer's layout.
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            int m = m0 + ty * TM + i;
            if (m >= p.M) continue;
            int wo = m % p.Wo;
            int t = m / p.Wo;
            int ho = t % p.Ho;
            int n_img = t / p.Ho;
            size_t out_row = p.out_f32 ? (size_t)m : (size_t)layout_row(p.out, n_img, ho, wo);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                int n = n0 + tx * TN + j;
                if (n >= p.Cout) continue;
                float v = acc[i][j];
                if (p.bias) v += p.bias[n];
                if (p.res.hi || p.res.f32) v += view_load(p.res, n_img, ho, wo, n);
                v = apply_act(v, p.relu);
                if (p.out_f32) {
                    p.out_f32[out_row * p.Cout + n] = v;
                } else {
                    // the row stride is the stored channel count, which may exceed Cout
                    planes_store1(p.out_hi, p.out_lo, out_row * p.out.C + n, p.out.fmt, v);
                }
            }
        }
        ++iter;
    }
    if (tid == 0) trace_end(blp, iter);
}

static void tile_dims(int tile, int &bm, int &bn) {
    switch (tile) {
        case CONV_TILE_128: bm = 128; bn = 128; break;
        case CONV_TILE_64: bm = 64; bn = 64; break;
        default: bm = 32; bn = 32; break;
    }
}

void conv_set_tiles(ConvParams &p, int tile) {
    int bm, bn;
    tile_dims(tile, bm, bn);
    p.tiles_m = (p.M + bm - 1) / bm;
    p.tiles_n = (p.Cout + bn - 1) / bn;
}

int conv_pick_tile(const ConvParams &p, int sm_count) {
    // Largest tile that still yields about two waves of CTAs; small-M layers fall through to
    // the smallest tile to expose parallelism.
    for (int tile = CONV_TILE_128; tile <= CONV_TILE_32; ++tile) {
        int bm, bn;
        tile_dims(tile, bm, bn);
        long long tiles = (long long)((p.M + bm - 1) / bm) * ((p.Cout + bn - 1) / bn);
        if (tiles >= 2LL * sm_count || tile == CONV_TILE_32) return tile;
    }
    return CONV_TILE_32;
}

template <int BM, int BN, int TM, int TN>
static int occupancy() {
    static int v = 0;
    if (!v) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, conv_simt_kernel<BM, BN, TM, TN>,
                                                          kConvThreads, 0) != cudaSuccess ||
            v < 1)
            v = 1;
    }
    return v;
}

int conv_grid(const ConvParams &p, int tile, int sm_count) {
    long long tiles = (long long)p.tiles_m * p.tiles_n;
    int occ = tile == CONV_TILE_128   ? occupancy<128, 128, 8, 8>()
              : tile == CONV_TILE_64 ? occupancy<64, 64, 4, 4>()
                                     : occupancy<32, 32, 2, 2>();
    // Persistent grid: min(total tiles, resident CTAs), as Model::add_block_preemption_param
    // sizes it in the reference (src/model.cpp:373-385).
    long long grid = (long long)sm_count * occ;
    if (grid > tiles) grid = tiles;
    if (grid < 1) grid = 1;
    return (int)grid;
}

cudaError_t conv_launch(const ConvParams &p, int tile, int grid, const BlpArgs &blp,
                        cudaStream_t s) {
    switch (tile) {
        case CONV_TILE_128:
            return launch_layer(conv_simt_kernel<128, 128, 8, 8>, grid, kConvThreads, 0, s, p, blp);
        case CONV_TILE_64:
            return launch_layer(conv_simt_kernel<64, 64, 4, 4>, grid, kConvThreads, 0, s, p, blp);
        default:
            return launch_layer(conv_simt_kernel<32, 32, 2, 2>, grid, kConvThreads, 0, s, p, blp);
    }
}

// ---- pooling / sub-sampling ---------------------------------------------------------------

constexpr int kPoolThreads = 256;

// Eight channels of one input pixel as fp32: the sum of the planes, then the optional
// per-channel affine + activation of PoolParams.
__device__ __forceinline__ void pool_load8(const PoolParams &p, size_t off, int c0, float (&x)[8]) {
    planes_load8(p.in.hi, p.in.lo, off, p.in.l.fmt, x);
    if (p.scale) {
        const float4 *sc = reinterpret_cast<const float4 *>(p.scale + c0);
        const float4 *sh = reinterpret_cast<const float4 *>(p.shift + c0);
        float4 s0 = __ldg(sc), s1 = __ldg(sc + 1), h0 = __ldg(sh), h1 = __ldg(sh + 1);
        const float sv[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        const float hv[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = fmaf(x[j], sv[j], hv[j]);
        apply_act_n(x, p.act);
    }
}

__device__ __forceinline__ void pool_store8(const PoolParams &p, size_t off, const float (&x)[8]) {
    planes_store8(p.out_hi, p.out_lo, off, p.out.fmt, x);
}

// The tiles of a CTA.  Under the preemptible schedule a claim is two dependent round trips to L2 (the
// word, the cursor), more than a tile of 256 vectors takes; ahead(), called once the loads of a tile are
// on their way, claims the following tile while they travel.  The tile so claimed is run whatever the
// word says by then: a CTA leaves after at most two tiles instead of one, a few microseconds.
struct TileClaims {
    const BlpArgs &blp;
    const bool dynamic;
    int &s_tile;  // shared
    int iter = 0, upcoming = 0;
    bool asked = false;
    __device__ __forceinline__ TileClaims(const BlpArgs &b, bool d, int &s) : blp(b), dynamic(d), s_tile(s) {}
    __device__ __forceinline__ int first() {
        if (!dynamic) return blp_claim(blp, 0);
        if (threadIdx.x == 0) s_tile = blp_claim(blp, 0);
        __syncthreads();
        return s_tile;
    }
    __device__ __forceinline__ void ahead() {
        if (dynamic && threadIdx.x == 0 && !asked) {
            upcoming = blp_claim(blp, iter + 1);
            asked = true;
        }
    }
    __device__ __forceinline__ int next() {
        ++iter;
        if (!dynamic) return blp_claim(blp, iter);
        __syncthreads();  // every thread has read this round's number
        if (threadIdx.x == 0) s_tile = asked ? upcoming : blp_claim(blp, iter);
        asked = false;
        __syncthreads();
        return s_tile;
    }
    __device__ __forceinline__ int done() const { return iter; }
};

// 3x3 max pooling (K = 3) and 2x2 pooling of either kind (K = 2), without an affine map.  Bound by how many loads
// are under way: a thread requests all taps of its vector (of two planes, a row of them and the next one) before it
// looks at any, the largest of 16-bit values is taken as they are, and division by reciprocals keeps the
// registers of 24 to 32 warps an SM.  112x112x64, 64 images bf16, 3x3: 70 us at two CTAs an SM with fp32 maxima, 38
// like this (128 MB: 20 us); 299x299 Inception-v3 b16 fp16, first 3x3: 31 us, 14.
template <int K, bool TWO>
__global__ void __launch_bounds__(kPoolThreads, K == 3 ? (TWO ? 3 : 4) : 4)
pool_window_kernel(const __grid_constant__ PoolParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    if (threadIdx.x == 0) trace_begin(blp);
    const int C8 = p.channels / 8, H = p.in.l.H, W = p.in.l.W;
    const unsigned total = (unsigned)p.out.N * p.out.H * p.out.W * C8;  // < 2^31, checked when the model is built
    const bool plain = p.in.l.order == ACT_PLAIN, is_max = K == 3 || p.mode == 0;
    const int fmt = TWO ? (int)PF_SPLIT : p.in.l.fmt;
    TileClaims claims(blp, blp.preempted != nullptr, s_tile);
    for (int tile = claims.first(); tile >= 0; tile = claims.next()) {
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = begin + p.tile_elems < total ? begin + p.tile_elems : total;
        for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
            const unsigned px = p.by_c8.div(e), py = p.by_w.div(px), n = p.by_h.div(py);
            const int c0 = (int)(e - px * C8) * 8, wo = (int)(px - py * p.out.W), ho = (int)(py - n * p.out.H);
            const int h0 = ho * p.stride - p.pad, w0 = wo * p.stride - p.pad;
            const size_t out = (size_t)layout_row(p.out, n, ho, wo) * p.out.C + c0;
            if (c0 >= p.in_valid) {
                float zero[8] = {};
                planes_store8(p.out_hi, p.out_lo, out, TWO ? (int)PF_SPLIT : p.out.fmt, zero);
                continue;
            }
            const long long at = ((long long)((int)n * p.in.l.Hs + h0) * p.in.l.Ws + w0) * p.in.l.C + c0;
            const long long row_step = (long long)p.in.l.Ws * p.in.l.C;
            auto inside = [&](int t) { return (unsigned)(h0 + t / K) < (unsigned)H && (unsigned)(w0 + t % K) < (unsigned)W; };
            auto fetch = [&](int t, uint4 &a, uint4 &b) {
                if (!inside(t)) return;
                const long long off = plain ? at + t / K * row_step + t % K * p.in.l.C
                                            : (long long)layout_row(p.in.l, n, h0 + t / K, w0 + t % K) * p.in.l.C + c0;
                planes_fetch8(p.in.hi, p.in.lo, (size_t)off, fmt, a, b);
            };
            float acc[8];
            int cnt = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = is_max ? -INFINITY : 0.f;
            auto take = [&](const uint4 &a, const uint4 &b) {
                float x[8];
                planes_decode8(a, b, fmt, x);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = is_max ? fmaxf(acc[j], x[j]) : acc[j] + x[j];
                ++cnt;
            };
            if (TWO) {
                uint4 ra[2][K], rb[2][K];
#pragma unroll
                for (int t = 0; t < K; ++t) fetch(t, ra[0][t], rb[0][t]);
#pragma unroll
                for (int r = 0; r < K; ++r) {
                    if (r + 1 < K)
#pragma unroll
                        for (int t = 0; t < K; ++t) fetch((r + 1) * K + t, ra[(r + 1) & 1][t], rb[(r + 1) & 1][t]);
                    if (r == 0) claims.ahead();
#pragma unroll
                    for (int t = 0; t < K; ++t)
                        if (inside(r * K + t)) take(ra[r & 1][t], rb[r & 1][t]);
                }
            } else {
                uint4 ra[K * K], none;
#pragma unroll
                for (int t = 0; t < K * K; ++t) fetch(t, ra[t], none);
                claims.ahead();
                if (is_max) {
                    const unsigned low = fmt == PF_F16 ? 0xfc00fc00u : 0xff80ff80u;  // -infinity
                    uint4 m = make_uint4(low, low, low, low);
#pragma unroll
                    for (int t = 0; t < K * K; ++t)
                        if (inside(t)) {
                            m.x = max_packed(m.x, ra[t].x, fmt), m.y = max_packed(m.y, ra[t].y, fmt);
                            m.z = max_packed(m.z, ra[t].z, fmt), m.w = max_packed(m.w, ra[t].w, fmt);
                        }
                    *reinterpret_cast<uint4 *>(p.out_hi + out) = m;
                    continue;
                }
#pragma unroll
                for (int t = 0; t < K * K; ++t)
                    if (inside(t)) take(ra[t], none);
            }
            if (!is_max) {
                const float inv = 1.0f / (float)(p.mode == 1 ? cnt : K * K);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] *= inv;
            }
            planes_store8(p.out_hi, p.out_lo, out, TWO ? (int)PF_SPLIT : p.out.fmt, acc);
        }
    }
    if (threadIdx.x == 0) trace_end(blp, claims.done());
}

// Other pooling windows, pooling behind an affine map, or a strided copy, over split-plane activations; eight channels (one
// 16-byte vector per plane) per thread-iteration.  A tile is tile_elems consecutive output
// vectors in (n, ho, wo, c/8) order.
__global__ void __launch_bounds__(kPoolThreads)
pool_kernel(const __grid_constant__ PoolParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int Cin = p.in.l.C, Cout = p.out.C;  // row strides
    const int C8 = p.channels / 8;
    const int Ho = p.out.H, Wo = p.out.W;
    const int H = p.in.l.H, W = p.in.l.W;
    const unsigned total = (unsigned)p.out.N * Ho * Wo * C8;  // < 2^31, checked when the model is built
    TileClaims claims(blp, dynamic, s_tile);
    for (int tile = claims.first(); tile >= 0; tile = claims.next()) {
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = begin + p.tile_elems < total ? begin + p.tile_elems : total;
        if (p.mode == 1 && p.k * p.k >= 16) {
            // Large averaging window (global average pool): one warp per output vector, lanes
            // take taps lane, lane+32, ...; a fixed shuffle tree adds the lane sums, so the
            // result is the same on every run.
            const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
            for (unsigned e = begin + wid; e < end; e += kPoolThreads / 32) {
                int c8 = (int)(e % C8);
                unsigned t = e / C8;
                int wo = (int)(t % Wo);
                t /= Wo;
                int ho = (int)(t % Ho);
                int n = (int)(t / Ho);
                float acc[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] = 0.f;
                int cnt = 0;
                const bool readable = c8 * 8 < p.in_valid;
                for (int tap = lane; tap < p.k * p.k; tap += 32) {
                    int fh = tap / p.k, fw = tap - fh * p.k;
                    int hi = ho * p.stride - p.pad + fh, wi = wo * p.stride - p.pad + fw;
                    if (hi < 0 || hi >= H || wi < 0 || wi >= W) continue;
                    if (readable) {
                        float x[8];
                        pool_load8(p, (size_t)layout_row(p.in.l, n, hi, wi) * Cin + c8 * 8, c8 * 8, x);
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[j] += x[j];
                    }
                    ++cnt;
                }
#pragma unroll
                for (int sh = 16; sh >= 1; sh >>= 1) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], sh);
                    cnt += __shfl_xor_sync(0xffffffffu, cnt, sh);
                }
                if (lane == 0) {
                    float inv = 1.0f / (float)cnt;
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[j] *= inv;
                    pool_store8(p, (size_t)layout_row(p.out, n, ho, wo) * Cout + c8 * 8, acc);
                }
            }
            continue;
        }
        for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
            int c8 = (int)(e % C8);
            unsigned t = e / C8;
            int wo = (int)(t % Wo);
            t /= Wo;
            int ho = (int)(t % Ho);
            int n = (int)(t / Ho);
            float acc[8];
            const bool readable = c8 * 8 < p.in_valid;
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = (p.mode == 0 && readable) ? -INFINITY : 0.f;
            int cnt = 0;
            const int kk = p.mode == 2 ? 1 : p.k;
            for (int fh = 0; fh < kk; ++fh) {
                int hi = ho * p.stride - p.pad + fh;
                if (hi < 0 || hi >= H) continue;
                for (int fw = 0; fw < kk; ++fw) {
                    int wi = wo * p.stride - p.pad + fw;
                    if (wi < 0 || wi >= W) continue;
                    ++cnt;
                    if (!readable) continue;
                    float x[8];
                    pool_load8(p, (size_t)layout_row(p.in.l, n, hi, wi) * Cin + c8 * 8, c8 * 8, x);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (p.mode == 0)
                            acc[j] = fmaxf(acc[j], x[j]);
                        else
                            acc[j] += x[j];
                    }
                }
            }
            if (p.mode == 1 || p.mode == 3) {
                float inv = 1.0f / (float)(p.mode == 1 ? cnt : p.k * p.k);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] *= inv;
            }
            pool_store8(p, (size_t)layout_row(p.out, n, ho, wo) * Cout + c8 * 8, acc);
        }
    }
    if (threadIdx.x == 0) trace_end(blp, claims.done());
}

// Patch matrix for the tensor-core GEMM: one thread-iteration writes eight consecutive columns
// (one 16-byte vector per plane) of one row.
__global__ void __launch_bounds__(kPoolThreads)
im2col_kernel(const __grid_constant__ Im2colParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int K8 = p.Kp / 8;
    const unsigned total = (unsigned)p.M * K8;
    const int H = p.in.l.H, W = p.in.l.W;
    // Column k of the patch matrix is filter tap (fh, fw) of channel ci; the decomposition and,
    // for an fp32 NCHW input, the element offset relative to the window origin are tabulated
    // once per CTA (K <= 1024).
    __shared__ int s_off[1024];
    __shared__ unsigned char s_fh[1024], s_fw[1024], s_ci[1024];
    for (int k = threadIdx.x; k < p.Kp && !p.planes_vec; k += kPoolThreads) {
        int tap = k / p.Cin;
        int ci = k - tap * p.Cin;
        int fh = tap / p.kw;
        int fw = tap - fh * p.kw;
        s_fh[k] = k < p.K ? (unsigned char)fh : 255;
        s_fw[k] = (unsigned char)fw;
        s_ci[k] = (unsigned char)ci;
        s_off[k] = (ci * H + fh) * W + fw;
    }
    __syncthreads();
    int iter = 0;
    if (p.s2d) {
        // Space-to-depth windows.  One thread-iteration gathers eight of the sixteen channels of one
        // 2x2 block (hb, wb'), splits them once and stores them into the up to four pixels
        // wb' - j (j = 0..3) whose window holds that block, at channel group j.  Blocks wb' >= Wo lie
        // past the padded image and are zero; they fill the tail groups of a row's last pixels.
        const int Wx = p.Wo + 3;
        const unsigned vectors = (unsigned)p.in.l.N * p.Ho * Wx * 2;
        // channel c of a block = (dy*2 + dx)*Cin + ci: the decomposition is tabulated once
        for (int c = threadIdx.x; c < 16; c += kPoolThreads) {
            const int q = c / p.Cin;
            s_fh[c] = q < 4 ? (unsigned char)q : 255;
            s_ci[c] = (unsigned char)(c - q * p.Cin);
        }
        for (;;) {
            int tile;
            __syncthreads();
            if (dynamic) {
                if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
                __syncthreads();
                tile = s_tile;
            } else {
                tile = blp_claim(blp, iter);
            }
            if (tile < 0) break;
            const unsigned begin = (unsigned)tile * p.tile_elems;
            const unsigned end = begin + p.tile_elems < vectors ? begin + p.tile_elems : vectors;
            for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
                const int half = (int)(e & 1);
                const unsigned b = e >> 1;
                const int wb = (int)(b % Wx);
                const unsigned t = b / Wx;
                const int hb = (int)(t % p.Ho), n = (int)(t / p.Ho);
                float x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int c = half * 8 + u;
                    const int q = s_fh[c];
                    const int hi = 2 * hb + (q >> 1) - p.pad, wi = 2 * wb + (q & 1) - p.pad;
                    float v = 0.f;
                    if (q != 255 && hi >= 0 && hi < H && wi >= 0 && wi < W)
                        v = p.in.f32[(((size_t)n * p.Cin + s_ci[c]) * H + hi) * W + wi];
                    x[u] = v;
                }
                const size_t row0 = ((size_t)n * p.Ho + hb) * p.Wo;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int wp = wb - j;  // the pixel whose window has this block at position j
                    if (wp >= 0 && wp < p.Wo)
                        planes_store8(p.out_hi, p.out_lo, (row0 + wp) * 64 + j * 16 + half * 8, p.fmt, x);
                }
            }
            ++iter;
        }
        if (threadIdx.x == 0) trace_end(blp, iter);
        return;
    }
    if (p.planes_vec) {
        const int Cs = p.in.l.C;            // stored channels of the input
        const unsigned vectors = (unsigned)p.M * K8;
        const int c8_per_tap = Cs / 8;
        const int fmt = p.fmt;
        for (;;) {
            int tile;
            __syncthreads();
            if (dynamic) {
                if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
                __syncthreads();
                tile = s_tile;
            } else {
                tile = blp_claim(blp, iter);
            }
            if (tile < 0) break;
            const unsigned begin = (unsigned)tile * p.tile_elems;
            const unsigned end = begin + p.tile_elems < vectors ? begin + p.tile_elems : vectors;
            for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
                const int k8 = (int)(e % K8);
                const unsigned m = e / K8;
                const int wo = (int)(m % p.Wo);
                const unsigned t = m / p.Wo;
                const int ho = (int)(t % p.Ho), n = (int)(t / p.Ho);
                const int tap = k8 / c8_per_tap, c8 = k8 - tap * c8_per_tap;
                const int fh = tap / p.kw, fw = tap - fh * p.kw;
                const int hi = ho * p.stride - p.pad + fh, wi = wo * p.stride - p.pad_w + fw;
                uint4 a = make_uint4(0, 0, 0, 0), b = make_uint4(0, 0, 0, 0);
                if (fh < p.kh && hi >= 0 && hi < H && wi >= 0 && wi < W)
                    planes_fetch8(p.in.hi, p.in.lo, (size_t)layout_row(p.in.l, n, hi, wi) * Cs + c8 * 8, fmt, a, b);
                const size_t off = (size_t)m * p.Kp + k8 * 8;
                *reinterpret_cast<uint4 *>(p.out_hi + off) = a;
                if (fmt == PF_SPLIT) *reinterpret_cast<uint4 *>(p.out_lo + off) = b;
            }
            ++iter;
        }
        if (threadIdx.x == 0) trace_end(blp, iter);
        return;
    }
    if (p.win_w > 0) {
        // Row-window mode.  The window of the tile - Cin x kh input rows, (win_w-1)*stride + kw
        // wide, zeros outside the image - is staged with coalesced loads; a patch-matrix element
        // is then one table lookup and one shared-memory read, and the stores stay row-contiguous.
        __shared__ float s_win[kIm2colWindowFloats];
        const int win_cols = (p.win_w - 1) * p.stride + p.kw;
        const int seg = p.Cin * p.kh;  // window rows
        for (int k = threadIdx.x; k < p.Kp; k += kPoolThreads)
            s_off[k] = s_fh[k] == 255 ? -1 : ((int)s_ci[k] * p.kh + (int)s_fh[k]) * win_cols + (int)s_fw[k];
        for (;;) {
            int tile;
            __syncthreads();  // the table is complete / the previous window has been consumed
            if (dynamic) {
                if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
                __syncthreads();
                tile = s_tile;
            } else {
                tile = blp_claim(blp, iter);
            }
            if (tile < 0) break;
            const int chunk = tile % p.win_chunks;
            const int t = tile / p.win_chunks;
            const int ho = t % p.Ho, n = t / p.Ho;
            const int wo0 = chunk * p.win_w;
            const int nw = min(p.win_w, p.Wo - wo0);
            const int h0 = ho * p.stride - p.pad, w0 = wo0 * p.stride - p.pad;
            for (int e = threadIdx.x; e < seg * win_cols; e += kPoolThreads) {
                const int r = e / win_cols, c = e - r * win_cols;
                const int ci = r / p.kh, fh = r - ci * p.kh;
                const int hi = h0 + fh, wi = w0 + c;
                float v = 0.f;
                if (hi >= 0 && hi < H && wi >= 0 && wi < W)
                    v = p.in.f32[(((size_t)n * p.Cin + ci) * H + hi) * W + wi];
                s_win[e] = v;
            }
            __syncthreads();
            const size_t m0 = ((size_t)n * p.Ho + ho) * p.Wo + wo0;
            for (int e = threadIdx.x; e < nw * K8; e += kPoolThreads) {
                const int wl = e / K8, k8 = e - wl * K8;
                const int shift = wl * p.stride;
                float x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int off = s_off[k8 * 8 + u];
                    x[u] = off < 0 ? 0.f : s_win[off + shift];
                }
                planes_store8(p.out_hi, p.out_lo, (m0 + wl) * p.Kp + k8 * 8, p.fmt, x);
            }
            ++iter;
        }
        if (threadIdx.x == 0) trace_end(blp, iter);
        return;
    }
    for (;;) {
        int tile;
        if (dynamic) {
            if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = begin + p.tile_elems < total ? begin + p.tile_elems : total;
        for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
            int k8 = (int)(e % K8);
            int m = (int)(e / K8);
            int wo = m % p.Wo;
            int t = m / p.Wo;
            int ho = t % p.Ho;
            int n = t / p.Ho;
            const int h0 = ho * p.stride - p.pad, w0 = wo * p.stride - p.pad;
            const long long origin = ((long long)n * p.Cin * H + h0) * W + w0;
            float x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                int k = k8 * 8 + u;
                float v = 0.f;
                int fh = s_fh[k];
                int hi = h0 + fh, wi = w0 + s_fw[k];
                if (fh != 255 && hi >= 0 && hi < H && wi >= 0 && wi < W)
                    v = p.in.f32 ? p.in.f32[origin + s_off[k]] : view_load(p.in, n, hi, wi, s_ci[k]);
                x[u] = v;
            }
            planes_store8(p.out_hi, p.out_lo, (size_t)m * p.Kp + k8 * 8, p.fmt, x);
        }
        ++iter;
        if (dynamic) __syncthreads();
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

// Patch matrix of a 3x3 filter over a three-channel fp32 NCHW input (VGG, MobileNetV2, Inception-v3): a thread
// takes one pixel and writes its whole row of 27 values and five zeros.  Neighbouring threads read
// neighbouring elements, 27 independent loads each that L1 and L2 serve after the first, and a row is two
// 32-byte stores a plane, whole sectors.  Bound by the writes and, at one image, by one chain
// load - convert - store.  (A window of the image in shared memory, a vector of eight columns a thread: four barriers
// and ~2 800 cycles a tile of one image row, 63 us for 224x224, 16 images fp16; 28 like this.  MobileNetV2, stride 2, 64 images: 86 -> 28 us.)
constexpr int kRgbK = 27, kRgbKp = 32;

template <int FMT>
__global__ void __launch_bounds__(kPoolThreads)
patches_rgb_kernel(const __grid_constant__ Im2colParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    if (threadIdx.x == 0) trace_begin(blp);
    const int H = p.in.l.H, W = p.in.l.W;
    TileClaims claims(blp, blp.preempted != nullptr, s_tile);
    for (int tile = claims.first(); tile >= 0; tile = claims.next()) {
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = min(begin + (unsigned)p.tile_elems, (unsigned)p.M);
        for (unsigned m = begin + threadIdx.x; m < end; m += kPoolThreads) {
            const int wo = (int)(m % (unsigned)p.Wo);
            const unsigned t = m / (unsigned)p.Wo;
            const int ho = (int)(t % (unsigned)p.Ho), n = (int)(t / (unsigned)p.Ho);
            const int h0 = ho * p.stride - p.pad, w0 = wo * p.stride - p.pad;
            const float *img = p.in.f32 + (size_t)n * 3 * H * W;
            float x[kRgbKp];
#pragma unroll
            for (int k = 0; k < kRgbKp; ++k) {  // columns are (fh, fw, channel)
                x[k] = 0.f;
                if (k < kRgbK) {
                    const int hi = h0 + k / 9, wi = w0 + k / 3 % 3;
                    if (hi >= 0 && hi < H && wi >= 0 && wi < W) x[k] = __ldg(img + ((size_t)(k % 3) * H + hi) * W + wi);
                }
            }
            claims.ahead();
            const size_t off = (size_t)m * kRgbKp;
#pragma unroll
            for (int c = 0; c < kRgbKp; c += 16) {
                unsigned hi[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) hi[q] = pf_pack2(x[c + 2 * q], x[c + 2 * q + 1], FMT);
                st_sector(p.out_hi + off + c, hi);
                if (FMT == PF_SPLIT) {
                    unsigned lo[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        lo[q] = pf_pack2(x[c + 2 * q] - __uint_as_float(hi[q] << 16),
                                         x[c + 2 * q + 1] - __uint_as_float(hi[q] & 0xffff0000u), PF_SPLIT);
                    st_sector(p.out_lo + off + c, lo);
                }
            }
        }
    }
    if (threadIdx.x == 0) trace_end(blp, claims.done());
}

static auto patches_rgb_instance(int fmt) {
    return fmt == PF_SPLIT ? patches_rgb_kernel<PF_SPLIT> : (fmt == PF_F16 ? patches_rgb_kernel<PF_F16> : patches_rgb_kernel<PF_BF16>);
}

int im2col_rgb_grid(int sm_count, int total_tiles) {
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, patches_rgb_instance(PF_SPLIT), kPoolThreads, 0);
    return (int)std::min<long long>((long long)sm_count * std::max(per_sm, 1), total_tiles);
}

cudaError_t im2col_launch(const Im2colParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    if (p.rgb) return launch_layer(patches_rgb_instance(p.fmt), grid, kPoolThreads, 0, s, p, blp);
    return launch_layer(im2col_kernel, grid, kPoolThreads, 0, s, p, blp);
}

// Finishing pass of a split-K tensor-core convolution: one thread-iteration handles eight
// channels of one GEMM row.  The per-split sums are added in split order, so the result does
// not depend on which CTA produced which split or in which order they finished.
__global__ void __launch_bounds__(kPoolThreads)
splitk_finish_kernel(const __grid_constant__ SplitKParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int C8 = p.cout_padded / 8;
    const unsigned total = (unsigned)p.m_rows * C8;
    const int img = p.in_hs * p.in_ws;
    int iter = 0;
    for (;;) {
        int tile;
        if (dynamic) {
            if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = begin + p.tile_elems < total ? begin + p.tile_elems : total;
        for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
            const int c8 = (int)(e % C8);
            const int vrow = (int)(e / C8);
            const int n_img = vrow / img;
            const int r = vrow - n_img * img;
            const int hs = r / p.in_ws;
            const int h = hs - p.in_off;
            const int w = r - hs * p.in_ws - p.in_off;
            if (h < 0 || h >= p.out.H || w < 0 || w >= p.out.W) continue;
            float f[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = 0.f;
            for (int s = 0; s < p.k_splits; ++s) {
                const float4 *src = reinterpret_cast<const float4 *>(
                    p.partial + ((size_t)s * p.partial_rows + vrow) * p.partial_ld + c8 * 8);
                float4 a = src[0], b = src[1];
                f[0] += a.x; f[1] += a.y; f[2] += a.z; f[3] += a.w;
                f[4] += b.x; f[5] += b.y; f[6] += b.z; f[7] += b.w;
            }
            splitk_apply(p, n_img, h, w, c8 * 8, f);
        }
        ++iter;
        if (dynamic) __syncthreads();
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

__global__ void __launch_bounds__(kPoolThreads)
dense_rows_kernel(const __grid_constant__ DenseRowsParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    __shared__ float s_part[kPoolThreads / 32][8];
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    constexpr int kStep = kPoolThreads * 8;  // elements of one row the CTA reads per step (4 KB per plane)
    constexpr int kU = 4;
    int iter = 0;
    for (;;) {
        int tile;
        __syncthreads();
        if (dynamic) {
            if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        // A tile is eight output columns, one after the other; the whole CTA walks one weight row
        // with consecutive threads on consecutive 16-byte vectors, so that DRAM sees long
        // contiguous reads (one warp per row opened a new DRAM page with every 512 bytes and
        // reached a quarter of the bandwidth).
        for (int c = 0; c < 8; ++c) {
            const int n = tile * 8 + c;
            if (n >= p.cout) break;
            float acc[8];
#pragma unroll
            for (int m = 0; m < 8; ++m) acc[m] = 0.f;
            const size_t w_row = (size_t)n * p.w_ld;
            for (int k0 = threadIdx.x * 8; k0 < p.K; k0 += kStep * kU) {
                uint4 wa[kU], wb[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    wa[u] = wb[u] = make_uint4(0, 0, 0, 0);
                    if (k0 + u * kStep < p.K) planes_fetch8(p.w_hi, p.w_lo, w_row + k0 + u * kStep, p.fmt, wa[u], wb[u]);
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    if (k0 + u * kStep >= p.K) break;
                    float w[8];
                    planes_decode8(wa[u], wb[u], p.fmt, w);
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        if (m < p.M) {
                            float a[8];
                            planes_load8(p.a_hi, p.a_lo, (size_t)m * p.a_ld + k0 + u * kStep, p.fmt, a);
#pragma unroll
                            for (int j = 0; j < 8; ++j) acc[m] = fmaf(a[j], w[j], acc[m]);
                        }
                    }
                }
            }
#pragma unroll
            for (int sh = 16; sh >= 1; sh >>= 1)
#pragma unroll
                for (int m = 0; m < 8; ++m) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], sh);
            __syncthreads();  // the previous column's partial sums have been consumed
            if (lane == 0)
#pragma unroll
                for (int m = 0; m < 8; ++m) s_part[wid][m] = acc[m];
            __syncthreads();
            if (threadIdx.x < p.M) {
                const int m = threadIdx.x;
                float v = 0.f;
#pragma unroll
                for (int w8 = 0; w8 < kPoolThreads / 32; ++w8) v += s_part[w8][m];  // fixed order
                v = apply_act(v + (p.bias ? p.bias[n] : 0.f), p.relu);
                if (p.out_f32)
                    p.out_f32[(size_t)m * p.cout + n] = v;
                else
                    planes_store1(p.out_hi, p.out_lo, (size_t)m * p.out_ld + n, p.fmt, v);
            }
        }
        ++iter;
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

// The same layer with short rows (at most kDenseShortK input elements: the classifiers behind a global
// average pool): one warp per output column, eight columns per tile.  Such a row is a few KB, the matrix
// a few MB that L2 keeps; what costs is the chain of steps, so the columns of a tile run side by side
// instead of one after the other with a block-wide sum each, and every lane's part of its first row is
// requested ahead of the wait for the predecessor (weights are never written by a kernel).
// ResNet-50's 2048 -> 1000 at batch 1: 12.5 us with the whole CTA on one row, 2.3 like this.
constexpr int kDenseShortVec = kDenseShortK / 256;  // 16-byte vectors per lane and plane

__global__ void __launch_bounds__(kPoolThreads)
dense_short_kernel(const __grid_constant__ DenseRowsParams p, BlpArgs blp) {
    extern __shared__ float s_a[];  // [M][K] input rows
    __shared__ int s_tile;
    const bool dynamic = blp.preempted != nullptr;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint4 wa[kDenseShortVec], wb[kDenseShortVec];
    auto fetch = [&](int n) {
#pragma unroll
        for (int u = 0; u < kDenseShortVec; ++u)
            if (n < p.cout && (u * 32 + lane) * 8 < p.K)
                planes_fetch8(p.w_hi, p.w_lo, (size_t)n * p.w_ld + (u * 32 + lane) * 8, p.fmt, wa[u], wb[u]);
    };
    int have = dynamic ? -1 : (int)blockIdx.x;  // tile whose weights are in wa, wb
    if (have >= 0) fetch(have * 8 + wid);
    pdl_enter();
    if (threadIdx.x == 0) trace_begin(blp);
    for (int v = threadIdx.x; v < p.M * (p.K / 8); v += kPoolThreads) {
        const int m = v / (p.K / 8), k = (v - m * (p.K / 8)) * 8;
        float a[8];
        planes_load8(p.a_hi, p.a_lo, (size_t)m * p.a_ld + k, p.fmt, a);
        float4 *dst = reinterpret_cast<float4 *>(s_a + m * p.K + k);
        dst[0] = make_float4(a[0], a[1], a[2], a[3]);
        dst[1] = make_float4(a[4], a[5], a[6], a[7]);
    }
    __syncthreads();
    int iter = 0;
    for (;;) {
        int tile;
        if (dynamic) {
            __syncthreads();
            if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        const int n = tile * 8 + wid;
        if (tile != have) fetch(n);
        have = -1;
        if (n < p.cout) {
            float w[kDenseShortVec][8];
#pragma unroll
            for (int u = 0; u < kDenseShortVec; ++u) planes_decode8(wa[u], wb[u], p.fmt, w[u]);
            const float bias = p.bias ? __ldg(p.bias + n) : 0.f;
#pragma unroll 1
            for (int m = 0; m < p.M; ++m) {
                float acc = 0.f;
#pragma unroll
                for (int u = 0; u < kDenseShortVec; ++u) {
                    const int k0 = (u * 32 + lane) * 8;
                    if (k0 < p.K) {
                        const float4 *a4 = reinterpret_cast<const float4 *>(s_a + m * p.K + k0);
                        const float4 x = a4[0], y = a4[1];
                        const float a[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc = fmaf(a[j], w[u][j], acc);
                    }
                }
#pragma unroll
                for (int sh = 16; sh >= 1; sh >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, sh);
                if (lane == 0) {
                    const float v = apply_act(acc + bias, p.relu);
                    if (p.out_f32)
                        p.out_f32[(size_t)m * p.cout + n] = v;
                    else
                        planes_store1(p.out_hi, p.out_lo, (size_t)m * p.out_ld + n, p.fmt, v);
                }
            }
        }
        ++iter;
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

// The whole CTA reads every input row again for each of a tile's columns, from L1: it gets all of an SM's memory as cache.
// Behind a kernel that uses it as shared memory it was left 28 KB of it, or not, by what ran between: 25088 -> 4096 of three
// images 192 or 228 us float32, 105 or 140 bf16; 194 and 105 like this, and never the other.
cudaError_t dense_rows_prepare() {
    return cudaFuncSetAttribute(dense_rows_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1);
}

cudaError_t dense_rows_launch(const DenseRowsParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    // (input rows of the short form, beside its own variables, in the default 48 KB of shared memory)
    const size_t rows = (size_t)p.M * p.K * sizeof(float);
    if (p.K <= kDenseShortK && rows + 256 <= 48 * 1024)
        return launch_layer(dense_short_kernel, grid, kPoolThreads, rows, s, p, blp);
    return launch_layer(dense_rows_kernel, grid, kPoolThreads, 0, s, p, blp);
}

cudaError_t splitk_launch(const SplitKParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    return launch_layer(splitk_finish_kernel, grid, kPoolThreads, 0, s, p, blp);
}

// Output pixel and channel group of element e of a tensor walked in (n, ho, wo, c / 8) order.
struct PixelAt {
    int c8, wo, ho, n;
};
__device__ __forceinline__ PixelAt pixel_at(unsigned e, int C8, int Wo, int Ho) {
    PixelAt a;
    a.c8 = (int)(e % C8);
    unsigned t = e / C8;
    a.wo = (int)(t % Wo);
    t /= Wo;
    a.ho = (int)(t % Ho);
    a.n = (int)(t / Ho);
    return a;
}

// Depthwise convolution: one thread-iteration produces eight channels of one output pixel,
// taps walked in (fh, fw) order with one FMA each, so the result is independent of the tiling.  Channels that only
// pad the stored width are left as the zeros they are (MobileNetV2's first layers: 32 of 64, 96 of 128, 144 of 192).
// At batch 1 this is latency: ahead of the wait for the predecessor the filter (never written by a kernel) is
// copied to shared memory, and for the element a thread starts with the addresses, the taps inside the image
// and the bias are found; behind it the nine taps of a 3x3 filter are requested before any is used
// (MobileNetV2 b1, us a layer: 4.4 a tap at a time, 3.3 to 4.9 with nine in flight and addresses behind the wait,
// 2.5 to 3.7 like this).
//
// BATCH: taps of a 3x3 filter in flight at once.  Nine where all vectors are at work at once at two CTAs an SM; three (a
// filter row) in larger tensors that the strips below do not take (fewer than four vectors a thread, rows stored with a
// border, strides from three on), which want the occupancy that the registers of nine take; 0: a tap at a time (other
// filter sizes), at that occupancy too.  Six such layers between a 1x1 layer and a classifier, us, all with the registers
// of nine / like this: 3x3 over padded rows, 32 images of 56x56x64 bf16 343 / 258, stride 3 over the same image 87 / 74,
// stride 2, 14x14x512 76 / 67; 7x7, 32 images of 14x14x512 float32 584 / 432.
struct DwElem {
    long long in;    // element offset of tap (0, 0) in a plain input (it may lie outside)
    size_t out;      // element offset of the output
    int c0;
    unsigned taps;   // of a 3x3 filter: inside the image
};
__device__ __forceinline__ DwElem dw_elem(const DwConvParams &p, const PixelAt &at) {
    DwElem a;
    a.c0 = at.c8 * 8;
    const int h0 = at.ho * p.stride - p.pad, w0 = at.wo * p.stride - p.pad;
    a.in = ((long long)(at.n * p.in.l.Hs + h0) * p.in.l.Ws + w0) * p.in.l.C + a.c0;
    a.out = (size_t)layout_row(p.out, at.n, at.ho, at.wo) * p.out.C + a.c0;
    unsigned rows = 0, cols = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        rows |= (unsigned)(h0 + i) < (unsigned)p.in.l.H ? 7u << (3 * i) : 0u;
        cols |= (unsigned)(w0 + i) < (unsigned)p.in.l.W ? 0x49u << i : 0u;
    }
    a.taps = rows & cols;
    return a;
}

template <int BATCH, bool TWO>
__global__ void __launch_bounds__(kPoolThreads, BATCH == 9 ? 2 : 4)
dwconv_kernel(const __grid_constant__ DwConvParams p, BlpArgs blp) {
    extern __shared__ float s_w[];  // [k * k][C], or nothing where it does not fit
    __shared__ int s_tile;
    const bool dynamic = blp.preempted != nullptr;
    const int C = p.out.C;
    const int C8 = p.channels / 8;
    const int H = p.in.l.H, W = p.in.l.W;
    const unsigned total = (unsigned)p.out.N * p.out.H * p.out.W * C8;  // < 2^31, checked when the model is built
    const float *wts = p.w;
    if (p.w_in_smem) {
        const int n4 = p.k * p.k * C / 4;
        for (int i = threadIdx.x; i < n4; i += kPoolThreads)
            reinterpret_cast<float4 *>(s_w)[i] = __ldg(reinterpret_cast<const float4 *>(p.w) + i);
        wts = s_w;
    }
    unsigned known = (unsigned)blockIdx.x * p.tile_elems + threadIdx.x;  // found ahead for a static schedule
    if (dynamic || known >= total) known = ~0u;
    const PixelAt first = pixel_at(known == ~0u ? 0 : known, C8, p.out.W, p.out.H);
    DwElem ahead;
    float4 bias_a = make_float4(0.f, 0.f, 0.f, 0.f), bias_b = bias_a;
    auto fetch_bias = [&](int c0) {
        if (!p.bias) return;
        bias_a = __ldg(reinterpret_cast<const float4 *>(p.bias + c0));
        bias_b = __ldg(reinterpret_cast<const float4 *>(p.bias + c0) + 1);
    };
    if constexpr (BATCH == 9) {
        ahead = dw_elem(p, first);
        fetch_bias(ahead.c0);
    }
    __syncthreads();
    pdl_enter();
    if (threadIdx.x == 0) trace_begin(blp);
    TileClaims claims(blp, dynamic, s_tile);
    const int fmt = TWO ? (int)PF_SPLIT : p.in.l.fmt;
    for (int tile = claims.first(); tile >= 0; tile = claims.next()) {
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = begin + p.tile_elems < total ? begin + p.tile_elems : total;
        for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
            float2 acc[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = make_float2(0.f, 0.f);
            auto tap = [&](const float (&x)[8], int t, int c0) {
                const float4 *wv = reinterpret_cast<const float4 *>(wts + (size_t)t * C + c0);
                const float4 a = wv[0], b = wv[1];
                if (BATCH == 9) {
                    acc[0] = fma2(make_float2(x[0], x[1]), make_float2(a.x, a.y), acc[0]);
                    acc[1] = fma2(make_float2(x[2], x[3]), make_float2(a.z, a.w), acc[1]);
                    acc[2] = fma2(make_float2(x[4], x[5]), make_float2(b.x, b.y), acc[2]);
                    acc[3] = fma2(make_float2(x[6], x[7]), make_float2(b.z, b.w), acc[3]);
                } else {
                    acc[0].x = fmaf(x[0], a.x, acc[0].x), acc[0].y = fmaf(x[1], a.y, acc[0].y);
                    acc[1].x = fmaf(x[2], a.z, acc[1].x), acc[1].y = fmaf(x[3], a.w, acc[1].y);
                    acc[2].x = fmaf(x[4], b.x, acc[2].x), acc[2].y = fmaf(x[5], b.y, acc[2].y);
                    acc[3].x = fmaf(x[6], b.z, acc[3].x), acc[3].y = fmaf(x[7], b.w, acc[3].y);
                }
            };
            size_t out;
            if constexpr (BATCH == 9) {
                const PixelAt px = e == known ? first : pixel_at(e, C8, p.out.W, p.out.H);
                const DwElem at = e == known ? ahead : dw_elem(p, px);
                out = at.out;
                uint4 ra[9], rb[TWO ? 9 : 1];
                if (p.in.l.order == ACT_PLAIN) {
                    const long long row_step = (long long)p.in.l.Ws * p.in.l.C;
#pragma unroll
                    for (int t = 0; t < 9; ++t)
                        if (at.taps >> t & 1)
                            planes_fetch8(p.in.hi, p.in.lo, (size_t)(at.in + t / 3 * row_step + t % 3 * p.in.l.C), fmt, ra[t], rb[TWO ? t : 0]);
                } else {
#pragma unroll
                    for (int t = 0; t < 9; ++t)
                        if (at.taps >> t & 1)
                            planes_fetch8(p.in.hi, p.in.lo,
                                          (size_t)layout_row(p.in.l, px.n, px.ho * p.stride - p.pad + t / 3, px.wo * p.stride - p.pad + t % 3) *
                                                  p.in.l.C + at.c0,
                                          fmt, ra[t], rb[TWO ? t : 0]);
                }
                claims.ahead();
                if (e != known) fetch_bias(at.c0);
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    if (!(at.taps >> t & 1)) continue;
                    float x[8];
                    planes_decode8(ra[t], rb[TWO ? t : 0], fmt, x);
                    tap(x, t, at.c0);
                }
            } else {
                const PixelAt px = BATCH == 0 && e == known ? first : pixel_at(e, C8, p.out.W, p.out.H);
                const int c0 = px.c8 * 8, h0 = px.ho * p.stride - p.pad, w0 = px.wo * p.stride - p.pad;
                const int k = BATCH ? 3 : p.k;
#pragma unroll 1
                for (int fh = 0; fh < k; ++fh) {
                    const int hi = h0 + fh;
                    if constexpr (BATCH == 3) {
                        uint4 ra[3], rb[TWO ? 3 : 1];
                        bool ok[3];
#pragma unroll
                        for (int t = 0; t < 3; ++t) {
                            const int wi = w0 + t;
                            ok[t] = hi >= 0 && hi < H && wi >= 0 && wi < W;
                            if (ok[t])
                                planes_fetch8(p.in.hi, p.in.lo, (size_t)layout_row(p.in.l, px.n, hi, wi) * p.in.l.C + c0, fmt, ra[t], rb[TWO ? t : 0]);
                        }
                        if (fh == 0) claims.ahead();
#pragma unroll
                        for (int t = 0; t < 3; ++t) {
                            if (!ok[t]) continue;
                            float x[8];
                            planes_decode8(ra[t], rb[TWO ? t : 0], fmt, x);
                            tap(x, fh * 3 + t, c0);
                        }
                    } else {
                        if (hi < 0 || hi >= H) continue;
                        for (int fw = 0; fw < k; ++fw) {
                            const int wi = w0 + fw;
                            if (wi < 0 || wi >= W) continue;
                            float x[8];
                            planes_load8(p.in.hi, p.in.lo, (size_t)layout_row(p.in.l, px.n, hi, wi) * p.in.l.C + c0, p.in.l.fmt, x);
                            tap(x, fh * k + fw, c0);
                        }
                    }
                }
                fetch_bias(c0);
                out = (size_t)layout_row(p.out, px.n, px.ho, px.wo) * C + c0;
            }
            float f[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) f[2 * j] = acc[j].x, f[2 * j + 1] = acc[j].y;
            if (p.bias) {
                f[0] += bias_a.x, f[1] += bias_a.y, f[2] += bias_a.z, f[3] += bias_a.w;
                f[4] += bias_b.x, f[5] += bias_b.y, f[6] += bias_b.z, f[7] += bias_b.w;
            }
            apply_act_n(f, p.act);
            planes_store8(p.out_hi, p.out_lo, out, TWO ? (int)PF_SPLIT : p.out.fmt, f);
        }
    }
    if (threadIdx.x == 0) trace_end(blp, claims.done());
}

// The 3x3 filter over a large tensor in plain rows: a thread produces eight channels of four neighbouring output
// pixels, so that a vector of the input is fetched and unpacked 1.5 times (2.25 at stride 2) instead of
// nine, and a tap's filter values are read once for four pixels.  Bound by instruction issue: 56x56x144, 64 images
// fp16, 142 us a pixel at a time over the padded width of 192, 122 over 144, 71 in strips
// (its bytes alone: 18); all of MobileNetV2 b64 fp16 1 302 -> 1 013.  The order of an output's taps is that of the other form, so its bits are too.
constexpr int dw_strip(int stride, bool two) { return stride == 2 && two ? 2 : 4; }  // (nine columns of two planes spill)
template <int STRIDE, bool TWO>
__global__ void __launch_bounds__(kPoolThreads, 2)
dwconv_strip_kernel(const __grid_constant__ DwConvParams p, BlpArgs blp) {
    extern __shared__ float s_w[];
    __shared__ int s_tile;
    constexpr int kDwStrip = dw_strip(STRIDE, TWO), kCols = (kDwStrip - 1) * STRIDE + 3;
    const bool dynamic = blp.preempted != nullptr;
    const int C = p.out.C, C8 = p.channels / 8;
    const int H = p.in.l.H, W = p.in.l.W, strips = (p.out.W + kDwStrip - 1) / kDwStrip;
    const unsigned total = (unsigned)p.out.N * p.out.H * strips * C8;
    const float *wts = p.w;
    if (p.w_in_smem) {
        const int n4 = 9 * C / 4;
        for (int i = threadIdx.x; i < n4; i += kPoolThreads)
            reinterpret_cast<float4 *>(s_w)[i] = __ldg(reinterpret_cast<const float4 *>(p.w) + i);
        wts = s_w;
    }
    __syncthreads();
    pdl_enter();
    if (threadIdx.x == 0) trace_begin(blp);
    TileClaims claims(blp, dynamic, s_tile);
    const int fmt = TWO ? (int)PF_SPLIT : p.in.l.fmt;
    for (int tile = claims.first(); tile >= 0; tile = claims.next()) {
        const unsigned begin = (unsigned)tile * p.tile_elems;
        const unsigned end = begin + p.tile_elems < total ? begin + p.tile_elems : total;
        for (unsigned e = begin + threadIdx.x; e < end; e += kPoolThreads) {
            const PixelAt at = pixel_at(e, C8, strips, p.out.H);
            const int c0 = at.c8 * 8, wo0 = at.wo * kDwStrip;
            const int h0 = at.ho * STRIDE - p.pad, w0 = wo0 * STRIDE - p.pad;
            float2 acc[kDwStrip][4];
#pragma unroll
            for (int o = 0; o < kDwStrip; ++o)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[o][j] = make_float2(0.f, 0.f);
#pragma unroll 1
            for (int fh = 0; fh < 3; ++fh) {
                if ((unsigned)(h0 + fh) >= (unsigned)H) continue;
                const long long row = ((long long)(at.n * H + h0 + fh) * W + w0) * p.in.l.C + c0;
                uint4 ra[kCols], rb[TWO ? kCols : 1];
#pragma unroll
                for (int c = 0; c < kCols; ++c)
                    if ((unsigned)(w0 + c) < (unsigned)W)
                        planes_fetch8(p.in.hi, p.in.lo, (size_t)(row + (long long)c * p.in.l.C), fmt, ra[c], rb[TWO ? c : 0]);
                if (fh == 1) claims.ahead();
                float2 wt[3][4];
#pragma unroll
                for (int fw = 0; fw < 3; ++fw) {
                    const float4 *wv = reinterpret_cast<const float4 *>(wts + (size_t)(fh * 3 + fw) * C + c0);
                    const float4 a = wv[0], b = wv[1];
                    wt[fw][0] = make_float2(a.x, a.y), wt[fw][1] = make_float2(a.z, a.w);
                    wt[fw][2] = make_float2(b.x, b.y), wt[fw][3] = make_float2(b.z, b.w);
                }
#pragma unroll
                for (int c = 0; c < kCols; ++c) {
                    if ((unsigned)(w0 + c) >= (unsigned)W) continue;
                    float x[8];
                    planes_decode8(ra[c], rb[TWO ? c : 0], fmt, x);
#pragma unroll
                    for (int o = 0; o < kDwStrip; ++o) {
                        const int fw = c - o * STRIDE;
                        if (fw < 0 || fw > 2) continue;
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[o][j] = fma2(make_float2(x[2 * j], x[2 * j + 1]), wt[fw][j], acc[o][j]);
                    }
                }
            }
            float4 bias_a = make_float4(0.f, 0.f, 0.f, 0.f), bias_b = bias_a;
            if (p.bias) {
                bias_a = __ldg(reinterpret_cast<const float4 *>(p.bias + c0));
                bias_b = __ldg(reinterpret_cast<const float4 *>(p.bias + c0) + 1);
            }
            const size_t out = (size_t)layout_row(p.out, at.n, at.ho, wo0) * C + c0;
#pragma unroll
            for (int o = 0; o < kDwStrip; ++o) {
                if (wo0 + o >= p.out.W) break;
                float f[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) f[2 * j] = acc[o][j].x, f[2 * j + 1] = acc[o][j].y;
                if (p.bias) {
                    f[0] += bias_a.x, f[1] += bias_a.y, f[2] += bias_a.z, f[3] += bias_a.w;
                    f[4] += bias_b.x, f[5] += bias_b.y, f[6] += bias_b.z, f[7] += bias_b.w;
                }
                apply_act_n(f, p.act);
                const size_t off = p.out.order == ACT_PHASED ? (size_t)layout_row(p.out, at.n, at.ho, wo0 + o) * C + c0 : out + (size_t)o * C;
                planes_store8(p.out_hi, p.out_lo, off, TWO ? (int)PF_SPLIT : p.out.fmt, f);
            }
        }
    }
    if (threadIdx.x == 0) trace_end(blp, claims.done());
}

static auto dwconv_instance(const DwConvParams &p) {
    const bool two = p.out.fmt == PF_SPLIT;
    if (p.strip) {
        if (p.stride == 1) return two ? dwconv_strip_kernel<1, true> : dwconv_strip_kernel<1, false>;
        return two ? dwconv_strip_kernel<2, true> : dwconv_strip_kernel<2, false>;
    }
    if (p.k != 3) return two ? dwconv_kernel<0, true> : dwconv_kernel<0, false>;
    if (p.small) return two ? dwconv_kernel<9, true> : dwconv_kernel<9, false>;
    return two ? dwconv_kernel<3, true> : dwconv_kernel<3, false>;
}
static size_t dwconv_smem(const DwConvParams &p) { return p.w_in_smem ? (size_t)p.k * p.k * p.out.C * sizeof(float) : 0; }

// Tiles, form and grid of a layer whose shapes, filter and stride are set.  Strips of four pixels where the tensor
// has more than four tiles of 256 vectors an SM; below that a thread per pixel has more threads at work.  Nine taps in flight
// up to two tiles an SM, which is what their registers leave resident (MobileNetV2, us a latency-critical request with
// the line at two / at four tiles: 2 images bf16 204 / 210, 8 images 277 / 283, float32 the same).
int dwconv_plan(DwConvParams &p, int sm_count) {
    const long long pixels = (long long)p.out.N * p.out.H * p.out.W, c8 = p.channels / 8;
    p.small = pixels * c8 <= 2LL * 256 * sm_count;
    p.strip = p.k == 3 && p.in.l.order == ACT_PLAIN && (p.stride == 1 || p.stride == 2) && pixels * c8 > 4LL * 256 * sm_count;
    const int len = dw_strip(p.stride, p.out.fmt == PF_SPLIT);
    const long long total = p.strip ? (long long)p.out.N * p.out.H * ((p.out.W + len - 1) / len) * c8 : pixels * c8;
    p.tile_elems = 256;
    p.total_tiles = (int)((total + p.tile_elems - 1) / p.tile_elems);
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dwconv_instance(p), kPoolThreads, dwconv_smem(p));
    return (int)std::min<long long>((long long)sm_count * std::max(per_sm, 1), p.total_tiles);
}

cudaError_t dwconv_launch(const DwConvParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    return launch_layer(dwconv_instance(p), grid, kPoolThreads, dwconv_smem(p), s, p, blp);
}

// Taps along a side of the windows that have an instance of their own, else 0.
static int pool_taps(const PoolParams &p) {
    if (p.scale) return 0;
    if (p.mode == 0 && p.k == 3) return 3;
    return p.mode != 2 && p.k == 2 ? 2 : 0;
}
typedef void (*PoolKernel)(const PoolParams, BlpArgs);
static PoolKernel pool_instance(const PoolParams &p) {
    const bool two = p.out.fmt == PF_SPLIT;
    switch (pool_taps(p)) {
        case 3: return two ? pool_window_kernel<3, true> : pool_window_kernel<3, false>;
        case 2: return two ? pool_window_kernel<2, true> : pool_window_kernel<2, false>;
        default: return pool_kernel;
    }
}

// Tiles and grid of a launch whose shapes are set.
int pool_plan(PoolParams &p, int sm_count) {
    const long long total = (long long)p.out.N * p.out.H * p.out.W * (p.channels / 8);
    const int t = pool_taps(p);
    int per_sm = 8;
    if (t) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pool_instance(p), kPoolThreads, 0);
        if (per_sm < 1) per_sm = 1;
        // A small tensor is cut so that each CTA that fits runs one tile (ResNet's 3x3 at batch 1: 392 tiles of 64
        // vectors on 296 CTAs were two rounds), a large one into tiles of whole CTAs.  2x2 windows take two warps a tile
        // at least, and four CTAs an SM without spills (bf16, us six latency-critical layers: five CTAs and from 32
        // vectors on / like this: 56x56x256 47 / 43, 28x28x512 of two images 38 / 35, 112x112x64 81 / 77).
        const long long slots = (long long)per_sm * sm_count, even = (total + slots - 1) / slots;
        p.tile_elems = even <= 256 ? (int)std::max<long long>(t == 3 ? 32 : 64, (even + 7) / 8 * 8) : (t == 2 && even >= 1024 ? 512 : 256);
        p.by_c8 = FastDiv::of((unsigned)(p.channels / 8)), p.by_w = FastDiv::of((unsigned)p.out.W), p.by_h = FastDiv::of((unsigned)p.out.H);
    } else {
        // the cap is per unit of work: a copy or an affine map reads one tap per vector
        const int taps_per_vec = p.mode == 2 ? 1 : p.k * p.k;
        const long long cap = std::min<long long>(2048, std::max<long long>(256, 9 * 256 / taps_per_vec));
        if (p.mode == 1 && p.k * p.k >= 16)  // (a warp to a vector: one tile a CTA while that is a few vectors a warp)
            p.tile_elems = (int)std::max<long long>(8, std::min<long long>(64, (total + 8LL * sm_count - 1) / (8LL * sm_count) / 8 * 8 + 8));
        else
            p.tile_elems = (int)std::max<long long>(64, std::min<long long>(cap, total / (4LL * sm_count) / 8 * 8));
    }
    p.total_tiles = (int)((total + p.tile_elems - 1) / p.tile_elems);
    return (int)std::max<long long>(1, std::min<long long>((long long)sm_count * per_sm, p.total_tiles));
}

cudaError_t pool_launch(const PoolParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    return launch_layer(pool_instance(p), grid, kPoolThreads, 0, s, p, blp);
}

}  // namespace gpx
