// Storage layout of an activation tensor in HBM.
//
// Activations between layers are kept as two bf16 planes (hi, lo) with x ~= hi + lo: 16 bits of
// mantissa, which is what the tensor-core convolution consumes directly (three bf16 products
// hi*hi + hi*lo + lo*hi stand in for one fp32 product).  Each plane is a row-major matrix
// [rows][C]: one row per stored pixel, channels contiguous, so every convolution is a GEMM over
// rows and a filter tap is a constant row shift.  Three row orders exist:
//   plain            row = (n*H + h)*W + w
//   padded           one zero pixel around every image: row = (n*(H+2) + h+1)*(W+2) + w+1
//                    (input of a 3x3 stride-1 convolution: a tap (fh,fw) is the row shift
//                    (fh-1)*(W+2) + (fw-1), and the zero border supplies the padding)
//   phased           the padded image split into its four (row parity, column parity) planes,
//                    plane-major (input of a 3x3 stride-2 convolution: tap (fh,fw) reads plane
//                    (fh&1, fw&1) shifted by (fh>>1, fw>>1), again a constant row shift)
// Border rows are zeroed once at allocation and never written.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define GPX_HD __host__ __device__ __forceinline__
#else
#define GPX_HD inline
#endif

namespace gpx {

enum ActOrder : int { ACT_PLAIN = 0, ACT_PADDED = 1, ACT_PHASED = 2 };

// Element format of the planes: two bf16 planes hi + lo (float32 models), or one plane of bf16
// or fp16 (the reduced-precision models).
enum PlaneFmt : int { PF_SPLIT = 0, PF_BF16 = 1, PF_F16 = 2 };

struct ActLayout {
    int N, H, W, C;  // logical shape
    int order;       // ActOrder
    int Hs, Ws;      // stored rows / columns per image (per phase plane when phased)
    int plane;       // rows of one phase plane (N*Hs*Ws); equals rows when not phased
    int rows;        // stored rows in total
    int fmt;         // PlaneFmt of the planes that hold the tensor
};

inline ActLayout make_layout(int N, int H, int W, int C, int order) {
    ActLayout l;
    l.N = N;
    l.H = H;
    l.W = W;
    l.C = C;
    l.order = order;
    l.fmt = PF_SPLIT;
    if (order == ACT_PLAIN) {
        l.Hs = H;
        l.Ws = W;
    } else if (order == ACT_PADDED) {
        l.Hs = H + 2;
        l.Ws = W + 2;
    } else {
        l.Hs = (H + 2) / 2;
        l.Ws = (W + 2) / 2;
    }
    l.plane = N * l.Hs * l.Ws;
    l.rows = order == ACT_PHASED ? 4 * l.plane : l.plane;
    return l;
}

// Stored row of logical pixel (n, h, w).
GPX_HD int layout_row(const ActLayout &l, int n, int h, int w) {
    if (l.order == ACT_PLAIN) return (n * l.Hs + h) * l.Ws + w;
    if (l.order == ACT_PADDED) return (n * l.Hs + h + 1) * l.Ws + w + 1;
    int hp = h + 1, wp = w + 1;
    int ph = ((hp & 1) << 1) | (wp & 1);
    return ph * l.plane + (n * l.Hs + (hp >> 1)) * l.Ws + (wp >> 1);
}

// Activation fused into a layer's epilogue.
enum ActKind : int { ACT_NONE = 0, ACT_RELU = 1, ACT_GELU = 2, ACT_RELU6 = 3 };

#if defined(__CUDACC__)
// Exact GELU, v * Phi(v) with Phi(v) = erfc(-v / sqrt 2) / 2.  The complementary error function is the
// Chebyshev fit t * exp(-z*z + P(t)), t = 1 / (1 + z/2), z = |v| / sqrt 2, of W. J. Cody's form as
// printed in Press et al., Numerical Recipes, section 6.2 ("erfcc"): relative error below 1.2e-7
// everywhere, so the tail of negative v keeps its leading digits, which 1 + erf(v / sqrt 2) cancels
// away.  Two elements share each step (packed fp32 FMA); with erff per element the epilogue of a
// 768 -> 3072 layer took longer than its products (175 us against 115 us for 3072 -> 768 at 16 384 rows).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)),
          "l"(reinterpret_cast<unsigned long long &>(c)));
    return r;
}
__device__ __forceinline__ float2 gelu2(float a, float b) {
    const float2 z = make_float2(fabsf(a) * 0.70710678118654752440f, fabsf(b) * 0.70710678118654752440f);
    float2 t;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.x) : "f"(fmaf(0.5f, z.x, 1.0f)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.y) : "f"(fmaf(0.5f, z.y, 1.0f)));
    auto c = [](float v) { return make_float2(v, v); };
    float2 p = fma2(c(0.17087277f), t, c(-0.82215223f));
    p = fma2(p, t, c(1.48851587f));
    p = fma2(p, t, c(-1.13520398f));
    p = fma2(p, t, c(0.27886807f));
    p = fma2(p, t, c(-0.18628806f));
    p = fma2(p, t, c(0.09678418f));
    p = fma2(p, t, c(0.37409196f));
    p = fma2(p, t, c(1.00002368f));
    p = fma2(p, t, c(-1.26551223f));
    p = fma2(make_float2(-z.x, -z.y), z, p);
    const float log2e = 1.4426950408889634f;
    float2 e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(p.x * log2e));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(p.y * log2e));
    const float hx = 0.5f * t.x * e.x, hy = 0.5f * t.y * e.y;  // Phi(-|v|)
    return make_float2(a * (a > 0.f ? 1.0f - hx : hx), b * (b > 0.f ? 1.0f - hy : hy));
}

__device__ __forceinline__ float apply_act(float v, int act) {
    if (act == ACT_RELU) return fmaxf(v, 0.f);
    if (act == ACT_GELU) return gelu2(v, v).x;
    if (act == ACT_RELU6) return fminf(fmaxf(v, 0.f), 6.f);
    return v;
}

// The same over a register array, with the (warp-uniform) choice made once outside the element
// loop: inside it the compiler would otherwise evaluate the erf of GELU for every element of every
// layer and select afterwards.  N is even.
template <int N>
__device__ __forceinline__ void apply_act_n(float (&f)[N], int act) {
    if (act == ACT_RELU) {
#pragma unroll
        for (int j = 0; j < N; ++j) f[j] = fmaxf(f[j], 0.f);
    } else if (act == ACT_RELU6) {
#pragma unroll
        for (int j = 0; j < N; ++j) f[j] = fminf(fmaxf(f[j], 0.f), 6.f);
    } else if (act == ACT_GELU) {
#pragma unroll
        for (int j = 0; j < N; j += 2) {
            const float2 g = gelu2(f[j], f[j + 1]);
            f[j] = g.x;
            f[j + 1] = g.y;
        }
    }
}
#endif

}  // namespace gpx
