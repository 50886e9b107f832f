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
// Packed fp32 arithmetic on two values (one instruction each on sm_100).
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)),
          "l"(reinterpret_cast<unsigned long long &>(c)));
    return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
    return r;
}

// Exact GELU, v * Phi(v) = max(v, 0) - |v| * Phi(-|v|), for two values.  Phi(-|v|) = erfc(z) / 2 with
// z = |v| / sqrt 2, and erfc(z) = exp(-z*z) * t * Q(t) with t = 1 / (1 + 0.37 z): the substitution of
// Hastings (Abramowitz and Stegun 7.1.26) with the exponential and the leading t factored out, and Q
// the degree-6 minimax polynomial of that quotient (own fit over 0 <= z <= 6.5: relative error 3.7e-7,
// 7e-7 evaluated in fp32).  The error is relative, so the tail of negative v keeps its leading digits,
// which 1 + erf(v / sqrt 2) cancels away.  Both reciprocals come from one: the special-function unit
// bounds this (1.5 of its operations an element).  With erff per element the epilogue of a
// 768 -> 3072 layer took longer than its products (175 us against 115 us for 3072 -> 768, 16 384 rows).
__device__ __forceinline__ float2 gelu2(float a, float b) {
    auto c = [](float v) { return make_float2(v, v); };
    // (beyond 64 the exponential is zero: the bound only keeps infinities out of the products)
    const float ua = fminf(fabsf(a), 64.f), ub = fminf(fabsf(b), 64.f);
    const float d0 = fmaf(0.261629508f, ua, 1.0f), d1 = fmaf(0.261629508f, ub, 1.0f);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d0 * d1));
    const float2 t = mul2(c(r), make_float2(d1, d0));
    // Q / 2
    float2 q = fma2(c(-0.0729324635f), t, c(0.22384969f));
    q = fma2(q, t, c(-0.102016685f));
    q = fma2(q, t, c(0.1653087285f));
    q = fma2(q, t, c(0.073651064f));
    q = fma2(q, t, c(0.107995136f));
    q = fma2(q, t, c(0.104144361f));
    const float2 v = make_float2(a, b);
    const float2 x = mul2(mul2(v, c(-0.72134752044f)), v);  // -z*z * log2(e)
    float2 e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(x.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(x.y));
    const float2 h = mul2(mul2(q, t), e);
    return make_float2(fmaf(-ua, h.x, fmaxf(a, 0.f)), fmaf(-ub, h.y, fmaxf(b, 0.f)));
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
