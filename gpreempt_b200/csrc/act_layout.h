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
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 x, y, r;\n\t"
        "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 r, x, y;\n\tmov.b64 {%0, %1}, r;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long &>(r))
        : "l"(reinterpret_cast<unsigned long long &>(a)), "l"(reinterpret_cast<unsigned long long &>(b)));
    return r;
}

// Exact GELU, v * Phi(v), for two values, as accurate as 0.5 v (1 + erff(v / sqrt 2)) or more so everywhere.
// |v| < 1.25: Phi(v) = 1/2 + v W(v*v), W of degree 5 (minimax, 2.2e-9 in Phi).  Beyond: v Phi(v) =
// max(v, 0) - |v| Phi(-|v|) with Phi(-z) = 2^p(z), p of degree 7 (minimax of log2 Phi(-z) weighted for
// the error of the product, 5e-9, fitted over 1.25 <= z <= 6; it falls on until 2^p is zero, which the
// bound of 14 on z reaches).  The tail of negative v so keeps its leading digits, which 1 + erf cancels
// away.  Largest error against double, in brackets that of the form with erff: |v| < 0.1 5.0e-9
// (5.2e-9), < 1 7.4e-8 (8.6e-8), < 3 1.4e-7 (3.0e-7), < 6 2.4e-7 (4.9e-7); relative, between -4 and -3, 4e-6
// (9e-4).  A 768 -> 3072 layer of 16 384 rows, whose epilogue this is: 175 us with erff when its products took 115,
// 79 with both as they are now.
__device__ __forceinline__ float2 gelu2(float a, float b) {
    auto c = [](float v) { return make_float2(v, v); };
    const float2 v = make_float2(a, b), u = mul2(v, v);
    float2 w = fma2(c(-6.65244033e-06f), u, c(0.000110361892f));
    w = fma2(w, u, c(-0.00118276756f));
    w = fma2(w, u, c(0.00997154508f));
    w = fma2(w, u, c(-0.066490002f));
    w = fma2(w, u, c(0.398942262f));
    const float2 mid = mul2(v, fma2(v, w, c(0.5f)));
    const float2 z = make_float2(fminf(fabsf(a), 14.f), fminf(fabsf(b), 14.f));
    float2 q = fma2(c(-2.00619388e-06f), z, c(6.50551447e-05f));
    q = fma2(q, z, c(-0.000957242271f));
    q = fma2(q, z, c(0.00860437006f));
    q = fma2(q, z, c(-0.0541074574f));
    q = fma2(q, z, c(-0.458460182f));
    q = fma2(q, z, c(-1.15104771f));
    q = fma2(q, z, c(-1.0001303f));
    float2 e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(q.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(q.y));
    // (NaN takes the middle form and stays NaN)
    return make_float2(fabsf(a) >= 1.25f ? fmaf(-z.x, e.x, fmaxf(a, 0.f)) : mid.x,
                       fabsf(b) >= 1.25f ? fmaf(-z.y, e.y, fmaxf(b, 0.f)) : mid.y);
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
