// Sweeps of the device functions that stand in for divisions, pow and erff, against double or long double
// on the host and against the functions they stand in for.  Prints one line "name value..." per sweep.
#include "act_layout.h"
#include "quotients.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

using namespace gpx;

#define CHECK(x)                                                                      \
    do {                                                                              \
        cudaError_t e_ = (x);                                                         \
        if (e_ != cudaSuccess) {                                                      \
            printf("error %s: %s\n", #x, cudaGetErrorString(e_));                     \
            exit(1);                                                                  \
        }                                                                             \
    } while (0)

__device__ unsigned long long g_count[4];

static void counts(unsigned long long (&out)[4]) {
    CHECK(cudaDeviceSynchronize());
    CHECK(cudaMemcpyFromSymbol(out, g_count, sizeof(out)));
    unsigned long long zero[4] = {0, 0, 0, 0};
    CHECK(cudaMemcpyToSymbol(g_count, zero, sizeof(zero)));
}

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

// What became of one quotient: 0 the division's, 1 an infinity or NaN (callers keep clear of those), 2 a numerator below
// 2^-100 that misses by one or two in the last place, 3 wrong.
__device__ int judge(float a, float b, float q) {
    if (!(largest(q, 0.f, 0.f) <= 3.402823466e38f)) return 1;
    const float want = __fdiv_rn(a, b);
    if (same(q, want)) return 0;
    const int off = abs((int)(__float_as_uint(q) & 0x7fffffffu) - (int)(__float_as_uint(want) & 0x7fffffffu));
    return fabsf(a) < 7.8886091e-31f && off <= 2 && q * want >= 0.f ? 2 : 3;
}

// Counts of each over every float as numerator; `any`: div_by_any, of which infinite quotients count too unless
// a negative one overflows.
__global__ void every_numerator(float b, bool given, float y_given, bool any) {
    const float y = given ? y_given : __frcp_rn(b);
    unsigned n[4] = {0, 0, 0, 0};
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32); i += (unsigned long long)gridDim.x * blockDim.x) {
        const float a = __uint_as_float((unsigned)i);
        const float q = any ? div_by_any(a, b, y) : div_by(a, b, y);
        int j = judge(a, b, q);
        if (any && j == 1 && !(a < 0.f && a >= -3.402823466e38f) && !same(q, __fdiv_rn(a, b))) j = 3;
        for (int k = 0; k < 4; ++k) n[k] += j == k;
    }
    for (int k = 0; k < 4; ++k) atomicAdd(&g_count[k], n[k]);
}

__global__ void every_reciprocal() {
    unsigned wrong = 0, wrong_d = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (1u << 23); i += gridDim.x * blockDim.x)
        for (int e = -125; e < 100; e += 25) {
            const float b = __uint_as_float((unsigned)(e + 127) << 23 | i);
            if (!same(reciprocal(b), __frcp_rn(b))) ++wrong;
            if (fabs(reciprocal((double)b) * b - 1.0) > 4.5e-16) ++wrong_d;
        }
    atomicAdd(&g_count[0], wrong);
    atomicAdd(&g_count[1], wrong_d);
}

__device__ unsigned mix(unsigned long long x) {
    x ^= x >> 31, x *= 0x7fb5d329728ea185ull, x ^= x >> 27, x *= 0x81dadef4bc2dd44dull, x ^= x >> 33;
    return (unsigned)x;
}

// Counts of each over pseudo-random pairs with 2^-24 <= b < 2^24, every eighth numerator and divisor from a list of
// extremes; in double over all positive finite b, wrong ones counted as 3.
__global__ void pairs(unsigned long long n) {
    const unsigned extreme[] = {0u, 0x80000000u, 1u, 0x80000001u, 0x007fffffu, 0x00800000u, 0x7f7fffffu, 0x7f800000u, 0xff800000u, 0x7fc00000u,
                                0x3f800000u, 0xbf800000u, 0x3f7fffffu, 0x3fffffffu, 0x0d800000u, 0x4b7fffffu};
    unsigned c[4] = {0, 0, 0, 0};
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
        unsigned ua = mix(2 * i + 1), ub = mix(2 * i + 2) & 0x7fffffffu;
        if (i % 8 == 0) ua = extreme[ua % 16];
        if (i % 16 < 2) ub = extreme[ub % 16] & 0x7fffffffu;
        const float a = __uint_as_float(ua), any = __uint_as_float(ub);
        const float b = __uint_as_float((ub & 0x007fffffu) | (127 - 24 + ub / 0x00800000u % 48) << 23);
        const int j = judge(a, b, div_by(a, b, reciprocal(b)));
        for (int k = 0; k < 4; ++k) c[k] += j == k;
        // in double the divisor is positive and both are finite floats
        if (any > 0.f && any <= 3.402823466e38f && fabsf(a) <= 3.402823466e38f) {
            const double d = div_by((double)a, (double)any, reciprocal((double)any)), want = __ddiv_rn((double)a, (double)any);
            if (__double_as_longlong(d) != __double_as_longlong(want)) ++c[3];
        }
    }
    for (int k = 0; k < 4; ++k) atomicAdd(&g_count[k], c[k]);
}

__global__ void powers(int n, const double *x, double g, double *mine, double *cuda) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        mine[i] = power(x[i], g);
        cuda[i] = pow(x[i], g);
    }
}

__global__ void gelus(int n, const float *x, float *mine, float *with_erff) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        mine[i] = apply_act(x[i], ACT_GELU);
        with_erff[i] = 0.5f * x[i] * (1.0f + erff(x[i] * 0.70710678118654752440f));
    }
}

template <typename T>
struct Buf {
    T *d;
    std::vector<T> h;
    explicit Buf(size_t n) : h(n) { CHECK(cudaMalloc(&d, n * sizeof(T))); }
    ~Buf() { cudaFree(d); }
    void up() { CHECK(cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice)); }
    void down() { CHECK(cudaMemcpy(h.data(), d, h.size() * sizeof(T), cudaMemcpyDeviceToHost)); }
};

int main() {
    unsigned long long c[4];
    CHECK(cudaFree(nullptr));
    counts(c);
    every_reciprocal<<<1024, 256>>>();
    counts(c);
    printf("reciprocal %llu %llu\n", c[0], c[1]);
    for (float b : {12.f, 6.25f, 5.9999995f, 20000.f / 3200, 20000.f / 2999, 10000.f / 1601, 10000.f / 53, 0.3f}) {
        for (bool any : {false, true}) {
            every_numerator<<<2368, 256>>>(b, b == 12.f, 1.f / 12.f, any);
            counts(c);
            printf("numerators %llu %llu %llu %llu\n", c[0], c[1], c[2], c[3]);
        }
    }
    pairs<<<2368, 256>>>(1ull << 32);
    counts(c);
    printf("pairs %llu %llu %llu %llu\n", c[0], c[1], c[2], c[3]);

    // power: relative error in units of 1e-16, this and pow's, inside the range and at its edges
    const double gamma = (double)1.40027894002789400278940027894f;
    const double ranges[][2] = {{1.6e-5, 1e-3}, {1e-3, 0.5}, {0.5, 2.0}, {2.0, 400.0}, {400.0, 65535.0}};
    const int n = 1 << 20;
    Buf<double> x(n), a(n), b(n);
    for (auto &r : ranges) {
        for (int i = 0; i < n; ++i) x.h[i] = r[0] * pow(r[1] / r[0], (i + 0.37) / n);
        x.up();
        powers<<<1024, 256>>>(n, x.d, gamma, a.d, b.d);
        a.down(), b.down();
        long double worst = 0, worst_pow = 0;
        for (int i = 0; i < n; ++i) {
            const long double e = powl((long double)x.h[i], (long double)gamma);
            worst = fmaxl(worst, fabsl(a.h[i] - e) / e);
            worst_pow = fmaxl(worst_pow, fabsl(b.h[i] - e) / e);
        }
        int differ = 0;  // as a float pressure
        for (int i = 0; i < n; ++i) differ += (float)(27.562941f * a.h[i]) != (float)(27.562941f * b.h[i]);
        printf("power %.3f %.3f %d\n", (double)(worst * 1e16L), (double)(worst_pow * 1e16L), differ);
    }
    {
        const double odd[] = {0.0, -0.0, -1.0, 1e-300, 1e300, INFINITY, -INFINITY, NAN, 1.52587890625e-05, 65536.0, 1e-5, 1e5, 5e-324};
        const int m = (int)(sizeof(odd) / sizeof(odd[0]));
        for (int i = 0; i < m; ++i) x.h[i] = odd[i];
        x.up();
        powers<<<1, 32>>>(m, x.d, gamma, a.d, b.d);
        a.down(), b.down();
        int differ = 0;
        for (int i = 0; i < m; ++i) differ += memcmp(&a.h[i], &b.h[i], 8) != 0 && !(std::isnan(a.h[i]) && std::isnan(b.h[i]));
        printf("power_outside %d\n", differ);
    }

    // GELU: largest and mean square error against double, this and the form with erff
    const float bounds[] = {-20.f, -13.f, -9.f, -6.f, -4.f, -3.f, -2.f, -1.25f, -0.5f, -0.1f, 0.f, 0.1f, 0.5f, 1.f, 1.25f, 2.f, 3.f, 6.f, 20.f};
    const int k = 1 << 21;
    Buf<float> v(k), p(k), q(k);
    for (size_t r = 0; r + 1 < sizeof(bounds) / sizeof(bounds[0]); ++r) {
        for (int i = 0; i < k; ++i) v.h[i] = bounds[r] + (bounds[r + 1] - bounds[r]) * ((float)i / k);
        v.up();
        gelus<<<1024, 256>>>(k, v.d, p.d, q.d);
        p.down(), q.down();
        double worst[2] = {0, 0}, sum[2] = {0, 0}, rel = 0;
        for (int i = 0; i < k; ++i) {
            const double t = v.h[i], e = 0.5 * t * erfc(-t * 0.70710678118654752440);
            const double d[2] = {fabs(p.h[i] - e), fabs(q.h[i] - e)};
            for (int j = 0; j < 2; ++j) worst[j] = fmax(worst[j], d[j]), sum[j] += d[j] * d[j];
            if (e != 0) rel = fmax(rel, d[0] / fabs(e));
        }
        printf("gelu %g %g %.4g %.4g %.4g %.4g %.4g\n", bounds[r], bounds[r + 1], worst[0], worst[1], sqrt(sum[0] / k), sqrt(sum[1] / k), rel);
    }
    {
        const float odd[] = {INFINITY, -INFINITY, NAN, 3e38f, -3e38f, 0.f, -0.f, 1e-40f, -1e-40f, 1.25f, -1.25f};
        const int m = (int)(sizeof(odd) / sizeof(odd[0]));
        for (int i = 0; i < m; ++i) v.h[i] = odd[i];
        v.up();
        gelus<<<1, 32>>>(m, v.d, p.d, q.d);
        p.down();
        printf("gelu_odd");
        for (int i = 0; i < m; ++i) printf(" %.9g", p.h[i]);
        printf("\n");
    }
    return 0;
}
