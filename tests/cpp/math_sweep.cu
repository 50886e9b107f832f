// Sweep of the device function that stands in for erff in GELU, against double on the host and against the form
// with erff.  Prints one line "name value..." per sweep.
#include "act_layout.h"

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
