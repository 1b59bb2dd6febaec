// Host program of test_gpu_fft_codelets.py: the register transforms of fft.cuh on packed values (one complex
// value, or a pair) against the same transforms written one part at a time for the compiler to contract,
// bit for bit; with twiddles the two packed forms against each other (how a scalar product contracts there
// depends on what surrounds it).
#include "../optimizec_b200/csrc/fft.cuh"

#include <cstdio>
#include <cstring>
#include <vector>

using namespace dns2d;

// one butterfly per thread: twiddles (as before the second and later stages of a transform; butterflies 2i
// and 2i + 1 have the same, as a pair has), then the R-point transform
template <int R, bool INV, bool TW, class V>
__global__ void k_single(const float2 *x, const float2 *w, float2 *y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    V v[R];
    for (int r = 0; r < R; ++r) v[r] = V{x[i * R + r].x, x[i * R + r].y};
    if (TW)
        for (int r = 1; r < R; ++r) v[r] = ctwiddle<INV>(v[r], w[(i / 2) * R + r]);
    DFT<R, INV>::run(v);
    for (int r = 0; r < R; ++r) y[i * R + r] = make_float2(v[r].x, v[r].y);
}

// butterflies 2i and 2i + 1 side by side
template <int R, bool INV, bool TW>
__global__ void k_pair(const float2 *x, const float2 *w, float2 *y, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n / 2) return;
    cpair v[R];
    const float2 *a = x + (size_t)2 * i * R, *b = a + R;
    for (int r = 0; r < R; ++r) v[r] = {make_float2(a[r].x, b[r].x), make_float2(a[r].y, b[r].y)};
    if (TW)
        for (int r = 1; r < R; ++r) v[r] = ctwiddle<INV>(v[r], w[i * R + r]);
    DFT<R, INV>::run(v);
    float2 *ya = y + (size_t)2 * i * R, *yb = ya + R;
    for (int r = 0; r < R; ++r) {
        ya[r] = make_float2(v[r].re.x, v[r].im.x);
        yb[r] = make_float2(v[r].re.y, v[r].im.y);
    }
}

static int failed = 0;
static float2 *x, *w, *a, *b;
constexpr int kN = 4096;

static void compare(const char *what, int R, bool inv, bool tw)
{
    std::vector<float2> A((size_t)kN * R), B(A.size());
    const cudaError_t e = cudaDeviceSynchronize();
    cudaMemcpy(A.data(), a, A.size() * 8, cudaMemcpyDeviceToHost);
    cudaMemcpy(B.data(), b, B.size() * 8, cudaMemcpyDeviceToHost);
    size_t d = 0;
    for (size_t i = 0; i < A.size(); ++i) d += A[i].x != B[i].x || A[i].y != B[i].y;
    if (d || e != cudaSuccess) {
        std::printf("%s R=%d inverse=%d twiddles=%d: %zu of %zu differ (%s)\n", what, R, inv, tw, d, A.size(),
                    cudaGetErrorString(e));
        ++failed;
    }
}

template <int R, bool INV>
static void check()
{
    const int g = (kN + 127) / 128;
    k_single<R, INV, false, cscalar><<<g, 128>>>(x, w, a, kN);
    k_single<R, INV, false, float2><<<g, 128>>>(x, w, b, kN);
    compare("packed, scalar", R, INV, false);
    k_pair<R, INV, false><<<g, 128>>>(x, w, b, kN);
    compare("pair, scalar", R, INV, false);
    k_single<R, INV, true, float2><<<g, 128>>>(x, w, a, kN);
    k_pair<R, INV, true><<<g, 128>>>(x, w, b, kN);
    compare("pair, packed", R, INV, true);
}

template <int R>
static void all()
{
    check<R, false>();
    check<R, true>();
}

int main()
{
    const size_t m = (size_t)kN * 32;
    std::vector<float2> hx(m), hw(m);
    unsigned s = 12345u;
    auto next = [&] { return (float)((s = s * 1664525u + 1013904223u) >> 8) * (1.0f / 16777216.0f) - 0.5f; };
    for (auto &v : hx) v = make_float2(next(), next());
    for (auto &v : hw) v = make_float2(next(), next());
    for (float2 **p : {&x, &w, &a, &b})
        if (cudaMalloc((void **)p, m * 8) != cudaSuccess) return 2;
    cudaMemcpy(x, hx.data(), m * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(w, hw.data(), m * 8, cudaMemcpyHostToDevice);
    all<3>();
    all<4>();
    all<6>();
    all<8>();
    all<12>();
    all<16>();
    all<24>();
    std::printf(failed ? "%d comparisons failed\n" : "ok\n", failed);
    return failed != 0;
}
