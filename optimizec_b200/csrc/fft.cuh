// fft.cuh — shared-memory Stockham FFT engine for the B200 (sm_100a) DNS kernels.
//
// A transform of compile-time length L runs as a sequence of radix-R stages
// (radix plan = template list).  Each stage reads its R inputs per butterfly from shared
// memory into registers, applies the inter-stage twiddles W_{Ns*R}^{r*k} (looked up in
// FP64-built, once-rounded per-stage tables held in global memory / L1), performs the R-point
// DFT fully unrolled in registers (generic Cooley-Tukey codelets whose constants are folded at
// compile time) and writes the R outputs back in Stockham auto-sort order.  Several arrays
// (rows or columns of the DNS fields) can be transformed together by one CTA.
//
// Conventions: forward = exp(-2 pi i jk/L), inverse = exp(+2 pi i jk/L), both unnormalised,
// the same as the reference's cuFFT R2C/C2R calls (cuda/vfft_cuda.cu:14-42).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

namespace dns2d {

// ------------------------------------------------------------------------------------------
// compile-time trigonometry for codelet constants: cos/sin(2 pi k / R) by Taylor series on an
// angle reduced to [-pi, pi]; the results are rounded to float, so double accuracy suffices.
// ------------------------------------------------------------------------------------------
constexpr double kPi = 3.14159265358979323846264338327950288;

constexpr double ct_series_sin(double x)
{
    double x2 = x * x, term = x, sum = x;
    for (int n = 1; n < 20; ++n) {
        term *= -x2 / (double)((2 * n) * (2 * n + 1));
        sum += term;
    }
    return sum;
}

constexpr double ct_series_cos(double x)
{
    double x2 = x * x, term = 1.0, sum = 1.0;
    for (int n = 1; n < 20; ++n) {
        term *= -x2 / (double)((2 * n - 1) * (2 * n));
        sum += term;
    }
    return sum;
}

constexpr double ct_angle(int k, int R)
{
    int m = ((k % R) + R) % R;
    if (2 * m > R) m -= R;  // reduce to [-pi, pi]
    return 2.0 * kPi * (double)m / (double)R;
}

constexpr double ct_cos(int k, int R) { return ct_series_cos(ct_angle(k, R)); }
constexpr double ct_sin(int k, int R) { return ct_series_sin(ct_angle(k, R)); }

constexpr int ct_first_factor(int R)
{
    if (R % 4 == 0 && R != 4) return 4;
    for (int f = 2; f * f <= R; ++f)
        if (R % f == 0) return f;
    return R;
}

constexpr bool ct_is_prime(int R) { return R > 1 && ct_first_factor(R) == R; }

template <int B, int E, class F>
__device__ __forceinline__ void static_for(F &&f)
{
    if constexpr (B < E) {
        f(std::integral_constant<int, B>{});
        static_for<B + 1, E>(f);
    }
}

// ------------------------------------------------------------------------------------------
// complex helpers
// ------------------------------------------------------------------------------------------
// Additions, scalings and rotations of both parts are packed FP32 instructions (two results for one issue
// slot; the butterflies are mostly additions): N = 256 / 512 step 12.5 / 22.3 -> 12.0 / 20.6 us, the
// 64-member ensemble 130 -> 125 us per step on B200, with the rounding of the scalar expressions (see crot).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 cmul_mi(float2 a)
{
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// a + (-i) b (forward) or a + i b (inverse)
template <bool INV>
__device__ __forceinline__ float2 cadd_mi(float2 a, float2 b)
{
    return cadd(a, cmul_mi<INV>(b));
}
// m + f t, f real
__device__ __forceinline__ float2 cfma(float2 t, float f, float2 m) { return __ffma2_rn(t, make_float2(f, f), m); }
// m + (-i) f t (forward) or m + i f t (inverse), f real
template <bool INV>
__device__ __forceinline__ float2 cfma_mi(float2 t, float f, float2 m)
{
    return INV ? make_float2(fmaf(-t.y, f, m.x), fmaf(t.x, f, m.y)) : make_float2(fmaf(t.y, f, m.x), fmaf(-t.x, f, m.y));
}
// a (c + i s)
//
// Which of its two products an FMA rounds is fixed here so that the results equal, bit for bit, those of
// the scalar expression (a.x c - a.y s, a.x s + a.y c) as the compiler contracts it: the real part keeps
// a.x c exact, the imaginary part a.x s, or (ALT) a.y c where the sum is written as a difference.  Which
// rotations take ALT was found by comparison with nvcc 12.9's scalar code, not derived: tests/fft_codelets.cu
// compares the packed forms with the scalar one (cscalar) bit for bit, so a compiler that contracts otherwise
// shows there.
template <bool ALT = false>
__device__ __forceinline__ float2 crot(float2 a, float c, float s)
{
    if (ALT) return __ffma2_rn(a, make_float2(c, c), __fmul2_rn(make_float2(a.y, a.x), make_float2(-s, s)));
    return __ffma2_rn(make_float2(a.x, a.x), make_float2(c, s), __fmul2_rn(make_float2(a.y, a.y), make_float2(-s, c)));
}
__device__ __forceinline__ void czero(float2 &a) { a = make_float2(0.f, 0.f); }

// A complex value whose operations are written one part at a time, for the compiler to contract: the
// 4-CTA cluster kernels (radices that the packed forms below were not compared for) and the large-grid
// diagnostics.
struct cscalar {
    float x, y;
};
__device__ __forceinline__ cscalar cadd(cscalar a, cscalar b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ cscalar csub(cscalar a, cscalar b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ cscalar cscale(cscalar a, float s) { return {a.x * s, a.y * s}; }
__device__ __forceinline__ cscalar cmul(cscalar a, float2 b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
template <bool INV>
__device__ __forceinline__ cscalar cmul_mi(cscalar a)
{
    return INV ? cscalar{-a.y, a.x} : cscalar{a.y, -a.x};
}
template <bool INV>
__device__ __forceinline__ cscalar cadd_mi(cscalar a, cscalar b)
{
    return cadd(a, cmul_mi<INV>(b));
}
__device__ __forceinline__ cscalar cfma(cscalar t, float f, cscalar m) { return {m.x + f * t.x, m.y + f * t.y}; }
template <bool INV>
__device__ __forceinline__ cscalar cfma_mi(cscalar t, float f, cscalar m)
{
    return cadd(m, cmul_mi<INV>(cscale(t, f)));
}
template <bool ALT = false>
__device__ __forceinline__ cscalar crot(cscalar a, float c, float s)
{
    return {a.x * c - a.y * s, a.x * s + a.y * c};
}
__device__ __forceinline__ void czero(cscalar &a) { a = {0.f, 0.f}; }

// Two complex values side by side, (re, re') and (im, im'): every operation of a butterfly is one
// packed instruction on both, with no exchange of halves (a float2 value needs the halves swapped
// for each multiplication by i or by a twiddle).
struct cpair {
    float2 re, im;
};
__device__ __forceinline__ cpair cadd(cpair a, cpair b) { return {cadd(a.re, b.re), cadd(a.im, b.im)}; }
__device__ __forceinline__ cpair csub(cpair a, cpair b) { return {csub(a.re, b.re), csub(a.im, b.im)}; }
__device__ __forceinline__ cpair cscale(cpair a, float s) { return {cscale(a.re, s), cscale(a.im, s)}; }
__device__ __forceinline__ cpair cfma(cpair t, float f, cpair m) { return {cfma(t.re, f, m.re), cfma(t.im, f, m.im)}; }
template <bool INV>
__device__ __forceinline__ cpair cfma_mi(cpair t, float f, cpair m)
{
    return INV ? cpair{cfma(t.im, -f, m.re), cfma(t.re, f, m.im)} : cpair{cfma(t.im, f, m.re), cfma(t.re, -f, m.im)};
}
template <bool ALT = false>
__device__ __forceinline__ cpair crot(cpair a, float c, float s)
{
    return {cfma(a.re, c, cscale(a.im, -s)), ALT ? cfma(a.im, c, cscale(a.re, s)) : cfma(a.re, s, cscale(a.im, c))};
}
template <bool INV>
__device__ __forceinline__ cpair cmul_mi(cpair a)
{
    if constexpr (INV) return {cscale(a.im, -1.f), a.re};
    else return {a.im, cscale(a.re, -1.f)};
}
template <bool INV>
__device__ __forceinline__ cpair cadd_mi(cpair a, cpair b)
{
    if constexpr (INV) return {csub(a.re, b.im), cadd(a.im, b.re)};
    else return {cadd(a.re, b.im), csub(a.im, b.re)};
}
// the squares (u + i w)^2 = u^2 - w^2 + 2 i u w of a pair, the imaginary part as its two factors: the sum or
// difference of two is one rounding fewer, a FMA on one product (again as the compiler contracts the
// scalar expressions)
struct csquare {
    float2 re, u2, w;
};
__device__ __forceinline__ csquare square(cpair a)
{
    return {__ffma2_rn(a.re, a.re, __fmul2_rn(cscale(a.im, -1.f), a.im)), cadd(a.re, a.re), a.im};
}
__device__ __forceinline__ cpair cadd(csquare a, csquare b)
{
    return {cadd(a.re, b.re), __ffma2_rn(a.u2, a.w, __fmul2_rn(b.u2, b.w))};
}
__device__ __forceinline__ cpair csub(csquare a, csquare b)
{
    return {csub(a.re, b.re), __ffma2_rn(a.u2, a.w, __fmul2_rn(cscale(b.u2, -1.f), b.w))};
}
__device__ __forceinline__ void czero(cpair &a) { a = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}; }

// a w (forward) or a conj(w) (inverse): the twiddles before a butterfly
template <bool INV, class V>
__device__ __forceinline__ V ctwiddle(V a, float2 w)
{
    if constexpr (std::is_same_v<V, cscalar>) return cmul(a, INV ? cconj(w) : w);
    else return INV ? crot<true>(a, w.x, -w.y) : crot(a, w.x, w.y);
}

// a * W_R^K with W_R = exp(-+ 2 pi i / R); trivial angles become sign swaps.  SWAP: the other order of the
// imaginary part's sum (see crot; where |c| = |s| the compiler shares the products and has one order).
template <int R, int K, bool INV, bool SWAP = false, class V>
__device__ __forceinline__ V twid(V a)
{
    constexpr int k = ((K % R) + R) % R;
    if constexpr (k == 0) {
        return a;
    } else if constexpr (2 * k == R) {
        return cscale(a, -1.f);
    } else if constexpr (4 * k == R) {
        return cmul_mi<INV>(a);
    } else if constexpr (4 * k == 3 * R) {
        return cmul_mi<!INV>(a);
    } else {
        constexpr float c = (float)ct_cos(k, R);
        constexpr float s = INV ? (float)ct_sin(k, R) : -(float)ct_sin(k, R);
        return crot<c != s && c != -s && (c > 0.f && s < 0.f) != SWAP>(a, c, s);
    }
}

// ------------------------------------------------------------------------------------------
// R-point DFT in registers, in place, natural order in and out.
// ------------------------------------------------------------------------------------------
template <int R, bool INV>
struct DFT;

template <bool INV>
struct DFT<1, INV> {
    template <class V>
    static __device__ __forceinline__ void run(V (&)[1]) {}
};

template <bool INV>
struct DFT<2, INV> {
    template <class V>
    static __device__ __forceinline__ void run(V (&v)[2])
    {
        const V a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <bool INV>
struct DFT<3, INV> {
    template <class V>
    static __device__ __forceinline__ void run(V (&v)[3])
    {
        constexpr float h = 0.5f;
        constexpr float s3 = 0.86602540378443864676f;
        const V t1 = cadd(v[1], v[2]);
        const V t2 = csub(v[1], v[2]);
        const V m1 = cfma(t1, -h, v[0]);
        v[0] = cadd(v[0], t1);
        v[1] = cfma_mi<INV>(t2, s3, m1);
        v[2] = cfma_mi<!INV>(t2, s3, m1);
    }
};

template <bool INV>
struct DFT<4, INV> {
    template <class V>
    static __device__ __forceinline__ void run(V (&v)[4])
    {
        run(v, v);
    }
    template <class In, class V>
    static __device__ __forceinline__ void run(const In (&x)[4], V (&v)[4])
    {
        const V t0 = cadd(x[0], x[2]), t1 = csub(x[0], x[2]);
        const V t2 = cadd(x[1], x[3]), t3 = csub(x[1], x[3]);
        v[0] = cadd(t0, t2);
        v[2] = csub(t0, t2);
        v[1] = cadd_mi<INV>(t1, t3);
        v[3] = cadd_mi<!INV>(t1, t3);
    }
};

// odd prime R (5, 7, ...): symmetric pair form with folded constants
template <int R, bool INV, bool PRIME = ct_is_prime(R)>
struct DFTGeneric;

template <int R, bool INV>
struct DFTGeneric<R, INV, true> {
    template <class V>
    static __device__ __forceinline__ void run(V (&v)[R])
    {
        constexpr int M = (R - 1) / 2;
        V s[M + 1], d[M + 1];
        const V x0 = v[0];
        V sum = x0;
        static_for<1, M + 1>([&](auto nc) {
            constexpr int n = decltype(nc)::value;
            s[n] = cadd(v[n], v[R - n]);
            d[n] = csub(v[n], v[R - n]);
            sum = cadd(sum, s[n]);
        });
        static_for<1, M + 1>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            V A = x0;
            V B;
            czero(B);
            static_for<1, M + 1>([&](auto nc) {
                constexpr int n = decltype(nc)::value;
                A = cfma(s[n], (float)ct_cos(n * k, R), A);
                B = cfma(d[n], (float)ct_sin(n * k, R), B);
            });
            // forward: X[k] = A - iB, X[R-k] = A + iB (inverse swaps)
            v[k] = cadd_mi<INV>(A, B);
            v[R - k] = cadd_mi<!INV>(A, B);
        });
        v[0] = sum;
    }
};

template <int SWAP_N2, int R, bool INV, class V>
__device__ __forceinline__ void dft_swapped(V (&v)[R])
{
    if constexpr (SWAP_N2 > 0) DFTGeneric<R, INV>::template run<SWAP_N2>(v);
    else DFT<R, INV>::run(v);
}

// composite R = P * Q, decimation in time:
// X[k1 + P k2] = sum_{n2} W_R^{n2 k1} W_Q^{n2 k2} sum_{n1} x[Q n1 + n2] W_P^{n1 k1}
template <int R, bool INV>
struct DFTGeneric<R, INV, false> {
    // SWAP_N2: a pair whose rotations take the other order of crot in the place that this transform has in a
    // larger one; the rotations of i t differences (INV, P = 4, odd k1) always do
    template <int SWAP_N2 = 0, class V>
    static __device__ __forceinline__ void run(V (&v)[R])
    {
        run<SWAP_N2>(v, v);
    }
    template <int SWAP_N2 = 0, class In, class V>
    static __device__ __forceinline__ void run(const In (&x)[R], V (&v)[R])
    {
        constexpr int P = ct_first_factor(R);
        constexpr int Q = R / P;
        V t[R];
        static_for<0, Q>([&](auto n2c) {
            constexpr int n2 = decltype(n2c)::value;
            In b[P];
            V a[P];
            static_for<0, P>([&](auto n1c) {
                constexpr int n1 = decltype(n1c)::value;
                b[n1] = x[Q * n1 + n2];
            });
            if constexpr (std::is_same_v<In, V>) {
                static_for<0, P>([&](auto n1c) { a[decltype(n1c)::value] = b[decltype(n1c)::value]; });
                DFT<P, INV>::run(a);
            } else {
                DFT<P, INV>::run(b, a);
            }
            static_for<0, P>([&](auto k1c) {
                constexpr int k1 = decltype(k1c)::value;
                constexpr bool SWAP = (INV && P == 4 && k1 % 2 == 1) != (SWAP_N2 > 0 && n2 == SWAP_N2);
                t[k1 * Q + n2] = twid<R, n2 * k1, INV, SWAP>(a[k1]);
            });
        });
        static_for<0, P>([&](auto k1c) {
            constexpr int k1 = decltype(k1c)::value;
            V b[Q];
            static_for<0, Q>([&](auto n2c) {
                constexpr int n2 = decltype(n2c)::value;
                b[n2] = t[k1 * Q + n2];
            });
            dft_swapped<R == 24 && INV && k1 == 3 ? 1 : 0, Q, INV>(b);
            static_for<0, Q>([&](auto k2c) {
                constexpr int k2 = decltype(k2c)::value;
                v[k1 + P * k2] = b[k2];
            });
        });
    }
};

template <int R, bool INV>
struct DFT {
    template <class V>
    static __device__ __forceinline__ void run(V (&v)[R])
    {
        DFTGeneric<R, INV>::run(v);
    }
    template <class In, class V>
    static __device__ __forceinline__ void run(const In (&x)[R], V (&v)[R])
    {
        DFTGeneric<R, INV>::run(x, v);
    }
};

// ------------------------------------------------------------------------------------------
// Shared-memory layout: one float2 of padding every 2^PS elements (PS = 5 by default: bank-
// conflict-free strided butterfly writes for radix 8/16; a plan whose first stage writes at
// stride 16 uses PS = 4), and a per-array stride that shifts consecutive arrays by 8 banks.
// A warp's 8-byte accesses are served per half-warp: conflict-free when the 16 padded indices of
// a half-warp are distinct modulo 16.
// ------------------------------------------------------------------------------------------
template <int PS = 5>
__device__ __forceinline__ int sidx(int i) { return i + (i >> PS); }

// array stride of L padded elements, rounded up to 16 float2 plus EX (EX = 4 by default: consecutive
// arrays 8 banks apart)
template <int L, int PS = 5, int EX = 4>
struct SmemLen {
    static constexpr int raw = L + (L >> PS) + 1;
    static constexpr int value = ((raw + 15) / 16) * 16 + EX;
};

template <int... Rs>
struct Radices {};

template <int... Rs>
constexpr int radix_product(Radices<Rs...>)
{
    return (1 * ... * Rs);
}

// ------------------------------------------------------------------------------------------
// Per-stage twiddle tables.  Stage (R, Ns) of a length-L transform multiplies input r of
// butterfly j by W_{Ns R}^{r k}, k = j mod Ns.  Its table holds those factors as [r-1][k]
// (FP64-built, rounded once), so for fixed r the threads of a warp read consecutive entries.
// A catalog lists the (R, Ns > 1) stages of every plan compiled for one L and their offsets in
// one contiguous table; kernels get the table base and find their stage's offset at compile
// time.
// ------------------------------------------------------------------------------------------
struct TwCatalog {
    int n = 0;
    int total = 0;
    int R[64] = {};
    int NS[64] = {};
    int off[64] = {};
    int outer[64] = {};  // P > 0: index k = i1 + P i2 is stored at i1 (NS / P) + i2
    constexpr int find(int r, int ns, int p = 0) const
    {
        for (int i = 0; i < n; ++i)
            if (R[i] == r && NS[i] == ns && outer[i] == p) return off[i];
        return -1;
    }
    constexpr void add_stage(int r, int ns, int p = 0)
    {
        if (find(r, ns, p) >= 0) return;
        R[n] = r;
        NS[n] = ns;
        outer[n] = p;
        off[n] = total;
        total += (r - 1) * ns;
        ++n;
    }
    // power k of entry `loc` of stage i (its r is loc / NS + 1)
    __host__ __device__ constexpr int index(int i, int loc) const
    {
        const int e = loc % NS[i], p = outer[i], w = p ? NS[i] / p : 1;
        return p ? e / w + p * (e % w) : e;
    }
    constexpr void add_plan(const int *rs, int nr)
    {
        int ns = 1;
        for (int i = 0; i < nr; ++i) {
            if (ns > 1) add_stage(rs[i], ns);
            ns *= rs[i];
        }
    }
    template <int... Rs>
    constexpr void add(Radices<Rs...>)
    {
        const int a[] = {Rs...};
        add_plan(a, (int)sizeof...(Rs));
    }
};

// The thread index read so that the compiler cannot treat it as loop-invariant: inside a
// persistent kernel's work loop, expressions of threadIdx.x would otherwise be hoisted out of
// the loop for every stage of every transform and kept live across it (register spills).
__device__ __forceinline__ int opaque_tid()
{
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

// One Stockham stage over B arrays of length L (array b at s + b*LP); OPQ: read the thread
// index with opaque_tid().
template <class Cat, int L, int LP, int R, int NS, bool INV, int B, int NT, int PS = 5, bool OPQ = false, class V = float2>
__device__ __forceinline__ void fft_stage(float2 *__restrict__ s, const float2 *__restrict__ tw)
{
    const int tid = OPQ ? opaque_tid() : (int)threadIdx.x;
    constexpr int LR = L / R;
    constexpr int TOT = B * LR;
    constexpr int NBF = (TOT + NT - 1) / NT;
    V v[NBF][R];
#pragma unroll
    for (int i = 0; i < NBF; ++i) {
        const int t = tid + i * NT;
        if ((NBF * NT == TOT) || t < TOT) {
            const int b = t / LR;
            const int j = t - b * LR;
            const float2 *x = s + b * LP;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float2 e = x[sidx<PS>(j + r * LR)];
                v[i][r] = V{e.x, e.y};
            }
            if constexpr (NS > 1) {
                constexpr int OFF = Cat::off(R, NS);
                static_assert(OFF >= 0, "stage missing from the twiddle catalog");
                const float2 *t = tw + OFF + j % NS;
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    v[i][r] = ctwiddle<INV>(v[i][r], __ldg(t + (r - 1) * NS));
                }
            }
            DFT<R, INV>::run(v[i]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NBF; ++i) {
        const int t = tid + i * NT;
        if ((NBF * NT == TOT) || t < TOT) {
            const int b = t / LR;
            const int j = t - b * LR;
            float2 *y = s + b * LP;
            const int k = j % NS;
            const int base = (j / NS) * NS * R + k;
#pragma unroll
            for (int q = 0; q < R; ++q) y[sidx<PS>(base + q * NS)] = make_float2(v[i][q].x, v[i][q].y);
        }
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------------------
// One-butterfly-per-thread building blocks (the large-grid kernels).  Butterfly j of a stage
// (radix R, Ns) reads x[j + r L/R] and writes y[(j/Ns) Ns R + j%Ns + q Ns]; with Ns = 1 the
// reads of the first stage can come straight from global memory, and the last stage's outputs
// (Ns = L/R: positions j + q L/R) can go straight back, skipping two shared-memory passes.
// ------------------------------------------------------------------------------------------
template <int R, bool INV>
__device__ __forceinline__ void dft_scalar(float2 (&v)[R])
{
    cscalar c[R];
#pragma unroll
    for (int r = 0; r < R; ++r) c[r] = {v[r].x, v[r].y};
    DFT<R, INV>::run(c);
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = make_float2(c[r].x, c[r].y);
}

template <class Cat, int L, int R, int NS, bool INV>
__device__ __forceinline__ void bfly(float2 (&v)[R], int j, const float2 *__restrict__ tw)
{
    if constexpr (NS > 1) {
        constexpr int OFF = Cat::off(R, NS);
        static_assert(OFF >= 0, "stage missing from the twiddle catalog");
        const float2 *t = tw + OFF + j % NS;
#pragma unroll
        for (int r = 1; r < R; ++r) {
            float2 w = __ldg(t + (r - 1) * NS);
            if constexpr (INV) w.y = -w.y;
            const cscalar c = cmul(cscalar{v[r].x, v[r].y}, w);
            v[r] = make_float2(c.x, c.y);
        }
    }
    dft_scalar<R, INV>(v);
}

// 1: shared-memory addresses of a butterfly as one base plus compile-time offsets where the
// padding allows it (N = 4096: rows 0.361 -> 0.348 ms, columns 0.375 -> 0.371 ms on B200)
#ifndef DNS2D_IDX
#define DNS2D_IDX 1
#endif

// Butterfly j reads x[j + r L/R].  When L/R is a multiple of G = 2^PS the padded index is
// sidx(j) + r (L/R + L/R/G): one address, the rest compile-time offsets.
template <int L, int R, int PS = 5>
__device__ __forceinline__ void sm_load(float2 (&v)[R], const float2 *__restrict__ x, int j)
{
    constexpr int LR = L / R, G = 1 << PS;
    if constexpr (DNS2D_IDX && LR % G == 0) {
        const float2 *__restrict__ b = x + sidx<PS>(j);
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = b[r * (LR + LR / G)];
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = x[sidx<PS>(j + r * LR)];
    }
}

// Butterfly j writes y[A + k + q Ns], A = (j / Ns) Ns R, k = j % Ns.  Compile-time offsets from
// one address when the G-element padding groups (G = 2^PS) allow it:
//   Ns % G == 0:                  sidx(A + k) + q (Ns + Ns/G)
//   G % Ns == 0, (Ns R) % G == 0: A + A/G + k + q Ns + (q Ns)/G   (k + q Ns never crosses a group)
//   Ns == 1, G % R == 0:          sidx(A) + q                     (A .. A+R-1 in one group)
template <int L, int R, int NS, int PS = 5>
__device__ __forceinline__ void sm_store(float2 *__restrict__ y, const float2 (&v)[R], int j)
{
    constexpr int G = 1 << PS;
    const int k = j % NS;
    const int A = (j / NS) * NS * R;
    if constexpr (DNS2D_IDX && NS % G == 0) {
        float2 *__restrict__ b = y + sidx<PS>(A + k);
#pragma unroll
        for (int q = 0; q < R; ++q) b[q * (NS + NS / G)] = v[q];
    } else if constexpr (DNS2D_IDX && G % NS == 0 && (NS * R) % G == 0) {
        float2 *__restrict__ b = y + A + (A >> PS) + k;
#pragma unroll
        for (int q = 0; q < R; ++q) b[q * NS + ((q * NS) >> PS)] = v[q];
    } else if constexpr (DNS2D_IDX && NS == 1 && G % R == 0) {
        float2 *__restrict__ b = y + sidx<PS>(A);
#pragma unroll
        for (int q = 0; q < R; ++q) b[q] = v[q];
    } else {
        const int base = A + k;
#pragma unroll
        for (int q = 0; q < R; ++q) y[sidx<PS>(base + q * NS)] = v[q];
    }
}

// Bands known at compile time.  A first stage (Ns = 1) reads positions j + r L/R, a last stage
// (Ns = L/R) writes positions j + q L/R, j < L/R: slot r (q) covers [r L/R, r L/R + L/R - 1].
// When that whole range lies in [B0, B1] (the 3/2 padding band of a spectrum), the input is zero
// for every j, or the output is never read: loads become constants and stores are dropped, and
// the compiler removes the arithmetic that only fed them.
template <int L, int R, int B0, int B1>
__device__ __forceinline__ constexpr bool slot_in_band(int r)
{
    return r * (L / R) >= B0 && r * (L / R) + L / R - 1 <= B1;
}

// smem -> smem stage, one butterfly per thread (threads >= L/R idle); in place, so reads and
// writes are separated by a barrier.  Leading barrier included; no trailing barrier.
template <class Cat, int L, int R, int NS, bool INV, int PS = 5>
__device__ __forceinline__ void stage1(float2 *s, const float2 *tw)
{
    constexpr int LR = L / R;
    const int j = threadIdx.x;
    float2 v[R];
    __syncthreads();
    if (j < LR) {
        sm_load<L, R, PS>(v, s, j);
        bfly<Cat, L, R, NS, INV>(v, j, tw);
    }
    __syncthreads();
    if (j < LR) sm_store<L, R, NS, PS>(s, v, j);
}

// asynchronous global -> shared copies (cp.async; 16-byte elements, not kept in L1)
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(PENDING) : "memory");
}
// the first i + 1 of ND commit groups have landed
template <int ND>
__device__ __forceinline__ void cp_async_wait_first(int i)
{
    static_for<0, ND>([&](auto k) {
        if (i == decltype(k)::value) cp_async_wait<ND - 1 - decltype(k)::value>();
    });
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <class V, class Cat, int L, int LP, bool INV, int B, int NT, int PS, bool OPQ, int NS, int R0, int... Rs>
__device__ __forceinline__ void fft_stages(float2 *s, const float2 *tw)
{
    fft_stage<Cat, L, LP, R0, NS, INV, B, NT, PS, OPQ, V>(s, tw);
    if constexpr (sizeof...(Rs) > 0) fft_stages<V, Cat, L, LP, INV, B, NT, PS, OPQ, NS * R0, Rs...>(s, tw);
}

// PS: the padding of sidx<PS>; OPQ: read the thread index with opaque_tid(); V: the type a complex value is computed in
template <class Cat, int L, int LP, bool INV, int B, int NT, int PS = 5, bool OPQ = false, class V = float2, int... Rs>
__device__ __forceinline__ void fft_run(float2 *s, const float2 *tw, Radices<Rs...>)
{
    static_assert((1 * ... * Rs) == L, "radix plan does not multiply to L");
    fft_stages<V, Cat, L, LP, INV, B, NT, PS, OPQ, 1, Rs...>(s, tw);
}

}  // namespace dns2d
