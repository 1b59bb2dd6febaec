// inplace.cuh — the step's row and column passes on in-place transforms (the sizes with CfgI).
//
// A CTA holds two sequences of length L = R1 R2 R3 side by side: two physical rows (row pass), or
// the D and E (then U and W) columns of one kx (column pass).  An element is 16 bytes in shared
// memory, (re, re', im, im'), so one 128-bit access moves both sequences' values and every butterfly
// operation is one packed instruction on both (cpair, fft.cuh).
//
// Every stage is in place: a butterfly writes its outputs to the positions its inputs came from,
// so nothing is held in registers across a barrier and one barrier separates two stages (the
// auto-sort stages of fft.cuh need two, and the registers of all threads in between).  The first
// transform of a pass runs natural -> digit-reversed order (radix R1 over the L/R1-strided digit, then
// R2, then R3 over R3 contiguous elements), the second one digit-reversed -> natural (R3, R2, R1), and what lies between the two (the
// products of the row pass, the spectral update of the column pass) works in any order.  So no
// reordering pass exists, and the R3 stages of both transforms with everything between them run in
// registers: a pass touches shared memory 4 times in each direction.
//   position p = i1 B1 + i2 R3 + i3 (B1 = R2 R3) holds
//     row pass:     kx = p before, x = i1 + R1 (i2 + R2 i3) between, kx = p after
//     column pass:  z = p before, kz = i1 + R1 (i2 + R2 i3) between, z = p after
// In the row pass, between the two outer stages a warp works on its own blocks of B1 elements only
// (no CTA barrier: two per pass in all).  Bank conflicts: i3 is stored as i3 ^ ((i1 ^ i2) & 7), so
// eight neighbouring lanes find eight different 16-byte columns in every stage, along i3, i2 or i1.
//
// Rounding: both transforms compute node by node what auto-sort plans do (decimation in time: twiddles
// before a butterfly), and the packed operations round where the scalar expressions of those plans round
// (fft.cuh), so that with the plans (16, 12, 16) and (16, 24, 16), the same in both directions, N = 2048
// and 4096 have the auto-sort kernels' results bit for bit: the default configuration of a size keeps its
// rounding from build to build (dns2d.h), so that runs and restarts can be compared across builds mode by
// mode.  FP32 rounding of the products, times k^2, is 1e-3 of the field's RMS in single modes of the corners.
// Measured with other rounding and not kept for that reason alone: a first transform by decimation in
// frequency (twiddles after a butterfly, fetched once; N = 4096 386 us per step where decimation in time
// took 392 in the same build, 2048 89.7 / 98), N = 8192 / 9216 on three-stage in-place passes (1.75 / 2.55 ms,
// 3.44 / 4.70 on the clusters), N = 512 and 256 (15.3 and 10.6 us; 20.1 and 11.9 now) and the 64-member ensemble
// (77 us per step; 119 now).  Auto-sort stages within one CTA could keep the rounding there; not built.
//
// Bounds (N = 4096 on B200, 1965 MHz; ncu): the row pass is bound by the L1 / shared-memory data
// pipe (66 % of its cycles busy), the column pass by the latency of its phases at two CTAs per SM (HBM
// 38 %, issue 35 %).  Measured (rows / columns, one launch): N = 4096 0.254 / 0.293 -> 0.194 / 0.200 ms,
// N = 2048 67.6 / 71.7 -> 52.1 / 54.7 us,
// N = 1024 27.0 / 28.2 -> 20.3 / 23.2 us against the auto-sort kernels that these replace (one row,
// or one array and thread group, per 384 threads).
// Tried and slower, or no faster: each sequence on its own lane with scalar butterflies (rows 0.185,
// columns 0.223 ms at N = 4096), fetching the next round's twiddles, state or rows into registers in the
// column pass (0.220-0.239 ms), prefetching a later CTA's input to L2 (columns +4 us), twice the threads at
// half the registers (rows 0.200 ms), 2-row tiles of the work buffer (columns 0.259 ms).
#pragma once
#include "dns2d_kernels.cuh"

namespace dns2d {

// shared-memory element <-> the two complex values of a butterfly input
__device__ __forceinline__ cpair ip_get(const float4 *s, int i)
{
    const float4 x = s[i];
    return {make_float2(x.x, x.y), make_float2(x.z, x.w)};
}
__device__ __forceinline__ void ip_put(float4 *s, int i, cpair v)
{
    s[i] = make_float4(v.re.x, v.re.y, v.im.x, v.im.y);
}
// element r of a butterfly whose element 0 has the (swizzled) index b; the elements are STRIDE apart
template <int R, int STRIDE>
__device__ __forceinline__ void ip_load(cpair (&v)[R], const float4 *s, int b)
{
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ip_get(s, (b ^ (r & 7)) + r * STRIDE);
}
template <int R, int STRIDE>
__device__ __forceinline__ void ip_store(float4 *s, const cpair (&v)[R], int b)
{
#pragma unroll
    for (int r = 0; r < R; ++r) ip_put(s, (b ^ (r & 7)) + r * STRIDE, v[r]);
}
// the same for the R contiguous elements of a group
template <int R>
__device__ __forceinline__ void ip_load_run(cpair (&v)[R], const float4 *s, int b)
{
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ip_get(s, (b ^ (r & 7)) + (r & ~7));
}
template <int R>
__device__ __forceinline__ void ip_store_run(float4 *s, const cpair (&v)[R], int b)
{
#pragma unroll
    for (int r = 0; r < R; ++r) ip_put(s, (b ^ (r & 7)) + (r & ~7), v[r]);
}

// w[r] = W^{r k}, r >= 1: the twiddles of the stage (R, NS) at index k of the table's order
template <class Cat, int R, int NS, int OUTER = 0>
__device__ __forceinline__ void ip_tw_load(float2 (&w)[R], const float2 *__restrict__ tw, int k)
{
    constexpr int OFF = Cat::off(R, NS, OUTER);
    static_assert(OFF >= 0, "stage missing from the twiddle catalog");
    const float2 *t = tw + OFF + k;
#pragma unroll
    for (int r = 1; r < R; ++r)
        asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(w[r].x), "=f"(w[r].y) : "l"(t + (r - 1) * NS));
}
// v[r] *= w[r] (conjugate when INV)
template <int R, bool INV>
__device__ __forceinline__ void ip_twiddle(cpair (&v)[R], const float2 (&w)[R])
{
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = ctwiddle<INV>(v[r], w[r]);
}

// the two components of one mode on two neighbouring rows: 32 contiguous bytes of the work buffer
struct row2 {
    float4 a, b;
};
__device__ __forceinline__ row2 ld_row2(const float2 *p)
{
    row2 v;
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v.a.x), "=f"(v.a.y), "=f"(v.a.z), "=f"(v.a.w), "=f"(v.b.x), "=f"(v.b.y), "=f"(v.b.z), "=f"(v.b.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ void st_row2(float2 *p, const row2 &v)
{
    asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(v.a.x), "f"(v.a.y), "f"(v.a.z),
                 "f"(v.a.w), "f"(v.b.x), "f"(v.b.y), "f"(v.b.z), "f"(v.b.w), "l"(p)
                 : "memory");
}
__device__ __forceinline__ cpair shfl_xor16(cpair m)
{
    cpair h;
    h.re.x = __shfl_xor_sync(0xffffffffu, m.re.x, 16);
    h.re.y = __shfl_xor_sync(0xffffffffu, m.re.y, 16);
    h.im.x = __shfl_xor_sync(0xffffffffu, m.im.x, 16);
    h.im.y = __shfl_xor_sync(0xffffffffu, m.im.y, 16);
    return h;
}

// ------------------------------------------------------------------------------------------
// Row pass by NT threads (tid < NT): rows 2 pair and + 1: U, W -> C2R -> (u + iw)^2 -> R2C -> D, E.
// The Hermitian packing needs modes k and L - k together: k = j + r B1 is slot r of butterfly j, and
// L - k is slot R1 - 1 - r of butterfly B1 - j, so butterflies j and B1 - j run 16 lanes apart in one
// warp and exchange those slots by shuffle, on the way in and on the way out (butterflies 0 and
// B1 / 2 are their own mirrors).
// ------------------------------------------------------------------------------------------
template <int N, int NT>
__device__ __forceinline__ void rows_ip(const Pointers &p, int pair, float4 *s4, int tid)
{
    using C = CfgI<N>;
    using P = typename C::RowPlan;
    using Cat = TwCat<N>;
    constexpr int L = C::L, H = C::H, R1 = P::R1, R2 = P::R2, R3 = P::R3, B1 = P::B1;
    constexpr int NW = NT / 32, BPW = R1 / NW;  // blocks of B1 elements per warp
    static_assert(R1 % NW == 0 && B1 % 32 == 0, "whole blocks per warp");
    constexpr int NLO = (H + B1 - 1) / B1;  // slots with retained modes below H
    const int lane = tid & 31, warp = tid >> 5;
    float2 *row = p.work + widx<L, H>(0, 2 * pair, 0);
    auto jof = [](int t) {  // butterfly of index t
        const int l = t & 31, q = (t >> 5) * 16 + (l & 15);
        return (l < 16) ? q : (q == 0 ? B1 / 2 : B1 - q);
    };
    // a round's twiddles on their way before the round, where a thread has the registers (N = 4096: rows
    // 198 -> 193 us; 2048 and 1024, at 128 registers, 52.5 -> 53.7 and 20.6 -> 20.8)
    constexpr bool AHEAD = 65536 / (C::MBR * C::NTR) >= 255;
    float2 w1[R1], w2[R2], w3[R3];
    auto first_w2 = [&] { ip_tw_load<Cat, R2, R1>(w2, p.tw, warp * BPW + (lane < BPW * R3 ? lane / R3 : 0)); };
    auto first_w3 = [&] { ip_tw_load<Cat, R3, R1 * R2, R1>(w3, p.tw, warp * BPW * R2 + (lane < BPW * R2 ? lane : 0)); };
#pragma unroll 1
    for (int t = tid; t < B1; t += NT) {
        const int j = jof(t);
        cpair v[R1], m[NLO + 1];
        czero(m[NLO]);
#pragma unroll
        for (int r = 0; r < R1; ++r) czero(v[r]);
#pragma unroll
        for (int r = 0; r < NLO; ++r) {
            const int k = j + r * B1;
            czero(m[r]);
            if ((r + 1) * B1 <= H || k < H) {
                const row2 x = ld_row2(row + (size_t)k * widx_kx_stride);
                if (r == 0 && k == 0) {
                    v[r] = {make_float2(x.a.x, x.b.x), make_float2(x.a.z, x.b.z)};
                } else {
                    v[r] = {make_float2(x.a.x - x.a.w, x.b.x - x.b.w), make_float2(x.a.y + x.a.z, x.b.y + x.b.z)};
                }
                m[r] = {make_float2(x.a.x + x.a.w, x.b.x + x.b.w), make_float2(x.a.z - x.a.y, x.b.z - x.b.y)};
            }
        }
#pragma unroll
        for (int r = R1 - NLO; r < R1; ++r) {
            cpair h = shfl_xor16(m[R1 - 1 - r]);
            if (j == 0) h = m[R1 - r];
            else if (j == B1 / 2) h = m[R1 - 1 - r];
            v[r] = h;
        }
        DFT<R1, true>::run(v);
        ip_store<R1, B1>(s4, v, j ^ ((j / R3) & 7));
    }
    if constexpr (AHEAD) first_w2();
    __syncthreads();
#pragma unroll 1
    for (int t = lane; t < BPW * R3; t += 32) {
        const int i3 = t % R3, i1 = warp * BPW + t / R3;
        const int b = i1 * B1 + (i3 ^ (i1 & 7));
        cpair v[R2];
        if (!AHEAD) ip_tw_load<Cat, R2, R1>(w2, p.tw, i1);
        ip_load<R2, R3>(v, s4, b);
        ip_twiddle<R2, true>(v, w2);
        if (AHEAD && t + 32 < BPW * R3) ip_tw_load<Cat, R2, R1>(w2, p.tw, warp * BPW + (t + 32) / R3);
        DFT<R2, true>::run(v);
        ip_store<R2, R3>(s4, v, b);
    }
    if constexpr (AHEAD) first_w3();
    __syncwarp();
    // last inverse stage -> products (u + iw)^2 -> first forward stage, in registers
#pragma unroll 1
    for (int t = lane; t < BPW * R2; t += 32) {
        const int i2 = t % R2, i1 = warp * BPW + t / R2;
        const int b = i1 * B1 + i2 * R3 + ((i1 ^ i2) & 7);
        cpair v[R3];
        if (!AHEAD) ip_tw_load<Cat, R3, R1 * R2, R1>(w3, p.tw, i1 * R2 + i2);
        ip_load_run<R3>(v, s4, b);
        ip_twiddle<R3, true>(v, w3);
        if (AHEAD && t + 32 < BPW * R2) ip_tw_load<Cat, R3, R1 * R2, R1>(w3, p.tw, warp * BPW * R2 + t + 32);
        DFT<R3, true>::run(v);
        csquare sq[R3];
#pragma unroll
        for (int q = 0; q < R3; ++q) sq[q] = square(v[q]);
        DFT<R3, false>::run(sq, v);
        ip_store_run<R3>(s4, v, b);
    }
    static_assert(32 % R3 == 0, "a thread's index within a block's R3 is the same in every round");
    ip_tw_load<Cat, R2, R3>(w2, p.tw, lane % R3);
    __syncwarp();
#pragma unroll 1
    for (int t = lane; t < BPW * R3; t += 32) {
        const int i3 = t % R3, i1 = warp * BPW + t / R3;
        const int b = i1 * B1 + (i3 ^ (i1 & 7));
        cpair v[R2];
        ip_load<R2, R3>(v, s4, b);
        ip_twiddle<R2, false>(v, w2);
        DFT<R2, false>::run(v);
        ip_store<R2, R3>(s4, v, b);
    }
    ip_tw_load<Cat, R1, B1>(w1, p.tw, jof(tid < B1 ? tid : 0));
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < B1; t += NT) {
        const int j = jof(t);
        cpair v[R1];
        ip_load<R1, B1>(v, s4, j ^ ((j / R3) & 7));
        ip_twiddle<R1, false>(v, w1);
        if (t + NT < B1) ip_tw_load<Cat, R1, B1>(w1, p.tw, jof(t + NT));
        DFT<R1, false>::run(v);
        // mode k = j + r B1 < H and its mirror L - k: slot R1 - 1 - r of butterfly B1 - j
#pragma unroll
        for (int r = 0; r < NLO; ++r) {
            const int k = j + r * B1;
            cpair m = shfl_xor16(v[R1 - 1 - r]);
            if (j == 0) m = v[r == 0 ? 0 : R1 - r];
            else if (j == B1 / 2) m = v[R1 - 1 - r];
            if ((r + 1) * B1 <= H || k < H) {
                row2 o;
                o.a = make_float4(0.5f * (v[r].re.x + m.re.x), 0.5f * (v[r].im.x - m.im.x),
                                  0.25f * (v[r].im.x + m.im.x), -0.25f * (v[r].re.x - m.re.x));
                o.b = make_float4(0.5f * (v[r].re.y + m.re.y), 0.5f * (v[r].im.y - m.im.y),
                                  0.25f * (v[r].im.y + m.im.y), -0.25f * (v[r].re.y - m.re.y));
                st_row2(row + (size_t)k * widx_kx_stride, o);
            }
        }
    }
}

template <int N>
__global__ void __launch_bounds__(CfgI<N>::NTR, CfgI<N>::MBR) k_rows_ip(Pointers p0)
{
    const Pointers p = p0.member(blockIdx.y);
    using C = CfgI<N>;
    extern __shared__ __align__(16) float4 s4[];
    rows_ip<N, C::NTR>(p, blockIdx.x, s4, threadIdx.x);
}

// The factors of cn_update and recover_velocity for one mode, in FP64 and each rounded once to float as
// there, from one reciprocal in place of two divisions: r = 1 / (K^2 (1 + a)), 1 / (1 + a) = r K^2,
// 1 / K^2 = r (1 + a).  The reciprocal is the PTX instruction's approximation (relative error 2^-20) and two
// steps of Newton's iteration x <- x + x (1 - d x), which squares the error each time.  The column pass
// waits for the chains of these (N = 4096 on B200: columns 211 -> 201 us; 2048 58.6 -> 54.7).
struct ModeFactors {
    float d1, c2, c3, gu, gw;
    double invK2;  // 0 at K = 0
};
__device__ __forceinline__ ModeFactors mode_factors(int kx, int kz, double hvdt, double c2n, double c3n)
{
    const int k2 = kx * kx + kz * kz;
    const double K2 = (double)k2, a = hvdt * K2, q = 1.0 + a, s = k2 ? K2 : 1.0, d = s * q;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.0), r);
    r = fma(r, fma(-d, r, 1.0), r);
    const double inv = r * s, invK2 = k2 ? r * q : 0.0;
    ModeFactors f;
    f.d1 = (float)(-2.0 * a * inv);
    f.c2 = (float)(c2n * inv);
    f.c3 = (float)(c3n * inv);
    f.gu = (float)((double)kz * invK2);
    f.gw = (float)((double)kx * invK2);
    f.invK2 = invK2;
    return f;
}

// ------------------------------------------------------------------------------------------
// Column pass: column kx: D, E -> z-forward -> FN, Crank-Nicolson / AB2, FNM1 <- FN, velocity
// recovery -> z-inverse -> U, W.  The column arrives by cp.async in natural order; a thread waits
// only for its own copies (it copies what its first butterflies read).  In the R3 stage the threads
// run along kz, so om2 and fnm1 are read and written coalesced; the 3/2 band's slots are zeros known
// at compile time where they lie wholly in it.
// ------------------------------------------------------------------------------------------
// First half, by NT threads: up to the first stage of the inverse; returns this thread's (E, Z) sums.
// The threads must pass a barrier before cols_ip_inverse.
template <int N, int NT>
__device__ __forceinline__ double2 cols_ip_forward(const Pointers &p, int kx, int first, float4 *s4, int tid)
{
    using C = CfgI<N>;
    using P = typename C::ColPlan;
    using Cat = TwCat<N>;
    constexpr int L = C::L, H = C::H, R1 = P::R1, R2 = P::R2, R3 = P::R3, B1 = P::B1;
    constexpr int S3 = R1 * R2, NLO = (H + S3 - 1) / S3, HI0 = (L - H) / S3;
    static_assert(HI0 + NLO == R3 && NLO <= HI0, "retained slots");
    static_assert(B1 % 32 == 0, "whole warps in the first and last stage");
    float2 *om2c = p.om2 + (size_t)kx * N;
    float2 *fnc = p.fnm1 + (size_t)kx * N;
    static_assert(B1 % widx_rows == 0, "stride");
    constexpr size_t ZS = (size_t)(B1 / widx_rows) * H * widx_kx_stride;  // float2 between z and z + B1
    constexpr int ND1 = (B1 + NT - 1) / NT;
#pragma unroll
    for (int i = 0; i < ND1; ++i) {
        const int j = tid + i * NT;
        if (B1 % NT == 0 || j < B1) {
            const float2 *ptr = p.work + widx<L, H>(0, j, kx);
#pragma unroll
            for (int r = 0; r < R1; ++r) cp_async16(s4 + j + r * B1, ptr + r * ZS);
        }
        cp_async_commit();
    }
    for (int o = tid * 16; o < N; o += NT * 16) {
        prefetch_l2(om2c + o);
        prefetch_l2(fnc + o);
    }
    float2 w2[R2], w3[R3];
#pragma unroll 1
    for (int i = 0; i < ND1; ++i) {
        const int j = tid + i * NT;
        if (B1 % NT != 0 && j >= B1) break;
        cpair v[R1];
        cp_async_wait_first<ND1>(i);
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            const float4 x = s4[j + r * B1];
            v[r] = {make_float2(x.x, x.z), make_float2(x.y, x.w)};
        }
        DFT<R1, false>::run(v);
        __syncwarp();  // the swizzled positions are other lanes' inputs
        ip_store<R1, B1>(s4, v, j ^ ((j / R3) & 7));
    }
    __syncthreads();
#pragma unroll 1
    for (int t = tid; t < R1 * R3; t += NT) {
        const int i3 = t % R3, i1 = t / R3;
        const int b = i1 * B1 + (i3 ^ (i1 & 7));
        cpair v[R2];
        ip_tw_load<Cat, R2, R1>(w2, p.tw, i1);
        ip_load<R2, R3>(v, s4, b);
        ip_twiddle<R2, false>(v, w2);
        DFT<R2, false>::run(v);
        ip_store<R2, R3>(s4, v, b);
    }
    const StepParams prm = *p.prm;
    const float dt = prm.dt;
    const float cnm1 = first ? prm.cnm1_first : prm.cn;
    const double hvdt = 0.5 * (double)prm.visc * (double)dt;
    const double c2n = 0.5 * (double)dt * (2.0 + (double)cnm1);
    const double c3n = -0.5 * (double)dt * (double)cnm1;
    const float divxz = (float)(1.0 / ((double)L * (double)L));
    double2 ez = make_double2(0.0, 0.0);
    __syncthreads();
#pragma unroll 1
    for (int j = tid; j < S3; j += NT) {
        const int i1 = j % R1, i2 = j / R1;
        const int b = i1 * B1 + i2 * R3 + ((i1 ^ i2) & 7);
        float2 om[2 * NLO], fo[2 * NLO];
#pragma unroll
        for (int q = 0; q < 2 * NLO; ++q) {
            const int kzi = j + S3 * (q < NLO ? q : HI0 - NLO + q);
            const int iz = q < NLO ? kzi : kzi - (L - N);
            om[q] = fo[q] = make_float2(0.f, 0.f);
            if (q < NLO ? kzi < H : kzi >= L - H) {
                om[q] = om2c[iz];
                fo[q] = fnc[iz];
            }
        }
        cpair v[R3];
        ip_tw_load<Cat, R3, R1 * R2>(w3, p.tw, j);
        ip_load_run<R3>(v, s4, b);
        ip_twiddle<R3, false>(v, w3);
        DFT<R3, false>::run(v);
#pragma unroll
        for (int q = NLO; q < HI0; ++q) czero(v[q]);
#pragma unroll
        for (int q = 0; q < 2 * NLO; ++q) {
            const int slot = q < NLO ? q : HI0 - NLO + q;
            const int kzi = j + S3 * slot;
            const int kz = q < NLO ? kzi : kzi - L, iz = q < NLO ? kzi : kzi - (L - N);
            cpair uw;
            czero(uw);
            if (q < NLO ? kzi < H : kzi >= L - H) {
                const float2 d = make_float2(v[slot].re.x, v[slot].im.x), e = make_float2(v[slot].re.y, v[slot].im.y);
                float2 fn = make_float2(0.f, 0.f);
                if (kz != -H) {
                    const float ga = (float)kz * (float)kx;
                    const float g2a2 = (float)kz * (float)kz - (float)kx * (float)kx;
                    fn.x = (ga * d.x + g2a2 * e.x) * divxz;
                    fn.y = (ga * d.y + g2a2 * e.y) * divxz;
                    if (p.force) fn = add_forcing(fn, p, kx, iz, N);
                }
                const ModeFactors f = mode_factors(kx, kz, hvdt, c2n, c3n);
                const float2 on = make_float2(om[q].x + fmaf(f.d1, om[q].x, fmaf(f.c2, fn.x, f.c3 * fo[q].x)),
                                              om[q].y + fmaf(f.d1, om[q].y, fmaf(f.c2, fn.y, f.c3 * fo[q].y)));
                om2c[iz] = on;
                fnc[iz] = fn;
                // u = -i gu om, w = i gw om
                uw = {make_float2(f.gu * on.y, -f.gw * on.y), make_float2(-f.gu * on.x, f.gw * on.x)};
                const double pw = (double)on.x * on.x + (double)on.y * on.y;
                ez.x = fma(pw, f.invK2, ez.x);
                ez.y += pw;
            }
            v[slot] = uw;
        }
        DFT<R3, true>::run(v);
        ip_store_run<R3>(s4, v, b);
    }
    const double wgt = (kx == 0) ? 0.5 : 1.0;  // 1/2 * (1 on kx = 0, else 2)
    return make_double2(ez.x * wgt, ez.y * wgt);
}

// Second half: the inverse transform's other stages and the U, W column.
template <int N, int NT>
__device__ __forceinline__ void cols_ip_inverse(const Pointers &p, int kx, float4 *s4, int tid)
{
    using C = CfgI<N>;
    using P = typename C::ColPlan;
    using Cat = TwCat<N>;
    constexpr int L = C::L, H = C::H, R1 = P::R1, R2 = P::R2, R3 = P::R3, B1 = P::B1;
    constexpr size_t ZS = (size_t)(B1 / widx_rows) * H * widx_kx_stride;
    float2 w1[R1], w2[R2];
    ip_tw_load<Cat, R2, R3>(w2, p.tw, tid % R3);
#pragma unroll 1
    for (int t = tid; t < R1 * R3; t += NT) {
        const int i3 = t % R3, i1 = t / R3;
        const int b = i1 * B1 + (i3 ^ (i1 & 7));
        cpair v[R2];
        ip_load<R2, R3>(v, s4, b);
        ip_twiddle<R2, true>(v, w2);
        DFT<R2, true>::run(v);
        ip_store<R2, R3>(s4, v, b);
    }
    ip_tw_load<Cat, R1, B1>(w1, p.tw, tid < B1 ? tid : 0);
    __syncthreads();
#pragma unroll 1
    for (int j = tid; j < B1; j += NT) {
        cpair v[R1];
        ip_load<R1, B1>(v, s4, j ^ ((j / R3) & 7));
        ip_twiddle<R1, true>(v, w1);
        if (j + NT < B1) ip_tw_load<Cat, R1, B1>(w1, p.tw, j + NT);
        DFT<R1, true>::run(v);
        float4 *ptr = reinterpret_cast<float4 *>(p.work + widx<L, H>(0, j, kx));
#pragma unroll
        for (int r = 0; r < R1; ++r) ptr[r * (ZS / 2)] = make_float4(v[r].re.x, v[r].im.x, v[r].re.y, v[r].im.y);
    }
}

template <int N>
__global__ void __launch_bounds__(CfgI<N>::NTC, CfgI<N>::MBC) k_cols_ip(Pointers p0, int first, int hist_slot)
{
    const Pointers p = p0.member(blockIdx.y);
    using C = CfgI<N>;
    constexpr int H = C::H, NT = C::NTC;
    extern __shared__ __align__(16) float4 s4[];
    __shared__ double2 red[NT / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kx = blockIdx.x;
    double2 ez = cols_ip_forward<N, NT>(p, kx, first, s4, tid);
    for (int o = 16; o > 0; o >>= 1) {
        ez.x += __shfl_xor_sync(0xffffffffu, ez.x, o);
        ez.y += __shfl_xor_sync(0xffffffffu, ez.y, o);
    }
    if (lane == 0) red[warp] = ez;
    __syncthreads();
    // energy / enstrophy: per-column partials, the last column's first warp sums them (deterministic)
    if (warp == 0) {
        ez = lane < NT / 32 ? red[lane] : make_double2(0.0, 0.0);
        for (int o = 16; o > 0; o >>= 1) {
            ez.x += __shfl_xor_sync(0xffffffffu, ez.x, o);
            ez.y += __shfl_xor_sync(0xffffffffu, ez.y, o);
        }
        unsigned int n = 0;
        if (lane == 0) {
            p.part[kx] = ez;
            __threadfence();
            n = atomicAdd(p.counter, 1u);
        }
        n = __shfl_sync(0xffffffffu, n, 0);
        if (n == gridDim.x - 1) {
            __threadfence();
            double2 acc = make_double2(0.0, 0.0);
            for (int i = lane; i < H; i += 32) {
                const double2 q = __ldcg(&p.part[i]);
                acc.x += q.x;
                acc.y += q.y;
            }
            for (int o = 16; o > 0; o >>= 1) {
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
                acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            }
            if (lane == 0) {
                p.hist[hist_slot] = acc;
                *p.counter = 0u;
            }
        }
    }
    cols_ip_inverse<N, NT>(p, kx, s4, tid);
}

}  // namespace dns2d
