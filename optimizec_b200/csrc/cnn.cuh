// cnn.cuh — periodic 3x3 convolutional network of the learned subgrid closure.
//
// Network: L layers of 3x3 convolutions with periodic padding; layer 0 maps the 3 input
// channels (filtered vorticity, u, w) to C channels, layers 1..L-2 map C -> C, the last maps
// C -> 1 (the subgrid forcing); GELU(x) = x Phi(x) after every layer but the last.
// Activations are [B][C][H][W] float; weights [Co][Ci][3][3] then bias [Co], layer after
// layer, in one flat parameter vector.  Forward, backward (data and weight gradients) and Adam
// are hand-written kernels; all reductions are in fixed order (deterministic).
#pragma once
#include "cnn_math.cuh"

#include <type_traits>

namespace dns2d {
namespace cnn {

// ------------------------------------------------------------------------------------------
// One convolution in FP32, forward or data gradient:
//   y[b][co][p] = sum_{ci, tap} w(ci, co, tap) x[b][ci][p + tap - 1]  (periodic)
//   forward: z = y + bias and, when a is set, a = GELU(z); data gradient: y * GELU'(zprev)
// w: the layer's weights packed [ci][tap][NP] by k_pack_fp32, co contiguous (read straight from
// [co][ci][tap], each lane of a copy touched another line: 62 -> 49 us).
// A CTA computes 8 COG output channels of a tile 16 pixels wide and kConvRows<COG> rows high; a thread 4
// neighbouring pixels x 8 channels, its sums packed in pairs of channels (one packed FMA per pixel,
// tap and pair): per input channel and kernel row 2 + 6 loads from shared memory feed 48 packed FMAs, so
// the FMA pipe is the bound (one pixel x 8 channels per thread took a load for every FMA).  Measured on
// B200 at 48^2, batch 32, 32 -> 32 channels: 49 us = 28 TFLOP/s of FP32's 74 (0.26 ms
// before, with the GELU in a kernel of its own); 3.9 CTAs per SM leave its copies partly exposed.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ void cp_async4(float *smem_dst, const float *gmem_src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async16f(float *smem_dst, const float *gmem_src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_all()
{
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

constexpr int kConvThreads = 128, kConvCols = 16, kConvCi = 16, kConvPitch = 20;
template <int COG>
constexpr int kConvRows = kConvThreads / COG / 4;
template <int COG>
constexpr int kConvStage = kConvCi * (kConvRows<COG> + 2) * kConvPitch + kConvCi * 9 * 8 * COG;  // floats
template <int COG>
constexpr size_t conv_smem()
{
    return (size_t)kConvStage<COG> * sizeof(float);
}

// output channels of a packed row: a whole number of the convolution's channel tiles
__host__ __device__ constexpr int packed_channels(int Co) { return Co <= 8 ? 8 : (Co + 31) / 32 * 32; }
// packed weights of up to kPackLayers layers: forward w[co][ci][tap] -> [ci][tap][co], data gradient
// w[co][ci][8 - tap] -> [co][tap][ci], channels beyond the layer's zero
constexpr int kPackLayers = 32;
struct PackFp32 {
    int ci[kPackLayers], co[kPackLayers];
    unsigned int woff[kPackLayers], fwd[kPackLayers], bwd[kPackLayers];
};
__global__ void k_pack_fp32(const float *__restrict__ params, const __grid_constant__ PackFp32 a, float *__restrict__ out)
{
    const int l = blockIdx.y >> 1, flip = blockIdx.y & 1;
    const int Ci = a.ci[l], Co = a.co[l], K = flip ? Co : Ci, N = flip ? Ci : Co, NP = packed_channels(N);
    const float *w = params + a.woff[l];
    float *o = out + (flip ? a.bwd[l] : a.fwd[l]);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < K * 9 * NP; e += gridDim.x * blockDim.x) {
        const int r = e / NP, n = e - r * NP, k = r / 9, tap = r - k * 9;
        o[e] = n >= N ? 0.0f : (flip ? w[((size_t)k * Ci + n) * 9 + 8 - tap] : w[((size_t)n * Ci + k) * 9 + tap]);
    }
}

template <int COG>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3(const float *__restrict__ x, const float *__restrict__ w,
                                                          const float *__restrict__ bias, const float *__restrict__ zprev,
                                                          float *__restrict__ y, float *__restrict__ a, int Ci, int Co,
                                                          int H, int W, int NP)
{
    constexpr int TR = kConvRows<COG>, NCO = 8 * COG;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, cg = tid / (kConvThreads / COG), pg = tid % (kConvThreads / COG);
    const int tiles_x = (W + kConvCols - 1) / kConvCols;
    const int x0 = (blockIdx.x % tiles_x) * kConvCols, y0 = (blockIdx.x / tiles_x) * TR;
    const int co0 = blockIdx.y * NCO, b = blockIdx.z;
    const int px = (pg & 3) * 4, py = pg >> 2, oy = y0 + py, ox = x0 + px;
    const float *xb = x + (size_t)b * Ci * H * W;
    float2 acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[p][j] = make_float2(0.f, 0.f);
    float *tin = sm, *tw = sm + kConvCi * (TR + 2) * kConvPitch;  // [ci][TR + 2][pitch], [ci][tap][NCO]
    // the tile's rows of nc channels; a last tile that reaches beyond the image takes the image's rows only
    // (16 rows, 8 channels, one CTA: 14.7 -> 13.0 us)
    auto load_rows = [&](int c0, int nc, auto whole) {
        const int per = (decltype(whole)::value ? TR + 2 : H - y0 + 2) * (kConvCols + 2);
        for (int e = tid; e < nc * per; e += kConvThreads) {
            const int ci = e / per, r = e - ci * per;
            const int ry = r / (kConvCols + 2), rx = r - ry * (kConvCols + 2);
            int yy = y0 + ry - 1, xx = x0 + rx - 1;  // periodic; tiles may reach beyond the image
            if (yy < 0) yy += H;
            while (yy >= H) yy -= H;
            if (xx < 0) xx += W;
            while (xx >= W) xx -= W;
            cp_async4(tin + (ci * (TR + 2) + ry) * kConvPitch + rx, xb + ((size_t)(c0 + ci) * H + yy) * W + xx);
        }
    };
    for (int c0 = 0; c0 < Ci; c0 += kConvCi) {
        const int nc = min(kConvCi, Ci - c0);
        if (c0 > 0) __syncthreads();
        for (int e = tid; e < nc * 9 * (NCO / 4); e += kConvThreads) {
            const int r = e / (NCO / 4), q = (e % (NCO / 4)) * 4;
            cp_async16f(tw + r * NCO + q, w + (size_t)(c0 * 9 + r) * NP + co0 + q);
        }
        if (y0 + TR <= H) load_rows(c0, nc, std::true_type{});
        else load_rows(c0, nc, std::false_type{});
        cp_async_all();
        __syncthreads();
        for (int ci = 0; ci < nc && oy < H; ++ci) {
            const float *ti = tin + (ci * (TR + 2) + py) * kConvPitch + px;
            const float *wi = tw + ci * 9 * NCO + cg * 8;
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                const float4 u = *reinterpret_cast<const float4 *>(ti + ky * kConvPitch);
                const float2 u2 = *reinterpret_cast<const float2 *>(ti + ky * kConvPitch + 4);
                const float v[6] = {u.x, u.y, u.z, u.w, u2.x, u2.y};
#pragma unroll
                for (int kx = 0; kx < 3; ++kx) {
                    const float4 wa = *reinterpret_cast<const float4 *>(wi + (ky * 3 + kx) * NCO);
                    const float4 wb = *reinterpret_cast<const float4 *>(wi + (ky * 3 + kx) * NCO + 4);
                    const float2 wp[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y),
                                          make_float2(wb.z, wb.w)};
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float2 vv = make_float2(v[p + kx], v[p + kx]);
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc[p][j] = __ffma2_rn(vv, wp[j], acc[p][j]);
                    }
                }
            }
        }
    }
    if (oy >= H || ox >= W) return;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int co = co0 + cg * 8 + j;
        if (co >= Co) break;
        const size_t o = (((size_t)b * Co + co) * H + oy) * W + ox;
        const float bi = bias ? __ldg(bias + co) : 0.0f;
        float v[4];
#pragma unroll
        for (int p = 0; p < 4; ++p) v[p] = ((j & 1) ? acc[p][j >> 1].y : acc[p][j >> 1].x) + bi;
        if (zprev) {
#pragma unroll
            for (int p = 0; p < 4; ++p)
                if (ox + p < W) v[p] *= gelu_grad(__ldg(zprev + o + p));
        }
        if ((W & 3) == 0) {
            *reinterpret_cast<float4 *>(y + o) = make_float4(v[0], v[1], v[2], v[3]);
            if (a) *reinterpret_cast<float4 *>(a + o) = make_float4(gelu(v[0]), gelu(v[1]), gelu(v[2]), gelu(v[3]));
        } else {
#pragma unroll
            for (int p = 0; p < 4; ++p)
                if (ox + p < W) {
                    y[o + p] = v[p];
                    if (a) a[o + p] = gelu(v[p]);
                }
        }
    }
}

// One output channel (the network's last layer), forward: a thread per pixel straight from global memory
// (L1 serves the taps), the weights from shared memory.  With a single channel the tile of 8 above
// spends its time on loads (48^2, batch 32: 99 -> 20 us).
__global__ void __launch_bounds__(128) k_conv3x3_one(const float *__restrict__ x, const float *__restrict__ w,
                                                     const float *__restrict__ bias, float *__restrict__ y, int Ci, int H,
                                                     int W)
{
    extern __shared__ __align__(16) float sm[];
    for (int e = threadIdx.x; e < Ci * 9; e += 128) sm[e] = w[e];
    __syncthreads();
    const int p = blockIdx.x * 128 + threadIdx.x, b = blockIdx.y;
    if (p >= H * W) return;
    const int oy = p / W, ox = p - oy * W;
    const int cx[3] = {ox == 0 ? W - 1 : ox - 1, ox, ox == W - 1 ? 0 : ox + 1};
    const int ry[3] = {(oy == 0 ? H - 1 : oy - 1) * W, oy * W, (oy == H - 1 ? 0 : oy + 1) * W};
    const float *xb = x + (size_t)b * Ci * H * W;
    float acc = 0.0f;
#pragma unroll 4
    for (int ci = 0; ci < Ci; ++ci)
#pragma unroll
        for (int k = 0; k < 9; ++k)
            acc = fmaf(sm[ci * 9 + k], __ldg(xb + (size_t)ci * H * W + ry[k / 3] + cx[k % 3]), acc);
    y[(size_t)b * H * W + p] = acc + __ldg(bias);
}

// ------------------------------------------------------------------------------------------
// Weight gradient: dw[co][ci][tap] = sum_{b, p} dy[b][co][p] x[b][ci][p + tap - 1], db[co] = sum dy.
// blockIdx.y: a tile of 32 input x 32 output channels; lane = input channel, warp = 4 output channels, 9
// taps x 4 sums per thread.  blockIdx.x takes a contiguous range of row pieces (kWgCols pixels of one
// image row; three rows of x are held, the next piece below loads one): per pixel 3 new x values and
// one 16-byte load of dy feed 18 packed FMAs (before: a load for every FMA, every pixel read by each of
// the Ci Co CTAs).  Each CTA writes its sums; k_wgrad_reduce adds them in order in FP64.
// Measured on B200 at 48^2, batch 32, 32 x 32 channels: 55 us, 20 of them its FMAs (0.45 ms before).
// ------------------------------------------------------------------------------------------
constexpr int kWgCols = 64, kWgThreads = 256, kWgXs = 33, kWgDs = 36, kWgCtas = 2;  // CTAs per SM
constexpr size_t wgrad_smem() { return ((size_t)4 * (kWgCols + 2) * kWgXs + (size_t)2 * kWgCols * kWgDs) * sizeof(float); }
constexpr int kWgPart = 9 * 32 * 32 + 32;  // sums of one CTA: [tap][ci][co], then db[co]

__global__ void __launch_bounds__(kWgThreads, kWgCtas) k_conv3x3_wgrad(const float *__restrict__ x, const float *__restrict__ dy,
                                                                 float *__restrict__ part, int B, int Ci, int Co, int H, int W)
{
    extern __shared__ __align__(16) float sm[];
    constexpr int ROW = (kWgCols + 2) * kWgXs, DS = kWgCols * kWgDs;
    float *ds = sm, *xs = sm + 2 * DS;  // dy [piece % 2][px][co], x [row % 4][px][ci]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nco = (Co + 31) / 32, ci0 = (blockIdx.y / nco) * 32, co0 = (blockIdx.y % nco) * 32;
    const int nseg = (W + kWgCols - 1) / kWgCols, rows = B * H;
    const long long units = (long long)nseg * rows;
    const long long u0 = units * blockIdx.x / gridDim.x, u1 = units * (blockIdx.x + 1) / gridDim.x;
    // x row yy + d of a piece into slot (yy + d + 4) % 4, and its dy, asynchronously; channels beyond Ci or
    // Co are zero
    auto load_x = [&](int b, int yy, int x0, int nw, int d) {
        int sy = yy + d;
        float *t = xs + ((sy + 4) & 3) * ROW;
        if (sy < 0) sy += H;
        if (sy >= H) sy -= H;
        for (int c = warp; c < 32; c += 8) {
            const bool on = ci0 + c < Ci;
            const float *src = x + (((size_t)b * Ci + (on ? ci0 + c : 0)) * H + sy) * W;
            for (int p = lane; p < nw + 2; p += 32) {
                int sx = x0 + p - 1;
                if (sx < 0) sx += W;
                if (sx >= W) sx -= W;
                if (on) cp_async4(t + p * kWgXs + c, src + sx);
                else t[p * kWgXs + c] = 0.0f;
            }
        }
    };
    auto load_dy = [&](int b, int yy, int x0, int nw, int buf) {
        for (int c = warp; c < 32; c += 8) {
            const bool on = co0 + c < Co;
            const float *src = dy + (((size_t)b * Co + (on ? co0 + c : 0)) * H + yy) * W + x0;
            for (int p = lane; p < nw; p += 32) {
                if (on) cp_async4(ds + buf * DS + p * kWgDs + c, src + p);
                else ds[buf * DS + p * kWgDs + c] = 0.0f;
            }
        }
    };
    float2 tot[9][2], sb[2];
#pragma unroll
    for (int k = 0; k < 9; ++k) tot[k][0] = tot[k][1] = make_float2(0.f, 0.f);
    sb[0] = sb[1] = make_float2(0.f, 0.f);
    for (long long u = u0; u < u1; ++u) {
        const int sg = (int)(u / rows), r = (int)(u - (long long)sg * rows), b = r / H, yy = r - b * H;
        const int x0 = sg * kWgCols, nw = min(kWgCols, W - x0), buf = (int)((u - u0) & 1);
        if (u == u0 || yy == 0) {  // a new image or column of pieces: nothing was brought ahead
            __syncthreads();
            for (int d = -1; d <= 1; ++d) load_x(b, yy, x0, nw, d);
            load_dy(b, yy, x0, nw, buf);
        }
        cp_async_all();
        __syncthreads();
        if (u + 1 < u1 && yy + 1 < H) {  // the piece below, while this one is summed
            load_x(b, yy + 1, x0, nw, 1);
            load_dy(b, yy + 1, x0, nw, buf ^ 1);
        }
        const float *t[3], *dsb = ds + buf * DS;
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = xs + ((yy + k + 3) & 3) * ROW + lane;
        float2 v[3][3];  // [kernel row][column], each value twice
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int c = 0; c < 2; ++c) v[k][c + 1] = make_float2(t[k][c * kWgXs], t[k][c * kWgXs]);
        float2 acc[9][2], sp[2];  // of this piece: short sums, added to the CTA's afterwards
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k][0] = acc[k][1] = make_float2(0.f, 0.f);
        sp[0] = sp[1] = make_float2(0.f, 0.f);
#pragma unroll 3
        for (int p = 0; p < nw; ++p) {
            const float4 g = *reinterpret_cast<const float4 *>(dsb + p * kWgDs + warp * 4);
            const float2 ga = make_float2(g.x, g.y), gb = make_float2(g.z, g.w);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                v[k][0] = v[k][1];
                v[k][1] = v[k][2];
                const float n = t[k][(p + 2) * kWgXs];
                v[k][2] = make_float2(n, n);
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                acc[k][0] = __ffma2_rn(v[k / 3][k % 3], ga, acc[k][0]);
                acc[k][1] = __ffma2_rn(v[k / 3][k % 3], gb, acc[k][1]);
            }
            sp[0] = __fadd2_rn(sp[0], ga);
            sp[1] = __fadd2_rn(sp[1], gb);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
#pragma unroll
            for (int k = 0; k < 9; ++k) tot[k][j] = __fadd2_rn(tot[k][j], acc[k][j]);
            sb[j] = __fadd2_rn(sb[j], sp[j]);
        }
    }
    float *o = part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kWgPart;
#pragma unroll
    for (int k = 0; k < 9; ++k)
        *reinterpret_cast<float4 *>(o + (k * 32 + lane) * 32 + warp * 4) =
            make_float4(tot[k][0].x, tot[k][0].y, tot[k][1].x, tot[k][1].y);
    if (lane == 0)
        *reinterpret_cast<float4 *>(o + 9 * 1024 + warp * 4) = make_float4(sb[0].x, sb[0].y, sb[1].x, sb[1].y);
}

// dw and db from the G partials of every channel tile (blockIdx.y): one CTA per row (tap, ci) and one
// for db
__global__ void __launch_bounds__(256) k_wgrad_reduce(const float *__restrict__ part, int G, float *__restrict__ dw,
                                                      float *__restrict__ db, int Ci, int Co)
{
    const int m = blockIdx.x, nco = (Co + 31) / 32, ci = (blockIdx.y / nco) * 32 + (m & 31), tap = m >> 5;
    const int co = (blockIdx.y % nco) * 32 + (threadIdx.x & 31);
    if (tap == 9 ? blockIdx.y / nco != 0 : ci >= Ci) return;
    const double s = sum_partials(part + (size_t)blockIdx.y * G * kWgPart + m * 32, G, kWgPart);
    if (threadIdx.x >= 32 || co >= Co) return;
    if (tap == 9) db[co] = (float)s;
    else dw[((size_t)co * Ci + ci) * 9 + tap] = (float)s;
}

// The same for few pixels and channels: a CTA per (ci, co) over all pixels, one launch.  Two launches and the
// latency of a CTA's first pieces bound the kernels above there: 10.4 us at 16^2, 8 x 8 channels, where this
// one takes 4.8.  wgrad_pairs: where it is the faster one (measured, this against those, in us, at B H W pixels
// and Ci x Co channels: 2304 and 16 x 16 12.1 / 14.5, 4096 18.5 / 16.2; 576 and 32 x 32 11.9 / 12.5, 1152
// 17.4 / 12.8; 64 and 64 x 64 17.6 / 12.1; with the threads' sums as an FP32 tree of eight barriers, 0.4 more
// than in FP64 behind one).
constexpr bool wgrad_pairs(long long pixels, int Ci, int Co)
{
    return pixels <= 2048 && Ci * Co <= 1024 && pixels * Ci * Co <= 1 << 19;
}
__global__ void __launch_bounds__(256) k_wgrad_pairs(const float *__restrict__ x, const float *__restrict__ dy,
                                                     float *__restrict__ dw, float *__restrict__ db, int B, int Ci, int Co,
                                                     int H, int W)
{
    __shared__ float red[10][256];
    const int ci = blockIdx.x, co = blockIdx.y, HW = H * W;
    float acc[10];  // 9 taps, db
#pragma unroll
    for (int k = 0; k < 10; ++k) acc[k] = 0.0f;
    for (int p = threadIdx.x; p < B * HW; p += 256) {
        const int b = p / HW, r = p - b * HW, yy = r / W, xx = r - yy * W;
        const int sy[3] = {(yy == 0 ? H - 1 : yy - 1) * W, yy * W, (yy == H - 1 ? 0 : yy + 1) * W};
        const int sx[3] = {xx == 0 ? W - 1 : xx - 1, xx, xx == W - 1 ? 0 : xx + 1};
        const float g = __ldg(dy + ((size_t)b * Co + co) * HW + r);
        const float *xc = x + ((size_t)b * Ci + ci) * HW;
#pragma unroll
        for (int k = 0; k < 9; ++k) acc[k] = fmaf(g, __ldg(xc + sy[k / 3] + sx[k % 3]), acc[k]);
        acc[9] += g;
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) red[k][threadIdx.x] = acc[k];
    __syncthreads();
    // the threads' sums in FP64 and a fixed order, one warp per tap
    const int lane = threadIdx.x & 31;
    for (int k = threadIdx.x >> 5; k < 10; k += 8) {
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s += (double)red[k][i * 32 + lane];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0 && k < 9) dw[((size_t)co * Ci + ci) * 9 + k] = (float)s;
        if (lane == 0 && k == 9 && ci == 0) db[co] = (float)s;
    }
}

// one minibatch from the resident data set: sample src[blockIdx.y] (xs inputs, ts targets) to place
// blockIdx.y.  One launch for all samples (a device copy per tensor and sample took 64 launches at
// batch 32: 48^2 iteration 0.63 -> 0.33 ms).
constexpr int kGather = 512;
struct GatherIdx {
    int n = 0;
    int src[kGather];
};
__global__ void k_gather(const float *__restrict__ dx, const float *__restrict__ dt, const __grid_constant__ GatherIdx g,
                         float *__restrict__ x, float *__restrict__ t, size_t xs, size_t ts)
{
    const size_t k = (size_t)g.src[blockIdx.y], b = blockIdx.y;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < xs + ts; i += (size_t)gridDim.x * blockDim.x) {
        if (i < xs) x[b * xs + i] = dx[k * xs + i];
        else t[b * ts + i - xs] = dt[k * ts + i - xs];
    }
}

// mean squared error over n values and its gradient 2 (p - t) / n; per-block partial losses
__global__ void k_mse(const float *__restrict__ pred, const float *__restrict__ tgt, float *__restrict__ grad,
                      double *__restrict__ part, size_t n)
{
    __shared__ double red[256];
    double acc = 0.0;
    const float sc = 2.0f / (float)n;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float d = pred[i] - tgt[i];
        grad[i] = sc * d;
        acc += (double)d * d;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// Adam (bias-corrected) on the flat parameter vector.  With tensor-core training e0 / e1 (nullable) are the wait
// flags of its kernels: a gradient from a pass in which a wait ran out is not applied, and *steps counts
// the iterations that were.
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2, const int *e0,
                       const int *e1, int *steps)
{
    if ((e0 && *e0) || (e1 && *e1)) return;
    if (steps && blockIdx.x == 0 && threadIdx.x == 0) *steps += 1;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

}  // namespace cnn
}  // namespace dns2d
