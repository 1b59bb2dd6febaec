// cnn_train.cu — training convolutions on chunk planes (cnn_train.cuh).
#include "cnn_math.cuh"
#include "cnn_train.cuh"
#include "cnn_tc.cuh"

#include <algorithm>
#include <vector>

namespace dns2d {
namespace cnntrain {
namespace {

using cnntc::bulk_g2s;
using cnntc::idesc_bf16;
using cnntc::mbar_arrive;
using cnntc::mbar_expect_tx;
using cnntc::mbar_init;
using cnntc::mbar_wait;
using cnntc::mma_bf16;
using cnntc::mma_commit;
using cnntc::saddr;
using cnntc::smem_desc;
using cnntc::tmem_ld32;

using cnn::gelu;
using cnn::gelu_grad;

__device__ __forceinline__ uint4 pack8(const float *v)
{
    uint4 u;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    return u;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *holder, int cols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(holder)), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
}

// the chunk of pixel (y, x) of one plane, at its place and at every frame position that repeats it
__device__ __forceinline__ void store_halo(uint4 *plane, int H, int W, int y, int x, uint4 v)
{
    const int Wp = W + 2;
    uint4 *d = plane + (size_t)(y + 1) * Wp + x + 1;
    *d = v;
    const bool l = x == 0, r = x == W - 1;
    if (l) d[W] = v;
    if (r) d[-W] = v;
    if (y == 0) {
        uint4 *e = d + (size_t)H * Wp;
        *e = v;
        if (l) e[W] = v;
        if (r) e[-W] = v;
    }
    if (y == H - 1) {
        uint4 *e = d - (size_t)H * Wp;
        *e = v;
        if (l) e[W] = v;
        if (r) e[-W] = v;
    }
}

// FP32 [B][C][H][W] -> a point tensor: one thread per image pixel and chunk
template <int C>
__global__ void k_to_points(const float *__restrict__ x, int B, int H, int W, uint4 *__restrict__ pl)
{
    static_assert(point_of(C), "all products of a pixel in its chunks");
    constexpr int NCH = planes_of(C);
    const int Wp = W + 2, PS = (H + 2) * Wp, HW = H * W;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < B * HW; e += gridDim.x * blockDim.x) {
        const int b = e / HW, p = e - b * HW, y = p / W, xx = p - y * W;
        const int sy[3] = {(y == 0 ? H - 1 : y - 1) * W, y * W, (y == H - 1 ? 0 : y + 1) * W};
        const int sx[3] = {xx == 0 ? W - 1 : xx - 1, xx, xx == W - 1 ? 0 : xx + 1};
        const float *xb = x + (size_t)b * C * HW;
        float v[NCH * 8];
#pragma unroll
        for (int k = 0; k < NCH * 8; ++k)
            v[k] = k < 9 * C ? __ldg(xb + (size_t)(k % C) * HW + sy[(k / C) / 3 % 3] + sx[(k / C) % 3]) : 0.0f;
        uint4 *o = pl + (size_t)b * NCH * PS + (size_t)(y + 1) * Wp + xx + 1;
#pragma unroll
        for (int c = 0; c < NCH; ++c) o[(size_t)c * PS] = pack8(v + 8 * c);
    }
}

// Packed weights of every layer: per layer the forward operand (K = taps x input channels, N = co)
// and the data-gradient operand (K = flipped taps x output channels, N = ci), each ksteps_of(K
// channels) blocks of [k / 8][n][k % 8] (16 k x 32 n).  K step s: tap s / (nch / 2) and its chunk pair,
// or the 16 products k = 16 s ... of a point tensor.
struct PackArgs {
    int L = 0;
    int ci[kMaxLayers], co[kMaxLayers];
    unsigned int woff[kMaxLayers], fwd[kMaxLayers], bwd[kMaxLayers];
};

__global__ void k_pack_planes(const float *__restrict__ params, const __grid_constant__ PackArgs a,
                              __nv_bfloat16 *__restrict__ out)
{
    const int l = blockIdx.y >> 1, flip = blockIdx.y & 1;
    const int Ci = a.ci[l], Co = a.co[l], Kin = flip ? Co : Ci, Nout = flip ? Ci : Co;
    const int hp = planes_of(Kin) / 2, KS = ksteps_of(Kin);
    const float *w = params + a.woff[l];
    __nv_bfloat16 *o = out + (flip ? a.bwd[l] : a.fwd[l]);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < KS * 512; e += gridDim.x * blockDim.x) {
        const int s = e >> 9, h = (e >> 8) & 1, n = (e >> 3) & 31, k = e & 7;
        int tap, ch;
        if (point_of(Kin)) {
            const int kk = s * 16 + h * 8 + k;
            tap = kk / Kin;
            ch = kk - tap * Kin;
        } else {
            tap = s / hp;
            ch = ((s - tap * hp) * 2 + h) * 8 + k;
        }
        float v = 0.0f;
        if (tap < 9 && ch < Kin && n < Nout)
            v = flip ? w[((size_t)ch * Ci + n) * 9 + (8 - tap)] : w[((size_t)n * Ci + ch) * 9 + tap];
        o[e] = __float2bfloat16_rn(v);
    }
}

struct ConvArgs {
    const uint4 *in = nullptr;          // planes (after the guard)
    const __nv_bfloat16 *w = nullptr;   // KS packed blocks
    int nch = 4, KS = 18, rows = 3;     // of the input; rows: 3, or 1 for a point tensor
    int B = 0, H = 0, W = 0, Nv = 0;    // Nv output channels
    int tiles_img = 0, tiles = 0;
    const float *bias = nullptr;        // forward
    float *z = nullptr;                 // forward: pre-activations [B][Nv][H][W]
    const float *zprev = nullptr;       // data gradient: GELU'(zprev) factor [B][Nv][H][W]
    uint4 *out = nullptr;               // planes of GELU(z) or of dz of the layer below; nullptr: none
    int *err = nullptr;
};

constexpr int kSeg = 2176;         // bytes of one row copy in shared memory (130 pixels, 2080 bytes used)
constexpr int kSegPx = 130;
constexpr int kConvStages = 3, kConvCtas = 2;  // 4 stages leave one CTA per SM: iteration 1.01 -> 1.21 ms
constexpr int kConvThreads = 320;  // warps 0-7 epilogue, 8 producer, 9 MMA issuer

// One convolution over planes (forward or data gradient).  CTA c takes tiles c, c + G, ...  At 384^2,
// batch 4, 32 channels (B200): 57 us forward, 62 for a data gradient.  Bound by the epilogue's erf and stores
// (issue 68-70 % busy); without them (one output channel, no GELU) the chain of a tile's 18 dependent MMAs
// alone takes 36 (tensor pipe 15 % busy); the tensors moved (z, planes in and out, 150 MB) would take 23.
// Against 97 us of im2col expansion and 88 us of GEMM before.  Two CTAs per SM give 16 epilogue warps.
// Every wait is bounded (2 s): one that runs out sets *err, and each role ends after the copies and
// MMAs in flight.
__global__ void __launch_bounds__(kConvThreads, kConvCtas) k_conv_planes(const __grid_constant__ ConvArgs q)
{
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t full[kConvStages], empty[kConvStages], tfull[2], tempty[2], wbar;
    __shared__ uint32_t tmem_holder;
    __shared__ float sbias[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KS = q.KS, nch = q.nch, Wp = q.W + 2, PS = (q.H + 2) * Wp, G = (int)gridDim.x;
    const int ncopy = q.rows * nch, stageB = ncopy * kSeg;
    unsigned char *sB = sm, *sA = sm + KS * 1024;
    if (tid < 32) sbias[tid] = (q.bias && tid < q.Nv) ? q.bias[tid] : 0.0f;
    if (warp == 0) tmem_alloc(&tmem_holder, 64);
    if (tid == 0) {
        for (int s = 0; s < kConvStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], 1);
            mbar_init(&tempty[b], 8);
        }
        mbar_init(&wbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_holder;

    if (warp == 8) {
        if (lane == 0) {
            mbar_expect_tx(&wbar, (uint32_t)(KS * 1024));
            bulk_g2s(sB, q.w, (uint32_t)(KS * 1024), &wbar);
        }
        int k = 0;
        for (int tile = (int)blockIdx.x; tile < q.tiles; tile += G, ++k) {
            const int s = k % kConvStages;
            bool ok = true;
            if (lane == 0) {
                ok = k < kConvStages || mbar_wait(&empty[s], (uint32_t)((k / kConvStages - 1) & 1));
                if (ok) mbar_expect_tx(&full[s], (uint32_t)(ncopy * kSegPx * 16));
                else atomicExch(q.err, 1);
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) break;
            if (lane < ncopy) {
                const int dy = q.rows == 3 ? lane / nch : 1, c = q.rows == 3 ? lane - dy * nch : lane;
                const int b = tile / q.tiles_img, q0 = Wp + (tile - b * q.tiles_img) * 128;
                const uint4 *src = q.in + ((ptrdiff_t)(b * nch + c) * PS + q0 + (dy - 1) * Wp - 1);
                bulk_g2s(sA + (size_t)s * stageB + lane * kSeg, src, (uint32_t)(kSegPx * 16), &full[s]);
            }
        }
        if (lane == 0) {  // the copies issued have landed before the CTA can end
            for (int kk = std::max(0, k - kConvStages); kk < k; ++kk)
                mbar_wait(&full[kk % kConvStages], (uint32_t)((kk / kConvStages) & 1));
            mbar_wait(&wbar, 0);
        }
        __syncwarp();
    } else if (warp == 9) {
        if (lane == 0) {
            bool ok = mbar_wait(&wbar, 0);
            const uint64_t db0 = smem_desc(saddr(sB), 512, 128);
            constexpr uint32_t idesc = idesc_bf16(32);
            int k = 0;
            for (int tile = (int)blockIdx.x; ok && tile < q.tiles; tile += G, ++k) {
                const int s = k % kConvStages, bb = k & 1;
                ok = mbar_wait(&full[s], (uint32_t)((k / kConvStages) & 1)) &&
                     (k < 2 || mbar_wait(&tempty[bb], (uint32_t)((k / 2 - 1) & 1)));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t a0 = saddr(sA) + (uint32_t)(s * stageB), d = tmem + (uint32_t)(bb * 32);
                const uint64_t da = smem_desc(a0, kSeg, 128);  // the second 8 k: the next chunk plane
                const int hp = nch / 2;
                int ks = 0;
                for (int tap = q.rows == 3 ? 0 : 4; tap < (q.rows == 3 ? 9 : 5); ++tap) {
                    const int row = q.rows == 3 ? tap / 3 : 0;
                    for (int h = 0; h < hp; ++h, ++ks)
                        mma_bf16(d, da + (uint64_t)(((row * nch + 2 * h) * kSeg + (tap % 3) * 16) >> 4),
                                 db0 + (uint64_t)(ks * 64), idesc, ks > 0 ? 1u : 0u);
                }
                mma_commit(&empty[s]);
                mma_commit(&tfull[bb]);
            }
            if (!ok) atomicExch(q.err, 1);
            // the MMAs issued are done before tensor memory is given back
            if (k > 0) mbar_wait(&empty[(k - 1) % kConvStages], (uint32_t)(((k - 1) / kConvStages) & 1));
        }
        __syncwarp();
    } else {
        // warp w: TMEM lanes 32 (w % 4) .. (pixels), columns 16 (w / 4) .. + 15 (channels)
        const int qd = warp & 3, c0 = 16 * (warp >> 2);
        const size_t HW = (size_t)q.H * q.W;
        const int ncho = chunks_of(q.Nv);  // of the output planes
        int k = 0;
        for (int tile = (int)blockIdx.x; tile < q.tiles; tile += G, ++k) {
            const int bb = k & 1;
            const int b = tile / q.tiles_img, p = Wp + (tile - b * q.tiles_img) * 128 + qd * 32 + lane;
            const int py = p / Wp, px = p - py * Wp;
            const bool on = py <= q.H && px >= 1 && px <= q.W && c0 < q.Nv;
            const int y = py - 1, x = px - 1;
            const size_t o0 = ((size_t)b * q.Nv + c0) * HW + (size_t)(on ? y * q.W + x : 0);
            float zp[16];
            if (q.zprev && on) {  // while the MMAs run
#pragma unroll
                for (int j = 0; j < 16; ++j) zp[j] = c0 + j < q.Nv ? __ldg(q.zprev + o0 + j * HW) : 0.0f;
            }
            const bool got = mbar_wait(&tfull[bb], (uint32_t)((k / 2) & 1));
            if (!__all_sync(0xffffffffu, got)) {
                if (lane == 0) atomicExch(q.err, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            uint32_t r[16];
            tmem_ld16(tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(bb * 32 + c0), r);
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[bb]);
            float v[16];
            if (!on) {
                // a frame position, or columns without a channel
            } else if (q.zprev) {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) * gelu_grad(zp[j]);
            } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) + sbias[c0 + j];
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c0 + j < q.Nv) q.z[o0 + j * HW] = v[j];
                if (q.out) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = gelu(v[j]);
                }
            }
            if (on && q.out) {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (c0 + j >= q.Nv) v[j] = 0.0f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int c = (c0 >> 3) + h;
                    if (c < ncho) store_halo(q.out + (size_t)(b * ncho + c) * PS, q.H, q.W, y, x, pack8(v + 8 * h));
                }
            }
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(64));
}

struct WgradArgs {
    const uint4 *x = nullptr, *dz = nullptr;  // planes (after the guard)
    int nchi = 4, ncho = 4, rows = 3;         // rows: kernel rows of x, 3, or 1 for a point tensor
    int H = 0, W = 0;
    int ksteps = 0, items = 0;                // 16-pixel K steps in all; items of kKC of them
    float *part = nullptr;                    // [G][rows][128][32]
    int *err = nullptr;
};

constexpr int kKC = 4;              // K steps per item
constexpr int kPlanePx = 16 * kKC + 2 * kKC;
constexpr int kPlane = kPlanePx * 16;  // bytes of a plane in shared memory: an item's pixels and 2 more per image row
constexpr int kWgradStages = 8;
constexpr int kProducers = 2;       // producer warps, items in turn (one: iteration 1.13 -> 1.10 ms)
constexpr int kWgradThreads = 160 + 32 * kProducers;  // warps 0-3 epilogue, 4 MMA issuer, 5 ... producers

// A and B M-major / N-major: bits 15 and 16 of the instruction descriptor
constexpr uint32_t kBothMajor = (1u << 15) | (1u << 16);

// shared-memory planes of a stage: rows nchi of x, the ones plane, ncho of dz
__host__ __device__ constexpr int wgrad_planes(int rows, int nchi, int ncho) { return rows * nchi + 1 + ncho; }

// Weight gradient: an item is 4 K steps, 64 consecutive image pixels (W a multiple of 16, so a K step
// stays within an image row), of dz and, for each kernel row dy, of the x planes dy rows on with one
// pixel more on either side of each image row's piece; a kernel column dx is the same operand started
// dx pixels further on.  Accumulator dx: row m = (dy nchi + chunk) 8 + channel, row 8 x planes the
// product with a plane of ones (db).  The M tile's 16 planes reach beyond those into whatever lies
// behind them in shared memory: those rows are not read.  CTA c takes items c, c + G, ... into
// accumulators that it writes once: part[c].  Measured 63 us at 384^2, batch 4, 32 channels against
// 0.41 ms of expansion, packing and GEMM before; bound by the chain of MMAs on an accumulator (252 of
// them, about 290 cycles apart when none lies between), whose grouping fixes the rounding of the sums.
// Waits are bounded as in k_conv_planes.
__global__ void __launch_bounds__(kWgradThreads, 1) k_wgrad_planes(const __grid_constant__ WgradArgs q)
{
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ __align__(8) uint64_t full[kWgradStages], empty[kWgradStages], tfull;
    __shared__ uint32_t tmem_holder;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, G = (int)gridDim.x;
    const int nA = q.rows * q.nchi, stageB = wgrad_planes(q.rows, q.nchi, q.ncho) * kPlane, halo = q.rows == 3 ? 2 : 0;
    if (warp == 0) tmem_alloc(&tmem_holder, 128);
    if (tid == 0) {
        for (int s = 0; s < kWgradStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&tfull, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    for (int e = tid; e < kWgradStages * (kPlane / 16); e += kWgradThreads)  // channel 0 of the ones plane: 1.0 (0x3f80)
        *reinterpret_cast<uint4 *>(sm + (size_t)(e / (kPlane / 16)) * stageB + nA * kPlane + (e % (kPlane / 16)) * 16) =
            make_uint4(0x3f80u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tmem_holder;
    const int Wp = q.W + 2, PS = (q.H + 2) * Wp, KW = q.W / 16;

    if (warp >= 5) {
        const int my_dy = q.rows == 3 ? lane / q.nchi : 1, my_c = q.rows == 3 ? lane - my_dy * q.nchi : lane;
        const int my_off = (my_dy - 1) * Wp - halo / 2;
        int k = warp - 5, last = -1;
        for (int it = (int)blockIdx.x + k * G; it < q.items; it += kProducers * G, k += kProducers) {
            const int s = k % kWgradStages, s0 = it * kKC, nks = min(kKC, q.ksteps - s0), r0 = s0 / KW;
            const int nseg = (s0 + nks - 1) / KW - r0 + 1;  // image rows that the item touches
            bool ok = true;
            if (lane == 0) {
                ok = k < kWgradStages || mbar_wait(&empty[s], (uint32_t)((k / kWgradStages - 1) & 1));
                if (ok) mbar_expect_tx(&full[s], (uint32_t)((nA * (16 * nks + halo * nseg) + q.ncho * 16 * nks) * 16));
                else atomicExch(q.err, 1);
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) break;
            unsigned char *st = sm + (size_t)s * stageB;
            if (nseg == 1) {  // one copy per plane (at most 16)
                const int b = r0 / q.H, pix = (r0 - b * q.H + 1) * Wp + (s0 - r0 * KW) * 16 + 1;
                if (lane < nA)
                    bulk_g2s(st + lane * kPlane, q.x + ((ptrdiff_t)(b * q.nchi + my_c) * PS + pix + my_off),
                             (uint32_t)((16 * nks + halo) * 16), &full[s]);
                else if (lane < nA + q.ncho)
                    bulk_g2s(st + (lane + 1) * kPlane, q.dz + ((ptrdiff_t)(b * q.ncho + lane - nA) * PS + pix),
                             (uint32_t)(nks * 256), &full[s]);
            }
            for (int e = lane; nseg > 1 && e < (nA + q.ncho) * nseg; e += 32) {
                const int pl = e / nseg, g = e - pl * nseg;
                const int a = max(s0, (r0 + g) * KW), z = min(s0 + nks, (r0 + g + 1) * KW);  // its K steps
                const int b = (r0 + g) / q.H, y = (r0 + g) - b * q.H, x0 = (a - (r0 + g) * KW) * 16, n = (z - a) * 16;
                if (pl < nA) {
                    const int dy = q.rows == 3 ? pl / q.nchi : 1, c = q.rows == 3 ? pl - dy * q.nchi : pl;
                    bulk_g2s(st + (size_t)pl * kPlane + ((a - s0) * 16 + halo * g) * 16,
                             q.x + ((ptrdiff_t)(b * q.nchi + c) * PS + (y + dy) * Wp + x0 + 1 - halo / 2),
                             (uint32_t)((n + halo) * 16), &full[s]);
                } else {
                    bulk_g2s(st + (size_t)(pl + 1) * kPlane + (a - s0) * 256,
                             q.dz + ((ptrdiff_t)(b * q.ncho + pl - nA) * PS + (y + 1) * Wp + x0 + 1), (uint32_t)(n * 16),
                             &full[s]);
                }
            }
            last = k;
            __syncwarp();
        }
        if (lane == 0)  // the copies issued have landed before the CTA can end
            for (int kk = last; kk >= 0 && kk > last - kWgradStages; kk -= kProducers)
                mbar_wait(&full[kk % kWgradStages], (uint32_t)((kk / kWgradStages) & 1));
        __syncwarp();
    } else if (warp == 4) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(q.ncho > 2 ? 32 : 16) | kBothMajor;
            int k = 0;
            bool ok = true;
            for (int it = (int)blockIdx.x; it < q.items; it += G, ++k) {
                const int s = k % kWgradStages;
                ok = mbar_wait(&full[s], (uint32_t)((k / kWgradStages) & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t st = saddr(sm) + (uint32_t)(s * stageB);
                // 8 pixels (a core matrix) further along K: 128 bytes; 8 channels further along M or N: a plane
                const uint64_t da = smem_desc(st, 128, kPlane), db = smem_desc(st + (uint32_t)((nA + 1) * kPlane), 128, kPlane);
                const int s0 = it * kKC, nks = min(kKC, q.ksteps - s0);
                int row_end = KW - s0 % KW, px = 0;  // the K step that begins the next image row's piece
                for (int ks = 0; ks < nks; ++ks, px += 16) {
                    if (ks == row_end) {
                        row_end += KW;
                        px += halo;
                    }
                    for (int dx = 0; dx < q.rows; ++dx)
                        mma_bf16(tmem + (uint32_t)(dx * 32), da + (uint64_t)(px + dx), db + (uint64_t)(16 * ks), idesc,
                                 (k > 0 || ks > 0) ? 1u : 0u);
                }
                mma_commit(&empty[s]);
            }
            if (!ok) atomicExch(q.err, 1);
            mma_commit(&tfull);  // arrives when every MMA issued is done
            if (k > 0) mbar_wait(&empty[(k - 1) % kWgradStages], (uint32_t)(((k - 1) / kWgradStages) & 1));
        }
        __syncwarp();
    } else {
        const bool got = mbar_wait(&tfull, 0u);  // G <= items: every CTA has one
        if (!__all_sync(0xffffffffu, got)) {
            if (lane == 0) atomicExch(q.err, 1);
        } else {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            for (int dx = 0; dx < q.rows; ++dx) {
                uint32_t r[32];
                tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(dx * 32), r);
                float4 *dst = reinterpret_cast<float4 *>(
                    q.part + (((size_t)blockIdx.x * q.rows + dx) * 128 + warp * 32 + lane) * 32);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    dst[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                         __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(128));
}

// dw[co][ci][tap] and db[co] from the G partials: one CTA per row of an accumulator (output channel
// co in column c0 + co).  Row m: of the planes of one
// kernel row after another, or (rows 1) the products k = tap Ci + ci of a point tensor; row 8 x planes: db.
__global__ void __launch_bounds__(256) k_reduce_planes(const float *__restrict__ part, int G, int rows, int nchi, int c0,
                                                       int Ci, int Co, float *__restrict__ dw, float *__restrict__ db)
{
    const int m = blockIdx.x, dx = blockIdx.y, co = (threadIdx.x & 31) - c0;
    const bool ones = m == 8 * rows * nchi;
    int tap, ci;
    if (rows == 3) {
        const int dy = m / (8 * nchi);
        ci = m - dy * 8 * nchi;
        tap = dy * 3 + dx;
    } else {
        tap = m / Ci;
        ci = m - tap * Ci;
    }
    if (ones ? dx != 0 : (ci >= Ci || tap >= 9)) return;
    const double s = cnn::sum_partials(part + ((size_t)dx * 128 + m) * 32, G, (size_t)rows * 128 * 32);
    if (threadIdx.x >= 32 || co < 0 || co >= Co) return;
    if (ones) db[co] = (float)s;
    else dw[((size_t)co * Ci + ci) * 9 + tap] = (float)s;
}

cudaError_t grow(void **p, size_t *cap, size_t need, size_t elem, bool clear, cudaStream_t st)
{
    if (need <= *cap) return cudaSuccess;
    cudaError_t e = cudaStreamSynchronize(st);  // the old buffer may be in use
    if (e != cudaSuccess) return e;
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    if ((e = cudaMalloc(p, need * elem)) != cudaSuccess) return e;
    *cap = need;
    return clear ? cudaMemsetAsync(*p, 0, need * elem, st) : cudaSuccess;
}

int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return std::max(sms, 1);
}

// planes of layer l's input within Planes::act (after its guard)
uint4 *input_planes(const Net &n, const Planes &p, int l)
{
    size_t off = kGuard;
    for (int i = 0; i < l; ++i) off += plane_pixels(n.B, n.ci[i], n.H, n.W);
    return p.act + off;
}

// dynamic shared memory of k_conv_planes for Cin input channels, and of k_wgrad_planes
constexpr size_t conv_smem(int Cin)
{
    return (size_t)ksteps_of(Cin) * 1024 + (size_t)kConvStages * (point_of(Cin) ? 1 : 3) * planes_of(Cin) * kSeg;
}
constexpr size_t wgrad_smem(int rows, int nchi, int ncho)
{
    // the last stage's M tile reaches 16 planes from its start
    const int planes = wgrad_planes(rows, nchi, ncho), tail = planes < 16 ? 16 - planes : 0;
    return (size_t)(kWgradStages * planes + tail) * kPlane;
}
constexpr int kMaxC = 32;  // of supported()
static_assert(conv_smem(kMaxC) >= conv_smem(16) && conv_smem(kMaxC) >= conv_smem(3) && conv_smem(kMaxC) >= conv_smem(1) &&
                  wgrad_smem(3, 4, 4) >= wgrad_smem(3, 2, 2) && wgrad_smem(3, 4, 4) >= wgrad_smem(1, 4, 4) &&
                  wgrad_smem(3, 4, 4) <= 227 * 1024,
              "the most shared memory that any layer asks for");

cudaError_t conv(const Net &n, ConvArgs a, int Cin, cudaStream_t st)
{
    a.nch = planes_of(Cin);
    a.KS = ksteps_of(Cin);
    a.rows = point_of(Cin) ? 1 : 3;
    a.B = n.B;
    a.H = n.H;
    a.W = n.W;
    a.tiles_img = (n.H * (n.W + 2) + 127) / 128;
    a.tiles = a.tiles_img * n.B;
    k_conv_planes<<<std::min(a.tiles, kConvCtas * sm_count()), kConvThreads, conv_smem(Cin), st>>>(a);
    return cudaGetLastError();
}

cudaError_t wgrad(const Net &n, const uint4 *x, const uint4 *dz, int l, Planes &p, cudaStream_t st)
{
    WgradArgs a;
    a.x = x;
    a.dz = dz;
    a.nchi = planes_of(n.ci[l]);
    a.ncho = planes_of(n.co[l]);
    a.rows = point_of(n.ci[l]) ? 1 : 3;
    a.H = n.H;
    a.W = n.W;
    a.ksteps = n.B * n.H * (n.W / 16);
    a.items = (a.ksteps + kKC - 1) / kKC;
    a.part = p.part;
    a.err = p.err;
    const int G = std::min(a.items, sm_count());
    k_wgrad_planes<<<G, kWgradThreads, wgrad_smem(a.rows, a.nchi, a.ncho), st>>>(a);
    float *dw = n.grad + n.woff[l], *db = dw + (size_t)n.co[l] * n.ci[l] * 9;
    // a point tensor's centre tap is the tensor itself
    k_reduce_planes<<<dim3(8 * a.rows * a.nchi + 1, a.rows), 256, 0, st>>>(
        p.part, G, a.rows, a.nchi, point_of(n.co[l]) ? 4 * n.co[l] : 0, n.ci[l], n.co[l], dw, db);
    return cudaGetLastError();
}

int blocks_for(long long items) { return (int)std::max<long long>(1, std::min<long long>(2048, (items + 255) / 256)); }

}  // namespace

cudaError_t reserve(const Net &n, Planes &p, cudaStream_t st)
{
    size_t act = 0, w = 0;
    int cmax = 1;
    for (int l = 0; l < n.L; ++l) {
        act += plane_pixels(n.B, n.ci[l], n.H, n.W);
        w += (size_t)(ksteps_of(n.ci[l]) + ksteps_of(n.co[l])) * 512;
        cmax = std::max(cmax, n.co[l]);
    }
    cudaError_t e;
    if (!p.err) {
        // the limit belongs to the function: the most that any layer of any network asks for, so that networks
        // on several host threads set the same value
        const cudaFuncAttribute sm = cudaFuncAttributeMaxDynamicSharedMemorySize;
        if ((e = cudaFuncSetAttribute(k_conv_planes, sm, (int)conv_smem(kMaxC))) != cudaSuccess) return e;
        if ((e = cudaFuncSetAttribute(k_wgrad_planes, sm, (int)wgrad_smem(3, 4, 4))) != cudaSuccess) return e;
        if ((e = cudaMalloc((void **)&p.err, 4)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(p.err, 0, 4, st)) != cudaSuccess) return e;
    }
    if ((e = grow((void **)&p.act, &p.act_cap, act, 16, true, st)) != cudaSuccess) return e;
    const size_t dz = std::max(plane_pixels(n.B, cmax, n.H, n.W), plane_pixels(n.B, n.co[n.L - 1], n.H, n.W));
    if (dz > p.dz_cap) {
        size_t c0 = p.dz_cap, c1 = p.dz_cap;
        p.dz_cap = 0;
        if ((e = grow((void **)&p.dz[0], &c0, dz, 16, true, st)) != cudaSuccess) return e;
        if ((e = grow((void **)&p.dz[1], &c1, dz, 16, true, st)) != cudaSuccess) return e;
        p.dz_cap = dz;
    }
    if ((e = grow((void **)&p.w, &p.w_cap, w, 2, false, st)) != cudaSuccess) return e;
    return grow((void **)&p.part, &p.part_cap, (size_t)sm_count() * 3 * 128 * 32, 4, false, st);
}

cudaError_t forward(const Net &n, Planes &p, cudaStream_t st)
{
    cudaError_t e = reserve(n, p, st);
    if (e != cudaSuccess) return e;
    std::vector<size_t> fwd(n.L);
    size_t off = 0;
    for (int l = 0; l < n.L; ++l) {
        fwd[l] = off;
        off += (size_t)(ksteps_of(n.ci[l]) + ksteps_of(n.co[l])) * 512;
    }
    for (int l0 = 0; l0 < n.L; l0 += kMaxLayers) {
        PackArgs pa;
        pa.L = std::min(kMaxLayers, n.L - l0);
        for (int i = 0; i < pa.L; ++i) {
            pa.ci[i] = n.ci[l0 + i];
            pa.co[i] = n.co[l0 + i];
            pa.woff[i] = (unsigned)n.woff[l0 + i];
            pa.fwd[i] = (unsigned)fwd[l0 + i];
            pa.bwd[i] = (unsigned)(fwd[l0 + i] + (size_t)ksteps_of(n.ci[l0 + i]) * 512);
        }
        k_pack_planes<<<dim3(4, 2 * pa.L), 256, 0, st>>>(n.params, pa, p.w);
    }
    if (n.ci[0] != 3 || n.co[n.L - 1] != 1) return cudaErrorInvalidValue;
    k_to_points<3><<<blocks_for((long long)n.B * n.H * n.W), 256, 0, st>>>(n.x, n.B, n.H, n.W, input_planes(n, p, 0));
    for (int l = 0; l < n.L; ++l) {
        ConvArgs a;
        a.in = input_planes(n, p, l);
        a.w = p.w + fwd[l];
        a.Nv = n.co[l];
        a.bias = n.params + n.woff[l] + (size_t)n.co[l] * n.ci[l] * 9;
        a.z = n.z[l];
        a.out = l + 1 < n.L ? input_planes(n, p, l + 1) : nullptr;
        a.err = p.err;
        if ((e = conv(n, a, n.ci[l], st)) != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

cudaError_t backward(const Net &n, Planes &p, cudaStream_t st)
{
    uint4 *dz = p.dz[0] + kGuard, *other = p.dz[1] + kGuard;
    k_to_points<1><<<blocks_for((long long)n.B * n.H * n.W), 256, 0, st>>>(n.dout, n.B, n.H, n.W, dz);
    size_t off = 0;
    std::vector<size_t> fwd(n.L);
    for (int l = 0; l < n.L; ++l) {
        fwd[l] = off;
        off += (size_t)(ksteps_of(n.ci[l]) + ksteps_of(n.co[l])) * 512;
    }
    cudaError_t e = cudaGetLastError();
    for (int l = n.L - 1; l >= 0 && e == cudaSuccess; --l) {
        if ((e = wgrad(n, input_planes(n, p, l), dz, l, p, st)) != cudaSuccess) break;
        if (l == 0) break;
        ConvArgs a;
        a.in = dz;
        a.w = p.w + fwd[l] + (size_t)ksteps_of(n.ci[l]) * 512;
        a.Nv = n.ci[l];
        a.zprev = n.z[l - 1];
        a.out = other;
        a.err = p.err;
        e = conv(n, a, n.co[l], st);
        std::swap(dz, other);
    }
    return e;
}

void release(Planes &p)
{
    cudaFree(p.act);
    cudaFree(p.dz[0]);
    cudaFree(p.dz[1]);
    cudaFree(p.w);
    cudaFree(p.part);
    cudaFree(p.err);
    p = Planes{};
}

}  // namespace cnntrain
}  // namespace dns2d
