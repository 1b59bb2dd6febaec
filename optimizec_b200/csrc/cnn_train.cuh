// cnn_train.cuh — the closure network's training convolutions straight from chunk planes.
//
// The GEMMs are those of cnn_gemm.cuh (bf16 operands, FP32 accumulators in tensor memory), but no
// im2col expansion is written: the operand tensors (activations, and the gradients dz of the
// pre-activations) are kept as bf16 chunk planes, and each tap of a 3x3 kernel is the same plane read
// one pixel or one row further on.
//
// Planes: a tensor of C channels has nch = 2 or 4 chunks of 8 channels (channels beyond C zero);
// element (image b, chunk c, padded row py, padded column px) is 16 bytes at pixel
//     (b nch + c) (H + 2)(W + 2) + py (W + 2) + px,
// px = 1 .. W, py = 1 .. H the image, the frame around it the periodic halo, written by whoever
// writes the tensor.  kGuard zero pixels lie before and after (a tile may reach beyond the last row).
//
//   forward / data gradient (k_conv_planes): an M tile is 128 consecutive padded pixels of one image,
//     so tap (dy, dx) of every pixel of the tile lies (dy - 1)(W + 2) + dx - 1 pixels on: three bulk
//     copies of 130 pixels per chunk bring all nine taps, and a tap is a K-major operand started
//     16 dx bytes into its row's copy.  Positions of the frame are computed and not stored.
//   weight gradient (k_wgrad_planes): K is the pixels and M = (tap, channel): a plane's 16-byte pixel
//     (8 channels) is a row of an M-major core matrix, so the planes are M-major operands as they
//     are, a kernel column dx started dx pixels further on.
//   The 3-channel input and the 1-channel output gradient would fill a third and an eighth of a
//     chunk: their planes hold the 27 (9) products' operands of a pixel themselves, k = tap C + channel
//     in 4 (2) chunks, and enter as a 1 x 1 convolution ("point" tensors).
//
// Operands, their order along K and the pixels that one accumulator sums are those of the im2col GEMMs
// (cnn_gemm.cuh), so for 32 channels the results are the same bit for bit.  The planes hold exactly the
// bf16 operands that the expansions held (rounded once from the same FP32 values); pre-activations,
// loss, weights, accumulators and gradients stay FP32.  One Adam iteration of the 6 x 32 network on
// B200: 384^2, batch 4 4.92 -> 1.10 ms; 48^2, batch 32 1.31 -> 0.34 ms.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace dns2d {
namespace cnntrain {

constexpr int kGuard = 512;     // pixels before and after a tensor's planes
constexpr int kMaxLayers = 32;  // of one packing launch

__host__ __device__ constexpr int chunks_of(int C) { return C <= 16 ? 2 : 4; }
// point tensors: all 9 C products of a pixel
__host__ __device__ constexpr bool point_of(int C) { return 9 * C <= 32; }
__host__ __device__ constexpr int planes_of(int C) { return point_of(C) ? (9 * C <= 16 ? 2 : 4) : chunks_of(C); }
// 16-byte pixels of a tensor's planes with both guards
inline size_t plane_pixels(int B, int C, int H, int W)
{
    return (size_t)B * planes_of(C) * (H + 2) * (W + 2) + 2 * kGuard;
}
// K steps of a convolution over C channels
__host__ __device__ constexpr int ksteps_of(int C) { return (point_of(C) ? 1 : 9) * planes_of(C) / 2; }

// sizes that the planes path takes: the weight gradient's K steps are 16 pixels of one image row (fewer
// than 4 hidden channels would be point tensors)
inline bool supported(int C, int H, int W) { return C >= 4 && C <= 32 && H >= 1 && W >= 16 && W % 16 == 0; }

// operand buffers of a network (grown on demand)
struct Planes {
    uint4 *act = nullptr;   // per layer input: x, a_0 .. a_{L-2}
    uint4 *dz[2] = {nullptr, nullptr};
    __nv_bfloat16 *w = nullptr;  // packed weights: per layer forward, then data gradient
    float *part = nullptr;       // weight-gradient partials
    int *err = nullptr;          // 1: a wait ran out
    size_t act_cap = 0, dz_cap = 0, w_cap = 0, part_cap = 0;  // pixels, pixels, elements, floats
};

// everything a pass needs of one network and batch; layer l maps ci[l] -> co[l] channels
struct Net {
    int L = 0, B = 0, H = 0, W = 0;
    const int *ci = nullptr, *co = nullptr;
    const size_t *woff = nullptr;
    const float *params = nullptr;
    float *grad = nullptr;
    const float *x = nullptr;      // [B][ci[0]][H][W]
    float *const *z = nullptr;     // pre-activations per layer, [B][co][H][W]
    const float *dout = nullptr;   // loss gradient of the output [B][co[L-1]][H][W]
};

cudaError_t reserve(const Net &n, Planes &p, cudaStream_t st);
cudaError_t forward(const Net &n, Planes &p, cudaStream_t st);   // fills z of every layer
cudaError_t backward(const Net &n, Planes &p, cudaStream_t st);  // after forward: fills grad
void release(Planes &p);

}  // namespace cnntrain
}  // namespace dns2d
