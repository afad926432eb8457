// Learned 2x flow upsampler for the FLOWDOWNSCALE fast mode (no counterpart
// in the reference, whose fast mode upsamples the flow bilinearly,
// flowmodel.cpp:158-161).
//
// Input at the full resolution: the bilinear upsampling of the coarse flow
// with its vectors scaled to the full-resolution grid (the "base" flow) and
// the luma of the full-resolution frame.  Four 3x3 convolutions (3 -> 32 ->
// 32 -> 32 -> 2, zero padding, ReLU between) predict a residual r; the
// output flow is base + r where max(|r_u|, |r_v|) <= max_residual, else the
// base flow (the bilinear fallback).  19,970 parameters, kept in FP32 for
// training and rounded to FP16 for inference.
//
// The training kernels are written here, in FP32: direct convolutions on the
// CUDA cores over planar activations (register tiles of pixels and channels
// fed from shared memory, fused multiply-adds), a backward pass for the data
// and the weights, an L1 loss against the full-resolution flow and Adam.  The
// input preparation is shared with the inference, which runs on the tensor
// cores (vsc_upsampler_tc.cu).  Nothing here has a bit-exact contract
// (contraction is spelled out with __fmaf_rn, the library being built
// without automatic contraction).
#include "vsc_device.h"
#include "vsc_internal.h"
#include "vsc_math.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace vsc {
namespace {

constexpr int kParams = 19970;
static_assert(kUpLayers[3].b_off + 2 == kParams, "parameter layout");

__device__ __forceinline__ float luma(const float* p) { return 0.299f * p[0] + 0.587f * p[1] + 0.114f * p[2]; }

// ---- input: base flow and luma ------------------------------------------------------
// base = bilinear(coarse) at the frame's size (kernel_bilinear's sampling,
// flowconsistency.cu:50-75) times the size ratio per axis.  plane, if given:
// the same values as the tensor-core inference's first chunk plane (FP16, five
// zero channels).
__global__ void prepare_kernel(const float* __restrict__ coarse, int cw, int ch, int cfc, const float* __restrict__ img,
    float* __restrict__ input, int w, int h, int64_t s_coarse, int64_t s_img, int64_t s_in,
    uint4* __restrict__ plane)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int n = blockIdx.z;
    if (x >= w || y >= h)
        return;
    const float* cf = coarse + n * s_coarse;
    const float xx = static_cast<float>(x) * static_cast<float>(cw) / static_cast<float>(w);
    const float yy = static_cast<float>(y) * static_cast<float>(ch) / static_cast<float>(h);
    const int ix = min(static_cast<int>(floorf(xx)), cw - 1), iy = min(static_cast<int>(floorf(yy)), ch - 1);
    const float fx = xx - static_cast<float>(ix), fy = yy - static_cast<float>(iy);
    const int ix1 = min(ix + 1, cw - 1), iy1 = min(iy + 1, ch - 1);
    const float sx = static_cast<float>(w) / static_cast<float>(cw), sy = static_cast<float>(h) / static_cast<float>(ch);
    float v[2];
    for (int k = 0; k < 2; ++k) {
        const float v00 = cf[pix_index(ix, iy, cw) * cfc + k], v10 = cf[pix_index(ix1, iy, cw) * cfc + k];
        const float v01 = cf[pix_index(ix, iy1, cw) * cfc + k], v11 = cf[pix_index(ix1, iy1, cw) * cfc + k];
        v[k] = v00 * (1 - fx) * (1 - fy) + v10 * fx * (1 - fy) + v01 * (1 - fx) * fy + v11 * fx * fy;
    }
    float* o = input + n * s_in + pix_index(x, y, w) * 3;
    const float u = v[0] * sx, t = v[1] * sy, l = luma(img + n * s_img + pix_index(x, y, w) * 3);
    o[0] = u;
    o[1] = t;
    o[2] = l;
    if (plane) {
        const __half2 a = __floats2half2_rn(u, t), b = __floats2half2_rn(l, 0.0f);
        plane[(static_cast<int64_t>(n) * h + y) * w + x] =
            make_uint4(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b), 0u, 0u);
    }
}

// ---- training: 3x3 convolutions on register tiles ---------------------------------------
// Inner activations and their gradients are planes ([image][channel][y][x]);
// the input (NHWC, 3 channels) is read as the caller holds it.
//
// The convolutions (forward, and backward for the data with the taps
// flipped) and the weight gradients are FP32 contractions of 9 CI CO products
// a pixel, bound by the FMA issue rate as long as shared memory keeps up.
// One thread per pixel with the weights read one by one from shared memory
// (one 4-byte broadcast load per FMA) ran the 32 -> 32 layer of a 32 x 64 x
// 64 batch in 274 us forward and 369 us backward; weight gradients with one
// block per (output, tap), which re-read the whole activation with a stride
// for each of the 288 blocks, took 919 us.  The layer's 1.2 G FMAs are 30 us
// at 152 x 128 lanes; now 70 forward, 68 backward, 72 for the weights.

__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
        "l"(src), "r"(valid ? 4 : 0)
        : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ bool finite_f(float v) { return fabsf(v) <= 3.402823466e38f; }

constexpr int kTileW = 32;   // pixels of a tile row
constexpr int kPitch = 36;   // its shared-memory pitch: 34 with the halo; 4 mod 32 keeps 16-byte reads of
                             // 4 groups x 8 rows free of bank conflicts

enum ConvMode { kConvRelu, kConvLoss, kConvBwd };

// The convolution of one 32 x 8 pixel tile.  A thread keeps PX adjacent pixels
// x OCT output channels; its weight reads are broadcasts.  Every sum runs over
// the taps in order with the channels of a tap inside, as the per-pixel loops
// it replaces had it, so activations and ReLU signs keep their bits; all
// channels of the tile and all weights are therefore in shared memory at once (93
// KB for 32 channels, two blocks an SM).  The pixels' window at a horizontal
// tap is 8 of 10 values: two 16-byte words and at most one value more, rows on a
// pitch that keeps them free of bank conflicts; weights in the parameters' own
// layout, read four channels (forward) or four outputs (backward) at a time.
// Per tap and four channels 8 x 8 registers take 8 + 11 reads for 256 FMAs.
constexpr int kConvPitch = 44;  // columns x0 - 4 ... x0 + 39: x0 on a 16-byte boundary; 12 mod 32

template <int CI, int CO, int OCT>
struct ConvShape {
    static constexpr int OG = CO / OCT;             // channel groups
    static constexpr int rows = 8;
    static constexpr int PX = 32 * rows * OG / 128;  // pixels a thread
    static constexpr int kG = kTileW / PX;          // threads of a tile row
    static constexpr int plane = (rows + 2) * kConvPitch;
    static constexpr int weights = CI * 9 * CO;
    static constexpr int smem = (CI * plane + weights) * 4;
    static_assert((PX == 8 || PX == 2) && weights % 4 == 0 && (CI * plane) % 4 == 0, "tile");
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
        "l"(src), "r"(valid ? 16 : 0)
        : "memory");
}

// v[i] = p[kx + i], p four bytes below a 16-byte boundary
template <int PX>
__device__ __forceinline__ void conv_window(const float* p, int kx, float (&v)[PX])
{
    if constexpr (PX == 8) {
        const float4 a = *reinterpret_cast<const float4*>(p + 1), b = *reinterpret_cast<const float4*>(p + 5);
        const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        const float e = kx == 0 ? p[0] : kx == 2 ? p[9] : 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int j = i + kx - 1;
            v[i] = j < 0 || j > 7 ? e : w[j & 7];
        }
    } else {
#pragma unroll
        for (int i = 0; i < PX; ++i)
            v[i] = p[kx + i];
    }
}

// Output (thread's pixel i, channel oc) of conv3x3_kernel again, with the taps
// outside the image left out rather than multiplied with the zeros that the tile
// holds there: w * 0 is not 0 for a weight that is not finite.  xr: the tile at
// the thread's first pixel's window; the sum in the kernel's order.
template <int CI, int CO, int OCT, int kMode>
__device__ __noinline__ float conv_inside(const float* xr, const float* sw, float b, int oc, int i, int py, int px,
    int H, int W)
{
    using S = ConvShape<CI, CO, OCT>;
    constexpr bool kBwd = kMode == kConvBwd;
    float acc = b;
    for (int t = 0; t < 9; ++t) {
        const int dy = kBwd ? 2 - t / 3 : t / 3, dx = kBwd ? 2 - t % 3 : t % 3;
        const int yy = py + dy - 1, xx = px + i + dx - 1;
        if (yy < 0 || yy >= H || xx < 0 || xx >= W)
            continue;
        for (int c = 0; c < CI; ++c)
            acc = __fmaf_rn(kBwd ? sw[(c * 9 + t) * CO + oc] : sw[(oc * 9 + t) * CI + c],
                xr[c * S::plane + dy * kConvPitch + i + dx], acc);
    }
    return acc;
}

// x: planes (kInter: interleaved CI-channel pixels).  kConvRelu: y = ReLU(conv
// + bias).  kConvLoss (the last layer): the L1 sum of base + r against the
// target and the loss's gradient dr = sign / pixels as planes in y.  kConvBwd: x is
// dz of the layer's CI outputs, y = dz of its CO inputs where a_prev > 0.
// nonfinite: set when a value the weight gradients will multiply (the input,
// an activation or a dz) is not finite.
template <int CI, int CO, int OCT, int kMode, bool kInter>
__global__ void __launch_bounds__(128, 2) conv3x3_kernel(const float* __restrict__ x, const float* __restrict__ wts,
    const float* __restrict__ bias, const float* __restrict__ a_prev, float* __restrict__ y, int H, int W, int tiles_x,
    const float* __restrict__ input, const float* __restrict__ target, double* __restrict__ loss, float inv,
    int* __restrict__ nonfinite)
{
    using S = ConvShape<CI, CO, OCT>;
    constexpr int PX = S::PX;
    extern __shared__ __align__(16) float sm[];
    float* sw = sm + CI * S::plane;
    const int tid = threadIdx.x, lane = tid & 31;
    const int og = tid / (8 * S::kG), g = tid % S::kG, r = tid / S::kG % 8;  // channel group, pixel group, tile row
    const int x0 = (blockIdx.x % tiles_x) * kTileW, y0 = (blockIdx.x / tiles_x) * S::rows;
    const int64_t HW = static_cast<int64_t>(H) * W;
    const int n = blockIdx.y;
    const float* xn = x + static_cast<int64_t>(n) * HW * CI;

    for (int i = tid; i < S::weights / 4; i += 128)
        cp_async16(sw + 4 * i, wts + 4 * i, true);
    if (!kInter && (W & 3) == 0) {  // planes and rows start on the 16-byte grid: a vector is in the image or not
        for (int i = tid; i < CI * (S::rows + 2) * 8; i += 128) {
            const int q = i & 7, row = i / 8 % (S::rows + 2), c = i / (8 * (S::rows + 2));
            const int gy = y0 - 1 + row, gx = x0 + 4 * q;
            const bool ok = gy >= 0 && gy < H && gx < W;
            cp_async16(sm + c * S::plane + row * kConvPitch + 4 + 4 * q,
                xn + c * HW + (ok ? static_cast<int64_t>(gy) * W + gx : 0), ok);
        }
        for (int i = tid; i < CI * (S::rows + 2) * 2; i += 128) {
            const int q = i & 1, row = i / 2 % (S::rows + 2), c = i / (2 * (S::rows + 2));
            const int gy = y0 - 1 + row, gx = x0 + (q ? 32 : -1);
            const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
            cp_async4(sm + c * S::plane + row * kConvPitch + (q ? 36 : 3),
                xn + c * HW + (ok ? static_cast<int64_t>(gy) * W + gx : 0), ok);
        }
    } else {
        for (int i = tid; i < CI * (S::rows + 2) * 34; i += 128) {
            const int col = i % 34, row = i / 34 % (S::rows + 2), c = i / (34 * (S::rows + 2));
            const int gy = y0 - 1 + row, gx = x0 - 1 + col;
            const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
            const int64_t p = ok ? static_cast<int64_t>(gy) * W + gx : 0;
            cp_async4(sm + c * S::plane + row * kConvPitch + 3 + col, xn + (kInter ? p * CI + c : c * HW + p), ok);
        }
    }
    cp_async_commit();

    float acc[PX][OCT];
#pragma unroll
    for (int o = 0; o < OCT; ++o) {
        const float b = kMode == kConvBwd ? 0.0f : bias[og * OCT + o];
#pragma unroll
        for (int i = 0; i < PX; ++i)
            acc[i][o] = b;
    }
    bool bad = false;
    cp_async_wait<0>();
    __syncthreads();
    if (kInter && kMode == kConvRelu)  // the layer's own input feeds its weight gradient
        for (int i = tid; i < CI * (S::rows + 2) * 34; i += 128) {
            const int col = i % 34, row = i / 34 % (S::rows + 2), c = i / (34 * (S::rows + 2));
            bad = bad || !finite_f(sm[c * S::plane + row * kConvPitch + 3 + col]);
        }
    // tap (ky, kx) of the layer; backward reads the output pixel whose tap it was
#pragma unroll 1
    for (int ky = 0; ky < 3; ++ky) {
        const float* xr = sm + (r + (kMode == kConvBwd ? 2 - ky : ky)) * kConvPitch + 3 + PX * g;
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) {
            constexpr int kC = CI % 4 == 0 ? 4 : 1;
            const int t = ky * 3 + kx, dx = kMode == kConvBwd ? 2 - kx : kx;
#pragma unroll 1
            for (int c0 = 0; c0 < CI; c0 += kC) {
                float w[kC][OCT];
                if constexpr (kMode == kConvBwd) {  // [in = its outputs][tap][out]
#pragma unroll
                    for (int c = 0; c < kC; ++c)
#pragma unroll
                        for (int q = 0; q < OCT / 4; ++q) {
                            const float4 f =
                                *reinterpret_cast<const float4*>(sw + ((c0 + c) * 9 + t) * CO + og * OCT + 4 * q);
                            w[c][4 * q] = f.x;
                            w[c][4 * q + 1] = f.y;
                            w[c][4 * q + 2] = f.z;
                            w[c][4 * q + 3] = f.w;
                        }
                } else {  // [out][tap][in]
#pragma unroll
                    for (int o = 0; o < OCT; ++o) {
                        const float* q = sw + ((og * OCT + o) * 9 + t) * CI + c0;
                        if constexpr (kC == 4) {
                            const float4 f = *reinterpret_cast<const float4*>(q);
                            w[0][o] = f.x;
                            w[1][o] = f.y;
                            w[2][o] = f.z;
                            w[3][o] = f.w;
                        } else {
                            w[0][o] = q[0];
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < kC; ++c) {
                    float v[PX];
                    conv_window<PX>(xr + (c0 + c) * S::plane, dx, v);
#pragma unroll
                    for (int i = 0; i < PX; ++i)
#pragma unroll
                        for (int o = 0; o < OCT; ++o)
                            acc[i][o] = __fmaf_rn(w[c][o], v[i], acc[i][o]);
                }
            }
        }
    }

    const int py = y0 + r, px = x0 + PX * g;
    const bool row_in = py < H;
    const int64_t p = static_cast<int64_t>(py) * W + px;
    // sums of pixels at the image's edge that are not finite may have come from a tap outside it
    bool redo = false;
    const float* const x_thread = sm + r * kConvPitch + 3 + PX * g;
    if (py == 0 || py == H - 1 || px == 0 || px + PX >= W) {
#pragma unroll
        for (int i = 0; i < PX; ++i)
#pragma unroll
            for (int o = 0; o < OCT; ++o)
                redo = redo || !finite_f(acc[i][o]);
    }
    if constexpr (kMode == kConvLoss) {
        if (redo)
#pragma unroll
            for (int i = 0; i < PX; ++i)
#pragma unroll
                for (int o = 0; o < OCT; ++o)
                    acc[i][o] = conv_inside<CI, CO, OCT, kMode>(x_thread, sw, bias[o], o, i, py, px, H, W);
        float l = 0.0f;
#pragma unroll
        for (int i = 0; i < PX; ++i) {
            if (!row_in || px + i >= W)
                continue;
            const int64_t q = n * HW + p + i;
#pragma unroll
            for (int o = 0; o < OCT; ++o) {
                const float d = input[q * 3 + o] + acc[i][o] - target[q * 2 + o];
                l += fabsf(d);
                y[(static_cast<int64_t>(n) * CO + o) * HW + p + i] = d > 0.0f ? inv : (d < 0.0f ? -inv : 0.0f);
            }
        }
        for (int o = 16; o > 0; o >>= 1)
            l += __shfl_xor_sync(0xffffffffu, l, o);
        // One add a block, in 64 bits: 512 additions in a row in 32 were up to 8 units
        // of 2^-24 off (32 x 64 x 64 pixels), in the order in which the blocks end.
        __syncthreads();
        if (lane == 0)
            sm[tid >> 5] = l;
        __syncthreads();
        if (tid == 0)
            atomicAdd(loss, static_cast<double>((sm[0] + sm[1]) + (sm[2] + sm[3])));
    } else {
        const bool vec = (W & 3) == 0;  // planes and rows then start on the 16-byte grid
#pragma unroll
        for (int o = 0; o < OCT; ++o) {
            const int64_t q = (static_cast<int64_t>(n) * CO + og * OCT + o) * HW + p;
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const bool in = row_in && px + i < W;
                v[i] = acc[i][o];
                if (kMode == kConvRelu) {
                    v[i] = fmaxf(v[i], 0.0f);
                    bad = bad || (in && !finite_f(v[i]));
                } else {
                    v[i] = in && a_prev[q + i] > 0.0f ? v[i] : 0.0f;
                    bad = bad || !finite_f(v[i]);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (vec && row_in && px + 4 * h + 3 < W) {
                    *reinterpret_cast<float4*>(y + q + 4 * h) =
                        make_float4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
                } else {
#pragma unroll
                    for (int i = 4 * h; i < 4 * h + 4; ++i)
                        if (row_in && px + i < W)
                            y[q + i] = v[i];
                }
            }
        }
        if (redo && row_in) {  // (the thread's own stores, written over)
#pragma unroll 1
            for (int k = 0; k < PX * OCT; ++k) {
                const int i = k % PX, oc = og * OCT + k / PX;
                if (px + i >= W)
                    continue;
                const int64_t q = (static_cast<int64_t>(n) * CO + oc) * HW + p + i;
                float v = conv_inside<CI, CO, OCT, kMode>(x_thread, sw, kMode == kConvBwd ? 0.0f : bias[oc], oc, i, py,
                    px, H, W);
                v = kMode == kConvRelu ? fmaxf(v, 0.0f) : a_prev[q] > 0.0f ? v : 0.0f;
                bad = bad || !finite_f(v);
                y[q] = v;
            }
        }
        if (bad)
            atomicOr(nonfinite, 1);
    }
}

// ---- weight gradients ---------------------------------------------------------------
// dw[o][t][c] += sum over pixels of dz[o] * x[tap t][c]; db[o] += sum dz[o].
// Blocks walk 32 x 2 pixel tiles, two cp.async buffers, and add their sums to
// the gradient at the end, and every kWgFlush tiles.  The gradient is kept in
// copies, one for 16 blocks and 32 at most, which the update sums: all 608 blocks
// on one sum were 608 additions in a row and five times as far from the float64 sum
// (32 x 64 x 64 pixels of equal dz: 5.9 units of 2^-24 in the root mean square, now
// 1.1; the per-pixel kernels 1.7), and slower (a step 590 us, now 560); a thread's
// own sum is at most 2,048 products long, whatever the batch.  A pixel with dz = 0 adds nothing, whatever x
// holds there, nor does a tap outside the image, whatever dz is (kSafe, taken
// when some x or dz is not finite; else the product with 0 is 0 anyway).
constexpr int kGradCopies = 32;
constexpr int kGradPitch = (kParams + 31) / 32 * 32;  // of a copy, in floats
constexpr int kWgFlush = 32;
constexpr int kWgRows = 2;
constexpr int kWgPx = kTileW * kWgRows;
constexpr int kWgPlane = 148;  // x plane: 4 rows x 36, + 4: 20 mod 32, 16-byte reads across channels conflict-free

// CI = 32: a lane is an input channel with OGT outputs x 9 taps in registers,
// a warp one group of outputs (its dz reads are broadcasts); with fewer than
// four groups the warps split the tile's columns.  Per 4 pixels a thread
// reads 3 + OGT 16-byte words for 36 OGT FMAs.
template <int CO, int OGT>
struct WgShape {
    static constexpr int NOG = CO / OGT, KS = 4 / NOG;
    static constexpr int dzp = kWgPx;  // dz pitch
    static constexpr int buf = 32 * kWgPlane + CO * dzp;
    static constexpr int smem = 2 * buf * 4;
};

// inside: the tap lies in the image (looked at where safe only)
__device__ __forceinline__ float wg_add(bool safe, float g, float v, float acc, bool inside)
{
    return safe && (g == 0.0f || !inside) ? acc : __fmaf_rn(g, v, acc);
}

// bit i of n: the coordinate first + i lies in [0, size)
__device__ __forceinline__ unsigned inside_bits(int first, int n, int size)
{
    unsigned m = 0;
    for (int i = 0; i < n; ++i)
        m |= first + i >= 0 && first + i < size ? 1u << i : 0u;
    return m;
}

template <int CO, int OGT, bool kSafe>
__device__ __forceinline__ void wg_tile(const float* sx, const float* sz, int ks, int lane, float (&acc)[OGT][9])
{
    using S = WgShape<CO, OGT>;
    constexpr int J = 8 / S::KS;  // 4-pixel groups of a row this warp takes
#pragma unroll 1
    for (int row = 0; row < kWgRows; ++row) {
        const float* xr = sx + lane * kWgPlane + row * kPitch + 4 * J * ks;
        const float* zr = sz + row * kTileW + 4 * J * ks;
        float4 cur[3];
#pragma unroll
        for (int ky = 0; ky < 3; ++ky)
            cur[ky] = *reinterpret_cast<const float4*>(xr + ky * kPitch);
#pragma unroll 2
        for (int j = 0; j < J; ++j) {
            float v[3][6];
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                const float4 nx = *reinterpret_cast<const float4*>(xr + ky * kPitch + 4 * j + 4);
                v[ky][0] = cur[ky].x;
                v[ky][1] = cur[ky].y;
                v[ky][2] = cur[ky].z;
                v[ky][3] = cur[ky].w;
                v[ky][4] = nx.x;
                v[ky][5] = nx.y;
                cur[ky] = nx;
            }
#pragma unroll
            for (int o = 0; o < OGT; ++o) {
                const float4 z = *reinterpret_cast<const float4*>(zr + o * S::dzp + 4 * j);
                const float gz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int t = 0; t < 9; ++t) {
                        const float a = v[t / 3][i + t % 3];
                        acc[o][t] = wg_add(kSafe, gz[i], a, acc[o][t], a == a);
                    }
            }
        }
    }
}

template <int CO, int OGT>
__global__ void __launch_bounds__(128, 4) wgrad_kernel(const float* __restrict__ x, const float* __restrict__ dz,
    float* __restrict__ dw, float* __restrict__ db, int H, int W, int tiles_x, int tiles, int N,
    int copies, const int* __restrict__ nonfinite)
{
    using S = WgShape<CO, OGT>;
    extern __shared__ __align__(16) float sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int og = warp % S::NOG, ks = warp / S::NOG;
    const int64_t HW = static_cast<int64_t>(H) * W;
    const int total = tiles * N;

    auto stage = [&](int tile, float* b) {
        const int n = tile / tiles, rem = tile % tiles;
        const int x0 = (rem % tiles_x) * kTileW, y0 = (rem / tiles_x) * kWgRows;
        const float* xn = x + static_cast<int64_t>(n) * HW * 32;
        const float* zn = dz + static_cast<int64_t>(n) * HW * CO;
        for (int i = tid; i < 32 * 4 * 34; i += 128) {
            const int c = i / (4 * 34), q = i % (4 * 34), row = q / 34, col = q % 34;
            const int gy = y0 - 1 + row, gx = x0 - 1 + col;
            const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
            cp_async4(b + c * kWgPlane + row * kPitch + col,
                ok ? xn + c * HW + static_cast<int64_t>(gy) * W + gx : xn, ok);
        }
        float* sz = b + 32 * kWgPlane;
        for (int i = tid; i < CO * kWgPx; i += 128) {
            const int o = i / kWgPx, q = i % kWgPx, gy = y0 + q / kTileW, gx = x0 + q % kTileW;
            const bool ok = gy < H && gx < W;
            cp_async4(sz + o * S::dzp + q, ok ? zn + o * HW + static_cast<int64_t>(gy) * W + gx : zn, ok);
        }
    };

    dw += blockIdx.x % copies * kGradPitch;
    db += blockIdx.x % copies * kGradPitch;
    const bool safe = *nonfinite != 0;
    int tile = blockIdx.x, k = 0;
    if (tile < total)
        stage(tile, sm);
    cp_async_commit();
    while (tile < total) {
        float acc[OGT][9], bsum[OGT];
#pragma unroll
        for (int o = 0; o < OGT; ++o) {
            bsum[o] = 0.0f;
#pragma unroll
            for (int t = 0; t < 9; ++t)
                acc[o][t] = 0.0f;
        }
        for (int m = 0; m < kWgFlush && tile < total; ++m, tile += gridDim.x, ++k) {
            const float* b = sm + (k & 1) * S::buf;
            if (tile + static_cast<int>(gridDim.x) < total)
                stage(tile + gridDim.x, sm + ((k + 1) & 1) * S::buf);
            cp_async_commit();
            cp_async_wait<1>();
            __syncthreads();
            const float* sz = b + 32 * kWgPlane + og * OGT * S::dzp;
            if (safe) {
                // x is a ReLU's output, never NaN: NaN marks the tile's places outside the image
                const int x0 = (tile % tiles % tiles_x) * kTileW, y0 = (tile % tiles / tiles_x) * kWgRows;
                for (int i = tid; i < 32 * 4 * 34; i += 128) {
                    const int c = i / (4 * 34), q = i % (4 * 34), gy = y0 - 1 + q / 34, gx = x0 - 1 + q % 34;
                    if (gy < 0 || gy >= H || gx < 0 || gx >= W)
                        sm[(k & 1) * S::buf + c * kWgPlane + q / 34 * kPitch + q % 34] = __int_as_float(0x7fffffff);
                }
                __syncthreads();
                wg_tile<CO, OGT, true>(b, sz, ks, lane, acc);
            } else {
                wg_tile<CO, OGT, false>(b, sz, ks, lane, acc);
            }
            if (ks == 0)
#pragma unroll
                for (int o = 0; o < OGT; ++o)
                    bsum[o] += sz[o * S::dzp + lane] + sz[o * S::dzp + 32 + lane];
            __syncthreads();
        }
#pragma unroll
        for (int o = 0; o < OGT; ++o) {
            const int oc = og * OGT + o;
#pragma unroll
            for (int t = 0; t < 9; ++t)
                atomicAdd(&dw[(oc * 9 + t) * 32 + lane], acc[o][t]);  // a warp's 32 channels: one 128-byte line
            if (ks == 0) {
                float s = bsum[o];
                for (int d = 16; d > 0; d >>= 1)
                    s += __shfl_xor_sync(0xffffffffu, s, d);
                if (lane == 0)
                    atomicAdd(&db[oc], s);
            }
        }
    }
}

// The first layer (3 -> 32, interleaved input): a lane is an output with 3 x 9
// sums, the warps split each tile's columns.
constexpr int kWg1Dz = kWgPx + 4;  // dz pitch: 4 mod 32, 16-byte reads across outputs conflict-free
constexpr int kWg1X = 3 * 4 * kPitch;
constexpr int kWg1Buf = 32 * kWg1Dz + kWg1X;

__global__ void __launch_bounds__(128) wgrad_first_kernel(const float* __restrict__ x, const float* __restrict__ dz,
    float* __restrict__ dw, float* __restrict__ db, int H, int W, int tiles_x, int tiles, int N,
    int copies, const int* __restrict__ nonfinite)
{
    __shared__ __align__(16) float sm[2 * kWg1Buf];
    __shared__ float red[32 * 28];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t HW = static_cast<int64_t>(H) * W;
    const int total = tiles * N;
    for (int i = tid; i < 32 * 28; i += 128)
        red[i] = 0.0f;

    auto stage = [&](int tile, float* b) {
        const int n = tile / tiles, rem = tile % tiles;
        const int x0 = (rem % tiles_x) * kTileW, y0 = (rem / tiles_x) * kWgRows;
        const float* xn = x + static_cast<int64_t>(n) * HW * 3;
        const float* zn = dz + static_cast<int64_t>(n) * HW * 32;
        for (int i = tid; i < 32 * kWgPx; i += 128) {
            const int o = i / kWgPx, q = i % kWgPx, gy = y0 + q / kTileW, gx = x0 + q % kTileW;
            const bool ok = gy < H && gx < W;
            cp_async4(b + o * kWg1Dz + q, ok ? zn + o * HW + static_cast<int64_t>(gy) * W + gx : zn, ok);
        }
        float* sx = b + 32 * kWg1Dz;
        for (int i = tid; i < 3 * 4 * 34; i += 128) {
            const int c = i % 3, q = i / 3, row = q / 34, col = q % 34;
            const int gy = y0 - 1 + row, gx = x0 - 1 + col;
            const bool ok = gy >= 0 && gy < H && gx >= 0 && gx < W;
            cp_async4(sx + (c * 4 + row) * kPitch + col, ok ? xn + (static_cast<int64_t>(gy) * W + gx) * 3 + c : xn, ok);
        }
    };

    dw += blockIdx.x % copies * kGradPitch;
    db += blockIdx.x % copies * kGradPitch;
    float acc[27], bsum8 = 0.0f, bsum = 0.0f;  // dz in short chains: of a tile, of 8 tiles, of the eights
#pragma unroll
    for (int t = 0; t < 27; ++t)
        acc[t] = 0.0f;
    const bool safe = *nonfinite != 0;
    int tile = blockIdx.x, k = 0;
    if (tile < total)
        stage(tile, sm);
    cp_async_commit();
    for (; tile < total; tile += gridDim.x, ++k) {
        const float* b = sm + (k & 1) * kWg1Buf;
        if (tile + static_cast<int>(gridDim.x) < total)
            stage(tile + gridDim.x, sm + ((k + 1) & 1) * kWg1Buf);
        cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        const float* sx = b + 32 * kWg1Dz;
        const int x0 = (tile % tiles % tiles_x) * kTileW, y0 = (tile % tiles / tiles_x) * kWgRows;
        auto add_tile = [&](auto safe_tile) {
            constexpr bool kSafe = decltype(safe_tile)::value;
            float tsum = 0.0f;
            const unsigned ym = kSafe ? inside_bits(y0 - 1, kWgRows + 2, H) : 0;
#pragma unroll 1
            for (int q = 2 * warp; q < 2 * warp + 2; ++q) {  // this warp's 4-pixel groups of each row
                const unsigned xm = kSafe ? inside_bits(x0 + 4 * q - 1, 6, W) : 0;
#pragma unroll
                for (int row = 0; row < kWgRows; ++row) {
                    const float4 z = *reinterpret_cast<const float4*>(b + lane * kWg1Dz + row * kTileW + 4 * q);
                    const float gz[4] = {z.x, z.y, z.z, z.w};
                    tsum += (z.x + z.y) + (z.z + z.w);
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int ky = 0; ky < 3; ++ky) {
                            const float* xr = sx + (c * 4 + row + ky) * kPitch + 4 * q;
                            const float4 v0 = *reinterpret_cast<const float4*>(xr);
                            const float2 v1 = *reinterpret_cast<const float2*>(xr + 4);
                            const float v[6] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y};
#pragma unroll
                            for (int i = 0; i < 4; ++i)
#pragma unroll
                                for (int kx = 0; kx < 3; ++kx) {
                                    float& a = acc[(ky * 3 + kx) * 3 + c];
                                    a = wg_add(kSafe, gz[i], v[i + kx], a,
                                        (xm >> (i + kx) & ym >> (row + ky) & 1u) != 0);
                                }
                        }
                }
            }
            bsum8 += tsum;
        };
        if (safe)
            add_tile(std::true_type{});
        else
            add_tile(std::false_type{});
        if ((k & 7) == 7) {
            bsum += bsum8;
            bsum8 = 0.0f;
        }
        __syncthreads();
        if ((k + 1) % kWgFlush != 0 && tile + static_cast<int>(gridDim.x) < total)
            continue;
        // the four warps' sums, then one coalesced addition per weight and block
#pragma unroll
        for (int t = 0; t < 27; ++t) {
            atomicAdd(&red[lane * 27 + t], acc[t]);
            acc[t] = 0.0f;
        }
        atomicAdd(&red[32 * 27 + lane], bsum + bsum8);
        bsum = bsum8 = 0.0f;
        __syncthreads();
        for (int i = tid; i < 32 * 28; i += 128) {
            atomicAdd(i < 32 * 27 ? &dw[i] : &db[i - 32 * 27], red[i]);
            red[i] = 0.0f;
        }
        __syncthreads();
    }
}

// The update; also the loss, from its sum over the batch's pixels.
__global__ void adam_kernel(float* __restrict__ prm, const float* __restrict__ g, float* __restrict__ m,
    float* __restrict__ v, int n, int copies, float lr, float b1, float b2, float c1, float c2, float eps,
    const double* __restrict__ sum, double px, float* __restrict__ loss)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0)
        *loss = static_cast<float>(*sum / px);
    if (i >= n)
        return;
    float part[4] = {};  // (copies in four chains: shorter sums, loads ahead)
    for (int c = 0; c < copies; c += 4)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            part[k] += c + k < copies ? g[(c + k) * kGradPitch + i] : 0.0f;
    const float gi = (part[0] + part[1]) + (part[2] + part[3]);
    m[i] = b1 * m[i] + (1.0f - b1) * gi;
    v[i] = b2 * v[i] + (1.0f - b2) * gi * gi;
    prm[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
}

uint64_t splitmix(uint64_t* s)
{
    uint64_t z = (*s += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// Dynamic shared memory of the training kernels, opted into once per device.
cudaError_t train_prepare_device(int* sms)
{
    static PerDevice<int> device;
    return device.get(
        [](int* count) {
            constexpr auto kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
            cudaError_t e = cudaSuccess;
            auto set = [&](auto* k, int smem) {
                if (e == cudaSuccess)
                    e = cudaFuncSetAttribute(k, kAttr, smem);
            };
            set(conv3x3_kernel<3, 32, 8, kConvRelu, true>, ConvShape<3, 32, 8>::smem);
            set(conv3x3_kernel<32, 32, 8, kConvRelu, false>, ConvShape<32, 32, 8>::smem);
            set(conv3x3_kernel<32, 2, 2, kConvLoss, false>, ConvShape<32, 2, 2>::smem);
            set(conv3x3_kernel<2, 32, 8, kConvBwd, false>, ConvShape<2, 32, 8>::smem);
            set(conv3x3_kernel<32, 32, 8, kConvBwd, false>, ConvShape<32, 32, 8>::smem);
            set(wgrad_kernel<2, 2>, WgShape<2, 2>::smem);
            set(wgrad_kernel<32, 8>, WgShape<32, 8>::smem);
            int dev = 0;
            if (e == cudaSuccess)
                e = cudaGetDevice(&dev);
            return e != cudaSuccess ? e : cudaDeviceGetAttribute(count, cudaDevAttrMultiProcessorCount, dev);
        },
        sms);
}

template <int CI, int CO, int OCT, int kMode, bool kInter>
void launch_conv(const float* x, const float* prm, int layer, const float* a_prev, float* y, int N, int H, int W,
    int* nonfinite, cudaStream_t st, const float* input = nullptr, const float* target = nullptr,
    double* loss = nullptr, float inv = 0.0f)
{
    using S = ConvShape<CI, CO, OCT>;
    const int tx = (W + kTileW - 1) / kTileW, ty = (H + S::rows - 1) / S::rows;
    conv3x3_kernel<CI, CO, OCT, kMode, kInter><<<dim3(static_cast<unsigned>(tx) * ty, N), 128, S::smem, st>>>(x,
        prm + kUpLayers[layer].w_off, prm + kUpLayers[layer].b_off, a_prev, y, H, W, tx, input, target, loss, inv,
        nonfinite);
}

}  // namespace

int upsampler_param_count() { return kParams; }
size_t upsampler_grad_floats() { return static_cast<size_t>(kGradCopies) * kGradPitch; }

void upsampler_init_params(float* host, uint64_t seed)
{
    uint64_t s = seed;
    for (const UpLayer& l : kUpLayers) {
        const float bound = std::sqrt(6.0f / static_cast<float>(9 * l.ci));  // He-uniform
        for (int i = 0; i < l.co * 9 * l.ci; ++i)
            host[l.w_off + i] = (static_cast<float>(splitmix(&s) >> 40) * (1.0f / 16777216.0f) * 2.0f - 1.0f) * bound;
        for (int i = 0; i < l.co; ++i)
            host[l.b_off + i] = 0.0f;
    }
    // the last layer starts near zero: the initial prediction is the base flow
    for (int i = 0; i < kUpLayers[3].co * 9 * kUpLayers[3].ci; ++i)
        host[kUpLayers[3].w_off + i] *= 0.01f;
}

cudaError_t launch_upsampler_prepare(const float* coarse, int cw, int ch, int cfc, const float* img, float* input, int w,
    int h, int N, int64_t s_coarse, int64_t s_img, int64_t s_in, cudaStream_t st, void* plane)
{
    const dim3 b(32, 8);
    const dim3 g((w + 31) / 32, (h + 7) / 8, N);
    prepare_kernel<<<g, b, 0, st>>>(coarse, cw, ch, cfc, img, input, w, h, s_coarse, s_img, s_in,
        static_cast<uint4*>(plane));
    return cudaGetLastError();
}

// One Adam step on a batch: forward, L1 loss, backward, update.  grad:
// upsampler_grad_floats floats; work: upsampler_train_work_floats; state (4 floats, 8-byte
// aligned): the loss, as an int the non-finite flag, as a double the loss's sum.
cudaError_t upsampler_train_step(float* prm, float* grad, float* m, float* v, int step, const float* input,
    const float* target, int N, int H, int W, float lr, float* work, float* state, cudaStream_t st)
{
    int sms = 0;
    cudaError_t e = train_prepare_device(&sms);
    if (e != cudaSuccess)
        return e;
    const int64_t px = static_cast<int64_t>(N) * H * W;
    float* a1 = work;
    float* a2 = a1 + px * 32;
    float* a3 = a2 + px * 32;
    float* dz3 = a3 + px * 32;
    float* dz2 = dz3 + px * 32;
    float* dz1 = dz2 + px * 32;
    float* dr = dz1 + px * 32;
    int* bad = reinterpret_cast<int*>(state + 1);
    double* sum = reinterpret_cast<double*>(state + 2);
    if ((e = cudaMemsetAsync(state, 0, 4 * sizeof(float), st)) != cudaSuccess)
        return e;
    launch_conv<3, 32, 8, kConvRelu, true>(input, prm, 0, nullptr, a1, N, H, W, bad, st);
    launch_conv<32, 32, 8, kConvRelu, false>(a1, prm, 1, nullptr, a2, N, H, W, bad, st);
    launch_conv<32, 32, 8, kConvRelu, false>(a2, prm, 2, nullptr, a3, N, H, W, bad, st);
    launch_conv<32, 2, 2, kConvLoss, false>(a3, prm, 3, nullptr, dr, N, H, W, bad, st, input, target, sum,
        1.0f / static_cast<float>(px));
    // weight gradients: resident blocks walk the tiles, so a block's sums are added once
    const int tx = (W + kTileW - 1) / kTileW, tiles = tx * ((H + kWgRows - 1) / kWgRows);
    const int wb = static_cast<int>(std::min<int64_t>(static_cast<int64_t>(tiles) * N, 4 * sms));
    const int copies = std::min((wb + 15) / 16, kGradCopies);
    if ((e = cudaMemsetAsync(grad, 0, static_cast<size_t>(copies) * kGradPitch * sizeof(float), st)) != cudaSuccess)
        return e;
    float* gw[4];
    float* gb[4];
    for (int l = 0; l < 4; ++l) {
        gw[l] = grad + kUpLayers[l].w_off;
        gb[l] = grad + kUpLayers[l].b_off;
    }
    wgrad_kernel<2, 2><<<wb, 128, WgShape<2, 2>::smem, st>>>(a3, dr, gw[3], gb[3], H, W, tx, tiles, N, copies, bad);
    launch_conv<2, 32, 8, kConvBwd, false>(dr, prm, 3, a3, dz3, N, H, W, bad, st);
    wgrad_kernel<32, 8><<<wb, 128, WgShape<32, 8>::smem, st>>>(a2, dz3, gw[2], gb[2], H, W, tx, tiles, N, copies, bad);
    launch_conv<32, 32, 8, kConvBwd, false>(dz3, prm, 2, a2, dz2, N, H, W, bad, st);
    wgrad_kernel<32, 8><<<wb, 128, WgShape<32, 8>::smem, st>>>(a1, dz2, gw[1], gb[1], H, W, tx, tiles, N, copies, bad);
    launch_conv<32, 32, 8, kConvBwd, false>(dz2, prm, 1, a1, dz1, N, H, W, bad, st);
    wgrad_first_kernel<<<wb, 128, 0, st>>>(input, dz1, gw[0], gb[0], H, W, tx, tiles, N, copies, bad);
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - std::pow(b1, static_cast<float>(step)), c2 = 1.0f - std::pow(b2, static_cast<float>(step));
    adam_kernel<<<(kParams + 255) / 256, 256, 0, st>>>(prm, grad, m, v, kParams, copies, lr, b1, b2, c1, c2, 1e-8f, sum,
        static_cast<double>(px), state);
    return cudaGetLastError();
}

size_t upsampler_train_work_floats(int N, int H, int W)
{
    const size_t px = static_cast<size_t>(N) * H * W;
    return px * (32 * 6 + 2);
}

}  // namespace vsc
