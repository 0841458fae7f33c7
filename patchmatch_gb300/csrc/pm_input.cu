// Input preparation on the GPU: the keyframe thumbnails the densifier reads
// (data/frame.cc:53-54,136-138: gray and mask resized to the densification
// size, colour thumbnail via set_rgb_thumb) and the FP16 image pyramid of the
// precision form.  All buffers are caller-owned device memory; work is
// enqueued on the context's stream.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pm_gb300.h"

namespace {

// All of these move a few bytes per pixel and are bound by HBM, once the
// accesses are wide: a thread that handles one byte leaves the memory system
// waiting for instructions.  The vector kernels take 16 pixels (or 8 outputs)
// per thread with 16-byte accesses; the scalar kernels remain for rows that do
// not start on a 16-byte boundary.  Measured at 3840x1920 (scalar -> vector):
// gray of 3 channels 23 -> 7.0 us (4.2 TB/s), u8 to FP16 22 -> 6.5 us, half
// size of 1 and 3 channels 13 -> 4.2 and 15 -> 7.3 us, the pyramid's second
// and third level 8.6 -> 5.4 and 4.6 -> 3.5 us.
constexpr int kVecThreads = 256;
bool aligned16(const void *p, size_t pitch) { return (((uintptr_t)p | pitch) & 15) == 0; }

// Colour -> gray with the BT.601 weights in 14-bit fixed point, rounded
// (0.299, 0.587, 0.114 -> 4899, 9617, 1868 of 16384; the published
// fixed-point form of COLOR_BGR2GRAY, util/image_converter.cc:8-39).
__device__ __forceinline__ uint32_t gray_of(uint32_t c0, uint32_t c1, uint32_t c2, int rgb) {
    const uint32_t b = rgb ? c2 : c0, r = rgb ? c0 : c2;
    return (r * 4899u + c1 * 9617u + b * 1868u + 8192u) >> 14;
}

__global__ void to_gray_kernel(const uint8_t *src, int W, int H, size_t pitch, int ch, int rgb, uint8_t *dst,
                               size_t dpitch) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    const uint8_t *p = src + (size_t)y * pitch + (size_t)x * ch;
    dst[(size_t)y * dpitch + x] = ch == 1 ? p[0] : (uint8_t)gray_of(p[0], p[1], p[2], rgb);
}

// One row of n pixels per blockIdx.y (a tightly packed image is one long
// row), 16 pixels per thread: CH 16-byte loads, one store.  Rows start on
// 16-byte boundaries; the last n % 16 pixels are done one by one.
template <int CH>
__global__ void __launch_bounds__(kVecThreads)
    to_gray_vec_kernel(const uint8_t *src, size_t n, size_t pitch, int rgb, uint8_t *dst, size_t dpitch) {
    const size_t x = ((size_t)blockIdx.x * kVecThreads + threadIdx.x) * 16;
    if (x >= n) return;
    const uint8_t *p = src + (size_t)blockIdx.y * pitch + x * CH;
    uint8_t *q = dst + (size_t)blockIdx.y * dpitch + x;
    if (x + 16 > n) {
        for (size_t k = 0; k < n - x; ++k)
            q[k] = CH == 1 ? p[k * CH] : (uint8_t)gray_of(p[k * CH], p[k * CH + 1], p[k * CH + 2], rgb);
        return;
    }
    uint32_t w[4 * CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p) + c);
        w[4 * c] = v.x;
        w[4 * c + 1] = v.y;
        w[4 * c + 2] = v.z;
        w[4 * c + 3] = v.w;
    }
    uint4 o;
    if (CH == 1) {
        o = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
        uint32_t g[4] = {0, 0, 0, 0};
        const auto byte = [&](int k) { return (w[k >> 2] >> (8 * (k & 3))) & 0xffu; };
#pragma unroll
        for (int k = 0; k < 16; ++k)
            g[k >> 2] |= gray_of(byte(k * CH), byte(k * CH + 1), byte(k * CH + 2), rgb) << (8 * (k & 3));
        o = make_uint4(g[0], g[1], g[2], g[3]);
    }
    *reinterpret_cast<uint4 *>(q) = o;
}

// Bilinear resize with pixel-centre alignment (source coordinate
// (x + 0.5) * sw / dw - 0.5, clamped to the image) and 11-bit fixed-point
// weights, rounded once at the end: the scheme of an 8-bit linear resize
// (cv::resize INTER_LINEAR).  ch interleaved channels; rx = sw / dw and
// ry = sh / dh as rounded FP32 quotients.
__global__ void resize_kernel(const uint8_t *src, int sw, int sh, size_t spitch, int ch, uint8_t *dst, int dw, int dh,
                              size_t dpitch, float rx, float ry) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= dw || y >= dh) return;
    // separately rounded operations (no contraction), as the restatement computes them
    const float fx0 = __fsub_rn(__fmul_rn(__fadd_rn((float)x, 0.5f), rx), 0.5f);
    const float fy0 = __fsub_rn(__fmul_rn(__fadd_rn((float)y, 0.5f), ry), 0.5f);
    int sx = (int)floorf(fx0), sy = (int)floorf(fy0);
    float fx = fx0 - (float)sx, fy = fy0 - (float)sy;
    if (sx < 0) { sx = 0; fx = 0.f; }
    if (sx >= sw - 1) { sx = sw - 1; fx = 0.f; }
    if (sy < 0) { sy = 0; fy = 0.f; }
    if (sy >= sh - 1) { sy = sh - 1; fy = 0.f; }
    const int cx1 = __float2int_rn(fx * 2048.f), cx0 = 2048 - cx1;
    const int cy1 = __float2int_rn(fy * 2048.f), cy0 = 2048 - cy1;
    const int sx1 = min(sx + 1, sw - 1), sy1 = min(sy + 1, sh - 1);
    const uint8_t *r0 = src + (size_t)sy * spitch, *r1 = src + (size_t)sy1 * spitch;
    for (int c = 0; c < ch; ++c) {
        const int a = r0[(size_t)sx * ch + c] * cx0 + r0[(size_t)sx1 * ch + c] * cx1;
        const int b = r1[(size_t)sx * ch + c] * cx0 + r1[(size_t)sx1 * ch + c] * cx1;
        const int v = (a * cy0 + b * cy1 + (1 << 21)) >> 22;
        dst[(size_t)y * dpitch + (size_t)x * ch + c] = (uint8_t)min(max(v, 0), 255);
    }
}

// The same at exactly half the size (sw = 2 dw, sh = 2 dh): the source
// coordinate of output x is 2 x + 1/2, so every weight is 1024 of 2048 and the
// rounding (1024^2 S + 2^21) >> 22 of the 2x2 sum S is (S + 2) >> 2.  A thread
// makes 8 outputs from 16 pixels of two rows (CH 16-byte loads each, 8 CH
// bytes out); rows start on 16- and 8-byte boundaries.
template <int CH>
__global__ void __launch_bounds__(kVecThreads)
    halve_vec_kernel(const uint8_t *src, size_t spitch, uint8_t *dst, int dw, size_t dpitch) {
    const int x = (blockIdx.x * kVecThreads + threadIdx.x) * 8;
    if (x >= dw) return;
    const uint8_t *r0 = src + (size_t)(2 * blockIdx.y) * spitch + (size_t)2 * x * CH, *r1 = r0 + spitch;
    uint8_t *q = dst + (size_t)blockIdx.y * dpitch + (size_t)x * CH;
    if (x + 8 > dw) {
        for (int k = 0; k < (dw - x) * CH; ++k) {
            const int o = (k / CH) * 2 * CH + k % CH;
            q[k] = (uint8_t)(((int)r0[o] + r0[o + CH] + r1[o] + r1[o + CH] + 2) >> 2);
        }
        return;
    }
    uint32_t a[4 * CH], b[4 * CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(r0) + c);
        const uint4 w = __ldg(reinterpret_cast<const uint4 *>(r1) + c);
        a[4 * c] = v.x; a[4 * c + 1] = v.y; a[4 * c + 2] = v.z; a[4 * c + 3] = v.w;
        b[4 * c] = w.x; b[4 * c + 1] = w.y; b[4 * c + 2] = w.z; b[4 * c + 3] = w.w;
    }
    uint32_t g[2 * CH] = {};
    const auto sum = [&](int k) {
        return ((a[k >> 2] >> (8 * (k & 3))) & 0xffu) + ((b[k >> 2] >> (8 * (k & 3))) & 0xffu);
    };
#pragma unroll
    for (int k = 0; k < 8 * CH; ++k) {
        const int o = (k / CH) * 2 * CH + k % CH;
        g[k >> 2] |= ((sum(o) + sum(o + CH) + 2u) >> 2) << (8 * (k & 3));
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) reinterpret_cast<uint2 *>(q)[c] = make_uint2(g[2 * c], g[2 * c + 1]);
}

// FP16 pyramid: level 0 = the image; level k+1 entry (y, x) = mean of the 2x2
// block (2y, 2x) of level k (rows/columns past the edge repeat the last one),
// summed in FP32 (exact for FP16 inputs) and rounded once to FP16.
__global__ void u8_to_half_kernel(const uint8_t *src, int W, int H, size_t pitch, __half *dst) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= W || y >= H) return;
    dst[(size_t)y * W + x] = __float2half_rn((float)src[(size_t)y * pitch + x]);
}

// Two bytes of w (k and k + 1) as FP16 values (whole numbers up to 255: exact).
__device__ __forceinline__ uint32_t half2_bytes(uint32_t w, int k) {
    const __half2 h = __halves2half2(__ushort2half_rn((unsigned short)((w >> (8 * k)) & 0xffu)),
                                     __ushort2half_rn((unsigned short)((w >> (8 * k + 8)) & 0xffu)));
    return *reinterpret_cast<const uint32_t *>(&h);
}

// Tightly packed or 16-byte aligned rows of n pixels, 16 pixels per thread.
__global__ void __launch_bounds__(kVecThreads)
    u8_to_half_vec_kernel(const uint8_t *src, size_t n, size_t pitch, __half *dst, size_t dpitch) {
    const size_t x = ((size_t)blockIdx.x * kVecThreads + threadIdx.x) * 16;
    if (x >= n) return;
    const uint8_t *p = src + (size_t)blockIdx.y * pitch + x;
    __half *q = dst + (size_t)blockIdx.y * dpitch + x;
    if (x + 16 > n) {
        for (size_t k = 0; k < n - x; ++k) q[k] = __float2half_rn((float)p[k]);
        return;
    }
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p));
    reinterpret_cast<uint4 *>(q)[0] =
        make_uint4(half2_bytes(v.x, 0), half2_bytes(v.x, 2), half2_bytes(v.y, 0), half2_bytes(v.y, 2));
    reinterpret_cast<uint4 *>(q)[1] =
        make_uint4(half2_bytes(v.z, 0), half2_bytes(v.z, 2), half2_bytes(v.w, 0), half2_bytes(v.w, 2));
}

// Mean of a 2x2 block, in the order ((a + b) + c) + d.
__device__ __forceinline__ __half mean4(float a, float b, float c, float d) {
    return __float2half_rn(0.25f * (a + b + c + d));
}

__global__ void half_down_kernel(const __half *src, int sw, int sh, __half *dst, int dw, int dh) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= dw || y >= dh) return;
    const int x0 = min(2 * x, sw - 1), x1 = min(2 * x + 1, sw - 1);
    const int y0 = min(2 * y, sh - 1), y1 = min(2 * y + 1, sh - 1);
    dst[(size_t)y * dw + x] =
        mean4(__half2float(src[(size_t)y0 * sw + x0]), __half2float(src[(size_t)y0 * sw + x1]),
              __half2float(src[(size_t)y1 * sw + x0]), __half2float(src[(size_t)y1 * sw + x1]));
}

// The same for rows of 8 n pixels on 16-byte boundaries: 4 outputs per thread
// from 8 pixels of two rows (the last row repeats at an odd height).
__global__ void __launch_bounds__(kVecThreads)
    half_down_vec_kernel(const __half *src, int sw, int sh, __half *dst, int dw) {
    const int x = (blockIdx.x * kVecThreads + threadIdx.x) * 4;
    if (x >= dw) return;
    const int y0 = 2 * blockIdx.y, y1 = min(y0 + 1, sh - 1);
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(src + (size_t)y0 * sw + 2 * x));
    const uint4 w = __ldg(reinterpret_cast<const uint4 *>(src + (size_t)y1 * sw + 2 * x));
    const auto pair = [](uint32_t u) { return __half22float2(*reinterpret_cast<const __half2 *>(&u)); };
    const auto one = [&](uint32_t p, uint32_t q) {
        const float2 t = pair(p), b = pair(q);
        return mean4(t.x, t.y, b.x, b.y);
    };
    const __half2 o0 = __halves2half2(one(v.x, w.x), one(v.y, w.y)), o1 = __halves2half2(one(v.z, w.z), one(v.w, w.w));
    *reinterpret_cast<uint2 *>(dst + (size_t)blockIdx.y * dw + x) =
        make_uint2(*reinterpret_cast<const uint32_t *>(&o0), *reinterpret_cast<const uint32_t *>(&o1));
}

// Blocks of kVecThreads threads for n items of `per` each along a row.
unsigned vec_blocks(size_t n, int per) {
    const size_t items = (size_t)kVecThreads * per;
    return (unsigned)((n + items - 1) / items);
}

constexpr int kMaxGridY = 65535;  // rows of a launch with one row per blockIdx.y

dim3 grid2(int W, int H) { return dim3((W + 31) / 32, (H + 7) / 8); }

}  // namespace

extern "C" {

void *pm_stream(const pm_ctx *ctx);

int pm_image_to_gray(pm_ctx *ctx, const void *src, int W, int H, size_t pitch, int channels, int order, void *gray,
                     size_t gray_pitch) {
    if (!ctx || !src || !gray || W < 1 || H < 1 || (channels != 1 && channels != 3 && channels != 4) ||
        (order != PM_ORDER_BGR && order != PM_ORDER_RGB) || pitch < (size_t)W * channels || gray_pitch < (size_t)W)
        return PM_EINVAL;
    cudaStream_t st = (cudaStream_t)pm_stream(ctx);
    const uint8_t *s = (const uint8_t *)src;
    uint8_t *d = (uint8_t *)gray;
    // a tightly packed image is one row
    const bool packed = pitch == (size_t)W * channels && gray_pitch == (size_t)W;
    const size_t n = packed ? (size_t)W * H : (size_t)W;
    const int rows = packed ? 1 : H;
    if (aligned16(s, rows > 1 ? pitch : 0) && aligned16(d, rows > 1 ? gray_pitch : 0) && rows <= kMaxGridY) {
        const dim3 grid(vec_blocks(n, 16), rows);
        const int rgb = order == PM_ORDER_RGB;
        if (channels == 1) to_gray_vec_kernel<1><<<grid, kVecThreads, 0, st>>>(s, n, pitch, rgb, d, gray_pitch);
        else if (channels == 3) to_gray_vec_kernel<3><<<grid, kVecThreads, 0, st>>>(s, n, pitch, rgb, d, gray_pitch);
        else to_gray_vec_kernel<4><<<grid, kVecThreads, 0, st>>>(s, n, pitch, rgb, d, gray_pitch);
    } else {
        to_gray_kernel<<<grid2(W, H), dim3(32, 8), 0, st>>>(s, W, H, pitch, channels, order == PM_ORDER_RGB, d,
                                                            gray_pitch);
    }
    return cudaGetLastError() == cudaSuccess ? PM_OK : PM_ECUDA;
}

int pm_image_resize(pm_ctx *ctx, const void *src, int sw, int sh, size_t spitch, int channels, void *dst, int dw,
                    int dh, size_t dpitch) {
    if (!ctx || !src || !dst || sw < 1 || sh < 1 || dw < 1 || dh < 1 || channels < 1 || channels > 4 ||
        spitch < (size_t)sw * channels || dpitch < (size_t)dw * channels)
        return PM_EINVAL;
    cudaStream_t st = (cudaStream_t)pm_stream(ctx);
    const uint8_t *s = (const uint8_t *)src;
    uint8_t *d = (uint8_t *)dst;
    // (2 x + 1/2 is exact in FP32 up to 2^22 outputs)
    if (sw == 2 * (int64_t)dw && sh == 2 * (int64_t)dh && dw <= (1 << 21) && aligned16(s, spitch) &&
        (((uintptr_t)d | dpitch) & 7) == 0 && dh <= kMaxGridY) {
        const dim3 grid(vec_blocks(dw, 8), dh);
        switch (channels) {
            case 1: halve_vec_kernel<1><<<grid, kVecThreads, 0, st>>>(s, spitch, d, dw, dpitch); break;
            case 2: halve_vec_kernel<2><<<grid, kVecThreads, 0, st>>>(s, spitch, d, dw, dpitch); break;
            case 3: halve_vec_kernel<3><<<grid, kVecThreads, 0, st>>>(s, spitch, d, dw, dpitch); break;
            default: halve_vec_kernel<4><<<grid, kVecThreads, 0, st>>>(s, spitch, d, dw, dpitch); break;
        }
    } else {
        resize_kernel<<<grid2(dw, dh), dim3(32, 8), 0, st>>>(s, sw, sh, spitch, channels, d, dw, dh, dpitch,
                                                             (float)sw / (float)dw, (float)sh / (float)dh);
    }
    return cudaGetLastError() == cudaSuccess ? PM_OK : PM_ECUDA;
}

int pm_build_pyramid_f16(pm_ctx *ctx, const void *src, int W, int H, size_t pitch, int src_format, int levels,
                         void *const *out) {
    const size_t es = src_format == PM_IMAGE_F16 ? 2 : 1;
    if (!ctx || !src || !out || W < 1 || H < 1 || levels < 1 || levels > 16 || pitch < (size_t)W * es ||
        (src_format != PM_IMAGE_U8 && src_format != PM_IMAGE_F16))
        return PM_EINVAL;
    for (int k = 0; k < levels; ++k)
        if (!out[k]) return PM_EINVAL;
    cudaStream_t st = (cudaStream_t)pm_stream(ctx);
    if (src_format == PM_IMAGE_U8) {
        const bool packed = pitch == (size_t)W;
        const size_t n = packed ? (size_t)W * H : (size_t)W;
        const int rows = packed ? 1 : H;
        if (aligned16(src, rows > 1 ? pitch : 0) && aligned16(out[0], rows > 1 ? (size_t)W * 2 : 0) &&
            rows <= kMaxGridY)
            u8_to_half_vec_kernel<<<dim3(vec_blocks(n, 16), rows), kVecThreads, 0, st>>>((const uint8_t *)src, n, pitch,
                                                                                         (__half *)out[0], W);
        else
            u8_to_half_kernel<<<grid2(W, H), dim3(32, 8), 0, st>>>((const uint8_t *)src, W, H, pitch, (__half *)out[0]);
    } else if (out[0] != src || pitch != (size_t)W * 2) {
        if (cudaMemcpy2DAsync(out[0], (size_t)W * 2, src, pitch, (size_t)W * 2, H, cudaMemcpyDeviceToDevice, st) !=
            cudaSuccess)
            return PM_ECUDA;
    }
    int w = W, h = H;
    for (int k = 1; k < levels; ++k) {
        const int dw = (w + 1) / 2, dh = (h + 1) / 2;
        const __half *s = (const __half *)out[k - 1];
        __half *d = (__half *)out[k];
        if (w % 8 == 0 && aligned16(s, 0) && ((uintptr_t)d & 7) == 0 && dh <= kMaxGridY)
            half_down_vec_kernel<<<dim3(vec_blocks(dw, 4), dh), kVecThreads, 0, st>>>(s, w, h, d, dw);
        else
            half_down_kernel<<<grid2(dw, dh), dim3(32, 8), 0, st>>>(s, w, h, d, dw, dh);
        w = dw;
        h = dh;
    }
    return cudaGetLastError() == cudaSuccess ? PM_OK : PM_ECUDA;
}

}  // extern "C"
