// Device-side building blocks of the densifier: counter-based random numbers,
// equirectangular angle evaluation, quad-packed bilinear sampling and the
// per-tap NCC moment accumulation shared by every cost kernel.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pm_types.h"

namespace pm {

// ---------------------------------------------------------------------------
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy
// as 1, 2, 3", SC'11).  Key = (seed, keyframe); counter = (pixel, tag, draw,
// constant).  tag 0 = initialisation, tag s+1 = the pixel's visit in sweep s.
// Replaces the clock-seeded cuRAND XORWOW states of the reference
// (PatchMatchCuda.cu:246-252), which made runs irreproducible.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        if (r) { k.x += 0x9E3779B9u; k.y += 0xBB67AE85u; }
        const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    }
    return c;
}

__device__ __forceinline__ uint4 philox_block(uint32_t seed, uint32_t kf, uint32_t pixel, uint32_t tag,
                                              uint32_t draw) {
    return philox4x32_10(make_uint4(pixel, tag, draw, 0x504d4742u), make_uint2(seed, kf));
}

// 24-bit uniform in (0, 1), exactly representable.
__device__ __forceinline__ float u24(uint32_t x) {
    return __fmul_rn(__fadd_rn((float)(x >> 8), 0.5f), 1.0f / 16777216.0f);
}

// Box-Muller pair from two words.
__device__ __forceinline__ float2 box_muller(uint32_t a, uint32_t b) {
    const float u1 = u24(a), u2 = u24(b);
    const float r = sqrtf(__fmul_rn(-2.0f, logf(u1)));
    const float th = __fmul_rn(6.28318530717958647692f, u2);
    return make_float2(__fmul_rn(r, cosf(th)), __fmul_rn(r, sinf(th)));
}

// ---------------------------------------------------------------------------
// atan on [0, 1]: atan(t) ~ t * P(t^2), P of degree 7, a minimax (Remez
// exchange) fit made for this project (max error 3.7e-8 rad before float
// rounding).  sample_coords scales it to turns (1/2pi), so the angles come out
// directly in image-fraction units.
// ---------------------------------------------------------------------------
#define PM_ATAN_C0 0.9999993443489075f
#define PM_ATAN_C1 -0.33329859375953674f
#define PM_ATAN_C2 0.19946566224098206f
#define PM_ATAN_C3 -0.1390862911939621f
#define PM_ATAN_C4 0.0964219719171524f
#define PM_ATAN_C5 -0.0559123270213604f
#define PM_ATAN_C6 0.021862957626581192f
#define PM_ATAN_C7 -0.004054567310959101f

// Packed FP32 pairs (fma.rn.f32x2 and friends): two independent IEEE
// operations per instruction, each rounded exactly as its scalar form.  A pair
// occupies both FMA pipes for the two cycles that two scalar operations take,
// but one issue slot instead of two, and the sample loop was bound by issue
// slots: 72.6 -> 55 warp instructions per sample with the rotation, the two
// angle polynomials and the moments in pairs (1920x960, 6 sources, 8 sweeps:
// 61.3 -> 58.0 ms; 3840x1920, 8 FP16 sources: 389 -> 373 ms; maps
// bit-identical).  What binds now is the FMA pipes and their register reads:
// three register pairs as operands take three cycles instead of two, which is
// why the last step of the coordinates is scalar, with the scale a constant
// (69 against 71 cycles per sample in a loop of the cost alone).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ f32x2 pack2(float2 v) { return pack2(v.x, v.y); }
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Both angles use atan2(a, b) = pi/4 + atan((a - b) / (a + b)) for a, b >= 0,
// whose argument lies in [-1, 1] without an octant select.  The approximate
// division can leave |t| an ulp or two above 1; with kBound each angle is
// clamped to keep |lon| <= 1/2 and |lat| <= 1/2 exactly, so sample
// coordinates stay in [0, W] x [0, H], which the quad samplers index without
// further checks (texture reads clamp in hardware and skip the two clamps).

// Sample coordinates (u, v) of direction (X, Y, Z), as a pair:
//   u = W lon + halfW, lon = atan2(X, Z) / (2 pi) in [-1/2, 1/2], the
//       equirectangular longitude in image widths (PatchMatchCuda.cu:140,143);
//       X = Z = 0 gives t = -1 and an angle of 0, like atan2(0, 0);
//   v = H lat + halfH, lat = asin(Y / |(X, Y, Z)|) / pi in [-1/2, 1/2], minus
//       the latitude in image heights (PatchMatchCuda.cu:139,144), evaluated
//       as atan2(|Y|, sqrt(X^2 + Z^2)) with the sign of Y.
// The two polynomials run as one pair in units of turns; a half turn is 2
// turns exactly, so scale = (W, 2 H) gives v the same bits as a latitude
// polynomial in half turns.  The result's halves are adjacent registers, as
// the texture fetch reads them.
template <bool kBound>
__device__ __forceinline__ f32x2 sample_coords(float X, float Y, float Z, f32x2 scale, f32x2 half) {
    constexpr float s = 0.159154943091895335769f;  // 1 / (2 pi)
    const float ax = fabsf(X), az = fabsf(Z) + 1e-30f;
    const float r2 = fmaxf(fmaf(X, X, Z * Z), 1e-30f);
    const float rho = r2 * rsqrtf(r2);
    const float ay = fabsf(Y);
    float rx, ry;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rx) : "f"(ax + az));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ry) : "f"(ay + rho));
    const f32x2 t = mul2(pack2(ax - az, ay - rho), pack2(rx, ry));
    const f32x2 q = mul2(t, t);
    f32x2 p = pack2(PM_ATAN_C7 * s, PM_ATAN_C7 * s);
    p = fma2(p, q, pack2(PM_ATAN_C6 * s, PM_ATAN_C6 * s));
    p = fma2(p, q, pack2(PM_ATAN_C5 * s, PM_ATAN_C5 * s));
    p = fma2(p, q, pack2(PM_ATAN_C4 * s, PM_ATAN_C4 * s));
    p = fma2(p, q, pack2(PM_ATAN_C3 * s, PM_ATAN_C3 * s));
    p = fma2(p, q, pack2(PM_ATAN_C2 * s, PM_ATAN_C2 * s));
    p = fma2(p, q, pack2(PM_ATAN_C1 * s, PM_ATAN_C1 * s));
    p = fma2(p, q, pack2(PM_ATAN_C0 * s, PM_ATAN_C0 * s));
    float2 a = unpack2(fma2(p, t, pack2(0.125f, 0.125f)));
    if (kBound) {
        a.x = fmaxf(a.x, 0.0f);
        a.y = fminf(a.y, 0.25f);
    }
    a.x = (Z < 0.0f) ? 0.5f - a.x : a.x;
    const float2 sc = unpack2(scale), hf = unpack2(half);
    return pack2(fmaf(copysignf(a.x, X), sc.x, hf.x), fmaf(copysignf(a.y, Y), sc.y, hf.y));
}

// ---------------------------------------------------------------------------
// Quad-packed source images.  Entry (y, x) of a (H+1) x (W+1) array holds the
// 2x2 bilinear footprint {T(x,y), T(x+1,y), T(x,y+1), T(x+1,y+1)} with the
// border policy baked in (x+1 clamps at W-1 or wraps to 0; y+1 clamps), so a
// sample is one aligned load.  Texel k sits at coordinate k, matching the
// reference's texture reads at u + 0.5 (PatchMatchCuda.cu:146).
// ---------------------------------------------------------------------------
// Split a sample coordinate c in [0, N] into cell index k = floor(c) and
// weight a = c - k.  A NaN coordinate (a degenerate plane hypothesis) gives
// k = 0, so every index stays inside the (N+1)-entry quad array.
__device__ __forceinline__ void split_coord(float c, int &k, float &a) {
    const float f = floorf(c);
    k = (int)f;
    a = c - f;
}

struct QuadU8 {
    // sample coordinates: texel k at coordinate k, indexed unchecked
    static constexpr float kCoordOffset = 0.0f;
    static constexpr bool kBound = true;
    // shift: value subtracted from every texel, given as 2^23 + I_c so the
    // byte-to-float conversion and the centring are one subtraction.
    static __device__ __forceinline__ float shift_for(float centre) { return 8388608.0f + centre; }
    // Footprint of one sample: the packed texels and the bilinear weights.
    struct Raw {
        uint32_t w;
        float ax, ay;
    };
    static __device__ __forceinline__ Raw fetch(const void *quad, unsigned long long, int qpitch, float u, float v) {
        // u in [0, W], v in [0, H] by construction of sample_coords
        int x0, y0;
        Raw f;
        split_coord(u, x0, f.ax);
        split_coord(v, y0, f.ay);
        f.w = __ldg(static_cast<const uint32_t *>(quad) + (y0 * qpitch + x0));
        return f;
    }
    static __device__ __forceinline__ float centred(const Raw &f, float shift) {
        // texels as 2^23 + byte; differences are exact, the shift is applied once per row
        const float m00 = __uint_as_float(__byte_perm(f.w, 0x4B000000u, 0x7540));
        const float m01 = __uint_as_float(__byte_perm(f.w, 0x4B000000u, 0x7541));
        const float m10 = __uint_as_float(__byte_perm(f.w, 0x4B000000u, 0x7542));
        const float m11 = __uint_as_float(__byte_perm(f.w, 0x4B000000u, 0x7543));
        const float a = fmaf(f.ax, m01 - m00, m00 - shift);
        const float b = fmaf(f.ax, m11 - m10, m10 - shift);
        return fmaf(f.ay, b - a, a);
    }
    static __device__ __forceinline__ f32x2 centred2(const Raw &f, const Raw &g, float shift) {
        return pack2(centred(f, shift), centred(g, shift));
    }
};

struct QuadF16 {
    static constexpr float kCoordOffset = 0.0f;
    static constexpr bool kBound = true;
    static __device__ __forceinline__ float shift_for(float centre) { return centre; }
    struct Raw {
        uint2 w;
        float ax, ay;
    };
    static __device__ __forceinline__ Raw fetch(const void *quad, unsigned long long, int qpitch, float u, float v) {
        int x0, y0;
        Raw f;
        split_coord(u, x0, f.ax);
        split_coord(v, y0, f.ay);
        f.w = __ldg(static_cast<const uint2 *>(quad) + (y0 * qpitch + x0));
        return f;
    }
    static __device__ __forceinline__ float centred(const Raw &f, float shift) {
        const float2 r0 = __half22float2(*reinterpret_cast<const __half2 *>(&f.w.x));
        const float2 r1 = __half22float2(*reinterpret_cast<const __half2 *>(&f.w.y));
        const float t00 = r0.x - shift, t01 = r0.y - shift, t10 = r1.x - shift, t11 = r1.y - shift;
        const float a = fmaf(f.ax, t01 - t00, t00);
        const float b = fmaf(f.ax, t11 - t10, t10);
        return fmaf(f.ay, b - a, a);
    }
    static __device__ __forceinline__ f32x2 centred2(const Raw &f, const Raw &g, float shift) {
        return pack2(centred(f, shift), centred(g, shift));
    }
};

// Texture sampling (PM_SAMPLER_TEXTURE): the texture unit's bilinear filter
// over the source image, read at the texel-centre convention of the
// reference (coordinate + 0.5, PatchMatchCuda.cu:146), clamped at the border.
// u8 images are bound as normalised 8-bit textures (value / 255).
struct TexU8 {
    static constexpr float kCoordOffset = 0.5f;
    static constexpr bool kBound = false;
    static __device__ __forceinline__ float shift_for(float centre) { return centre; }
    typedef float Raw;
    static __device__ __forceinline__ float fetch(const void *, unsigned long long tex, int, float u, float v) {
        return tex2D<float>((cudaTextureObject_t)tex, u, v);
    }
    static __device__ __forceinline__ float centred(float raw, float shift) { return fmaf(raw, 255.0f, -shift); }
    static __device__ __forceinline__ f32x2 centred2(float f, float g, float shift) {
        return fma2(pack2(f, g), pack2(255.0f, 255.0f), pack2(-shift, -shift));
    }
};

struct TexF16 {
    static constexpr float kCoordOffset = 0.5f;
    static constexpr bool kBound = false;
    static __device__ __forceinline__ float shift_for(float centre) { return centre; }
    typedef float Raw;
    static __device__ __forceinline__ float fetch(const void *, unsigned long long tex, int, float u, float v) {
        return tex2D<float>((cudaTextureObject_t)tex, u, v);
    }
    static __device__ __forceinline__ float centred(float raw, float shift) { return raw - shift; }
    static __device__ __forceinline__ f32x2 centred2(float f, float g, float shift) {
        return add2(pack2(f, g), pack2(-shift, -shift));
    }
};

// Bilateral window weight exp(-dI^2 / (2 sigma_c^2) - d^2 / (2 sigma_x^2))
// (PatchMatchCuda.cu:148-149) as exp2 of a pre-scaled exponent:
// ncf = -log2(e) / (2 sigma_c^2), dk = -log2(e) (dx^2 + dy^2) / (2 sigma_x^2).
__device__ __forceinline__ float bilateral_weight(float xs, float ncf, float dk) {
    return exp2f(fmaf(xs * xs, ncf, dk));
}

// The six standard normals of refinements t and t + 1 (t even) of one pixel
// visit: normals 3t..3t+5 of the Box-Muller stream whose pair p uses Philox
// block p / 2, words (x, y) for even p and (z, w) for odd p.  Two refinements
// at a time take two blocks and three pairs; one at a time took two blocks and
// two pairs each, a third of the draws twice.
__device__ __forceinline__ void refine_normals2(uint32_t seed, uint32_t kf, uint32_t pix, uint32_t tag, int t,
                                                float (&z)[6]) {
    const int p0 = (3 * t) >> 1;
    const uint4 b0 = philox_block(seed, kf, pix, tag, (uint32_t)(p0 >> 1));
    const uint4 b1 = philox_block(seed, kf, pix, tag, (uint32_t)(p0 >> 1) + 1u);
    const bool odd = p0 & 1;
    const float2 n0 = box_muller(odd ? b0.z : b0.x, odd ? b0.w : b0.y);
    const float2 n1 = box_muller(odd ? b1.x : b0.z, odd ? b1.y : b0.w);
    const float2 n2 = box_muller(odd ? b1.z : b1.x, odd ? b1.w : b1.y);
    z[0] = n0.x;
    z[1] = n0.y;
    z[2] = n1.x;
    z[3] = n1.y;
    z[4] = n2.x;
    z[5] = n2.y;
}

// The four standard normals of refinement t of the plain (host-variant)
// propagation: Philox block t, words (x, y) and (z, w), one depth draw
// followed by three normal draws (depthmap.cc:1041-1050).
__device__ __forceinline__ void refine_normals4(uint32_t seed, uint32_t kf, uint32_t pix, uint32_t tag, int t,
                                                float &z0, float &z1, float &z2, float &z3) {
    const uint4 blk = philox_block(seed, kf, pix, tag, (uint32_t)t);
    const float2 a = box_muller(blk.x, blk.y), b = box_muller(blk.z, blk.w);
    z0 = a.x;
    z1 = a.y;
    z2 = b.x;
    z3 = b.y;
}

// ---------------------------------------------------------------------------
// One tap of the plane-induced warp for all S sources (PatchMatchCuda.cu:107-157,
// restructured).  The reference maps X_c = b / (pi . b) through
// R_r (R_1^T X_c - R_1^T t_1) + t_r and normalises.  Only the direction of the
// source-frame point matters, so with M_r = R_r R_1^T and c_r = t_r - M_r t_1
// (composed in FP64 on the host) we evaluate |s| * X_r = sign(s) M_r b + |s| c_r,
// s = pi . b, which has the same direction and no division.  M_r b does not
// depend on the hypothesis: the tile kernels stage its row and column factors.
// Moments are accumulated shifted by the centre intensity (y - I_c), which is
// exact algebra for the NCC and avoids float cancellation in the variances.
// ---------------------------------------------------------------------------
// Where the per-source constants of the sample loop come from.  ParamAccess:
// kernel parameters (constant bank, usable directly as instruction operands).
// SharedAccess: a request's arguments staged in shared memory by the batched
// executor, re-read at every use: the loads are volatile so that the compiler
// does not hoist all sources' rows into registers (that spills).
struct ParamAccess {
    static __device__ __forceinline__ float val(const float &x) { return x; }
    static __device__ __forceinline__ float2 pair(const float &x) { return make_float2((&x)[0], (&x)[1]); }
    static __device__ __forceinline__ float4 row(const float4 &g) { return g; }
    static __device__ __forceinline__ unsigned long long tex(const unsigned long long &t) { return t; }
    static __device__ __forceinline__ const void *ptr(const void *const &p) { return p; }
};
struct SharedAccess {
    static __device__ __forceinline__ float val(const float &x) {
        float v;
        const unsigned a = (unsigned)__cvta_generic_to_shared(&x);
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
        return v;
    }
    static __device__ __forceinline__ float2 pair(const float &x) {
        float2 v;
        const unsigned a = (unsigned)__cvta_generic_to_shared(&x);
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
        return v;
    }
    static __device__ __forceinline__ float4 row(const float4 &g) {
        float4 v;
        const unsigned a = (unsigned)__cvta_generic_to_shared(&g);
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
        return v;
    }
    static __device__ __forceinline__ unsigned long long tex(const unsigned long long &t) {
        unsigned long long v;
        const unsigned a = (unsigned)__cvta_generic_to_shared(&t);
        asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
        return v;
    }
    static __device__ __forceinline__ const void *ptr(const void *const &p) {
        unsigned long long v;
        const unsigned a = (unsigned)__cvta_generic_to_shared(&p);
        asm volatile("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"(a));
        return reinterpret_cast<const void *>(v);
    }
};

// M b of one source: the first two components as a pair and the third, the
// hypothesis-independent part of the warp.
struct Rotated {
    f32x2 xy;
    float z;
};

// M b for a source's pose block, evaluated directly; bx2, by2, bz2 hold each
// bearing component in both halves.
__device__ __forceinline__ Rotated rotate(const float4 &g0, const float4 &g1, const float4 &g2, f32x2 bx2, f32x2 by2,
                                          f32x2 bz2) {
    const float bx = unpack2(bx2).x, by = unpack2(by2).x, bz = unpack2(bz2).x;
    Rotated m;
    m.xy = fma2(pack2(g0.x, g0.y), bx2, fma2(pack2(g0.z, g0.w), by2, mul2(pack2(g1.x, g1.y), bz2)));
    m.z = fmaf(g2.x, bx, fmaf(g2.y, by, g2.z * bz));
    return m;
}

// Factored form over the equirectangular grid: with b = (cos lat sin lon,
// -sin lat, cos lat cos lon),  M b = cos(lat) A(lon) + B(lat),
//   A = sin(lon) M e_x + cos(lon) M e_z   (per image column and source),
//   B = -sin(lat) M e_y                   (per image row and source),
// so a tile kernel stages A per column and B per row once and a tap costs
// three FMAs and two shared-memory reads per source instead of nine FMAs.
// Used from PM_FACTOR_MIN_SOURCES to PM_FACTOR_MAX_SOURCES sources: with
// fewer sources the shared-memory reads cost as much as the FMAs they
// replace and the staged factors take L1 from the texture samples (measured,
// 8 sweeps: 1920x960 u8 - 4-6 sources faster direct, 8 even, 10 sources 4 %
// faster factored; 3840x1920 - 8 sources FP16 4 % faster direct, 9-10
// sources 0-3 % faster factored).  The staged factors take 1760 bytes of
// shared memory per source.
#ifndef PM_FACTOR_MIN_SOURCES
#define PM_FACTOR_MIN_SOURCES 9
#endif
#ifndef PM_FACTOR_MAX_SOURCES
#define PM_FACTOR_MAX_SOURCES 10
#endif
template <int S>
__host__ __device__ constexpr bool factored_warp() {
    return S >= PM_FACTOR_MIN_SOURCES && S <= PM_FACTOR_MAX_SOURCES;
}
__device__ __forceinline__ float3 col_factor(const float4 &g0, const float4 &g1, const float4 &g2, float sin_lon,
                                             float cos_lon) {
    return make_float3(fmaf(sin_lon, g0.x, cos_lon * g1.x), fmaf(sin_lon, g0.y, cos_lon * g1.y),
                       fmaf(sin_lon, g2.x, cos_lon * g2.z));
}
__device__ __forceinline__ float3 row_factor(const float4 &g0, const float4 &g1, const float4 &g2, float sin_lat) {
    return make_float3(-sin_lat * g0.z, -sin_lat * g0.w, -sin_lat * g2.y);
}

// x with its sign bit flipped when sg (0 or 0x80000000) is set.
__device__ __forceinline__ float flip_sign(float x, uint32_t sg) { return __uint_as_float(__float_as_uint(x) ^ sg); }

template <int S, class Img, class Acc = ParamAccess>
struct TapAccum {
    // moments of sources 2k and 2k + 1 as pairs; an odd last source on its own
    static constexpr int kPairs = S / 2;
    f32x2 py[kPairs + 1], pyy[kPairs + 1], pxy[kPairs + 1];
    float oy, oyy, oxy;
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < kPairs; ++k) py[k] = pyy[k] = pxy[k] = 0ull;
        oy = oyy = oxy = 0.0f;
    }
    __device__ __forceinline__ static float part(const f32x2 (&p)[kPairs + 1], float odd, int r) {
        if (r >= 2 * kPairs) return odd;
        const float2 v = unpack2(p[r >> 1]);
        return (r & 1) ? v.y : v.x;
    }
    __device__ __forceinline__ float swy(int r) const { return part(py, oy, r); }
    __device__ __forceinline__ float swyy(int r) const { return part(pyy, oyy, r); }
    __device__ __forceinline__ float swxy(int r) const { return part(pxy, oxy, r); }
    // One tap given |s| (s = pi . b) and the sources' signed rotated
    // bearings mb(r) = sign(s) M_r b (a Rotated): X_r = sign(s) M_r b + |s| c_r.
    // P and src live in kernel parameter space (or shared memory, through
    // Acc); w: bilateral weight, xs: tap intensity minus centre; scale =
    // (W, 2 H), half = (W / 2, H / 2) plus the sampler's coordinate offset.
    template <class MB>
    __device__ __forceinline__ void add_rot(const PmPoses &P, const SrcSet &src, f32x2 scale, f32x2 half, float shift,
                                            float as, MB mb, float w, float xs) {
        typename Img::Raw raw[S];
        fetch(P, src, scale, half, as, mb, raw);
        add(raw, shift, w, xs);
    }
    template <class MB>
    __device__ __forceinline__ static void fetch(const PmPoses &P, const SrcSet &src, f32x2 scale, f32x2 half,
                                                 float as, MB mb, typename Img::Raw (&raw)[S]) {
        // phase 1: all S sample coordinates, so the S footprint loads issue
        // back to back; phase 2: bilinear + moments as they arrive
        f32x2 uv[S];
        const f32x2 as2 = pack2(as, as);
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const Rotated m = mb(r);
            const float2 c = Acc::pair(P.G[r][1].z);
            const float2 XY = unpack2(fma2(as2, pack2(c), m.xy));
            const float Z = fmaf(as, Acc::val(P.G[r][2].w), m.z);
            uv[r] = sample_coords<Img::kBound>(XY.x, XY.y, Z, scale, half);
        }
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const float2 c = unpack2(uv[r]);
            raw[r] = Img::fetch(Acc::ptr(src.quad[r]), Acc::tex(src.tex[r]), src.qpitch, c.x, c.y);
        }
    }
    __device__ __forceinline__ void add(const typename Img::Raw (&raw)[S], float shift, float w, float xs) {
        const f32x2 w2 = pack2(w, w), xs2 = pack2(xs, xs);
#pragma unroll
        for (int k = 0; k < kPairs; ++k) add_pair(k, Img::centred2(raw[2 * k], raw[2 * k + 1], shift), w2, xs2);
        if constexpr (S & 1) add_odd(Img::centred(raw[S - 1], shift), w, xs);
    }
    __device__ __forceinline__ void add_pair(int k, f32x2 y, f32x2 w2, f32x2 xs2) {
        const f32x2 wy = mul2(w2, y);
        py[k] = add2(py[k], wy);
        pyy[k] = fma2(wy, y, pyy[k]);
        pxy[k] = fma2(wy, xs2, pxy[k]);
    }
    __device__ __forceinline__ void add_odd(float y, float w, float xs) {
        const float wy = w * y;
        oy += wy;
        oyy = fmaf(wy, y, oyy);
        oxy = fmaf(wy, xs, oxy);
    }
    // One tap with bearing b = (bx, by, bz), rotated per source directly.
    __device__ __forceinline__ void add_bearing(const PmPoses &P, const SrcSet &src, f32x2 scale, f32x2 half,
                                                float shift, float px, float py_, float pz, float bx, float by,
                                                float bz, float w, float xs) {
        const float s = fmaf(px, bx, fmaf(py_, by, pz * bz));
        const uint32_t sg = __float_as_uint(s) & 0x80000000u;
        const float sbx = flip_sign(bx, sg), sby = flip_sign(by, sg), sbz = flip_sign(bz, sg);
        const f32x2 bx2 = pack2(sbx, sbx), by2 = pack2(sby, sby), bz2 = pack2(sbz, sbz);
        add_rot(P, src, scale, half, shift, fabsf(s),
                [&](int r) {
                    return rotate(Acc::row(P.G[r][0]), Acc::row(P.G[r][1]), Acc::row(P.G[r][2]), bx2, by2, bz2);
                },
                w, xs);
    }
    // The footprints of the tap at the grid point with row trig rt = (cos lat,
    // sin lat) and column trig ct = (sin lon, cos lon): the factored form when
    // factored_warp<S>() (the arithmetic of the staged tile factors), the direct
    // rotation of the bearing otherwise; the bearing is (cos lat sin lon,
    // -sin lat, cos lat cos lon), as in the staged tile.
    __device__ __forceinline__ static void fetch_trig(const PmPoses &P, const SrcSet &src, f32x2 scale, f32x2 half,
                                                      float px, float py_, float pz, float2 rt, float2 ct,
                                                      typename Img::Raw (&raw)[S]) {
        const float bx = rt.x * ct.x, by = -rt.y, bz = rt.x * ct.y;
        const float s = fmaf(px, bx, fmaf(py_, by, pz * bz));
        const uint32_t sg = __float_as_uint(s) & 0x80000000u;
        if constexpr (factored_warp<S>()) {
            const float sc = flip_sign(rt.x, sg);
            fetch(P, src, scale, half, fabsf(s),
                  [&](int r) {
                      const float4 g0 = Acc::row(P.G[r][0]), g1 = Acc::row(P.G[r][1]), g2 = Acc::row(P.G[r][2]);
                      const float3 A = col_factor(g0, g1, g2, ct.x, ct.y);
                      const float3 B = row_factor(g0, g1, g2, rt.y);
                      return Rotated{pack2(fmaf(sc, A.x, flip_sign(B.x, sg)), fmaf(sc, A.y, flip_sign(B.y, sg))),
                                     fmaf(sc, A.z, flip_sign(B.z, sg))};
                  },
                  raw);
        } else {
            const float sbx = flip_sign(bx, sg), sby = flip_sign(by, sg), sbz = flip_sign(bz, sg);
            const f32x2 bx2 = pack2(sbx, sbx), by2 = pack2(sby, sby), bz2 = pack2(sbz, sbz);
            fetch(P, src, scale, half, fabsf(s),
                  [&](int r) {
                      return rotate(Acc::row(P.G[r][0]), Acc::row(P.G[r][1]), Acc::row(P.G[r][2]), bx2, by2, bz2);
                  },
                  raw);
        }
    }
};

// NCC from shifted moments (PatchMatchCuda.cu:161-170): -1 when either
// weighted variance is below 0.1.  RefMoments: the reference window's part,
// the same for every source.
struct RefMoments {
    float prob, mx, vx;
    __device__ __forceinline__ RefMoments(float sw, float swx, float swxx)
        : prob(1.0f / sw), mx(swx * prob), vx(fmaf(-mx, mx, swxx * prob)) {}
};
struct SrcMoments {
    float vy, cov;
    __device__ __forceinline__ SrcMoments(const RefMoments &x, float swy, float swyy, float swxy) {
        const float my = swy * x.prob;
        vy = fmaf(-my, my, swyy * x.prob);
        cov = fmaf(-x.mx, my, swxy * x.prob);
    }
};
__device__ __forceinline__ float ncc_of(const RefMoments &x, const SrcMoments &y) {
    const float ncc = y.cov / sqrtf(x.vx * y.vy);
    return (x.vx < 0.1f || y.vy < 0.1f) ? -1.0f : ncc;
}

// View combination; best = argmax of the per-source NCCs (sep).
//  PM_COMBINE_FOLD: the reference GPU kernel: NCC of the moments accumulated
//    over sources 0..r (cum[r], the reference never resets its sums between
//    views, PatchMatchCuda.cu:57-62,100-176), folded from -1 with "average
//    when within 25 %, else max" (PatchMatchCuda.cu:93,171);
//  PM_COMBINE_FOLD_SEPARATE: the same fold over the per-source NCCs;
//  PM_COMBINE_MAX: maximum (the reference CPU path, depthmap.cc:1104-1127);
//  PM_COMBINE_TOPK: mean of the top_k best sources (per-pixel view selection).
template <int S>
__device__ __forceinline__ float fold_scores(const float (&v)[S]) {
    float score = -1.0f;
#pragma unroll
    for (int r = 0; r < S; ++r) {
        const float s2 = v[r];
        score = (fabsf(__fdiv_rn(__fsub_rn(score, s2), s2)) < 0.25f) ? __fmul_rn(0.5f, __fadd_rn(score, s2))
                                                                     : fmaxf(score, s2);
    }
    return score;
}

template <int S>
__device__ __forceinline__ int argmax(const float (&v)[S]) {
    int b = 0;
    float m = v[0];
#pragma unroll
    for (int r = 1; r < S; ++r) {
        b = v[r] > m ? r : b;
        m = v[r] > m ? v[r] : m;
    }
    return b;
}

// PM_COMBINE_TOPK: mean of the k largest by repeated selection, summed in
// descending order.
template <int S>
__device__ __forceinline__ float top_mean(const float (&sep)[S], int top_k) {
    float v[S];
#pragma unroll
    for (int r = 0; r < S; ++r) v[r] = sep[r];
    const int k = top_k < 1 ? 1 : (top_k > S ? S : top_k);
    float accf = 0.0f;
    for (int a = 0; a < k; ++a) {
        const int bi = argmax<S>(v);
        float m = v[0];
#pragma unroll
        for (int r = 0; r < S; ++r) m = (r == bi) ? v[r] : m;
        accf += m;
#pragma unroll
        for (int r = 0; r < S; ++r) v[r] = (r == bi) ? -3.0e38f : v[r];
    }
    return accf / (float)k;
}

// Per-source NCCs of one hypothesis from the window moments.
template <int S, class Img, class Acc>
__device__ __forceinline__ void source_nccs(const TapAccum<S, Img, Acc> &acc, float sw, float swx, float swxx,
                                            float (&sep)[S]) {
    const RefMoments x(sw, swx, swxx);
#pragma unroll
    for (int r = 0; r < S; ++r) sep[r] = ncc_of(x, SrcMoments(x, acc.swy(r), acc.swyy(r), acc.swxy(r)));
}

// Combined score of one hypothesis from the window moments, and its best
// source.  The fold over accumulated moments and the maximum need the
// per-source NCCs only for the best source, so those are ranked by
// cov * rsqrt(vx vy): that is within 1e-6 of the NCC, relatively, so a lead of
// more than 1e-5 decides, and closer races (ties among them) are settled by
// the NCCs themselves.  A square root and a division per source fall away.
template <int S, class Img, class Acc>
__device__ __forceinline__ float score_moments(const TapAccum<S, Img, Acc> &acc, float sw, float swx, float swxx,
                                               int mode, int top_k, int *best) {
    if (mode == PM_COMBINE_FOLD || mode == PM_COMBINE_MAX) {
        const RefMoments x(sw, swx, swxx);
        float v[S];
#pragma unroll
        for (int r = 0; r < S; ++r) {
            const SrcMoments y(x, acc.swy(r), acc.swyy(r), acc.swxy(r));
            v[r] = y.vy < 0.1f ? -1.0f : y.cov * rsqrtf(x.vx * y.vy);
        }
        int b = argmax<S>(v);
        float top = v[0], next = -3.0e38f;
#pragma unroll
        for (int r = 1; r < S; ++r) {
            next = fmaxf(next, fminf(top, v[r]));
            top = fmaxf(top, v[r]);
        }
        if (x.vx < 0.1f) {
            b = 0;  // every NCC is -1
        } else if (!(v[0] == v[0] && top - next > 1e-5f * fmaxf(1.0f, fabsf(top)))) {
            float sep[S];
            source_nccs(acc, sw, swx, swxx, sep);
            b = argmax<S>(sep);
            if (mode == PM_COMBINE_MAX) {
                float m = sep[0];
#pragma unroll
                for (int r = 1; r < S; ++r) m = fmaxf(m, sep[r]);
                *best = b;
                return m;
            }
        }
        *best = b;
        if (mode == PM_COMBINE_MAX) {
            float y = 0.f, yy = 0.f, xy = 0.f;
#pragma unroll
            for (int r = 0; r < S; ++r) {
                y = r == b ? acc.swy(r) : y;
                yy = r == b ? acc.swyy(r) : yy;
                xy = r == b ? acc.swxy(r) : xy;
            }
            return ncc_of(x, SrcMoments(x, y, yy, xy));
        }
        float cum[S];
        float cy = 0.f, cyy = 0.f, cxy = 0.f;
#pragma unroll
        for (int r = 0; r < S; ++r) {
            cy += acc.swy(r);
            cyy += acc.swyy(r);
            cxy += acc.swxy(r);
            const float n = (float)(r + 1);
            const RefMoments xn(n * sw, n * swx, n * swxx);
            cum[r] = ncc_of(xn, SrcMoments(xn, cy, cyy, cxy));
        }
        return fold_scores<S>(cum);
    }
    float sep[S];
    source_nccs(acc, sw, swx, swxx, sep);
    *best = argmax<S>(sep);
    return mode == PM_COMBINE_FOLD_SEPARATE ? fold_scores<S>(sep) : top_mean<S>(sep, top_k);
}

}  // namespace pm
