// Post-filter, export, geometric-consistency filter and point fusion kernels.
#include <cuda_runtime.h>

#include "pm_device.cuh"
#include "pm_kernels.h"

namespace pm {

namespace {

constexpr float kPiF = 3.14159265358979323846f;

__device__ __forceinline__ void cswap(float &a, float &b) {
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo;
    b = hi;
}
__device__ __forceinline__ float med3(float a, float b, float c) {
    return fmaxf(fminf(a, b), fminf(fmaxf(a, b), c));
}

// 3x3 median with replicated borders (OpenCV medianBlur ksize 3 on CV_32F):
// sort each row, then median(max of minima, median of medians, min of maxima).
__device__ __forceinline__ float median3x3(const float *m, int W, int H, int i, int j) {
    float r[3][3];
#pragma unroll
    for (int di = 0; di < 3; ++di) {
        const int y = min(max(i + di - 1, 0), H - 1);
#pragma unroll
        for (int dj = 0; dj < 3; ++dj) {
            const int x = min(max(j + dj - 1, 0), W - 1);
            r[di][dj] = m[(size_t)y * W + x];
        }
        cswap(r[di][0], r[di][1]);
        cswap(r[di][1], r[di][2]);
        cswap(r[di][0], r[di][1]);
    }
    const float lo = fmaxf(fmaxf(r[0][0], r[1][0]), r[2][0]);
    const float mid = med3(r[0][1], r[1][1], r[2][1]);
    const float hi = fminf(fminf(r[0][2], r[1][2]), r[2][2]);
    return med3(lo, mid, hi);
}

// Window of the host copy-back (depthmap.cc:731-760): rows/cols
// [patch_half, N - patch_half - 4); mask; low-variance mask over the taps
// (PatchVariance, depthmap.cc:963-973, averaged over the taps it fills).
__global__ void post_window_kernel(const PostArgs a) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.H || j >= a.W) return;
    const size_t idx = (size_t)i * a.W + j;
    const int ph = a.patch_half;
    float d = 0.0f, s = -1.0f;
    if (i >= ph && i < a.H - ph - 4 && j >= ph && j < a.W - ph - 4 && (!a.mask || a.mask[idx])) {
        bool low = false;
        if (a.min_var > 0.0f) {
            float sum = 0.0f;
            int n = 0;
            for (int u = -ph; u <= ph; u += 2)
                for (int v = -ph; v <= ph; v += 2, ++n) sum = __fadd_rn(sum, a.ref[(size_t)(i + u) * a.W + (j + v)]);
            const float mean = __fdiv_rn(sum, (float)n);
            float sum2 = 0.0f;
            for (int u = -ph; u <= ph; u += 2)
                for (int v = -ph; v <= ph; v += 2) {
                    const float dd = __fsub_rn(a.ref[(size_t)(i + u) * a.W + (j + v)], mean);
                    sum2 = __fadd_rn(sum2, __fmul_rn(dd, dd));
                }
            low = __fdiv_rn(sum2, (float)n) < a.min_var;
        }
        if (low) {
            d = 0.0f;
            s = 0.0f;
        } else {
            d = a.plane[idx].w;
            s = a.score[idx];
        }
    }
    a.d0[idx] = d;
    a.s0[idx] = s;
}

__global__ void median_kernel(const float *in, float *out, int W, int H) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= H || j >= W) return;
    out[(size_t)i * W + j] = median3x3(in, W, H, i, j);
}

// Second median + PostProcess thresholds (depthmap.cc:1176-1197).
__global__ void post_threshold_kernel(const PostArgs a) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.H || j >= a.W) return;
    const size_t idx = (size_t)i * a.W + j;
    const float m = median3x3(a.m1, a.W, a.H, i, j);
    const float d = a.d0[idx], s = a.s0[idx];
    // (float) q > 0.05 (double) is q >= 0.05f for a float q
    const bool reject = d == 0.0f || __fdiv_rn(fabsf(__fsub_rn(d, m)), d) >= 0.05f || d < a.min_depth ||
                        d > a.max_depth || s <= a.min_score;
    a.out_depth[idx] = reject ? 0.0f : m;
    a.out_score[idx] = reject ? -1.0f : s;
}

__global__ void export_kernel(const float4 *plane, const float *score, const int8_t *best, const float *fd,
                              const float *fs, const float2 *row_trig, const float2 *col_trig, int W, int H, int raw,
                              float *depth, float *score_out, float *plane3, float *normal3, int32_t *best32) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= H || j >= W) return;
    const size_t idx = (size_t)i * W + j;
    const float4 p = plane[idx];
    const float d = raw ? p.w : fd[idx];
    if (depth) depth[idx] = d;
    if (score_out) score_out[idx] = raw ? score[idx] : fs[idx];
    if (plane3) {
        plane3[3 * idx] = p.x;
        plane3[3 * idx + 1] = p.y;
        plane3[3 * idx + 2] = p.z;
    }
    if (normal3) {
        // unit normal facing the camera: -pi / |pi| (pi . b = 1 / depth > 0)
        const float n = sqrtf(p.x * p.x + p.y * p.y + p.z * p.z);
        const float2 rt = row_trig[i], ct = col_trig[j];
        const float s = p.x * rt.x * ct.x - p.y * rt.y + p.z * rt.x * ct.y;
        const float k = (d > 0.0f && n > 0.0f) ? (s > 0.0f ? -1.0f : 1.0f) / n : 0.0f;
        normal3[3 * idx] = p.x * k;
        normal3[3 * idx + 1] = p.y * k;
        normal3[3 * idx + 2] = p.z * k;
    }
    if (best32) best32[idx] = best[idx];
}

// Equirect projection of a camera-frame point (ReprojectEquirect,
// depthmap.cc:143-161, in float).  Returns false when nearer than 1e-4.
__device__ __forceinline__ bool project(float X, float Y, float Z, float Wf, float Hf, float &x, float &y, float &r) {
    r = sqrtf(X * X + Y * Y + Z * Z);
    if (r < 1e-4f) return false;
    const float lat = -asinf(fminf(1.0f, fmaxf(-1.0f, Y / r)));
    const float lon = atan2f(X, Z);
    x = Wf * (0.5f + lon / (2.0f * kPiF));
    y = Hf * (0.5f - lat / kPiF);
    return true;
}

// LinearInterpolation<float> (depthmap.cc:34-50)
__device__ __forceinline__ float interp_depth(const float *img, int W, int H, float y, float x) {
    if (x < 0.0f || x >= (float)(W - 1) || y < 0.0f || y >= (float)(H - 1)) return 0.0f;
    const int ix = (int)x, iy = (int)y;
    const float dx = x - ix, dy = y - iy;
    const float *r0 = img + (size_t)iy * W + ix, *r1 = r0 + W;
    const float im0 = (1 - dx) * r0[0] + dx * r0[1];
    const float im1 = (1 - dx) * r1[0] + dx * r1[1];
    return (1 - dy) * im0 + dy * im1;
}

// DepthmapCleaner::Clean (depthmap.cc:1337-1373) for every pixel of view 0.
// Bound by the instructions of the projections and their inverses (some 470
// a view and warp, 90 % issue-active), so a pixel stops at the view that
// settles it: 3840x1920 with 5 views, 2 needed, 401 -> 246 us where 98 % are
// kept; 405 -> 400 us with 3 needed and noise that leaves 59 %.  (Packing a
// block's open pixels before each view gave 241 and 383 us, and cost small
// maps 10 %.)
__global__ void clean_kernel(const __grid_constant__ CleanArgs a) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.H || j >= a.W) return;
    const size_t idx = (size_t)i * a.W + j;
    const float d = a.depths[0][idx];
    float out = 0.0f;
    // depth < 1e-6 (double) is depth <= 1e-6f for a float depth
    if (!(d <= 1e-6f)) {
        const float2 rt = a.row_trig[i], ct = a.col_trig[j];
        const float Xc = d * rt.x * ct.x, Yc = -d * rt.y, Zc = d * rt.x * ct.y;
        const float Wf = (float)a.W, Hf = (float)a.H;
        int consistent = 1;
        // until the views left cannot change the outcome
        for (int k = 1; k < a.n && consistent < a.min_consistent && consistent + a.n - k >= a.min_consistent; ++k) {
            const float *M = a.M[k], *c = a.c[k];
            const float X = M[0] * Xc + M[1] * Yc + M[2] * Zc + c[0];
            const float Y = M[3] * Xc + M[4] * Yc + M[5] * Zc + c[1];
            const float Z = M[6] * Xc + M[7] * Yc + M[8] * Zc + c[2];
            float x, y, dop;
            if (!project(X, Y, Z, Wf, Hf, x, y, dop)) continue;
            const int ix = (int)x, iy = (int)y;
            if (!(iy >= 0 && iy < a.H && ix >= 0 && ix < a.W)) continue;
            const float dat = interp_depth(a.depths[k], a.W, a.H, y, x);
            if (!(fabsf(dat - dop) < dop * a.thr)) continue;
            if (a.reproj_px > 0.0f) {
                // round trip through view k's depth back into view 0
                const float lon = 2.0f * kPiF * (x / Wf - 0.5f), lat = -kPiF * (y / Hf - 0.5f);
                float sl, cl, sn, cn;
                sincosf(lat, &sl, &cl);
                sincosf(lon, &sn, &cn);
                const float qx = dat * cl * sn, qy = -dat * sl, qz = dat * cl * cn;
                const float *Mi = a.Minv[k], *ci = a.cinv[k];
                const float X0 = Mi[0] * qx + Mi[1] * qy + Mi[2] * qz + ci[0];
                const float Y0 = Mi[3] * qx + Mi[4] * qy + Mi[5] * qz + ci[1];
                const float Z0 = Mi[6] * qx + Mi[7] * qy + Mi[8] * qz + ci[2];
                float x0, y0, r0;
                if (!project(X0, Y0, Z0, Wf, Hf, x0, y0, r0)) continue;
                float ex = fabsf(x0 - (float)j);
                const float ey = fabsf(y0 - (float)i);
                if (ex > 0.5f * Wf) ex = Wf - ex;
                if (ex > a.reproj_px || ey > a.reproj_px) continue;
            }
            ++consistent;
        }
        if (consistent >= a.min_consistent) out = d;
    }
    a.out[idx] = out;
}

// ---------------------------------------------------------------------------
// Point fusion (DepthmapPruner::Prune, depthmap.cc:1556-1695).  The reference
// walks the head map in raster order and, per pixel, visits views 1..n-1 in
// order; a nearer head pixel zeroes the matching pixel of a later view, which
// later head pixels then see as empty.  Within view k, a target pixel q is
// therefore zeroed by the first (raster order) head pixel that reaches view k
// and qualifies; head pixels after it see 0, head pixels before it see the
// original value.  Processing views in order with an atomicMin per target
// reproduces that exactly, independent of thread scheduling.
// ---------------------------------------------------------------------------
//
// All of these kernels move a few bytes per pixel; with one pixel per thread
// they waited for their own dependent loads.  A thread takes V = 4 consecutive
// pixels with vector accesses and keeps their gathers in flight together;
// V = 1 where rows or maps are not aligned for that, and for small maps (see
// kFuseVecPixels).  Measured at 3840x1920 with 5 views (one pixel -> four per
// thread, us): init 33 -> 15, classify 59/51/43/40 -> 48/42/35/31 (bound by the
// projection's arithmetic), resolve 47/41/35/33 -> 23/17/15/14, count 21 -> 4,
// scan 14 -> 5; the scatter's figures stand at its kernel.
enum : int8_t { kSkip = 0, kZero = 1, kDrop = 2 };

template <int V, class T>
struct alignas(sizeof(T) * V) Vec {
    T v[V];
};
template <int V, class T>
__device__ __forceinline__ Vec<V, T> load_vec(const T *p) {
    return *reinterpret_cast<const Vec<V, T> *>(p);
}
template <int V, class T>
__device__ __forceinline__ void store_vec(T *p, const Vec<V, T> &x) {
    *reinterpret_cast<Vec<V, T> *>(p) = x;
}

template <int V>
__global__ void fuse_init_kernel(const __grid_constant__ FuseArgs a) {
    const int j0 = (blockIdx.x * blockDim.x + threadIdx.x) * V, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.H || j0 >= a.W) return;
    const size_t idx = (size_t)i * a.W + j0;
    const float *D0 = a.depths[0];
    const Vec<V, float> d = load_vec<V>(D0 + idx);
    Vec<V, float> up, down;
    const bool has_up = i - 1 > 0, has_down = i + 1 < a.H;
    if (has_up) up = load_vec<V>(D0 + idx - a.W);
    if (has_down) down = load_vec<V>(D0 + idx + a.W);
    const float left = j0 - 1 > 0 ? D0[idx - 1] : 1.0f, right = j0 + V < a.W ? D0[idx + V] : 1.0f;
    Vec<V, uint8_t> alive;
    Vec<V, float> pruned;
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const int j = j0 + k;
        bool f = d.v[k] == 0.0f;
        if (has_up) f = f || up.v[k] == 0.0f;
        if (has_down) f = f || down.v[k] == 0.0f;
        if (j - 1 > 0) f = f || (k ? d.v[k ? k - 1 : 0] : left) == 0.0f;
        if (j + 1 < a.W) f = f || (k + 1 < V ? d.v[k + 1 < V ? k + 1 : 0] : right) == 0.0f;
        alive.v[k] = f ? 0 : 1;
        pruned.v[k] = f ? 0.0f : d.v[k];
    }
    store_vec(a.alive + idx, alive);
    store_vec(a.pruned + idx, pruned);
}

template <int V>
__global__ void fuse_classify_kernel(const __grid_constant__ FuseArgs a, int k) {
    const int j0 = (blockIdx.x * blockDim.x + threadIdx.x) * V, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.H || j0 >= a.W) return;
    const size_t idx = (size_t)i * a.W + j0;
    const Vec<V, uint8_t> alive = load_vec<V>(a.alive + idx);
    const Vec<V, float> d = load_vec<V>(a.depths[0] + idx);
    const float2 rt = a.row_trig[i];
    const float *M = a.M[k], *c = a.c[k];
    Vec<V, int> q;
    Vec<V, int8_t> cls;
    float dop[V], dat[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        q.v[v] = -1;
        if (alive.v[v]) {
            const float2 ct = a.col_trig[j0 + v];
            const float Xc = d.v[v] * rt.x * ct.x, Yc = -d.v[v] * rt.y, Zc = d.v[v] * rt.x * ct.y;
            const float X = M[0] * Xc + M[1] * Yc + M[2] * Zc + c[0];
            const float Y = M[3] * Xc + M[4] * Yc + M[5] * Zc + c[1];
            const float Z = M[6] * Xc + M[7] * Yc + M[8] * Zc + c[2];
            float x, y;
            if (project(X, Y, Z, (float)a.W, (float)a.H, x, y, dop[v])) {
                const int iu = (int)x, iv = (int)y;
                if (iv >= 0 && iv < a.H && iu >= 0 && iu < a.W && !(dop[v] < 1e-5f)) q.v[v] = iv * a.W + iu;
            }
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) dat[v] = q.v[v] >= 0 ? a.depths[k][q.v[v]] : 0.0f;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        cls.v[v] = kSkip;
        if (q.v[v] >= 0 && !(dat[v] == 0.0f || fabsf(dat[v] - dop[v]) > a.thr * dop[v])) {
            cls.v[v] = d.v[v] < dat[v] ? kZero : kDrop;
            if (cls.v[v] == kZero) atomicMin(a.first + q.v[v], (unsigned)(idx + v));
        }
    }
    store_vec(a.cls + idx, cls);
    store_vec(a.target + idx, q);
}

template <int V>
__global__ void fuse_resolve_kernel(const __grid_constant__ FuseArgs a, int k) {
    const int j0 = (blockIdx.x * blockDim.x + threadIdx.x) * V, i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= a.H || j0 >= a.W) return;
    const size_t idx = (size_t)i * a.W + j0;
    const Vec<V, int8_t> cls = load_vec<V>(a.cls + idx);
    const Vec<V, int> q = load_vec<V>(a.target + idx);
    unsigned first[V];
#pragma unroll
    for (int v = 0; v < V; ++v) first[v] = cls.v[v] != kSkip ? a.first[q.v[v]] : 0u;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const unsigned me = (unsigned)(idx + v);
        if (cls.v[v] == kSkip || me > first[v]) continue;  // target already zeroed: skipped
        if (me == first[v]) {                              // first qualifying nearer pixel zeroes it
            a.depths[k][q.v[v]] = 0.0f;
        } else if (cls.v[v] == kDrop) {                    // sees the original, farther-or-equal: dropped
            a.alive[me] = 0;
            a.pruned[me] = 0.0f;
        }
    }
}

// Kept pixels of compaction block b (kCompactBlock consecutive pixels): 64
// threads with 16 flags each, four blocks per CTA.
__global__ void __launch_bounds__(256) compact_count_kernel(const uint8_t *alive, size_t N, unsigned *counts) {
    __shared__ unsigned part[8];
    const size_t i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 16;
    unsigned c = 0;
    if (i + 16 <= N) {
        const uint4 w = *reinterpret_cast<const uint4 *>(alive + i);  // flags are 0 or 1
        c = __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
    } else {
        for (size_t k = i; k < N; ++k) c += alive[k];
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
    __syncthreads();
    const unsigned b = blockIdx.x * 4 + threadIdx.x;
    if (threadIdx.x < 4 && (size_t)b * kCompactBlock < N) counts[b] = part[2 * threadIdx.x] + part[2 * threadIdx.x + 1];
}
static_assert(kCompactBlock == 1024, "compact_count_kernel sums 64 x 16 flags per block");

// Inclusive prefix sum over a warp.
__device__ __forceinline__ unsigned warp_scan(unsigned v) {
    const unsigned lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= (unsigned)off) v += t;
    }
    return v;
}

// exclusive scan of nb block counts (single block of 1024, four counts per
// thread and step); counts[nb] = total
__global__ void __launch_bounds__(1024) compact_scan_kernel(unsigned *counts, int nb, unsigned *total) {
    __shared__ unsigned warp_tot[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned carry = 0;
    for (int base = 0; base < nb; base += 4096) {
        const int i = base + 4 * (int)threadIdx.x;
        unsigned v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = i + k < nb ? counts[i + k] : 0u;
            sum += v[k];
        }
        const unsigned inc = warp_scan(sum);
        if (lane == 31) warp_tot[wid] = inc;
        __syncthreads();
        const unsigned all = warp_scan(warp_tot[lane]);  // every warp scans the warp totals
        const unsigned before = wid ? __shfl_sync(0xffffffffu, all, wid - 1) : 0u;
        unsigned run = carry + before + inc - sum;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i + k < nb) counts[i + k] = run;
            run += v[k];
        }
        carry += __shfl_sync(0xffffffffu, all, 31);
        __syncthreads();  // before the next step replaces warp_tot
    }
    if (threadIdx.x == 0) {
        counts[nb] = carry;
        *total = carry;
    }
}

// Points of compaction block blockIdx.x, in two steps: the kept pixels of the
// block are listed in order (256 threads with 4 flags each), then thread t
// writes the points t, t + 256, ..., so that the lanes of a warp write
// neighbouring points whatever the share of kept pixels.  3840x1920, one pixel
// per thread / four neighbours per thread (whose stores lie 48 bytes apart) /
// every 256th pixel per thread / this: all pixels kept 59 / 113 / 36 / 36 us, 58 %
// kept 46 / 72 / 26 / 27, 10 % kept, with colours, 28 / 27 / 17 / 19, noisy maps with
// few kept 38 / 19 / 21 / 16.
__global__ void __launch_bounds__(256) compact_scatter_kernel(const __grid_constant__ FuseArgs a) {
    __shared__ unsigned warp_tot[8];
    __shared__ uint16_t list[kCompactBlock];  // offsets of the kept pixels in the block
    const size_t N = (size_t)a.W * a.H, base = (size_t)blockIdx.x * kCompactBlock;
    const unsigned t4 = 4 * threadIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Vec<4, uint8_t> keep = {};
    if (base + t4 + 4 <= N) {
        keep = load_vec<4>(a.alive + base + t4);
    } else {
        for (int k = 0; k < 4; ++k)
            if (base + t4 + k < N) keep.v[k] = a.alive[base + t4 + k];
    }
    const unsigned cnt = keep.v[0] + keep.v[1] + keep.v[2] + keep.v[3];
    const unsigned inc = warp_scan(cnt);
    if (lane == 31) warp_tot[wid] = inc;
    __syncthreads();
    unsigned at = inc - cnt, total = 0;
#pragma unroll
    for (unsigned w = 0; w < 8; ++w) {
        at += w < wid ? warp_tot[w] : 0u;
        total += warp_tot[w];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (keep.v[k]) list[at++] = (uint16_t)(t4 + k);
    __syncthreads();
    const size_t first = a.block_counts[blockIdx.x], row0 = base / a.W;
    const unsigned col0 = (unsigned)(base - row0 * a.W);
#pragma unroll
    for (unsigned k = 0; k < 4; ++k) {
        const unsigned e = 256 * k + threadIdx.x;
        if (e >= total) break;
        const unsigned off = list[e], down = (col0 + off) / (unsigned)a.W;
        const int row = (int)(row0 + down), col = (int)(col0 + off - down * (unsigned)a.W);
        const size_t i = base + off, pos = first + e;
        const float d = a.depths[0][i];
        const float2 rt = a.row_trig[row], ct = a.col_trig[col];
        const float Xc = d * rt.x * ct.x, Yc = -d * rt.y, Zc = d * rt.x * ct.y;
        a.xyz[3 * pos] = a.Rinv[0] * Xc + a.Rinv[1] * Yc + a.Rinv[2] * Zc + a.tw[0];
        a.xyz[3 * pos + 1] = a.Rinv[3] * Xc + a.Rinv[4] * Yc + a.Rinv[5] * Zc + a.tw[1];
        a.xyz[3 * pos + 2] = a.Rinv[6] * Xc + a.Rinv[7] * Yc + a.Rinv[8] * Zc + a.tw[2];
        if (a.bgr_out && a.bgr) {
            a.bgr_out[3 * pos] = a.bgr[3 * i];
            a.bgr_out[3 * pos + 1] = a.bgr[3 * i + 1];
            a.bgr_out[3 * pos + 2] = a.bgr[3 * i + 2];
        }
        if (a.ij_out) {
            a.ij_out[2 * pos] = row;
            a.ij_out[2 * pos + 1] = col;
        }
    }
}

}  // namespace

void launch_postprocess(cudaStream_t st, const PostArgs &a) {
    dim3 b(32, 8), g((a.W + 31) / 32, (a.H + 7) / 8);
    post_window_kernel<<<g, b, 0, st>>>(a);
    median_kernel<<<g, b, 0, st>>>(a.d0, a.m1, a.W, a.H);
    post_threshold_kernel<<<g, b, 0, st>>>(a);
}

void launch_export(cudaStream_t st, const float4 *plane, const float *score, const int8_t *best,
                   const float *filt_depth, const float *filt_score, const float2 *row_trig, const float2 *col_trig,
                   int W, int H, int raw, float *depth, float *score_out, float *plane3, float *normal3,
                   int32_t *best32) {
    dim3 b(32, 8), g((W + 31) / 32, (H + 7) / 8);
    export_kernel<<<g, b, 0, st>>>(plane, score, best, filt_depth, filt_score, row_trig, col_trig, W, H, raw, depth,
                                   score_out, plane3, normal3, best32);
}

void clean_set_poses(CleanArgs &a, int n, const double *R, const double *t, int center, int *order) {
    order[0] = center;
    for (int k = 0, s = 1; k < n; ++k)
        if (k != center) order[s++] = k;
    const double *R0 = R + 9 * center, *t0 = t + 3 * center;
    for (int s = 1; s < n; ++s) {
        const int k = order[s];
        compose_pose(R0, t0, R + 9 * k, t + 3 * k, a.M[s], a.c[s]);
        compose_pose(R + 9 * k, t + 3 * k, R0, t0, a.Minv[s], a.cinv[s]);
    }
    a.n = n;
}

void launch_clean(cudaStream_t st, const CleanArgs &a) {
    dim3 b(32, 8), g((a.W + 31) / 32, (a.H + 7) / 8);
    clean_kernel<<<g, b, 0, st>>>(a);
}

namespace {
inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }
inline int compact_blocks(int W, int H) { return (int)(((size_t)W * H + kCompactBlock - 1) / kCompactBlock); }
}  // namespace

size_t fuse_workspace_bytes(int W, int H) {
    const size_t N = (size_t)W * H;
    return al256(N) + al256(N * 4) + al256(N) + al256(N * 4) + al256((size_t)(compact_blocks(W, H) + 1) * 4);
}

void fuse_bind_workspace(FuseArgs &a, void *ws) {
    const size_t N = (size_t)a.W * a.H;
    char *p = static_cast<char *>(ws);
    auto take = [&](size_t b) { char *q = p; p += al256(b); return q; };
    a.alive = reinterpret_cast<uint8_t *>(take(N));
    a.target = reinterpret_cast<int *>(take(N * 4));
    a.cls = reinterpret_cast<int8_t *>(take(N));
    a.first = reinterpret_cast<unsigned *>(take(N * 4));
    a.block_counts = reinterpret_cast<unsigned *>(take((size_t)(compact_blocks(a.W, a.H) + 1) * 4));
}

void fuse_set_poses(FuseArgs &a, int n, const double *R, const double *t) {
    for (int k = 1; k < n; ++k) compose_pose(R, t, R + 9 * k, t + 3 * k, a.M[k], a.c[k]);
    for (int r0 = 0; r0 < 3; ++r0) {
        for (int c0 = 0; c0 < 3; ++c0) a.Rinv[3 * r0 + c0] = (float)R[3 * c0 + r0];
        a.tw[r0] = (float)(-(R[r0] * t[0] + R[3 + r0] * t[1] + R[6 + r0] * t[2]));
    }
    a.n = n;
}

namespace {
// Four pixels per thread where every row of every map starts on a 16-byte
// boundary and the map has this many pixels.  Below, the chip holds one pixel
// per thread in some two waves, and a thread's four projections in a row only
// add latency.  All kernels of a fusion, one -> four pixels per thread, us:
// 5 views 260x130 29.2 -> 37.1, 960x480 42.8 -> 48.0, 1152x576 (663,552 pixels)
// 50.5 -> 53.3, 1216x608 (739,328) 52.6 -> 52.0, 1280x640 55.7 -> 54.8, 1920x960
// 101 -> 92; 8 views 260x130 45.3 -> 57.5, 1152x576 71.4 -> 75.1, 1216x608 75.4 ->
// 72.9; 2 views 260x130 14.0 -> 16.2, 1216x608 29.9 -> 30.2, 1536x768 40.0 -> 38.1.
constexpr size_t kFuseVecPixels = 700000;

bool fuse_vector(const FuseArgs &a) {
    if (a.W % 4 || (size_t)a.W * a.H < kFuseVecPixels) return false;
    uintptr_t p = (uintptr_t)a.pruned | (uintptr_t)a.target | (uintptr_t)a.depths[0];
    return (p & 15) == 0 && (((uintptr_t)a.alive | (uintptr_t)a.cls) & 3) == 0;
}

template <int V>
cudaError_t launch_fuse_views(cudaStream_t st, const FuseArgs &a) {
    const dim3 b(32, 8), g((a.W + 32 * V - 1) / (32 * V), (a.H + 7) / 8);
    const size_t N = (size_t)a.W * a.H;
    fuse_init_kernel<V><<<g, b, 0, st>>>(a);
    for (int k = 1; k < a.n; ++k) {
        const cudaError_t e = cudaMemsetAsync(a.first, 0xFF, N * sizeof(unsigned), st);
        if (e != cudaSuccess) return e;
        fuse_classify_kernel<V><<<g, b, 0, st>>>(a, k);
        fuse_resolve_kernel<V><<<g, b, 0, st>>>(a, k);
    }
    return cudaSuccess;
}
}  // namespace

cudaError_t launch_fuse(cudaStream_t st, const FuseArgs &a) {
    const size_t N = (size_t)a.W * a.H;
    const cudaError_t e = fuse_vector(a) ? launch_fuse_views<4>(st, a) : launch_fuse_views<1>(st, a);
    if (e != cudaSuccess) return e;
    const int nb = compact_blocks(a.W, a.H);
    compact_count_kernel<<<(nb + 3) / 4, 256, 0, st>>>(a.alive, N, a.block_counts);
    compact_scan_kernel<<<1, 1024, 0, st>>>(a.block_counts, nb, a.count);
    compact_scatter_kernel<<<nb, 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace pm
