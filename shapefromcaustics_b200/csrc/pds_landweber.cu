// Projected Landweber update of the height-field offset, fused (sm_100a).
//
// The reference's per-iteration update (shape_from_caustics.py:386-398, default options):
//   d = d - tau * grad                                  (gradient step, :387)
//   d = mask * extShrink(d, tau * alpha, lower, upper)  (:397, extShrink :184-189)
//   d = VconsHeur(d, d1, d2, mask, gamma, r)            (:398, VconsHeur :228-241)
// with extShrink(x) = clamp(max(|x| - a, 0) sign(x), lower, upper) and
// VconsHeur: v = sum(d); m = (2r+1)^2 box mean of d (zero padded, count_include_pad);
//   v <= d1: d += mask m sin(v/d1 pi) gamma;  v >= d2: d -= mask m sin((v/d2 - 1) pi) gamma.
// Two kernels: (1) step + shrink + mask into a scratch image, with per-block partial sums;
// (2) every block reduces the partial sums in a fixed order (deterministic v), then applies
// the volume heuristic with the box mean of the scratch image. The reference's volume test
// is a host-side branch on a device scalar; here it stays on the device.
#include <cstdint>
#include <mutex>
#include <cuda_runtime.h>

#include "../../include/pds_b200.h"
#include "pds_internal.h"

namespace pds {
namespace {

constexpr int kThreads = 256;
constexpr float kPi = 3.14159265358979323846f;

__device__ __forceinline__ float ext_shrink(float x, float a, float lo, float hi) {
    const float s = x > 0.f ? 1.f : (x < 0.f ? -1.f : 0.f);
    const float v = fmaxf(fabsf(x) - a, 0.f) * s;
    return fmaxf(fminf(v, hi), lo);
}

__global__ __launch_bounds__(kThreads) void lw_shrink_kernel(const float* __restrict__ d,
                                                             const float* __restrict__ g,
                                                             const float* __restrict__ mask,
                                                             int64_t n, pds_landweber p,
                                                             float* __restrict__ t,
                                                             float* __restrict__ partial) {
    __shared__ float red[kThreads / 32];
    float acc = 0.f;
    const int64_t stride = int64_t(gridDim.x) * kThreads;
    const int64_t first = int64_t(blockIdx.x) * kThreads + threadIdx.x;
    // four pixels at a time where every array starts on 16 bytes, then the last n % 4
    const bool quads = ((reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(g) |
                         reinterpret_cast<uintptr_t>(mask) | reinterpret_cast<uintptr_t>(t)) & 15) == 0;
    const int64_t nq = quads ? n >> 2 : 0;
    const auto step = [&](float x, float gv, float mv) {
        return mv * ext_shrink(x - p.tau * gv, p.shrink, p.lower, p.upper);
    };
    for (int64_t i = first; i < nq; i += stride) {
        const float4 x = reinterpret_cast<const float4*>(d)[i];
        const float4 gv = reinterpret_cast<const float4*>(g)[i];
        const float4 mv = reinterpret_cast<const float4*>(mask)[i];
        const float4 v = make_float4(step(x.x, gv.x, mv.x), step(x.y, gv.y, mv.y),
                                     step(x.z, gv.z, mv.z), step(x.w, gv.w, mv.w));
        reinterpret_cast<float4*>(t)[i] = v;
        acc += (v.x + v.y) + (v.z + v.w);
    }
    for (int64_t i = 4 * nq + first; i < n; i += stride) {
        const float v = step(d[i], g[i], mask[i]);
        t[i] = v;
        acc += v;
    }
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
        for (int w = 0; w < kThreads / 32; ++w) s += red[w];
        partial[blockIdx.x] = s;
    }
}

// The factor of the volume heuristic's box mean, 0 where the volume is inside (d1, d2). All
// threads of the CTA call it; every CTA sums the partial sums in the same order (a thread's
// share, then a warp's by shuffles, then the warps'). (One thread adding 256 shared values in
// turn took 4 us of every CTA.)
__device__ __forceinline__ float volume_coef(const float* __restrict__ partial, int nparts,
                                             const pds_landweber& p) {
    __shared__ float red[kThreads / 32];
    float s = 0.f;
    for (int k = threadIdx.x; k < nparts; k += kThreads) s += partial[k];
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) v += red[w];
    if (v <= p.d1) return sinf(v / p.d1 * kPi) * p.gamma;
    if (v >= p.d2) return -sinf((v / p.d2 - 1.f) * kPi) * p.gamma;
    return 0.f;
}

// Volume heuristic of a tile of kTileW x kTileH pixels a CTA, for box radii up to kTileRadius: the
// tile and its margin are read once into shared memory and the box is summed along rows, then
// along columns, so a pixel costs 2 (2 r + 1) shared reads. Bound by launch and L2 latency at
// the sizes fields have (1024^2: 4 MB an array, L2-resident); read per pixel through the cache
// with a 64-bit division for its row, the same box took 28 us there.
constexpr int kTileW = 64, kTileH = 16, kTileRadius = 8;

__global__ __launch_bounds__(kThreads) void lw_volume_tile_kernel(
    const float* __restrict__ t, const float* __restrict__ mask, int rows, int cols,
    pds_landweber p, const float* __restrict__ partial, int nparts, float* __restrict__ d) {
    __shared__ float in[(kTileH + 2 * kTileRadius) * (kTileW + 2 * kTileRadius)];
    __shared__ float across[(kTileH + 2 * kTileRadius) * kTileW];
    const int x0 = blockIdx.x * kTileW, y0 = blockIdx.y * kTileH;
    const int tx = threadIdx.x % kTileW, ty = threadIdx.x / kTileW;
    constexpr int kStep = kThreads / kTileW;
    const int r = p.radius, w = kTileW + 2 * r, h = kTileH + 2 * r;
    // the tile's loads do not wait for the volume (nothing but the pixels themselves is needed
    // where the heuristic does not act, which is not known yet), nor for one another:
    // asynchronous copies, zero-filled outside the field
    for (int y = ty; y < h; y += kStep) {
        const int gy = y0 - r + y;
        const bool row = gy >= 0 && gy < rows;
        for (int x = tx; x < w; x += kTileW) {
            const int gx = x0 - r + x;
            const bool inside = row && gx >= 0 && gx < cols;
            const float* src = inside ? t + int64_t(gy) * cols + gx : t;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                         :: "r"(uint32_t(__cvta_generic_to_shared(in + y * w + x))), "l"(src),
                            "r"(inside ? 4 : 0)
                         : "memory");
        }
    }
    float m[kTileH / kStep];
#pragma unroll
    for (int k = 0; k < kTileH / kStep; ++k) {
        const int gy = y0 + ty + k * kStep;
        m[k] = gy < rows && x0 + tx < cols ? mask[int64_t(gy) * cols + x0 + tx] : 0.f;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const float coef = volume_coef(partial, nparts, p);  // (with a barrier)
    if (coef == 0.f) {
        for (int y = ty; y < kTileH; y += kStep)
            if (y0 + y < rows && x0 + tx < cols)
                d[int64_t(y0 + y) * cols + x0 + tx] = in[(y + r) * w + tx + r];
        return;
    }
    for (int y = ty; y < h; y += kStep) {
        float s = 0.f;
        for (int k = 0; k <= 2 * r; ++k) s += in[y * w + tx + k];
        across[y * kTileW + tx] = s;
    }
    __syncthreads();
    const float scale = coef / float((2 * r + 1) * (2 * r + 1));
#pragma unroll
    for (int j = 0; j < kTileH / kStep; ++j) {
        const int y = ty + j * kStep;
        float s = 0.f;
        for (int k = 0; k <= 2 * r; ++k) s += across[(y + k) * kTileW + tx];
        if (y0 + y < rows && x0 + tx < cols)
            d[int64_t(y0 + y) * cols + x0 + tx] = in[(y + r) * w + tx + r] + m[j] * (s * scale);
    }
}

// The same for any radius, a pixel a thread.
__global__ __launch_bounds__(kThreads) void lw_volume_kernel(const float* __restrict__ t,
                                                             const float* __restrict__ mask,
                                                             int64_t rows, int64_t cols,
                                                             pds_landweber p,
                                                             const float* __restrict__ partial,
                                                             int nparts, float* __restrict__ d) {
    const float coef = volume_coef(partial, nparts, p);
    const int r = p.radius;
    const float inv_area = 1.f / float((2 * r + 1) * (2 * r + 1));
    const int64_t n = rows * cols;
    const int64_t stride = int64_t(gridDim.x) * kThreads;
    for (int64_t i = int64_t(blockIdx.x) * kThreads + threadIdx.x; i < n; i += stride) {
        const float x = t[i];
        if (coef == 0.f) {
            d[i] = x;
            continue;
        }
        const int64_t y = i / cols, xx = i - y * cols;
        float box = 0.f;
        for (int dy = -r; dy <= r; ++dy) {
            const int64_t yy = y + dy;
            if (yy < 0 || yy >= rows) continue;
            for (int dx = -r; dx <= r; ++dx) {
                const int64_t xc = xx + dx;
                if (xc < 0 || xc >= cols) continue;
                box += t[yy * cols + xc];
            }
        }
        d[i] = x + mask[i] * (box * inv_area) * coef;
    }
}

// Fixed block count (independent of the device, so the scratch size is too): grid-stride
// loops cover any image size. Every CTA of the second kernel reads all partial sums, so no more
// blocks than a resident wave or two of the four-pixel loop.
int lw_blocks(int64_t n) {
    const int64_t b = (n + 4 * kThreads - 1) / (4 * kThreads);
    return int(b < 512 ? (b > 0 ? b : 1) : 512);
}

}  // namespace

size_t landweber_scratch_bytes(int64_t n) {
    return align_up(size_t(n > 0 ? n : 1) * sizeof(float), 256) + size_t(lw_blocks(n)) * sizeof(float);
}

cudaError_t launch_landweber(float* d, const float* g, const float* mask, int64_t rows,
                             int64_t cols, const pds_landweber& p, float* t, float* partial,
                             cudaStream_t st) {
    const int64_t n = rows * cols;
    if (n <= 0) return cudaSuccess;
    const int nb = lw_blocks(n);
    lw_shrink_kernel<<<nb, kThreads, 0, st>>>(d, g, mask, n, p, t, partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // the tile kernel indexes rows and columns in 32 bits and puts row tiles on the grid's second
    // axis (at most 65535)
    const int64_t tiles_y = (rows + kTileH - 1) / kTileH;
    if (p.radius >= 0 && p.radius <= kTileRadius && tiles_y <= 65535 && cols <= (int64_t(1) << 30)) {
        const dim3 grid(unsigned((cols + kTileW - 1) / kTileW), unsigned(tiles_y));
        lw_volume_tile_kernel<<<grid, kThreads, 0, st>>>(t, mask, int(rows), int(cols), p, partial,
                                                         nb, d);
    } else {
        lw_volume_kernel<<<nb, kThreads, 0, st>>>(t, mask, rows, cols, p, partial, nb, d);
    }
    return cudaGetLastError();
}

// ---- the allocation-free variant -------------------------------------------------------
// Scratch of pds_landweber_update_noalloc_f32: the shrunk image (up to kNoAllocMaxPixels
// floats) followed by the per-block partial sums (at most 1024 floats, see lw_blocks).
// Every GPU that loads this library holds it (4 MiB + 4 KiB) until the process exits.
constexpr int64_t kNoAllocMaxPixels = int64_t(1) << 20;  // 1024 x 1024
constexpr size_t kNoAllocImageBytes = size_t(kNoAllocMaxPixels) * sizeof(float);
constexpr size_t kNoAllocBytes = kNoAllocImageBytes + 1024 * sizeof(float);
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

int64_t landweber_noalloc_max_pixels() { return kNoAllocMaxPixels; }

// Device addresses of the scratch's two parts on the current device: the shrunk image `t`
// (kNoAllocMaxPixels floats) and the per-block partial sums `partial` right after it. In host
// code the symbol is only a host-side stand-in, so the array's address is looked up once per
// device (with that device current) and cached.
cudaError_t landweber_noalloc_scratch(float** t, float** partial) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static void* addr[kMaxDevices] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (addr[dev] == nullptr) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        addr[dev] = p;
    }
    unsigned char* base = static_cast<unsigned char*>(addr[dev]);
    *t = reinterpret_cast<float*>(base);
    *partial = reinterpret_cast<float*>(base + kNoAllocImageBytes);
    return cudaSuccess;
}

}  // namespace pds
