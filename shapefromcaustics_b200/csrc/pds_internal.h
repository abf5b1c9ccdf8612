// Internal (non-ABI) declarations shared by the library's translation units.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/pds_b200.h"

namespace pds {

inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Photons per tile-kernel work chunk of a call with n photons: the configured chunk, lowered for
// small photon counts so that every resident CTA of the tile kernels (3 per SM) gets about four
// chunks; at least 256 photons (one CTA-wide batch). The default chunk, whether a configuration
// names it or leaves it out, grows with the photon count, up to 8192, while 48 chunks an SM are left:
// a chunk ends with its tile's pixels added to the image or the next tile's staged, 6% of the
// forward at 2048 photons.
constexpr int32_t kDefaultChunk = 2048;
inline int32_t effective_chunk(int32_t chunk, int64_t n, int64_t sms) {
    const auto share = [&](int64_t per_sm) {
        const int64_t target = (n + sms * per_sm - 1) / (sms * per_sm);
        return (target + 255) / 256 * 256;
    };
    if (chunk == kDefaultChunk) chunk = int32_t(std::clamp<int64_t>(share(48), chunk, 8192));
    return int32_t(std::clamp<int64_t>(share(12), 256, chunk));
}

// The current device (0 where there is none).
inline int current_device() {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess ? dev : 0;
}

// Multiprocessors of the current device (148 where there is none), asked of the driver once per
// device: a fact of the hardware that every launch's grid needs.
inline int num_sms() {
    constexpr int kDevices = 64;
    static std::atomic<int> known[kDevices];
    const int dev = current_device();
    if (dev >= 0 && dev < kDevices) {
        const int k = known[dev].load(std::memory_order_relaxed);
        if (k > 0) return k;
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        return 148;
    if (dev >= 0 && dev < kDevices) known[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

// Lets a kernel use up to kMaxDynamicSmem bytes of dynamic shared memory (always the same
// limit, so that threads raising it for different launches cannot undo one another), once per
// device. A larger request fails here as its launch would.
constexpr size_t kMaxDynamicSmem = 226 * 1024;  // 227 KB less what the kernels hold statically
template <auto Kernel>
cudaError_t allow_smem(size_t smem) {
    constexpr int kDevices = 64;
    static std::atomic<bool> done[kDevices];
    if (smem <= 48 * 1024) return cudaSuccess;
    if (smem > kMaxDynamicSmem) return cudaErrorInvalidValue;
    const int dev = current_device();
    const bool cached = dev >= 0 && dev < kDevices;
    if (cached && done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(kMaxDynamicSmem));
    if (e == cudaSuccess && cached) done[dev].store(true, std::memory_order_release);
    return e;
}

// Resident CTAs of a kernel on one SM (at least 1) for a block size and dynamic shared memory:
// a function of the kernel and the device; the last answer per device is kept.
template <auto Kernel>
int resident_ctas(int threads, size_t smem) {
    constexpr int kDevices = 64;
    static std::atomic<uint64_t> last[kDevices];  // smem << 16 | threads' warps << 8 | CTAs
    const int dev = current_device();
    const bool cached = dev >= 0 && dev < kDevices;
    const uint64_t key = uint64_t(smem) << 16 | uint64_t(threads / 32) << 8;
    if (cached) {
        const uint64_t v = last[dev].load(std::memory_order_relaxed);
        if ((v & ~uint64_t(0xFF)) == key && (v & 0xFF)) return int(v & 0xFF);
    }
    int per_sm = 0;
    if (allow_smem<Kernel>(smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, Kernel, threads, smem) != cudaSuccess ||
        per_sm < 1)
        return 1;
    if (cached) last[dev].store(key | uint64_t(per_sm), std::memory_order_relaxed);
    return per_sm;
}

// refraction to the receiver (pds_refract.cu)
// A splat plan's per-photon gradient records (the backward's output before the spread into
// grad_Ep / grad_xp / grad_Mp): the inverse map, the 32-byte records, the plan's counters.
struct GradRecords {
    const uint32_t* inv;
    const float* stage;
    const uint32_t* counters;
};

// backward: the splat gradients from gE / gX / gM, or from rec when rec is non-null
cudaError_t launch_refract(bool backward, const float* h, int H, int W, const pds_plate& plate,
                           const pds_plate* plates, const int64_t* begins, int32_t n_sims,
                           const float* px, const float* py, const float* flux,
                           const int64_t* channel, int64_t n, float* Ep, float* xp, float* Mp,
                           int64_t* cp, float* radius, const float* gE, const float* gX,
                           const float* gM, float* gh, cudaStream_t st,
                           const GradRecords* rec = nullptr);

cudaError_t launch_refract_point(bool backward, const float* h, int H, int W,
                                 const pds_plate& plate, const pds_point_light& light,
                                 const float* dir, const float* dth, const float* dph,
                                 const float* flux, const int64_t* channel, int64_t n, float* Ep,
                                 float* xp, float* Mp, int64_t* cp, float* radius,
                                 const float* gE, const float* gX, const float* gM, float* gh,
                                 cudaStream_t st, const GradRecords* rec = nullptr);

// splat inputs of traced photons (pds_basis.cu); vectors [3][n]
struct BasisArgs {
    const float *Du, *Dv, *normal, *flux;
    int64_t n;
    // forward
    const int64_t* channel;
    float *Ep, *Mp, *radius;
    int64_t* cp;
    // backward: the plan's gradient records; gX [2][n], the others may be null (not wanted)
    const uint32_t* rec_inv;
    const float4* rec_stage;
    const uint32_t* rec_counters;
    float *gDu, *gDv, *gN, *gflux, *gX;
};
cudaError_t launch_basis(bool backward, const BasisArgs& a, cudaStream_t st);

// photon source (pds_source.cu)
cudaError_t launch_source(int32_t rows, int32_t cols, int32_t per_texel, float texel,
                          uint64_t seed, uint64_t offset, int64_t n, float* px, float* py,
                          cudaStream_t st);

cudaError_t launch_point_light(const pds_point_light& L, int64_t n_dir, uint64_t seed,
                               uint64_t offset, const float* coeffs, float* dir, float* dth,
                               float* dph, float* flux, cudaStream_t st);

// Landweber update (pds_landweber.cu)
size_t landweber_scratch_bytes(int64_t n);
cudaError_t launch_landweber(float* d, const float* g, const float* mask, int64_t rows,
                             int64_t cols, const pds_landweber& p, float* t, float* partial,
                             cudaStream_t st);
int64_t landweber_noalloc_max_pixels();
cudaError_t landweber_noalloc_scratch(float** t, float** partial);

}  // namespace pds
