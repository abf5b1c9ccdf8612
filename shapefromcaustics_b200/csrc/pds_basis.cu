// Splat inputs of traced photons from their receiver-plane differentials, and their backward
// (sm_100a).
//
// Reference: model/caustics.py:224-239 (change_of_basis_matrix, splat_photons): with T = Dv x n,
// S = n x Du and den = Du . T,
//   Mp = 2 / den [T ; S],  radius = max(|Du|, |Dv|) / 2,  Ep = 4 flux / |Du x Dv|,
// and photons with den = 0 (dropped there) keep their slot with channel -1.
//
// Bound by memory: one thread a photon reads each input once and writes each output once (88 B
// forward). As torch operations the same took some thirty launches forward and backward
// (2.8 10^5 photons: 230 us of device time spread over 600 us of host time). The backward reads
// the splat gradients where the splat backward left them, in the plan's records, so their spread
// into grad_Ep / grad_Mp and its re-read do not happen.
#include <cstdint>
#include <cuda_runtime.h>

#include "pds_device.cuh"
#include "pds_internal.h"

namespace pds {
namespace {

struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 load3(const float* p, int64_t n, int64_t i) {
    return {p[i], p[n + i], p[2 * n + i]};
}
__device__ __forceinline__ void store3(float* p, int64_t n, int64_t i, V3 v) {
    p[i] = v.x;
    p[n + i] = v.y;
    p[2 * n + i] = v.z;
}
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 scale(float s, V3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ V3 add(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }

__global__ __launch_bounds__(256) void basis_fwd_kernel(BasisArgs a) {
    const int64_t n = a.n;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        const V3 u = load3(a.Du, n, i), v = load3(a.Dv, n, i), m = load3(a.normal, n, i);
        const V3 t = cross(v, m), s = cross(m, u);
        const float den = dot(u, t);
        const bool good = den != 0.f;
        const float f = 2.f / (good ? den : 1.f);
        store3(a.Mp, n, i, scale(f, t));
        store3(a.Mp + 3 * n, n, i, scale(f, s));
        a.radius[i] = 0.5f * fmaxf(sqrtf(dot(u, u)), sqrtf(dot(v, v)));
        const V3 c = cross(u, v);
        a.Ep[i] = a.flux[i] / (good ? sqrtf(dot(c, c)) : 1.f) * 4.f;
        a.cp[i] = good ? a.channel[i] : -1;
    }
}

__global__ __launch_bounds__(256) void basis_bwd_kernel(BasisArgs a) {
    const int64_t n = a.n;
    const int64_t n_tile = min(int64_t(__ldg(a.rec_counters)), n);
    const V3 zero = {0.f, 0.f, 0.f};
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        // the photon's record (none: it touches no pixel, and all its gradients are zero)
        const uint32_t r = __ldg(a.rec_inv + i);
        const int64_t slot = (r & kWideBit) ? n_tile + int64_t(r & ~kWideBit) : int64_t(r);
        const bool have = r != kInvalidPos && slot < n;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (have) {
            const Words8 w = load_words8(a.rec_stage + 2 * slot);
            lo = w.lo;
            hi = w.hi;
        }
        const float gE = lo.x;
        a.gX[i] = lo.y;
        a.gX[n + i] = lo.z;
        const V3 u = load3(a.Du, n, i), v = load3(a.Dv, n, i), m = load3(a.normal, n, i);
        const V3 t = cross(v, m), c = cross(u, v);
        const float den = dot(u, t), area = sqrtf(dot(c, c));
        V3 gu = zero, gv = zero, gm = zero;
        float gf = 0.f;
        if (have && den != 0.f) {
            const V3 s = cross(m, u);
            const V3 g0 = {lo.w, hi.x, 0.f}, g1 = {hi.y, hi.z, 0.f};  // (Mp's third column is unused)
            const float f = 2.f / den;
            // Mp = f [t ; s], f = 2 / den, den = u . t, t = v x m, s = m x u
            const float gden = -(f / den) * (dot(g0, t) + dot(g1, s));
            const V3 gt = add(scale(f, g0), scale(gden, u)), gs = scale(f, g1);
            gu = add(scale(gden, t), cross(gs, m));
            gv = cross(m, gt);
            // Ep = 4 flux / area, area = |u x v| (no direction at 0, as for torch's norm)
            gf = 4.f / area * gE;
            if (area > 0.f) {
                const V3 gc = scale(-(a.flux[i] * gf) / (area * area), c);
                gu = add(gu, cross(v, gc));
                gv = add(gv, cross(gc, u));
            }
            if (a.gN) gm = add(cross(gt, v), cross(u, gs));
        }
        if (a.gDu) store3(a.gDu, n, i, gu);
        if (a.gDv) store3(a.gDv, n, i, gv);
        if (a.gN) store3(a.gN, n, i, gm);
        if (a.gflux) a.gflux[i] = gf;
    }
}

}  // namespace

cudaError_t launch_basis(bool backward, const BasisArgs& a, cudaStream_t st) {
    if (a.n <= 0) return cudaSuccess;
    const int64_t blocks = (a.n + 255) / 256, cap = int64_t(num_sms()) * 16;
    const unsigned grid = unsigned(blocks < cap ? blocks : cap);
    if (backward)
        basis_bwd_kernel<<<grid, 256, 0, st>>>(a);
    else
        basis_fwd_kernel<<<grid, 256, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace pds
