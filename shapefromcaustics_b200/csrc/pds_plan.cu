// Photon binning of the splatting plan, for sm_100a.
//
// Reference: PyOptix/kernel/photon_differentials.cu:76-89 (the footprint each photon's
// threads recompute in both kernels). Here every photon is binned once per plan, by a
// counting sort over its bucket (simulation, channel, screen tile of the centre pixel,
// footprint class) in two passes over the photon inputs:
//
//   count pass       (coalesced SoA reads) the exact integer footprint and the bucket of every
//                    photon; each CTA takes a contiguous photon range (one or two simulations)
//                    and counts its buckets in a shared-memory histogram over the window of
//                    buckets (up to 32768) that starts at its first photon's simulation; the
//                    histogram is added into the global counts and kept per CTA. Photons wider
//                    than the apron go to the wide list.
//   bucket scan      exclusive scan of the bucket counts, giving each bucket its first sorted
//                    position; a copy serves as the place pass's cursors. Up to kFusedBuckets
//                    buckets every place CTA scans the counts itself (no kernel of its own), up
//                    to kOneScanBuckets one kernel does it, beyond that three.
//   place pass       the same CTA ranges: each CTA reserves its share of every bucket with one
//                    atomic on the bucket's cursor, hands positions out from shared memory,
//                    re-bins its photons and writes each one's 32-byte record at its position
//                    (one whole sector), keeping the position per photon (coalesced) for the
//                    backward's gradient spread. The photon placed first in a tile-kernel work
//                    chunk also writes down the chunk's tile.
//
// Nothing per photon is kept between the passes but the inverse map of wide and untouched
// photons: the place pass recomputes the keys from the inputs (40 bytes a photon read twice)
// instead of writing and reading back keys and photon-order records. Global atomics are per
// CTA and bucket rather than per photon (buckets outside a CTA's window, possible for
// simulations with more buckets than the window, take one global atomic per photon). Photons
// of one bucket land in an arbitrary order; every photon's result is independent of it
// (forward sums are reassociated, as the reference's atomics also do).
#include <cstdint>
#include <cuda_runtime.h>

#include "pds_device.cuh"
#include "pds_internal.h"
#include "pds_splat.h"

namespace pds {

namespace {

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Few large CTAs: the histogram flush and the cursor reservations cost one global atomic per
// CTA and touched bucket, so fewer, larger CTAs make fewer of them. A CTA of 768 threads gives
// each thread the registers to hold the next photon's inputs while it bins the current one
// (measured 3% faster than 1024 threads with one photon in flight).
constexpr int kPlanKernelThreads = 768;
// CTAs of a plan pass at most (each keeps its window histogram between the passes)
constexpr int64_t kPlanMaxCtas = 512;
// buckets of a CTA's shared histogram (128 KB: a 2048^2 image's buckets at 5 class bits; the
// SM keeps about 100 KB of L1 cache for the streamed loads)
constexpr int kMaxWindow = 32768;
// Buckets up to which every place CTA scans the counts itself (six a thread): a 512^2 image has
// 2048 at 5 class bits, two of them 4096. The scan's re-reads (16 KB a CTA from the L2) cost
// about a microsecond; the kernels they replace took 11 us a plan with their launches.
constexpr int kFusedPer = 6;
constexpr int64_t kFusedBuckets = int64_t(kFusedPer) * kPlanKernelThreads;
// Buckets up to which one kernel scans them, each CTA summing the counts before its own (at
// most 512 KB from the L2); beyond, the sums are formed once, by a kernel of their own.
constexpr int64_t kOneScanBuckets = 131072;

// Photons of a plan CTA at least: one per thread, and a quarter of its window's buckets, so that
// the window's clear and flush stay in proportion. (A fixed 8192 left small calls on a handful
// of CTAs, each running 11 photons a thread in a row: count and place together took 37 us for
// 2^14 photons and 46 us for 3 10^5.)
__host__ __device__ constexpr int64_t min_range(int64_t window) {
    const int64_t q = window / 4;
    return q <= kPlanKernelThreads
               ? kPlanKernelThreads
               : (q + kPlanKernelThreads - 1) / kPlanKernelThreads * kPlanKernelThreads;
}

// First bucket of a CTA's window: the first of the simulation owning its first photon i, or the
// first of all where the window holds every bucket.
__device__ __forceinline__ uint32_t window_base(const PlanArgs& a, int64_t i) {
    if (uint32_t(a.window) >= a.key_big) return 0u;
    return uint32_t(load_sim(a.sims, find_sim_of_photon(a.sims, i)).tile_base) << a.cfg.class_bits;
}

__device__ __forceinline__ void zero_window(uint32_t* hist, int window) {
    for (int j = threadIdx.x; j < window; j += blockDim.x) hist[j] = 0u;
}

// Clears a buffer by all CTAs of the grid: 16 bytes a store from its first 16-byte boundary on.
__device__ __forceinline__ void clear_image(float* p, int64_t n) {
    const int64_t head = min(int64_t((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / 4, n);
    const int64_t quads = (n - head) >> 2, tail = head + 4 * quads;
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    float4* q = reinterpret_cast<float4*>(p + head);
    for (int64_t k = t; k < quads; k += int64_t(gridDim.x) * blockDim.x)
        q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (t < head) p[t] = 0.f;
    if (tail + t < n) p[tail + t] = 0.f;
}

// What binning needs of a simulation, kept by each thread along its photons.
struct SimGeo {
    int32_t W, H, tiles_x, tiles_y, channels;
    uint32_t tile_base;
    float sx, sy;     // 2 / W, 2 / H
    double s2w, s2h;  // the same, for the corner offsets
    uint32_t end;     // first photon after the simulation's
};

__device__ __forceinline__ SimGeo load_geo(const SimTable& t, int s) {
    const pds_sim sim = load_sim(t, s);
    SimGeo g;
    g.W = sim.width;
    g.H = sim.height;
    g.tiles_x = sim.tiles_x;
    g.tiles_y = sim.tiles_y;
    g.channels = sim.channels;
    g.tile_base = uint32_t(sim.tile_base);
    g.s2w = corner_step(sim.width);
    g.s2h = corner_step(sim.height);
    g.sx = float(g.s2w);
    g.sy = float(g.s2h);
    g.end = uint32_t(min(sim_end(t, s), int64_t(UINT32_MAX)));
    return g;
}

// One photon's inputs.
struct PhotonIn {
    int64_t ch;
    float x, y, rad, e, m00, m01, m10, m11;
};

template <bool PLACE>
__device__ __forceinline__ PhotonIn load_photon(const PlanArgs& a, uint32_t i) {
    PhotonIn p;
    p.ch = __ldg(a.ph.cp + i);
    p.x = __ldg(a.ph.X + i);
    p.y = __ldg(a.Y + i);
    p.rad = __ldg(a.ph.R + i);
    p.m00 = __ldg(a.ph.M + i);
    p.m01 = __ldg(a.M01 + i);
    p.m10 = __ldg(a.M10 + i);
    p.m11 = __ldg(a.M11 + i);
    p.e = PLACE ? __ldg(a.ph.E + i) : 0.f;
    return p;
}

// The bucket of one photon (key_invalid, key_big, or (tile << cb) | class), for the tile path
// its box radius max(rx, ry) in rmax, and when PLACE its 32-byte record. Both passes run it on
// the same inputs, so they agree on every key. The passes are bound by instruction issue, so
// all but the reference's double-precision footprint is 32-bit integer and float work.
template <bool PLACE>
__device__ __forceinline__ uint32_t bin_photon(const PlanArgs& a, const SimGeo& g,
                                               const PhotonIn& p, Rec& r, int& rmax) {
    const int A = a.cfg.apron, cb = a.cfg.class_bits;
    const uint32_t cls_max = (1u << cb) - 1u;
    if (uint64_t(p.ch) >= uint64_t(g.channels)) return a.key_invalid;  // (negative ones too)
    const Footprint f = make_footprint(p.x, p.y, p.rad, g.H, g.W, a.mpr);
    if (f.rx < 0 || f.ry < 0) return a.key_invalid;
    // the clipped box; the centre is held within reach of 32 bits, far outside any image (an
    // empty box stays empty: tile-path radii are at most A), and wider footprints are clipped
    // in 64 bits
    if (f.rx > A || f.ry > A) {
        int32_t x0, x1, y0, y1;
        return clip_box(f, g.H, g.W, x0, x1, y0, y1) ? a.key_big : a.key_invalid;
    }
    const int pxc = min(max(f.px_c, -65536), 131072), pyc = min(max(f.py_c, -65536), 131072);
    const int x0 = max(pxc - f.rx, 0), x1 = min(pxc + f.rx, g.W - 1);
    const int y0 = max(pyc - f.ry, 0), y1 = min(pyc + f.ry, g.H - 1);
    if (x0 > x1 || y0 > y1) return a.key_invalid;
    rmax = max(f.rx, f.ry);
    // the tile edge is a power of two (16, 32 or 64, checked by the configuration), so the
    // tile of a (non-negative) centre pixel is a shift, not an integer division
    const int tx = min(max(pxc, 0), g.W - 1) >> a.tile_shift;
    const int ty = min(max(pyc, 0), g.H - 1) >> a.tile_shift;
    const uint32_t tile = g.tile_base + uint32_t((int32_t(p.ch) * g.tiles_y + ty) * g.tiles_x + tx);
    const float dy0 = corner_offset_step(f.py_c, g.s2h, p.y);
    uint32_t cls = min(uint32_t(rmax), cls_max);
    if (cb == kRowClassBits) {
        // the row walk's classes: rows and row width inside the box
        cls = f.ellipse_all ? plan_row_class(p.m00, p.m01, p.m10, p.m11, dy0, g.W, g.H, f.rx,
                                             x0 - pxc, x1 - pxc, y0 - pyc, y1 - pyc)
                            : cls_max;
    } else if (a.cfg.band) {
        // photons of a warp then have similar trip counts of the band walk: classes of 1/k octave
        // of its pixels, k = 1, 2, 3 for up to 3, 4 and 5 class bits
        int area = (2 * f.rx + 1) * (2 * f.ry + 1);
        if (f.ellipse_all)
            area = 2 * band_steps(p.m00 * g.sx, p.m01 * g.sy, p.m10 * g.sx, p.m11 * g.sy,
                                  dy0 * (0.5f * float(g.H)), f.rx, f.ry);
        // floor(k log2 area), from the exponent of area^k in float
        const int k = cb <= 3 ? 1 : cb - 2;
        const float a1 = float(max(area, 1));
        const float ak = k == 1 ? a1 : (k == 2 ? a1 * a1 : a1 * a1 * a1);
        const int lg = (__float_as_int(ak) >> 23) - 127;
        cls = min(uint32_t(max(lg - k, 0)), cls_max);
    }
    if (PLACE) {
        const uint32_t flags =
            (f.ellipse_all ? kFlagEllipseAll : 0u) | (p.e > 0.f ? 0u : kFlagFwdSkip);
        r.dx0 = corner_offset_step(f.px_c, g.s2w, p.x);
        r.dy0 = dy0;
        r.m00 = p.m00;
        r.m01 = p.m01;
        r.m10 = p.m10;
        r.m11 = p.m11;
        r.e = p.e;
        r.packed = pack_rec(pxc - ((tx << a.tile_shift) - A), pyc - ((ty << a.tile_shift) - A), f.rx,
                            f.ry, flags);
    }
    return (tile << cb) | cls;
}

// Exclusive scan of the counts of all buckets (at most kFusedPer a thread, the window holds
// them all) by one place CTA, then the reservation of the CTA's share: hist[j] = bucket j's
// first position + what other CTAs have taken before. CTA 0 writes the starts down for the
// tile kernels.
__device__ __forceinline__ void fused_scan(const PlanArgs& a, uint32_t* hist,
                                           const uint32_t* mine) {
    constexpr int kWarps = kPlanKernelThreads / 32;
    __shared__ uint32_t wsum[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b0 = int(threadIdx.x) * kFusedPer, nb = int(a.key_big);
    uint32_t v[kFusedPer], s = 0;
#pragma unroll
    for (int k = 0; k < kFusedPer; ++k) {
        v[k] = b0 + k < nb ? __ldcg(a.counts + b0 + k) : 0u;
        s += v[k];
    }
    uint32_t x = s;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    uint32_t run = x - s;
    for (int w = 0; w < warp; ++w) run += wsum[w];
#pragma unroll
    for (int k = 0; k < kFusedPer; ++k) {
        const int j = b0 + k;
        if (j < nb) {
            const uint32_t c = mine[j];
            hist[j] = c ? run + atomicAdd(a.cursor + j, c) : run;
            if (blockIdx.x == 0) a.start[j] = run;
        }
        run += v[k];
    }
    if (blockIdx.x == 0 && threadIdx.x == kPlanKernelThreads - 1) a.start[nb] = run;
}

// One pass of the plan over a CTA's contiguous photon range (coalesced SoA reads; each thread
// loads its next photon's inputs while it bins the current one).
//   count (PLACE = false): every photon's bucket into the CTA's shared histogram window (global
//       atomics for buckets outside it), the histogram added into the global counts and kept
//       per CTA in cta_hist; wide photons appended to the wide list; the inverse map of wide
//       and untouched photons.
//   place (PLACE = true, after the scan): the CTA reserves its share of every window bucket
//       with one atomic on the bucket's cursor (from its kept histogram), re-bins its photons,
//       builds each tile-path photon's record and writes it at its sorted position (one whole
//       32-byte sector), keeping the position in the inverse map. With few buckets (a.fused) it
//       first scans the counts itself; a.cursor then starts at zero and holds what the CTAs
//       have taken.
template <bool PLACE>
__global__ __launch_bounds__(kPlanKernelThreads) void plan_pass_kernel(PlanArgs a) {
    extern __shared__ uint32_t hist[];  // a.window buckets
    const int64_t n = a.ph.n;
    const int lane = threadIdx.x & 31;
    const int64_t r0 = int64_t(blockIdx.x) * a.range, r1 = min(r0 + a.range, n);
    const uint32_t kb0 = window_base(a, r0);
    const int64_t wend = min(int64_t(a.window), int64_t(a.key_big) - int64_t(kb0));
    uint32_t* mine = a.cta_hist + int64_t(blockIdx.x) * a.window;
    if (PLACE) {
        // hist[j] becomes the CTA's first position in window bucket j
        if (a.fused) {
            fused_scan(a, hist, mine);
        } else {
            for (int j = threadIdx.x; j < a.window; j += blockDim.x) {
                const uint32_t c = j < wend ? mine[j] : 0u;
                hist[j] = c ? atomicAdd(a.cursor + kb0 + j, c) : 0u;
            }
        }
    } else {
        zero_window(hist, a.window + a.window_tiles);
        // the image that the forward after this plan adds to: its stores ride along with the
        // pass, a memset of its own is a launch more (3 us of the host, 2 of the device)
        if (a.image) clear_image(a.image, a.image_elems);
    }
    __syncthreads();
    // the window's tiles' largest radii (kb0 is a tile's first bucket)
    uint32_t* radii = hist + a.window;
    uint32_t c_tile = 0, c_inv = 0;
    // The thread's simulation is followed along its photons (contiguous per simulation) rather
    // than searched per photon: one table load when a simulation boundary is crossed.
    const uint32_t end = uint32_t(r1);
    uint32_t i = uint32_t(r0) + threadIdx.x;
    int sidx = find_sim_of_photon(a.sims, min(int64_t(i), n - 1));
    SimGeo geo = load_geo(a.sims, sidx);
    PhotonIn next = {};
    if (i < end) next = load_photon<PLACE>(a, i);
    // whole warps step together (the wide list's ballot needs every lane)
    for (uint32_t base = uint32_t(r0); base < end; base += blockDim.x, i += blockDim.x) {
        const bool valid = i < end;
        const PhotonIn ph = next;
        if (i + blockDim.x < end) next = load_photon<PLACE>(a, i + blockDim.x);
        uint32_t key = a.key_invalid;
        int rmax = 0;
        Rec r;
        if (valid) {
            while (i >= geo.end) geo = load_geo(a.sims, ++sidx);  // at most the table's length in all
            key = bin_photon<PLACE>(a, geo, ph, r, rmax);
        }
        const bool tile_path = key < a.key_big;
        if (PLACE) {
            if (tile_path) {
                const uint32_t j = key - kb0;
                const uint32_t pos = j < uint32_t(a.window) ? atomicAdd(hist + j, 1u)
                                                           : atomicAdd(a.cursor + key, 1u);
                // both passes bin with the same code on the same inputs, so every position is
                // below the tile-path count; the guard keeps a mismatch inside the arrays
                if (pos < uint32_t(n)) {
                    store_rec(a.srecs + pos, r);
                    a.inv[i] = pos;
                    // the first photon of a work chunk (a multiple of 256 positions)
                    if ((pos & 255u) == 0u && pos % uint32_t(a.cfg.chunk) == 0u)
                        a.chunk_tile[pos / uint32_t(a.cfg.chunk)] = key >> a.cfg.class_bits;
                }
            }
            continue;
        }
        const bool wide = key == a.key_big;
        c_tile += tile_path;
        c_inv += valid && key == a.key_invalid;
        if (valid && key == a.key_invalid) a.inv[i] = kInvalidPos;
        if (tile_path) {
            const uint32_t j = key - kb0;
            if (j < uint32_t(a.window)) atomicAdd(hist + j, 1u);
            else atomicAdd(a.counts + key, 1u);
            // the tile's largest box radius (the backward stages, and the forward flushes, only
            // the tile's pixels within it), kept per CTA like the histogram: an atomic only
            // where the photon's radius exceeds the value seen (a stale, lower value only costs
            // a redundant atomic; the value only grows)
            uint32_t* tr = a.tile_r + (key >> a.cfg.class_bits);
            if (j < uint32_t(a.window) && a.window_tiles) tr = radii + (j >> a.cfg.class_bits);
            if (uint32_t(rmax) > *tr) atomicMax(tr, uint32_t(rmax));
        }
        // wide photons: appended to the wide list (one atomic per warp)
        const uint32_t wm = __ballot_sync(0xFFFFFFFFu, wide);
        if (wm) {
            uint32_t wbase = 0;
            if (lane == __ffs(wm) - 1) wbase = atomicAdd(a.counters + 1, uint32_t(__popc(wm)));
            wbase = __shfl_sync(0xFFFFFFFFu, wbase, __ffs(wm) - 1);
            if (wide) {
                const uint32_t k = wbase + __popc(wm & lanemask_lt());
                a.wide[k] = i;
                a.inv[i] = kWideBit | k;
            }
        }
    }
    if (PLACE) return;
    // block totals -> the tile-path and untouched counters; the window -> the bucket counts
    // and this CTA's kept histogram
    __shared__ uint32_t red[2];
    if (threadIdx.x < 2) red[threadIdx.x] = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < wend; j += blockDim.x) {
        const uint32_t c = hist[j];
        mine[j] = c;
        if (c) atomicAdd(a.counts + kb0 + j, c);
    }
    for (int j = threadIdx.x; j < a.window_tiles; j += blockDim.x) {
        const uint32_t m = radii[j];
        if (m) atomicMax(a.tile_r + (kb0 >> a.cfg.class_bits) + j, m);
    }
    c_tile = __reduce_add_sync(0xFFFFFFFFu, c_tile);
    c_inv = __reduce_add_sync(0xFFFFFFFFu, c_inv);
    if (lane == 0) {
        atomicAdd(&red[0], c_tile);
        atomicAdd(&red[1], c_inv);
    }
    __syncthreads();
    if (threadIdx.x == 0 && red[0]) atomicAdd(a.counters + 0, red[0]);
    if (threadIdx.x == 1 && red[1]) atomicAdd(a.counters + 2, red[1]);
}

// ------------------------------------------------------------------ bucket scan --------
// Exclusive scan of counts[0, nb) into start[0, nb] (start[nb] = the total) and cursor[0, nb).
// Up to kOneScanBuckets: bucket_down alone, whose CTAs each sum the counts before theirs.
// Beyond: per-CTA sums of kScanItems buckets, one CTA scanning those sums, then bucket_down.

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanItems = kScanThreads * kScanPer;

// Exclusive scan of one value per thread over the CTA; *total gets the CTA's sum.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
    __shared__ uint32_t wsum[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = wsum[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, off);
            if (lane >= off) w += y;
        }
        wsum[lane] = w;
    }
    __syncthreads();
    const uint32_t before = warp > 0 ? wsum[warp - 1] : 0u;
    *total = wsum[kScanThreads / 32 - 1];
    __syncthreads();
    return before + x - v;
}
static_assert(kScanThreads == 1024, "one warp scans the warps' sums");

// Sum of the counts of one CTA's buckets; four a thread (the counts start 256-byte aligned and
// are padded to a multiple of 256 bytes, so a group of four that begins before nb is inside).
__device__ __forceinline__ uint4 count_group(const uint32_t* counts, int64_t j, int64_t nb) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (j < nb) {
        v = __ldg(reinterpret_cast<const uint4*>(counts + j));
        if (j + 1 >= nb) v.y = 0u;
        if (j + 2 >= nb) v.z = 0u;
        if (j + 3 >= nb) v.w = 0u;
    }
    return v;
}

__global__ __launch_bounds__(kScanThreads) void bucket_reduce(const uint32_t* __restrict__ counts,
                                                              int64_t nb,
                                                              uint32_t* __restrict__ part) {
    const uint4 v = count_group(counts, int64_t(blockIdx.x) * kScanItems + threadIdx.x * kScanPer,
                                nb);
    uint32_t total;
    block_exclusive_scan(v.x + v.y + v.z + v.w, &total);
    if (threadIdx.x == 0) part[blockIdx.x] = total;
}

__global__ __launch_bounds__(kScanThreads) void bucket_top(uint32_t* __restrict__ part,
                                                           int64_t np) {
    uint32_t carry = 0;
    for (int64_t b = 0; b < np; b += kScanThreads) {
        const int64_t j = b + threadIdx.x;
        const uint32_t v = j < np ? part[j] : 0u;
        uint32_t total;
        const uint32_t ex = block_exclusive_scan(v, &total);
        if (j < np) part[j] = carry + ex;
        carry += total;
    }
}

// part: the scanned sums of the CTAs' buckets, or null to sum the counts before this CTA's here.
__global__ __launch_bounds__(kScanThreads) void bucket_down(const uint32_t* __restrict__ counts,
                                                            int64_t nb,
                                                            const uint32_t* __restrict__ part,
                                                            uint32_t* __restrict__ start,
                                                            uint32_t* __restrict__ cursor) {
    // thread t owns buckets [b0 + t * kScanPer, + kScanPer)
    const int64_t b0 = int64_t(blockIdx.x) * kScanItems;
    uint32_t base, total;
    if (part) {
        base = part[blockIdx.x];
    } else {
        uint32_t s = 0;
        for (int64_t j = int64_t(threadIdx.x) * kScanPer; j < b0; j += kScanItems) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(counts + j));
            s += v.x + v.y + v.z + v.w;
        }
        block_exclusive_scan(s, &base);
    }
    const int64_t j = b0 + int64_t(threadIdx.x) * kScanPer;
    const uint4 v = count_group(counts, j, nb);
    const uint32_t sum = v.x + v.y + v.z + v.w;
    uint32_t run = base + block_exclusive_scan(sum, &total);
    const uint32_t c[kScanPer] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        if (j + k < nb) {
            start[j + k] = run;
            cursor[j + k] = run;
        }
        run += c[k];
    }
    if (threadIdx.x == 0 && b0 + kScanItems >= nb) start[nb] = base + total;
}

// The plan's binning per photon: its bucket (from its sorted position and the bucket starts)
// and its slot (sorted position, wide-list index, or kInvalidPos).
__global__ __launch_bounds__(256) void plan_export_kernel(const uint32_t* __restrict__ inv,
                                                          const uint32_t* __restrict__ start,
                                                          int64_t nb, uint32_t key_big,
                                                          uint32_t key_invalid, int64_t n,
                                                          uint32_t* bucket, uint32_t* slot) {
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        const uint32_t v = inv[i];
        uint32_t b;
        if (v == kInvalidPos) {
            b = key_invalid;
        } else if (v & kWideBit) {
            b = key_big;
        } else {
            // the last bucket whose first position is at or before v (empty buckets start
            // where their successor does, so this is v's own bucket)
            int64_t lo = 0, hi = nb - 1;
            while (lo < hi) {
                const int64_t mid = (lo + hi + 1) >> 1;
                if (start[mid] <= v) lo = mid; else hi = mid - 1;
            }
            b = uint32_t(lo);
        }
        bucket[i] = b;
        slot[i] = v == kInvalidPos ? kInvalidPos : (v & ~kWideBit);
    }
}

unsigned capped_blocks(int64_t items, int per_sm) {
    const int64_t blocks = (items + 255) / 256;
    const int64_t cap = int64_t(num_sms()) * per_sm;
    return unsigned(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

}  // namespace

bool plan_fused(int64_t nb) { return nb <= kFusedBuckets; }

int64_t bucket_scan_parts(int64_t nb) { return (nb + kScanItems - 1) / kScanItems; }

// Tiles of a window whose radii the count pass keeps in shared memory after the histogram (with
// global atomics, the first photons of every CTA all met on a few tiles: 262144 photons of a plate
// 37 us, 11 us this way): all of them, or none where the two do not fit together (no class bits).
int32_t plan_window_tiles(int32_t window, int32_t class_bits) {
    const int64_t tiles = (int64_t(window) + (int64_t(1) << class_bits) - 1) >> class_bits;
    return size_t(window + tiles) * 4 <= kMaxDynamicSmem ? int32_t(tiles) : 0;
}

// Window and photons per CTA of the two plan passes: the window holds a simulation's buckets
// where it can (at most kMaxWindow); as many CTAs per SM as the window's shared memory allows,
// at most kPlanMaxCtas in all (the size of the kept histograms), and the photons are split
// evenly over one wave of them (at least min_range a CTA).
void plan_shape(int64_t n, int64_t nb, int32_t* window, int64_t* range) {
    const int64_t w = nb < kMaxWindow ? nb : kMaxWindow;
    *window = int32_t(w > 0 ? w : 1);
    int64_t ctas = int64_t(num_sms()) *
                   resident_ctas<plan_pass_kernel<false>>(kPlanKernelThreads, size_t(*window) * 4);
    if (ctas > kPlanMaxCtas) ctas = kPlanMaxCtas;
    int64_t r = (n + ctas - 1) / ctas;
    r = (r + kPlanKernelThreads - 1) / kPlanKernelThreads * kPlanKernelThreads;
    const int64_t least = min_range(*window);
    *range = r < least ? least : r;
}

int64_t plan_hist_entries(int64_t n, int64_t nb) {
    const int64_t w = nb < kMaxWindow ? (nb > 0 ? nb : 1) : kMaxWindow;
    const int64_t by_n = (n + min_range(w) - 1) / min_range(w);
    return (by_n < kPlanMaxCtas ? (by_n > 0 ? by_n : 1) : kPlanMaxCtas) * w;
}

template <bool PLACE>
cudaError_t launch_pass(const PlanArgs& a, cudaStream_t st) {
    if (a.ph.n <= 0) return cudaSuccess;
    const size_t smem = size_t(a.window + (PLACE ? 0 : a.window_tiles)) * 4;
    const cudaError_t e = allow_smem<plan_pass_kernel<PLACE>>(smem);
    if (e != cudaSuccess) return e;
    plan_pass_kernel<PLACE><<<unsigned((a.ph.n + a.range - 1) / a.range), kPlanKernelThreads, smem,
                              st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_plan_count(const PlanArgs& a, cudaStream_t st) { return launch_pass<false>(a, st); }

cudaError_t launch_plan_place(const PlanArgs& a, cudaStream_t st) { return launch_pass<true>(a, st); }

cudaError_t launch_plan_export(const uint32_t* inv, const uint32_t* start, int64_t nb,
                               uint32_t key_big, uint32_t key_invalid, int64_t n,
                               uint32_t* bucket, uint32_t* slot, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    plan_export_kernel<<<capped_blocks(n, 8), 256, 0, st>>>(inv, start, nb, key_big, key_invalid,
                                                            n, bucket, slot);
    return cudaGetLastError();
}

cudaError_t launch_bucket_scan(const ScanArgs& a, cudaStream_t st) {
    const int64_t np = bucket_scan_parts(a.nb);
    uint32_t* part = nullptr;
    if (a.nb > kOneScanBuckets) {
        part = a.part;
        bucket_reduce<<<unsigned(np), kScanThreads, 0, st>>>(a.counts, a.nb, part);
        bucket_top<<<1, kScanThreads, 0, st>>>(part, np);
    }
    bucket_down<<<unsigned(np), kScanThreads, 0, st>>>(a.counts, a.nb, part, a.start, a.cursor);
    return cudaGetLastError();
}

}  // namespace pds
