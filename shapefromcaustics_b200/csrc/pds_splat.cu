// Photon-differential splatting kernels for sm_100a.
//
// Reference: PyOptix/kernel/photon_differentials.cu. The reference runs one thread per
// photon over its whole footprint box with one global atomicAdd per covered pixel (forward,
// :60-113) and the same walk reading the upstream gradient (backward, :136-221). Here the
// photons come binned by the plan (pds_plan.cu: records in (simulation, channel, screen tile,
// footprint class) order) and
//
//   fwd_tiles_kernel persistent CTAs take fixed-size chunks of the sorted photons from a work
//                    counter; each tile segment is rasterised into a shared-memory accumulator
//                    covering the tile plus an apron of the largest footprint radius, then
//                    flushed with one coalesced pass of global adds over the touched box.
//   bwd_tiles_kernel same walk; the segment's tile+apron of the upstream gradient is staged
//                    in shared memory once, each photon gathers over its footprint from there
//                    and writes one gradient record (no atomics). The per-pixel work is reduced
//                    to the moments sum(t g), sum(t^2 g), sum(t g d), sum(t g d d^T) of the
//                    offset d, from which dL/dE, dL/dx and dL/dM follow by 2x2 algebra.
//   tail_*           footprints wider than the apron (direct global path, a warp per photon), by
//                    the tile kernels' CTAs once no chunk is left.
//   grad_scatter     gradient records into the reference's SoA outputs, zero for photons that
//                    touch no pixel.
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

#include "pds_device.cuh"
#include "pds_internal.h"
#include "pds_splat.h"

namespace pds {

namespace {

// ------------------------------------------------------------------ tiles --------------

// Photon counts of the plan, clamped to the photon count so that a workspace without a plan
// cannot send the kernels outside their arrays.
__device__ __forceinline__ int64_t tile_count(const TileArgs& a) {
    return min(int64_t(a.counters[0]), a.ph.n);
}
__device__ __forceinline__ int64_t wide_count(const TileArgs& a) {
    return min(int64_t(a.counters[1]), a.ph.n - tile_count(a));
}

struct TileInfo {
    int64_t img_off;  // element offset of the (simulation, channel) image plane
    bool in_image;    // the plane lies inside the caller's image buffer
    int32_t W, H;
    int32_t ox, oy;   // pixel coordinates of the accumulator's (0, 0)
    float sx, sy;     // 2 / W, 2 / H
    float isx, isy;   // W / 2, H / 2
};

// float(W), float(H) in double: the reference's w, h of the :93 ellipse test
__device__ __forceinline__ double img_wd(const TileInfo& t) { return double(float(t.W)); }
__device__ __forceinline__ double img_hd(const TileInfo& t) { return double(float(t.H)); }

__device__ __forceinline__ TileInfo decode_tile(const SimTable& st, uint32_t tile, const Cfg& cfg,
                                                int64_t image_elems) {
    const int s = find_sim_of_tile(st, tile);
    const pds_sim sim = load_sim(st, s);
    const int32_t local = int32_t(tile) - sim.tile_base;
    const int32_t tx = local % sim.tiles_x;
    const int32_t r = local / sim.tiles_x;
    const int32_t ty = r % sim.tiles_y;
    const int32_t ch = r / sim.tiles_y;
    TileInfo t;
    t.W = sim.width;
    t.H = sim.height;
    t.img_off = sim.image_offset + int64_t(ch) * sim.height * sim.width;
    t.in_image = t.img_off >= 0 && t.img_off + int64_t(sim.height) * sim.width <= image_elems;
    t.ox = tx * cfg.tile - cfg.apron;
    t.oy = ty * cfg.tile - cfg.apron;
    t.sx = float(2.0 / double(sim.width));
    t.sy = float(2.0 / double(sim.height));
    t.isx = 0.5f * float(sim.width);
    t.isy = 0.5f * float(sim.height);
    return t;
}

// A run of sorted positions [begin, end) holding one screen tile's photons (positions and tiles
// fit in 31 bits: the entry points reject larger calls).
struct Segment {
    int tile;
    uint32_t begin, end;
};

// End of tile t's photons: the start of its successor's first bucket.
__device__ __forceinline__ uint32_t tile_end(const TileArgs& a, int t) {
    return __ldg(a.start + ((int64_t(t) + 1) << a.cfg.class_bits));
}

__device__ __forceinline__ Segment first_segment(const TileArgs& a, uint32_t chunk, uint32_t p0) {
    Segment s;
    // (clamped, like the counters, so that a workspace without a plan stays in its arrays)
    s.tile = int(min(int64_t(__ldg(a.chunk_tile + chunk)), a.n_tiles - 1));
    s.begin = p0;
    s.end = tile_end(a, s.tile);
    return s;
}

// The segment after sg (sg.end below the tile path's photon count): the first tile after
// sg.tile whose range is not empty, found by doubling steps then bisection (empty tiles are
// usually few, so one probe mostly suffices).
__device__ __forceinline__ Segment next_segment(const TileArgs& a, const Segment& sg) {
    const uint32_t p = sg.end;
    const int t = sg.tile, last = int(a.n_tiles) - 1;
    int k = 1;
    while (k < last - t && tile_end(a, t + k) <= p) k <<= 1;
    int lo = t + (k >> 1) + 1, hi = k < last - t ? t + k : last;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (tile_end(a, mid) > p) hi = mid; else lo = mid + 1;
    }
    Segment s;
    s.tile = lo;
    s.begin = p;
    s.end = tile_end(a, lo);
    return s;
}

// The current segment and its tile, held in shared memory: one thread finds and decodes the next
// one while the others flush the last (two slots), and the photon loops read the fields they
// need instead of keeping them all in registers across a walk.
struct TileState {
    Segment sg;
    TileInfo ti;
    int x0, x1, y0, y1;  // pixels its photons can touch: the tile and the plan's largest radius
                         // around it, inside the image
    float scale, unit;   // forward: accumulator counts per unit of energy density (a power of
                         // two) and its inverse; both 0: the accumulator holds floats
    uint32_t stop;       // forward: end of the photons that are summed together
    uint32_t wrapped;    // forward: non-zero where a pixel's count has wrapped
    uint32_t groups;     // groups of 32 photons that warps have taken
};

__device__ __forceinline__ void set_tile(const TileArgs& a, const Segment& sg, TileState* t) {
    t->sg = sg;
    t->groups = 0u;
    const TileInfo ti = decode_tile(a.sims, uint32_t(sg.tile), a.cfg, a.image_elems);
    t->ti = ti;
    const int m = a.cfg.apron - int(min(__ldg(a.tile_r + sg.tile), uint32_t(a.cfg.apron)));
    t->x0 = max(ti.ox + m, 0);
    t->y0 = max(ti.oy + m, 0);
    t->x1 = min(ti.ox + a.cfg.tile + 2 * a.cfg.apron - 1 - m, ti.W - 1);
    t->y1 = min(ti.oy + a.cfg.tile + 2 * a.cfg.apron - 1 - m, ti.H - 1);
}

// ---- the forward's accumulator -----------------------------------------------------------
// A tile's pixels are summed as 32-bit fixed-point counts: a shared integer add is one native
// instruction whatever the lanes' addresses, where a shared float add is a compare-and-swap loop
// of about eight (measured a warp and SM, random pixels of a tile: 3.1 against 8.9 cycles with
// the loop around it; all lanes in 32 pixels, as in a focused caustic: 3.1 against 34).
//
// What a count is worth is a power of two chosen per segment from a sample of its photons
// (set_scale): with c the photons' mean number of covers of a pixel if they were spread over the
// tile, 2^32 counts hold at least 64 c typical peaks (or all of the segment's photons on one
// pixel). Where the peak of the sample's dimmest photon would then be below 2^kMinCountBits counts,
// half the room is given up; then a large segment is summed in pieces (kPiece), which need less; and
// what is still missing is taken from the room.
//
// An add is rounded to half a count (0.29 in the mean square): at most 2^-20 of its photon's peak,
// mostly 2^-22 and less, as far as a photon evaluated in float32 is off anyway. Measured against 64
// bits, and with sums in float instead:
// - single photons of 0.5 to 4 px: 6.3e-8 of their peak in the mean square, 6.9e-8;
// - a pixel of 2^24 photons on caustic curves, in chunks of 8192: 3.7e-9 of the peaks that cover
//   it, 9.1e-9; the whole image 5.5e-8, 3.0e-7;
// - of 2^22 uniform photons: 4.9e-9, 4.5e-9; the whole image 1.07e-7, 1.01e-7 (mostly the float
//   sums of the segments in the image).
//
// - A pixel whose count wraps (photons gathered on few pixels) is seen by the lane that causes
//   it, from the old count that the add returns. Every walk only marks the segment, and a marked
//   segment is summed again from zero by redo_segment, whose adds put each wrap's 2^32 counts into
//   the image pixel (carry_pixel). (Carried on the spot, the band walk has a branch a step that
//   its lanes leave apart: 2^22 photons on caustic curves 600 against 402 us. And no walk may
//   carry where another one marks: what it carried would be added again.)
// - A photon with a peak below 2^kDimBits counts, or of 2^31 and more, is added to the image
//   directly, in float (deposit_direct).
// - Where no scale holds the sample's dimmest and brightest photons, or none is in float range,
//   the whole segment is summed in float, in shared memory (scale 0, deposit_slow): 2^22 photons
//   with energies over six decades 190 us, all those out of range sent to the image 765.
// A floor of 23 bits for the dimmest photon instead of 21 makes dense segments wrap (2^22 photons on
// caustic curves 1043 us against 402), and a quarter of the room does so where photons gather (2^22
// of them within 2 px: 107 us, with 16 c peaks 191).
constexpr int kMaxCountBits = 25;  // counts of a typical peak at most, leaving the 2^6 above
constexpr int kMinCountBits = 21, kDimBits = 19;
constexpr float kCountLimit = 2147483648.f;
// Photons of a piece at least (each is added to the image by itself): 2^26 photons on caustic curves
// in chunks of 8192 4.29 ms (4.36 with no room given up first, and then 4.70 in pieces from 512 on,
// 4.58 to 4.77 from 2048 on, where some wrap); 7.00 in whole segments; 4.22 with the typical peak
// at 18 bits.
constexpr uint32_t kPiece = 1024;

// Sets t's stop, and its scale, from at most 32 photons spread evenly over the sorted positions
// [begin, end), one a lane (the whole warp calls it): the geometric mean, the least and the greatest
// of their energies as powers of two, and their mean support pi / |det M|, at most their box.
__device__ __forceinline__ void set_scale(const TileArgs& a, uint32_t begin, uint32_t end,
                                          TileState* t) {
    const uint32_t lane = threadIdx.x & 31, n = end > begin ? end - begin : 0u;
    float e = 0.f, area = 0.f;
    if (n > 0) {
        const Rec r = load_rec(a.srecs + (begin + uint32_t((uint64_t(n) * lane) >> 5)));
        e = r.e;
        const float det = fabsf(fmaf(r.m00, r.m11, -r.m01 * r.m10)) * t->ti.sx * t->ti.sy;
        const float box = float((2 * rec_rx(r.packed) + 1) * (2 * rec_ry(r.packed) + 1));
        area = fminf(__fdividef(3.1415927f, det), box);  // (NaN, inf: the box)
    }
    const bool use = e > 0.f && e < __int_as_float(0x7F800000);
    const int lg = (__float_as_int(e) >> 23) - 127;  // floor(log2 e)
    const int sum = __reduce_add_sync(0xFFFFFFFFu, use ? lg : 0);
    const int least = __reduce_min_sync(0xFFFFFFFFu, use ? lg : 128);
    const int most = __reduce_max_sync(0xFFFFFFFFu, use ? lg : -127);
    const int count = __popc(__ballot_sync(0xFFFFFFFFu, use));
    const int area16 = __reduce_add_sync(0xFFFFFFFFu, int(area * 16.f));  // mean area * 512
    if (lane == 0) {
        const int tile = a.cfg.tile;
        const float pixels = float(min(tile, t->ti.W) * min(tile, t->ti.H));
        const float peaks = 32.f * float(n) * (float(area16) * (1.f / 512.f)) / pixels;
        // ceil(log2) of min(peaks, n): the exponent of the next float below, plus one
        const int room = (__float_as_int(fmaxf(fminf(peaks, float(n)), 1.f) * 0.99999994f) >> 23) - 126;
        const int mean = __float2int_rd(float(sum) / float(max(count, 1)));
        const int lift = kMinCountBits - least + mean;  // bits of a typical peak that this takes
        int halvings = 0;
        while (lift > 31 - room + halvings && (n >> (halvings + 1)) >= kPiece) ++halvings;
        t->stop = begin + ((n + (1u << halvings) - 1u) >> halvings);
        const int k = max(min(kMaxCountBits, 30 - room + halvings), lift) - mean;
        const bool fits = count > 0 && most + k <= 30 && k <= 126;
        t->scale = fits ? __int_as_float((k + 127) << 23) : 0.f;
        t->unit = fits ? __int_as_float((127 - k) << 23) : 0.f;
        t->wrapped = 0u;
    }
}

// The photon's peak E 3/pi in counts, or 0 for one that is not counted.
__device__ __forceinline__ float count_peak(const TileState& t, float e) {
    const float p = (e * kThreeOverPi) * t.scale;
    return p >= float(1 << kDimBits) && p < kCountLimit ? p : 0.f;
}

// Adds the 2^32 counts that the pixel at shared byte address `at` has wrapped by to the image.
__device__ __forceinline__ void carry_pixel(const TileArgs& a, const TileState& t,
                                            uint32_t acc_base, uint32_t at) {
    const uint32_t idx = (at - acc_base) >> 2;
    const int sw = a.cfg.sw;
    // idx / sw: exact, (idx + 1/2) / sw is at least 1 / (2 sw) from an integer
    const int y = __float2int_rd((float(idx) + 0.5f) * (1.f / float(sw)));
    const int x = int(idx) - y * sw;
    if (t.ti.in_image)
        atomicAdd(a.out + t.ti.img_off + int64_t(t.ti.oy + y) * t.ti.W + (t.ti.ox + x),
                  t.unit * 4294967296.f);
}

// One pixel of a deposit: s = |u|^2 and the photon's peak in counts; adds peak (1 - s)^2 where
// s < 1 and in (the reference's value > 0, photon_differentials.cu:105-106). A wrap is carried on
// (kCarry: when the segment is summed again) or recorded in wraps. kFloat: the peak is E 3/pi and
// the sum is in float.
enum AddMode { kMark, kCarry, kFloat };
__device__ __forceinline__ bool add_count(uint32_t at, uint32_t v) {
    uint32_t old;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(at), "r"(v) : "memory");
    return old + v < v;
}
__device__ __forceinline__ void add_carry(const TileArgs& a, const TileState& t, uint32_t acc_base,
                                          uint32_t at, uint32_t v) {
    if (add_count(at, v)) carry_pixel(a, t, acc_base, at);
}
__device__ __forceinline__ void add_shared(uint32_t at, float v) {
    asm volatile("red.shared.add.f32 [%0], %1;" :: "r"(at), "f"(v) : "memory");
}
template <AddMode MODE>
__device__ __forceinline__ void add_pixel(const TileArgs& a, const TileState& t, uint32_t acc_base,
                                          uint32_t at, float s, float peak, bool& wraps,
                                          bool in = true) {
    if (!(in && s < 1.f)) return;
    const float d = 1.f - s;
    if (MODE == kFloat) return add_shared(at, (d * peak) * d);
    const uint32_t v = __float2uint_rn((d * peak) * d);
    if (MODE == kCarry)
        add_carry(a, t, acc_base, at, v);
    else
        wraps |= add_count(at, v);
}

// Adds the counts v0, v1 to the pixels at shared byte addresses at, at + 4 and counts the wraps.
// Unconditional (a pixel outside the support gets 0): ptxas branches around a predicated atomic.
__device__ __forceinline__ void add_pair(uint32_t at, uint32_t v0, uint32_t v1, uint32_t& wraps) {
    asm volatile(
        "{\n\t.reg .b32 a, b;\n\t"
        "atom.shared.add.u32 a, [%1], %2;\n\tatom.shared.add.u32 b, [%1+4], %3;\n\t"
        "add.cc.u32 a, a, %2;\n\taddc.u32 %0, %0, 0;\n\t"
        "add.cc.u32 b, b, %3;\n\taddc.u32 %0, %0, 0;\n\t}"
        : "+r"(wraps) : "r"(at), "r"(v0), "r"(v1) : "memory");
}

// One row of a forward deposit: n pixels from shared byte address `at`, with
// u = (k M00 sx + b0, k M10 sx + b1) at the k-th pixel.
template <AddMode MODE>
__device__ __forceinline__ void fwd_row(const TileArgs& a, const TileState& t, uint32_t acc_base,
                                        int n, uint32_t at, float b0, float b1, float a00,
                                        float a10, float peak, bool& wraps) {
    for (int k = 0; k < n; ++k, at += 4u) {
        const float u0 = fmaf(float(k), a00, b0), u1 = fmaf(float(k), a10, b1);
        add_pixel<MODE>(a, t, acc_base, at, fmaf(u0, u0, u1 * u1), peak, wraps);
    }
}

// Clipped box of a record in pixel coordinates.
__device__ __forceinline__ void rec_box(const Rec& r, const TileInfo& ti, int& pxc, int& pyc,
                                        int& x0, int& x1, int& y0, int& y1) {
    const uint32_t p = r.packed;
    pxc = ti.ox + rec_lx(p);
    pyc = ti.oy + rec_ly(p);
    const int rx = rec_rx(p), ry = rec_ry(p);
    x0 = max(pxc - rx, 0);
    x1 = min(pxc + rx, ti.W - 1);
    y0 = max(pyc - ry, 0);
    y1 = min(pyc + ry, ti.H - 1);
}

// Forward deposit of one photon straight into the image, in float: the few photons that the
// segment's counts cannot hold. Out of line.
__device__ __noinline__ void deposit_direct(const TileArgs& a, const TileState* tp, const Rec* rp) {
    const Rec r = *rp;
    const TileInfo ti = tp->ti;
    if (!ti.in_image) return;
    int pxc, pyc, x0, x1, y0, y1;
    rec_box(r, ti, pxc, pyc, x0, x1, y0, y1);
    const bool all = rec_flags(r.packed) & kFlagEllipseAll;
    const Support sup = make_support(r.m00, r.m01, r.m10, r.m11, all);
    const float e3 = r.e * kThreeOverPi;
    int ky0 = y0 - pyc, ky1 = y1 - pyc;
    support_rows(sup, r.dy0, ti.isy, ky0, ky1);
    for (int ky = ky0; ky <= ky1; ++ky) {
        const float dy = fmaf(float(ky), ti.sy, r.dy0);
        int kx0 = x0 - pxc, kx1 = x1 - pxc;
        if (!support_cols(sup, dy, r.dx0, ti.isx, kx0, kx1)) continue;
        float* row = a.out + ti.img_off + int64_t(pyc + ky) * ti.W + pxc;
        for (int kx = kx0; kx <= kx1; ++kx) {
            if (!all && !ellipse_ok(kx, ky, img_wd(ti), img_hd(ti))) continue;
            const float dx = fmaf(float(kx), ti.sx, r.dx0);
            const float u0 = fmaf(r.m00, dx, r.m01 * dy), u1 = fmaf(r.m10, dx, r.m11 * dy);
            const float s = fmaf(u0, u0, u1 * u1);
            const float d = 1.f - s;
            if (s < 1.f) atomicAdd(row + kx, (d * e3) * d);
        }
    }
}

// The band walks: the rows of a photon's band (see Band) inside its box, two pixels at a time. A
// row is w = min(2 floor(hw + 1), box width) pixels wide and starts at the first pixel at or
// after the band's left edge xc - hw, clamped into [kxb0, kxb1 - w + 1]. The support's pixels of
// a row are at most floor(2 hw) + 1 <= 2 floor(hw + 1) in a row, so the window holds them all;
// clamping slides it into the box without dropping any that lies there, and when w is the box
// width the row is the whole box row, so no pixel needs an in-box test. When w is odd, the second
// pixel of each row's last pair lies just outside the box and is masked: the remaining-pair count
// is tail there. (A pixel that rounding puts just outside the window is at the support's edge to
// within some 1e-6 of a pixel: it adds (1 - s)^2 ~ 1e-12 of the peak. Supports narrower than
// 2 kMinHalf, whose centre that could be, are walked that wide: still one pair.)
//
// With rho = ky + dy0 / sy the photon's row offset in pixels, the support of a row is centred on
// the column xc = beta rho - dx0 / sx, and with e = kx - xc
//   s = |M d|^2 = A e^2 + B rho^2,  A = |M (sx, 0)|^2,  B = (det M sx sy)^2 / A,
// so a pixel costs three operations (e, e^2, 1 - s = (1 - B rho^2) - A e^2) where u = M d and
// |u|^2 cost six, and nothing cancels: both terms of s are positive.
//
// Row starts are formed without conversions: round-to-nearest of xc - hw + 1/2, by adding and
// taking off 1.5 * 2^23 (the sum's low mantissa bits are then the integer itself).

struct PairWalk {
    int rows, npairs, tail;
    float ky0;            // first row
    float dyp, dxp, beta; // dy0 / sy, dx0 / sx, the centre's shift a row
    float A, B;
    float hw5, lo, hi;    // hw - 1/2, the clamp range of the row starts
    uint32_t row;         // 4 * (accumulator index of the first row's column 0 - kRoundMagicBits)
};

// False where the photon has no band (make_band's conditions, and photons that fail the
// reference's image-half-size ellipse test somewhere in their box). It is a third of a small
// photon's instructions, so everything is in pixel units and the reciprocals are the hardware's;
// what s depends on is then made exact to the last place: det M and the columns' product are
// formed without cancellation (a product's rounding error is added back) and the quotients by A
// corrected by their residue.
__device__ __forceinline__ bool pair_walk(const Rec& r, const TileInfo& ti, int sw, PairWalk& p) {
    const float m00 = r.m00 * ti.sx, m10 = r.m10 * ti.sx, m01 = r.m01 * ti.sy, m11 = r.m11 * ti.sy;
    const float A = fmaf(m00, m00, m10 * m10);
    const float cd = m01 * m10, cb = m10 * m11;
    const float d1 = fmaf(m00, m11, -cd);
    const float det = d1 - fmaf(m01, m10, -cd);
    const float hw = rsqrt_fast(A), iA = rcp_fast(A);
    const float ey = A * hw * rcp_fast(fabsf(det));  // the support's half-height, sqrt(A) / |det|
    const uint32_t bits = r.packed;
    const int rx = rec_rx(bits), ry = rec_ry(bits), lx = rec_lx(bits), ly = rec_ly(bits);
    if (!((bits & kFlagEllipseAll) && A > 0.f && A < 1e30f && hw <= float(rx) + 1.f && ey < 1e6f &&
          fabsf(det) > 1e-3f * (fabsf(d1 + cd) + fabsf(cd))))
        return false;
    const float bco = fmaf(m00, m01, cb) + fmaf(m10, m11, -cb);
    const float qd = det * iA, qb = bco * iA;
    p.A = A;
    p.B = fmaf(fmaf(-A, qd, det), iA, qd) * det;
    p.beta = -fmaf(fmaf(-A, qb, bco), iA, qb);
    p.dxp = r.dx0 * ti.isx;
    p.dyp = r.dy0 * ti.isy;
    // the clipped box, in offsets from the centre pixel
    const int pxc = ti.ox + lx, pyc = ti.oy + ly;
    const int kxb0 = -min(rx, pxc), kxb1 = min(rx, ti.W - 1 - pxc);
    const int boxw = kxb1 - kxb0 + 1;
    const float wide = fmaxf(hw, kMinHalf);
    const int w = min(2 * band_pairs(wide), boxw);
    const int ky0 = max(__float2int_ru(-ey - p.dyp), -min(ry, pyc));
    p.rows = min(__float2int_rd(ey - p.dyp), min(ry, ti.H - 1 - pyc)) - ky0 + 1;
    p.npairs = (w + 1) >> 1;
    p.tail = w & 1;
    p.ky0 = float(ky0);
    p.hw5 = wide - 0.5f;
    p.lo = float(kxb0);
    p.hi = float(kxb1 - w + 1);
    p.row = 4u * (uint32_t((ly + ky0) * sw + lx) - kRoundMagicBits);
    return true;
}

// The start of a row: its first pixel's offset e from the row's centre, the magic sum whose bits
// hold its column, and 1 - B rho^2.
struct PairRow {
    float m, e, d, rho;
};

__device__ __forceinline__ PairRow pair_row(const PairWalk& p, float ky) {
    PairRow r;
    r.rho = ky + p.dyp;
    const float xc = fmaf(r.rho, p.beta, -p.dxp);
    r.m = fminf(fmaxf(xc - p.hw5, p.lo), p.hi) + kRoundMagic;
    r.e = (r.m - kRoundMagic) - xc;
    r.d = fmaf(-p.B * r.rho, r.rho, 1.f);
    return r;
}

__device__ __forceinline__ float2 pair(float v) { return make_float2(v, v); }
__device__ __forceinline__ float hsum(float2 v) { return v.x + v.y; }

// Forward deposit of one photon over its band: one flattened loop over the rows' pixel pairs, so
// the trip count depends only on the band's area (photons of a warp share an area class), the
// row changing every npairs steps. False: the photon has no band.
//
// Bound by instruction issue. A row change, which some lane of the warp makes on nearly every
// step, is selected rather than branched to (2^22 photons on caustic curves 403 against 430 us;
// the backward, with more to select, is faster with the branch).
template <AddMode MODE>
__device__ __forceinline__ bool deposit_band(const TileArgs& a, TileState& t, const Rec& r,
                                             float peak, uint32_t acc_base) {
    const int sw = a.cfg.sw;
    PairWalk p;
    if (!pair_walk(r, t.ti, sw, p)) return false;
    const float2 P = pair(peak);
    float ky = p.ky0;
    PairRow c = pair_row(p, ky);
    // (wrapping arithmetic: the magic number's bits come off with each row's start)
    uint32_t row = acc_base + p.row;
    uint32_t at = row + 4u * __float_as_uint(c.m);
    int rem = p.npairs;
    uint32_t wraps = 0u;
    for (int q = p.rows * p.npairs; q > 0; --q) {
        const float e1 = c.e + 1.f;
        // 1 - s, or 0 outside the support and at the pixel after an odd row
        const float t0 = fmaxf(fmaf(-p.A * c.e, c.e, c.d), 0.f);
        const float t1 = rem == p.tail ? 0.f : fmaxf(fmaf(-p.A * e1, e1, c.d), 0.f);
        const float2 T = make_float2(t0, t1);
        const float2 V = __fmul2_rn(__fmul2_rn(T, P), T);
        if (MODE == kFloat) {
            if (V.x > 0.f) add_shared(at, V.x);
            if (V.y > 0.f) add_shared(at + 4u, V.y);
        } else if (MODE == kCarry) {
            add_carry(a, t, acc_base, at, __float2uint_rn(V.x));
            add_carry(a, t, acc_base, at + 4u, __float2uint_rn(V.y));
        } else {
            add_pair(at, __float2uint_rn(V.x), __float2uint_rn(V.y), wraps);
        }
        // the next pair: two columns on, or the next row's start
        const bool wrap = --rem == 0;
        const PairRow n = pair_row(p, ky + 1.f);
        const uint32_t row1 = row + 4u * uint32_t(sw);
        at = wrap ? row1 + 4u * __float_as_uint(n.m) : at + 8u;
        c.e = wrap ? n.e : c.e + 2.f;
        c.d = wrap ? n.d : c.d;
        ky = wrap ? ky + 1.f : ky;
        row = wrap ? row1 : row;
        rem = wrap ? p.npairs : rem;
    }
    if (wraps) t.wrapped = 1u;
    return true;
}

// Forward deposit of one photon without a band walk (photon_differentials.cu:91-110): the whole
// box, or with spans on only the support's rows and row spans (the other box pixels add exactly
// zero in the reference: value > 0 fails, :106). Photons that fail the reference's
// image-half-size ellipse test somewhere in their box (tiny images only) take the per-pixel test
// path. Out of line: with the band walk on, hardly any photon comes here, and inlined its
// registers were spilled around every photon's band walk.
template <AddMode MODE>
__device__ __noinline__ void deposit_generic(const TileArgs& a, TileState* tp, const Rec* rp,
                                             float peak, uint32_t acc_base) {
    bool wraps = false;
    const Rec r = *rp;
    const TileState& t = *tp;
    const TileInfo ti = t.ti;
    const int sw = a.cfg.sw;
    int pxc, pyc, x0, x1, y0, y1;
    rec_box(r, ti, pxc, pyc, x0, x1, y0, y1);
    const bool all = rec_flags(r.packed) & kFlagEllipseAll;
    const Support sup = make_support(r.m00, r.m01, r.m10, r.m11, (a.cfg.spans || a.cfg.band) && all);
    const float a00 = r.m00 * ti.sx, a10 = r.m10 * ti.sx;
    const float m01sy = r.m01 * ti.sy, m11sy = r.m11 * ti.sy;
    // u at the centre pixel's corner: M (dx0, dy0)
    const float c00 = fmaf(r.m00, r.dx0, r.m01 * r.dy0), c10 = fmaf(r.m10, r.dx0, r.m11 * r.dy0);
    int ky0 = y0 - pyc, ky1 = y1 - pyc;
    support_rows(sup, r.dy0, ti.isy, ky0, ky1);
    for (int ky = ky0; ky <= ky1; ++ky) {
        const float dy = fmaf(float(ky), ti.sy, r.dy0);
        int kx0 = x0 - pxc, kx1 = x1 - pxc;
        if (!support_cols(sup, dy, r.dx0, ti.isx, kx0, kx1)) continue;
        const uint32_t at = acc_base + 4u * uint32_t((pyc + ky - ti.oy) * sw + (pxc + kx0 - ti.ox));
        if (all) {
            const float kf = float(kx0);
            fwd_row<MODE>(a, t, acc_base, kx1 - kx0 + 1, at,
                           fmaf(kf, a00, fmaf(float(ky), m01sy, c00)),
                           fmaf(kf, a10, fmaf(float(ky), m11sy, c10)), a00, a10, peak,
                           wraps);
        } else {
            const float c0 = fmaf(r.m00, r.dx0, r.m01 * dy);
            const float c1 = fmaf(r.m10, r.dx0, r.m11 * dy);
            for (int kx = kx0; kx <= kx1; ++kx) {
                if (!ellipse_ok(kx, ky, img_wd(ti), img_hd(ti))) continue;
                const float u0 = fmaf(float(kx), a00, c0), u1 = fmaf(float(kx), a10, c1);
                add_pixel<MODE>(a, t, acc_base, at + 4u * uint32_t(kx - kx0),
                                 fmaf(u0, u0, u1 * u1), peak, wraps);
            }
        }
    }
    if (wraps) tp->wrapped = 1u;
}

// Forward deposit of a photon of a segment that is summed again with carries, or in float. Out of
// line.
template <AddMode MODE>
__device__ __noinline__ void deposit_slow(const TileArgs& a, TileState* t, const Rec* rp,
                                          float peak, uint32_t acc_base) {
    const Rec r = *rp;
    if (!((a.cfg.band || a.cfg.rows) && deposit_band<MODE>(a, *t, r, peak, acc_base)))
        deposit_generic<MODE>(a, t, rp, peak, acc_base);
}

// Forward deposit of a photon that is not counted.
__device__ __forceinline__ void deposit_uncounted(const TileArgs& a, TileState* t, const Rec* rp,
                                                  float e, uint32_t acc_base) {
    if (t->scale > 0.f)
        deposit_direct(a, t, rp);
    else
        deposit_slow<kFloat>(a, t, rp, e * kThreeOverPi, acc_base);
}

// ---- the padded-row walk (walk 4) -------------------------------------------------------
// Each lane holds one photon and walks its band's rows inside the clipped box (RowWalk). The
// warp pads every lane to the warp's largest row count and row width, so all lanes change
// rows on the same iteration and the loops stay converged; the plan's row classes group
// photons of nearly equal rows and widths into a warp, so little of the padding is wasted.
// Along a row, s = |M d|^2 is a quadratic in the column c, stepped by its first and second
// differences (two adds per pixel). Padding pixels (c >= the lane's width, rows past the
// lane's count) are predicated off.

// Per-lane constants of the row walk of one photon.
struct RowGeo {
    float xs0, beta;        // band start of row ky: floor(xs0 + beta ky) (xs0 = alpha - hw)
    int ky0, rows, w;       // rows ky0 .. ky0 + rows - 1 of w pixels (RowWalk)
    int kxb0, kxlast;       // clamp range of the row starts
    int off;                // accumulator index of the centre pixel: (pyc - oy) sw + pxc - ox
    float a00, a10;         // u step per pixel column: M (sx, 0)
    float b0, b1;           // u step per pixel row: M (0, sy)
    float c00, c10;         // u at the centre pixel's corner: M (dx0, dy0)
    float A;                // |M (sx, 0)|^2: half the second difference of s along a row
};

// Row walk of a record inside its clipped box (x0..y1, from rec_box); false when the photon
// needs the generic walk (the image-half-size ellipse quirk of tiny images, or an M without a
// band).
__device__ __forceinline__ bool prep_rows(const Rec& r, const TileInfo& ti, int sw, int pxc,
                                          int pyc, int x0, int x1, int y0, int y1, RowGeo& g) {
    if (!(rec_flags(r.packed) & kFlagEllipseAll)) return false;
    const Band band = make_band(r.m00, r.m01, r.m10, r.m11, r.dx0, r.dy0, ti.sy, ti.isx, ti.isy,
                                float(rec_rx(r.packed)) + 1.f);
    if (!band.on) return false;
    const RowWalk rw = row_walk(band, x0 - pxc, x1 - pxc, y0 - pyc, y1 - pyc);
    g.xs0 = band.alpha - band.hw;
    g.beta = band.beta;
    g.ky0 = rw.ky0;
    g.rows = rw.rows;
    g.w = rw.w;
    g.kxb0 = rw.kxb0;
    g.kxlast = rw.kxlast;
    g.off = (pyc - ti.oy) * sw + (pxc - ti.ox);
    g.a00 = r.m00 * ti.sx;
    g.a10 = r.m10 * ti.sx;
    g.b0 = r.m01 * ti.sy;
    g.b1 = r.m11 * ti.sy;
    g.c00 = fmaf(r.m00, r.dx0, r.m01 * r.dy0);
    g.c10 = fmaf(r.m10, r.dx0, r.m11 * r.dy0);
    g.A = fmaf(g.a00, g.a00, g.a10 * g.a10);
    return true;
}

// First column of row ky (band start clamped into the box), s and its first difference there.
__device__ __forceinline__ int row_begin(const RowGeo& g, int ky, float& s, float& d) {
    const float kyf = float(ky);
    const int xs = min(max(__float2int_rd(fmaf(kyf, g.beta, g.xs0)), g.kxb0), g.kxlast);
    const float kxf = float(xs);
    const float u0 = fmaf(kxf, g.a00, fmaf(kyf, g.b0, g.c00));
    const float u1 = fmaf(kxf, g.a10, fmaf(kyf, g.b1, g.c10));
    s = fmaf(u0, u0, u1 * u1);
    d = fmaf(2.f, fmaf(u0, g.a00, u1 * g.a10), g.A);  // s(c + 1) - s(c) at c = 0
    return xs;
}

// Shared load of the float at shared byte address a when c < w, else 0.
__device__ __forceinline__ float lds_row(uint32_t a, int c, int w) {
    float v;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.lt.s32 q, %2, %3;\n\tmov.b32 %0, 0;\n\t"
        "@q ld.shared.f32 %0, [%1];\n\t}"
        : "=f"(v) : "r"(a), "r"(c), "r"(w) : "memory");
    return v;
}

// Forward deposit of the warp's photons by padded rows. rows = 0 for lanes with nothing to
// walk (their g is not read). Every lane of the warp calls it.
__device__ __forceinline__ void deposit_rows(const TileArgs& a, TileState& t, const RowGeo& g,
                                             int rows, float peak, uint32_t acc_base) {
    const int rm = __reduce_max_sync(0xFFFFFFFFu, rows);
    if (rm == 0) return;
    bool wraps = false;
    const int wm = __reduce_max_sync(0xFFFFFFFFu, rows > 0 ? g.w : 0);
    const float dd = 2.f * g.A;
    for (int j = 0; j < rm; ++j) {
        const int wl = j < rows ? g.w : 0;
        const int ky = g.ky0 + j;
        float s, d;
        const int xs = row_begin(g, ky, s, d);
        uint32_t at = acc_base + 4u * uint32_t(g.off + ky * a.cfg.sw + xs);
        for (int c = 0; c < wm; ++c, at += 4u) {
            add_pixel<kMark>(a, t, acc_base, at, s, peak, wraps, c < wl);
            s += d;
            d += dd;
        }
    }
    if (wraps) t.wrapped = 1u;
}

// Backward moments of the warp's photons by padded rows (no rotation: the gathers read).
// Per row it keeps sum t g, sum t g c and sum t g c^2 over the row's columns c and folds them
// into the photon's moments in the integer x offset kx = xs + c and the normalised y offset,
// at the row's end. Every lane of the warp calls it.
struct RowMoments {
    float sE, A0t, B1t, B2t, Sy, Sxy, Syy;
};

__device__ __forceinline__ RowMoments gather_rows(const RowGeo& g, int rows, uint32_t tg_base,
                                                 int sw, float sy, float dy0) {
    RowMoments m = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const int rm = __reduce_max_sync(0xFFFFFFFFu, rows);
    if (rm == 0) return m;
    const int wm = __reduce_max_sync(0xFFFFFFFFu, rows > 0 ? g.w : 0);
    const float dd = 2.f * g.A;
    for (int j = 0; j < rm; ++j) {
        const bool act = j < rows;
        const int wl = act ? g.w : 0;
        const int ky = g.ky0 + j;
        float s, d;
        const int xs = row_begin(g, ky, s, d);
        // lanes without this row read nothing (their address is not formed from their rows)
        uint32_t a = act ? tg_base + 4u * uint32_t(g.off + ky * sw + xs) : tg_base;
        float A0 = 0.f, Bc = 0.f, Bcc = 0.f, sEr = 0.f, cf = 0.f;
        int c = 0;
        for (; c + 2 <= wm; c += 2) {
            const float q0 = lds_row(a, c, wl);
            const float q1 = lds_row(a + 4u, c + 1, wl);
            const float t0 = fmaxf(1.f - s, 0.f);
            s += d;
            d += dd;
            const float t1 = fmaxf(1.f - s, 0.f);
            s += d;
            d += dd;
            const float g0 = t0 * q0, g1 = t1 * q1;
            sEr = fmaf(t0, g0, sEr);
            sEr = fmaf(t1, g1, sEr);
            A0 += g0 + g1;
            const float h0 = g0 * cf, h1 = g1 * (cf + 1.f);
            Bc += h0 + h1;
            Bcc = fmaf(h0, cf, Bcc);
            Bcc = fmaf(h1, cf + 1.f, Bcc);
            cf += 2.f;
            a += 8u;
        }
        if (c < wm) {
            const float q0 = lds_row(a, c, wl);
            const float t0 = fmaxf(1.f - s, 0.f);
            const float g0 = t0 * q0;
            sEr = fmaf(t0, g0, sEr);
            A0 += g0;
            const float h0 = g0 * cf;
            Bc += h0;
            Bcc = fmaf(h0, cf, Bcc);
        }
        // sum g kx and sum g kx^2 with kx = xs + c
        const float xf = float(xs);
        const float B1 = fmaf(xf, A0, Bc);
        const float B2 = fmaf(xf, fmaf(xf, A0, 2.f * Bc), Bcc);
        const float dy = fmaf(float(ky), sy, dy0);
        m.sE += sEr;
        m.A0t += A0;
        m.B1t += B1;
        m.B2t += B2;
        m.Sy = fmaf(dy, A0, m.Sy);
        m.Syy = fmaf(dy * dy, A0, m.Syy);
        m.Sxy = fmaf(dy, B1, m.Sxy);  // sum g kx dy; finish_rows adds the dx0 part
    }
    return m;
}


// Photons with a footprint radius of at least cfg.coop_r are splatted by their whole warp:
// lane j takes rows j, j + 32, ... of the photon and walks each row's span of the support
// (|M d| < 1 solved per row, one pixel of margin) rather than the whole box row. Large and
// thin footprints then cost about their support area, co-located photons of a caustic no
// longer make a warp's lanes add into one shared address at once, and with an odd
// accumulator pitch the 32 rows of one column fall in 32 different banks.
__device__ __forceinline__ bool use_coop(const Rec& r, int coop_r) {
    const uint32_t p = r.packed;
    const uint32_t fl = rec_flags(p);
    return coop_r > 0 && (fl & kFlagEllipseAll) && !(fl & kFlagFwdSkip) &&
           (rec_rx(p) >= coop_r || rec_ry(p) >= coop_r);
}

// Forward deposit of one photon by the whole warp (see use_coop).
__device__ __noinline__ void deposit_coop(const TileArgs& a, TileState* tp, const Rec* rp,
                                          uint32_t acc_base) {
    const Rec r = *rp;
    const TileState& t = *tp;
    const TileInfo ti = t.ti;
    const float peak = count_peak(t, r.e);
    int pxc, pyc, x0, x1, y0, y1;
    rec_box(r, ti, pxc, pyc, x0, x1, y0, y1);
    const float a00 = r.m00 * ti.sx, a10 = r.m10 * ti.sx;
    const float m01sy = r.m01 * ti.sy, m11sy = r.m11 * ti.sy;
    const float c00 = fmaf(r.m00, r.dx0, r.m01 * r.dy0), c10 = fmaf(r.m10, r.dx0, r.m11 * r.dy0);
    const Support sup = make_support(r.m00, r.m01, r.m10, r.m11, true);
    bool wraps = false;
    int ky0 = y0 - pyc, ky1 = y1 - pyc;
    support_rows(sup, r.dy0, ti.isy, ky0, ky1);
    for (int ky = ky0 + int(threadIdx.x & 31); ky <= ky1; ky += 32) {
        const float dy = fmaf(float(ky), ti.sy, r.dy0);
        int kx0 = x0 - pxc, kx1 = x1 - pxc;
        if (!support_cols(sup, dy, r.dx0, ti.isx, kx0, kx1)) continue;
        const float kf = float(kx0);
        fwd_row<kMark>(
            a, t, acc_base, kx1 - kx0 + 1,
            acc_base + 4u * uint32_t((pyc + ky - ti.oy) * a.cfg.sw + (pxc + kx0 - ti.ox)),
            fmaf(kf, a00, fmaf(float(ky), m01sy, c00)), fmaf(kf, a10, fmaf(float(ky), m11sy, c10)),
            a00, a10, peak, wraps);
    }
    if (wraps) tp->wrapped = 1u;
}

// Next chunk of sorted photons for this CTA (the whole warp calls it): a shared work counter
// (zero when the kernel starts) hands chunks out in order as CTAs finish, so CTAs that drew
// chunks of large footprints do not hold up the others. Nothing waits on it.
__device__ __forceinline__ uint32_t take_chunk(uint32_t* queue) {
    uint32_t c = 0u;
    if ((threadIdx.x & 31) == 0) c = atomicAdd(queue, 1u);
    return __shfl_sync(0xFFFFFFFFu, c, 0);
}

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" :: "l"(p));
}

// Calls walk(i, valid) with whole warps over the photons [begin, end) of t's segment, a group of 32
// at a time: warps take groups as they finish, from the end of the range (the footprint classes
// ascend, so the long walks come first and the short ones fill the gaps), and each warp prefetches
// the records of its next group. With fixed groups the warps that drew long walks, or that
// prepared the next tile, kept the others waiting at the segment's end (a quarter of the
// warps' time in the forward of 2^22 photons on caustic curves). Each warp calls ending() once,
// after the first of its groups that leaves at most one a warp, or when there is none left.
template <class Walk, class Ending>
__device__ __forceinline__ void walk_segment(const TileArgs& a, TileState* t, uint32_t begin,
                                             uint32_t end, Walk walk, Ending ending) {
    const uint32_t lane = threadIdx.x & 31, n = end > begin ? end - begin : 0u;
    uint32_t g = take_chunk(&t->groups) * 32u;
    bool ended = false;
    while (g < n) {
        const uint32_t next = take_chunk(&t->groups) * 32u;
        if (next + lane < n) prefetch_l1(a.srecs + (end - 1u - next - lane));
        walk(end - 1u - g - lane, g + lane < n);
        // lanes wait for their warp's longest walk here: without it they would run on into the
        // next group a few at a time
        __syncwarp();
        if (!ended && next + blockDim.x >= n) {
            ended = true;
            ending();
        }
        g = next;
    }
    if (!ended) ending();
}

// Called by every CTA after it drew its last chunk: the last CTA to do so leaves the work counter
// at zero for the next launch on this plan (the count of finished CTAs wraps to zero by itself).
// Nothing waits.
__device__ __forceinline__ void finish_queue(uint32_t* queue) {
    if (threadIdx.x == 0 && atomicInc(queue + 1, gridDim.x - 1u) == gridDim.x - 1u) *queue = 0u;
}

// ------------------------------------------------------------------ tail ---------------
// Footprints wider than the apron (the plan's wide list) are splatted straight into global
// memory, one warp per photon; their gradient records follow the tile path's in the stage. The
// tile kernels do it after their last chunk: as kernels of their own they cost every call a
// launch (1.5 us and the gap before it), and hardly any call has such footprints.

struct Direct {
    int pxc, pyc, x0, x1, y0, y1;
    bool all;
    float dx0, dy0, m00, m01, m10, m11, e;
    float sx, sy;
    double wd, hd;
    int64_t img_off;
    int W;
};

__device__ __forceinline__ bool direct_setup(const TileArgs& a, uint32_t rid, Direct& d) {
    const int64_t n = a.ph.n;
    const int s = find_sim_of_photon(a.sims, rid);
    const pds_sim sim = load_sim(a.sims, s);
    const int64_t ch = a.ph.cp[rid];
    const float x = a.ph.X[rid], y = a.ph.X[n + rid];
    const Footprint f = make_footprint(x, y, a.ph.R[rid], sim.height, sim.width, a.mpr);
    if (!clip_box(f, sim.height, sim.width, d.x0, d.x1, d.y0, d.y1)) return false;
    d.pxc = f.px_c;
    d.pyc = f.py_c;
    d.all = f.ellipse_all;
    d.dx0 = corner_offset(f.px_c, sim.width, x);
    d.dy0 = corner_offset(f.py_c, sim.height, y);
    d.m00 = a.ph.M[rid];
    d.m01 = a.ph.M[n + rid];
    d.m10 = a.ph.M[3 * n + rid];
    d.m11 = a.ph.M[4 * n + rid];
    d.e = a.ph.E[rid];
    d.sx = float(2.0 / double(sim.width));
    d.sy = float(2.0 / double(sim.height));
    d.wd = double(float(sim.width));
    d.hd = double(float(sim.height));
    d.img_off = sim.image_offset + ch * sim.height * sim.width;
    if (d.img_off < 0 || d.img_off + int64_t(sim.height) * sim.width > a.image_elems) return false;
    d.W = sim.width;
    return true;
}

// (Out of line, so that its registers do not burden the walk before it.)
__device__ __noinline__ void tail_forward(const TileArgs& a) {
    const int64_t n_big = wide_count(a);
    const int lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t w = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n_big;
         w += warps) {
        const uint32_t rid = __ldg(a.wide + w);
        Direct d;
        if (!direct_setup(a, rid, d) || !(d.e > 0.f)) continue;
        const float e3 = d.e * kThreeOverPi;
        const int bw = d.x1 - d.x0 + 1;
        const int64_t total = int64_t(bw) * (d.y1 - d.y0 + 1);
        float* img = a.out + d.img_off;
        for (int64_t k = lane; k < total; k += 32) {
            const int py = d.y0 + int(k / bw), px = d.x0 + int(k % bw);
            const int kx = px - d.pxc, ky = py - d.pyc;
            if (!d.all && !ellipse_ok(kx, ky, d.wd, d.hd)) continue;
            const float dx = fmaf(float(kx), d.sx, d.dx0), dy = fmaf(float(ky), d.sy, d.dy0);
            const float u0 = fmaf(d.m00, dx, d.m01 * dy), u1 = fmaf(d.m10, dx, d.m11 * dy);
            const float s = fmaf(u0, u0, u1 * u1);
            if (s < 1.f) {
                const float t = 1.f - s;
                atomicAdd(img + int64_t(py) * d.W + px, t * t * e3);
            }
        }
    }
}

// Adds the pixels that the segment's photons can touch from the accumulator into the image and
// clears them: warps take rows, lanes take consecutive columns. When image rows are 16-byte
// aligned the adds are 4-wide vector reductions (red.global.add.v4.f32) over 4-aligned column
// groups; columns of a group outside the range add zero. All-zero groups are skipped.
__device__ __forceinline__ void flush_rows(uint32_t* acc, int sw, const TileState& t, float* out) {
    const float unit = t.unit;
    const auto value = [&](uint32_t v) {
        return unit > 0.f ? float(v) * unit : __uint_as_float(v);
    };
    const int x0 = t.x0, x1 = t.x1, y1 = t.y1;
    const int ox = t.ti.ox, oy = t.ti.oy, W = t.ti.W;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    float* img = out + t.ti.img_off;
    const bool vec = (W & 3) == 0 && (reinterpret_cast<uintptr_t>(img) & 15) == 0;
    if (!t.ti.in_image) {
        // a plane outside the caller's buffer (an inconsistent simulation table): clear only
        for (int gy = t.y0 + warp; gy <= y1; gy += nw) {
            uint32_t* arow = acc + (gy - oy) * sw - ox;
            for (int gx = x0 + lane; gx <= x1; gx += 32) arow[gx] = 0u;
        }
    } else if (vec) {
        const int g0 = x0 >> 2, g1 = x1 >> 2;
        for (int gy = t.y0 + warp; gy <= y1; gy += nw) {
            uint32_t* arow = acc + (gy - oy) * sw - ox;
            float* grow = img + int64_t(gy) * W;
            for (int g = g0 + lane; g <= g1; g += 32) {
                const int gx = g << 2;
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = gx + j;
                    v[j] = 0.f;
                    if (c >= x0 && c <= x1) {
                        v[j] = value(arow[c]);
                        arow[c] = 0u;
                    }
                }
                if (v[0] != 0.f || v[1] != 0.f || v[2] != 0.f || v[3] != 0.f)
                    atomicAdd(reinterpret_cast<float4*>(grow + gx),
                              make_float4(v[0], v[1], v[2], v[3]));
            }
        }
    } else {
        for (int gy = t.y0 + warp; gy <= y1; gy += nw) {
            uint32_t* arow = acc + (gy - oy) * sw - ox;
            float* grow = img + int64_t(gy) * W;
            for (int gx = x0 + lane; gx <= x1; gx += 32) {
                const uint32_t v = arow[gx];
                if (v != 0u) {
                    atomicAdd(grow + gx, value(v));
                    arow[gx] = 0u;
                }
            }
        }
    }
}

// Starts a segment of the forward whose photons below p1 are to be splatted (a whole warp calls
// it).
__device__ __forceinline__ void start_segment(const TileArgs& a, const Segment& sg, uint32_t p1,
                                              TileState* t) {
    if ((threadIdx.x & 31) == 0) set_tile(a, sg, t);
    __syncwarp();
    set_scale(a, sg.begin, min(sg.end, p1), t);
}

// Sums the segment's photons [begin, end) again where a pixel's count has wrapped: from zero, by
// the walk whose adds carry a wrap on (the photons that went to the image directly stay there).
// All threads call it, between barriers.
__device__ __noinline__ void redo_segment(const TileArgs& a, uint32_t* acc, TileState* t,
                                          uint32_t begin, uint32_t end) {
    const int sw = a.cfg.sw;
    for (int k = threadIdx.x; k < sw * sw; k += blockDim.x) acc[k] = 0u;
    __syncthreads();
    const uint32_t acc_base = static_cast<uint32_t>(__cvta_generic_to_shared(acc));
    for (uint32_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
        const float peak = count_peak(*t, a.srecs[i].e);
        if (!(rec_flags(a.srecs[i].packed) & kFlagFwdSkip) && peak > 0.f)
            deposit_slow<kCarry>(a, t, a.srecs + i, peak, acc_base);
    }
    __syncthreads();
}

// The forward's chunks (all threads of the CTA call it): walk(t, i, valid) splats photon i of
// segment t's tile into acc (whole warps call it), which each segment's end adds to the image.
// Warp 0 takes and prepares the next chunk while the others end the current one, and the last
// warp (which has the fewest rows to flush) the next segment while the others flush.
template <class Walk>
__device__ __forceinline__ void forward_chunks(const TileArgs& a, uint32_t* acc, Walk walk) {
    __shared__ TileState ts[3];
    __shared__ uint32_t chunks[2];
    const int sw = a.cfg.sw;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t n_tile = uint32_t(tile_count(a)), chunk = uint32_t(a.cfg.chunk);
    const uint32_t nchunks = (n_tile + chunk - 1) / chunk;
    auto prepare = [&](TileState* t, uint32_t* slot) {
        const uint32_t c = take_chunk(a.queue);
        if (c < nchunks)
            start_segment(a, first_segment(a, c, c * chunk), min(c * chunk + chunk, n_tile), t);
        if (threadIdx.x == 0) *slot = c;
    };
    if (warp == 0) prepare(ts, chunks);
    for (int k = threadIdx.x; k < sw * sw; k += blockDim.x) acc[k] = 0u;
    __syncthreads();
    int cur = 0, alt = 1, pre = 2;
    for (int par = 0;; par ^= 1) {
        const uint32_t c = chunks[par];
        if (c >= nchunks) break;
        const uint32_t p0 = c * chunk, p1 = min(p0 + chunk, n_tile);
        // every pass but the first covers at least one photon, so chunk + 1 passes suffice
        for (uint32_t pass = 0; pass <= chunk; ++pass) {
            const Segment sg = ts[cur].sg;
            const uint32_t stop = ts[cur].stop;
            const bool more = stop < p1;
            walk_segment(
                a, ts + cur, sg.begin, stop,
                [&](uint32_t i, bool valid) { walk(ts[cur], i, valid); },
                [&] { if (!more && warp == 0) prepare(ts + pre, chunks + (par ^ 1)); });
            __syncthreads();
            if (ts[cur].wrapped) redo_segment(a, acc, ts + cur, sg.begin, stop);
            if (more && threadIdx.x >= blockDim.x - 32)
                start_segment(a, stop < sg.end ? Segment{sg.tile, stop, sg.end} : next_segment(a, sg),
                              p1, ts + alt);
            flush_rows(acc, sw, ts[cur], a.out);
            __syncthreads();
            if (!more) break;
            const int old = cur;
            cur = alt;
            alt = old;
        }
        const int old = cur;
        cur = pre;
        pre = old;
    }
    finish_queue(a.queue);
    tail_forward(a);
}

template <int NT, int MINB>
__global__ __launch_bounds__(NT, MINB) void fwd_tiles_kernel(const __grid_constant__ TileArgs a) {
    extern __shared__ uint32_t acc[];
    const uint32_t acc_base = static_cast<uint32_t>(__cvta_generic_to_shared(acc));
    forward_chunks(a, acc, [&](TileState& t, uint32_t i, bool valid) {
        bool coop = false;
        if (valid) {
            const Rec r = load_rec(a.srecs + i);
            const float peak = count_peak(t, r.e);
            coop = peak > 0.f && use_coop(r, a.cfg.coop_r);
            if (!coop && !(rec_flags(r.packed) & kFlagFwdSkip)) {
                if (!(peak > 0.f))
                    deposit_uncounted(a, &t, a.srecs + i, r.e, acc_base);
                else if (!(a.cfg.band && deposit_band<kMark>(a, t, r, peak, acc_base)))
                    deposit_generic<kMark>(a, &t, a.srecs + i, peak, acc_base);
            }
        }
        if (a.cfg.coop_r > 0) {
            __syncwarp();
            for (uint32_t cm = __ballot_sync(0xFFFFFFFFu, coop); cm; cm &= cm - 1)
                deposit_coop(a, &t, a.srecs + __shfl_sync(0xFFFFFFFFu, i, __ffs(cm) - 1), acc_base);
        }
    });
}

// Stages the upstream gradient that a tile's photons read (clipped to the image): the tile and
// the pixels within r of it, r the largest box radius of the tile's photons (the plan's
// tile_r, at most the apron), and the column after them (the band walk reads, and discards,
// the pixel after an odd row's end; the pitch sw = tile + 2 apron + 1 has room for it). The
// apron's outer margin, which no photon of the tile reaches, is not loaded. Warps take rows,
// lanes take consecutive columns; the copies are asynchronous, so that a warp's rows are all in
// flight together (four-byte copies: the odd pitch aligns nothing wider).
__device__ __forceinline__ void load_region(float* tg, int sw, const TileState& t,
                                            const float* grad) {
    const int gx1 = min(t.x1 + 1, t.ti.W - 1), y1 = t.y1;
    const int ox = t.ti.ox, oy = t.ti.oy, W = t.ti.W;
    const bool in_image = t.ti.in_image;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nw = blockDim.x >> 5;
    const float* img = grad + t.ti.img_off;
    for (int gy = t.y0 + warp; gy <= y1; gy += nw) {
        float* trow = tg + (gy - oy) * sw - ox;
        const float* grow = img + int64_t(gy) * W;
        for (int gx = t.x0 + lane; gx <= gx1; gx += 32) {
            if (in_image)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
                             :: "r"(uint32_t(__cvta_generic_to_shared(trow + gx))), "l"(grow + gx)
                             : "memory");
            else
                trow[gx] = 0.f;
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// WIDE: one 256-bit store. (Not in functions that are called: there this toolkit's ptxas loses the
// alignment of the eight registers, or crashes.)
template <bool WIDE>
__device__ __forceinline__ void store_grad(GradRec* stage, uint32_t rid, float gE, float gx0,
                                           float gx1, float g00, float g01, float g10,
                                           float g11) {
    const float4 lo = make_float4(gE, gx0, gx1, g00), hi = make_float4(g01, g10, g11, 0.f);
    if (WIDE) {
        store_words8(stage + rid, lo, hi);
    } else {
        float4* d = reinterpret_cast<float4*>(stage + rid);
        d[0] = lo;
        d[1] = hi;
    }
}

// The moments of one photon turned into its gradients. With a = -12/pi E t g (the
// reference's d_silverman(r) E g / r, :193), sums over the support of
//   S  = sum t^2 g,  Sd = sum t g d,  Sdd = sum t g d d^T  (d the normalised offset)
// give  dL/dE = 3/pi S,  dL/dx = -M^T (c M Sd),  dL/dM = c M Sdd  with c = -12/pi E
// (:195-205 summed over the pixels; u = M d).
template <bool WIDE>
__device__ __forceinline__ void finish_grad(GradRec* stage, uint32_t rid, float e, float m00,
                                            float m01, float m10, float m11, float sE, float Sx,
                                            float Sy, float Sxx, float Sxy, float Syy) {
    const float c = -kTwelveOverPi * e;
    const float v0 = c * fmaf(m00, Sx, m01 * Sy);
    const float v1 = c * fmaf(m10, Sx, m11 * Sy);
    store_grad<WIDE>(stage, rid, kThreeOverPi * sE, -fmaf(m00, v0, m10 * v1),
               -fmaf(m01, v0, m11 * v1), c * fmaf(m00, Sxx, m01 * Sxy),
               c * fmaf(m00, Sxy, m01 * Syy), c * fmaf(m10, Sxx, m11 * Sxy),
               c * fmaf(m10, Sxy, m11 * Syy));
}

// The gradients of one photon from its row moments: sum g dx = sx B1t + dx0 A0t and
// sum g dx dy = sx (sum g kx dy) + dx0 Sy, with dx = kx sx + dx0.
__device__ __forceinline__ void finish_rows(GradRec* stage, uint32_t slot, const Rec& r,
                                            const TileInfo& ti, const RowMoments& m) {
    const float Sx = fmaf(ti.sx, m.B1t, r.dx0 * m.A0t);
    const float Sxx = fmaf(ti.sx * ti.sx, m.B2t,
                           fmaf(2.f * ti.sx * r.dx0, m.B1t, r.dx0 * r.dx0 * m.A0t));
    const float Sxy = fmaf(ti.sx, m.Sxy, r.dx0 * m.Sy);
    finish_grad<true>(stage, slot, r.e, r.m00, r.m01, r.m10, r.m11, m.sE, Sx, m.Sy, Sxx, Sxy, m.Syy);
}

// One row of a backward gather: n pixels from q, the first at pixel offset k0 (relative to
// the centre pixel). With t = max(1 - s, 0) and g the upstream gradient it accumulates
// sum t^2 g, and over the row sum t g and sum t g k (k the pixel offset); the caller folds
// those into the photon's moments. Unrolled by two; n is nearly always warp-uniform.
__device__ __forceinline__ void bwd_row(int n, const float* q, float k0, float b0, float b1,
                                        float a00, float a10, float& sE, float& A0, float& B1,
                                        float& B2) {
    float kf = 0.f;
    int k = 0;
    for (; k + 1 < n; k += 2) {
        const float u0 = fmaf(kf, a00, b0), u1 = fmaf(kf, a10, b1);
        const float v0 = u0 + a00, v1 = u1 + a10;
        const float s = fmaf(u0, u0, u1 * u1), s2 = fmaf(v0, v0, v1 * v1);
        const float t = fmaxf(1.f - s, 0.f), t2 = fmaxf(1.f - s2, 0.f);
        const float g = t * q[k], g2 = t2 * q[k + 1];
        const float kk = k0 + kf;
        sE = fmaf(t, g, sE);
        sE = fmaf(t2, g2, sE);
        A0 += g + g2;
        const float tk = g * kk, tk2 = g2 * (kk + 1.f);
        B1 += tk + tk2;
        B2 = fmaf(tk, kk, B2);
        B2 = fmaf(tk2, kk + 1.f, B2);
        kf += 2.f;
    }
    if (k < n) {
        const float u0 = fmaf(kf, a00, b0), u1 = fmaf(kf, a10, b1);
        const float s = fmaf(u0, u0, u1 * u1);
        const float t = fmaxf(1.f - s, 0.f);
        const float g = t * q[k];
        const float kk = k0 + kf;
        sE = fmaf(t, g, sE);
        A0 += g;
        const float tk = g * kk;
        B1 += tk;
        B2 = fmaf(tk, kk, B2);
    }
}

// Backward gather of one photon over its band's rows in the box, two pixels a step (PairWalk;
// the pixel after an odd row is read from the staged tile's spare column, the pitch is odd: tile +
// 2 apron + 1, and a box never reaches past column tile + 2 apron - 1, and its value discarded).
// With no row inside the box its gradients are zero. False: the photon has no band.
//
// Bound by the FP32 pipe and instruction issue. The moments run over the whole band, in the walk's own coordinates: with
// t = 1 - s, sums of t^2 g, t g e, t g e^2, t g rho, t g e rho, t g rho^2, from which those
// of the offset d = (sx (e + beta rho), sy rho) follow once per photon. The two pixels of a step
// are the two lanes of packed FP32 instructions with partial sums of their own. (Folding a row's
// sums at its end instead cost about 28 instructions that some lane of the warp ran on nearly
// every step, and kept the lanes apart.)
__device__ __forceinline__ bool gather_band(const Rec& r, const TileInfo& ti, int sw,
                                            const float* tg, uint32_t slot, GradRec* stage) {
    float2 SE = pair(0.f), GE = pair(0.f), GEE = pair(0.f), GR = pair(0.f),
           GER = pair(0.f), GRR = pair(0.f);
    PairWalk p;
    if (!pair_walk(r, ti, sw, p)) return false;
    {
        float ky = p.ky0;
        PairRow c = pair_row(p, ky);
        float2 R = pair(c.rho);
        // (wrapping arithmetic, as in deposit_band)
        uint32_t row = p.row;
        uint32_t at = row + 4u * __float_as_uint(c.m);
        const char* base = reinterpret_cast<const char*>(tg);
        int rem = p.npairs;
        for (int q = p.rows * p.npairs; q > 0; --q) {
            const float* g = reinterpret_cast<const float*>(base + at);
            const float2 Q = make_float2(g[0], rem == p.tail ? 0.f : g[1]);
            const float2 E = make_float2(c.e, c.e + 1.f);
            const float2 T = make_float2(fmaxf(fmaf(-p.A * E.x, E.x, c.d), 0.f),
                                         fmaxf(fmaf(-p.A * E.y, E.y, c.d), 0.f));
            const float2 G = __fmul2_rn(T, Q);
            const float2 X = __fmul2_rn(G, E), Y = __fmul2_rn(G, R);
            SE = __ffma2_rn(T, G, SE);
            GE = __fadd2_rn(GE, X);
            GEE = __ffma2_rn(X, E, GEE);
            GR = __fadd2_rn(GR, Y);
            GER = __ffma2_rn(X, R, GER);
            GRR = __ffma2_rn(Y, R, GRR);
            at += 8u;
            c.e += 2.f;
            if (--rem == 0) {
                ky += 1.f;
                c = pair_row(p, ky);
                R = pair(c.rho);
                row += 4u * uint32_t(sw);
                at = row + 4u * __float_as_uint(c.m);
                rem = p.npairs;
            }
        }
    }
    const float gr = hsum(GR), grr = hsum(GRR), ger = hsum(GER);
    const float bgr = p.beta * grr;
    const float Sx = ti.sx * fmaf(p.beta, gr, hsum(GE)), Sy = ti.sy * gr;
    const float Sxx = (ti.sx * ti.sx) * fmaf(p.beta, fmaf(2.f, ger, bgr), hsum(GEE));
    const float Sxy = (ti.sx * ti.sy) * (ger + bgr), Syy = (ti.sy * ti.sy) * grr;
    finish_grad<true>(stage, slot, r.e, r.m00, r.m01, r.m10, r.m11, hsum(SE), Sx, Sy, Sxx, Sxy, Syy);
    return true;
}

// Backward gather of one photon without a band walk (photon_differentials.cu:169-218) from the
// staged gradient. Pixels outside the support contribute 0 * g in the reference; with spans on
// they are not visited. The offset d of pixel (kx, ky) is (kx sx + dx0, ky sy + dy0); moments in
// x are kept in the integer offset kx and converted once per photon. Out of line, like
// deposit_generic.
__device__ __noinline__ void gather_generic(const Rec* rp, TileInfo ti, int sw, bool spans,
                                            const float* tg, uint32_t rid, GradRec* stage) {
    const Rec r = *rp;
    const uint32_t p = r.packed;
    const int pxc = ti.ox + rec_lx(p), pyc = ti.oy + rec_ly(p);
    const int rx = rec_rx(p), ry = rec_ry(p);
    const int x0 = max(pxc - rx, 0), x1 = min(pxc + rx, ti.W - 1);
    const int y0 = max(pyc - ry, 0), y1 = min(pyc + ry, ti.H - 1);
    const bool all = rec_flags(p) & kFlagEllipseAll;
    const Support sup = make_support(r.m00, r.m01, r.m10, r.m11, spans && all);
    const float a00 = r.m00 * ti.sx, a10 = r.m10 * ti.sx;
    int ky0 = y0 - pyc, ky1 = y1 - pyc;
    support_rows(sup, r.dy0, ti.isy, ky0, ky1);
    float sE = 0.f, A0t = 0.f, B1t = 0.f, B2 = 0.f, Sy = 0.f, Sxy = 0.f, Syy = 0.f;
    for (int ky = ky0; ky <= ky1; ++ky) {
        const float dy = fmaf(float(ky), ti.sy, r.dy0);
        int kx0 = x0 - pxc, kx1 = x1 - pxc;
        if (!support_cols(sup, dy, r.dx0, ti.isx, kx0, kx1)) continue;
        const float c0 = fmaf(r.m00, r.dx0, r.m01 * dy);
        const float c1 = fmaf(r.m10, r.dx0, r.m11 * dy);
        const float* q = tg + (pyc + ky - ti.oy) * sw + (pxc - ti.ox);
        float A0 = 0.f, B1 = 0.f;
        if (all) {
            const float kf = float(kx0);
            bwd_row(kx1 - kx0 + 1, q + kx0, kf, fmaf(kf, a00, c0), fmaf(kf, a10, c1), a00, a10,
                    sE, A0, B1, B2);
        } else {
            for (int kx = kx0; kx <= kx1; ++kx) {
                if (!ellipse_ok(kx, ky, img_wd(ti), img_hd(ti))) continue;
                const float kf = float(kx);
                const float u0 = fmaf(kf, a00, c0), u1 = fmaf(kf, a10, c1);
                const float s = fmaf(u0, u0, u1 * u1);
                const float t = fmaxf(1.f - s, 0.f);
                const float tgv = t * q[kx];
                sE = fmaf(t, tgv, sE);
                A0 += tgv;
                const float tk = tgv * kf;
                B1 += tk;
                B2 = fmaf(tk, kf, B2);
            }
        }
        A0t += A0;
        B1t += B1;
        const float sdx = fmaf(ti.sx, B1, r.dx0 * A0);  // sum t g dx over the row
        Sy = fmaf(dy, A0, Sy);
        Sxy = fmaf(dy, sdx, Sxy);
        Syy = fmaf(dy * dy, A0, Syy);
    }
    const float Sx = fmaf(ti.sx, B1t, r.dx0 * A0t);
    const float Sxx = fmaf(ti.sx * ti.sx, B2, fmaf(2.f * ti.sx * r.dx0, B1t, r.dx0 * r.dx0 * A0t));
    finish_grad<false>(stage, rid, r.e, r.m00, r.m01, r.m10, r.m11, sE, Sx, Sy, Sxx, Sxy, Syy);
}

// Backward gather of one photon by the whole warp (see use_coop): lanes take rows and walk
// their support spans, and a warp reduction hands the moments to the owning lane.
__device__ __noinline__ void gather_coop(const Rec* rp, TileInfo ti, int sw, const float* tg,
                                         uint32_t rid, int owner, GradRec* stage) {
    const Rec r = *rp;
    const int lane = threadIdx.x & 31;
    int pxc, pyc, x0, x1, y0, y1;
    rec_box(r, ti, pxc, pyc, x0, x1, y0, y1);
    const float a00 = r.m00 * ti.sx, a10 = r.m10 * ti.sx;
    const Support sup = make_support(r.m00, r.m01, r.m10, r.m11, true);
    int ky0 = y0 - pyc, ky1 = y1 - pyc;
    support_rows(sup, r.dy0, ti.isy, ky0, ky1);
    float sE = 0.f, A0t = 0.f, B1t = 0.f, B2 = 0.f, Sy = 0.f, Sxy = 0.f, Syy = 0.f;
    for (int ky = ky0 + lane; ky <= ky1; ky += 32) {
        const float dy = fmaf(float(ky), ti.sy, r.dy0);
        int kx0 = x0 - pxc, kx1 = x1 - pxc;
        if (!support_cols(sup, dy, r.dx0, ti.isx, kx0, kx1)) continue;
        const float c0 = fmaf(r.m00, r.dx0, r.m01 * dy);
        const float c1 = fmaf(r.m10, r.dx0, r.m11 * dy);
        const float* q = tg + (pyc + ky - ti.oy) * sw + (pxc - ti.ox);
        float A0 = 0.f, B1 = 0.f;
        const float kf = float(kx0);
        bwd_row(kx1 - kx0 + 1, q + kx0, kf, fmaf(kf, a00, c0), fmaf(kf, a10, c1), a00, a10, sE,
                A0, B1, B2);
        A0t += A0;
        B1t += B1;
        const float sdx = fmaf(ti.sx, B1, r.dx0 * A0);
        Sy = fmaf(dy, A0, Sy);
        Sxy = fmaf(dy, sdx, Sxy);
        Syy = fmaf(dy * dy, A0, Syy);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        sE += __shfl_xor_sync(0xFFFFFFFFu, sE, off);
        A0t += __shfl_xor_sync(0xFFFFFFFFu, A0t, off);
        B1t += __shfl_xor_sync(0xFFFFFFFFu, B1t, off);
        B2 += __shfl_xor_sync(0xFFFFFFFFu, B2, off);
        Sy += __shfl_xor_sync(0xFFFFFFFFu, Sy, off);
        Sxy += __shfl_xor_sync(0xFFFFFFFFu, Sxy, off);
        Syy += __shfl_xor_sync(0xFFFFFFFFu, Syy, off);
    }
    if (lane == owner) {
        const float Sx = fmaf(ti.sx, B1t, r.dx0 * A0t);
        const float Sxx = fmaf(ti.sx * ti.sx, B2, fmaf(2.f * ti.sx * r.dx0, B1t, r.dx0 * r.dx0 * A0t));
        finish_grad<false>(stage, rid, r.e, r.m00, r.m01, r.m10, r.m11, sE, Sx, Sy, Sxx, Sxy, Syy);
    }
}

__device__ __noinline__ void tail_backward(const TileArgs& a) {
    const int64_t n_tile = tile_count(a), n_big = wide_count(a);
    const int lane = threadIdx.x & 31;
    const int64_t warps = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t w = int64_t(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); w < n_big;
         w += warps) {
        const uint32_t rid = __ldg(a.wide + w);
        Direct d;
        float sE = 0.f, Sx = 0.f, Sy = 0.f, Sxx = 0.f, Sxy = 0.f, Syy = 0.f;
        const bool any = direct_setup(a, rid, d);
        if (any) {
            const int bw = d.x1 - d.x0 + 1;
            const int64_t total = int64_t(bw) * (d.y1 - d.y0 + 1);
            const float* img = a.grad + d.img_off;
            for (int64_t k = lane; k < total; k += 32) {
                const int py = d.y0 + int(k / bw), px = d.x0 + int(k % bw);
                const int kx = px - d.pxc, ky = py - d.pyc;
                if (!d.all && !ellipse_ok(kx, ky, d.wd, d.hd)) continue;
                const float dx = fmaf(float(kx), d.sx, d.dx0), dy = fmaf(float(ky), d.sy, d.dy0);
                const float u0 = fmaf(d.m00, dx, d.m01 * dy), u1 = fmaf(d.m10, dx, d.m11 * dy);
                const float s = fmaf(u0, u0, u1 * u1);
                const float t = s < 1.f ? 1.f - s : 0.f;
                const float tgv = t * __ldg(img + int64_t(py) * d.W + px);
                sE = fmaf(t, tgv, sE);
                Sx = fmaf(tgv, dx, Sx);
                Sy = fmaf(tgv, dy, Sy);
                Sxx = fmaf(tgv * dx, dx, Sxx);
                Sxy = fmaf(tgv * dx, dy, Sxy);
                Syy = fmaf(tgv * dy, dy, Syy);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            sE += __shfl_xor_sync(0xFFFFFFFFu, sE, off);
            Sx += __shfl_xor_sync(0xFFFFFFFFu, Sx, off);
            Sy += __shfl_xor_sync(0xFFFFFFFFu, Sy, off);
            Sxx += __shfl_xor_sync(0xFFFFFFFFu, Sxx, off);
            Sxy += __shfl_xor_sync(0xFFFFFFFFu, Sxy, off);
            Syy += __shfl_xor_sync(0xFFFFFFFFu, Syy, off);
        }
        if (lane == 0) {
            if (!any) {
                d.m00 = d.m01 = d.m10 = d.m11 = d.e = 0.f;
            }
            finish_grad<false>(a.stage, uint32_t(n_tile + w), d.e, d.m00, d.m01, d.m10, d.m11, sE, Sx,
                        Sy, Sxx, Sxy, Syy);
        }
    }
}

// The backward's chunks (all threads of the CTA call it): walk(t, i, valid) gathers photon i of
// segment t's tile from tg (whole warps call it). Warp 0 prepares the next segment, or takes and
// prepares the next chunk, while the others end the current one.
template <class Walk>
__device__ __forceinline__ void backward_chunks(const TileArgs& a, float* tg, Walk walk) {
    __shared__ TileState ts[3];
    __shared__ uint32_t chunks[2];
    const int sw = a.cfg.sw;
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t n_tile = uint32_t(tile_count(a)), chunk = uint32_t(a.cfg.chunk);
    const uint32_t nchunks = (n_tile + chunk - 1) / chunk;
    auto prepare = [&](TileState* t, uint32_t* slot) {
        const uint32_t c = take_chunk(a.queue);
        if (threadIdx.x == 0) {
            if (c < nchunks) set_tile(a, first_segment(a, c, c * chunk), t);
            *slot = c;
        }
    };
    if (warp == 0) prepare(ts, chunks);
    __syncthreads();
    int cur = 0, alt = 1, pre = 2;
    for (int par = 0;; par ^= 1) {
        const uint32_t c = chunks[par];
        if (c >= nchunks) break;
        const uint32_t p0 = c * chunk, p1 = min(p0 + chunk, n_tile);
        for (uint32_t pass = 0; pass <= chunk; ++pass) {
            load_region(tg, sw, ts[cur], a.grad);
            __syncthreads();
            const Segment sg = ts[cur].sg;
            const uint32_t begin = max(sg.begin, p0), end = min(sg.end, p1);
            const bool more = sg.end < p1;
            walk_segment(
                a, ts + cur, begin, end, [&](uint32_t i, bool valid) { walk(ts[cur], i, valid); },
                [&] {
                    if (warp != 0) return;
                    if (!more)
                        prepare(ts + pre, chunks + (par ^ 1));
                    else if (threadIdx.x == 0)
                        set_tile(a, next_segment(a, sg), ts + alt);
                });
            __syncthreads();
            if (!more) break;
            const int old = cur;
            cur = alt;
            alt = old;
        }
        const int old = cur;
        cur = pre;
        pre = old;
    }
    finish_queue(a.queue);
    tail_backward(a);
}

template <int NT, int MINB>
__global__ __launch_bounds__(NT, MINB) void bwd_tiles_kernel(const __grid_constant__ TileArgs a) {
    extern __shared__ float tg[];
    backward_chunks(a, tg, [&](TileState& t, uint32_t i, bool valid) {
        const int sw = a.cfg.sw;
        bool coop = false;
        if (valid) {
            const Rec r = load_rec(a.srecs + i);
            coop = use_coop(r, a.cfg.coop_r);
            // a photon's gradient record goes to its sorted position
            if (!coop && !(a.cfg.band && gather_band(r, t.ti, sw, tg, i, a.stage)))
                gather_generic(a.srecs + i, t.ti, sw, a.cfg.spans, tg, i, a.stage);
        }
        if (a.cfg.coop_r > 0) {
            __syncwarp();
            for (uint32_t cm = __ballot_sync(0xFFFFFFFFu, coop); cm; cm &= cm - 1) {
                const int src = __ffs(cm) - 1;
                const uint32_t slot = __shfl_sync(0xFFFFFFFFu, i, src);
                gather_coop(a.srecs + slot, t.ti, sw, tg, slot, src, a.stage);
            }
        }
    });
}

// ---- the padded-row walk's kernels (walk 4) ---------------------------------------------
// The same persistent chunk and segment loop as fwd_tiles_kernel / bwd_tiles_kernel, with the
// padded-row walk for the photons that have a band. A lane loads its record in the pass of its
// segment only, and keeps just the row walk's constants across the walk.

template <int NT, int MINB>
__global__ __launch_bounds__(NT, MINB) void fwd_rows_kernel(const __grid_constant__ TileArgs a) {
    extern __shared__ uint32_t acc[];
    const uint32_t acc_base = static_cast<uint32_t>(__cvta_generic_to_shared(acc));
    forward_chunks(a, acc, [&](TileState& t, uint32_t i, bool valid) {
        RowGeo g;
        int rows = 0;
        float peak = 0.f;
        bool generic = false, coop = false;
        if (valid) {
            const Rec r = load_rec(a.srecs + i);
            peak = count_peak(t, r.e);
            coop = peak > 0.f && use_coop(r, a.cfg.coop_r);
            if (!coop && !(rec_flags(r.packed) & kFlagFwdSkip)) {
                int pxc, pyc, x0, x1, y0, y1;
                rec_box(r, t.ti, pxc, pyc, x0, x1, y0, y1);
                if (!(peak > 0.f)) {
                    deposit_uncounted(a, &t, a.srecs + i, r.e, acc_base);
                } else {
                    generic = !prep_rows(r, t.ti, a.cfg.sw, pxc, pyc, x0, x1, y0, y1, g);
                    rows = generic ? 0 : g.rows;
                }
            }
        }
        __syncwarp();
        deposit_rows(a, t, g, rows, peak, acc_base);
        if (generic) deposit_generic<kMark>(a, &t, a.srecs + i, peak, acc_base);
        __syncwarp();
        for (uint32_t cm = __ballot_sync(0xFFFFFFFFu, coop); cm; cm &= cm - 1)
            deposit_coop(a, &t, a.srecs + __shfl_sync(0xFFFFFFFFu, i, __ffs(cm) - 1), acc_base);
    });
}

template <int NT, int MINB>
__global__ __launch_bounds__(NT, MINB) void bwd_rows_kernel(const __grid_constant__ TileArgs a) {
    extern __shared__ float tg[];
    const uint32_t tg_base = static_cast<uint32_t>(__cvta_generic_to_shared(tg));
    backward_chunks(a, tg, [&](TileState& t, uint32_t i, bool valid) {
        const int sw = a.cfg.sw;
        RowGeo g;
        int rows = 0;
        float dy0 = 0.f;
        bool walk = false, generic = false, coop = false;
        if (valid) {
            const Rec r = load_rec(a.srecs + i);
            coop = use_coop(r, a.cfg.coop_r);
            if (!coop) {
                int pxc, pyc, x0, x1, y0, y1;
                rec_box(r, t.ti, pxc, pyc, x0, x1, y0, y1);
                walk = prep_rows(r, t.ti, sw, pxc, pyc, x0, x1, y0, y1, g);
                generic = !walk;
                rows = walk ? g.rows : 0;
                dy0 = r.dy0;
            }
        }
        __syncwarp();
        const RowMoments m = gather_rows(g, rows, tg_base, sw, t.ti.sy, dy0);
        if (walk) finish_rows(a.stage, i, load_rec(a.srecs + i), t.ti, m);
        if (generic) gather_generic(a.srecs + i, t.ti, sw, a.cfg.spans, tg, i, a.stage);
        __syncwarp();
        for (uint32_t cm = __ballot_sync(0xFFFFFFFFu, coop); cm; cm &= cm - 1) {
            const int src = __ffs(cm) - 1;
            const uint32_t slot = __shfl_sync(0xFFFFFFFFu, i, src);
            gather_coop(a.srecs + slot, t.ti, sw, tg, slot, src, a.stage);
        }
    });
}

// Spreads the gradient records into the reference's outputs grad_Ep[N], grad_xp[2][N],
// grad_Mp[2][3][N] (column 2 of grad_Mp is zero, :212, :218) in photon order: each photon's
// record is one 32-byte gather through the plan's inverse map, the writes are coalesced.
// Photons that touch no pixel get zeros.
__device__ __forceinline__ void grad_record(const TileArgs& a, int64_t n, int64_t n_tile,
                                            uint32_t v, float4& lo, float4& hi) {
    const int64_t slot = (v & kWideBit) ? n_tile + int64_t(v & ~kWideBit) : int64_t(v);
    lo = make_float4(0.f, 0.f, 0.f, 0.f);
    hi = lo;
    if (v != kInvalidPos && slot < n) {
        const Words8 w = load_words8(a.stage + slot);
        lo = w.lo;
        hi = w.hi;
    }
}

__global__ __launch_bounds__(256) void grad_scatter_kernel(TileArgs a) {
    const int64_t n = a.ph.n;
    const int64_t n_tile = tile_count(a);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += int64_t(gridDim.x) * blockDim.x) {
        float4 lo, hi;
        grad_record(a, n, n_tile, __ldg(a.inv + i), lo, hi);
        a.gE[i] = lo.x;
        a.gX[i] = lo.y;
        a.gX[n + i] = lo.z;
        a.gM[i] = lo.w;
        a.gM[n + i] = hi.x;
        a.gM[2 * n + i] = 0.f;
        a.gM[3 * n + i] = hi.y;
        a.gM[4 * n + i] = hi.z;
        a.gM[5 * n + i] = 0.f;
    }
}

// The same for 4 photons per thread: quad q holds photons 4q..4q+3 and each output row takes
// them in one 16-byte store, two 8-byte stores or four 4-byte stores, as the row's start
// allows (row r starts N * r elements after its array's start, so for N not a multiple of 4
// rows differ in alignment). The last N % 4 photons are written one by one.
__device__ __forceinline__ void store_quad(float* p, float4 v) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    if ((a & 15) == 0) {
        *reinterpret_cast<float4*>(p) = v;
    } else if ((a & 7) == 0) {
        reinterpret_cast<float2*>(p)[0] = make_float2(v.x, v.y);
        reinterpret_cast<float2*>(p)[1] = make_float2(v.z, v.w);
    } else {
        p[0] = v.x; p[1] = v.y; p[2] = v.z; p[3] = v.w;
    }
}

__global__ __launch_bounds__(256) void grad_scatter4_kernel(TileArgs a) {
    const int64_t n = a.ph.n, nq = n >> 2;
    const int64_t n_tile = tile_count(a);
    const uint4* inv4 = reinterpret_cast<const uint4*>(a.inv);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int64_t q = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < nq;
         q += int64_t(gridDim.x) * blockDim.x) {
        const uint4 v = __ldg(inv4 + q);
        float4 l0, h0, l1, h1, l2, h2, l3, h3;
        grad_record(a, n, n_tile, v.x, l0, h0);
        grad_record(a, n, n_tile, v.y, l1, h1);
        grad_record(a, n, n_tile, v.z, l2, h2);
        grad_record(a, n, n_tile, v.w, l3, h3);
        const int64_t i = 4 * q;
        store_quad(a.gE + i, make_float4(l0.x, l1.x, l2.x, l3.x));
        store_quad(a.gX + i, make_float4(l0.y, l1.y, l2.y, l3.y));
        store_quad(a.gX + n + i, make_float4(l0.z, l1.z, l2.z, l3.z));
        store_quad(a.gM + i, make_float4(l0.w, l1.w, l2.w, l3.w));
        store_quad(a.gM + n + i, make_float4(h0.x, h1.x, h2.x, h3.x));
        store_quad(a.gM + 2 * n + i, z);
        store_quad(a.gM + 3 * n + i, make_float4(h0.y, h1.y, h2.y, h3.y));
        store_quad(a.gM + 4 * n + i, make_float4(h0.z, h1.z, h2.z, h3.z));
        store_quad(a.gM + 5 * n + i, z);
    }
    // the last n % 4 photons
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < (n & 3)) {
        const int64_t i = 4 * nq + t;
        float4 lo, hi;
        grad_record(a, n, n_tile, __ldg(a.inv + i), lo, hi);
        a.gE[i] = lo.x;
        a.gX[i] = lo.y;
        a.gX[n + i] = lo.z;
        a.gM[i] = lo.w;
        a.gM[n + i] = hi.x;
        a.gM[2 * n + i] = 0.f;
        a.gM[3 * n + i] = hi.y;
        a.gM[4 * n + i] = hi.z;
        a.gM[5 * n + i] = 0.f;
    }
}


constexpr int kTileThreads = 256;

// Grid of a persistent tile kernel: resident CTAs per SM x SMs, capped by the work.
template <auto Kernel>
int persistent_grid(size_t smem, int64_t n_units) {
    const int64_t g = int64_t(num_sms()) * resident_ctas<Kernel>(kTileThreads, smem);
    const int64_t need = n_units > 0 ? n_units : 1;
    return int(g < need ? g : need);
}

}  // namespace


// Dynamic shared memory of a tile kernel: the tile's region, sw x sw words.
size_t tile_smem(const TileArgs& a) { return size_t(a.cfg.sw) * size_t(a.cfg.sw) * 4; }

template <int MINB, bool ROWS>
cudaError_t launch_forward_t(const TileArgs& a, cudaStream_t st) {
    const size_t smem = tile_smem(a);
    constexpr auto kern = ROWS ? fwd_rows_kernel<kTileThreads, MINB>
                               : fwd_tiles_kernel<kTileThreads, MINB>;
    const cudaError_t e = allow_smem<kern>(smem);
    if (e != cudaSuccess) return e;
    const int64_t chunks = (a.ph.n + a.cfg.chunk - 1) / a.cfg.chunk;
    if (chunks <= 0) return cudaSuccess;
    kern<<<persistent_grid<kern>(smem, chunks), kTileThreads, smem, st>>>(a);
    return cudaGetLastError();
}

template <int MINB, bool ROWS>
cudaError_t launch_backward_t(const TileArgs& a, cudaStream_t st) {
    const size_t smem = tile_smem(a);
    constexpr auto kern = ROWS ? bwd_rows_kernel<kTileThreads, MINB>
                               : bwd_tiles_kernel<kTileThreads, MINB>;
    cudaError_t e = allow_smem<kern>(smem);
    if (e != cudaSuccess) return e;
    const int64_t chunks = (a.ph.n + a.cfg.chunk - 1) / a.cfg.chunk;
    if (chunks <= 0) return cudaSuccess;
    kern<<<persistent_grid<kern>(smem, chunks), kTileThreads, smem, st>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // no outputs: the gradients stay in the workspace as records (read by the refraction
    // backward's records mode)
    if (!a.gE) return cudaSuccess;
    // the quad form needs the inverse map 16-byte aligned (the workspace is) and every
    // output 4-byte aligned; the rows' own alignment is handled per store
    const auto al = [](const void* p, uintptr_t m) {
        return (reinterpret_cast<uintptr_t>(p) & m) == 0;
    };
    const bool vec = al(a.inv, 15) && al(a.gE, 3) && al(a.gX, 3) && al(a.gM, 3);
    const int64_t items = vec ? a.ph.n / 4 : a.ph.n;
    const int64_t sblocks = items > 0 ? (items + 255) / 256 : 1;
    const int64_t scap = int64_t(num_sms()) * 16;
    const unsigned sgrid = unsigned(sblocks < scap ? sblocks : scap);
    if (vec)
        grad_scatter4_kernel<<<sgrid, 256, 0, st>>>(a);
    else
        grad_scatter_kernel<<<sgrid, 256, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_forward(const TileArgs& a, cudaStream_t st) {
    if (a.cfg.rows) {
        if (a.cfg.min_blocks >= 4) return launch_forward_t<4, true>(a, st);
        return a.cfg.min_blocks == 3 ? launch_forward_t<3, true>(a, st)
                                     : launch_forward_t<2, true>(a, st);
    }
    if (a.cfg.min_blocks >= 4) return launch_forward_t<4, false>(a, st);
    return a.cfg.min_blocks == 3 ? launch_forward_t<3, false>(a, st)
                                 : launch_forward_t<2, false>(a, st);
}

cudaError_t launch_backward(const TileArgs& a, cudaStream_t st) {
    if (a.cfg.rows) {
        if (a.cfg.min_blocks >= 4) return launch_backward_t<4, true>(a, st);
        return a.cfg.min_blocks == 3 ? launch_backward_t<3, true>(a, st)
                                     : launch_backward_t<2, true>(a, st);
    }
    if (a.cfg.min_blocks >= 4) return launch_backward_t<4, false>(a, st);
    return a.cfg.min_blocks == 3 ? launch_backward_t<3, false>(a, st)
                                 : launch_backward_t<2, false>(a, st);
}

}  // namespace pds
