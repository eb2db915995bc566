// blend.cu — kernel (e): per-tile front-to-back alpha blending, and its adjoint.
//
// Reference: blend.slang:24-105 (one 16x16 workgroup per tile; rounds of 256
// splats staged in shared memory; per pixel: power, alpha = min(0.99,
// o*exp(power)), skip below 1/255, stop when T*(1-alpha) < 1e-4; colour
// gathered per contributing pair) dispatched by GaussianEngine.cpp:857-862.
// The reference has no backward pass; blend_backward_kernel is new.
//
// GB300 form: one CTA of 128 threads per tile, each lane on two pixels whose
// pair arithmetic runs in packed f32x2 operations; each round stages
// position, conic+opacity and colour of the next list entries into shared
// memory (colour is staged with the rest instead of gathered per pair), the
// whole CTA leaves as soon as every pixel is done (__syncthreads_count), and
// per pixel the final transmittance and the number of list entries up to the
// last contributor are kept for the adjoint. The adjoint walks each tile's
// list back to front, recomputing transmittance as T / (1 - alpha) from the
// final T (no per-pixel lists). It stores each entry's sums per 8x4 block in
// shared memory and adds them to the Gaussian's record with vector atomics, once
// per round and entry.
//
// Every per-pixel operation (n2, alpha, the skip and stop tests) has the same
// operations and explicit rounding in the forward and in the adjoint, so both
// take identical decisions.
//
// Block culling: the tile is four blocks of 8x8 pixels (the forward: one per
// warp) or eight of 8x4 (the adjoint: four per warp). The thread that
// stages a list entry also works out, once for the whole CTA, which of the
// tile's blocks the entry can reach: for each block row (a slab of
// pixel rows) it takes the x extent of the entry's alpha >= 1/255 ellipse
// within the slab (closed form, two square roots), enlarged for rounding,
// and compares it with the two block columns. Only the entries whose bit for
// a block is set are walked for it (found by one ballot per 32 entries). A
// culled pair lies outside that ellipse, where the pair's own test finds
// alpha below 1/255 and skips it, as the reference does; so the culling
// changes which skipped pairs are visited, never a result.
#include <algorithm>
#include <type_traits>

#include "tpd_common.cuh"
#include "tpd_kernels.h"
#include "tpd_scan.cuh"

namespace tpd {
namespace {

constexpr float kAlphaMax = 0.99f;
constexpr float kTMin = 0.0001f;

constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// Per (pixel, entry) pair, with the conic pre-scaled at staging
//   qa = 0.5 log2e cx, qb = log2e cy, qc = 0.5 log2e cz,
//   dx = x - px, dy = y - py (rounded subtractions),
//   n2 = fma(fma(qb, dy, qa dx), dx, (qc dy) dy) = -log2(e) * power,
//   power = -0.5 * (cx*dx*dx + cz*dy*dy) - cy*dx*dy  (blend.slang:83-84),
// five multiply/fma operations; exp(power) = 2^-n2 is one ex2, and
//   alpha = min(0.99, o * 2^-n2) < 1/255  <=>  n2 > -thr, thr = log2(1 / (255 o))
// is decided before the exponential. The pair counts when power <= 0 and alpha
// >= 1/255, i.e. 0 <= n2 <= -thr: floats of that range ascend as unsigned
// integers and negative ones lie above them, so one integer comparison of n2's
// bits with keep_limit decides both. ((qc dy) dy is taken as a fused
// multiply-add onto +0, so that n2 is never -0 unless its terms underflow.)
// With a comparison for each the blend of 1M Gaussians at 1080p took 249 us,
// with one 239 (8 views of 1.5M: 1621 and 1525); the adjoint of 500,000 in 8
// views 1140 and 1124.

constexpr float kInf = __builtin_huge_valf();

__device__ __forceinline__ float sqrt_approx(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Blocks of the tile at pixel origin (ox, oy) that the entry can reach, for
// blocks 8 pixels wide and 16 / kSlabs high: bit 2k + c for block row k
// (pixel rows oy + hk .. oy + hk + h - 1, h = 16 / kSlabs) and block column c
// (pixel columns ox + 8c .. ox + 8c + 7), the block of warp 2k + c.
//
// With a = -qa, b = -qb / 2, c = -qc and d = centre - pixel, a pixel is kept
// only when n2 <= -thr, i.e. inside the ellipse a dx^2 + 2b dx dy + c dy^2 <= R
// for R = -thr. R is enlarged by 4e-3 (relative and absolute) plus 1e-5 ac/det
// relative, which bounds the rounding of the per-pixel n2 even for thin
// ellipses (its terms are at most 4 R ac / det in size there). For dy in a
// slab, the ellipse spans dx in [(-b dy - s) / a, (-b dy + s) / a],
// s = sqrt(a R - det dy^2); over the slab the extremes are +-hx (hx =
// sqrt(c R / det)) when the slab holds the extreme point's dy (-+b hx / c),
// else the values at the slab's ends. The x extent is widened by 0.02 px +
// 1e-4 hx for the rounding of this computation. thr > 0 (opacity below
// 1/255) never blends: no block; a conic that is not positive definite is
// never culled: every block.
template <int kSlabs>
__device__ __forceinline__ uint32_t block_mask(float cx, float cy, float4 q, float ox, float oy) {
    constexpr float kSlabRows = float(kBlockY / kSlabs);  // pixel rows per block row
    const float thr = q.w;
    if (!(thr <= 0.0f)) return 0u;
    const float a = -q.x, c = -q.z, b = -0.5f * q.y;
    const float w = b * b;
    const float det = __fmaf_rn(a, c, -w) + __fmaf_rn(-b, b, w);  // compensated a c - b^2
    if (!(a > 0.0f && c > 0.0f && det > 0.0f)) return 0xFFu;
    const float inv_det = rcp_approx(det), inv_a = rcp_approx(a);
    const float R = -thr * (1.0f + 4e-3f + 1e-5f * (a * c * inv_det)) + 4e-3f;
    const float hx = sqrt_approx(c * R * inv_det), hy = sqrt_approx(a * R * inv_det);
    const float dyr = -b * hx * rcp_approx(c);  // dy of the rightmost point; the leftmost at -dyr
    const float aR = a * R;
    const float wx = 0.02f + 1e-4f * hx;
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < kSlabs; ++k) {
        const float y0 = oy + kSlabRows * float(k);
        float dlo = cy - (y0 + (kSlabRows - 1.0f)) - 0.01f, dhi = cy - y0 + 0.01f;
        if (dhi < -hy || dlo > hy) continue;
        dlo = fmaxf(dlo, -hy);
        dhi = fminf(dhi, hy);
        const float s0 = sqrt_approx(fmaxf(__fmaf_rn(-det, dlo * dlo, aR), 0.0f));
        const float s1 = sqrt_approx(fmaxf(__fmaf_rn(-det, dhi * dhi, aR), 0.0f));
        float xmax = fmaxf((-b * dlo + s0) * inv_a, (-b * dhi + s1) * inv_a);
        float xmin = fminf((-b * dlo - s0) * inv_a, (-b * dhi - s1) * inv_a);
        if (dyr >= dlo && dyr <= dhi) xmax = hx;
        if (-dyr >= dlo && -dyr <= dhi) xmin = -hx;
        const float pxlo = cx - xmax - wx, pxhi = cx - xmin + wx;  // pixel x = centre x - dx
        if (pxlo <= ox + 7.0f && pxhi >= ox) m |= 1u << (2 * k);
        if (pxlo <= ox + 15.0f && pxhi >= ox + 8.0f) m |= 2u << (2 * k);
    }
    return m;
}

__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// UNORM RGBA8 of (r, g, b, 1): round(clamp(c, 0, 1) * 255) per channel.
__device__ __forceinline__ uint32_t rgba8_unorm(float r, float g, float b) {
    const float c[3] = {r, g, b};
    uint32_t out = 0xFF000000u;
#pragma unroll
    for (int k = 0; k < 3; ++k) out |= uint32_t(__float2uint_rn(fminf(fmaxf(c[k], 0.0f), 1.0f) * 255.0f)) << (8 * k);
    return out;
}

// The bits of n2 below which a pair counts, for q = (-qa, -qb, -qc, thr):
// one above the bits of -thr, or 0 (no pair) when thr > 0. A conic that is not a
// number (its covariance's determinant overflowed) gives n2 = NaN in every
// pixel, which neither test skips: all bits are below the limit then. (No conic
// is infinite: a determinant that is not 0 is at least an ulp of the products,
// of numbers of at least 0.3, whose difference it is.)
__device__ __forceinline__ uint32_t keep_limit(float4 q) {
    const float sum = q.x + q.y + q.z;
    return sum != sum ? 0xFFFFFFFFu : q.w <= 0.0f ? __float_as_uint(0.0f - q.w) + 1u : 0u;
}

// View of a global tile id, that view's size, and the tile's (column, row) in it.
__device__ __forceinline__ void load_view_tile(const ViewConst* views, const uint32_t* tile_view, uint32_t tile,
                                               uint32_t& vi, uint32_t& width, uint32_t& height, uint32_t& tx,
                                               uint32_t& ty) {
    vi = tile_view ? tile_view[tile] : 0u;
    const ViewConst& v = views[vi];
    width = v.width;
    height = v.height;
    const uint32_t local = tile - v.tile_base;
    const uint32_t gx = grid_x(width);
    tx = local % gx;
    ty = local / gx;
}

// ---- forward
//
// A CTA of 128 threads per tile. Warp w owns the 8x8 block at (8 (w & 1),
// 8 (w >> 1)) of the tile, and lane l the two pixels (l & 7, l >> 3) and
// (l & 7, (l >> 3) + 4) of that block. The two pixels of a lane share dx, and
// the arithmetic of a (pixel, entry) pair runs on both pixels at once with
// packed f32x2 operations: per pixel the operations, order and rounding
// given above for n2, alpha and the tests, as in the adjoint. A staged entry
// holds its values duplicated in register-pair order, so the packed operands
// come straight out of five broadcast shared-memory loads.
constexpr uint32_t kFwdThreads = 128;
// List entries per staged round (the blend's batch depth, an engine setting
// the autotuner picks): 128 by default (20 KB of shared memory, 8 CTAs per
// SM at 64 registers); 64 (8 CTAs) or 256 (41 KB, 5 CTAs).
template <uint32_t kRound>
constexpr int fwd_min_blocks() { return kRound >= 256 ? 5 : 8; }

struct PairStaged {  // 80 bytes
    float4 xy;       // x, x, y, y
    float4 qab;      // qa, qa, qb, qb
    float4 qco;      // qc, qc, opacity, opacity
    float4 rg;       // r, r, g, g
    float4 bt;       // b, b, keep_limit (bits), 0
};

template <uint32_t kRound>
struct FwdStage {
    PairStaged e[2][kRound];
    uint8_t mask[2][kRound];  // bit w: the entry can reach warp w's 8x8 block
    uint32_t wlast[kFwdThreads / 32];
};

__device__ __forceinline__ void stage_pair_values(float4 c, float4 tex, float4 co, float ox, float oy, PairStaged& d,
                                                  uint8_t& mask) {
    const float thr = co.w > 0.0f ? -__log2f(255.0f * co.w) : kInf;  // +inf: never blends
    const float4 q = make_float4(-0.5f * kLog2e * co.x, -kLog2e * co.y, -0.5f * kLog2e * co.z, thr);
    d.xy = make_float4(tex.x, tex.x, tex.y, tex.y);
    d.qab = make_float4(-q.x, -q.x, -q.y, -q.y);
    d.qco = make_float4(-q.z, -q.z, co.w, co.w);
    d.rg = make_float4(c.x, c.x, c.y, c.y);
    d.bt = make_float4(c.z, c.z, __uint_as_float(keep_limit(q)), 0.0f);
    mask = uint8_t(block_mask<2>(tex.x, tex.y, q, ox, oy));
}

__device__ __forceinline__ void stage_pair_entry(const Splat* sp, float ox, float oy, PairStaged& d, uint8_t& mask) {
    const float4* p = reinterpret_cast<const float4*>(sp);
    stage_pair_values(__ldg(p + 0), __ldg(p + 1), __ldg(p + 2), ox, oy, d, mask);
}

__device__ __forceinline__ void stage_pair_empty(PairStaged& d, uint8_t& mask) {
    d.xy = d.qab = d.qco = d.rg = d.bt = make_float4(0.f, 0.f, 0.f, 0.f);  // (limit 0: no pair counts)
    mask = 0u;
}

// A gradient or a pixel's colour beyond this is walked apart by the adjoint (see
// there); the blend marks the tile_len of tiles with such a colour.
constexpr float kHuge = 1e18f;
constexpr uint32_t kTileHuge = 1u << 31;

// Class of a walk of len entries, longer walks first: quarter octaves of len + 1.
__device__ __forceinline__ uint32_t tile_class(uint32_t len) {
    const uint32_t o = 31u - __clz(len + 1u);  // len < 2^31: the class is below 128
    const uint32_t quarter = o >= 2u ? ((len + 1u) >> (o - 2u)) & 3u : ((len + 1u) << (2u - o)) & 3u;
    return 127u - (4u * o + quarter);
}

// One tile: rounds of kRound list entries, double-buffered: while the warps
// walk round r, each thread stages its entry of round r + 1 into the other
// buffer, and one barrier per round (which also counts finished pixels)
// separates the two. Called by the whole CTA; the first barrier comes after
// the first staging and the last one after every read of S. kState: also
// track and store each pixel's final transmittance and last contributor (the
// adjoint's inputs); a frame that no backward follows skips that work.
template <uint32_t kRound, bool kState>
__device__ __forceinline__ void blend_tile(const BlendArgs& a, uint32_t tile, FwdStage<kRound>& S) {
    uint32_t vi, W, H, tx, ty;
    load_view_tile(a.views, a.tile_view, tile, vi, W, H, tx, ty);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t px = tx * kBlockX + 8u * (warp & 1u) + (lane & 7u);
    const uint32_t pya = ty * kBlockY + 8u * (warp >> 1) + (lane >> 3), pyb = pya + 4u;
    const float ox = float(tx * kBlockX), oy = float(ty * kBlockY);
    const bool in_a = px < W && pya < H, in_b = px < W && pyb < H;
    const float2 npx = make_float2(-float(px), -float(px));
    const float2 npy = make_float2(-float(pya), -float(pyb));
    const uint32_t K = min(a.ctl->total_keys, a.capacity);
    const uint32_t raw_start = a.ranges[tile * 2 + 0], raw_end = a.ranges[tile * 2 + 1];
    const uint32_t end = min(raw_end, K), start = min(raw_start, end);
    // a tile without keys still holds the sort's preset (0xFFFFFFFF, 0): store
    // the reference's empty range (0, 0)
    if (tid == 0 && raw_start > raw_end) a.ranges[tile * 2 + 0] = 0u;
    const Splat* vsplats = a.splats + size_t(vi) * a.n;

    // entries j0 + tid, j0 + tid + 128, ... (below j0 + kRound) of the list into buffer buf
    auto stage = [&](uint32_t buf, uint32_t j0) {
#pragma unroll
        for (uint32_t k = tid; k < kRound; k += kFwdThreads) {
            const uint32_t j = j0 + k;
            if (j >= end || !TPD_INBOUNDS(a.ctl, 40, j, a.capacity)) continue;
            const uint32_t idx = a.vals[j];
            if (idx < a.n && TPD_INBOUNDS(a.ctl, 42, idx, a.n))
                stage_pair_entry(vsplats + idx, ox, oy, S.e[buf][k], S.mask[buf][k]);
            else
                stage_pair_empty(S.e[buf][k], S.mask[buf][k]);  // only reachable with corrupted lists
        }
    };

    // A pixel that stops is frozen at T = 0: every later pair then adds
    // exactly nothing, so no per-pixel done flags are needed (pixels outside
    // the image start frozen). With the adjoint's inputs, Tk keeps the
    // transmittance at the stop, which is what the reference leaves.
    float2 T = make_float2(in_a ? 1.0f : 0.0f, in_b ? 1.0f : 0.0f);
    float2 Tk = make_float2(1.0f, 1.0f);  // kState: the transmittance to store (it stays at the stop)
    float2 C0 = make_float2(0.f, 0.f), C1 = C0, C2 = C0;
    uint32_t last_a = 0, last_b = 0;
    const float2 one = make_float2(1.0f, 1.0f), mone = make_float2(-1.0f, -1.0f);
    auto pixels_done = [&]() { return T.x == 0.0f && T.y == 0.0f; };
    if (start < end) stage(0, start);
    bool all_done = __syncthreads_count(pixels_done()) == kFwdThreads;
    uint32_t r = 0;
    for (uint32_t b0 = start; b0 < end && !all_done; b0 += kRound, ++r) {
        const uint32_t b = r & 1u;
        // the next round's entries, into the buffer the last barrier released
        if (b0 + kRound < end) stage(b ^ 1u, b0 + kRound);
        const uint32_t n = min(kRound, end - b0);
        const uint32_t lbase = b0 - start + 1u;  // n_contrib of entry jj of this round: lbase + jj
        for (uint32_t g = 0; g < n; g += 32) {
            if (__all_sync(0xFFFFFFFFu, pixels_done())) break;
            const uint32_t e = g + lane;
            uint32_t m = __ballot_sync(0xFFFFFFFFu, e < n && ((S.mask[b][e] >> warp) & 1u));
            // branch-free body: every lane evaluates both pairs and selects
            // the update, so lanes taking different decisions do not run the
            // paths one after another. A skipped pair gets alpha = 0, which
            // leaves T and C exactly as they were.
            // alpha of a staged entry for both pixels (0 when the pair is skipped)
            auto alpha_of = [&](const PairStaged& E) {
                const float4 xy = E.xy, qab = E.qab, qco = E.qco, bt = E.bt;
                const float2 dx = __fadd2_rn(make_float2(xy.x, xy.y), npx);
                const float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), npy);
                const float2 t = __ffma2_rn(make_float2(qab.z, qab.w), dy, __fmul2_rn(make_float2(qab.x, qab.y), dx));
                const float2 qcdy = __fmul2_rn(make_float2(qco.x, qco.y), dy);
                const float2 n2 = __ffma2_rn(t, dx, __ffma2_rn(qcdy, dy, make_float2(0.0f, 0.0f)));
                const float2 ao =
                    __fmul2_rn(make_float2(qco.z, qco.w), make_float2(ex2_approx(-n2.x), ex2_approx(-n2.y)));
                const uint32_t limit = __float_as_uint(bt.z);
                return make_float2(__float_as_uint(n2.x) < limit ? fminf(kAlphaMax, ao.x) : 0.0f,
                                   __float_as_uint(n2.y) < limit ? fminf(kAlphaMax, ao.y) : 0.0f);
            };
            // the pair's update, in list order. T becomes 0 at the stop and
            // stays so after it (T = 0 gives tn = 0): the pair adds alpha * 0
            // and leaves T = 0; before the stop the second product with 1 -
            // alpha is tn again. With the adjoint's inputs, Tk keeps the transmittance at
            // the stop and the last entry that added is the last with w > 0
            // (alpha >= 1/255 times T >= 1e-4).
            auto apply = [&](float2 alpha, const PairStaged& E, uint32_t jj) {
                const float4 rg = E.rg, bt = E.bt;
                const float2 om = __ffma2_rn(mone, alpha, one);
                const float2 tn = __fmul2_rn(T, om);  // T (1 - alpha)
                const bool go_a = !(tn.x < kTMin), go_b = !(tn.y < kTMin);
                T = make_float2(go_a ? T.x : 0.0f, go_b ? T.y : 0.0f);
                const float2 w = __fmul2_rn(alpha, T);
                C0 = __ffma2_rn(make_float2(rg.x, rg.y), w, C0);
                C1 = __ffma2_rn(make_float2(rg.z, rg.w), w, C1);
                C2 = __ffma2_rn(make_float2(bt.x, bt.y), w, C2);
                T = __fmul2_rn(T, om);
                if constexpr (kState) {
                    Tk = make_float2(go_a ? tn.x : Tk.x, go_b ? tn.y : Tk.y);
                    last_a = w.x > 0.0f ? lbase + jj : last_a;
                    last_b = w.y > 0.0f ? lbase + jj : last_b;
                }
            };
            // two entries per step when there are two: their alphas are
            // independent, only the updates run in order (with the adjoint's
            // inputs: 670 -> 652 us for 8 views of 500,000 at 720p, 1514 -> 1470
            // for 8 of 1.5M at 1080p)
            while (m) {
                const uint32_t j0 = g + uint32_t(__ffs(m) - 1);
                m &= m - 1u;
                if (m) {
                    const uint32_t j1 = g + uint32_t(__ffs(m) - 1);
                    m &= m - 1u;
                    const PairStaged &E0 = S.e[b][j0], &E1 = S.e[b][j1];
                    const float2 a0 = alpha_of(E0), a1 = alpha_of(E1);
                    apply(a0, E0, j0);
                    apply(a1, E1, j1);
                } else {
                    const PairStaged& E0 = S.e[b][j0];
                    apply(alpha_of(E0), E0, j0);
                }
            }
        }
        all_done = __syncthreads_count(pixels_done()) == kFwdThreads;
    }
    if constexpr (kState) {
        const uint32_t wl = __reduce_max_sync(0xFFFFFFFFu, max(last_a, last_b));
        // (an infinite colour makes every pixel that meets it infinite or not a
        // number, whether the pixel counts it or not: 0 times infinity)
        const float sum = fabsf(C0.x) + fabsf(C1.x) + fabsf(C2.x) + fabsf(C0.y) + fabsf(C1.y) + fabsf(C2.y);
        const bool huge = __any_sync(0xFFFFFFFFu, !(sum <= kHuge));
        if (lane == 0) S.wlast[warp] = wl | (huge ? kTileHuge : 0u);
        __syncthreads();
        if (tid == 0 && TPD_INBOUNDS(a.ctl, 43, tile, a.n_tiles)) {
            const uint32_t w0 = S.wlast[0], w1 = S.wlast[1], w2 = S.wlast[2], w3 = S.wlast[3];
            const uint32_t len = max(max(w0 & ~kTileHuge, w1 & ~kTileHuge), max(w2 & ~kTileHuge, w3 & ~kTileHuge));
            a.tile_len[tile] = len | ((w0 | w1 | w2 | w3) & kTileHuge);
            atomicAdd(&a.ctl->tile_hist[tile_class(len)], 1u);
        }
    }
    if (TPD_INBOUNDS(a.ctl, 41, tile, a.n_tiles)) {
        const size_t img0 = a.image_offset ? a.image_offset[vi] : 0ull;
        if (in_a) {
            const size_t p = img0 + size_t(pya) * W + px;
            a.image[p * 3 + 0] = C0.x;
            a.image[p * 3 + 1] = C1.x;
            a.image[p * 3 + 2] = C2.x;
            if (a.rgba) a.rgba[p] = rgba8_unorm(C0.x, C1.x, C2.x);
            if constexpr (kState) {
                a.final_T[p] = Tk.x;
                a.n_contrib[p] = last_a;
            }
        }
        if (in_b) {
            const size_t p = img0 + size_t(pyb) * W + px;
            a.image[p * 3 + 0] = C0.y;
            a.image[p * 3 + 1] = C1.y;
            a.image[p * 3 + 2] = C2.y;
            if (a.rgba) a.rgba[p] = rgba8_unorm(C0.y, C1.y, C2.y);
            if constexpr (kState) {
                a.final_T[p] = Tk.y;
                a.n_contrib[p] = last_b;
            }
        }
    }
}

// The tile scheduler of a persistent launch: the CTA takes the next item of
// the frame's tile queue (an atomic ticket in FrameCtl) until the queue is
// empty; item i is tile order[i] (nullptr: tile i). Every tile of every view
// is one item, so one launch balances all views' tiles at once.
__device__ __forceinline__ bool next_tile(FrameCtl* ctl, uint32_t slot, const uint32_t* order, uint32_t n_tiles,
                                          uint32_t& tile) {
    __shared__ uint32_t s_item;
    if (threadIdx.x == 0) s_item = atomicAdd(&ctl->ticket[slot], 1u);
    __syncthreads();
    const uint32_t i = s_item;
    __syncthreads();  // every thread has read s_item before it is written again
    if (i >= n_tiles) return false;
    tile = order ? order[i] : i;
    return true;
}

// Item i of the tiles in class order (buckets as launch_list_classes fills
// them): the class whose tiles item i falls among, by a scan of their counts.
__device__ __forceinline__ uint32_t class_tile(const FrameCtl* ctl, const uint32_t* buckets, uint32_t n_tiles, uint32_t i) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t incl = warp_inclusive_scan(lane < kListClasses ? __ldcg(&ctl->list_class[lane]) : 0u);
    const uint32_t after = __ballot_sync(0xFFFFFFFFu, incl > i);  // classes that end past item i
    const uint32_t c = after ? uint32_t(__ffs(after) - 1) : 0u;
    const uint32_t before = c ? __shfl_sync(0xFFFFFFFFu, incl, c - 1u) : 0u;
    return after ? __ldcg(buckets + size_t(c) * n_tiles + (i - before)) : i;
}

// One CTA per tile, or (kPersistent) one CTA per resident slot taking tiles
// from the queue.
template <uint32_t kRound, bool kPersistent, bool kState>
__global__ void __launch_bounds__(kFwdThreads, fwd_min_blocks<kRound>()) blend_kernel(BlendArgs a) {
    __shared__ FwdStage<kRound> S;
    pdl_wait();  // launched as a dependent of the key sort's last pass: its lists and ranges
    pdl_trigger();
    // an overflowed frame is re-rendered with larger key buffers; nothing to draw
    if (a.ctl->status & (kStatusFatal | kStatusKeyOverflow)) return;
    if constexpr (kPersistent) {
        uint32_t tile;
        while (next_tile(a.ctl, kTicketBlend, nullptr, a.n_tiles, tile))
            blend_tile<kRound, kState>(a, a.list_buckets ? class_tile(a.ctl, a.list_buckets, a.n_tiles, tile) : tile, S);
    } else {
        blend_tile<kRound, kState>(
            a, a.list_buckets ? class_tile(a.ctl, a.list_buckets, a.n_tiles, blockIdx.x) : blockIdx.x, S);
    }
}

// UNORM conversion of (r, g, b, 1): round(clamp(c, 0, 1) * 255).
__global__ void pack_rgba8_kernel(const float* rgb, uint32_t* rgba, size_t pixels) {
    pdl_wait();  // launched as a dependent of the blend
    pdl_trigger();
    const size_t i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= pixels) return;
    rgba[i] = rgba8_unorm(rgb[i * 3 + 0], rgb[i * 3 + 1], rgb[i * 3 + 2]);
}

// ---- adjoint
//
// A CTA of 64 threads per tile. The tile is eight blocks of 8x4 pixels (block
// 2k + c: rows 4k .. 4k + 3, columns 8c .. 8c + 7); eight lanes own a block,
// one pixel column of four rows each, so warp w holds blocks 4w .. 4w + 3.
// Every block walks its own list of the entries that reach it (from the back:
// slot k of a round holds its k-th entry from the end): a warp's step takes
// one entry per block, and the four entries usually differ. The pixels of a
// lane share dx, and their arithmetic runs two rows at a time in packed f32x2
// operations, per pixel with the forward's operations, order and rounding for
// n2, alpha and the tests. A staged entry holds the values that the packed
// operations take duplicated in register-pair order.
//
// Per pixel, with g = dL/dimage, and going from the back: T after an entry
// gives T / (1 - alpha) in front of it, w = alpha T_front is its weight, and
// A, the colours behind it blended with each other and dotted with g, follows
// A <- A + alpha (g.c - A); then dL/dalpha = T_front (g.c - A). A skipped pair
// has alpha = 0, which leaves T and A as they are (1 / (1 - 0) is exactly 1).
//
// Sums per (block, entry). With P = dL/dpower (power = -n2 ln2) the record's
// gradients follow from nine sums over pixels: P, P dx, P dy, P dx^2, P dx dy,
// P dy^2 and w g (three). A lane's four pixels share dx, so it adds P, P dy
// and P dy^2 over them first and multiplies by dx afterwards; eight of the
// nine are then summed over the block's eight lanes by a transposed butterfly
// (seven exchanges, lane j ends with sum j), the ninth by three more. A block
// meets an entry once per round, so the sums are stored, not added: no
// shared-memory atomics. At the end of the round one thread per entry adds
// the blocks' sums (those whose bit is set), turns them into gradients with
// the entry's conic, and adds them to the global record with vector atomics.
//
// Against one 8x8 block per warp with two pixels a lane and the nine gradients
// of every pixel pair summed by shuffles and shared-memory atomics: 96M
// instead of 185M warp instructions for 200,000 Gaussians at 800x800, 234 ->
// 131 us; 8 views of 500,000 at 1280x720 1856 -> 1119 us; 5,003 at 201x151 90
// -> 58 us; 8 views of 6M at 2160p 20.5 -> 12.6 ms. It issues on 55% of the
// cycles (16 warps per SM, by its registers and the blocks' sums; rounds of 32
// with 20 warps measured 3% slower, rounds of 128 with 8 warps 38%), ALU and
// FMA pipes at 44% and 41%; the last tiles leave 15% of the SM time idle.
// The forward gained nothing from this layout (249 us at 1M Gaussians and
// 1080p either way, and a mid-sized frame's longest tile took 94 us on two
// warps instead of 72 on four), so it keeps one 8x8 block per warp.
//
// List entries per round (an engine setting the autotuner picks): 64 by
// default, 32 or 128.
constexpr uint32_t kAdjThreads = 64;
// A tile with a gradient or a colour beyond kHuge, an infinite one or one that is
// not a number is walked with arithmetic that keeps it to the entries its pixel
// counts: g.c may overflow, and 0 times infinity is no zero. There S, the
// colours behind an entry, takes A's place, dL/dalpha = g.(T_front c - S / (1 -
// alpha)), and a pair that does not count is selected away instead of
// multiplied by 0. The usual walk loses nothing by having it beside: a step of
// 8 views of 2160p 26810 us without it, 26828 with; selecting the power
// gradient in the usual walk, for infinite colours, 26920.
constexpr uint32_t kBlendBlocks = 8;  // 8x4 blocks of a tile

struct BlockStaged {  // 80 bytes
    float4 s;         // x, qa, keep_limit (bits), 0
    float4 yb;        // y, y, qb, qb
    float4 qco;       // qc, qc, opacity, opacity
    float4 rg;        // r, r, g, g
    float2 b;         // b, b
    float2 pad;
};

__device__ __forceinline__ void stage_block_values(float4 c, float4 tex, float4 co, float ox, float oy, BlockStaged& d,
                                                   uint8_t& mask) {
    const float thr = co.w > 0.0f ? -__log2f(255.0f * co.w) : kInf;  // +inf: never blends
    const float4 q = make_float4(-0.5f * kLog2e * co.x, -kLog2e * co.y, -0.5f * kLog2e * co.z, thr);
    d.s = make_float4(tex.x, -q.x, __uint_as_float(keep_limit(q)), 0.0f);
    d.yb = make_float4(tex.y, tex.y, -q.y, -q.y);
    d.qco = make_float4(-q.z, -q.z, co.w, co.w);
    d.rg = make_float4(c.x, c.x, c.y, c.y);
    d.b = make_float2(c.z, c.z);
    mask = uint8_t(block_mask<4>(tex.x, tex.y, q, ox, oy));
}

__device__ __forceinline__ void stage_block_empty(BlockStaged& d) {
    d.s = make_float4(0.f, 0.f, 0.f, 0.f);
    d.yb = d.qco = d.rg = make_float4(0.f, 0.f, 0.f, 0.f);
    d.b = make_float2(0.f, 0.f);
}

// Entries of a round for each block of a warp, in list order (BlockLists).
template <uint32_t kRound>
struct BlockLists {
    static constexpr uint32_t kEmpty = kRound;  // the staged slot that never blends
    uint16_t e[kBlendBlocks][kRound + 2];
};

// The lists of the calling warp's four blocks for a round of n entries:
// `nibble(e)` gives entry e's bits for them (called for e < n). Returns the
// steps of the walk, a multiple of two: the longest list's length, to which
// the shorter ones are filled up with the empty slot.
template <uint32_t kRound, typename Nibble>
__device__ __forceinline__ uint32_t build_block_lists(BlockLists<kRound>& L, uint32_t warp, uint32_t lane, uint32_t n,
                                                      Nibble nibble) {
    uint32_t cnt[4] = {0u, 0u, 0u, 0u};
    const uint32_t lt = (1u << lane) - 1u;
    for (uint32_t c = 0; c < n; c += 32u) {
        const uint32_t e = c + lane;
        const uint32_t m = e < n ? nibble(e) : 0u;
#pragma unroll
        for (uint32_t g = 0; g < 4; ++g) {
            const bool on = (m >> g) & 1u;
            const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
            if (on) L.e[4 * warp + g][cnt[g] + __popc(bal & lt)] = uint16_t(e);
            cnt[g] += __popc(bal);
        }
    }
    const uint32_t steps = (max(max(cnt[0], cnt[1]), max(cnt[2], cnt[3])) + 1u) & ~1u;
    const uint32_t g = lane >> 3;
    const uint32_t mine = g == 0 ? cnt[0] : g == 1 ? cnt[1] : g == 2 ? cnt[2] : cnt[3];
    for (uint32_t i = mine + (lane & 7u); i < steps; i += 8u) L.e[4 * warp + g][i] = uint16_t(L.kEmpty);
    __syncwarp();
    return steps;
}

// A lane's four pixels: the column and rows, in packed order.
struct LanePixels {
    uint32_t x, y;       // the first row's pixel
    float nx;            // -x
    float2 ny0, ny1;     // -(y, y + 1), -(y + 2, y + 3)
    bool in[4];
    __device__ __forceinline__ LanePixels(uint32_t tx, uint32_t ty, uint32_t warp, uint32_t lane, uint32_t W,
                                          uint32_t H) {
        const uint32_t block = 4u * warp + (lane >> 3);
        x = tx * kBlockX + 8u * (block & 1u) + (lane & 7u);
        y = ty * kBlockY + 4u * (block >> 1);
        nx = -float(x);
        ny0 = make_float2(-float(y), -float(y + 1u));
        ny1 = make_float2(-float(y + 2u), -float(y + 3u));
#pragma unroll
        for (uint32_t r = 0; r < 4; ++r) in[r] = x < W && y + r < H;
    }
};

template <uint32_t kBwdRound>
constexpr int bwd_min_blocks() { return kBwdRound >= 128 ? 4 : kBwdRound >= 64 ? 8 : 10; }
template <uint32_t kBwdRound>
struct BlendBackwardSmem {
    BlockStaged e[kBwdRound + 1];                     // slot kBwdRound: an entry that never blends
    float sums[kBlendBlocks][(kBwdRound + 1) * 8];   // eight per (block, entry); a row's length sets blocks 8 banks apart
    float sum9[kBlendBlocks][kBwdRound + 1];
    BlockLists<kBwdRound> lists;
    uint32_t idx[kBwdRound];
    uint32_t wmax[kAdjThreads / 32];
    uint8_t mask[kBwdRound];
    uint8_t met[kAdjThreads / 32][kBwdRound];  // blocks of the warp that have sums of the entry
};

__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float hsum(float2 a) { return a.x + a.y; }

// Sums v[0..7] over each group of eight lanes with a transposed butterfly:
// each exchange halves the values a lane holds. Lane j of a group returns the
// sum of v[j].
__device__ __forceinline__ float group_sum8_transposed(const float (&v)[8], uint32_t lane) {
    float a[4], b[2];
    const bool u2 = (lane >> 2) & 1u, u1 = (lane >> 1) & 1u, u0 = lane & 1u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float send = u2 ? v[i] : v[i + 4], keep = u2 ? v[i + 4] : v[i];
        a[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float send = u1 ? a[i] : a[i + 2], keep = u1 ? a[i + 2] : a[i];
        b[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, 2);
    }
    const float send = u0 ? b[0] : b[1], keep = u0 ? b[1] : b[0];
    return keep + __shfl_xor_sync(0xFFFFFFFFu, send, 1);
}

// One tile of the adjoint (the whole CTA). Two barriers per round: after the
// walk (the blocks' sums are complete) and after the flush, which also stages
// the next round's entries in place of this one's.
template <uint32_t kBwdRound>
__device__ __forceinline__ void blend_backward_tile(const BlendBackwardArgs& a, uint32_t tile,
                                                    BlendBackwardSmem<kBwdRound>& SM) {
    if (!TPD_INBOUNDS(a.ctl, 44, tile, a.n_tiles)) return;  // (uniform)
    uint32_t vi, W, H, tx, ty;
    load_view_tile(a.views, a.tile_view, tile, vi, W, H, tx, ty);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const LanePixels P(tx, ty, warp, lane, W, H);
    const float ox = float(tx * kBlockX), oy = float(ty * kBlockY);
    const uint32_t K = min(a.ctl->total_keys, a.capacity);
    const uint32_t end = min(a.ranges[tile * 2 + 1], K), start = min(a.ranges[tile * 2 + 0], end);
    const Splat* vsplats = a.splats + size_t(vi) * a.n;

    const size_t img0 = a.image_offset ? a.image_offset[vi] : 0ull;
    float Tp[4], gp[3][4];
    uint32_t last[4], blk_last = 0;
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
        Tp[q] = 1.0f;
        gp[0][q] = gp[1][q] = gp[2][q] = 0.0f;
        last[q] = 0;
        if (P.in[q]) {
            const size_t p = img0 + size_t(P.y + q) * W + P.x;
            Tp[q] = a.final_T[p];
            last[q] = min(a.n_contrib[p], end - start);
#pragma unroll
            for (uint32_t c = 0; c < 3; ++c) gp[c][q] = a.dL_dimage[p * 3 + c];
        }
        blk_last = max(blk_last, last[q]);
    }
    float2 T[2], g0[2], g1[2], g2[2];
    bool huge = a.tile_len[tile] & kTileHuge;  // a colour or a gradient beyond kHuge, or not a number
#pragma unroll
    for (uint32_t c = 0; c < 3; ++c)
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) huge |= !(fabsf(gp[c][q]) <= kHuge);
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
        T[h] = f2(Tp[2 * h], Tp[2 * h + 1]);
        g0[h] = f2(gp[0][2 * h], gp[0][2 * h + 1]);
        g1[h] = f2(gp[1][2 * h], gp[1][2 * h + 1]);
        g2[h] = f2(gp[2][2 * h], gp[2][2 * h + 1]);
    }
    // a block takes the entries below the largest last-contributor index over
    // its pixels; the tile is walked back from the largest of all
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) blk_last = max(blk_last, __shfl_xor_sync(0xFFFFFFFFu, blk_last, o));
    uint32_t bl[4];
#pragma unroll
    for (uint32_t g = 0; g < 4; ++g) bl[g] = __shfl_sync(0xFFFFFFFFu, blk_last, 8 * g);
    if (lane == 0) SM.wmax[warp] = max(max(bl[0], bl[1]), max(bl[2], bl[3]));
    if (tid == 0) stage_block_empty(SM.e[kBwdRound]);
    const bool any_huge = __syncthreads_or(huge);
    const uint32_t max_last = max(SM.wmax[0], SM.wmax[1]);
    float* g2d_view = a.g2d + size_t(vi) * a.g2d_view_stride;

    // A round's entries, kPer per thread (with fewer entries than threads the
    // warps take turns): their indices loaded two rounds before they are
    // walked, their splats one, and staged after that round's walk, so both
    // latencies hide behind walks. Slot k of the
    // round whose list positions end at r_end holds position r_end - 1 - k.
    constexpr uint32_t kPer = kBwdRound > kAdjThreads ? kBwdRound / kAdjThreads : 1u;
    uint32_t pf_idx[kPer], nx_idx[kPer];  // of the round being loaded, and of the one after it
    float4 pf_c[kPer], pf_tex[kPer], pf_co[kPer];
    auto load_indices = [&](uint32_t r_end, uint32_t turn) {
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u) {
            const uint32_t k = (tid ^ turn) + u * kAdjThreads;
            nx_idx[u] = k < min(kBwdRound, r_end) ? a.vals[start + r_end - 1u - k] : 0xFFFFFFFFu;
        }
    };
    auto load_round = [&]() {
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u) {
            pf_idx[u] = nx_idx[u];
            if (pf_idx[u] < a.n) {
                const float4* p = reinterpret_cast<const float4*>(vsplats + pf_idx[u]);
                pf_c[u] = __ldg(p + 0);
                pf_tex[u] = __ldg(p + 1);
                pf_co[u] = __ldg(p + 2);
            }
        }
    };
    auto store_round = [&](uint32_t r_end, uint32_t turn) {
#pragma unroll
        for (uint32_t u = 0; u < kPer; ++u) {
            const uint32_t k = (tid ^ turn) + u * kAdjThreads;
            if (k < min(kBwdRound, r_end)) {
                if (pf_idx[u] < a.n) {
                    stage_block_values(pf_c[u], pf_tex[u], pf_co[u], ox, oy, SM.e[k], SM.mask[k]);
                } else {  // only reachable with corrupted lists
                    stage_block_empty(SM.e[k]);
                    SM.mask[k] = 0u;
                }
                SM.idx[k] = pf_idx[u];
            }
        }
    };
    const float2 one = f2(1.0f, 1.0f), mone = f2(-1.0f, -1.0f);
    const uint32_t block = 4u * warp + (lane >> 3), j = lane & 7u;
    auto walk_tile = [&](auto apart_tag) {
        constexpr bool kApart = decltype(apart_tag)::value;
        float2 nA[2], S[3][2];  // -A; walked apart: the colours behind, instead
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) nA[h] = S[0][h] = S[1][h] = S[2][h] = f2(0.f, 0.f);
        load_indices(max_last, 0u);
        load_round();
        load_indices(max_last > kBwdRound ? max_last - kBwdRound : 0u, 32u);
        store_round(max_last, 0u);
        __syncthreads();
        // the first entry of the round that a pixel counts (its last contributor; the round is back to front)
        int from[4];
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) from[q] = int(max_last - last[q]);
        uint32_t turn = 0;
        for (uint32_t r_end = max_last; r_end > 0;) {
            const uint32_t n = min(kBwdRound, r_end), next_end = r_end - n;
            turn ^= 32u;
            if (next_end) {
                load_round();
                load_indices(next_end > kBwdRound ? next_end - kBwdRound : 0u, turn ^ 32u);
            }
            const uint32_t steps = build_block_lists<kBwdRound>(SM.lists, warp, lane, n, [&](uint32_t e) {
                uint32_t m = uint32_t(SM.mask[e]) >> (4u * warp);
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g)
                    if (e + bl[g] < r_end) m &= ~(1u << g);  // behind the block's last contributor
                SM.met[warp][e] = uint8_t(m & 15u);
                return m;
            });
            const uint16_t* list = SM.lists.e[block];
            for (uint32_t i = 0; i < steps; ++i) {
                const uint32_t jj = list[i];
                const BlockStaged& E = SM.e[jj];
                const float4 sc = E.s, yb = E.yb, qco = E.qco, rg = E.rg;
                const float2 bb = E.b;
                const float dx = __fadd_rn(sc.x, P.nx), qadx = __fmul_rn(sc.y, dx);
                float2 dpow[2], w[2], dy[2];
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    // n2 for both pixels, as in the forward
                    dy[h] = __fadd2_rn(f2(yb.x, yb.y), h ? P.ny1 : P.ny0);
                    const float2 t = __ffma2_rn(f2(yb.z, yb.w), dy[h], f2(qadx, qadx));
                    const float2 qcdy = __fmul2_rn(f2(qco.x, qco.y), dy[h]);
                    const float2 n2 = __ffma2_rn(t, f2(dx, dx), __ffma2_rn(qcdy, dy[h], f2(0.0f, 0.0f)));
                    const bool ca = int(jj) >= from[2 * h] && __float_as_uint(n2.x) < __float_as_uint(sc.z);
                    const bool cb = int(jj) >= from[2 * h + 1] && __float_as_uint(n2.y) < __float_as_uint(sc.z);
                    const float2 raw = __fmul2_rn(f2(qco.z, qco.w), f2(ex2_approx(-n2.x), ex2_approx(-n2.y)));
                    const float2 alpha =
                        f2(ca ? fminf(kAlphaMax, raw.x) : 0.0f, cb ? fminf(kAlphaMax, raw.y) : 0.0f);
                    const float2 om = __ffma2_rn(mone, alpha, one);  // 1 - alpha >= 0.01
                    // in front of the entry (an approximate division takes a reciprocal as well, and
                    // scales around it: 1178 us for 8 views of 500,000, 1140 without)
                    const float2 inv = f2(rcp_approx(om.x), rcp_approx(om.y));
                    T[h] = __fmul2_rn(T[h], inv);
                    w[h] = __fmul2_rn(alpha, T[h]);
                    if constexpr (kApart) {
                        const float2 ninv = __fmul2_rn(inv, mone);
                        const float2 d0 = __ffma2_rn(f2(rg.x, rg.y), T[h], __fmul2_rn(S[0][h], ninv));
                        const float2 d1 = __ffma2_rn(f2(rg.z, rg.w), T[h], __fmul2_rn(S[1][h], ninv));
                        const float2 d2 = __ffma2_rn(bb, T[h], __fmul2_rn(S[2][h], ninv));
                        const float2 dA = __ffma2_rn(g2[h], d2, __ffma2_rn(g1[h], d1, __fmul2_rn(g0[h], d0)));
                        S[0][h] = __ffma2_rn(f2(rg.x, rg.y), w[h], S[0][h]);
                        S[1][h] = __ffma2_rn(f2(rg.z, rg.w), w[h], S[1][h]);
                        S[2][h] = __ffma2_rn(bb, w[h], S[2][h]);
                        const float2 dp = __fmul2_rn(alpha, dA);
                        dpow[h] = f2(ca && raw.x <= kAlphaMax ? dp.x : 0.0f, cb && raw.y <= kAlphaMax ? dp.y : 0.0f);
                        continue;
                    }
                    const float2 gc =
                        __ffma2_rn(g2[h], bb, __ffma2_rn(g1[h], f2(rg.z, rg.w), __fmul2_rn(g0[h], f2(rg.x, rg.y))));
                    const float2 ad = __fmul2_rn(alpha, __fadd2_rn(gc, nA[h]));  // alpha (g.c - A)
                    nA[h] = __ffma2_rn(mone, ad, nA[h]);
                    const float2 dp = __fmul2_rn(T[h], ad);  // alpha dL/dalpha = dL/dpower, unless alpha is clamped
                    dpow[h] = f2(raw.x <= kAlphaMax ? dp.x : 0.0f, raw.y <= kAlphaMax ? dp.y : 0.0f);
                }
                // w g over the lane's pixels (an infinite g times the zero weight
                // of a pair that does not count would be a NaN)
                auto weighted = [&](const float2 (&g)[2]) {
                    if constexpr (kApart) {
                        auto of = [](float gi, float wi) { return wi > 0.0f ? gi * wi : 0.0f; };
                        return (of(g[0].x, w[0].x) + of(g[0].y, w[0].y)) + (of(g[1].x, w[1].x) + of(g[1].y, w[1].y));
                    } else {
                        return hsum(__ffma2_rn(g[1], w[1], __fmul2_rn(g[0], w[0])));
                    }
                };
                const float2 s0 = __fmul2_rn(dpow[0], dy[0]), s1 = __fmul2_rn(dpow[1], dy[1]);
                const float p0 = hsum(__fadd2_rn(dpow[0], dpow[1])), py = hsum(__fadd2_rn(s0, s1));
                const float pyy = hsum(__ffma2_rn(s1, dy[1], __fmul2_rn(s0, dy[0])));
                const float px = p0 * dx;
                const float v[8] = {px, py, px * dx, py * dx, pyy, p0, weighted(g0), weighted(g1)};
                float v9 = weighted(g2);
                SM.sums[block][jj * 8u + j] = group_sum8_transposed(v, lane);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) v9 += __shfl_xor_sync(0xFFFFFFFFu, v9, o);
                if (j == 0) SM.sum9[block][jj] = v9;
            }
            __syncthreads();  // the round's sums are complete
            // warp 0: the record's first 16 bytes; warp 1: the other 20
            for (uint32_t k = lane; k < n; k += 32u) {
                const uint32_t met = uint32_t(SM.met[0][k]) | uint32_t(SM.met[1][k]) << 4;
                if (!met) continue;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                float v9 = 0.f;
#pragma unroll
                for (uint32_t b = 0; b < kBlendBlocks; ++b) {
                    if (!((met >> b) & 1u)) continue;
                    const float4 x = *reinterpret_cast<const float4*>(&SM.sums[b][k * 8u + 4u * warp]);
                    v = make_float4(v.x + x.x, v.y + x.y, v.z + x.z, v.w + x.w);
                    if (warp) v9 += SM.sum9[b][k];
                }
                const BlockStaged& E = SM.e[k];
                float* rec = g2d_view + size_t(SM.idx[k]) * kG2DStride;
                if (warp == 0) {
                    // d power / d(dx, dy) = -ln2 (2 qa dx + qb dy, 2 qc dy + qb dx)
                    const float qa = E.s.y, qb = E.yb.z, qc = E.qco.x;
                    v = make_float4(-kLn2 * (2.0f * qa * v.x + qb * v.y), -kLn2 * (2.0f * qc * v.y + qb * v.x), -0.5f * v.z,
                                    -v.w);
                } else {
                    v = make_float4(-0.5f * v.x, __fdividef(v.y, E.qco.z), v.z, v.w);  // alpha = opacity exp(power)
                    if (v9 != 0.0f) atomicAdd(rec + 8, v9);
                }
                if (v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f)
                    atomicAdd(reinterpret_cast<float4*>(rec) + warp, v);
            }
            __syncthreads();  // (the flush has read the entries that are staged over)
            if (next_end) store_round(next_end, turn);
            __syncthreads();
            r_end = next_end;
#pragma unroll
            for (uint32_t q = 0; q < 4; ++q) from[q] -= int(n);
        }
    };
    if (any_huge)
        walk_tile(std::true_type{});
    else
        walk_tile(std::false_type{});
}

// One CTA per tile, tile order[b] for CTA b; or (kPersistent) one CTA per
// resident slot taking the tiles from the queue in that order.
template <uint32_t kBwdRound, bool kPersistent>
__global__ void __launch_bounds__(kAdjThreads, bwd_min_blocks<kBwdRound>())
    blend_backward_kernel(BlendBackwardArgs a) {
    extern __shared__ __align__(16) unsigned char bwd_smem[];
    BlendBackwardSmem<kBwdRound>& SM = *reinterpret_cast<BlendBackwardSmem<kBwdRound>*>(bwd_smem);
    pdl_wait();  // launched as a dependent of the stream's previous kernel: its output is read below
    pdl_trigger();
    if (a.ctl->status & (kStatusFatal | kStatusKeyOverflow)) return;  // no valid frame to differentiate
    if constexpr (kPersistent) {
        uint32_t tile;
        while (next_tile(a.ctl, kTicketBlendBackward, a.tile_order, a.n_tiles, tile))
            blend_backward_tile<kBwdRound>(a, tile, SM);
    } else {
        blend_backward_tile<kBwdRound>(a, a.tile_order ? a.tile_order[blockIdx.x] : blockIdx.x, SM);
    }
}

// The blend's order: tiles by octave of their list length, each class in a
// bucket of its own that a CTA's 1024 tiles fill from a cursor, so one launch
// is enough.
constexpr uint32_t kOrderThreads = 256;
constexpr uint32_t kOrderTiles = 1024;

__global__ void __launch_bounds__(kOrderThreads)
    list_classes_kernel(const uint32_t* __restrict__ ranges, uint32_t n_tiles, FrameCtl* __restrict__ ctl,
                        uint32_t* __restrict__ buckets) {
    __shared__ uint32_t count[kListClasses], base[kListClasses];
    pdl_wait();     // launched as a dependent of the key sort's last pass: its ranges
    pdl_trigger();  // the blend may be scheduled; it waits for this grid
    const uint32_t tid = threadIdx.x;
    if (tid < kListClasses) count[tid] = 0;
    __syncthreads();
    constexpr uint32_t kPer = kOrderTiles / kOrderThreads;
    uint32_t cls[kPer], rank[kPer];
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        const uint32_t t = blockIdx.x * kOrderTiles + u * kOrderThreads + tid;
        cls[u] = rank[u] = 0;
        if (t < n_tiles) {
            const uint2 r = reinterpret_cast<const uint2*>(ranges)[t];
            const uint32_t len = r.y > r.x ? r.y - r.x : 0u;
            cls[u] = kListClasses - 1u - min(kListClasses - 1u, 32u - uint32_t(__clz(len)));
            rank[u] = atomicAdd(&count[cls[u]], 1u);
        }
    }
    __syncthreads();
    if (tid < kListClasses && count[tid]) base[tid] = atomicAdd(&ctl->list_class[tid], count[tid]);
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        const uint32_t t = blockIdx.x * kOrderTiles + u * kOrderThreads + tid;
        if (t < n_tiles) buckets[size_t(cls[u]) * n_tiles + base[cls[u]] + rank[u]] = t;
    }
}

// The tiles in class order, the classes counted by the blend: a CTA counts
// its 1024 tiles per class, takes that many places of each class at once, and
// its tiles fill them. (One CTA counting list lengths for all tiles took 182 us
// for the 259,000 tiles of 8 views of 2160p; and a list's length
// says little about a walk that stops early.)
__global__ void __launch_bounds__(kOrderThreads)
    tile_order_kernel(const uint32_t* __restrict__ tile_len, uint32_t n_tiles, FrameCtl* __restrict__ ctl,
                      uint32_t* __restrict__ order) {
    __shared__ uint32_t count[128], base[128], wsum[4];
    pdl_wait();  // launched as a dependent of the stream's previous kernel: its output is read below
    pdl_trigger();
    // a frame that blended nothing has left no walk lengths (the buffer may
    // never have been written, and a class past the last would be counted out
    // of range); the adjoint does nothing either
    if (ctl->status & (kStatusFatal | kStatusKeyOverflow)) return;  // (uniform)
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    if (tid < 128) count[tid] = 0;
    if (blockIdx.x == 0 && tid == 0) ctl->ticket[kTicketBlendBackward] = 0;  // the adjoint's tile queue starts again
    __syncthreads();
    constexpr uint32_t kPer = kOrderTiles / kOrderThreads;
    uint32_t cls[kPer], rank[kPer];
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        const uint32_t t = blockIdx.x * kOrderTiles + u * kOrderThreads + tid;
        cls[u] = t < n_tiles ? tile_class(tile_len[t] & ~kTileHuge) : 0u;
        rank[u] = t < n_tiles ? atomicAdd(&count[cls[u]], 1u) : 0u;
    }
    __syncthreads();
    uint32_t h = 0, incl = 0;
    if (tid < 128) {
        h = ctl->tile_hist[tid];
        incl = warp_inclusive_scan(h);
        if (lane == 31) wsum[warp] = incl;
    }
    __syncthreads();
    if (tid < 128) {
        uint32_t first = incl - h;
        for (uint32_t w = 0; w < warp; ++w) first += wsum[w];
        base[tid] = first + (count[tid] ? atomicAdd(&ctl->tile_cursor[tid], count[tid]) : 0u);
    }
    __syncthreads();
#pragma unroll
    for (uint32_t u = 0; u < kPer; ++u) {
        const uint32_t t = blockIdx.x * kOrderTiles + u * kOrderThreads + tid;
        const uint32_t pos = base[cls[u]] + rank[u];
        if (t < n_tiles && pos < n_tiles) order[pos] = t;
    }
    // the last CTA leaves the cursors at zero for the next order of this frame
    __shared__ bool last;
    if (tid == 0) {
        __threadfence();
        last = atomicAdd(&ctl->tile_order_done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    if (tid < 128) ctl->tile_cursor[tid] = 0;
    if (tid == 0) ctl->tile_order_done = 0;
}

}  // namespace

// Between one and five waves of CTAs (8 per SM). In one wave every tile starts
// at once; in many, the end of the launch is short beside it and the order's
// own launch (3 us) is lost: blend with and without the order, its launch
// included, 120,000 Gaussians at 801x603 60 and 71 us, 500,000 at 720p 90 and
// 99, at 1080p (8160 tiles) 144 and 150, but 1M spread evenly at 720p 147 and
// 145, at 1080p 254 and 250, 3M at 2160p 763 and 751.
bool blend_takes_list_order(uint32_t n_tiles, int num_sms) {
    const uint32_t wave = 8u * uint32_t(num_sms > 0 ? num_sms : 148);
    return n_tiles > wave && n_tiles <= 5u * wave;
}

void launch_list_classes(const uint32_t* ranges, uint32_t n_tiles, FrameCtl* ctl, uint32_t* buckets, cudaStream_t s) {
    if (n_tiles == 0) return;
    launch_dependent(list_classes_kernel, dim3((n_tiles + kOrderTiles - 1) / kOrderTiles), dim3(kOrderThreads), 0, s,
                     ranges, n_tiles, ctl, buckets);
}

void launch_tile_order(const uint32_t* tile_len, uint32_t n_tiles, FrameCtl* ctl, uint32_t* order, cudaStream_t s) {
    if (n_tiles == 0) return;
    launch_dependent(tile_order_kernel, dim3((n_tiles + kOrderTiles - 1) / kOrderTiles), dim3(kOrderThreads), 0, s,
                     tile_len, n_tiles, ctl, order);
}

namespace {

template <typename Kernel>
int resident_ctas(Kernel k, uint32_t threads, size_t smem) {
    int r = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k, int(threads), smem);
    return r > 0 ? r : 1;
}
template <uint32_t R, bool P, bool K>
int blend_occupancy() { return resident_ctas(blend_kernel<R, P, K>, kFwdThreads, 0); }
// the adjoint's shared-memory opt-in (a round of 128 takes above 48 KB) and its resident CTAs
template <uint32_t R, bool P>
int blend_backward_setup() {
    cudaFuncSetAttribute(blend_backward_kernel<R, P>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(sizeof(BlendBackwardSmem<R>)));
    return resident_ctas(blend_backward_kernel<R, P>, kAdjThreads, sizeof(BlendBackwardSmem<R>));
}

template <uint32_t R, bool P, bool K>
void launch_blend_k(const BlendArgs& a, int num_sms, cudaStream_t s) {
    const uint32_t grid =
        P ? std::min<uint32_t>(a.n_tiles, uint32_t(num_sms * device_once(blend_occupancy<R, P, K>))) : a.n_tiles;
    if (P)  // a persistent grid is placed once: on SMs the key sort has left, not while its last CTAs run
        blend_kernel<R, P, K><<<grid, kFwdThreads, 0, s>>>(a);
    else
        launch_dependent(blend_kernel<R, P, K>, dim3(grid), dim3(kFwdThreads), 0, s, a);
}

// with the adjoint's inputs (final T, last contributor) when both buffers are given
template <uint32_t R, bool P>
void launch_blend_t(const BlendArgs& a, int num_sms, cudaStream_t s) {
    if (a.final_T && a.n_contrib)
        launch_blend_k<R, P, true>(a, num_sms, s);
    else
        launch_blend_k<R, P, false>(a, num_sms, s);
}

template <uint32_t R, bool P>
void launch_blend_backward_t(const BlendBackwardArgs& a, int num_sms, cudaStream_t s) {
    const int resident = device_once(blend_backward_setup<R, P>);
    const uint32_t grid = P ? std::min<uint32_t>(a.n_tiles, uint32_t(num_sms * resident)) : a.n_tiles;
    launch_dependent(blend_backward_kernel<R, P>, dim3(grid), dim3(kAdjThreads), sizeof(BlendBackwardSmem<R>), s, a);
}

}  // namespace

void launch_blend(const BlendArgs& a, const BlendLaunch& l, cudaStream_t s) {
    if (a.n_tiles == 0) return;
    const int sms = l.num_sms > 0 ? l.num_sms : 148;
    switch (l.round) {
        case 64: l.persistent ? launch_blend_t<64, true>(a, sms, s) : launch_blend_t<64, false>(a, sms, s); break;
        case 256: l.persistent ? launch_blend_t<256, true>(a, sms, s) : launch_blend_t<256, false>(a, sms, s); break;
        default: l.persistent ? launch_blend_t<128, true>(a, sms, s) : launch_blend_t<128, false>(a, sms, s); break;
    }
}

void launch_pack_rgba8(const float* rgb, uint32_t* rgba, size_t pixels, cudaStream_t s) {
    if (pixels == 0) return;
    launch_dependent(pack_rgba8_kernel, dim3(unsigned((pixels + 255) / 256)), dim3(256), 0, s,
                     static_cast<const float*>(rgb), rgba, pixels);
}

void launch_blend_backward(const BlendBackwardArgs& a, const BlendLaunch& l, cudaStream_t s) {
    if (a.n_tiles == 0) return;
    const int sms = l.num_sms > 0 ? l.num_sms : 148;
    switch (l.backward_round) {
        case 32:
            l.persistent ? launch_blend_backward_t<32, true>(a, sms, s) : launch_blend_backward_t<32, false>(a, sms, s);
            break;
        case 128:
            l.persistent ? launch_blend_backward_t<128, true>(a, sms, s)
                         : launch_blend_backward_t<128, false>(a, sms, s);
            break;
        default:
            l.persistent ? launch_blend_backward_t<64, true>(a, sms, s) : launch_blend_backward_t<64, false>(a, sms, s);
            break;
    }
}

}  // namespace tpd
