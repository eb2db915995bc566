// keygen.cu — kernel (b): the tile-count scan over the Gaussians in depth
// order, and key duplication over the keys it counts.
//
// Reference: prefix.slang:40-158 (the scan of the per-Gaussian tile counts)
// and keygen.slang:23-53 (one thread per Gaussian looping over its tile
// rect). It also presets the tile ranges (fillBuffer, GaussianEngine.cpp:843-848)
// that the key sort's last pass fills in (range.slang:18-35, in sort.cu), and
// counts the key sort's first-pass digits per 4096-key partition.
//
// Gaussians are visited in depth order (a prior sort of the (view | depth)
// keys), so the emitted keys only need a stable sort on their tile-id bits
// afterwards: per tile the order is (depth, index), exactly the reference's
// stable sort of (tile | depth) keys emitted in index order. Keys and values
// are bit-identical to the reference's.
//
// Two kernels, split by what they balance. scan_items_kernel goes over items
// (Gaussians in depth order) and stores each item's first key slot and tile
// rectangle. expand_keys_kernel goes over key slots, one CTA per 4096 of them
// (a partition of the key sort), and finds each slot's item. Splitting by
// slots matters because depth order puts the nearest Gaussians, with the
// largest rectangles, side by side: one kernel over 512-item partitions gave
// the first CTA up to a million keys to write while the others were done
// (1M Gaussians at 1080p from the edge of the cloud: 303 us, now 20 + 35;
// 3M at 2160p: 1189 us, now 74 + 242; 10,000 at 256x256: 11 us with the scan of
// the counts, now 6 + 5). In a large single view expand_strips_kernel takes the
// second one's place and writes column strips, a few per item, for the key sort
// to expand (sort.cu): 20 + 20 and 77 + 67 us for the first two.
#include <algorithm>
#include <type_traits>

#include "tpd_common.cuh"
#include "tpd_counted.cuh"
#include "tpd_kernels.h"
#include "tpd_scan.cuh"
#include "tpd_slots.cuh"

namespace tpd {
namespace {

constexpr uint32_t kScanItemsThreads = 256;
constexpr uint32_t kScanItemsChunks = kKeygenPart / kScanItemsThreads;  // items per thread
constexpr uint32_t kScanItemsWarps = kScanItemsThreads / 32;
static_assert(kScanItemsChunks * kScanItemsThreads == kKeygenPart, "a partition is whole chunks of every warp");

// An item's tile rectangle: its first tile (t0, row-major in its view), its
// width and the view's grid width (wgx = w | gx << 16), its key count (w h)
// and Gaussian index.
struct ItemRect {
    uint32_t t0, wgx, cnt, gi;
};

// For the strips of an item: its rectangle's first column, first row and height
// packed as a strip's key (strip_key), and its width (its strips).
struct ItemStrips {
    uint32_t key, w;
};

__device__ __forceinline__ ItemRect item_rect(uint32_t item, bool valid, float4 texel, uint32_t n_items, uint32_t n,
                                              const ViewConst* __restrict__ views, FrameCtl* ctl, ItemStrips& strips) {
    strips = ItemStrips{0u, 0u};
    uint32_t w = 1, h = 0, gx = 1, gi = 0, t0 = 0;
    if (valid && TPD_INBOUNDS(ctl, 21, item, n_items)) {
        const uint32_t v = n_items == n ? 0u : item / n;  // one view: no division
        gi = item - v * n;
        const ViewConst& vc = views[v];
        gx = grid_x(vc.width);
        if (texel.w > 0.0f) {
            uint32_t x0, y0, x1, y1;
            bounding_rect(texel.x, texel.y, texel.w, gx, grid_y(vc.height), x0, y0, x1, y1);
            if (x1 > x0 && y1 > y0) {
                w = x1 - x0;
                h = y1 - y0;
                t0 = vc.tile_base + y0 * gx + x0;
                strips = ItemStrips{strip_key(x0, y0, h), w};
            }
        }
    }
    return ItemRect{t0, w | (gx << 16), w * h, gi};
}

// The depth-order tile-count scan. Persistent CTAs take partitions of
// kKeygenPart consecutive items in depth order by an atomic ticket; warp w of
// a CTA owns the partition's items [w 32 kScanItemsChunks, ...), in chunks of
// 32 (one item per lane). Per partition:
//  1. each lane gathers its items' splat texels and works out their tile
//     rectangles, so their key counts;
//  2. the counts are scanned across the warp, then across the CTA;
//  3. one warp resolves the partition's exclusive prefix with the bounded
//     decoupled look-back (prefix.slang:100-114 as restated in tpd_scan.cuh):
//     the last partition's inclusive prefix is the frame's key count K. A
//     prefix has 32 bits, so a frame of 2^31 keys or more is flagged where they
//     are passed: the first partition to end past them has an exact exclusive
//     prefix (whatever those after it come round to);
//  4. each lane stores its items' key offsets (the scan's output), for
//     expand_keys_kernel their rectangles, offsets and Gaussians (16 bytes an
//     item), and, for every multiple of 4096 among an item's slots, the item's
//     position in part_first.
// A CTA takes a ticket only when it starts on the partition, so every
// partition a look-back waits on is being worked on by a running CTA and
// publishes its aggregate soon. Bound by the gathers (32 bytes of every
// 48-byte splat in depth order) and the look-back's latency.
struct ScanItemsSmem {
    uint32_t wtot[2][kScanItemsWarps];  // key counts of the warps' items; strip counts
    uint32_t ticket;                    // the partition being worked on
    uint32_t excl[2];                   // the partition's exclusive prefixes
};

// kStrips: the items' strips (one per column of the rectangle) are scanned as
// well, by a second look-back beside the first, and item_info and part_first
// are those of the strip slots. (Registers for six CTAs per SM, as without,
// with 12 bytes spilled: 48 -> 45 us with the expansion, 1M Gaussians at 1080p.)
template <bool kStrips>
__global__ void __launch_bounds__(kScanItemsThreads, 6)
    scan_items_kernel(const Splat* __restrict__ splats, const uint32_t* __restrict__ items,
                      const uint32_t* __restrict__ items_other, uint32_t n_items, uint32_t n,
                      const ViewConst* __restrict__ views, uint32_t* __restrict__ offsets,
                      uint4* __restrict__ item_info, uint32_t* __restrict__ part_first, uint32_t capacity,
                      uint32_t* __restrict__ ranges, uint32_t n_tiles, uint64_t* desc, uint64_t* strip_desc,
                      FrameCtl* ctl, uint32_t spin_limit, uint32_t never_publish) {
    constexpr uint32_t kSums = kStrips ? 2u : 1u;
    __shared__ ScanItemsSmem S;
    pdl_wait();     // launched as a dependent of the depth sort's last pass: its order is read below
    pdl_trigger();  // expand_keys_kernel may be scheduled (it waits for this grid)
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
    const uint32_t count = min(ctl->depth_count, n_items);
    if (ctl->depth_skips & 1u) items = items_other;  // a skipped depth pass left the order there
    // ranges: (0xFFFFFFFF, 0) until the key sort's last pass narrows them
    for (uint32_t t = blockIdx.x * blockDim.x + tid; t < n_tiles; t += gridDim.x * blockDim.x)
        reinterpret_cast<uint2*>(ranges)[t] = make_uint2(0xFFFFFFFFu, 0u);
    const uint32_t nparts = (count + kKeygenPart - 1) / kKeygenPart;
    const uint32_t tag = ctl->tag * 32u + kTagScan;
    for (;;) {
        // one thread reads the status for the whole CTA (a look-back of this
        // grid may raise a fatal bit meanwhile, and every thread must take the
        // same way through the barriers): a fatal status ends the CTA as a
        // ticket past the last partition does
        if (tid == 0)
            S.ticket = (ctl->status & kStatusFatal) ? 0xFFFFFFFFu : atomicAdd(&ctl->ticket[kTicketScan], 1u);
        __syncthreads();
        const uint32_t part = S.ticket;
        if (part >= nparts) break;  // (uniform)
        const uint32_t r0 = part * kKeygenPart + warp * (kScanItemsChunks * 32u) + lane;
        uint32_t item[kScanItemsChunks];
        float4 texel[kScanItemsChunks];
#pragma unroll
        for (uint32_t c = 0; c < kScanItemsChunks; ++c)
            item[c] = r0 + 32u * c < count ? items[r0 + 32u * c] : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t c = 0; c < kScanItemsChunks; ++c)
            texel[c] = item[c] < n_items ? reinterpret_cast<const float4*>(splats + item[c])[1]
                                         : make_float4(0.f, 0.f, 0.f, 0.f);
        ItemRect rect[kScanItemsChunks];
        ItemStrips strips[kScanItemsChunks];
        // [0]: keys, [1]: strips
        uint32_t incl[kSums][kScanItemsChunks], ctot[kSums][kScanItemsChunks], wtotal[kSums] = {}, vis = 0;
#pragma unroll
        for (uint32_t c = 0; c < kScanItemsChunks; ++c) {
            rect[c] = item_rect(item[c], r0 + 32u * c < count, texel[c], n_items, n, views, ctl, strips[c]);
#pragma unroll
            for (uint32_t u = 0; u < kSums; ++u) {
                incl[u][c] = warp_inclusive_scan(u ? strips[c].w : rect[c].cnt);
                ctot[u][c] = __shfl_sync(0xFFFFFFFFu, incl[u][c], 31);
                wtotal[u] += ctot[u][c];
            }
            vis += rect[c].cnt ? 1u : 0u;
        }
        vis = warp_sum(vis);
        if (lane == 0) {
#pragma unroll
            for (uint32_t u = 0; u < kSums; ++u) S.wtot[u][warp] = wtotal[u];
            if (vis) atomicAdd(&ctl->visible, vis);
        }
        __syncthreads();
        uint32_t wbase[kSums] = {}, total[kSums] = {};
#pragma unroll
        for (uint32_t u = 0; u < kSums; ++u)
#pragma unroll
            for (uint32_t w = 0; w < kScanItemsWarps; ++w) {
                const uint32_t sw = S.wtot[u][w];
                wbase[u] += w < warp ? sw : 0u;
                total[u] += sw;
            }
        if (warp < kSums) {
            const bool keys = warp == 0;
            const uint32_t sum = keys ? total[0] : total[kSums - 1u];
            const uint32_t ex = warp_lookback(keys ? desc : strip_desc, part, sum, tag, &ctl->status, spin_limit,
                                              never_publish != 0);
            if (lane == 0) {
                S.excl[warp] = ex;
                uint64_t end = ex;  // (a warp's count is at most 2^31: 128 items of 2^24 tiles)
#pragma unroll
                for (uint32_t w = 0; w < kScanItemsWarps; ++w) end += S.wtot[0][w];
                if (keys && end > 0x7FFFFFFFull) {
                    atomicMax(&ctl->total_keys, 0xFFFFFFFFu);
                    atomicOr(&ctl->status, kStatusKeyOverflow);
                }
                if (part == nparts - 1u) {
                    atomicMax(keys ? &ctl->total_keys : &ctl->total_strips, ex + sum);  // (0 at the frame's start)
                    if (keys && ex + sum > capacity) atomicOr(&ctl->status, kStatusKeyOverflow);
                }
            }
        }
        __syncthreads();
        uint32_t base[kSums];
#pragma unroll
        for (uint32_t u = 0; u < kSums; ++u) base[u] = S.excl[u] + wbase[u];
#pragma unroll
        for (uint32_t c = 0; c < kScanItemsChunks; ++c) {
            const uint32_t r = r0 + 32u * c, first_key = base[0] + incl[0][c] - rect[c].cnt;
            const uint32_t slots = kStrips ? strips[c].w : rect[c].cnt;
            const uint32_t first = kStrips ? base[kSums - 1u] + incl[kSums - 1u][c] - slots : first_key;
            if (r < count) {
                offsets[r] = first_key;
                item_info[r] = kStrips ? make_uint4(strips[c].key, 0u, first, rect[c].gi)
                                       : make_uint4(rect[c].t0, rect[c].wgx, first, rect[c].gi);
                // (slots past the capacity are not written: the frame is flagged)
                const uint32_t end = min(first + slots, capacity);
                for (uint32_t p = (first + kCountedTile - 1) / kCountedTile; p * kCountedTile < end; ++p)
                    part_first[p] = r;
            }
#pragma unroll
            for (uint32_t u = 0; u < kSums; ++u) base[u] += ctot[u][c];
        }
        __syncthreads();  // S is rewritten for the next partition
    }
}

// Key duplication by key slots: one CTA per 4096 slots, 16 per thread.
//  1. The partition's items are part_first[part] up to the one holding the
//     next partition's first slot; each marks its first slot in an owner map
//     in shared memory, and a prefix maximum over the map gives every slot its
//     item.
//  2. A thread takes four consecutive slots at a time, so that keys and values
//     are stored 16 bytes at once. The first slot's (row, column) in its item's
//     rectangle takes a division; the next slot is the next column or row of
//     the same item, or the first of the next item.
// A key is stored as its tile id alone: the low 32 bits of the reference's
// key are the depth, already in order, and the depth of a key is that of its
// value's splat, so the sort needs only the tile ids and the full keys can be
// rebuilt from (tile, value) when read.
// work != nullptr: the partition's low tile-id digits are counted as they are
// written and finished into the global digit offsets of the key sort's first
// pass (counted_finish), which then needs no counting kernel. work == nullptr
// (look-back passes): every digit of the tile ids is added to ctl->sort_hist.
// Bound by latency and issue; the stores are 8 bytes a key. With one key per
// thread and step (35 instructions a key, two dependent loads) 1M Gaussians at
// 1080p took 67 us with the scan, 8 views of 500,000 at 720p 216; now 55 and
// 162, with 64 registers for four CTAs per SM, which spill 8 to 16 bytes (71
// registers, three CTAs: 59 and 171; five: 57 and 164).
constexpr uint32_t kExpandThreads = 256;
constexpr uint32_t kExpandSlots = kCountedTile / kExpandThreads;
constexpr uint32_t kTileDigitsMax = 4;

// kDig: digits of the counted first pass (256 or 512), 0 for the look-back form.
template <uint32_t kDig>
__global__ void __launch_bounds__(kExpandThreads, 4)
    expand_keys_kernel(const uint4* __restrict__ item_info, const uint32_t* __restrict__ part_first,
                       uint32_t* __restrict__ tiles, uint32_t* __restrict__ vals, uint32_t n_items,
                       uint32_t capacity, uint32_t max_parts, uint32_t tile_bits, uint32_t* __restrict__ work, FrameCtl* ctl) {
    __shared__ __align__(16) uint16_t owner[kCountedTile];  // item of each slot, from the partition's first
    constexpr bool kCounted = kDig != 0;
    constexpr uint32_t kRows = kCounted ? 1u : kTileDigitsMax, kWidth = kCounted ? kDig : 256u;
    __shared__ uint32_t digits[kRows][kWidth];
    __shared__ uint32_t wsum[kExpandThreads / 32];
    __shared__ bool s_last;
    pdl_wait();
    pdl_trigger();
    const uint32_t tid = threadIdx.x;
    const uint32_t K = (ctl->status & (kStatusFatal | kStatusKeyOverflow)) ? 0u : min(ctl->total_keys, capacity);
    const uint32_t nparts = min((K + kCountedTile - 1) / kCountedTile, max_parts);
    const uint32_t part = blockIdx.x;
    if (part >= nparts) return;  // (uniform)
    const uint32_t base = part * kCountedTile, cnt = min(kCountedTile, K - base);
    const uint32_t n_all = min(ctl->depth_count, n_items);
    const uint32_t first = min(part_first[part], n_all - 1u);
    const uint32_t last = part + 1u < nparts ? min(part_first[part + 1u], n_all - 1u) : n_all - 1u;
    // an item has at least one key: a partition holds at most kCountedTile items
    const uint32_t m = min(last - first + 1u, kCountedTile + 1u);
#pragma unroll
    for (uint32_t p = 0; p < kRows * kWidth / kExpandThreads; ++p) (&digits[0][0])[p * kExpandThreads + tid] = 0;
    slot_owners(owner, m, cnt, wsum, [&](uint32_t k) { return item_info[first + k].z - base; });
    const uint32_t ndig = kCounted ? 1u : min(kTileDigitsMax, (tile_bits + 7u) / 8u);
    // kFull: a whole partition (all but the last), without per-slot checks
    auto expand = [&](auto full_tag) {
        constexpr bool kFull = decltype(full_tag)::value;
#pragma unroll
        for (uint32_t q = 0; q < kExpandSlots / 4u; ++q) {
            const uint32_t slot = q * (4u * kExpandThreads) + 4u * tid;
            if (!kFull && slot >= cnt) break;
            const uint2 own = *reinterpret_cast<const uint2*>(owner + slot);  // four 16-bit owners
            const uint32_t o[4] = {own.x & 0xFFFFu, own.x >> 16, own.y & 0xFFFFu, own.y >> 16};
            uint4 info[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) info[u] = __ldg(item_info + first + o[u]);
            uint32_t w = info[0].y & 0xFFFFu;
            const uint32_t local = base + slot - info[0].z;  // < 2^24: exact in a float
            // row = local / w from a float quotient, corrected by one step
            uint32_t ty = __float2uint_rz(__fdividef(float(local), float(w)));
            int32_t col = int32_t(local) - int32_t(ty * w);
            if (col < 0) {
                --ty;
                col += int32_t(w);
            } else if (col >= int32_t(w)) {
                ++ty;
                col -= int32_t(w);
            }
            uint32_t t[4], x = uint32_t(col);
            t[0] = info[0].x + ty * (info[0].y >> 16) + x;
#pragma unroll
            for (uint32_t u = 1; u < 4; ++u) {
                const bool next_item = o[u] != o[u - 1], next_row = x + 1u == w;
                const uint32_t step = next_row ? (info[u].y >> 16) - w + 1u : 1u;
                t[u] = next_item ? info[u].x : t[u - 1] + step;
                x = next_item || next_row ? 0u : x + 1u;
                w = info[u].y & 0xFFFFu;
            }
            if (kFull || slot + 4u <= cnt) {
                *reinterpret_cast<uint4*>(tiles + base + slot) = make_uint4(t[0], t[1], t[2], t[3]);
                *reinterpret_cast<uint4*>(vals + base + slot) = make_uint4(info[0].w, info[1].w, info[2].w, info[3].w);
            } else {
#pragma unroll
                for (uint32_t u = 0; u < 4; ++u)
                    if (slot + u < cnt) {
                        tiles[base + slot + u] = t[u];
                        vals[base + slot + u] = info[u].w;
                    }
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (!kFull && slot + u >= cnt) continue;
#pragma unroll
                for (uint32_t p = 0; p < kRows; ++p)
                    if (p < ndig) atomicAdd(&digits[p][(t[u] >> (8u * p)) & (kWidth - 1u)], 1u);
            }
        }
    };
    if (cnt == kCountedTile)
        expand(std::true_type{});
    else
        expand(std::false_type{});
    __syncthreads();
    if constexpr (kCounted) {
        constexpr uint32_t kPer = kWidth / kExpandThreads;
        RowDigits<kPer> count;
#pragma unroll
        for (uint32_t p = 0; p < kPer; ++p) count.v[p] = digits[0][kPer * tid + p];
        counted_finish<kWidth>(CountedWork<kWidth>(work, max_parts), nparts, part, count, wsum, s_last);
    } else {
        for (uint32_t p = 0; p < ndig; ++p)
            if (digits[p][tid]) atomicAdd(&ctl->sort_hist[p][tid], digits[p][tid]);
    }
}

// The strips' form (see sort.cu): a slot is a strip, one column of its item's
// rectangle. Its key is that column with the rectangle's rows (strip_key), its
// value the Gaussian. Counted per partition and column: the strips and, as
// digits 256 and up, their heights (the keys they hold). Bound by latency, as
// the keys' form: 3M Gaussians at 2160p 67 us (242 for the keys), 1M at 1080p
// 20 (35).
__global__ void __launch_bounds__(kExpandThreads, 4)
    expand_strips_kernel(const uint4* __restrict__ item_info, const uint32_t* __restrict__ part_first,
                         uint32_t* __restrict__ strips, uint32_t* __restrict__ vals, uint32_t n_items,
                         uint32_t capacity, uint32_t max_parts, uint32_t* __restrict__ work, FrameCtl* ctl) {
    __shared__ __align__(16) uint16_t owner[kCountedTile];  // item of each slot, from the partition's first
    __shared__ __align__(8) uint32_t sums[512];              // strips by column, heights by column
    __shared__ uint32_t wsum[kExpandThreads / 32];
    __shared__ bool s_last;
    pdl_wait();
    pdl_trigger();
    const uint32_t tid = threadIdx.x;
    const uint32_t K = (ctl->status & (kStatusFatal | kStatusKeyOverflow)) ? 0u : min(ctl->total_strips, capacity);
    const uint32_t nparts = min((K + kCountedTile - 1) / kCountedTile, max_parts);
    const uint32_t part = blockIdx.x;
    if (part >= nparts) return;  // (uniform)
    const uint32_t base = part * kCountedTile, cnt = min(kCountedTile, K - base);
    const uint32_t n_all = min(ctl->depth_count, n_items);
    const uint32_t first = min(part_first[part], n_all - 1u);
    const uint32_t last = part + 1u < nparts ? min(part_first[part + 1u], n_all - 1u) : n_all - 1u;
    const uint32_t m = min(last - first + 1u, kCountedTile + 1u);
    sums[tid] = sums[tid + 256u] = 0u;
    slot_owners(owner, m, cnt, wsum, [&](uint32_t k) { return item_info[first + k].z - base; });
#pragma unroll
    for (uint32_t q = 0; q < kExpandSlots / 4u; ++q) {
        const uint32_t slot = q * (4u * kExpandThreads) + 4u * tid;
        if (slot >= cnt) break;
        const uint2 own = *reinterpret_cast<const uint2*>(owner + slot);  // four 16-bit owners
        const uint32_t o[4] = {own.x & 0xFFFFu, own.x >> 16, own.y & 0xFFFFu, own.y >> 16};
        uint32_t key[4], gi[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint4 info = __ldg(item_info + first + o[u]);
            key[u] = info.x + (base + slot + u - info.z);  // (the columns stay below 256)
            gi[u] = info.w;
        }
        if (slot + 4u <= cnt) {
            *reinterpret_cast<uint4*>(strips + base + slot) = make_uint4(key[0], key[1], key[2], key[3]);
            *reinterpret_cast<uint4*>(vals + base + slot) = make_uint4(gi[0], gi[1], gi[2], gi[3]);
        } else {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                if (slot + u < cnt) {
                    strips[base + slot + u] = key[u];
                    vals[base + slot + u] = gi[u];
                }
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)
            if (slot + u < cnt) {
                atomicAdd(&sums[strip_col(key[u])], 1u);
                atomicAdd(&sums[256u + strip_col(key[u])], strip_height(key[u]));
            }
    }
    __syncthreads();
    RowDigits<2> count;
    const uint2 c = reinterpret_cast<const uint2*>(sums)[tid];
    count.v[0] = c.x;
    count.v[1] = c.y;
    counted_finish<512>(CountedWork<512>(work, max_parts), nparts, part, count, wsum, s_last);
}

int scan_items_setup() {
    int r = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, scan_items_kernel<false>, kScanItemsThreads, 0);
    return r > 0 ? r : 1;
}

}  // namespace

void launch_keygen(const KeygenArgs& a, int num_sms, cudaStream_t s) {
    if (a.n_items == 0 || a.n == 0) return;
    const uint64_t parts = (uint64_t(a.n_items) + kKeygenPart - 1) / kKeygenPart;
    const int per_sm = device_once(scan_items_setup);  // resident CTAs per SM
    const uint64_t cap = uint64_t(num_sms > 0 ? num_sms : 148) * uint64_t(per_sm);  // persistent
    const uint64_t blocks = parts < cap ? parts : cap;
    launch_dependent(a.strips ? scan_items_kernel<true> : scan_items_kernel<false>, dim3(unsigned(blocks)),
                     dim3(kScanItemsThreads), 0, s, a.splats, a.items, a.items_other, a.n_items, a.n, a.views,
                     a.offsets, a.item_info, a.part_first, a.capacity, a.ranges, a.n_tiles, a.desc, a.strip_desc,
                     a.ctl, a.spin_limit, a.never_publish);
    const uint32_t max_parts = std::max(1u, uint32_t((uint64_t(a.capacity) + kCountedTile - 1) / kCountedTile));
    if (a.strips) {
        launch_dependent(expand_strips_kernel, dim3(max_parts), dim3(kExpandThreads), 0, s,
                         static_cast<const uint4*>(a.item_info), static_cast<const uint32_t*>(a.part_first), a.tiles,
                         a.vals, a.n_items, a.capacity, max_parts, a.counted_work, a.ctl);
        return;
    }
    const auto expand = !a.counted_work                                ? expand_keys_kernel<0>
                        : counted_digit_bits(a.tile_bits) > 8 ? expand_keys_kernel<512>
                                                              : expand_keys_kernel<256>;
    launch_dependent(expand, dim3(max_parts), dim3(kExpandThreads), 0, s, static_cast<const uint4*>(a.item_info),
                     static_cast<const uint32_t*>(a.part_first), a.tiles, a.vals, a.n_items, a.capacity, max_parts,
                     a.tile_bits, a.counted_work, a.ctl);
}

namespace {

// One CTA per tile: the tile's range of values, with the tile and each value's
// depth. (A tile without keys has the range (0, 0) or (0xFFFFFFFF, 0).)
__global__ void materialize_keys_kernel(const uint32_t* __restrict__ ranges, const uint32_t* __restrict__ vals,
                                        const Splat* __restrict__ splats, uint32_t n,
                                        const uint32_t* __restrict__ tile_view, uint32_t capacity,
                                        const FrameCtl* __restrict__ ctl, uint64_t* __restrict__ keys) {
    const uint32_t t = blockIdx.x, v = tile_view ? tile_view[t] : 0u;
    const uint32_t K = min(ctl->total_keys, capacity), end = min(ranges[2 * t + 1], K);
    for (uint32_t i = ranges[2 * t] + threadIdx.x; i < end; i += blockDim.x) {
        const uint32_t g = vals[i];
        const uint32_t depth = g < n ? __float_as_uint(reinterpret_cast<const float4*>(splats + size_t(v) * n + g)[1].z)
                                     : 0xFFFFFFFFu;
        keys[i] = (uint64_t(t) << 32) | depth;
    }
}

}  // namespace

void launch_materialize_keys(const uint32_t* ranges, uint32_t n_tiles, const uint32_t* vals, const Splat* splats,
                             uint32_t n, const uint32_t* tile_view, uint32_t capacity, const FrameCtl* ctl,
                             uint64_t* keys, cudaStream_t s) {
    if (capacity == 0 || n_tiles == 0) return;
    materialize_keys_kernel<<<n_tiles, 128, 0, s>>>(ranges, vals, splats, n, tile_view, capacity, ctl, keys);
}

}  // namespace tpd
