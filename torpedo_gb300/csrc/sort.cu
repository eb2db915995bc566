// sort.cu — kernel (c): stable LSD radix sort of (u64 or u32 key, u32 value) pairs.
//
// Reference: the 4-way (2-bit digit) LSD sort of radix-shuffle.slang:39-151,
// radix-prefixA.slang:39-170, radix-prefixB.slang:39-169 and
// radix-mapping.slang:40-117, driven by GaussianEngine.cpp:820-841 with
// P = ceil((msb(tiles) + 32) / 2) passes (GaussianEngine.cpp:351-357): four
// dispatches per pass, 21-24 passes per frame.
//
// GB300 form (onesweep): 8-bit digits, so a 45-bit (tile | depth) key takes 6
// passes instead of 23.
//  1. In the frame the digit histograms come from earlier kernels (the
//     preprocess counts the depth keys' digits, key duplication those of the
//     tile ids for look-back passes); sort_histogram_kernel builds them for
//     standalone sorts (one read of the keys).
//  2. onesweep_kernel, once per pass: a persistent CTA takes 4096-key
//     partitions by atomic ticket, loads them with coalesced warp-striped
//     loads, ranks keys per warp (shared atomics where the digits are spread,
//     else bit ballots, or match-any in the 512-thread variant; stable within
//     the warp-striped order), combines warps per digit, publishes its digit counts, reorders the partition in shared
//     memory while predecessors publish, resolves each digit's global prefix
//     by a decoupled look-back (one thread per digit, four predecessors per
//     round trip, bounded spin) and writes digit runs out coalesced.
//  3. Counted passes (the frame's key sort, below): a counting kernel, then a
//     scatter kernel per pass, with every partition's digit offsets known
//     before it scatters, so no partition waits on another.
// In the frame the depth presort sorts 64-bit (view | depth) keys with
// onesweep passes and the key sort 32-bit tile ids (their depth order is
// already fixed) with counted passes; the standalone sort takes 64-bit keys
// (onesweep, 256 threads x 4, 8 or 16 keys by their number). Both 64-bit sorts
// are one counting launch up to 12288 pairs (sort_small.cu).
// The result is the stable sort of the pairs by the low key_bits bits, the
// same permutation as the reference's sort.
#include <algorithm>
#include <type_traits>

#include "tpd_common.cuh"
#include "tpd_counted.cuh"
#include "tpd_kernels.h"
#include "tpd_scan.cuh"
#include "tpd_slots.cuh"

namespace tpd {
namespace {

constexpr uint32_t kRadixBits = 8;
constexpr uint32_t kRadix = 1u << kRadixBits;
constexpr uint32_t kSortThreads = 256;
// Keys per thread of a radix pass: 16 (4096-key partitions) for large sorts;
// 8 or 4 give more, shorter partitions when the sort is too small to fill the
// GPU with 4096-key partitions (sort_items_for).
constexpr uint32_t kSortItemsMax = 16;
constexpr uint32_t kInvalidDigit = kRadix;                  // keys past K (and dropped keys)

// Pass kinds of onesweep_kernel. The depth sort compacts the culled items
// away in its first pass and sorts the remaining ctl->depth_count items in
// the others, where a pass whose digit is the same for every key is skipped
// (counted in ctl->depth_skips; the later passes swap their buffers).
constexpr int kPassPlain = 0;      // K = fixed_count, else ctl->total_keys
constexpr int kPassDropCulled = 1; // as plain; keys whose low 32 bits are 0xFFFFFFFF are not written
constexpr int kPassCompacted = 2;  // K = ctl->depth_count; a uniform digit skips the pass (ctl->depth_skips)

constexpr uint32_t kHistThreads = 256;
constexpr uint32_t kHistChunk = 2048;  // keys per grid-stride chunk of the histogram kernel (256 threads x 8)

// Reorder buffers hold one pad slot per 16 keys: digit runs of about 16 keys
// (8-bit digits over a 4096-key partition) put the runs of consecutive digits
// 128 B apart, which without padding lands a warp's stores on one bank when
// its lanes carry consecutive digits (keys of one Gaussian's tile rectangle).
__device__ __forceinline__ uint32_t pad16(uint32_t i) { return i + (i >> 4); }

template <int kItems, int kThreads, typename KeyT>
struct OnesweepSmem {
    static constexpr uint32_t kTile = kThreads * kItems;
    KeyT keys[kTile + kTile / 16];
    uint32_t vals[kTile + kTile / 16];
    uint32_t whist[kThreads / 32][kRadix];
    // per warp and digit (kInvalidDigit too), the lanes that have it (0 at rest)
    uint32_t match[kThreads == 256 ? kThreads / 32 : 1][kRadix + 4];
    uint32_t gdig[kRadix];    // global exclusive digit offsets of this pass
    uint32_t lstart[kRadix];  // block-local digit start
    uint32_t gmap[kRadix];    // global position of local index 0 of each digit
    uint32_t wsum[kThreads / 32];
    uint32_t part;
    uint32_t valid;  // keys of the partition that are written (all but dropped ones)
};

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__global__ void sort_begin_kernel(FrameCtl* ctl, uint32_t total) {
    const uint32_t t = threadIdx.x;
    for (uint32_t i = t; i < 32; i += blockDim.x) ctl->ticket[i] = 0;
    for (uint32_t i = t; i < 8 * 256; i += blockDim.x) {
        (&ctl->sort_hist[0][0])[i] = 0;
        (&ctl->depth_hist[0][0])[i] = 0;
    }
    if (t == 0) {
        ctl->tag = ctl->tag + 1;
        ctl->status = 0;
        ctl->total_keys = total;
    }
}

// Digit counts of a standalone sort: one read of the keys, one shared-memory
// increment per key and digit (an increment by one of one address from
// several lanes is a single operation of the hardware), in four copies by warp
// so that warps rarely meet, then one global atomic per non-zero bin and CTA.
// 9M keys of 45 bits: 25 us (72 MB, 11 us at copy speed); with match-any
// aggregation, six per key, it was 290 us. kHistKeys loads per thread are in flight at once.
constexpr uint32_t kHistCopies = 4;
constexpr uint32_t kHistKeys = 8;

template <typename KeyT>
__global__ void __launch_bounds__(kHistThreads)
    sort_histogram_kernel(const KeyT* __restrict__ keys, uint32_t capacity, uint32_t p0, uint32_t p1,
                          uint32_t key_bits, uint32_t (*hist)[256], FrameCtl* ctl) {
    __shared__ uint32_t sh[kHistCopies][8][kRadix];
    // launched as a dependent of the stream's previous kernel: its output is
    // read below. No early trigger: the next kernel is one wave of CTAs, which
    // must be placed on empty SMs, not onto the first ones this grid frees
    pdl_wait();
    const uint32_t tid = threadIdx.x;
    for (uint32_t i = tid; i < kHistCopies * 8 * kRadix; i += kHistThreads) (&sh[0][0][0])[i] = 0;
    __syncthreads();
    const uint32_t K = (ctl->status & kStatusFatal) ? 0u : min(ctl->total_keys, capacity);
    uint32_t(*mine)[kRadix] = sh[(tid >> 5) % kHistCopies];
    auto count = [&](KeyT k) {
#pragma unroll
        for (uint32_t p = 0; p < 8; ++p) {
            if (p < p0 || p >= p1) continue;  // (uniform)
            const uint32_t b = min(kRadixBits, key_bits - p * kRadixBits);
            atomicAdd(&mine[p][uint32_t(uint64_t(k) >> (p * kRadixBits)) & ((1u << b) - 1u)], 1u);
        }
    };
    const uint32_t nchunks = (K + kHistChunk - 1) / kHistChunk;
    for (uint32_t c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const uint32_t base = c * kHistChunk + tid;
        KeyT k[kHistKeys];
#pragma unroll
        for (uint32_t j = 0; j < kHistKeys; ++j)
            k[j] = base + j * kHistThreads < K ? keys[base + j * kHistThreads] : KeyT(0);
#pragma unroll
        for (uint32_t j = 0; j < kHistKeys; ++j)
            if (base + j * kHistThreads < K) count(k[j]);
    }
    __syncthreads();
    for (uint32_t p = p0; p < p1; ++p)
        for (uint32_t d = tid; d < kRadix; d += kHistThreads) {
            uint32_t c = 0;
#pragma unroll
            for (uint32_t q = 0; q < kHistCopies; ++q) c += sh[q][p][d];
            if (c) atomicAdd(&hist[p][d], c);
        }
}

// Resolves the exclusive prefix of one digit for partition `part` by walking
// predecessors; up to kLookbackWindow descriptors are loaded per round trip
// (8 measured the same, 16 slower: the extra registers spill).
constexpr int kLookbackWindow = 4;
__device__ __forceinline__ uint32_t digit_lookback(const uint64_t* __restrict__ desc, uint32_t part, uint32_t digit,
                                                   uint32_t tag, FrameCtl* ctl, uint32_t spin_limit) {
    constexpr int W = kLookbackWindow;
    uint32_t excl = 0;
    int64_t p = int64_t(part) - 1;
    uint32_t spins = 0;
    while (p >= 0) {
        uint64_t d[W];
        const int cnt = p >= W - 1 ? W : int(p) + 1;
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (j < cnt) d[j] = ld_relaxed_u64(desc + size_t(p - j) * kRadix + digit);  // 0 <= p - j < part
        bool stop = false, wait = false;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            if (j >= cnt || stop || wait) continue;
            const uint32_t f = desc_flag(d[j], tag);
            if (f == 0u) {
                wait = true;  // not yet published: retry from here
            } else {
                excl += uint32_t(d[j]);
                --p;
                if (f == uint32_t(kFlagPrefix)) stop = true;
            }
        }
        if (stop) break;
        if (wait) {
            if (++spins > spin_limit) {
                atomicOr(&ctl->status, kStatusLookbackTimeout);
                break;
            }
            __nanosleep(32);
        }
    }
    return excl;
}

// Tile ranges (range.slang:18-35) from the last pass of the key sort: the
// partition's keys sit in shared memory fully sorted within each digit run,
// and a digit run is contiguous in the output. A tile starts where the run's
// previous key has another tile and ends where the next one has; at the
// edges of a run the neighbour lies in another partition, and min / max
// reductions over all candidates give the range whatever the order.
// A key's tile id: the high 32 bits of a (tile | depth) key, or the whole of
// a 32-bit tile-id key.
__device__ __forceinline__ uint32_t tile_of(uint64_t key) { return uint32_t(key >> 32); }
__device__ __forceinline__ uint32_t tile_of(uint32_t key) { return key; }

template <int kItems, int kThreads, typename KeyT>
__device__ __forceinline__ void tile_range_bounds(const OnesweepSmem<kItems, kThreads, KeyT>& S, uint32_t* ranges,
                                                  uint32_t n_tiles, KeyT key, uint32_t j, uint32_t cnt,
                                                  uint32_t d, uint32_t g, uint32_t shift, uint32_t mask,
                                                  FrameCtl* ctl) {
    const uint32_t t = tile_of(key);
    if (!TPD_INBOUNDS(ctl, 18, t, n_tiles)) return;
    bool first = j == 0, last = j + 1 == cnt;
    if (!first) {
        const KeyT kp = S.keys[pad16(j - 1)];
        first = (uint32_t(kp >> shift) & mask) != d || tile_of(kp) != t;
    }
    if (!last) {
        const KeyT kn = S.keys[pad16(j + 1)];
        last = (uint32_t(kn >> shift) & mask) != d || tile_of(kn) != t;
    }
    if (first) atomicMin(&ranges[2 * t], g);
    if (last) atomicMax(&ranges[2 * t + 1], g + 1);
}

// kThreads = 256 (one digit per thread) or 512 (the digit-wide steps run on
// the first 256 threads); a partition is kThreads * kItems keys. kPass is a
// pass kind (kPassPlain ...): dropped keys are ranked as past-the-end keys.
// KeyT is uint64_t ((tile | depth) or (view | depth) keys) or uint32_t (tile
// ids, whose depth order the depth presort has already fixed).
template <int kItems, int kThreads, int kMinBlocks, int kPass, typename KeyT>
__global__ void __launch_bounds__(kThreads, kMinBlocks)
    onesweep_kernel(const KeyT* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                    KeyT* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t capacity,
                    uint32_t pass, uint32_t shift, uint32_t bits, const uint32_t (*hist)[256], uint32_t ticket_slot,
                    uint32_t tag_slot, uint32_t fixed_count, uint64_t* __restrict__ desc, FrameCtl* ctl,
                    uint32_t spin_limit, uint32_t* __restrict__ ranges, uint32_t n_tiles, uint32_t abort_mask) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr uint32_t kSortItems = kItems, kSortTile = kThreads * kItems, kWarps = kThreads / 32;
    // launched as a dependent of the stream's previous kernel: its output is
    // read below. No early trigger: the next kernel is one wave of CTAs, which
    // must be placed on empty SMs, not onto the first ones this grid frees
    pdl_wait();
    // digits ranked with match-any in the 512-thread variant (32 warps per SM
    // hide its latency), with shared atomics or bit ballots otherwise (below)
    constexpr bool kMatchRank = kThreads == 512;
    OnesweepSmem<kItems, kThreads, KeyT>& S = *reinterpret_cast<OnesweepSmem<kItems, kThreads, KeyT>*>(smem_raw);
    const bool digit_thread = threadIdx.x < kRadix;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    constexpr bool kDrop = kPass == kPassDropCulled;
    static_assert(kPass == kPassPlain || sizeof(KeyT) == 8, "depth-sort pass kinds take 64-bit keys");
    const uint32_t K = (ctl->status & abort_mask)
                           ? 0u
                           : min(kPass == kPassCompacted ? ctl->depth_count
                                                         : (fixed_count ? fixed_count : ctl->total_keys),
                                 capacity);
    if constexpr (kPass == kPassCompacted) {
        if (ctl->depth_skips & 1u) {  // an earlier pass was skipped: its input buffer holds the order
            KeyT* const k = const_cast<KeyT*>(keys_in);
            keys_in = keys_out;
            keys_out = k;
            uint32_t* const v = const_cast<uint32_t*>(vals_in);
            vals_in = vals_out;
            vals_out = v;
        }
    }
    const uint32_t nparts = (K + kSortTile - 1) / kSortTile;
    const uint32_t tag = ctl->tag * 32u + tag_slot;
    const uint32_t mask = (1u << bits) - 1u;
    // digits of this pass's width: only these count, publish and look back
    // (a 5-bit pass leaves 224 of the 256 digit threads idle)
    const bool live_digit = tid <= mask;

    // global exclusive digit offsets (histogram of this pass, scanned)
    const uint32_t h = digit_thread && TPD_INBOUNDS(ctl, 16, pass, 8) ? hist[pass][tid] : 0u;
    {
        const uint32_t ex = block_exclusive_scan<kWarps>(h, S.wsum);
        if (digit_thread) S.gdig[tid] = ex;
    }
    if constexpr (kPass == kPassCompacted) {
        // a pass whose digit is the same for all K keys leaves their order as
        // it is: it is skipped and counted, and the order stays in its input
        // buffer (every CTA takes the same decision from the same histogram)
        if (__syncthreads_or(digit_thread && K > 0 && h == K)) {
            if (blockIdx.x == 0 && tid == 0) atomicAdd(&ctl->depth_skips, 1u);
            return;
        }
    }

    // How a warp finds its lanes of one digit: an atomic OR into a shared word
    // per (warp, digit), where lanes that share a digit queue, or a ballot per
    // digit bit, whatever the digits. The OR is faster unless a digit has more
    // than a 24th of the keys, which the pass's histogram tells. 9M keys of 45
    // bits, us, OR / ballots: random digits 495 / 540, 64 digits of each byte
    // 548 / 551, 16 digits 663 / 573, 4 digits 634 / 535. With the choice (the
    // ballots are a little slower beside the other loop): 499, 568, 595, 561;
    // the depth sort of 3M 130 -> 124, of 500,000 in 8 views 220 -> 210.
    constexpr bool kMayMatch = kThreads == 256;
    bool by_match = false;
    if constexpr (kMayMatch) {
        for (uint32_t i = tid; i < kWarps * (kRadix + 4); i += kThreads) (&S.match[0][0])[i] = 0;
        by_match = !__syncthreads_or(h > K / 24u);
    }

    // Warp-striped items, loaded coalesced straight from global memory: warp w
    // owns [w*32*kItems, (w+1)*32*kItems), item i covers 32 consecutive keys.
    // Variants with registers to spare load the values with the keys. The
    // 256-thread variants load a CTA's next partition while they write out the
    // current one (thread 0 takes its ticket after its look-back), hiding the
    // load latency behind the write-out; the 512-thread variant, at 64
    // registers, takes its ticket and loads at the top of each partition.
    constexpr bool kValsEarly = kItems * kMinBlocks * (kThreads / 256) <= 32;
    constexpr bool kPrefetch = kThreads == 256;
    KeyT k[kSortItems];
    uint32_t vr[kValsEarly ? kSortItems : 1];
    auto load_partition = [&](uint32_t p) {
        const uint32_t b = p * kSortTile, c = p < nparts ? min(kSortTile, K - b) : 0u;
#pragma unroll
        for (uint32_t i = 0; i < kSortItems; ++i) {
            const uint32_t idx = warp * (kSortItems * 32) + i * 32 + lane;
            k[i] = idx < c ? keys_in[b + idx] : KeyT(~KeyT(0));
            if constexpr (kValsEarly) vr[i] = idx < c ? vals_in[b + idx] : 0u;
        }
    };
    uint32_t part = 0;
    if constexpr (kPrefetch) {
        if (tid == 0) S.part = atomicAdd(&ctl->ticket[ticket_slot], 1u);
        __syncthreads();
        part = S.part;
        load_partition(part);
    }

    while (true) {
        if constexpr (!kPrefetch) {
            if (tid == 0) S.part = atomicAdd(&ctl->ticket[ticket_slot], 1u);
        }
#pragma unroll
        for (uint32_t i = tid; i < kWarps * kRadix; i += kThreads) (&S.whist[0][0])[i] = 0;
        __syncthreads();
        if constexpr (!kPrefetch) part = S.part;
        if (part >= nparts) break;
        if constexpr (!kPrefetch) load_partition(part);
        const uint32_t base = part * kSortTile;
        const uint32_t cnt = min(kSortTile, K - base);

        // dr[i] packs the digit (bits 0..8, kInvalidDigit past K) and the
        // key's rank among equal digits earlier in the warp (bits 9..31).
        uint32_t dr[kSortItems];
        const uint32_t lt = lanemask_lt();
        auto rank = [&](auto match_tag) {
            constexpr bool kMatch = decltype(match_tag)::value;
#pragma unroll
            for (uint32_t i = 0; i < kSortItems; ++i) {
                const uint32_t idx = warp * (kSortItems * 32) + i * 32 + lane;
                const uint32_t d = idx < cnt && !(kDrop && uint32_t(k[i]) == 0xFFFFFFFFu) ? (uint32_t(k[i] >> shift) & mask)
                                                                                         : kInvalidDigit;
                uint32_t peers;
                if constexpr (kMatch) {
                    atomicOr(&S.match[warp][d], 1u << lane);
                    __syncwarp();
                    peers = S.match[warp][d];
                } else if constexpr (kMatchRank) {
                    peers = __match_any_sync(0xFFFFFFFFu, d);
                } else {
                    // lanes with the same digit: one ballot per digit bit (bits
                    // above the pass's width are zero in every valid lane and
                    // leave the mask as it is), and one for the past-the-end (or
                    // dropped) digit in the partitions that can have any
                    peers = 0xFFFFFFFFu;
#pragma unroll
                    for (uint32_t b = 0; b < kRadixBits; ++b) {
                        const bool on = (d >> b) & 1u;
                        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
                        peers &= on ? bal : ~bal;
                    }
                    if (kDrop || cnt < kSortTile) {
                        const bool on = d >= kRadix;
                        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
                        peers &= on ? bal : ~bal;
                    }
                }
                const uint32_t leader = __ffs(peers) - 1;
                uint32_t prev = 0;
                if (lane == leader && d < kRadix) {
                    prev = S.whist[warp][d];
                    S.whist[warp][d] = prev + __popc(peers);
                }
                if constexpr (kMatch) {
                    __syncwarp();  // (every lane has read its word)
                    if (lane == leader) S.match[warp][d] = 0u;
                }
                prev = __shfl_sync(0xFFFFFFFFu, prev, leader);
                dr[i] = d | ((prev + __popc(peers & lt)) << 9);
                __syncwarp();
            }
        };
        if constexpr (kMayMatch) {
            if (by_match)
                rank(std::true_type{});
            else
                rank(std::false_type{});
        } else {
            rank(std::false_type{});
        }
        __syncthreads();

        // per digit (thread = digit): warp prefixes, block count, local start
        uint32_t count = 0;
        uint64_t* dp = nullptr;
        if (live_digit) {
#pragma unroll
            for (uint32_t w = 0; w < kWarps; ++w) {
                const uint32_t c = S.whist[w][tid];
                S.whist[w][tid] = count;
                count += c;
            }
            dp = desc + size_t(TPD_INBOUNDS(ctl, 13, part, nparts) ? part : 0) * kRadix + tid;
            st_relaxed_u64(dp, make_desc(part == 0 ? kFlagPrefix : kFlagAggregate, tag, count));
        }
        const uint32_t lstart = block_exclusive_scan<kWarps>(count, S.wsum);  // (its barriers cover whist)
        if (digit_thread) S.lstart[tid] = lstart;
        if (kDrop && tid == kRadix - 1) S.valid = lstart + count;
        __syncthreads();

        // reorder the partition in shared memory (stable: warp, then item, then
        // lane) while predecessors publish; values not held in registers are
        // loaded now, coalesced
        if constexpr (kValsEarly) {
            // key and value go to the same slot: one position per item
#pragma unroll
            for (uint32_t i = 0; i < kSortItems; ++i) {
                const uint32_t d = dr[i] & 511u;
                if (d < kRadix) {
                    const uint32_t pos = S.lstart[d] + S.whist[warp][d] + (dr[i] >> 9);
                    if (TPD_INBOUNDS(ctl, 11, pos, cnt)) {
                        S.keys[pad16(pos)] = k[i];
                        S.vals[pad16(pos)] = vr[i];
                    }
                }
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < kSortItems; ++i) {
                const uint32_t d = dr[i] & 511u;
                if (d < kRadix) {
                    const uint32_t pos = S.lstart[d] + S.whist[warp][d] + (dr[i] >> 9);
                    if (TPD_INBOUNDS(ctl, 11, pos, cnt)) S.keys[pad16(pos)] = k[i];
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < kSortItems; ++i) {
                const uint32_t idx = warp * (kSortItems * 32) + i * 32 + lane;
                const uint32_t d = dr[i] & 511u;
                if (d < kRadix) {
                    const uint32_t v = vals_in[base + idx];
                    const uint32_t pos = S.lstart[d] + S.whist[warp][d] + (dr[i] >> 9);
                    if (TPD_INBOUNDS(ctl, 12, pos, cnt)) S.vals[pad16(pos)] = v;
                }
            }
        }

        // decoupled look-back for this thread's digit; then (prefetching
        // variants) thread 0 takes the next partition's ticket: every thread
        // has read S.part since it was last written
        if (live_digit) {
            if (part > 0) {
                const uint32_t excl = digit_lookback(desc, part, tid, tag, ctl, spin_limit);
                st_relaxed_u64(dp, make_desc(kFlagPrefix, tag, excl + count));
                S.gmap[tid] = S.gdig[tid] + excl - lstart;
            } else {
                S.gmap[tid] = S.gdig[tid] - lstart;
            }
        }
        if constexpr (kPrefetch) {
            if (tid == 0) S.part = atomicAdd(&ctl->ticket[ticket_slot], 1u);
        }
        __syncthreads();
        if constexpr (kPrefetch) {
            part = S.part;
            load_partition(part);  // k and vr are free since the reorder
        }

        // coalesced write-out of digit runs
        const uint32_t cntv = kDrop ? S.valid : cnt;
        for (uint32_t j = tid; j < cntv; j += kThreads) {
            const KeyT key = S.keys[pad16(j)];
            const uint32_t d = uint32_t(key >> shift) & mask;
            const uint32_t g = S.gmap[d] + j;
            if (g < capacity && TPD_INBOUNDS(ctl, 17, g, K + (K == 0))) {
                keys_out[g] = key;
                vals_out[g] = S.vals[pad16(j)];
                if (ranges) tile_range_bounds(S, ranges, n_tiles, key, j, cntv, d, g, shift, mask, ctl);
            }
        }
        __syncthreads();  // S.keys / S.vals / S.gmap are rewritten by the next partition
    }
}

// ---- counted passes: a radix pass without look-back
//
// The look-back of onesweep_kernel puts a wait on every partition's critical
// path (measured on the key sort of 1M Gaussians at 1080p: 4.4 of 10.5 us per
// partition, after load and rank 3.0, scan 0.4, write-out 2.6). A counted pass
// computes every partition's digit offsets beforehand instead:
//  1. partition_count_kernel, one CTA per 4096-key partition: the partition's
//     digit counts (per-warp shared-memory counts), stored as a row of the
//     work area and scanned by the last CTAs to arrive (counted_finish in
//     tpd_counted.cuh; nobody waits). The first pass of the frame's key sort
//     is counted by the kernel that writes its keys (keygen.cu) instead.
//  2. scatter_kernel, one CTA per partition: load, rank (bit ballots, or shared
//     atomics over strips; stable in warp-striped order), reorder in shared memory and write out at the
//     partition's global digit offsets, as onesweep_kernel does but with them
//     known: no partition waits for another.
// The permutation is the same stable one.
// Digits have 8 bits, or 9 (kDig = 512) where that takes a pass less. (The
// count's 40 registers for six CTAs per SM spill 4 bytes, 16 with 9 bits; the
// 9-bit scatters spill 4.)
template <int kItems, uint32_t kDig, typename KeyT>
__global__ void __launch_bounds__(256, 6) partition_count_kernel(const KeyT* __restrict__ keys, uint32_t capacity,
                                                              uint32_t shift, uint32_t bits, uint32_t fixed_count,
                                                              uint32_t max_parts, uint32_t* __restrict__ work,
                                                              FrameCtl* ctl, uint32_t abort_mask) {
    constexpr uint32_t kTile = 256 * kItems, kPer = kDig / 256;
    __shared__ uint32_t hw[8][kDig];  // per-warp counts
    __shared__ uint32_t wsum[8];
    __shared__ bool last;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // launched as a dependent of the kernel that wrote the keys: wait for it,
    // then let the scatter be scheduled (it loads its keys and values while
    // the last partitions are counted; they come from the kernel this one
    // waited for)
    pdl_wait();
    pdl_trigger();
    const uint32_t K = (ctl->status & abort_mask) ? 0u : min(fixed_count ? fixed_count : ctl->total_keys, capacity);
    const uint32_t nparts = min((K + kTile - 1) / kTile, max_parts);
    const uint32_t part = blockIdx.x;
    if (part >= nparts) return;  // (uniform)
    const uint32_t mask = (1u << bits) - 1u;
    const uint32_t base = part * kTile, cnt = min(kTile, K - base);
    KeyT k[kItems];
#pragma unroll
    for (uint32_t i = 0; i < kItems; ++i) {
        const uint32_t idx = i * 256 + tid;
        k[i] = idx < cnt ? keys[base + idx] : KeyT(0);
    }
    // (while the loads are in flight) each warp clears its own counts
#pragma unroll
    for (uint32_t j = 0; j < kDig / 32; ++j) hw[warp][lane + 32 * j] = 0;
    __syncwarp();
    // 32 consecutive keys often share a digit (a Gaussian's row of tiles, in
    // the high digit): then one add of 32, else one shared atomic per key
#pragma unroll
    for (uint32_t i = 0; i < kItems; ++i) {
        const uint32_t idx = i * 256 + tid;
        const uint32_t d = idx < cnt ? (uint32_t(k[i] >> shift) & mask) : kDig;
        const uint32_t d0 = __shfl_sync(0xFFFFFFFFu, d, 0);
        if (__all_sync(0xFFFFFFFFu, d == d0)) {
            if (lane == 0 && d < kDig) hw[warp][d] += 32u;
        } else if (d < kDig) {
            atomicAdd(&hw[warp][d], 1u);
        }
    }
    __syncthreads();
    RowDigits<kPer> total = {};
#pragma unroll
    for (uint32_t w = 0; w < 8; ++w)
#pragma unroll
        for (uint32_t p = 0; p < kPer; ++p) total.v[p] += hw[w][kPer * tid + p];
    counted_finish<kDig>(CountedWork<kDig>(work, max_parts), nparts, part, total, wsum, last);
}

// Strips. A rectangle of w x h tiles is w h keys but w column strips, and a key
// is its strip's column and one of its rows. So a frame of one view sorts the
// strips by column (a counted pass whose heights are counted too, which gives
// each sorted strip its first key slot), and its last pass, by row, makes the
// keys of 4096 consecutive slots from their strips instead of loading them:
// (row, column, depth) order with the keys ranked and moved once, not twice.
// 3M Gaussians at 2160p, us: expand 242 -> 67, counts 110 -> 52, first scatter
// 412 -> 98 (of strips), last 476 -> 480 (now with the expansion).

// What a scatter moves.
constexpr int kScatterPairs = 0;    // keys and values
constexpr int kScatterLast = 1;     // the last pass: values, and the tile ranges
constexpr int kScatterColumns = 2;  // strips, by column; also each strip's first key slot
constexpr int kScatterRows = 3;     // the keys of column-sorted strips, by row: the last pass

// Column-sorted strips (kScatterColumns writes them, kScatterRows expands them).
struct StripList {
    uint32_t *keys, *vals, *starts;  // strip_key, Gaussian, first key slot
    uint32_t* part_first;            // the strip that holds the first slot of every 4096-key partition
    uint32_t gx;                     // the image's tile columns
};

// The rows of every 4096-key partition of column-sorted strips: a strip covers
// consecutive rows, so it adds one where its slots of the partition begin and
// takes one where they end, and a prefix sum gives the counts (two shared
// atomics per strip, none per key). kParts partitions per CTA: latency is all
// it spends, of the loads and of the arrivals (keygen + key sort with 1 / 2 / 4
// / 8 of them: 817 / 798 / 789 / 816 us for 3M Gaussians at 2160p, 150 / 148 /
// 151 / 154 for 1M at 1080p, 98 / 101 / 102 / 106 for 2M seen from inside).
// (48 registers for five CTAs per SM spill 12 bytes; registers for six spill
// more: 2 us slower.)
template <uint32_t kParts>
__global__ void __launch_bounds__(256, 5) strip_rows_kernel(StripList strips, uint32_t capacity, uint32_t max_parts,
                                                            uint32_t* __restrict__ work, FrameCtl* ctl,
                                                            uint32_t abort_mask) {
    constexpr uint32_t kTile = 4096, kGroup = 256 / kParts;  // threads per partition
    __shared__ __align__(16) uint32_t edges[kParts][260];
    __shared__ uint32_t wsum[8];
    __shared__ bool s_last;
    pdl_wait();
    pdl_trigger();
    const uint32_t tid = threadIdx.x, at = tid % kGroup, group = tid / kGroup;
    const bool off = ctl->status & abort_mask;
    const uint32_t K = off ? 0u : min(ctl->total_keys, capacity), n_strips = min(ctl->total_strips, capacity);
    const uint32_t nparts = min((K + kTile - 1) / kTile, max_parts);
    const uint32_t part0 = blockIdx.x * kParts, part = part0 + group;
    if (part0 >= nparts) return;  // (uniform)
    const CountedWork<256> W(work, max_parts);
    for (uint32_t k = tid; k < kParts * 260; k += 256) (&edges[0][0])[k] = 0;
    uint32_t* edge = edges[group];
    const uint32_t base = part * kTile, end = part < nparts ? base + min(kTile, K - base) : base;
    uint32_t first = 1, last = 0;
    if (part < nparts) {
        first = min(strips.part_first[part], n_strips - 1u);
        last = part + 1u < nparts ? min(strips.part_first[part + 1u], n_strips - 1u) : n_strips - 1u;
    }
    __syncthreads();
    for (uint32_t q0 = first; q0 <= last; q0 += 4 * kGroup) {
        uint32_t strip[4], start[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t q = q0 + kGroup * u + at;
            strip[u] = q <= last ? strips.keys[q] : 0u;  // (no height: nothing is added)
            start[u] = q <= last ? strips.starts[q] : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t lo = max(start[u], base), hi = min(start[u] + strip_height(strip[u]), end);
            const uint32_t row = strip_row(strip[u]) + lo - start[u];
            if (lo < hi && TPD_INBOUNDS(ctl, 23, row + hi - lo, 257)) {
                atomicAdd(&edge[row], 1u);
                atomicSub(&edge[row + hi - lo], 1u);
            }
        }
    }
    __syncthreads();
    if (at < 32 && part < nparts) {  // a warp: rows 8 at .. 8 at + 7
        uint32_t v[8], sum = 0;
        *reinterpret_cast<uint4*>(v) = reinterpret_cast<const uint4*>(edge)[2 * at];
        *reinterpret_cast<uint4*>(v + 4) = reinterpret_cast<const uint4*>(edge)[2 * at + 1];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) sum = v[k] += sum;
        const uint32_t before = warp_inclusive_scan(sum) - sum;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) v[k] += before;
        uint4* row = reinterpret_cast<uint4*>(W.rows + size_t(part) * 256);
        row[2 * at] = *reinterpret_cast<const uint4*>(v);
        row[2 * at + 1] = *reinterpret_cast<const uint4*>(v + 4);
    }
    counted_arrive<256, kParts>(W, nparts, part0, wsum, s_last);
}
constexpr uint32_t kStripParts = 2;

// A partition of a scatter: its pairs reordered by digit, each in one 8-byte
// slot (one store and one load per pair), one pad slot per 16 (pad16).
template <uint32_t kDig, int kMode>
struct ScatterSmem {
    uint2 pairs[4096 + 4096 / 16];  // key, value
    uint32_t whist[8][kDig];        // per-warp digit counts, then the first slot of the warp's keys of each digit
    uint32_t gmap[kDig];            // global position of local index 0 of each digit
    uint32_t wsum[8];
    // strips: per warp and digit, the lanes that have it (0 at rest)
    uint32_t match[kMode >= kScatterColumns ? 8 : 1][kDig];
    // columns: the local prefix of the heights, and the columns' offsets (strips,
    // heights), then the key slot of local height 0 of each column
    uint32_t hpre[kMode == kScatterColumns ? 4096 + 4096 / 16 : 1];
    uint32_t hmap[kMode == kScatterColumns ? 512 : 2];
};

// kBits: the pass's digit width (1..9); the lanes with the same digit are
// found with one ballot per digit bit (the launch picks the variant of the
// pass's width: a 5-bit pass ranks with 5 ballots, not 8).
// kLast: the last pass. Nothing reads the sorted tile ids after it (the tile
// ranges hold them), so only the values are written, and the ranges: the
// partition's keys sit in shared memory fully sorted within each digit run, so
// a key that differs from the one before it ends that one's tile and starts
// its own; at the partition's edges min / max over the neighbours' candidates
// give the range whatever the order (range.slang:18-35). Against writing the
// keys too and comparing both neighbours of every key: 1M Gaussians at 1080p 57
// -> 51 us, 3M at 2160p 573 -> 501.
// Strips (kScatterColumns, kScatterRows; see above): the lanes of one digit are
// found by an atomic OR into a word per (warp, digit), as 32 strips or keys in
// a row seldom share one: 855 -> 816 us (keygen + key sort, 3M Gaussians at
// 2160p). With keys, whose last pass has most of a warp on one digit, ballots
// are faster (251 and 284 us for 8 views of 500,000). A CTA's strips are staged
// in shared memory while their slots are marked: 798 -> 699 us against two
// gathers per key.
// What bounds it: the shared-memory pipe (75% busy with keys and values in
// arrays of their own and the digit and warp offsets looked up apart) and the
// integer pipe (63%: ballots). Pairs in one slot and merged offsets took both
// passes and the count from 120 to 108 us at 1M Gaussians and 1080p; 64
// registers for a fourth CTA per SM spill (118).
template <int kMinBlocks, int kBits, int kMode, typename KeyT>
__global__ void __launch_bounds__(256, kMinBlocks)
    scatter_kernel(const KeyT* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, KeyT* __restrict__ keys_out,
                   uint32_t* __restrict__ vals_out, uint32_t capacity, uint32_t shift, uint32_t bits,
                   uint32_t fixed_count, uint32_t max_parts, uint32_t* __restrict__ work, FrameCtl* ctl,
                   uint32_t* __restrict__ ranges, uint32_t n_tiles, uint32_t abort_mask, bool keys_just_written,
                   StripList strips) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr bool kLast = kMode == kScatterLast || kMode == kScatterRows;
    constexpr bool kMatch = kMode >= kScatterColumns;  // lanes of one digit by shared atomics, not by ballots
    constexpr uint32_t kItems = 16, kSortTile = 4096, kWarps = 8;
    constexpr uint32_t kDig = kBits > 8 ? 512 : 256, kPer = kDig / 256;
    static_assert(sizeof(KeyT) == 4, "a pair is 8 bytes");
    ScatterSmem<kDig, kMode>& S = *reinterpret_cast<ScatterSmem<kDig, kMode>*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // the keys and values come from the kernel before the counting one, so they
    // are loaded while that one finishes; or (keys_just_written) from the
    // kernel right before this one, which counted them as it wrote them
    if (keys_just_written) pdl_wait();
    const uint32_t total = kMode == kScatterColumns ? ctl->total_strips : ctl->total_keys;
    const uint32_t K = (ctl->status & abort_mask) ? 0u : min(fixed_count ? fixed_count : total, capacity);
    const uint32_t nparts = min((K + kSortTile - 1) / kSortTile, max_parts);
    const uint32_t part = blockIdx.x;
    if (part >= nparts) return;  // (uniform)
    const uint32_t mask = (1u << bits) - 1u;
    const uint32_t base = part * kSortTile, cnt = min(kSortTile, K - base);
    // kFull: a whole partition (all but the last), without per-key bounds
    // checks and with a fixed write-out loop
    auto partition = [&](auto full_tag) {
        constexpr bool kFull = decltype(full_tag)::value;
        KeyT k[kMode == kScatterRows ? kItems / 2 : kItems];  // (rows: 16-bit keys, two to a register)
        uint32_t vr[kItems];
        auto key_at = [&](uint32_t i) -> KeyT {
            return kMode == kScatterRows ? (i & 1u ? k[i / 2] >> 16 : k[i / 2] & 0xFFFFu) : k[i];
        };
        // the strips of the partition's slots: the keys are column << 8 | row
        [[maybe_unused]] uint16_t* owner = reinterpret_cast<uint16_t*>(&S.whist[0][0]);
        [[maybe_unused]] uint32_t first = 0, col0 = 0;
        [[maybe_unused]] bool one_column = false;
        if constexpr (kMode == kScatterRows) {
            const uint32_t n_strips = min(ctl->total_strips, capacity);
            first = min(strips.part_first[part], n_strips - 1u);
            const uint32_t last = part + 1u < nparts ? min(strips.part_first[part + 1u], n_strips - 1u) : n_strips - 1u;
            const uint32_t m = min(last - first + 1u, kSortTile + 1u);
            // a strip's column << 8 | the row that it would have at the partition's slot 0, and its value
            slot_owners(owner, m, cnt, S.wsum, [&](uint32_t q) {
                const uint32_t strip = strips.keys[first + q], slot = strips.starts[first + q] - base;
                const uint32_t key = strip_col(strip) << 8 | ((strip_row(strip) - slot) & 0xFFu);
                S.pairs[q] = make_uint2(key, strips.vals[first + q]);
                return slot;
            });
            col0 = S.pairs[0].x >> 8;
            one_column = S.pairs[owner[cnt - 1]].x >> 8 == col0;
        }
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            const uint32_t idx = warp * (kItems * 32) + i * 32 + lane;
            if constexpr (kMode == kScatterRows) {
                const uint2 strip = S.pairs[owner[idx]];  // (past cnt: the last strip)
                const uint32_t key = (strip.x & 0xFF00u) | ((strip.x + idx) & 0xFFu);
                k[i / 2] = i & 1u ? k[i / 2] | key << 16 : key;
                vr[i] = strip.y;
            } else if (kFull || idx < cnt) {
                k[i] = keys_in[base + idx];
                vr[i] = vals_in[base + idx];
            } else {
                k[i] = KeyT(~KeyT(0));
                vr[i] = 0u;
            }
        }
        if constexpr (kMode == kScatterRows) __syncthreads();  // (the owners are read: their words are cleared next)
        // this partition's digit offsets, written by the counting kernel (this
        // kernel may have started while it ran)
        pdl_wait();
        pdl_trigger();  // the next kernel (the next counting kernel, or the blend) may be scheduled; it waits for this grid
        RowDigits<kPer> goff;
        [[maybe_unused]] uint32_t hoff = 0;
        if constexpr (kMode == kScatterColumns) {
            // 512 digits were counted: the heights' offsets start after all the strips
            const RowDigits<2> both = counted_offset<512>(CountedWork<512>(work, max_parts), nparts, part, S.wsum);
            S.hmap[2 * tid] = both.v[0];
            S.hmap[2 * tid + 1] = both.v[1];
            __syncthreads();
            goff.v[0] = S.hmap[tid];
            hoff = S.hmap[256 + tid] - K;
        } else {
            goff = counted_offset<kDig>(CountedWork<kDig>(work, max_parts), nparts, part, S.wsum);
        }
#pragma unroll
        for (uint32_t i = tid; i < kWarps * kDig / 4; i += 256)
            reinterpret_cast<uint4*>(&S.whist[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (kMatch)
#pragma unroll
            for (uint32_t i = tid; i < kWarps * kDig / 4; i += 256)
                reinterpret_cast<uint4*>(&S.match[0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        // stable rank within the warp (warp-striped order)
        uint32_t rank[kItems / 2];  // two 16-bit ranks each
        const uint32_t lt = lanemask_lt();
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            const uint32_t idx = warp * (kItems * 32) + i * 32 + lane;
            const uint32_t d = kFull || idx < cnt ? (uint32_t(key_at(i) >> shift) & mask) : kDig;
            uint32_t peers = 0xFFFFFFFFu;
            if constexpr (kMatch) {
                if (kFull || d < kDig) atomicOr(&S.match[warp][d], 1u << lane);
                __syncwarp();
                if (kFull || d < kDig) peers = S.match[warp][d];
            } else {
#pragma unroll
                for (int b = 0; b < kBits; ++b) {
                    const bool on = (d >> b) & 1u;
                    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
                    peers &= on ? bal : ~bal;
                }
                if constexpr (!kFull) {
                    const bool on = d >= kDig;
                    const uint32_t bal = __ballot_sync(0xFFFFFFFFu, on);
                    peers &= on ? bal : ~bal;
                }
            }
            const uint32_t leader = __ffs(peers) - 1;
            uint32_t prev = 0;
            if (lane == leader && (kFull || d < kDig)) {
                prev = S.whist[warp][d];
                S.whist[warp][d] = prev + __popc(peers);
            }
            __syncwarp();
            if (kMatch && lane == leader && (kFull || d < kDig)) S.match[warp][d] = 0u;
            prev = __shfl_sync(0xFFFFFFFFu, prev, leader);
            const uint32_t r = prev + __popc(peers & lt);
            rank[i / 2] = i & 1u ? rank[i / 2] | r << 16 : r;
            __syncwarp();
        }
        __syncthreads();
        RowDigits<kPer> c[kWarps], count = {};
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w)
#pragma unroll
            for (uint32_t p = 0; p < kPer; ++p) {
                c[w].v[p] = S.whist[w][kPer * tid + p];
                count.v[p] += c[w].v[p];
            }
        RowDigits<kPer> slot = scan_digits<kPer>(count, S.wsum);  // the digits' first slots
#pragma unroll
        for (uint32_t p = 0; p < kPer; ++p) S.gmap[kPer * tid + p] = goff.v[p] - slot.v[p];
        [[maybe_unused]] const uint32_t slot0 = slot.v[0];
        // rows of one column (most partitions of a large frame): each is one
        // tile's keys, and no key has to be compared with the one before it
        if (kMode == kScatterRows && one_column && count.v[0]) {
            const uint32_t tile = tid * strips.gx + col0;
            if (TPD_INBOUNDS(ctl, 18, tile, n_tiles)) {
                atomicMin(&ranges[2 * tile], goff.v[0]);
                atomicMax(&ranges[2 * tile + 1], goff.v[0] + count.v[0]);
            }
        }
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w)
#pragma unroll
            for (uint32_t p = 0; p < kPer; ++p) {
                S.whist[w][kPer * tid + p] = slot.v[p];
                slot.v[p] += c[w].v[p];
            }
        __syncthreads();
#pragma unroll
        for (uint32_t i = 0; i < kItems; ++i) {
            const uint32_t idx = warp * (kItems * 32) + i * 32 + lane;
            if (kFull || idx < cnt) {
                const uint32_t pos =
                    S.whist[warp][(key_at(i) >> shift) & mask] + (i & 1u ? rank[i / 2] >> 16 : rank[i / 2] & 0xFFFFu);
                if (TPD_INBOUNDS(ctl, 20, pos, cnt)) S.pairs[pad16(pos)] = make_uint2(key_at(i), vr[i]);
            }
        }
        __syncthreads();
        if constexpr (kMode == kScatterColumns) {  // the key slots of the sorted strips: a prefix of their heights
            uint32_t h[kItems], sum = 0;
#pragma unroll
            for (uint32_t q = 0; q < kItems; ++q) {
                const uint32_t j = kItems * tid + q;
                h[q] = kFull || j < cnt ? strip_height(S.pairs[pad16(j)].x) : 0u;
                sum += h[q];
            }
            uint32_t before = block_exclusive_scan<kWarps>(sum, S.wsum);
#pragma unroll
            for (uint32_t q = 0; q < kItems; ++q) {
                S.hpre[pad16(kItems * tid + q)] = before;
                before += h[q];
            }
            __syncthreads();
            if (count.v[0]) S.hmap[tid] = hoff - S.hpre[pad16(slot0)];
            __syncthreads();
        }
        // (g < K <= capacity: the bound check covers the buffer's end)
        auto write_out = [&](uint32_t j) {
            const uint2 pair = S.pairs[pad16(j)];
            const KeyT key = pair.x;
            const uint32_t g = S.gmap[(key >> shift) & mask] + j;
            if (!TPD_INBOUNDS(ctl, 22, g, K)) return;
            vals_out[g] = pair.y;
            if (kMode == kScatterRows && one_column) return;
            if constexpr (!kLast) {
                keys_out[g] = key;
                if constexpr (kMode == kScatterColumns) {
                    const uint32_t start = S.hmap[strip_col(key)] + S.hpre[pad16(j)];
                    strips.starts[g] = start;
                    const uint32_t p = (start + kSortTile - 1) / kSortTile;  // (a strip holds at most 256 slots)
                    if (p * kSortTile < start + strip_height(key) && p < max_parts) strips.part_first[p] = g;
                }
            } else {
                auto tile_of = [&](KeyT q) { return kMode == kScatterRows ? (q & 0xFFu) * strips.gx + (q >> 8) : q; };
                const uint32_t tile = tile_of(key);
                if (!TPD_INBOUNDS(ctl, 18, tile, n_tiles)) return;
                const KeyT before = j ? S.pairs[pad16(j - 1)].x : KeyT(~KeyT(0));
                if (before != key) {
                    atomicMin(&ranges[2 * tile], g);
                    if (j && TPD_INBOUNDS(ctl, 18, tile_of(before), n_tiles))
                        atomicMax(&ranges[2 * tile_of(before) + 1], S.gmap[uint32_t(before >> shift) & mask] + j);
                }
                if (j + 1 == cnt) atomicMax(&ranges[2 * tile + 1], g + 1);
            }
        };
        if constexpr (kFull) {
#pragma unroll 4
            for (uint32_t q = 0; q < kItems; ++q) write_out(tid + q * 256);
        } else {
            for (uint32_t j = tid; j < cnt; j += 256) write_out(j);
        }
    };
    if (cnt == kSortTile)
        partition(std::true_type{});
    else
        partition(std::false_type{});
}

// Residencies: the 256-thread, 16-key variant is compiled for 2 CTAs per SM
// (128 registers, no spills; the default) or 3 (80 registers); the 512-thread,
// 8-key variant for 2 (32 warps per SM); the 8- and 4-key 256-thread variants
// (shorter partitions, for small sorts) for 3 and 4 (registers for 4 and 5 spill
// and measured 4 to 8% slower).
// Shared-memory opt-in of every pass kind of a variant and its resident CTAs
// per SM, once per device.
template <int kItems, int kThreads, int kMinBlocks, typename KeyT>
int onesweep_setup() {
    const size_t smem = sizeof(OnesweepSmem<kItems, kThreads, KeyT>);
    cudaFuncSetAttribute(onesweep_kernel<kItems, kThreads, kMinBlocks, kPassPlain, KeyT>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if constexpr (sizeof(KeyT) == 8) {
        cudaFuncSetAttribute(onesweep_kernel<kItems, kThreads, kMinBlocks, kPassDropCulled, KeyT>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        cudaFuncSetAttribute(onesweep_kernel<kItems, kThreads, kMinBlocks, kPassCompacted, KeyT>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    }
    int r = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, onesweep_kernel<kItems, kThreads, kMinBlocks, kPassPlain, KeyT>,
                                                  kThreads, smem);
    return r > 0 ? r : 1;
}

template <int kItems, int kThreads, int kMinBlocks, typename KeyT>
int onesweep_occupancy() {
    return device_once(onesweep_setup<kItems, kThreads, kMinBlocks, KeyT>);
}

template <int kItems, int kThreads, int kMinBlocks, typename KeyT>
void launch_passes(KeyT* kin, uint32_t* vin, KeyT* kout, uint32_t* vout, uint32_t capacity, uint32_t p0,
                   uint32_t p1, const SortPlan& plan, uint32_t (*hist)[256], uint64_t* desc, FrameCtl* ctl,
                   uint32_t spin_limit, int sms, cudaStream_t s) {
    const size_t smem = sizeof(OnesweepSmem<kItems, kThreads, KeyT>);
    const int occ = onesweep_occupancy<kItems, kThreads, kMinBlocks, KeyT>();
    const uint32_t tile = kThreads * kItems;
    const uint32_t max_parts = (capacity + tile - 1) / tile;
    const uint32_t grid = std::max(1u, std::min<uint32_t>(max_parts, uint32_t(sms * occ)));
    for (uint32_t p = p0; p < p1; ++p) {
        const uint32_t shift = p * kRadixBits;
        const uint32_t bits = std::min(kRadixBits, plan.key_bits - shift);
        auto kernel = onesweep_kernel<kItems, kThreads, kMinBlocks, kPassPlain, KeyT>;
        if constexpr (sizeof(KeyT) == 8) {
            if (plan.compact_culled)
                kernel = p == p0 ? onesweep_kernel<kItems, kThreads, kMinBlocks, kPassDropCulled, KeyT>
                                 : onesweep_kernel<kItems, kThreads, kMinBlocks, kPassCompacted, KeyT>;
        }
        launch_dependent(kernel, dim3(grid), dim3(kThreads), smem, s, kin, vin, kout, vout, capacity, p, shift, bits,
                         static_cast<const uint32_t(*)[256]>(hist), plan.ticket_base + p, plan.tag_base + p,
                         plan.fixed_count, desc, ctl, spin_limit, p + 1 == p1 ? plan.ranges : nullptr, plan.n_tiles,
                         kStatusFatal | (plan.skip_on_overflow ? kStatusKeyOverflow : 0u));
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
}

template <int kMinBlocks, int kBits, int kMode, typename KeyT>
int scatter_setup() {
    cudaFuncSetAttribute(scatter_kernel<kMinBlocks, kBits, kMode, KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         int(sizeof(ScatterSmem<(kBits > 8 ? 512 : 256), kMode>)));
    return 1;
}

// Counted passes (see partition_count_kernel): per pass a counting launch and
// a scatter launch, one CTA per 4096-key partition each. work: the counted
// work area (counted_work_words(max partitions) u32, its arrival counts zero
// at rest). The scatter ranks with as many ballots as the pass has bits (the
// default variant; the 2-CTA one with 8 or 9).
template <int kMinBlocks, typename KeyT>
void launch_counted_passes(KeyT* kin, uint32_t* vin, KeyT* kout, uint32_t* vout, uint32_t capacity,
                           const SortPlan& plan, uint32_t* work, FrameCtl* ctl, cudaStream_t s) {
    const uint32_t max_parts = std::max(1u, (capacity + 4095u) / 4096u);
    const uint32_t abort = kStatusFatal | (plan.skip_on_overflow ? kStatusKeyOverflow : 0u);
    const uint32_t width = counted_digit_bits(plan.key_bits);
    for (uint32_t shift = 0; shift < plan.key_bits; shift += width) {
        const uint32_t bits = std::min(width, plan.key_bits - shift);
        const bool last = shift + width >= plan.key_bits && plan.ranges;
        const bool counted = shift == 0 && plan.precounted;
        if (!counted)
            launch_dependent(bits > 8 ? partition_count_kernel<16, 512, KeyT> : partition_count_kernel<16, 256, KeyT>,
                             dim3(max_parts), dim3(256), 0, s, kin, capacity, shift, bits, plan.fixed_count, max_parts,
                             work, ctl, abort);
        auto scatter = [&](auto bits_tag, auto last_tag) {
            constexpr int kBits = decltype(bits_tag)::value;
            constexpr int kMode = decltype(last_tag)::value ? kScatterLast : kScatterPairs;
            device_once(scatter_setup<kMinBlocks, kBits, kMode, KeyT>);
            launch_dependent(scatter_kernel<kMinBlocks, kBits, kMode, KeyT>, dim3(max_parts), dim3(256),
                             sizeof(ScatterSmem<(kBits > 8 ? 512 : 256), kMode>), s, kin, vin, kout, vout, capacity,
                             shift, bits, plan.fixed_count, max_parts, work, ctl, plan.ranges, plan.n_tiles, abort,
                             counted, StripList{});
        };
        auto either = [&](auto bits_tag) {
            last ? scatter(bits_tag, std::true_type{}) : scatter(bits_tag, std::false_type{});
        };
        if (kMinBlocks == 2 && bits <= 8) {
            either(std::integral_constant<int, 8>{});
        } else {
            switch (bits) {
                case 1: either(std::integral_constant<int, 1>{}); break;
                case 2: either(std::integral_constant<int, 2>{}); break;
                case 3: either(std::integral_constant<int, 3>{}); break;
                case 4: either(std::integral_constant<int, 4>{}); break;
                case 5: either(std::integral_constant<int, 5>{}); break;
                case 6: either(std::integral_constant<int, 6>{}); break;
                case 7: either(std::integral_constant<int, 7>{}); break;
                case 8: either(std::integral_constant<int, 8>{}); break;
                default: either(std::integral_constant<int, 9>{}); break;
            }
        }
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
}

template <int kBits, int kMode>
void launch_strip_scatter(const StripSort& a, const StripList& strips, const uint32_t* kin, const uint32_t* vin,
                          uint32_t* kout, uint32_t* vout, uint32_t bits, cudaStream_t s) {
    device_once(scatter_setup<3, kBits, kMode, uint32_t>);
    launch_dependent(scatter_kernel<3, kBits, kMode, uint32_t>, dim3(a.max_parts()), dim3(256),
                     sizeof(ScatterSmem<256, kMode>), s, kin, vin, kout, vout, a.capacity, 0u, bits, 0u,
                     a.max_parts(), a.work, a.ctl, a.ranges, a.n_tiles, kStatusFatal | kStatusKeyOverflow,
                     kMode == kScatterColumns, strips);
}

}  // namespace

size_t sort_counted_work_words(uint32_t capacity) {
    return counted_work_words(std::max(1u, (capacity + 4095u) / 4096u));
}

// Measured (scatters + counts, us): 16 mixed views, 17 bits as 8 + 8 + 1 690 +
// 157, as 9 + 8 514 + 68; 8 views of 2160p, 18 bits, 8 + 8 + 2 2207 + 448, 9 + 9
// 1719 + 255; 256x256, 9 bits, 8 + 1 16 + 2, 9 alone 9. Where both take the
// same passes 8-bit digits write longer runs.
uint32_t counted_digit_bits(uint32_t key_bits) { return (key_bits + 8) / 9 < (key_bits + 7) / 8 ? 9u : 8u; }

uint32_t sort_pass_count(uint32_t key_bits) { return (key_bits + kRadixBits - 1) / kRadixBits; }

size_t sort_desc_entries(uint32_t capacity, uint32_t items) {
    const size_t tile = size_t(kSortThreads) * (items ? items : kSortItemsMax);
    return (size_t(capacity) + tile - 1) / tile * kRadix + kRadix;
}

// Measured on the depth sort (4 passes, us): 30,000 items 42 / 34 / 30 with 16
// / 8 / 4 keys a thread, 120,000 47 / 39 / 38, 250,000 49 / 44 / 48, 500,000
// 56 / 55 / 66, 1M 67 / 70 / 90 (4 keys from 250,000 up: with ballots only).
uint32_t sort_items_limit(uint32_t items) { return items == 4 ? 1u << 17 : items == 8 ? 1u << 19 : 0xFFFFFFFFu; }
uint32_t sort_items_for(uint32_t n) { return n <= sort_items_limit(4) ? 4u : n <= sort_items_limit(8) ? 8u : 16u; }

// A strip's key has 8 bits for the column and 8 for the row, and the rows of
// several views would need more. Measured (keygen + key sort, us, keys / strips):
// 3M Gaussians at 2160p from the edge of the cloud 1106 / 699, from inside 207 /
// 161; 1M at 1080p 163 / 130, 2M inside 89 / 87, 500,000 104 / 93; 200,000 at
// 1440p 82 / 74. Smaller images have smaller rectangles, so fewer keys per
// strip, and their sorts are a few waves, where the rows' longer CTAs count:
// 300,000 at 720p (3600 tiles) 62 / 65, 120,000 at 801x603 51 / 54, 10,000 at
// 256x256 30 / 43.
bool takes_strips(uint32_t n_views, uint32_t gx, uint32_t gy) {
    return n_views == 1 && gx <= 256 && gy <= 256 && gx * gy > 4096;
}

void launch_strip_sort(const StripSort& a, cudaStream_t s) {
    const StripList strips{a.strips_alt, a.vals_alt, a.starts, a.part_first, a.gx};
    if (a.gx <= 128)
        launch_strip_scatter<7, kScatterColumns>(a, strips, a.strips, a.vals, a.strips_alt, a.vals_alt, 7, s);
    else
        launch_strip_scatter<8, kScatterColumns>(a, strips, a.strips, a.vals, a.strips_alt, a.vals_alt, 8, s);
    launch_dependent(strip_rows_kernel<kStripParts>, dim3((a.max_parts() + kStripParts - 1) / kStripParts), dim3(256),
                     0, s, strips, a.capacity, a.max_parts(), a.work, a.ctl, kStatusFatal | kStatusKeyOverflow);
    if (a.n_tiles <= 128 * a.gx)
        launch_strip_scatter<7, kScatterRows>(a, strips, nullptr, nullptr, nullptr, a.vals, 7, s);
    else
        launch_strip_scatter<8, kScatterRows>(a, strips, nullptr, nullptr, nullptr, a.vals, 8, s);
}

void launch_sort_begin(FrameCtl* ctl, uint32_t total, cudaStream_t s) {
    sort_begin_kernel<<<1, 256, 0, s>>>(ctl, total);
}

namespace {
template <typename KeyT>
bool launch_sort_t(KeyT* keys, uint32_t* vals, KeyT* keys_alt, uint32_t* vals_alt, uint32_t capacity,
                 const SortPlan& plan, uint64_t* desc, FrameCtl* ctl, uint32_t spin_limit, int num_sms,
                 cudaStream_t s) {
    const uint32_t p0 = plan.first_bit / kRadixBits;
    const uint32_t p1 = std::min(8u, sort_pass_count(plan.key_bits));
    if (p1 <= p0 || capacity == 0) return false;
    const int sms = num_sms > 0 ? num_sms : 148;
    uint32_t (*hist)[256] = plan.hist ? plan.hist : ctl->sort_hist;
    if (!plan.hist_ready) {
        const uint32_t hist_blocks = std::max(1u, std::min<uint32_t>(uint32_t(sms) * 4u, capacity / kHistChunk + 1u));
        launch_dependent(sort_histogram_kernel<KeyT>, dim3(hist_blocks), dim3(kHistThreads), 0, s,
                         static_cast<const KeyT*>(keys), capacity, p0, p1, plan.key_bits, hist, ctl);
    }
    if (plan.after_hist) cudaEventRecord(plan.after_hist, s);
    if constexpr (sizeof(KeyT) == 4) {  // counted passes: 32-bit keys (for 64-bit keys onesweep is faster)
        if (plan.counted_work) {
            if (plan.ctas_per_sm == 2)
                launch_counted_passes<2>(keys, vals, keys_alt, vals_alt, capacity, plan, plan.counted_work, ctl, s);
            else
                launch_counted_passes<3>(keys, vals, keys_alt, vals_alt, capacity, plan, plan.counted_work, ctl, s);
            const uint32_t width = counted_digit_bits(plan.key_bits);
            return ((plan.key_bits + width - 1) / width & 1u) != 0;
        }
    }
    if (plan.threads == 512)
        launch_passes<8, 512, 2>(keys, vals, keys_alt, vals_alt, capacity, p0, p1, plan, hist, desc, ctl, spin_limit,
                                 sms, s);
    else if (plan.items == 8)
        launch_passes<8, 256, 3>(keys, vals, keys_alt, vals_alt, capacity, p0, p1, plan, hist, desc, ctl, spin_limit,
                                 sms, s);
    else if (plan.items == 4)
        launch_passes<4, 256, 4>(keys, vals, keys_alt, vals_alt, capacity, p0, p1, plan, hist, desc, ctl, spin_limit,
                                 sms, s);
    else if (plan.ctas_per_sm == 3)
        launch_passes<16, 256, 3>(keys, vals, keys_alt, vals_alt, capacity, p0, p1, plan, hist, desc, ctl, spin_limit,
                                  sms, s);
    else
        launch_passes<16, 256, 2>(keys, vals, keys_alt, vals_alt, capacity, p0, p1, plan, hist, desc, ctl, spin_limit,
                                  sms, s);
    return ((p1 - p0) & 1u) != 0;
}
}  // namespace

bool launch_sort(uint64_t* keys, uint32_t* vals, uint64_t* keys_alt, uint32_t* vals_alt, uint32_t capacity,
                 const SortPlan& plan, uint64_t* desc, FrameCtl* ctl, uint32_t spin_limit, int num_sms,
                 cudaStream_t s) {
    return launch_sort_t(keys, vals, keys_alt, vals_alt, capacity, plan, desc, ctl, spin_limit, num_sms, s);
}

bool launch_sort(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, uint32_t capacity,
                 const SortPlan& plan, uint64_t* desc, FrameCtl* ctl, uint32_t spin_limit, int num_sms,
                 cudaStream_t s) {
    return launch_sort_t(keys, vals, keys_alt, vals_alt, capacity, plan, desc, ctl, spin_limit, num_sms, s);
}

}  // namespace tpd
