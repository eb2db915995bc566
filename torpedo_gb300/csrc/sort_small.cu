// sort_small.cu — the stable sort of few pairs (up to kSmallSortMax) in one
// launch: every key's final position is counted directly, against all keys.
//
// Reference: the same sorter as sort.cu's (radix-shuffle.slang:39-151 and the
// three shaders after it), which takes four dispatches per 2-bit digit
// whatever the size.
//
// A radix pass over a few thousand keys is a launch and a chain of global
// round trips (ticket, look-back, scattered stores): 9 us, four to six times
// per sort. A key's position in the stable sort is the number of keys below
// it, plus those equal to it and before it: n^2 comparisons, which the whole
// GPU makes in a few microseconds while n is small, without any exchange
// between CTAs. Bound by the integer pipe: two operations per pair of 32-bit
// keys, three for 64. 5,003 pairs of 40 bits: 12 us, 62 with the passes; the
// depth sort of 5,003 Gaussians 10 us instead of 38, of 10,000 22 instead of
// 37. The line at 12288 pairs lies where the depth sort's passes catch up
// (26 us against 37 there, 45 at 16384; pairs of 45 bits 33 against 78).
// (All radix passes in one CTA's shared memory measured no better than the
// passes over all SMs: 24 us for 5,003 pairs of 40 bits, 33 us for the depth
// sort of 10,000; one SM's shared-memory pipe bounds its scattered accesses.)
#include <type_traits>

#include "tpd_common.cuh"
#include "tpd_kernels.h"
#include "tpd_scan.cuh"

namespace tpd {
namespace {

constexpr uint32_t kThreads = 512;
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kStage = 4096;  // keys staged in shared memory at a time

// A CTA finds the positions of 32 keys (one per lane, the same for every
// warp); its warps share out the keys they are compared with, staged in
// rounds. (64 keys a CTA, or the comparisons as borrows of subtractions,
// measured slower.) KeyT: the bits that order the keys, uint32_t when 32
// suffice (a frame of one view: its depth keys' high half is zero).
// kDepth: the frame's depth sort. Culled items (low 32 bits 0xFFFFFFFF) come
// after all others and are not written; the position of a key in keys_in is
// its item. Otherwise keys and values go to (keys_out, vals_out), which must
// be other buffers than the inputs, and ctl->status is cleared.
template <typename KeyT, bool kDepth>
__global__ void __launch_bounds__(kThreads)
    small_sort_kernel(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                      uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, uint32_t n, uint64_t mask,
                      FrameCtl* ctl) {
    constexpr uint32_t kOwn = 32u;
    constexpr uint32_t kVec = 16u / sizeof(KeyT);  // keys per shared-memory load
    __shared__ __align__(16) KeyT stage[kStage];
    __shared__ uint32_t below[kOwn];
    pdl_wait();
    if (kDepth) pdl_trigger();  // the frame's next kernel may be scheduled (it waits for this grid)
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t i0 = blockIdx.x * kOwn;
    auto order_of = [&](uint64_t key) {  // a culled item of any view is above all others
        return kDepth && uint32_t(key) == 0xFFFFFFFFu ? KeyT(~KeyT(0)) : KeyT(key & mask);
    };
    const uint32_t i = i0 + lane;
    const KeyT own = i < n ? order_of(keys_in[i]) : KeyT(0);
    uint32_t cnt = 0;
    if (tid < kOwn) below[tid] = 0;
    for (uint32_t s0 = 0; s0 < n; s0 += kStage) {
        const uint32_t m = min(kStage, n - s0), whole = (m + kVec * kWarps - 1) / (kVec * kWarps) * (kVec * kWarps);
        __syncthreads();  // the last round's keys are read
        // (slots past the keys hold the largest: never below another)
        for (uint32_t j = tid; j < whole; j += kThreads)
            stage[j] = j < m ? order_of(keys_in[s0 + j]) : KeyT(~KeyT(0));
        __syncthreads();
        const uint32_t per = whole / kWarps, j0 = warp * per, j1 = j0 + per;  // this warp's keys, whole vectors
        // keys before all of this CTA's count when equal too, those after none do
        auto sweep = [&](uint32_t from, uint32_t to, auto le) {
#pragma unroll 4
            for (uint32_t j = from; j < to; j += kVec) {
                KeyT k[kVec];
                *reinterpret_cast<uint4*>(k) = *reinterpret_cast<const uint4*>(stage + j);
#pragma unroll
                for (uint32_t q = 0; q < kVec; ++q) {
                    if constexpr (decltype(le)::value) cnt += k[q] <= own ? 1u : 0u;
                    else cnt += k[q] < own ? 1u : 0u;
                }
            }
        };
        // [j0, a): before the CTA's own keys; [a, b): among them; [b, j1): after
        const uint32_t lo = i0 > s0 ? min(i0 - s0, whole) : 0u, hi = i0 + kOwn > s0 ? min(i0 + kOwn - s0, whole) : 0u;
        const uint32_t a = min(max(lo / kVec * kVec, j0), j1);
        const uint32_t b = min(max((hi + kVec - 1) / kVec * kVec, a), j1);
        sweep(j0, a, std::true_type{});
        for (uint32_t j = a; j < b; ++j) {
            const KeyT k = stage[j];
            cnt += k < own || (k == own && s0 + j < i) ? 1u : 0u;
        }
        sweep(b, j1, std::false_type{});
    }
    atomicAdd(&below[lane], cnt);
    __syncthreads();
    if (tid < kOwn && i0 + tid < n) {
        const uint32_t pos = below[tid];  // < n: a permutation
        const uint64_t key = keys_in[i0 + tid];
        if constexpr (kDepth) {
            if (uint32_t(key) != 0xFFFFFFFFu) vals_out[pos] = i0 + tid;
        } else {
            keys_out[pos] = key;
            vals_out[pos] = vals_in[i0 + tid];
        }
    }
    if (!kDepth && blockIdx.x == 0 && tid == 0) ctl->status = 0;
}

template <typename KeyT, bool kDepth>
void launch_t(const uint64_t* keys, const uint32_t* vals, uint64_t* keys_out, uint32_t* vals_out, uint32_t n,
              uint64_t mask, FrameCtl* ctl, cudaStream_t s) {
    launch_dependent(small_sort_kernel<KeyT, kDepth>, dim3((n + 31) / 32), dim3(kThreads), 0, s, keys, vals, keys_out,
                     vals_out, n, mask, ctl);
}

}  // namespace

void launch_small_depth_sort(const uint64_t* keys, uint32_t* items_out, uint32_t n, uint32_t key_bits, FrameCtl* ctl,
                             cudaStream_t s) {
    if (n == 0) return;
    if (key_bits <= 32)
        launch_t<uint32_t, true>(keys, nullptr, nullptr, items_out, n, 0xFFFFFFFFull, ctl, s);
    else
        launch_t<uint64_t, true>(keys, nullptr, nullptr, items_out, n, ~0ull, ctl, s);
}

void launch_small_sort(const uint64_t* keys, const uint32_t* vals, uint64_t* keys_out, uint32_t* vals_out, uint32_t n,
                       uint32_t key_bits, FrameCtl* ctl, cudaStream_t s) {
    if (n == 0) return;
    const uint64_t mask = key_bits >= 64 ? ~0ull : (1ull << key_bits) - 1ull;
    if (key_bits <= 32)
        launch_t<uint32_t, false>(keys, vals, keys_out, vals_out, n, mask, ctl, s);
    else
        launch_t<uint64_t, false>(keys, vals, keys_out, vals_out, n, mask, ctl, s);
}

}  // namespace tpd
