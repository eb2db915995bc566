// tpd_slots.cuh — key slots to owners: which item (keygen.cu) or strip
// (sort.cu) each of a partition's 4096 consecutive slots belongs to, when
// every owner has its first slot and at least one.
#pragma once
#include "tpd_counted.cuh"

namespace tpd {

// A column strip of an item's tile rectangle: its column (8 bits), first row (8
// bits) and height (9 bits).
__host__ __device__ __forceinline__ uint32_t strip_key(uint32_t col, uint32_t row, uint32_t height) {
    return col | row << 8 | height << 16;
}
__device__ __forceinline__ uint32_t strip_col(uint32_t key) { return key & 0xFFu; }
__device__ __forceinline__ uint32_t strip_row(uint32_t key) { return (key >> 8) & 0xFFu; }
__device__ __forceinline__ uint32_t strip_height(uint32_t key) { return key >> 16; }

// Called by the whole CTA of 256 threads. owner[s] = the last k < m with
// first_slot(k) <= s (first_slot(0) is taken as 0; a first slot of cnt or more
// is outside the partition): each owner marks its first slot, and a prefix
// maximum over the map gives every slot its owner. wmax: 8 words. Ends with a
// barrier.
template <typename FirstSlot>
__device__ __forceinline__ void slot_owners(uint16_t* owner, uint32_t m, uint32_t cnt, uint32_t* wmax,
                                            FirstSlot first_slot) {
    constexpr uint32_t kSlots = kCountedTile / 256;  // consecutive slots per thread
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint4* own4 = reinterpret_cast<uint4*>(owner);
    own4[2 * tid] = own4[2 * tid + 1] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (uint32_t k0 = tid; k0 < m; k0 += 1024u) {  // four loads at a time
        uint32_t slot[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) slot[u] = k0 + 256u * u < m ? first_slot(k0 + 256u * u) : cnt;
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u)  // (owner 0 has slot 0: the map's zeros)
            if (slot[u] < cnt) owner[slot[u]] = uint16_t(k0 + 256u * u);
    }
    __syncthreads();
    uint16_t o[kSlots];
    {
        const uint4 a = own4[2 * tid], b = own4[2 * tid + 1];
        *reinterpret_cast<uint4*>(o) = a;
        *reinterpret_cast<uint4*>(o + 8) = b;
    }
#pragma unroll
    for (uint32_t q = 1; q < kSlots; ++q) o[q] = max(o[q], o[q - 1]);
    uint32_t before = o[kSlots - 1];
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, before, d);
        if (lane >= d) before = max(before, x);
    }
    if (lane == 31) wmax[warp] = before;
    before = __shfl_up_sync(0xFFFFFFFFu, before, 1);
    if (lane == 0) before = 0;
    __syncthreads();
    for (uint32_t w = 0; w < warp; ++w) before = max(before, wmax[w]);
#pragma unroll
    for (uint32_t q = 0; q < kSlots; ++q) o[q] = max(o[q], uint16_t(before));
    own4[2 * tid] = *reinterpret_cast<const uint4*>(o);
    own4[2 * tid + 1] = *reinterpret_cast<const uint4*>(o + 8);
    __syncthreads();
}

}  // namespace tpd
