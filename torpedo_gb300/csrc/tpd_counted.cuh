// tpd_counted.cuh — the work area of a counted radix pass (sort.cu) and the
// scans that turn per-partition digit counts into global offsets, shared by
// the kernels that count a pass: partition_count_kernel (sort.cu) and
// expand_keys_kernel (keygen.cu), which counts the first pass's digits while
// it writes the keys.
#pragma once
#include "tpd_common.cuh"
#include "tpd_scan.cuh"

namespace tpd {

constexpr uint32_t kCountedTile = 4096;  // keys per partition
constexpr uint32_t kChunkParts = 32;     // partitions per chunk, and chunks per group

// Layout of a counted pass's work area (u32 words) for digits below kDig (256
// or 512) and at most P partitions, C = ceil(P / 32) chunks and G = ceil(C /
// 32) groups:
// [0, kDig P) rows of digit counts, then offsets within their chunk;
// kDig C words of chunk totals, then offsets within their group;
// kDig G words of group totals, then the groups' global offsets;
// at words 512 (P + C + G), whatever kDig: arrival counts, C (partitions of a
// chunk), G (chunks of a group), 1 (groups). Only these have to be zero at rest.
__host__ __device__ inline size_t counted_div(size_t n) { return (n + kChunkParts - 1) / kChunkParts; }
template <uint32_t kDig>
struct CountedWork {
    uint32_t *rows, *chunks, *groups, *chunk_arrivals, *group_arrivals, *done;
    __host__ __device__ CountedWork(uint32_t* work, uint32_t max_parts) {
        const size_t c = counted_div(max_parts), g = counted_div(c);
        rows = work;
        chunks = rows + kDig * size_t(max_parts);
        groups = chunks + kDig * c;
        chunk_arrivals = work + 512 * (size_t(max_parts) + c + g);
        group_arrivals = chunk_arrivals + c;
        done = group_arrivals + g;
    }
};
__host__ __device__ inline size_t counted_work_words(uint32_t parts) {
    const size_t c = counted_div(parts), g = counted_div(c);
    return 512 * (size_t(parts) + c + g) + c + g + 1;
}

// A thread's digits of a row: with 256 threads, digits kPer tid .. + kPer - 1.
template <uint32_t kPer>
struct RowDigits {
    uint32_t v[kPer];
};
template <uint32_t kPer>
__device__ __forceinline__ RowDigits<kPer> load_row(const uint32_t* rows, size_t row, uint32_t tid) {
    RowDigits<kPer> r;
    if constexpr (kPer == 1) {
        r.v[0] = __ldcg(rows + row * 256 + tid);
    } else {
        const uint2 x = __ldcg(reinterpret_cast<const uint2*>(rows + row * 512) + tid);
        r.v[0] = x.x;
        r.v[1] = x.y;
    }
    return r;
}
template <uint32_t kPer>
__device__ __forceinline__ void store_row(uint32_t* rows, size_t row, uint32_t tid, const RowDigits<kPer>& r) {
    if constexpr (kPer == 1)
        rows[row * 256 + tid] = r.v[0];
    else
        reinterpret_cast<uint2*>(rows + row * 512)[tid] = make_uint2(r.v[0], r.v[1]);
}

// Block-wide exclusive scan of one value per thread (kWarps warps); returns the exclusive prefix.
template <uint32_t kWarps>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* wsum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t incl = warp_inclusive_scan(v);
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t base = 0;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w)
        if (w < warp) base += wsum[w];
    __syncthreads();
    return base + incl - v;
}

// Exclusive prefix of each digit's total over all digits (thread = kPer digits).
template <uint32_t kPer>
__device__ __forceinline__ RowDigits<kPer> scan_digits(const RowDigits<kPer>& total, uint32_t* wsum) {
    RowDigits<kPer> r;
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t p = 0; p < kPer; ++p) {
        r.v[p] = sum;
        sum += total.v[p];
    }
    const uint32_t before = block_exclusive_scan<8>(sum, wsum);
#pragma unroll
    for (uint32_t p = 0; p < kPer; ++p) r.v[p] += before;
    return r;
}

// Rows [first, first + size) (size <= 32) -> exclusive prefixes within them,
// in place, and their total per digit into row total_row of totals (batches of
// rows are loaded together, then scanned).
template <uint32_t kPer>
__device__ __forceinline__ void scan_rows(uint32_t* rows, size_t first, uint32_t size, uint32_t* totals,
                                          size_t total_row, uint32_t tid) {
    constexpr uint32_t kBatch = kChunkParts / kPer;
    RowDigits<kPer> run = {};
    for (uint32_t q0 = 0; q0 < size; q0 += kBatch) {
        RowDigits<kPer> c[kBatch];
#pragma unroll
        for (uint32_t q = 0; q < kBatch; ++q)
            if (q0 + q < size) c[q] = load_row<kPer>(rows, first + q0 + q, tid);
#pragma unroll
        for (uint32_t q = 0; q < kBatch; ++q)
            if (q0 + q < size) {
                store_row<kPer>(rows, first + q0 + q, tid, run);
#pragma unroll
                for (uint32_t p = 0; p < kPer; ++p) run.v[p] += c[q].v[p];
            }
    }
    store_row<kPer>(totals, total_row, tid, run);
}

// Whether the calling CTA is the last of `expected` to arrive at *count (which
// the last arriver resets). The CTA's global writes before the call are
// visible to the last arriver after it: the barrier orders every thread's
// writes before thread 0's fence, which is cumulative.
__device__ __forceinline__ bool last_to_arrive(uint32_t* count, uint32_t expected, bool& s_last) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(count, 1u) == expected - 1u;
        if (s_last) {
            *count = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return s_last;
}

// The end of a counting CTA of 256 threads: stores the
// partition's digit counts as its row; the last CTA of a chunk of 32
// partitions scans the chunk's rows, the last chunk of a group of 32 scans the
// group's chunk totals, and the last group scans the group totals, starting
// each digit where the smaller digits' keys end. Nobody waits. Three levels
// keep the serial end short: 80M keys are 19,500 partitions but only 20
// groups. A sort of one chunk (up to 131072 keys) leaves its rows as counts,
// which counted_offset adds up itself: for the smallest frames the arrivals'
// round trips were half of the counting kernel's time (10,000 Gaussians at
// 256x256: 5.2 us of the frame with them, 2.4 without).
// counted_arrive is the same for a CTA that has stored the rows of kParts
// consecutive partitions, from a multiple of kParts, the first being part.
template <uint32_t kDig, uint32_t kParts = 1>
__device__ __forceinline__ void counted_arrive(const CountedWork<kDig>& W, uint32_t nparts, uint32_t part,
                                               uint32_t* wsum, bool& s_last) {
    constexpr uint32_t kPer = kDig / 256;
    const uint32_t tid = threadIdx.x;
    if (nparts <= kChunkParts) return;
    const uint32_t chunk = part / kChunkParts, nchunks = uint32_t(counted_div(nparts));
    const uint32_t first = chunk * kChunkParts, csize = min(kChunkParts, nparts - first);
    if (!last_to_arrive(W.chunk_arrivals + chunk, (csize + kParts - 1) / kParts, s_last)) return;
    scan_rows<kPer>(W.rows, first, csize, W.chunks, chunk, tid);
    const uint32_t group = chunk / kChunkParts, ngroups = uint32_t(counted_div(nchunks));
    const uint32_t gfirst = group * kChunkParts, gsize = min(kChunkParts, nchunks - gfirst);
    if (!last_to_arrive(W.group_arrivals + group, gsize, s_last)) return;
    scan_rows<kPer>(W.chunks, gfirst, gsize, W.groups, group, tid);
    // (a single group has arrived with its last chunk)
    if (ngroups > 1 && !last_to_arrive(W.done, ngroups, s_last)) return;
    RowDigits<kPer> total = {};
    for (uint32_t g = 0; g < ngroups; ++g) {
        const RowDigits<kPer> c = load_row<kPer>(W.groups, g, tid);
#pragma unroll
        for (uint32_t p = 0; p < kPer; ++p) total.v[p] += c.v[p];
    }
    RowDigits<kPer> run = scan_digits<kPer>(total, wsum);
    for (uint32_t g = 0; g < ngroups; ++g) {
        const RowDigits<kPer> c = load_row<kPer>(W.groups, g, tid);
        store_row<kPer>(W.groups, g, tid, run);
#pragma unroll
        for (uint32_t p = 0; p < kPer; ++p) run.v[p] += c.v[p];
    }
}

template <uint32_t kDig>
__device__ __forceinline__ void counted_finish(const CountedWork<kDig>& W, uint32_t nparts, uint32_t part,
                                               const RowDigits<kDig / 256>& count, uint32_t* wsum, bool& s_last) {
    store_row<kDig / 256>(W.rows, part, threadIdx.x, count);
    counted_arrive<kDig>(W, nparts, part, wsum, s_last);
}

// The global positions of the partition's first keys of the thread's digits
// (called by the whole CTA of 256 threads, after counted_finish's grid).
template <uint32_t kDig>
__device__ __forceinline__ RowDigits<kDig / 256> counted_offset(const CountedWork<kDig>& W, uint32_t nparts,
                                                                uint32_t part, uint32_t* wsum) {
    constexpr uint32_t kPer = kDig / 256;
    const uint32_t tid = threadIdx.x;
    if (nparts <= kChunkParts) {
        RowDigits<kPer> before = {}, total = {};
#pragma unroll 8
        for (uint32_t q = 0; q < nparts; ++q) {
            const RowDigits<kPer> c = load_row<kPer>(W.rows, q, tid);
#pragma unroll
            for (uint32_t p = 0; p < kPer; ++p) {
                before.v[p] += q < part ? c.v[p] : 0u;
                total.v[p] += c.v[p];
            }
        }
        RowDigits<kPer> r = scan_digits<kPer>(total, wsum);
#pragma unroll
        for (uint32_t p = 0; p < kPer; ++p) r.v[p] += before.v[p];
        return r;
    }
    RowDigits<kPer> r = load_row<kPer>(W.groups, part / (kChunkParts * kChunkParts), tid);
    const RowDigits<kPer> c = load_row<kPer>(W.chunks, part / kChunkParts, tid), o = load_row<kPer>(W.rows, part, tid);
#pragma unroll
    for (uint32_t p = 0; p < kPer; ++p) r.v[p] += c.v[p] + o.v[p];
    return r;
}

}  // namespace tpd
