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

// Layout of a counted pass's work area (u32 words), for at most P partitions,
// C = ceil(P / 32) chunks and G = ceil(C / 32) groups:
// [0, 256 P) rows of digit counts, then offsets within their chunk;
// 256 C words of chunk totals, then offsets within their group;
// 256 G words of group totals, then the groups' global offsets;
// arrival counts: C (partitions of a chunk), G (chunks of a group), 1 (groups).
// Only the arrival counts have to be zero at rest.
__host__ __device__ inline size_t counted_div(size_t n) { return (n + kChunkParts - 1) / kChunkParts; }
struct CountedWork {
    uint32_t *rows, *chunks, *groups, *chunk_arrivals, *group_arrivals, *done;
    __host__ __device__ CountedWork(uint32_t* work, uint32_t max_parts) {
        const size_t c = counted_div(max_parts), g = counted_div(c);
        rows = work;
        chunks = rows + 256 * size_t(max_parts);
        groups = chunks + 256 * c;
        chunk_arrivals = groups + 256 * g;
        group_arrivals = chunk_arrivals + c;
        done = group_arrivals + g;
    }
};
__host__ __device__ inline size_t counted_work_words(uint32_t parts) {
    const size_t c = counted_div(parts), g = counted_div(c);
    return 256 * (size_t(parts) + c + g) + c + g + 1;
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

// Rows [first, first + size) (size <= 32) -> exclusive prefixes within them,
// in place, and their total per digit into *total_row (thread = digit; the
// rows are loaded together, then scanned).
__device__ __forceinline__ void scan_rows(uint32_t* rows, size_t first, uint32_t size, uint32_t* total_row,
                                          uint32_t tid) {
    uint32_t c[kChunkParts];
#pragma unroll
    for (uint32_t q = 0; q < kChunkParts; ++q) c[q] = q < size ? __ldcg(rows + (first + q) * 256 + tid) : 0u;
    uint32_t run = 0;
#pragma unroll
    for (uint32_t q = 0; q < kChunkParts; ++q) {
        if (q < size) rows[(first + q) * 256 + tid] = run;
        run += c[q];
    }
    total_row[tid] = run;
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

// The end of a counting CTA of 256 threads (thread = digit): stores the
// partition's digit counts as its row; the last CTA of a chunk of 32
// partitions scans the chunk's rows, the last chunk of a group of 32 scans the
// group's chunk totals, and the last group scans the group totals, starting
// each digit where the smaller digits' keys end. Nobody waits. Three levels
// keep the serial end short: 80M keys are 19,500 partitions but only 20
// groups. A sort of one chunk (up to 131072 keys) leaves its rows as counts,
// which counted_offset adds up itself: for the smallest frames the arrivals'
// round trips were half of the counting kernel's time (10,000 Gaussians at
// 256x256: 5.2 us of the frame with them, 2.4 without).
__device__ __forceinline__ void counted_finish(const CountedWork& W, uint32_t nparts, uint32_t part, uint32_t count,
                                               uint32_t* wsum, bool& s_last) {
    const uint32_t tid = threadIdx.x;
    W.rows[size_t(part) * 256 + tid] = count;
    if (nparts <= kChunkParts) return;
    const uint32_t chunk = part / kChunkParts, nchunks = uint32_t(counted_div(nparts));
    const uint32_t first = chunk * kChunkParts, csize = min(kChunkParts, nparts - first);
    if (!last_to_arrive(W.chunk_arrivals + chunk, csize, s_last)) return;
    scan_rows(W.rows, first, csize, W.chunks + size_t(chunk) * 256, tid);
    const uint32_t group = chunk / kChunkParts, ngroups = uint32_t(counted_div(nchunks));
    const uint32_t gfirst = group * kChunkParts, gsize = min(kChunkParts, nchunks - gfirst);
    if (!last_to_arrive(W.group_arrivals + group, gsize, s_last)) return;
    scan_rows(W.chunks, gfirst, gsize, W.groups + size_t(group) * 256, tid);
    // (a single group has arrived with its last chunk)
    if (ngroups > 1 && !last_to_arrive(W.done, ngroups, s_last)) return;
    uint32_t total = 0;
    for (uint32_t g = 0; g < ngroups; ++g) total += __ldcg(W.groups + size_t(g) * 256 + tid);
    uint32_t run = block_exclusive_scan<8>(total, wsum);
    for (uint32_t g = 0; g < ngroups; ++g) {
        const uint32_t c = __ldcg(W.groups + size_t(g) * 256 + tid);
        W.groups[size_t(g) * 256 + tid] = run;
        run += c;
    }
}

// The global position of the partition's first key of a digit (thread =
// digit, called by the whole CTA of 256 threads, after counted_finish's grid).
__device__ __forceinline__ uint32_t counted_offset(const CountedWork& W, uint32_t nparts, uint32_t part,
                                                   uint32_t* wsum) {
    const uint32_t tid = threadIdx.x;
    if (nparts <= kChunkParts) {
        uint32_t before = 0, total = 0;
#pragma unroll 8
        for (uint32_t q = 0; q < nparts; ++q) {
            const uint32_t c = __ldcg(W.rows + size_t(q) * 256 + tid);
            before += q < part ? c : 0u;
            total += c;
        }
        return before + block_exclusive_scan<8>(total, wsum);
    }
    return __ldcg(W.groups + size_t(part / (kChunkParts * kChunkParts)) * 256 + tid) +
           __ldcg(W.chunks + size_t(part / kChunkParts) * 256 + tid) + __ldcg(W.rows + size_t(part) * 256 + tid);
}

}  // namespace tpd
