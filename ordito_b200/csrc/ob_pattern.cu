// a1: the "cotmatrix" mesh operator pattern, built deterministically from sorted keys.
//
// Follows ordito/laplacian.py:1212-1299 (directed build), ordito/kernels/laplacian.py:707-748
// (store_operator_keys) and ordito/array.py:1688-1807 (csr_from_keys). Keys are
// row * V + col (uint64), sorted stably: equal keys keep the producer's slot order, so an entry's
// contributors (its run of equal sorted keys) come out in face order. The sort is by row buckets,
// straight from the faces: a corner counts its (at most two) keys into its vertex's row with one
// atomic and later scatters them into the row's bucket with another, as (col, slot), each bucket is
// sorted by (col, slot) -- the order a stable sort by key gives, whatever order the scatter filled it
// in -- and its distinct columns counted; their scan is the row offsets, and one last pass writes the
// keys, payloads, columns and run starts. The out-of-range (sentinel) keys follow in slot order. No
// value is ever accumulated atomically: each entry's value is formed later from its run.
//
// What bounds it is traffic: the outputs (~16 bytes a key) and three trips of the buckets (8 bytes a
// key), the faces twice, and two atomics a corner. The unsorted keys are never stored, and no scan or
// pass runs over them: the form that stored them, with a general segmented sort and scans over
// every slot, took 0.50 ms on a 655 k-vertex torus (14 launches).
#include <cub/device/device_scan.cuh>

#include <algorithm>

#include "ob_internal.cuh"

namespace ob {
namespace {

constexpr int kThreads = 256;

// Slot 6 f + 2 e holds the key (i, j) of the edge opposite corner e (i = corner e + 1, j = corner
// e + 2), slot 6 f + 2 e + 1 its reverse, payload 3 f + e; slot 6 F + v the diagonal of a referenced
// vertex v (payload -1). A corner's own row so takes two of its face's slots: corner c's keys
// (c, c - 1) and (c, c + 1).
__device__ __forceinline__ int corner_column(const int* face, int c, int which) {
    return face[which == 0 ? (c + 2) % 3 : (c + 1) % 3];
}
__device__ __forceinline__ int corner_slot(int c, int which) {
    // (c, c - 1) is the reverse of the edge opposite c + 1, (c, c + 1) the edge opposite c - 1.
    return which == 0 ? 2 * ((c + 1) % 3) + 1 : 2 * ((c + 2) % 3);
}

// The payload of slot i: the corner 3 f + e of an edge slot 6 f + 2 e (+ 1), -1 for a tail slot.
__device__ __forceinline__ int slot_payload(long long i, long long tail) { return i < tail ? (int)(i / 2) : -1; }

__device__ __forceinline__ bool inside(int v, int n) { return v >= 0 && v < n; }

// Per face: its corners' in-range keys counted into their rows (integer atomics: the counts, not
// their order, are used), the rows flagged as referenced, and its sentinel slots counted.
__global__ void corner_counts(const int* __restrict__ faces, int n_faces, int n, int* __restrict__ counts,
                              int* __restrict__ referenced, int* __restrict__ sentinels) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f > n_faces) return;
    if (f == n_faces) {
        sentinels[f] = 0;  // the scan's total
        return;
    }
    const int c[3] = {faces[3 * f], faces[3 * f + 1], faces[3 * f + 2]};
    int outside = 6;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        if (!inside(c[e], n)) continue;
        const int keys = (int)inside(c[(e + 1) % 3], n) + (int)inside(c[(e + 2) % 3], n);
        outside -= keys;
        referenced[c[e]] = 1;
        if (keys) atomicAdd(&counts[c[e]], keys);
    }
    sentinels[f] = outside;
}

// Per row: its keys (the diagonal's among them) in the low half, whether its tail slot is a
// sentinel (an unreferenced vertex: an empty row) in the high half; the scan of both is one.
__global__ void row_totals(const int* __restrict__ counts, const int* __restrict__ referenced, int n,
                           unsigned long long* __restrict__ totals) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v > n) return;
    totals[v] = v == n            ? 0ULL
                : referenced[v]   ? (unsigned long long)(counts[v] + 1)
                                  : 1ULL << 32;
}

__device__ __forceinline__ int row_begin(const unsigned long long* starts, int row) {
    return (int)(starts[row] & 0xffffffffULL);
}

// Each corner's keys into its row's bucket as (col << 32 | slot), the place after the row's first
// (the diagonal's) taken by counting the row's counter down; each sentinel edge slot to its place
// after every in-range key.
__global__ void scatter_corners(const int* __restrict__ faces, int n_faces, int n,
                                const unsigned long long* __restrict__ starts, int* __restrict__ counts,
                                const int* __restrict__ sentinel_before, unsigned long long* __restrict__ bucket,
                                unsigned long long* __restrict__ keys_out, int* __restrict__ order_out) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_faces) return;
    const int c[3] = {faces[3 * f], faces[3 * f + 1], faces[3 * f + 2]};
    const int before = sentinel_before[f];
    const bool whole = before == sentinel_before[f + 1];
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        if (!inside(c[e], n)) continue;
        const int keys = (int)inside(c[(e + 1) % 3], n) + (int)inside(c[(e + 2) % 3], n);
        if (keys == 0) continue;
        int at = row_begin(starts, c[e]) + 1 + atomicSub(&counts[c[e]], keys) - keys;
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            const int col = corner_column(c, e, which);
            if (!inside(col, n)) continue;
            bucket[at++] = ((unsigned long long)col << 32) | (unsigned long long)(6LL * f + corner_slot(e, which));
        }
    }
    if (whole) return;
    const unsigned long long sentinel = (unsigned long long)n * (unsigned long long)n;
    long long at = (long long)row_begin(starts, n) + before;
    for (int slot = 0; slot < 6; ++slot) {
        const int i = c[(slot / 2 + 1) % 3], j = c[(slot / 2 + 2) % 3];
        if (inside(i, n) && inside(j, n)) continue;
        keys_out[at] = sentinel;
        order_out[at++] = slot_payload(6LL * f + slot, 6LL * n_faces);
    }
}

// Each row's tail slot: the diagonal's key first in the row's bucket, or a sentinel in its place.
__global__ void place_tail(const unsigned long long* __restrict__ starts, int n, int n_faces,
                           const int* __restrict__ referenced, const int* __restrict__ sentinel_before,
                           unsigned long long* __restrict__ bucket, unsigned long long* __restrict__ keys_out,
                           int* __restrict__ order_out) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    if (referenced[v]) {
        bucket[row_begin(starts, v)] = ((unsigned long long)v << 32) | (unsigned long long)(6LL * n_faces + v);
        return;
    }
    const long long at = (long long)row_begin(starts, n) + sentinel_before[n_faces] + (long long)(starts[v] >> 32);
    keys_out[at] = (unsigned long long)n * (unsigned long long)n;
    order_out[at] = -1;
}

// A CTA sorts the buckets of kSortRows consecutive rows, which are consecutive in memory: staged in
// shared memory with coalesced loads, a thread insertion-sorts its row there (13 keys on a mesh's
// usual vertex; a warp a row spends five times the instructions), counts its distinct columns, and
// the CTA writes the sorted segment back. Rows past kShortRow, and segments past the shared memory,
// are left to sort_long_rows by a list.
constexpr int kSortRows = 128;
constexpr int kSortKeys = 3072;  // 24 KB: 24 keys a row on average
constexpr int kShortRow = 96;

__global__ void __launch_bounds__(kSortRows) sort_rows(const unsigned long long* __restrict__ starts, int n,
                                                       unsigned long long* __restrict__ bucket,
                                                       int* __restrict__ distinct, int* __restrict__ long_rows,
                                                       int* __restrict__ n_long) {
    __shared__ unsigned long long keys[kSortKeys];
    const int first = blockIdx.x * kSortRows, row = first + threadIdx.x;
    const int begin = row_begin(starts, first), end = row_begin(starts, min(n, first + kSortRows));
    const bool staged = end - begin <= kSortKeys;
    if (staged) {
        for (int p = begin + threadIdx.x; p < end; p += kSortRows) keys[p - begin] = bucket[p];
        __syncthreads();
    }
    if (row < n) {
        const int from = row_begin(starts, row), count = row_begin(starts, row + 1) - from;
        if (!staged || count > kShortRow) {
            if (count > 1) long_rows[atomicAdd(n_long, 1)] = row;
            else distinct[row] = count;
        } else {
            unsigned long long* mine = keys + (from - begin);
            int columns = count > 0;
            for (int i = 1; i < count; ++i) {
                const unsigned long long key = mine[i];
                int j = i;
                for (; j > 0 && mine[j - 1] > key; --j) mine[j] = mine[j - 1];
                mine[j] = key;
            }
            for (int i = 1; i < count; ++i) columns += (mine[i] >> 32) != (mine[i - 1] >> 32);
            distinct[row] = columns;
        }
    }
    if (!staged) return;
    __syncthreads();
    for (int p = begin + threadIdx.x; p < end; p += kSortRows) bucket[p] = keys[p - begin];
}

// The listed rows, a CTA a row: runs of kRun keys sorted by rank in shared memory, then merged
// pairwise (a key's place is its own plus its rank in the other run, found by bisection), between
// the buckets and a second buffer of their size.
constexpr int kLongThreads = 1024;
constexpr int kRun = 1024;

__global__ void __launch_bounds__(kLongThreads) sort_long_rows(const unsigned long long* __restrict__ starts,
                                                               const int* __restrict__ long_rows,
                                                               const int* __restrict__ n_long,
                                                               unsigned long long* bucket, unsigned long long* spare,
                                                               int* __restrict__ distinct) {
    __shared__ unsigned long long run[kRun];
    __shared__ int scratch[32];
    const int listed = *n_long;
    for (int item = blockIdx.x; item < listed; item += gridDim.x) {
        const int row = long_rows[item];
        const int from = row_begin(starts, row), count = row_begin(starts, row + 1) - from;
        unsigned long long *source = bucket + from, *target = spare + from;
        for (int r = 0; r < count; r += kRun) {
            const int size = min(kRun, count - r);
            __syncthreads();
            if ((int)threadIdx.x < size) run[threadIdx.x] = source[r + threadIdx.x];
            __syncthreads();
            if ((int)threadIdx.x < size) {
                const unsigned long long key = run[threadIdx.x];
                int rank = 0;
                for (int i = 0; i < size; ++i) rank += run[i] < key;  // the keys differ by their slots
                source[r + rank] = key;
            }
        }
        __syncthreads();
        for (long long width = kRun; width < count; width *= 2) {
            for (int i = threadIdx.x; i < count; i += kLongThreads) {
                const unsigned long long key = source[i];
                const long long pair = i / (2 * width) * (2 * width), middle = min((long long)count, pair + width);
                const bool left = i < middle;
                long long lo = left ? middle : pair, hi = left ? min((long long)count, pair + 2 * width) : middle;
                const long long other = lo;
                while (lo < hi) {
                    const long long m = (lo + hi) / 2;
                    if (source[m] < key) lo = m + 1;
                    else hi = m;
                }
                target[(left ? i : pair + i - middle) + (lo - other)] = key;
            }
            __syncthreads();
            unsigned long long* swap = source;
            source = target;
            target = swap;
        }
        int columns = 0;
        for (int i = threadIdx.x; i < count; i += kLongThreads) {
            const unsigned long long key = source[i];
            columns += i == 0 || (key >> 32) != (source[i - 1] >> 32);
        }
        const int total = block_sum(columns, scratch);
        if (threadIdx.x == 0) distinct[row] = total;
        __syncthreads();
        if (source != bucket + from)
            for (int i = threadIdx.x; i < count; i += kLongThreads) bucket[from + i] = source[i];
        __syncthreads();
    }
}

// The sorted buckets out, a CTA kSortRows rows: each position's key and payload, and each run of
// one column as one entry (the entries of consecutive rows are consecutive: offsets of the CTA's
// first row plus the runs counted so far).
constexpr int kWriteThreads = 256;

__global__ void __launch_bounds__(kWriteThreads) write_rows(const unsigned long long* __restrict__ bucket,
                                                            const unsigned long long* __restrict__ starts,
                                                            const int* __restrict__ offsets, int n, long long tail,
                                                            unsigned long long* __restrict__ keys_out,
                                                            int* __restrict__ order_out, int* __restrict__ columns,
                                                            int* __restrict__ run_start) {
    __shared__ int row_start[kSortRows + 1];
    __shared__ int warp_runs[kWriteThreads / 32];
    const int first = blockIdx.x * kSortRows, rows = min(kSortRows, n - first);
    for (int i = threadIdx.x; i <= rows; i += kWriteThreads) row_start[i] = row_begin(starts, first + i);
    __syncthreads();
    const int begin = row_start[0], end = row_start[rows];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int entry = offsets[first];
    for (int base = begin; base < end; base += kWriteThreads) {
        const int p = base + threadIdx.x;
        bool opens = false;
        int col = 0;
        if (p < end) {
            // The row holding p: row_start[lo] <= p < row_start[lo + 1] (empty rows hold none).
            int lo = 0, hi = rows - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (row_start[mid] <= p) lo = mid;
                else hi = mid - 1;
            }
            const unsigned long long v = bucket[p];
            col = (int)(v >> 32);
            opens = p == row_start[lo] || (int)(bucket[p - 1] >> 32) != col;
            keys_out[p] = (unsigned long long)(first + lo) * (unsigned long long)n + (unsigned long long)col;
            order_out[p] = slot_payload((long long)(v & 0xffffffffULL), tail);
        }
        const unsigned runs = __ballot_sync(0xffffffffu, opens);
        if (lane == 0) warp_runs[warp] = __popc(runs);
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kWriteThreads / 32; ++w) {
            before += w < warp ? warp_runs[w] : 0;
            all += warp_runs[w];
        }
        if (opens) {
            const int at = entry + before + __popc(runs & ((1u << lane) - 1u));
            columns[at] = col;
            run_start[at] = p;
        }
        entry += all;
        __syncthreads();
    }
}

struct PatternLayout {
    size_t bucket = 0, spare = 0, counts = 0, totals = 0, starts = 0, sentinels = 0, distinct = 0, long_rows = 0,
           scan_temp = 0, total = 0;
};

int pattern_layout(int n, int n_faces, PatternLayout* out) {
    const long long count = 6LL * n_faces + n;
    PatternLayout l;
    size_t rows = 0, face = 0, entries = 0;
    if (count > 0) {
        OB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, rows, (const unsigned long long*)nullptr,
                                              (unsigned long long*)nullptr, n + 1));
        OB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, face, (const int*)nullptr, (int*)nullptr, n_faces + 1));
        OB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, entries, (const int*)nullptr, (int*)nullptr, n + 1));
    }
    l.bucket = 0;
    l.spare = align_up(l.bucket + 8 * (size_t)count);
    // Zeroed at the start of a build, in one piece: the rows' counters, their flags, the list's length.
    l.counts = align_up(l.spare + 8 * (size_t)count);
    l.totals = align_up(l.counts + 4 * (2 * (size_t)n + 1));
    l.starts = align_up(l.totals + 8 * ((size_t)n + 1));
    l.sentinels = align_up(l.starts + 8 * ((size_t)n + 1));
    l.distinct = align_up(l.sentinels + 4 * ((size_t)n_faces + 1));
    l.long_rows = align_up(l.distinct + 4 * ((size_t)n + 1));
    l.scan_temp = align_up(l.long_rows + 4 * (size_t)n);
    l.total = align_up(l.scan_temp + std::max(rows, std::max(face, entries))) + 256;
    *out = l;
    return OB_OK;
}

}  // namespace
}  // namespace ob

using namespace ob;

extern "C" {

int ob_pattern_workspace(int n_vertices, int n_faces, size_t* bytes) {
    OB_REQUIRE(bytes != nullptr, "ob_pattern_workspace: null output");
    OB_REQUIRE(n_vertices >= 0 && n_faces >= 0, "ob_pattern_workspace: negative size");
    OB_REQUIRE(6LL * n_faces + n_vertices < (1LL << 31),
               "ob_pattern_workspace: 6 F + V = %lld keys exceed int32 indexing",
               6LL * n_faces + n_vertices);
    OB_REQUIRE((long long)n_vertices * n_vertices < (1LL << 62), "ob_pattern_workspace: V too large");
    PatternLayout l;
    int st = pattern_layout(n_vertices, n_faces, &l);
    if (st) return st;
    *bytes = l.total;
    return OB_OK;
}

int ob_pattern_build(const int32_t* faces, int n_faces, int n_vertices, int32_t* offsets,
                     int32_t* columns, int32_t* run_start, uint64_t* keys, int32_t* order,
                     void* workspace, size_t workspace_bytes, ob_stream_t stream_) {
    cudaStream_t stream = as_stream(stream_);
    OB_REQUIRE(n_vertices >= 0 && n_faces >= 0, "ob_pattern_build: negative size");
    OB_REQUIRE(offsets != nullptr, "ob_pattern_build: null offsets");
    const long long count = 6LL * n_faces + n_vertices;
    PatternLayout l;
    int st = pattern_layout(n_vertices, n_faces, &l);
    if (st) return st;
    if (count == 0) {
        OB_CUDA(cudaMemsetAsync(offsets, 0, sizeof(int) * (size_t)(n_vertices + 1), stream));
        return OB_OK;
    }
    OB_REQUIRE(faces != nullptr || n_faces == 0, "ob_pattern_build: null faces");
    OB_REQUIRE(columns && run_start && keys && order, "ob_pattern_build: null output");
    OB_REQUIRE(workspace != nullptr && workspace_bytes >= l.total,
               "ob_pattern_build: workspace of %zu bytes, %zu needed", workspace_bytes, l.total);
    char* ws = reinterpret_cast<char*>(align_up(reinterpret_cast<size_t>(workspace)));
    auto* bucket = reinterpret_cast<unsigned long long*>(ws + l.bucket);
    auto* spare = reinterpret_cast<unsigned long long*>(ws + l.spare);
    auto* counts = reinterpret_cast<int*>(ws + l.counts);
    int *referenced = counts + n_vertices, *n_long = referenced + n_vertices;
    auto* totals = reinterpret_cast<unsigned long long*>(ws + l.totals);
    auto* starts = reinterpret_cast<unsigned long long*>(ws + l.starts);
    auto* sentinels = reinterpret_cast<int*>(ws + l.sentinels);
    auto* distinct = reinterpret_cast<int*>(ws + l.distinct);
    auto* long_rows = reinterpret_cast<int*>(ws + l.long_rows);
    void* scan_temp = ws + l.scan_temp;
    size_t scan_bytes = l.total - 256 - l.scan_temp;
    auto* keys_out = reinterpret_cast<unsigned long long*>(keys);
    const int n = n_vertices;
    OB_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * (2 * (size_t)n + 1), stream));
    corner_counts<<<ceil_div(n_faces + 1LL, kThreads), kThreads, 0, stream>>>(faces, n_faces, n, counts, referenced,
                                                                             sentinels);
    OB_CHECK_LAUNCH("corner_counts");
    row_totals<<<ceil_div(n + 1LL, kThreads), kThreads, 0, stream>>>(counts, referenced, n, totals);
    OB_CHECK_LAUNCH("row_totals");
    OB_CUDA(cub::DeviceScan::ExclusiveSum(scan_temp, scan_bytes, totals, starts, n + 1, stream));
    count_launch(1);
    // The sentinel slots' places among themselves.
    OB_CUDA(cub::DeviceScan::ExclusiveSum(scan_temp, scan_bytes, sentinels, sentinels, n_faces + 1, stream));
    count_launch(1);
    if (n_faces > 0) {
        scatter_corners<<<ceil_div(n_faces, kThreads), kThreads, 0, stream>>>(faces, n_faces, n, starts, counts,
                                                                             sentinels, bucket, keys_out, order);
        OB_CHECK_LAUNCH("scatter_corners");
    }
    if (n > 0) {
        place_tail<<<ceil_div(n, kThreads), kThreads, 0, stream>>>(starts, n, n_faces, referenced, sentinels, bucket,
                                                                   keys_out, order);
        OB_CHECK_LAUNCH("place_tail");
        sort_rows<<<ceil_div(n, kSortRows), kSortRows, 0, stream>>>(starts, n, bucket, distinct, long_rows, n_long);
        OB_CHECK_LAUNCH("sort_rows");
        sort_long_rows<<<sm_count(), kLongThreads, 0, stream>>>(starts, long_rows, n_long, bucket, spare, distinct);
        OB_CHECK_LAUNCH("sort_long_rows");
    }
    // (The scan reads distinct[n] and adds it to nothing.)
    OB_CUDA(cub::DeviceScan::ExclusiveSum(scan_temp, scan_bytes, distinct, offsets, n + 1, stream));
    count_launch(1);
    if (n > 0) {
        write_rows<<<ceil_div(n, kSortRows), kWriteThreads, 0, stream>>>(bucket, starts, offsets, n, 6LL * n_faces,
                                                                         keys_out, order, columns, run_start);
        OB_CHECK_LAUNCH("write_rows");
    }
    return OB_OK;
}

}  // extern "C"
