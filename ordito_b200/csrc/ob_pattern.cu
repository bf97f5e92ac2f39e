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
// the CTA writes the sorted segment back. Rows past kThreadRow, whose quadratic time would be one
// thread's, and segments past the shared memory are left to sort_listed_rows by lists.
constexpr int kSortRows = 128;
constexpr int kSortKeys = 3072;  // 24 KB: 24 keys a row on average
constexpr int kThreadRow = 24;
constexpr int kRunTile = 4096;
constexpr int kBlockKeys = 4 * kRunTile;  // the most of a block that write_rows leaves to one CTA

// Rows listed for a warp each (to kWarpRow keys), for 256 threads (to kMidRow) and for a CTA of 1 024.
constexpr int kWarpRow = 128, kMidRow = 1024;
struct RowLists {
    int* counts;  // of the three, then whether a block is past kBlockKeys
    int* rows;    // n for the first list, n for the second from the front and the third from the back
    int n;
    __device__ __forceinline__ int& row(int list, int i) const { return rows[list == 0 ? i : list == 1 ? n + i : 2 * n - 1 - i]; }
    __device__ __forceinline__ void add(int r, int keys) const {
        const int list = keys <= kWarpRow ? 0 : keys <= kMidRow ? 1 : 2;
        row(list, atomicAdd(&counts[list], 1)) = r;
    }
};

__global__ void __launch_bounds__(kSortRows) sort_rows(const unsigned long long* __restrict__ starts, int n,
                                                       unsigned long long* __restrict__ bucket,
                                                       int* __restrict__ distinct, const RowLists lists) {
    __shared__ unsigned long long keys[kSortKeys];
    const int first = blockIdx.x * kSortRows, row = first + threadIdx.x;
    const int begin = row_begin(starts, first), end = row_begin(starts, min(n, first + kSortRows));
    const bool staged = end - begin <= kSortKeys;
    if (threadIdx.x == 0 && end - begin > kBlockKeys) lists.counts[3] = 1;
    if (staged) {
        for (int p = begin + threadIdx.x; p < end; p += kSortRows) keys[p - begin] = bucket[p];
        __syncthreads();
    }
    if (row < n) {
        const int from = row_begin(starts, row), count = row_begin(starts, row + 1) - from;
        if (!staged || count > kThreadRow) {
            if (count > 1) lists.add(row, count);
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

// Merges give each thread consecutive places of the output, whose first pair it finds by bisection along
// the merge's diagonal (merge path; Odeh, Green, Mwassi, Shmueli and Birk, 2012): one bisection for
// several keys. How many of the first `diagonal` keys of the merge of a (na keys) and b (nb) are a's:
__device__ __forceinline__ int merge_split(const unsigned long long* a, int na, const unsigned long long* b, int nb,
                                           int diagonal) {
    int lo = max(0, diagonal - nb), hi = min(diagonal, na);
    while (lo < hi) {
        const int m = (lo + hi) / 2;
        if (a[m] < b[diagonal - 1 - m]) lo = m + 1;
        else hi = m;
    }
    return lo;
}

template <int K>
__device__ __forceinline__ void merge_keys(const unsigned long long* a, int na, const unsigned long long* b, int nb,
                                           int at, unsigned long long (&out)[K]) {
    const unsigned long long none = ~0ULL;  // above every key
    int i = merge_split(a, na, b, nb, min(at, na + nb)), j = min(at, na + nb) - i;
    unsigned long long x = i < na ? a[i] : none, y = j < nb ? b[j] : none;
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const bool left = x < y;
        out[q] = left ? x : y;
        if (left) {
            ++i;
            x = i < na ? a[i] : none;
        } else {
            ++j;
            y = j < nb ? b[j] : none;
        }
    }
}

// `size` keys of `source` (at most 4 T) in order in `tile`, by T threads that meet at `sync`: four a
// thread in registers, then merges, each thread four consecutive places of every output.
template <int T, typename Sync>
__device__ __forceinline__ void sort_tile(const unsigned long long* source, int size, unsigned long long* tile, int tid,
                                          Sync sync) {
    const int mine = 4 * tid;
    for (int i = tid; i < 4 * T; i += T) tile[i] = i < size ? source[i] : ~0ULL;
    sync();
    unsigned long long k[4] = {tile[mine], tile[mine + 1], tile[mine + 2], tile[mine + 3]};
    const auto order = [&k](int x, int y) {
        const unsigned long long low = min(k[x], k[y]), high = max(k[x], k[y]);
        k[x] = low;
        k[y] = high;
    };
    order(0, 1), order(2, 3), order(0, 2), order(1, 3), order(1, 2);
    for (int width = 4;; width *= 2) {
        sync();
#pragma unroll
        for (int q = 0; q < 4; ++q) tile[mine + q] = k[q];
        sync();
        if (width >= size) return;
        const int pair = mine / (2 * width) * (2 * width);
        merge_keys(tile + pair, width, tile + pair + width, width, mine - pair, k);
    }
}

// A row's `count` keys at `from` (all different), in order to `to`, by rank; returns its distinct columns.
__device__ __forceinline__ int rank_sort(const unsigned long long* from, int count, unsigned long long* to, int lane) {
    int columns = 0;
    for (int i = lane; i < count; i += 32) {
        const unsigned long long key = from[i];
        int rank = 0;
        bool first = true;
#pragma unroll 4
        for (int j = 0; j < count; ++j) {
            const unsigned long long other = from[j];
            rank += other < key;
            first = first && !(other < key && (other >> 32) == (key >> 32));
        }
        to[rank] = key;
        columns += first;
    }
    return warp_sum(columns);
}

// The listed rows, in one launch: a warp a row by rank (through the second buffer), 256 threads a row by a
// tile of four keys a thread, then a CTA a row by such tiles, merged pairwise between the buckets and the
// second buffer, each thread sixteen consecutive places of every output. A long row's runs up to each run
// tile's end stay in the second buffer, for write_rows. ms a build: 20 000 fans of 30 faces 0.28, one million
// random faces in rows of 60 keys 0.70, of 300 0.98, of 3 000 0.98, a fan of 200 000 faces 7.15; with every row past
// 96 keys, or of a crowded block, by 1 024 threads, runs of 1 024 by rank and a bisection a key 0.60, 1.76,
// 1.08, 3.20 and 18.7; by a general segmented sort of the stored keys 0.39, 3.1, 1.90, 1.50 and 7.1.
constexpr int kListedThreads = 1024, kGroup = 256;
constexpr int kMergeKeys = 16;

__global__ void __launch_bounds__(kListedThreads) sort_listed_rows(const unsigned long long* __restrict__ starts,
                                                                   const RowLists lists, unsigned long long* bucket,
                                                                   unsigned long long* spare,
                                                                   int* __restrict__ distinct) {
    constexpr int T = kListedThreads, kTile = 4 * T;
    __shared__ unsigned long long tile[kTile];
    __shared__ int scratch[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int item = blockIdx.x * (T / 32) + warp; item < lists.counts[0]; item += gridDim.x * (T / 32)) {
        const int r = lists.row(0, item), from = row_begin(starts, r), count = row_begin(starts, r + 1) - from;
        const int columns = rank_sort(bucket + from, count, spare + from, lane);
        if (lane == 0) distinct[r] = columns;
        __syncwarp();
        for (int i = lane; i < count; i += 32) bucket[from + i] = spare[from + i];
    }
    const int group = threadIdx.x / kGroup, at_group = threadIdx.x % kGroup;
    const auto group_sync = [group]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kGroup) : "memory"); };
    for (int item = blockIdx.x * (T / kGroup) + group; item < lists.counts[1]; item += gridDim.x * (T / kGroup)) {
        const int r = lists.row(1, item), from = row_begin(starts, r), count = row_begin(starts, r + 1) - from;
        unsigned long long* mine = tile + 4 * kGroup * group;
        group_sync();  // the row before is done with
        sort_tile<kGroup>(bucket + from, count, mine, at_group, group_sync);
        int columns = 0;
        for (int i = at_group; i < count; i += kGroup) {
            bucket[from + i] = mine[i];
            columns += i == 0 || (mine[i] >> 32) != (mine[i - 1] >> 32);
        }
        columns = warp_sum(columns);
        if (lane == 0) scratch[warp] = columns;
        group_sync();
        if (at_group == 0) {
            for (int w = 1; w < kGroup / 32; ++w) columns += scratch[warp + w];
            distinct[r] = columns;
        }
    }
    const auto sync = []() { __syncthreads(); };
    for (int item = blockIdx.x; item < lists.counts[2]; item += gridDim.x) {
        const int row = lists.row(2, item);
        const int from = row_begin(starts, row), count = row_begin(starts, row + 1) - from;
        unsigned long long *source = bucket + from, *target = spare + from;
        for (int r = 0; r < count; r += kTile) {
            const int size = min(kTile, count - r);
            __syncthreads();  // the tile and the row before are done with
            sort_tile<T>(source + r, size, tile, (int)threadIdx.x, sync);
            for (int i = threadIdx.x; i < size; i += T) source[r + i] = tile[i];
        }
        __syncthreads();
        for (long long width = kTile; width < count; width *= 2) {
            for (long long at = (long long)kMergeKeys * threadIdx.x; at < count; at += (long long)kMergeKeys * T) {
                const long long pair = at / (2 * width) * (2 * width);
                const int na = (int)min(width, count - pair), nb = (int)min(width, count - pair - na);
                unsigned long long k[kMergeKeys];
                merge_keys(source + pair, na, source + pair + na, nb, (int)(at - pair), k);
#pragma unroll
                for (int q = 0; q < kMergeKeys; ++q)
                    if (at + q < count) target[at + q] = k[q];
            }
            __syncthreads();
            unsigned long long* swap = source;
            source = target;
            target = swap;
        }
        if (source != bucket + from) {
            for (int i = threadIdx.x; i < count; i += T) bucket[from + i] = source[i];
            __syncthreads();
        }
        // The runs of one column up to each run tile's end.
        int total = 0;
        for (int r = 0; r < count; r += kRunTile) {
            int columns = 0;
            for (int i = r + threadIdx.x; i < min(count, r + kRunTile); i += T)
                columns += i == 0 || (bucket[from + i] >> 32) != (bucket[from + i - 1] >> 32);
            total += block_sum(columns, scratch);
            if (threadIdx.x == 0) spare[from + r / kRunTile] = (unsigned long long)total;
        }
        if (threadIdx.x == 0) distinct[row] = total;
    }
}

// The sorted buckets out: each position's key and payload, and each run of one column as one entry (the
// entries of consecutive rows are consecutive: offsets of the first row plus the runs counted so far).
constexpr int kWriteThreads = 256;

// The positions [begin, end) of the rows [first, first + rows), whose starts are row_start, from entry on.
template <typename Start>
__device__ __forceinline__ void write_positions(const unsigned long long* __restrict__ bucket, int begin, int end,
                                                int first, int rows, Start row_start, int entry, int n,
                                                long long tail, unsigned long long* __restrict__ keys_out,
                                                int* __restrict__ order_out, int* __restrict__ columns,
                                                int* __restrict__ run_start, int* warp_runs) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = begin; base < end; base += kWriteThreads) {
        const int p = base + threadIdx.x;
        bool opens = false;
        int col = 0;
        if (p < end) {
            // The row holding p: row_start(lo) <= p < row_start(lo + 1) (empty rows hold none).
            int lo = 0, hi = rows - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (row_start(mid) <= p) lo = mid;
                else hi = mid - 1;
            }
            const unsigned long long v = bucket[p];
            col = (int)(v >> 32);
            opens = p == row_start(lo) || (int)(bucket[p - 1] >> 32) != col;
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

// A CTA kSortRows rows; the CTAs past those take the blocks of rows with more than kBlockKeys keys, run
// tile by run tile of each row (two thousand rows of 3 000 keys are sixteen blocks: 1.6 ms by a CTA
// each).
__global__ void __launch_bounds__(kWriteThreads) write_rows(const unsigned long long* __restrict__ bucket,
                                                            const unsigned long long* __restrict__ spare,
                                                            const unsigned long long* __restrict__ starts,
                                                            const int* __restrict__ offsets, int n, long long tail,
                                                            const int* __restrict__ crowded,
                                                            unsigned long long* __restrict__ keys_out,
                                                            int* __restrict__ order_out, int* __restrict__ columns,
                                                            int* __restrict__ run_start) {
    __shared__ int row_start[kSortRows + 1];
    __shared__ int warp_runs[kWriteThreads / 32];
    const int blocks = (n + kSortRows - 1) / kSortRows;
    if ((int)blockIdx.x < blocks) {
        const int first = blockIdx.x * kSortRows, rows = min(kSortRows, n - first);
        for (int i = threadIdx.x; i <= rows; i += kWriteThreads) row_start[i] = row_begin(starts, first + i);
        __syncthreads();
        if (row_start[rows] - row_start[0] > kBlockKeys) return;
        write_positions(bucket, row_start[0], row_start[rows], first, rows, [&](int i) { return row_start[i]; },
                        offsets[first], n, tail, keys_out, order_out, columns, run_start, warp_runs);
        return;
    }
    if (*crowded == 0) return;
    // Tasks: run tile t of the bucket array, the rows' parts in it (a block of kBlockKeys at 128 rows has
    // few rows a tile, so their walk is short).
    const int total = row_begin(starts, n), helpers = gridDim.x - blocks;
    for (long long at = (long long)(blockIdx.x - blocks) * kRunTile; at < total; at += (long long)helpers * kRunTile) {
        const int begin = (int)at, end = (int)min((long long)total, at + kRunTile);
        // The row holding `begin`.
        int lo = 0, hi = n - 1;
        while (lo < hi) {
            const int mid = (int)(((long long)lo + hi + 1) / 2);
            if (row_begin(starts, mid) <= begin) lo = mid;
            else hi = mid - 1;
        }
        for (int row = lo, p = begin; p < end; ++row) {
            const int from = row_begin(starts, row), to = min(end, row_begin(starts, row + 1));
            if (to <= p) continue;
            const int block = row / kSortRows * kSortRows;
            const int keys = row_begin(starts, min(n, block + kSortRows)) - row_begin(starts, block);
            if (keys <= kBlockKeys) {
                // Written above, the block's other rows too.
                p = max(p, min(end, row_begin(starts, min(n, block + kSortRows))));
                row = block + kSortRows - 1;
                continue;
            }
            // The row's runs before p: a listed row's whole run tiles by its table, the rest counted.
            const int whole = (p - from) / kRunTile;
            int entry = offsets[row] + (whole > 0 ? (int)spare[from + whole - 1] : 0);
            for (int base = from + whole * kRunTile; base < p; base += kWriteThreads) {
                const int q = base + (int)threadIdx.x;
                const bool opens = q < p && (q == from || (bucket[q - 1] >> 32) != (bucket[q] >> 32));
                entry += __syncthreads_count(opens);
            }
            write_positions(bucket, p, to, row, 1, [&](int) { return from; }, entry, n, tail, keys_out, order_out,
                            columns, run_start, warp_runs);
            p = to;
        }
    }
}

struct PatternLayout {
    size_t bucket = 0, spare = 0, counts = 0, totals = 0, starts = 0, sentinels = 0, distinct = 0, listed = 0,
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
    // Zeroed at the start of a build, in one piece: the rows' counters, their flags, the lists' lengths.
    l.counts = align_up(l.spare + 8 * (size_t)count);
    l.totals = align_up(l.counts + 4 * (2 * (size_t)n + 4));
    l.starts = align_up(l.totals + 8 * ((size_t)n + 1));
    l.sentinels = align_up(l.starts + 8 * ((size_t)n + 1));
    l.distinct = align_up(l.sentinels + 4 * ((size_t)n_faces + 1));
    l.listed = align_up(l.distinct + 4 * ((size_t)n + 1));
    l.scan_temp = align_up(l.listed + 4 * 2 * (size_t)n);
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
    int* referenced = counts + n_vertices;
    auto* totals = reinterpret_cast<unsigned long long*>(ws + l.totals);
    auto* starts = reinterpret_cast<unsigned long long*>(ws + l.starts);
    auto* sentinels = reinterpret_cast<int*>(ws + l.sentinels);
    auto* distinct = reinterpret_cast<int*>(ws + l.distinct);
    const RowLists lists{referenced + n_vertices, reinterpret_cast<int*>(ws + l.listed), n_vertices};
    void* scan_temp = ws + l.scan_temp;
    size_t scan_bytes = l.total - 256 - l.scan_temp;
    auto* keys_out = reinterpret_cast<unsigned long long*>(keys);
    const int n = n_vertices;
    OB_CUDA(cudaMemsetAsync(counts, 0, sizeof(int) * (2 * (size_t)n + 4), stream));
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
        sort_rows<<<ceil_div(n, kSortRows), kSortRows, 0, stream>>>(starts, n, bucket, distinct, lists);
        OB_CHECK_LAUNCH("sort_rows");
        sort_listed_rows<<<sm_count(), kListedThreads, 0, stream>>>(starts, lists, bucket, spare, distinct);
        OB_CHECK_LAUNCH("sort_listed_rows");
    }
    // (The scan reads distinct[n] and adds it to nothing.)
    OB_CUDA(cub::DeviceScan::ExclusiveSum(scan_temp, scan_bytes, distinct, offsets, n + 1, stream));
    count_launch(1);
    if (n > 0) {
        const int helpers = std::min(ceil_div(count, kRunTile), sm_count());
        write_rows<<<ceil_div(n, kSortRows) + helpers, kWriteThreads, 0, stream>>>(
            bucket, spare, starts, offsets, n, 6LL * n_faces, lists.counts + 3, keys_out, order, columns, run_start);
        OB_CHECK_LAUNCH("write_rows");
    }
    return OB_OK;
}

}  // extern "C"
