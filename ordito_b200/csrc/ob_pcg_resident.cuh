// The conjugate gradient loop of ob_pcg.cu as ONE kernel that stays on the chip, for one right-hand
// side on an operator small enough to share out over the SMs' registers and shared memory.
//
// What bounds a round of a small system is not its bytes but its chain: a mat-vec and an update
// kernel (13 kernels under the Chebyshev polynomial), each with its launch, its first loads and
// its drain (4-5 us a kernel measured inside the loop graph, whatever the size below ~100 k rows).
// Here a thread owns R rows for the whole solve: their r, p, s, x, u and first seven entries (a
// mesh row's usual count) sit in registers, further entries in shared memory, and a round's kernels
// become barriers between the phases. Only the vector the next mat-vec gathers is published. Three
// forms, by how far it has to travel:
//
//   kBlock    one CTA: shared memory, __syncthreads;
//   kCluster  up to 16 CTAs, each holding its rows' values and a copy of the other CTAs' values its
//             rows read (its halo). A CTA publishes by storing its own values and pushing those
//             other CTAs hold copies of into their shared memory (a list made at the start), so
//             every gather is local. The pushes are asynchronous stores that count themselves off at
//             a barrier in the shared memory they arrive in (mbarrier transaction bytes), so a CTA
//             waits for the values it reads and nothing else: barrier.cluster between the phases
//             took 1.3 us each. (Gathering from the other CTAs took 3 us a mat-vec on a 10 k-vertex
//             icosphere, whose edge rows read nothing local. Where a halo does not fit, or a CTA
//             would push to one it does not read, the whole cluster gathers so, between
//             barrier.clusters.)
//   kGrid     up to one CTA an SM (a cooperative launch): global memory at L2, an arrival counter
//             between phases.
//
// Every wait is bounded: a CTA that gives up raises `abort`, the others then give up as well, and
// `gave_up` stays set until the host has reported OB_ERR_TIMEOUT. Rows longer than the entries a thread holds read the rest from the CSR arrays. A round's float64
// chain is kept short (two partial sums a row, one division behind the dots), since latency is what
// is left: the sums a row and the scalars agree with the loop graph's to rounding. The dots are
// folded thread, warp, CTA in a fixed order, so every run gives the same bits.
#pragma once

#include "ob_internal.cuh"

namespace ob {
namespace {

enum ResidentForm : int { kBlock = 0, kCluster = 1, kGrid = 2 };
constexpr int kClusterMax = 16;
constexpr int kHalo = 1024;      // other CTAs' values a cluster CTA holds copies of
constexpr int kHaloTable = 2048; // the hash table that numbers them
constexpr int kPushesARow = 4;   // a CTA's push list, of its rows (two rows a thread; half at four)
constexpr int kResidentWidth = 16;      // entries a row kept on the chip, at most
constexpr int kBaseEntries = 7;  // a mesh row's usual count: every row is padded to it
__host__ __device__ constexpr int register_entries(int rows_a_thread) { return rows_a_thread <= 2 ? kBaseEntries : 0; }
// Whether x, p and s of a thread's rows lie in shared memory: four rows' vectors under the polynomial
// take more than the 128 registers a thread has, and a step's loads then wait for one another (3 400
// cycles a mat-vec of 1 250 rows, 2 200 without the polynomial). Such a solver has no settle check.
__host__ __device__ constexpr bool far_vectors(int rows_a_thread, bool cheb) { return rows_a_thread == 4 && cheb; }
__host__ __device__ constexpr int resident_threads(int) { return 512; }
// Polls before a wait gives up, about a second: of a grid barrier (>= 0.3 us each), of a barrier in
// shared memory (2 us at most each).
constexpr int kGridPolls = 1 << 22, kClusterPolls = 1 << 19;

struct ResidentArgs {
    int n;
    const int* offsets;
    const int* columns;
    const double* values;
    const double* inv_diag;
    const double4* steps;  // the polynomial's, when preconditioned by it
    const double* rhs;
    double* x;
    double tol;
    int maxiter;
    int check_rounds;  // 0: stop by the residual
    double change_tolerance;
    int settle_rounds;
    LoopState* state;
    ColumnScalars* scalars;
    int narrow;  // the operator's values are rounded to float32
    int width;   // entries a row on the chip, those in registers among them
    int pushes;  // kCluster: the capacity of a CTA's push list
    int polls;   // before a wait gives up
    int* abort;  // 1 when a wait gave up (zero at the launch of kGrid, zeroed by the others)
    int* gave_up;  // the same, but not zeroed by a launch
    // kGrid: the published vector (two buffers of n), the CTAs' partial sums (6 a CTA) and the
    // arrival counter (zero at the launch).
    double* published;
    double* partials;
    unsigned int* counter;
};

__device__ __forceinline__ unsigned shared_address(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned cluster_address(unsigned local, int rank) {
    unsigned out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
    return out;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile(
        "barrier.cluster.arrive.release.aligned;\n\t"
        "barrier.cluster.wait.acquire.aligned;" ::
            : "memory");
}

__device__ __forceinline__ void store_cluster(unsigned at, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

// A value another SM has written: from L2, and read anew each time.
__device__ __forceinline__ double load_l2(const double* p) {
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Barriers in shared memory that count arriving bytes. A phase ends when the one arrival (which
// says how many bytes are due) and that many bytes have come.
__device__ __forceinline__ void arrivals_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void arrivals_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Waits for the phase of the given parity, `polls` tries of 2 us at most; false when it gave up.
__device__ __forceinline__ bool arrivals_wait(unsigned bar, unsigned parity, int polls) {
    for (int i = 0; i < polls; ++i) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, 2000;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// A value into a CTA's shared memory, counted at that CTA's barrier when it is there.
__device__ __forceinline__ void push_cluster(unsigned at, double v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(at), "d"(v), "r"(bar)
                 : "memory");
}

// Arrives at a grid barrier and waits until `goal` arrivals (monotonic, wrap-safe). False when
// this wait, or another CTA's, gave up. Called by every thread.
__device__ __forceinline__ bool grid_barrier(unsigned int* counter, unsigned int goal, int polls, int* abort,
                                             int* alive) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
        unsigned seen;
        int spins = 0, ok = 1;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
            if ((int)(seen - goal) >= 0) break;
            if (++spins >= polls || ((spins & 255) == 0 && *(volatile int*)abort != 0)) {
                atomicExch(abort, 1);
                ok = 0;
                break;
            }
        }
        __threadfence();
        *alive = ok;
    }
    __syncthreads();
    return *alive != 0;
}

// The warp's sums of three values: lane 8 q ends with the sum of value q (q < 3), in a fixed
// order. Two exchange steps hand each quarter of the warp one of the values, the last three add
// within the quarters: 6 shuffles where three plain sums take 15.
__device__ __forceinline__ double packed_sum(double v0, double v1, double v2, int lane) {
    const bool high = lane & 16, odd = lane & 8;
    const double s0 = __shfl_xor_sync(0xffffffffu, high ? v0 : v2, 16);
    const double s1 = __shfl_xor_sync(0xffffffffu, high ? v1 : 0.0, 16);
    double a = (high ? v2 : v0) + s0, b = high ? 0.0 : v1 + s1;
    a = (odd ? b : a) + __shfl_xor_sync(0xffffffffu, odd ? a : b, 8);
    a += __shfl_xor_sync(0xffffffffu, a, 4);
    a += __shfl_xor_sync(0xffffffffu, a, 2);
    return a + __shfl_xor_sync(0xffffffffu, a, 1);
}

// The sums of three rows of `count` <= 32 values at `from` (rows `stride` apart): a quarter of the
// warp a row. Every lane gets the three.
__device__ __forceinline__ void row_sums(const double* from, int stride, int count, int lane, double& v0,
                                         double& v1, double& v2) {
    const int q = lane >> 3;
    double v = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int w = (lane & 7) + 8 * j;
        if (q < 3 && w < count) v += from[q * stride + w];
    }
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v0 = __shfl_sync(0xffffffffu, v, 0);
    v1 = __shfl_sync(0xffffffffu, v, 8);
    v2 = __shfl_sync(0xffffffffu, v, 16);
}

template <int R, int FORM, bool CHEB>
__global__ void __launch_bounds__(resident_threads(R), 1) resident_pcg_kernel(const ResidentArgs a) {
    constexpr int E = register_entries(R);
    extern __shared__ double resident_smem[];
    const int T = blockDim.x, S = T * R, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int warps = T >> 5, cta = blockIdx.x, ctas = gridDim.x;
    // Shared memory: the published vector's two buffers (own rows, then the halo), the cluster's
    // partial sums (two rows of three values a CTA), the warps' (one), three totals, the entries past
    // the registers' (values, places), then the halo's table and the push list.
    const int buffer = FORM == kGrid ? 0 : S + (FORM == kCluster ? kHalo : 0);
    double* pub = resident_smem;
    double* parts = pub + 2 * buffer;
    double* scratch = parts + 6 * kClusterMax;
    double* totals = scratch + 3 * 32;
    int* alive = reinterpret_cast<int*>(totals + 3);
    double* bars = totals + 4;  // kCluster: a barrier a buffer of the halo, then of the partial sums
    double4* steps = reinterpret_cast<double4*>(bars + 4);
    // x, p and s, which a round needs once, where the polynomial's steps need their registers.
    constexpr bool kFar = far_vectors(R, CHEB);
    double* far = bars + 4 + 4 * kChebyshevDegree;
    double* vals = far + (kFar ? 3 * S : 0);
    const int more = a.width - E;
    int2* push = reinterpret_cast<int2*>(vals + (size_t)more * S);  // (own row, address); kCluster
    int* table = reinterpret_cast<int*>(push + (FORM == kCluster ? a.pushes : 0));
    int* table_slot = table + kHaloTable;
    int* counters = table_slot + kHaloTable;  // halo values, pushes, pulled entries
    unsigned* places = FORM == kCluster ? reinterpret_cast<unsigned*>(counters + 4) : reinterpret_cast<unsigned*>(push);
    const unsigned pub_at = FORM == kGrid ? 0u : shared_address(pub);
    unsigned goal = 0;  // grid arrivals due
    bool ok = true, pulls = false;
    int pushed = 0;
    // kCluster: exchanges so far of the published vector and of partial sums (each alternates between
    // two buffers and their barriers, and a barrier between its two phases), and the halo's bytes.
    unsigned sent = 0, summed = 0, due = 0;
    const unsigned bars_at = FORM == kCluster ? shared_address(bars) : 0u;
    if (FORM != kGrid && cta == 0 && tid == 0) *a.abort = 0;
    if (CHEB && tid < kChebyshevDegree - 1) steps[tid] = a.steps[tid];  // read behind the start's barriers

    auto barrier = [&]() {
        if (FORM == kBlock) __syncthreads();
        if (FORM == kCluster) cluster_barrier();
        if (FORM == kGrid) {
            goal += (unsigned)ctas;
            ok = grid_barrier(a.counter, goal, a.polls, a.abort, alive) && ok;
        }
    };
    // Sums over every row of the system, in two halves around a barrier: `fold` leaves the CTA's
    // three sums where `read` finds them after the next barrier(), or what stands for it (below).
    // `slot` 0: the dots; 1: the settle check's, a maximum and a sum. (Between two folds lies a
    // barrier after which the first's scratch is not read; one CTA reads it later.)
    auto fold = [&](double v0, double v1, double v2, int slot) {
        if (FORM == kBlock && slot == 1) __syncthreads();
        if (slot == 0) {
            v0 = packed_sum(v0, v1, v2, lane);
            if ((lane & 7) == 0 && lane < 24) scratch[4 * lane + warp] = v0;
        } else {
            v0 = warp_max(v0);
            v1 = warp_sum(v1);
            if (lane == 0) {
                scratch[warp] = v0;
                scratch[32 + warp] = v1;
            }
        }
        if (FORM == kBlock) return;
        ok = __syncthreads_and(ok);
        if (warp != 0) return;
        if (slot == 0) {
            row_sums(scratch, 32, warps, lane, v0, v1, v2);
        } else {
            v0 = warp_max(lane < warps ? scratch[lane] : 0.0);
            v1 = warp_sum(lane < warps ? scratch[32 + lane] : 0.0);
            v2 = 0.0;
        }
        if (FORM == kCluster) {
            const unsigned b = summed & 1u;
            if (!pulls && lane == 0) arrivals_expect(bars_at + 8u * (2u + b), 24u * (unsigned)ctas);
            if (lane < ctas) {
                const unsigned at = cluster_address(shared_address(parts + 3 * kClusterMax * b + cta), lane);
                if (pulls) {
                    store_cluster(at, v0);
                    store_cluster(at + 8u * kClusterMax, v1);
                    store_cluster(at + 16u * kClusterMax, v2);
                } else {
                    const unsigned bar = cluster_address(bars_at + 8u * (2u + b), lane);
                    push_cluster(at, v0, bar);
                    push_cluster(at + 8u * kClusterMax, v1, bar);
                    push_cluster(at + 16u * kClusterMax, v2, bar);
                }
            }
        } else if (lane == 0) {
            double* at = a.partials + (size_t)3 * ctas * slot + cta;
            __stcg(at, v0);
            __stcg(at + ctas, v1);
            __stcg(at + 2 * ctas, v2);
        }
    };
    // Where the cluster's exchanges count themselves off, a wait for one stands for the barrier. A
    // thread that gave up waits no more; the CTA agrees on `ok` behind the sums and at its next
    // barrier of its own (fold, publish), and leaves only where it has agreed.
    auto await_sums = [&]() {
        if (FORM == kCluster && !pulls) {
            ok = ok && arrivals_wait(bars_at + 8u * (2u + (summed & 1u)), (summed >> 1) & 1u, a.polls);
            ok = __syncthreads_and(ok);
        } else {
            barrier();
        }
    };
    auto await_published = [&]() {
        if (FORM == kCluster && !pulls) {
            ok = ok && arrivals_wait(bars_at + 8u * (sent & 1u), (sent >> 1) & 1u, a.polls);
            ++sent;
        } else {
            barrier();
        }
    };
    auto read = [&](double& v0, double& v1, double& v2, int slot) {
        if (FORM == kGrid) {
            // A warp a sum, so the CTAs' partials are read once a CTA.
            if (warp < 3) {
                const double* from = a.partials + (size_t)ctas * (3 * slot + warp);
                const bool largest = slot == 1 && warp == 0;
                double v = 0.0;
#pragma unroll 5
                for (int b = lane; b < ctas; b += 32) {
                    const double p = load_l2(from + b);
                    v = largest ? fmax(v, p) : v + p;
                }
                __syncwarp();
                v = largest ? warp_max(v) : warp_sum(v);
                if (lane == 0) totals[warp] = v;
            }
            __syncthreads();
            v0 = totals[0], v1 = totals[1], v2 = totals[2];
            return;
        }
        const double* from = FORM == kBlock ? scratch : parts + 3 * kClusterMax * (summed & 1u);
        ++summed;
        const int stride = FORM == kBlock ? 32 : kClusterMax, count = FORM == kBlock ? warps : ctas;
        if (slot == 0) {
            row_sums(from, stride, count, lane, v0, v1, v2);
        } else {
            v0 = warp_max(lane < count ? from[lane] : 0.0);
            v1 = warp_sum(lane < count ? from[stride + lane] : 0.0);
        }
    };

    // -- the rows: their entries, r = b - A x ----------------------------------------------------
    constexpr int N = kFar ? 1 : R;
    double x[N], r[R], p[N], s[N], u[R], inv[R], scaled[R], previous[N];
    double value[E ? E : 1][R];
    unsigned place[E ? E : 1][R];  // a column until the places are known
    int over = 0, span = kBaseEntries;
    double bb = 0.0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = cta * S + i * T + tid;
        const bool live = row < a.n;
        const int o = live ? a.offsets[row] : 0, d = live ? a.offsets[row + 1] - o : 0;
        const unsigned self = (unsigned)min(row, a.n - 1);
        double ax = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool has = e < d;
            const int col = has ? a.columns[o + e] : (int)self;
            const double v = has ? a.values[o + e] : 0.0;
            if (has) ax = fma(v, a.x[col], ax);
            value[e][i] = a.narrow ? (double)(float)v : v;
            place[e][i] = (unsigned)col;
        }
        for (int e = E; e < d; ++e) {
            const int col = a.columns[o + e];
            const double v = a.values[o + e];
            ax = fma(v, a.x[col], ax);
            if (e < a.width) {
                vals[((e - E) * R + i) * T + tid] = a.narrow ? (double)(float)v : v;
                places[((e - E) * R + i) * T + tid] = (unsigned)col;
            }
        }
        over |= d > a.width;
        span = max(span, min(d, a.width));
        const double b = live ? a.rhs[row] : 0.0;
        bb = fma(b, b, bb);
        const double start = live ? a.x[row] : 0.0;
        if constexpr (kFar) {
            far[i * T + tid] = start;
            far[S + i * T + tid] = far[2 * S + i * T + tid] = 0.0;
        } else {
            x[i] = previous[i] = start;
            p[i] = s[i] = 0.0;
        }
        r[i] = live ? b - ax : 0.0;
        inv[i] = live ? a.inv_diag[row] : 0.0;
        scaled[i] = u[i] = inv[i] * r[i];
    }
    // The warp's rows are padded to one span with zero entries on a live row.
    __syncwarp();
    over = __any_sync(0xffffffffu, over);
    span = __reduce_max_sync(0xffffffffu, span);
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = cta * S + i * T + tid;
        const int d = row < a.n ? a.offsets[row + 1] - a.offsets[row] : 0;
        for (int e = max(d, E); e < span; ++e) {
            vals[((e - E) * R + i) * T + tid] = 0.0;
            places[((e - E) * R + i) * T + tid] = (unsigned)min(row, a.n - 1);
        }
    }

    // -- the halo: each other CTA's column numbered once, its owner told to push it ------------
    auto mine = [&](int col) { return FORM != kCluster || (unsigned)(col - cta * S) < (unsigned)S; };
    // A column's place in the table (-1: the table was full when it came).
    auto find = [&](int col, bool insert) -> int {
        unsigned h = ((unsigned)col * 2654435761u) >> 21;  // kHaloTable = 2^11
        for (int probe = 0; probe < 64; ++probe, h = (h + 1) & (kHaloTable - 1)) {
            const int was = insert ? atomicCAS(&table[h], -1, col) : table[h];
            if (was == col || (insert && was == -1)) return (int)h;
            if (was == -1) return -1;
        }
        return -1;
    };
    // A column's shared address (its own row's, its halo copy's, or its owner's), or the column.
    auto place_of = [&](int col) -> unsigned {
        if (FORM == kGrid) return (unsigned)col;
        if (mine(col)) return pub_at + 8u * (unsigned)(FORM == kCluster ? col - cta * S : col);
        const int h = find(col, false);
        if (h >= 0 && table_slot[h] >= 0) return pub_at + 8u * (unsigned)(S + table_slot[h]);
        return cluster_address(pub_at + 8u * (unsigned)(col % S), col / S);
    };
    if (FORM == kCluster) {
        for (int h = tid; h < kHaloTable; h += T) table[h] = -1;
        if (tid < 4) counters[tid] = 0;
        if (tid == 0) {
            for (unsigned b = 0; b < 4; ++b) arrivals_init(bars_at + 8u * b);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int i = tid; i < 2 * kHalo; i += T) pub[(i / kHalo) * buffer + S + i % kHalo] = 0.0;
        cluster_barrier();  // every CTA of the cluster runs, its table, counters and barriers are ready
        bool pulled = false;
        unsigned from = 0;  // the CTAs this one holds copies from
#pragma unroll
        for (int i = 0; i < R; ++i) {
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (!mine((int)place[e][i])) pulled |= find((int)place[e][i], true) < 0;
            for (int e = E; e < span; ++e) {
                const int col = (int)places[((e - E) * R + i) * T + tid];
                if (!mine(col)) pulled |= find(col, true) < 0;
            }
        }
        __syncthreads();
        for (int h = tid; h < kHaloTable; h += T) {
            if (table[h] < 0) continue;
            const int slot = atomicAdd(&counters[0], 1), owner = table[h] / S;
            int taken = -1;
            if (slot < kHalo) {
                unsigned at;
                asm volatile("atom.shared::cluster.add.u32 %0, [%1], 1;"
                             : "=r"(at)
                             : "r"(cluster_address(shared_address(counters + 1), owner))
                             : "memory");
                if ((int)at < a.pushes) {
                    const unsigned entry = cluster_address(shared_address(push + at), owner);
                    asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(entry),
                                 "r"(table[h] - owner * S), "r"((cta << 16) | slot)
                                 : "memory");
                    taken = slot;
                    from |= 1u << owner;
                }
            }
            table_slot[h] = taken;
            pulled |= taken < 0;
        }
        if (over) pulled = true;  // entries read from the CSR arrays may lie anywhere
        from = __reduce_or_sync(0xffffffffu, from);
        if (lane == 0 && from) atomicOr(&counters[3], (int)from);
        cluster_barrier();  // every owner's list is whole
        pushed = min(counters[1], a.pushes);
        due = 8u * (unsigned)min(counters[0], kHalo);
        unsigned to_whom = 0;
        for (int q = tid; q < pushed; q += T) to_whom |= 1u << (push[q].y >> 16);
        to_whom = __reduce_or_sync(0xffffffffu, to_whom);
        // A CTA pushes again once it holds what it waits for: safe where those it pushes to are
        // those it reads. One that cannot takes the whole cluster back to barriers.
        if (lane == 0 && (to_whom & ~(unsigned)counters[3])) pulled = true;
        if (__any_sync(0xffffffffu, pulled) && lane < ctas)
            asm volatile("red.shared::cluster.or.b32 [%0], 1;" ::"r"(cluster_address(shared_address(counters + 2), lane))
                         : "memory");
        cluster_barrier();
        pulls = counters[2] != 0;
        for (int q = tid; q < pushed; q += T) {
            const int2 to = push[q];  // (own row, (CTA, slot)) to (own row, slot's address | CTA in the high bits)
            push[q].y = (int)cluster_address(pub_at + 8u * (unsigned)(S + (to.y & 0xffff)), to.y >> 16);
            push[q].x = to.x | (to.y & 0x7fff0000);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
#pragma unroll
        for (int e = 0; e < E; ++e) place[e][i] = place_of((int)place[e][i]);
        for (int e = E; e < span; ++e) {
            unsigned* at = places + ((e - E) * R + i) * T + tid;
            *at = place_of((int)*at);
        }
    }

    int parity = 0;
    auto publish = [&](const double* v) {
        parity ^= 1;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int at = i * T + tid;
            if (FORM != kGrid)
                pub[parity * buffer + at] = v[i];
            else if (cta * S + at < a.n)
                __stcg(a.published + (size_t)parity * a.n + cta * S + at, v[i]);
        }
        if (FORM == kCluster) {
            ok = __syncthreads_and(ok);
            const unsigned bar = bars_at + 8u * (sent & 1u);
            if (!pulls && tid == 0) arrivals_expect(bar, due);
            for (int q = tid; q < pushed; q += T) {
                const int2 to = push[q];
                const unsigned at = (unsigned)to.y + 8u * (unsigned)(parity * buffer);
                const double v = pub[parity * buffer + (to.x & 0xffff)];
                if (pulls) store_cluster(at, v);
                else push_cluster(at, v, cluster_address(bar, to.x >> 16));
            }
        }
    };
    auto gather = [&](unsigned at) -> double {
        double v;
        if (FORM == kGrid) {
            v = load_l2(a.published + (size_t)parity * a.n + at);
        } else if (FORM == kCluster && pulls) {
            asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at + 8u * (unsigned)(parity * buffer)));
        } else {
            asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at + 8u * (unsigned)(parity * buffer)));
        }
        return v;
    };
    // out = A (the published vector): two partial sums a row halve the chain.
    auto matvec = [&](double* out) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            double even = 0.0, odd = 0.0;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                if (e & 1) odd = fma(value[e][i], gather(place[e][i]), odd);
                else even = fma(value[e][i], gather(place[e][i]), even);
            }
            out[i] = even + odd;
        }
        // Four rows a thread: the base entries from shared memory, all their loads ahead of the sums.
        if (E == 0) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                double v[kBaseEntries], u_of[kBaseEntries];
#pragma unroll
                for (int e = 0; e < kBaseEntries; ++e) {
                    const int at = (e * R + i) * T + tid;
                    v[e] = vals[at];
                    u_of[e] = gather(places[at]);
                }
                double even = 0.0, odd = 0.0;
#pragma unroll
                for (int e = 0; e < kBaseEntries; ++e) {
                    if (e & 1) odd = fma(v[e], u_of[e], odd);
                    else even = fma(v[e], u_of[e], even);
                }
                out[i] = even + odd;
            }
        }
        for (int e = kBaseEntries; e < span; ++e) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int at = ((e - E) * R + i) * T + tid;
                out[i] = fma(vals[at], gather(places[at]), out[i]);
            }
        }
        if (over) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int row = cta * S + i * T + tid;
                const int o = row < a.n ? a.offsets[row] : 0, d = row < a.n ? a.offsets[row + 1] - o : 0;
                for (int e = a.width; e < d; ++e) {
                    const double v = a.narrow ? (double)(float)a.values[o + e] : a.values[o + e];
                    out[i] = fma(v, gather(place_of(a.columns[o + e])), out[i]);
                }
            }
            __syncwarp();
        }
    };
    // u = the polynomial of the published `scaled` (which is u itself under Jacobi), published.
    auto precondition = [&]() {
        if (!CHEB) return;
        double before[R], ax[R];
#pragma unroll
        for (int i = 0; i < R; ++i) u[i] = before[i] = scaled[i];
        for (int index = 0; index < kChebyshevDegree - 1; ++index) {
            const double4 st = steps[index];
            const double slope = st.w * st.x;
            double base[R];  // what the step takes from the vectors it has
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const double current = st.x * u[i];
                base[i] = fma(st.w, scaled[i], fma(st.z, current - st.y * before[i], current));
                before[i] = u[i];
            }
            matvec(ax);
#pragma unroll
            for (int i = 0; i < R; ++i) u[i] = fma(-slope * inv[i], ax[i], base[i]);
            publish(u);
            if (!ok) break;
            await_published();
        }
    };

    // -- the start: |b|^2, u published ---------------------------------------------------------
    double rr0 = 0.0, unused0, unused1;
    fold(bb, 0.0, 0.0, 0);
    publish(CHEB ? scaled : u);
    await_published();
    if (FORM == kCluster) await_sums();
    read(rr0, unused0, unused1, 0);
    barrier();  // the sums are read before the next fold writes them
    precondition();
    const double atol_sq = a.tol * a.tol * rr0;
    // 1 / gamma of the last step, formed beside its other division (0: its value has no such inverse).
    double gamma_old = INFINITY, inverse_old = 0.0, denominator_old = 0.0, rr = rr0;
    double settle_previous = 0.0, settle_reach = 0.0, settle_checks = 0.0;
    int round = 0, iterations = 0, status = OB_STATUS_CAPPED;
    bool done = false;
    while (!done) {
        double w[R], ag = 0.0, ad = 0.0, ar = 0.0;
        matvec(w);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            ag = fma(r[i], u[i], ag);
            ad = fma(w[i], u[i], ad);
            ar = fma(r[i], r[i], ar);
        }
        double gamma, delta;
        fold(ag, ad, ar, 0);
        await_sums();
        if (!ok) break;
        read(gamma, delta, rr, 0);
        double alpha = 0.0, beta = 0.0;
        bool step = false;
        if (rr > atol_sq && round <= a.maxiter && gamma != 0.0) {
            // beta gamma / alpha_old of the loop graph, with alpha_old = gamma_old / denominator_old.
            beta = inverse_old != 0.0 ? gamma * inverse_old : gamma / gamma_old;
            const double denominator = delta - beta * beta * denominator_old;
            if (denominator != 0.0) {
                alpha = gamma / denominator;
                const double inverse = 1.0 / gamma;
                step = true;
                inverse_old = gamma > 1e-290 && gamma < 1e290 ? inverse : 0.0;
                gamma_old = gamma;
                denominator_old = denominator;
            }
        }
        iterations += step ? 1 : 0;
        if (!step || round >= a.maxiter) {
            done = true;
            status = !(rr == rr) ? OB_STATUS_NONFINITE
                     : (!step && round <= a.maxiter) ? OB_STATUS_CONVERGED
                                                     : OB_STATUS_CAPPED;
        }
        ++round;
        if (step) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                if constexpr (kFar) {
                    double* at = far + i * T + tid;
                    const double pn = fma(beta, at[S], u[i]), sn = fma(beta, at[2 * S], w[i]);
                    at[S] = pn;
                    at[2 * S] = sn;
                    at[0] = fma(alpha, pn, at[0]);
                    r[i] = fma(-alpha, sn, r[i]);
                } else {
                    p[i] = fma(beta, p[i], u[i]);
                    s[i] = fma(beta, s[i], w[i]);
                    x[i] = fma(alpha, p[i], x[i]);
                    r[i] = fma(-alpha, s[i], r[i]);
                }
                scaled[i] = inv[i] * r[i];
                if (!CHEB) u[i] = scaled[i];
            }
        }
        if (done) break;
        const bool check = !kFar && a.check_rounds > 0 && round % a.check_rounds == 0;
        if constexpr (!kFar) if (check) {
            double change = 0.0, reached = 0.0;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                if (x[i] != 0.0) {
                    change = fmax(change, fabs(x[i] - previous[i]) / fabs(x[i]));
                    reached += 1.0;
                }
                previous[i] = x[i];
            }
            fold(change, reached, 0.0, 1);
        }
        publish(CHEB ? scaled : u);
        if (!ok) break;
        await_published();
        if (FORM == kCluster && check) await_sums();
        if ((FORM == kGrid || check) && !ok) break;
        if (check) {
            double change, reached;
            read(change, reached, unused0, 1);
            settle_checks += 1.0;
            if (reached + 1.0 != settle_previous) {
                settle_previous = reached + 1.0;
                settle_reach = settle_checks;
            } else if (change < a.change_tolerance ||
                       (settle_checks - settle_reach) * (double)a.check_rounds >= (double)a.settle_rounds) {
                done = true;
                status = change < a.change_tolerance ? OB_STATUS_SETTLED : OB_STATUS_SETTLE_BOUND;
            }
            if (FORM == kBlock) __syncthreads();  // the scratch is read before the next fold
        }
        if (!done) precondition();
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int row = cta * S + i * T + tid;
        if (row < a.n) a.x[row] = kFar ? far[i * T + tid] : x[kFar ? 0 : i];
    }
    if (cta == 0 && tid == 0) {
        a.state->round = round;
        a.state->iterations = iterations;
        a.state->done = 1;
        a.state->status = status;
        a.scalars->rr = rr;
        a.scalars->rr0 = rr0;
    }
    if (!ok) {
        atomicExch(a.abort, 1);
        atomicExch(a.gave_up, 1);
    }
    if (FORM == kCluster) {
        cluster_barrier();  // no CTA leaves while another may still read its memory
        // Where every CTA waited for what was pushed to it, nothing is on its way any more. After a wait
        // that was given up, pushes may be, and their sender cannot wait for them: none is sent past
        // the barrier, and the CTAs stay for about 100 us, where a store to shared memory takes one.
        if (*(volatile int*)a.abort != 0) {
            const long long start = clock64();
            while (clock64() - start < 200000) {
            }
            cluster_barrier();
        }
    }
}

}  // namespace
}  // namespace ob
