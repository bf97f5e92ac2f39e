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
//             icosphere, whose edge rows read nothing local. Where a halo does not quite fit, or a
//             CTA would push to one it does not read, the whole cluster gathers so, between
//             barrier.clusters; where far more is missing, the launch declines and the host takes
//             the grid.)
//   kGrid     up to one CTA an SM (a cooperative launch): global memory at L2, an arrival counter
//             between phases.
//
// Every wait is bounded: a CTA that gives up raises `abort`, the others then give up as well, and
// `gave_up` stays set until the host has reported OB_ERR_TIMEOUT. A round's float64 chain is kept short
// (two partial sums a row, one division behind the dots), since latency is what is left: the sums a
// row and the scalars agree with the loop graph's to rounding. The dots are folded thread, warp, CTA
// in a fixed order, so every run gives the same bits.
//
// Rows past the seven entries of a regular mesh (a scan has vertices of 7 to 20 neighbours, a pole any
// number) have a few more in place where many of a warp's rows have them; the rest is a list, whose
// entries all lanes of the warp take.
#pragma once

#include <type_traits>

#include "ob_internal.cuh"

namespace ob {
namespace {

enum ResidentForm : int { kBlock = 0, kCluster = 1, kGrid = 2 };
constexpr int kClusterMax = 16;
constexpr int kHalo = 1024;      // other CTAs' values a cluster CTA holds copies of
constexpr int kHaloTable = 2048; // the hash table that numbers them
constexpr int kPushesARow = 4;   // a CTA's push list, of its rows (two rows a thread; half at four)
constexpr int kBaseEntries = 7;  // a regular mesh's rows: every row is padded to it
// The most entries a row has in place, of a system's `mean`: the longest row's where the CTA's gathers are
// local, the mean's in the grid, whose loads in flight need the L1 that shared memory leaves (rows in
// random order, us a Chebyshev round at 64 and at 8: 140 000 rows 115 and 81).
constexpr int most_in_place(int form, int mean) { return form == kGrid ? mean : mean < 8 ? 16 : 2 * mean + 2; }
constexpr int kProducts = 64;    // of those, a warp's products at a time
constexpr int kLaneEntries = 16; // a row's listed entries that its own thread lists
// Values a CTA of a cluster may gather from the others, in place of a copy, before the launch leaves the
// system to the grid. Rows of a triangulation in random order, us a settle round / a Chebyshev one,
// cluster and grid: 5 000 rows (some 600 such values a CTA) 5.6 / 44 and 6.8 / 50, 6 000 7.0 / 53 and
// 6.7 / 51, 8 000 (1 500) 8.2 / 69 and 6.8 / 50, 10 000 10 / 84 and 7.3 / 52.
constexpr int kMayLose = 768;
// The same for the grid's four-row polynomial form where its shared memory leaves less than this of the
// 256 KB it has with L1: lines of 16 values a warp's gather reads on average (2 or 3 where rows lie in
// order, 31 in random order, which took 152 us a round of 200 000 rows where the loop graph takes 120;
// 94 and 106 at 160 000, whose shared memory leaves 100 KB).
constexpr size_t kScatterLeaves = 80 << 10;
constexpr int kMayScatter = 16;
constexpr int kDeclined = -1;    // LoopState::status of a launch that left the system to another form
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
    int width;   // entries a row has in place, at most, those in registers among them
    int more;    // entries past those that a CTA's list holds on the chip
    int pushes;  // kCluster: the capacity of a CTA's push list
    int polls;   // before a wait gives up
    int* abort;  // 1 when a wait gave up (zero at the launch of kGrid, zeroed by the others)
    int* gave_up;  // the same, but not zeroed by a launch
    int* scattered;  // kGrid: lines read by gathers (zero at the launch), null where the launch does not decline
    // The lists of the CTAs that have more of them: nnz entries, and R + 1 bounds a thread.
    double* more_values;
    unsigned* more_places;
    int* more_rows;
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
    // partial sums (two rows of three values a CTA), the warps' (one), three totals, the entries in
    // place past the registers' (values, places), the warps' products and the list of further entries
    // (values, places, the warps' and the rows' bounds), the push list and the halo's table (in a
    // cluster the products' place once the set-up is over).
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
    const int held = a.width - E;  // entries in place that lie in shared memory
    double* own_products = vals + (size_t)held * S;
    double* list_values = own_products + (FORM == kCluster ? 0 : kProducts * warps);
    int2* push = reinterpret_cast<int2*>(list_values + a.more);  // (own row, address); kCluster
    int* table = reinterpret_cast<int*>(push + (FORM == kCluster ? a.pushes : 0));
    int* table_slot = table + (FORM == kCluster ? kHaloTable : 0);
    // Halo values, pushes, the most values a CTA has no copy of, the CTAs read, this CTA's such values.
    int* counters = table_slot + (FORM == kCluster ? kHaloTable : 0);
    unsigned* places = reinterpret_cast<unsigned*>(counters + 8);
    unsigned* list_places = places + (size_t)held * S;
    int* list_warps = reinterpret_cast<int*>(list_places + a.more);  // each warp's first and last, in the CTA's
    int* list_rows = list_warps + 2 * 16 + 1;                        // (then whether the list lies here)
    double* products = (FORM == kCluster ? reinterpret_cast<double*>(table) : own_products) + kProducts * warp;
    static_assert(sizeof(double) * kProducts * 16 <= 2 * sizeof(int) * kHaloTable, "the table holds the products");
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
    double bb = 0.0;
    // A warp's rows have `span` entries in place, and every shorter row is padded to it with zero entries
    // on a live row: as many as the longest has where the gathers are local (a further entry a row is
    // then cheaper than the list), otherwise as many as half of the rows have. What longer rows have past
    // that is the warp's list, `listed` entries: in shared memory where the CTA's fit, otherwise in global
    // memory (consecutive, read at L2).
    int span = kBaseEntries, listed = 0;
    bool long_rows, lists;  // whether any row of the CTA has more than its base entries in place, and listed
    auto list = [&](double*& list_v, unsigned*& list_p, int*& bounds) {
        const bool here = list_warps[2 * 16] != 0;
        const size_t base = here ? 0 : (size_t)a.offsets[cta * S];  // entries of the CTAs before
        const int first = list_warps[2 * warp];
        list_v = (here ? list_values : a.more_values + base) + first;
        list_p = (here ? list_places : a.more_places + base) + first;
        bounds = (here ? list_rows : a.more_rows + (size_t)cta * T * (R + 1)) + tid * (R + 1);
    };
    {
        double ax[R];
        int from[R], length[R];
        int longest = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int row = cta * S + i * T + tid;
            const bool live = row < a.n;
            from[i] = live ? a.offsets[row] : 0;
            length[i] = live ? a.offsets[row + 1] - from[i] : 0;
            longest = max(longest, length[i]);
        }
        longest = __reduce_max_sync(0xffffffffu, longest);
        if (FORM != kGrid && longest <= a.width) {
            span = max(span, longest);
        } else {
            for (; span < min(longest, a.width); ++span) {
                int have = 0;
#pragma unroll
                for (int i = 0; i < R; ++i) have += __popc(__ballot_sync(0xffffffffu, length[i] > span));
                if (have < 16 * R) break;
            }
        }
        int mine = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const unsigned self = (unsigned)min(cta * S + i * T + tid, a.n - 1);
            auto entry = [&](int e, double& v, unsigned& at) {
                const bool has = e < length[i];
                at = has ? (unsigned)a.columns[from[i] + e] : self;
                v = has ? a.values[from[i] + e] : 0.0;
                if (has) ax[i] = fma(v, a.x[at], ax[i]);
                v = a.narrow ? (double)(float)v : v;
            };
            ax[i] = 0.0;
#pragma unroll
            for (int e = 0; e < E; ++e) entry(e, value[e][i], place[e][i]);
            for (int e = E; e < span; ++e)
                entry(e, vals[((e - E) * R + i) * T + tid], places[((e - E) * R + i) * T + tid]);
            mine += max(0, length[i] - span);
        }
        // Where the thread's listed entries start: the lanes' counts scanned, then the warps'.
        int before = mine;
#pragma unroll
        for (int step = 1; step < 32; step *= 2) {
            const int below = __shfl_up_sync(0xffffffffu, before, step);
            if (lane >= step) before += below;
        }
        int* of_warps = reinterpret_cast<int*>(scratch);
        listed = __shfl_sync(0xffffffffu, before, 31);
        if (lane == 0) of_warps[warp] = listed;
        long_rows = __syncthreads_or(span > kBaseEntries);
        lists = __syncthreads_or(listed);
        if (lists) {
            int all = 0, first = 0;
            for (int w = 0; w < warps; ++w) {
                first += w < warp ? of_warps[w] : 0;
                all += of_warps[w];
            }
            if (lane == 0) {
                list_warps[2 * warp] = first;
                list_warps[2 * warp + 1] = first + listed;
                if (warp == 0) list_warps[2 * 16] = all <= a.more;
            }
            __syncthreads();
        }
        if (listed) {
            double* list_v;
            unsigned* list_p;
            int* bounds;
            list(list_v, list_p, bounds);
            int at = before - mine;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int past = max(0, length[i] - span);
                bounds[i] = at;
                if (past <= kLaneEntries) {
                    for (int e = 0; e < past; ++e) {
                        const int col = a.columns[from[i] + span + e];
                        const double v = a.values[from[i] + span + e];
                        ax[i] = fma(v, a.x[col], ax[i]);
                        list_v[at + e] = a.narrow ? (double)(float)v : v;
                        list_p[at + e] = (unsigned)col;
                    }
                }
                // A long row by the whole warp.
                for (unsigned left = __ballot_sync(0xffffffffu, past > kLaneEntries); left; left &= left - 1) {
                    const int of = __ffs(left) - 1;
                    const int start = __shfl_sync(0xffffffffu, from[i], of) + span;
                    const int to = __shfl_sync(0xffffffffu, at, of), count = __shfl_sync(0xffffffffu, past, of);
                    double part = 0.0;
                    for (int e = lane; e < count; e += 32) {
                        const int col = a.columns[start + e];
                        const double v = a.values[start + e];
                        part = fma(v, a.x[col], part);
                        list_v[to + e] = a.narrow ? (double)(float)v : v;
                        list_p[to + e] = (unsigned)col;
                    }
                    part = warp_sum(part);
                    if (lane == of) ax[i] += part;
                }
                at += past;
            }
            bounds[R] = at;
            __syncwarp();  // other lanes' entries are read below
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int row = cta * S + i * T + tid;
            const bool live = row < a.n;
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
            r[i] = live ? b - ax[i] : 0.0;
            inv[i] = live ? a.inv_diag[row] : 0.0;
            scaled[i] = u[i] = inv[i] * r[i];
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
        if (tid < 8) counters[tid] = 0;
        if (tid == 0) {
            for (unsigned b = 0; b < 4; ++b) arrivals_init(bars_at + 8u * b);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        for (int i = tid; i < 2 * kHalo; i += T) pub[(i / kHalo) * buffer + S + i % kHalo] = 0.0;
        cluster_barrier();  // every CTA of the cluster runs, its table, counters and barriers are ready
        int lost = 0;
        unsigned from = 0;  // the CTAs this one holds copies from
#pragma unroll
        for (int i = 0; i < R; ++i) {
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (!mine((int)place[e][i])) lost += find((int)place[e][i], true) < 0;
            for (int e = E; e < span; ++e) {
                const int col = (int)places[((e - E) * R + i) * T + tid];
                if (!mine(col)) lost += find(col, true) < 0;
            }
        }
        if (listed) {
            double* list_v;
            unsigned* list_p;
            int* bounds;
            list(list_v, list_p, bounds);
            for (int q = lane; q < listed; q += 32)
                if (!mine((int)list_p[q])) lost += find((int)list_p[q], true) < 0;
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
            lost += taken < 0;
        }
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
        if (lane == 0 && (to_whom & ~(unsigned)counters[3])) ++lost;
        lost = __reduce_add_sync(0xffffffffu, lost);
        if (lane == 0 && lost) atomicAdd(&counters[4], lost);
        __syncthreads();
        if (counters[4] && warp == 0 && lane < ctas)
            asm volatile("red.shared::cluster.max.s32 [%0], %1;" ::"r"(cluster_address(shared_address(counters + 2), lane)),
                         "r"(counters[4])
                         : "memory");
        cluster_barrier();
        pulls = counters[2] != 0;
        if (counters[2] > kMayLose) {
            // Every CTA leaves here: none reads or writes another's memory past the barrier.
            if (cta == 0 && tid == 0) a.state->status = kDeclined;
            return;
        }
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
    if (listed) {
        double* list_v;
        unsigned* list_p;
        int* bounds;
        list(list_v, list_p, bounds);
        for (int q = lane; q < listed; q += 32) list_p[q] = place_of((int)list_p[q]);
        __syncwarp();
    }

    // (Grid: the lines that a gather of the base entries reads, counted over all CTAs by the first barrier.)
    const bool weighs = FORM == kGrid && kFar && a.scattered != nullptr;
    if (weighs) {
        int lines = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            for (int e = 0; e < kBaseEntries; ++e) {
                const unsigned line = places[(e * R + i) * T + tid] >> 4;
                const unsigned same = __match_any_sync(0xffffffffu, line);
                lines += __popc(__ballot_sync(0xffffffffu, __ffs(same) - 1 == lane));
            }
        }
        if (lane == 0) atomicAdd(a.scattered, lines);
    }

    // The solve, in three copies: a CTA runs one without the code for the kinds of entries it does not have
    // (beside which a cluster's Chebyshev round of 5 000 regular rows took 15.2 us, not 11.7).
    double rr0 = 0.0, rr = 0.0;
    int round = 0, iterations = 0, status = OB_STATUS_CAPPED;
    bool declined = false;
    auto solve = [&](auto kinds) {
        constexpr int kKinds = decltype(kinds)::value;
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
                for (int first = 0; first < R; first += 2) {
                    double u_of[2][kBaseEntries];
#pragma unroll
                    for (int i = first; i < first + 2; ++i)
#pragma unroll
                        for (int e = 0; e < kBaseEntries; ++e) u_of[i - first][e] = gather(places[(e * R + i) * T + tid]);
#pragma unroll
                    for (int i = first; i < first + 2; ++i) {
                        double even = 0.0, odd = 0.0;
#pragma unroll
                        for (int e = 0; e < kBaseEntries; ++e) {
                            const double v = vals[(e * R + i) * T + tid];
                            if (e & 1) odd = fma(v, u_of[i - first][e], odd);
                            else even = fma(v, u_of[i - first][e], even);
                        }
                        out[i] = even + odd;
                    }
                }
            }
            if constexpr (kKinds >= 1) {
                for (int e = kBaseEntries; e < span; ++e) {
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const int at = ((e - E) * R + i) * T + tid;
                        out[i] = fma(vals[at], gather(places[at]), out[i]);
                    }
                }
            }
            // The listed entries: a lane an entry, then each row its own products in order.
            if constexpr (kKinds == 2) {
                if (listed) {
                    double* list_v;
                    unsigned* list_p;
                    int* bounds;
                    list(list_v, list_p, bounds);
                    for (int from = 0; from < listed; from += kProducts) {
                        double v[kProducts / 32], u_of[kProducts / 32];
#pragma unroll
                        for (int h = 0; h < kProducts / 32; ++h) {
                            const int q = min(from + 32 * h + lane, listed - 1);
                            v[h] = list_v[q];
                            u_of[h] = gather(list_p[q]);
                        }
#pragma unroll
                        for (int h = 0; h < kProducts / 32; ++h) products[32 * h + lane] = v[h] * u_of[h];
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < R; ++i) {
                            const int end = min(bounds[i + 1] - from, kProducts);
#pragma unroll 4
                            for (int q = max(bounds[i] - from, 0); q < end; ++q) out[i] += products[q];
                        }
                        __syncwarp();
                    }
                }
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
        double unused0, unused1;
        fold(bb, 0.0, 0.0, 0);
        publish(CHEB ? scaled : u);
        await_published();
        if (FORM == kCluster) await_sums();
        if (weighs && ok && *(volatile int*)a.scattered > kMayScatter * kBaseEntries * R * warps * ctas) {
            declined = true;
            return;
        }
        read(rr0, unused0, unused1, 0);
        barrier();  // the sums are read before the next fold writes them
        precondition();
        const double atol_sq = a.tol * a.tol * rr0;
        // 1 / gamma of the last step, formed beside its other division (0: its value has no such inverse).
        double gamma_old = INFINITY, inverse_old = 0.0, denominator_old = 0.0;
        rr = rr0;
        double settle_previous = 0.0, settle_reach = 0.0, settle_checks = 0.0;
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
    };
    if (lists) solve(std::integral_constant<int, 2>{});
    else if (long_rows) solve(std::integral_constant<int, 1>{});
    else solve(std::integral_constant<int, 0>{});
    if (declined) {
        if (cta == 0 && tid == 0) a.state->status = kDeclined;
        return;
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
