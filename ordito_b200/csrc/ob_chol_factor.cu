// a11: the numeric sparse Cholesky factorisation on the device.
//
// Follows ordito/cholesky.py:1399 _factor (kernels/cholesky.py:434 factor_panel_tiled, :541
// panel_front_product, :591 update_panel_entries, :772-839 factor_front_panels /
// factor_level_panels): multifrontal over the dissection tree, one tree level at a time, every
// front of a level in the same launches. A front is the dense m x m matrix of a supernode's nc own
// columns and noff off-diagonal rows (m = nc + noff), column-major in one arena: it receives the
// operator's entries of its own columns (scattered once, for every front, before the first level)
// and its children's Schur complements (extend-add, child by child in a fixed order, so every
// front entry is summed in the same order on every run: no atomics). Its own columns are then
// eliminated in panels of 64:
//
//   K1  the panel's diagonal block D (b x b, b <= 64): Cholesky and its inverse D^-1, in registers
//       (one CTA a front); D^-1 goes straight into the stored block.
//   K2  the panel below the diagonal, L = F D^-T (in place), and the rows of the panel in the
//       stored block, Z_p = D^-1 Z_p (in place).
//   K3  the trailing update, F[j1:, j1:] -= L L^T (lower tiles), and Z[j1:, :j1] -= L Z_p.
//
// Z is the supernode's stored block [L11^-1; G] with G = -L21 L11^-1 -- the first nc columns of
// the inverse of [L11 0; L21 I], which forward elimination of [I; 0] builds panel by panel
// alongside the factorisation, so the partitioned inverse the solves read (ordito/cholesky.py
// notes: Alvarado, Pothen and Schreiber 1993) costs no separate pass. After the last panel the
// front's trailing block is the Schur complement its parent takes. K2 and K3 are batched float64
// tensor-core products (mma.sync m8n8k4) over 64 x 64 output tiles with an inner dimension of one
// panel; the whole schedule (every level's extend-add ranks, panels and tile lists) depends only
// on the analysis, so it is built once per analysis and kept.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ob_chol.cuh"
#include "ob_host.hpp"
#include "ob_scratch.cuh"

namespace ob {

namespace {

constexpr int kPanel = 64;         // columns eliminated a panel step; tile edge of K2 / K3
constexpr int kDiagThreads = 256;
constexpr int kTileThreads = 128;  // four warps, each a 16-row strip of the 64 x 64 output
constexpr int kSmemLd = kPanel + 4;
constexpr int kTileSmem = 2 * kPanel * kSmemLd * (int)sizeof(double);
constexpr int kExtendThreads = 256;
constexpr int kExtendColumns = 32;  // child columns an extend-add task takes
constexpr int kExtendFew = 8;       // where a launch would have too few tasks
// A row's entries sum to "zero" below this fraction of its diagonal (ordito/cholesky.py:76).
constexpr double kSingularRowSum = 1e-10;

// Extend-add: the child's Schur complement columns [b0, b1) added into its parent's front.
struct ExtendTask {
    int child, parent, b0, b1;
};

// One panel of one front: its front (offset f, leading dimension fld, m rows), its stored block
// (offset z, leading dimension zld), the panel's first column j0 and width b. K1 takes one task a
// CTA; K2 and K3 take 64 x 64 output tiles of [j1, m), j1 = j0 + b, numbered within the task from
// its first tile of the launch: K2 the row tiles of the panel below the diagonal, then the column
// tiles of the stored block's panel rows; K3 the lower tiles of the trailing front (column by
// column), then the tiles of the stored block below (row by row).
struct StepTask {
    long long f, z;
    int fld, zld, m, j0, b;
    int first_panel, first_trailing;
    int pad;
};

enum LaunchKind : int { kExtend = 0, kDiag = 1, kPanelProduct = 2, kTrailing = 3 };

}  // namespace

struct FactorPlan {
    int device = -1;
    long long front_total = 0;  // doubles in the front arena
    long long n_entries = 0;    // CSR entries of the operator
    // Per CSR entry (old numbering): its slot in the fronts (-1: the upper triangle, which the
    // lower one mirrors) and the new indices of its row and column.
    long long* entry_dest = nullptr;
    int2* entry_rc = nullptr;
    long long* diag_dest = nullptr;  // per new row: its diagonal slot in its front
    int* diag_pos = nullptr;         // per old row: the CSR position of its diagonal, or -1
    int* component = nullptr;        // per old row
    char* component_last = nullptr;  // per old row
    int* perm = nullptr;             // new -> old
    int* iperm = nullptr;            // old -> new
    int* node_of = nullptr;          // per new column: its supernode
    int* offsets = nullptr;          // the operator's row offsets (old numbering)
    // Per supernode: front offset, front leading dimension, own columns, off-diagonal rows, and
    // where its off-diagonal rows' positions in its parent's front start in `rel`.
    long long* front_at = nullptr;
    int* fld = nullptr;
    int* nc = nullptr;
    int* noff = nullptr;
    int* rel_at = nullptr;
    int* rel = nullptr;
    int* rows = nullptr;  // the off-diagonal rows themselves, starting as in `rel`
    // Per supernode: first column, parent, and where a factor's row lists of it start (BlockLayout).
    int* start = nullptr;
    int* parent = nullptr;
    int* rows_at = nullptr;
    int n_nodes = 0;
    struct Launch {
        int kind;
        const void* tasks;
        const int* owner;  // K2 / K3: each tile's task
        int count;
    };
    std::vector<Launch> launches;  // the whole numeric schedule, in order
    std::vector<void*> owned;
};

void release_plan(FactorPlan* plan) {
    if (plan == nullptr) return;
    if (!plan->owned.empty()) {
        int current = -1;
        cudaGetDevice(&current);
        if (plan->device >= 0 && plan->device != current) cudaSetDevice(plan->device);
        {
            std::lock_guard<std::recursive_mutex> guard(capture_mutex());
            cudaDeviceSynchronize();
        }
        for (void* p : plan->owned) cudaFree(p);
        if (current >= 0 && plan->device >= 0 && plan->device != current) cudaSetDevice(current);
    }
    delete plan;
}

namespace {

template <typename T>
int upload(FactorPlan* P, T** out, const std::vector<T>& host, cudaStream_t stream) {
    void* p = nullptr;
    OB_CUDA(pool_malloc(&p, sizeof(T) * std::max<size_t>(host.size(), 1), stream));
    P->owned.push_back(p);
    if (!host.empty())
        OB_CUDA(cudaMemcpyAsync(p, host.data(), sizeof(T) * host.size(), cudaMemcpyHostToDevice, stream));
    *out = static_cast<T*>(p);
    return OB_OK;
}

template <typename T>
int allocate(FactorPlan* P, T** out, size_t count, cudaStream_t stream) {
    void* p = nullptr;
    OB_CUDA(pool_malloc(&p, sizeof(T) * std::max<size_t>(count, 1), stream));
    P->owned.push_back(p);
    *out = static_cast<T*>(p);
    return OB_OK;
}

template <typename T>
int upload_scratch(Scratch& scratch, const T** out, const std::vector<T>& host, cudaStream_t stream) {
    T* p = scratch.take<T>(host.size());
    if (int st = scratch.commit()) return st;
    if (!host.empty())
        OB_CUDA(cudaMemcpyAsync(p, host.data(), sizeof(T) * host.size(), cudaMemcpyHostToDevice, stream));
    *out = p;
    return OB_OK;
}

// The tree as the plan kernels read it: per supernode its first column, own columns, front
// offset and leading dimension, and its off-diagonal rows (ascending) at rows + row_at[s] ..
// row_at[s + 1]; per new column its supernode.
struct PlanTree {
    const int* start;
    const int* nc;
    const long long* front_at;
    const int* fld;
    const int* row_at;
    const int* rows;
    const int* node_of;
};

// Row r's position in supernode s's front: its own column r - start, else nc + its index among
// the off-diagonal rows (which hold r: the symbolic structure puts it there).
__device__ __forceinline__ int front_position(const PlanTree& T, int s, int r) {
    const int start = T.start[s], count = T.nc[s];
    if (r < start + count) return r - start;
    int lo = T.row_at[s], hi = T.row_at[s + 1];
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (T.rows[mid] < r) lo = mid + 1;
        else hi = mid;
    }
    return count + (lo - T.row_at[s]);
}

// node_of[j] = s for each own column j of supernode s (a warp a supernode).
__global__ void node_of_kernel(int ns, const int* __restrict__ start, const int* __restrict__ nc, int* node_of) {
    const int s = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
    if (s >= ns) return;
    for (int j = threadIdx.x & 31; j < nc[s]; j += 32) node_of[start[s] + j] = s;
}

// Per CSR entry e of old row ro (a group of 8 lanes a row): its new (row, column) and its slot
// in the front of its row's supernode (-1 in the upper triangle, which the lower one mirrors);
// per old row the CSR position of its diagonal (left -1 when it has none).
constexpr int kEntryLanes = 8;
__global__ void entries_kernel(int n, const int* __restrict__ offsets, const int* __restrict__ columns,
                               const int* __restrict__ iperm, const PlanTree T, long long* __restrict__ dest,
                               int2* __restrict__ rc, int* __restrict__ diag_pos) {
    const long long lane_id = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int ro = (int)(lane_id / kEntryLanes);
    if (ro >= n) return;
    const int lane = (int)(lane_id % kEntryLanes);
    const int j = iperm[ro];
    const int s = T.node_of[j];
    const long long column_at = T.front_at[s] + (long long)(j - T.start[s]) * T.fld[s];
    for (int e = offsets[ro] + lane; e < offsets[ro + 1]; e += kEntryLanes) {
        const int co = columns[e];
        const int r = iperm[co];
        rc[e] = make_int2(j, r);
        if (co == ro) diag_pos[ro] = e;
        dest[e] = r < j ? -1LL : column_at + front_position(T, s, r);
    }
}

// rel: each child's off-diagonal rows as positions in its parent's front (a warp a supernode;
// a root's entries are left unset: nothing reads them).
__global__ void rel_kernel(int ns, const int* __restrict__ parent, const PlanTree T, int* __restrict__ rel) {
    const int s = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
    if (s >= ns || parent[s] < 0) return;
    for (int i = T.row_at[s] + (threadIdx.x & 31); i < T.row_at[s + 1]; i += 32)
        rel[i] = front_position(T, parent[s], T.rows[i]);
}

// Each new column's diagonal slot in its supernode's front.
__global__ void diag_dest_kernel(int n, const PlanTree T, long long* __restrict__ diag_dest) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int s = T.node_of[j];
    const long long lj = j - T.start[s];
    diag_dest[j] = T.front_at[s] + lj * T.fld[s] + lj;
}

// A factor's tables (a warp a supernode): its numbering, its rows' supernodes and the supernodes'
// parents, then its row lists: a supernode's off-diagonal rows (rows of B), then the backward product's
// inputs, its own rows of Y and its off-diagonal rows of X, in the stacked [B; Y; X]. The host filled
// and uploaded these before (as much as 60 MB at 2.6 M vertices), and made the tile lists after the
// factorisation instead of beside it: a factor of the 2.6 M-vertex torus took 102 ms where it now
// takes 57, of the 131k torus 3.81 and 3.08. (One launch: with four copies beside it the two factors of
// six vertices took 174 us, so 141.)
__global__ void factor_tables_kernel(int ns, int n, const int* __restrict__ start, const int* __restrict__ nc,
                                     const int* __restrict__ row_at, const int* __restrict__ rows,
                                     const int* __restrict__ rows_at, const int* __restrict__ old_of,
                                     const int* __restrict__ parent_of, const FactorTables to) {
    const int s = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (s >= ns) return;
    const int count = nc[s], own = start[s], first = row_at[s], noff = row_at[s + 1] - first;
    if (lane == 0) to.parent[s] = parent_of[s];
    int* off = to.idx + rows_at[s];
    int* back = off + noff;
    for (int i = lane; i < count; i += 32) {
        const int old = old_of[own + i];
        to.perm[own + i] = old;
        to.iperm[old] = own + i;
        to.node_of[own + i] = s;
        back[i] = n + own + i;
    }
    for (int i = lane; i < noff; i += 32) {
        const int r = rows[first + i];
        off[i] = r;
        back[count + i] = 2 * n + r;
    }
}

// The device tables and the launch schedule of an analysis (once). The per-entry and per-row
// tables are built on the device from the tree; the host builds the launch schedule.
int build_plan(const CholAnalysis& A, FactorPlan* P, cudaStream_t stream) {
    const int n = A.n, ns = (int)A.nodes.size();
    const BlockLayout layout = block_layout(A);
    // Front arena: node s is m x m column-major at front_at[s], leading dimension fld (m rounded
    // up to 8 doubles, so every front column starts on 64 bytes).
    std::vector<long long> front_at(ns);
    std::vector<int> fld(ns), nc(ns), noff(ns), start(ns), parent(ns), row_at(ns + 1, 0);
    long long total = 0;
    for (int s = 0; s < ns; ++s) {
        const CholNode& nd = A.nodes[s];
        nc[s] = nd.count;
        start[s] = nd.start;
        parent[s] = nd.parent;
        noff[s] = (int)nd.off_rows.size();
        row_at[s + 1] = row_at[s] + noff[s];
        const int m = nc[s] + noff[s];
        fld[s] = (m + 7) / 8 * 8;
        front_at[s] = total;
        total += (long long)fld[s] * m;
    }
    P->front_total = total;
    std::vector<int> rows(row_at[ns]);
    parallel_range(ns, row_at[ns] > (1 << 18), [&](long long lo, long long hi) {
        for (long long s = lo; s < hi; ++s)
            std::copy(A.nodes[s].off_rows.begin(), A.nodes[s].off_rows.end(), rows.begin() + row_at[s]);
    });
    std::vector<char> component_last(n);
    for (int i = 0; i < n; ++i) component_last[i] = (char)A.component_last[i];
    const long long nnz = A.offsets[n];
    P->n_entries = nnz;
    P->n_nodes = ns;
    int st = OB_OK;
    if ((st = upload(P, &P->component, A.component, stream)) ||
        (st = upload(P, &P->component_last, component_last, stream)) ||
        (st = upload(P, &P->perm, A.perm, stream)) || (st = upload(P, &P->iperm, A.iperm, stream)) ||
        (st = upload(P, &P->offsets, A.offsets, stream)) || (st = upload(P, &P->start, start, stream)) ||
        (st = upload(P, &P->parent, parent, stream)) || (st = upload(P, &P->rows, rows, stream)) ||
        (st = upload(P, &P->rows_at, layout.rows_at, stream)) || (st = allocate(P, &P->node_of, (size_t)n, stream)) ||
        (st = upload(P, &P->front_at, front_at, stream)) ||
        (st = upload(P, &P->fld, fld, stream)) || (st = upload(P, &P->nc, nc, stream)) ||
        (st = upload(P, &P->noff, noff, stream)) || (st = upload(P, &P->rel_at, row_at, stream)) ||
        (st = allocate(P, &P->rel, (size_t)row_at[ns], stream)) ||
        (st = allocate(P, &P->entry_dest, (size_t)nnz, stream)) ||
        (st = allocate(P, &P->entry_rc, (size_t)nnz, stream)) ||
        (st = allocate(P, &P->diag_pos, (size_t)n, stream)) ||
        (st = allocate(P, &P->diag_dest, (size_t)n, stream)))
        return st;
    {
        // The pattern's columns, for the table kernels only.
        Scratch scratch(stream);
        const int* d_columns = nullptr;
        if ((st = upload_scratch(scratch, &d_columns, A.columns, stream))) return st;
        const PlanTree T{P->start, P->nc, P->front_at, P->fld, P->rel_at, P->rows, P->node_of};
        const int threads = 256;
        node_of_kernel<<<ceil_div(32LL * ns, threads), threads, 0, stream>>>(ns, P->start, P->nc, P->node_of);
        OB_CHECK_LAUNCH("chol plan node_of");
        OB_CUDA(cudaMemsetAsync(P->diag_pos, 0xFF, sizeof(int) * (size_t)n, stream));
        entries_kernel<<<ceil_div((long long)kEntryLanes * n, threads), threads, 0, stream>>>(
            n, P->offsets, d_columns, P->iperm, T, P->entry_dest, P->entry_rc, P->diag_pos);
        OB_CHECK_LAUNCH("chol plan entries");
        rel_kernel<<<ceil_div(32LL * ns, threads), threads, 0, stream>>>(ns, P->parent, T, P->rel);
        OB_CHECK_LAUNCH("chol plan rel");
        diag_dest_kernel<<<ceil_div(n, threads), threads, 0, stream>>>(n, T, P->diag_dest);
        OB_CHECK_LAUNCH("chol plan diagonal slots");
        // The scratch is released in stream order, after these kernels.
    }
    // The schedule, level by level.
    std::vector<std::vector<int>> at_level(A.levels);
    for (int s = 0; s < ns; ++s) at_level[A.nodes[s].level].push_back(s);
    std::vector<ExtendTask> extend;
    std::vector<StepTask> steps;
    std::vector<int> owners;
    // Task lists are gathered on the host, then uploaded as one array each.
    struct Pending {
        int kind;
        size_t first, count, owner;
    };
    std::vector<Pending> pending;
    auto add = [&](int kind, size_t first, size_t count, size_t owner) {
        if (count > 0) pending.push_back(Pending{kind, first, count, owner});
    };
    const auto tiles_of = [](int extent) { return (extent + kPanel - 1) / kPanel; };
    for (int l = 0; l < A.levels; ++l) {
        const std::vector<int>& nodes = at_level[l];
        size_t ranks = 0;
        for (int s : nodes) ranks = std::max(ranks, A.nodes[s].children.size());
        for (size_t rank = 0; rank < ranks; ++rank) {
            const size_t first = extend.size();
            long long columns = 0;
            for (int p : nodes)
                if (A.nodes[p].children.size() > rank) columns += noff[A.nodes[p].children[rank]];
            // The top of the tree has few columns, and long ones: a column a warp there.
            const int width = columns < 8LL * kExtendColumns * sm_count() ? kExtendFew : kExtendColumns;
            for (int p : nodes) {
                if (A.nodes[p].children.size() <= rank) continue;
                const int c = A.nodes[p].children[rank];
                for (int b0 = 0; b0 < noff[c]; b0 += width)
                    extend.push_back(ExtendTask{c, p, b0, std::min(noff[c], b0 + width)});
            }
            add(kExtend, first, extend.size() - first, 0);
        }
        int panels = 0;
        for (int s : nodes) panels = std::max(panels, tiles_of(nc[s]));
        for (int panel = 0; panel < panels; ++panel) {
            const int j0 = panel * kPanel;
            const size_t first = steps.size(), k2_first = owners.size();
            size_t k2 = 0, k3 = 0;
            for (int s : nodes) {
                if (nc[s] <= j0) continue;
                StepTask t{};
                t.f = front_at[s];
                t.z = layout.inv_at[s];
                t.fld = fld[s];
                t.zld = layout.ld_at[s];
                t.m = nc[s] + noff[s];
                t.j0 = j0;
                t.b = std::min(kPanel, nc[s] - j0);
                t.first_panel = (int)k2;
                t.first_trailing = (int)k3;
                const size_t below = tiles_of(t.m - j0 - t.b);
                k2 += below + tiles_of(j0);
                k3 += below * (below + 1) / 2 + below * tiles_of(j0 + t.b);
                steps.push_back(t);
            }
            // Each tile's task, counted from the launch's first.
            owners.resize(k2_first + k2 + k3);
            for (size_t i = first; i < steps.size(); ++i) {
                const size_t end2 = i + 1 < steps.size() ? steps[i + 1].first_panel : k2;
                const size_t end3 = i + 1 < steps.size() ? steps[i + 1].first_trailing : k3;
                std::fill(owners.begin() + k2_first + steps[i].first_panel, owners.begin() + k2_first + end2,
                          (int)(i - first));
                std::fill(owners.begin() + k2_first + k2 + steps[i].first_trailing,
                          owners.begin() + k2_first + k2 + end3, (int)(i - first));
            }
            add(kDiag, first, steps.size() - first, 0);
            add(kPanelProduct, first, k2, k2_first);
            add(kTrailing, first, k3, k2_first + k2);
        }
    }
    ExtendTask* d_extend = nullptr;
    StepTask* d_steps = nullptr;
    int* d_owners = nullptr;
    if ((st = upload(P, &d_extend, extend, stream)) || (st = upload(P, &d_steps, steps, stream)) ||
        (st = upload(P, &d_owners, owners, stream)))
        return st;
    for (const Pending& q : pending) {
        const void* base = q.kind == kExtend ? (const void*)(d_extend + q.first) : (const void*)(d_steps + q.first);
        P->launches.push_back(FactorPlan::Launch{q.kind, base, d_owners + q.owner, (int)q.count});
    }
    OB_CUDA(cudaStreamSynchronize(stream));  // the host tables go out of scope
    return OB_OK;
}

// Per old row: whether its entries sum to zero (relative to its diagonal); a component with one
// row that does not is not singular (bad[component] = 1).
__global__ void zero_sum_rows_kernel(int n, const int* __restrict__ offsets, const double* __restrict__ values,
                                     const int* __restrict__ diag_pos, const int* __restrict__ component,
                                     int* __restrict__ bad) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double sum = 0.0;
    for (int e = offsets[r]; e < offsets[r + 1]; ++e) sum += values[e];
    const double d = diag_pos[r] >= 0 ? values[diag_pos[r]] : 0.0;
    if (!(fabs(sum) <= kSingularRowSum * fabs(d))) bad[component[r]] = 1;
}

// Per new row: pinned when its diagonal is missing or zero (an unreferenced vertex), or when it
// is the last row of a component that is pinned (every component, or every singular one). A
// pinned row's front column is the identity's.
__global__ void pin_rows_kernel(int n, const int* __restrict__ perm, const double* __restrict__ values,
                                const int* __restrict__ diag_pos, const int* __restrict__ component,
                                const char* __restrict__ component_last, const int* __restrict__ bad,
                                int mode, const long long* __restrict__ diag_dest, char* __restrict__ pinned,
                                double* __restrict__ fronts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int old = perm[i];
    const double d = diag_pos[old] >= 0 ? values[diag_pos[old]] : 0.0;
    bool pin = d == 0.0;
    if (component_last[old]) {
        if (mode == kPinAll) pin = true;
        if (mode == kPinZeroSum && bad[component[old]] == 0) pin = true;
    }
    pinned[i] = pin ? 1 : 0;
    if (pin) fronts[diag_dest[i]] = 1.0;
}

// The operator's lower-triangle entries into their fronts (rows and columns of pinned rows left
// out), times sign.
__global__ void scatter_entries_kernel(long long nnz, const double* __restrict__ values,
                                       const long long* __restrict__ dest, const int2* __restrict__ rc,
                                       const char* __restrict__ pinned, double sign, double* __restrict__ fronts) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    const long long d = dest[e];
    if (d < 0) return;
    const int2 ij = rc[e];
    if (pinned[ij.x] || pinned[ij.y]) return;
    fronts[d] = sign * values[e];
}

// The schedule's kernels are launched as the one before them starts its last blocks (launch_early)
// and wait here until it has finished, their tasks (the plan's, written before any of them) at hand:
// ~130 dependent launches on the 131k torus, 3.08 ms launched in turn and 2.78 so. What an earlier
// kernel wrote is read through no const __restrict__ pointer, so no such load moves above the wait.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// Extend-add: a warp a child column b, its lanes the rows a >= b of the child's Schur complement
// (contiguous in the child's front), added at the parent's positions rel[a], rel[b]. Bound by the
// trips of those loads and adds: one row in flight a lane and 32 columns a task, whatever the
// launch's columns, took the 131k torus' factorisation 4.14 ms where this takes 3.81.
__global__ void __launch_bounds__(kExtendThreads)
extend_add_kernel(const ExtendTask* __restrict__ tasks, const long long* __restrict__ front_at,
                  const int* __restrict__ fld, const int* __restrict__ nc, const int* __restrict__ noff,
                  const int* __restrict__ rel_at, const int* __restrict__ rel, double* __restrict__ fronts) {
    const ExtendTask t = tasks[blockIdx.x];
    const int cm = noff[t.child], cnc = nc[t.child], cld = fld[t.child], pld = fld[t.parent];
    const double* U = fronts + front_at[t.child];
    double* Pf = fronts + front_at[t.parent];
    const int* r = rel + rel_at[t.child];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    after_previous();
    for (int b = t.b0 + warp; b < t.b1; b += kExtendThreads / 32) {
        const double* src = U + (size_t)(cnc + b) * cld + cnc;
        double* dst = Pf + (size_t)r[b] * pld;
        // Four rows in flight a lane (a column's rows are distinct, and the child's front another).
        int a = b + lane;
        for (; a + 96 < cm; a += 128) {
            int to[4];
            double add[4], was[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) to[q] = r[a + 32 * q], add[q] = src[a + 32 * q];
#pragma unroll
            for (int q = 0; q < 4; ++q) was[q] = dst[to[q]];
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[to[q]] = was[q] + add[q];
        }
        for (; a < cm; a += 32) dst[r[a]] += src[a];
    }
}

// K1: the panel's diagonal block D = L L^T inverted to L^-1, in registers: a 16 x 16 grid of threads,
// each with 16 entries of the block (rows tx + 16 a, columns ty + 16 c) and 16 of the identity
// that forward elimination turns into the inverse (rows ty + 16 a, columns tx + 16 c). The
// eliminations run unnormalised (column j and the inverse's row j leave as they are, the update
// takes 1 / d_j once), so a step's chain is one reciprocal, one multiply-add and one barrier;
// the rows are scaled by d_i^-1/2 at the end. The next column and row are updated and published
// (two buffers) before the rest of a step's update, so the reciprocal of the next pivot runs
// beside it. A step in shared memory with a square root, a division and three barriers took
// 1.3 us (86 us a launch of any size on the 131k torus); this takes 0.2. A pivot that is not
// positive sets *status and is replaced by 1, so the launch completes.
__global__ void __launch_bounds__(kDiagThreads)
diag_block_kernel(const StepTask* __restrict__ tasks, const double* fronts, double* vals,
                  int* __restrict__ status) {
    __shared__ double col[2][kPanel], row[2][kPanel], reciprocal[2], pivot[kPanel];
    __shared__ double lift[kPanel];
    const StepTask t = tasks[blockIdx.x];
    const int b = t.b, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const double* F = fronts + t.f + (long long)t.j0 * t.fld + t.j0;
    after_previous();
    double A[4][4], X[4][4];  // A[a][c]: row tx + 16 a, column ty + 16 c; X[a][c]: row ty + 16 a, column tx + 16 c
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int r = tx + 16 * a, k = ty + 16 * c;
            A[a][c] = (r < b && k <= r) ? F[(size_t)k * t.fld + r] : 0.0;
            X[a][c] = ty + 16 * a == tx + 16 * c ? 1.0 : 0.0;
        }
    // A pivot below 2^-1024 has no reciprocal in range. Rows of such a diagonal are scaled by 2^500, and
    // their columns (exact; a block without any, which is every block of an ordinary operator, is left
    // as it is), and the inverse's columns at the end: D A D = (D L) (D L)^T, L^-1 = (D L)^-1 D.
    // Looking at each step's pivot instead took 3 % of the 131k torus' factorisation, this 0.6 %.
    bool small = false;
#pragma unroll
    for (int a = 0; a < 4; ++a)
        if (tx == ty) {
            const bool lifted = A[a][a] < 0x1p-900 && tx + 16 * a < b;
            lift[tx + 16 * a] = lifted ? 0x1p500 : 1.0;
            small |= lifted;
        }
    small = __syncthreads_or(small);
    if (small) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int a = 0; a < 4; ++a) A[a][c] = A[a][c] * lift[tx + 16 * a] * lift[ty + 16 * c];
    }
    auto take_pivot = [&](int j, double d) {
        const bool bad = !(d > 0.0);
        if (bad) *status = 1;
        d = bad ? 1.0 : d;
        pivot[j] = d;
        reciprocal[j & 1] = 1.0 / d;
    };
    // Publishes column j of the block (zero above the diagonal) and row j of the inverse.
    auto publish = [&](int j, const double (&column)[4], const double (&line)[4]) {
        if (ty == (j & 15)) {
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const int r = tx + 16 * a;
                col[j & 1][r] = r > j ? column[a] : 0.0;
                row[j & 1][r] = line[a];
                if (r == j) take_pivot(j, column[a]);
            }
        }
    };
    {
        const double column[4] = {A[0][0], A[1][0], A[2][0], A[3][0]};
        publish(0, column, X[0]);
    }
    __syncthreads();
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
        for (int jj = 0; jj < 16; ++jj) {
            const int j = 16 * jb + jj;
            if (j >= b) break;
            const double inv = reciprocal[j & 1];
            double cr[4], ck[4], xr[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                cr[a] = col[j & 1][tx + 16 * a];
                ck[a] = col[j & 1][ty + 16 * a] * inv;
                xr[a] = row[j & 1][tx + 16 * a];
            }
            // Column j + 1 and the inverse's row j + 1 first.
            if (j + 1 < b) {
                double column[4], line[4];
                if (jj < 15) {
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        column[a] = fma(-cr[a], ck[jb], A[a][jb]);
                        line[a] = fma(-ck[jb], xr[a], X[jb][a]);
                    }
                } else {
                    const int next = jb < 3 ? jb + 1 : 3;
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        column[a] = fma(-cr[a], ck[next], A[a][next]);
                        line[a] = fma(-ck[next], xr[a], X[next][a]);
                    }
                }
                publish(j + 1, column, line);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    A[a][c] = fma(-cr[a], ck[c], A[a][c]);
                    X[a][c] = fma(-ck[a], xr[c], X[a][c]);
                }
            __syncthreads();
        }
    }
    double* Z = vals + t.z + (long long)t.j0 * t.zld + t.j0;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const int r = ty + 16 * a;
        if (r >= b) continue;
        const double scale = rsqrt(pivot[r]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int k = tx + 16 * c;
            if (k <= r) Z[(size_t)r * t.zld + k] = X[a][c] * scale * (small ? lift[k] : 1.0);
        }
    }
}

__device__ __forceinline__ void copy_async_8(double* to, const double* from, bool take) {
    const unsigned at = (unsigned)__cvta_generic_to_shared(to);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(at), "l"(from), "r"(take ? 8 : 0) : "memory");
}

template <int N>
__device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// K2 (TRAILING false) / K3: one 64 x 64 output tile a CTA, C = or -= A (rows x inner) B (inner x
// cols), inner <= 64. The tile's place in its front follows from its index (StepTask), so the
// schedule holds one int a tile. A and B are staged by 8-byte asynchronous copies (a front's rows
// begin at any column after a short panel) in four groups of 16 inner steps, the products of a
// group running while the later ones arrive; C is fetched with them. Each operand lies in shared
// memory with its contiguous direction contiguous and a leading dimension of 68, in either
// orientation free of bank conflicts in the fragment loads (65 had four lanes to a bank). A tile
// may write the block it reads (the in-place products of K2): every copy has landed before the
// first store; no two tiles of a launch write the same entries, and none reads what another writes.
template <bool TRAILING>
__global__ void __launch_bounds__(kTileThreads, 3)
front_product_kernel(const StepTask* __restrict__ tasks, const int* __restrict__ owner, double* fronts, double* vals) {
    extern __shared__ double smem[];
    double* As = smem;
    double* Bs = smem + kPanel * kSmemLd;
    const StepTask t = tasks[owner[blockIdx.x]];
    const int j1 = t.j0 + t.b, below = (t.m - j1 + kPanel - 1) / kPanel;
    double* F = fronts + t.f;
    double* Z = vals + t.z;
    const long long panel = (long long)t.j0 * t.fld;  // the panel's first column in the front
    const double *A, *B;
    double* C;
    int a_ks, b_ld, c_rs, c_cs, rows, cols;
    bool a_rows = true, b_cols = true;  // A contiguous down its rows, B along its columns (else along inner)
    int q = blockIdx.x - (TRAILING ? t.first_trailing : t.first_panel);
    if (!TRAILING) {
        if (q < below) {
            // L = F D^-T in place: B(kk, c) = D^-1(c, kk).
            const int rb = j1 + q * kPanel;
            A = F + panel + rb;
            a_ks = t.fld;
            B = Z + (long long)t.j0 * t.zld + t.j0;
            b_ld = t.zld;
            b_cols = false;
            C = F + panel + rb;
            c_rs = 1, c_cs = t.fld;
            rows = min(kPanel, t.m - rb), cols = t.b;
        } else {
            // Z_p = D^-1 Z_p in place over columns [0, j0).
            const int cb = (q - below) * kPanel;
            A = Z + (long long)t.j0 * t.zld + t.j0;
            a_ks = t.zld;
            a_rows = false;
            B = Z + (long long)t.j0 * t.zld + cb;
            b_ld = t.zld;
            C = Z + (long long)t.j0 * t.zld + cb;
            c_rs = t.zld, c_cs = 1;
            rows = t.b, cols = min(kPanel, t.j0 - cb);
        }
    } else {
        const int triangle = below * (below + 1) / 2;
        a_ks = t.fld;
        if (q < triangle) {
            // F[rb, cb] -= L[rb] L[cb]^T over the lower tiles, column by column.
            int ct = 0;
            while (q >= below - ct) q -= below - ct, ++ct;
            const int cb = j1 + ct * kPanel, rb = cb + q * kPanel;
            A = F + panel + rb;
            B = F + panel + cb;
            b_ld = t.fld;
            C = F + (long long)cb * t.fld + rb;
            c_rs = 1, c_cs = t.fld;
            rows = min(kPanel, t.m - rb), cols = min(kPanel, t.m - cb);
        } else {
            // Z[rb, cb] -= L[rb] Z_p[:, cb] for rows [j1, m), columns [0, j1).
            q -= triangle;
            const int across = (j1 + kPanel - 1) / kPanel;
            const int rb = j1 + (q / across) * kPanel, cb = (q % across) * kPanel;
            A = F + panel + rb;
            B = Z + (long long)t.j0 * t.zld + cb;
            b_ld = t.zld;
            C = Z + (long long)rb * t.zld + cb;
            c_rs = t.zld, c_cs = 1;
            rows = min(kPanel, t.m - rb), cols = min(kPanel, j1 - cb);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wr = warp * 16, fr = lane >> 2, fk = lane & 3;
    // Shared strides of the operands: (row, inner) of A and (inner, column) of B.
    const int a_i = a_rows ? 1 : kSmemLd, a_k = a_rows ? kSmemLd : 1;
    const int b_k = b_cols ? kSmemLd : 1, b_c = b_cols ? 1 : kSmemLd;
    const int groups = (t.b + 15) / 16;
    after_previous();
    const int x = threadIdx.x & 63, y = threadIdx.x >> 6;       // across: 64 outer x 2 inner a step
    const int k = threadIdx.x & 15, outer = threadIdx.x >> 4;   // along: 16 inner x 8 outer a step
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        if (g < groups) {
#pragma unroll
            for (int step = 0; step < 8; ++step) {
                if (a_rows) {
                    const int kk = 16 * g + 2 * step + y;
                    const bool in = x < rows && kk < t.b;
                    copy_async_8(As + kk * kSmemLd + x, in ? A + (long long)kk * a_ks + x : A, in);
                } else {
                    const int kk = 16 * g + k, i = 8 * step + outer;
                    const bool in = i < rows && kk < t.b;
                    copy_async_8(As + i * kSmemLd + kk, in ? A + (long long)i * a_ks + kk : A, in);
                }
                if (b_cols) {
                    const int kk = 16 * g + 2 * step + y;
                    const bool in = x < cols && kk < t.b;
                    copy_async_8(Bs + kk * kSmemLd + x, in ? B + (long long)kk * b_ld + x : B, in);
                } else {
                    const int kk = 16 * g + k, c = 8 * step + outer;
                    const bool in = c < cols && kk < t.b;
                    copy_async_8(Bs + c * kSmemLd + kk, in ? B + (long long)c * b_ld + kk : B, in);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    double acc[2][8][2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = wr + 8 * i + fr;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = 8 * j + 2 * fk + h;
                acc[i][j][h] = TRAILING && r < rows && c < cols ? C[(long long)r * c_rs + (long long)c * c_cs] : 0.0;
            }
    }
    const int col_groups = (cols + 7) / 8;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        if (g == 0) copy_async_wait<3>();
        if (g == 1) copy_async_wait<2>();
        if (g == 2) copy_async_wait<1>();
        if (g == 3) copy_async_wait<0>();
        __syncthreads();
        if (g >= groups || wr >= rows) continue;
#pragma unroll
        for (int k4 = 16 * g; k4 < 16 * g + 16; k4 += 4) {
            double a[2], bv[8];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                a[i] = As[(wr + 8 * i + fr) * a_i + (k4 + fk) * a_k];
                if (TRAILING) a[i] = -a[i];
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) bv[j] = Bs[(k4 + fk) * b_k + (8 * j + fr) * b_c];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j < col_groups) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], bv[j]);
        }
    }
    if (wr >= rows) return;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = wr + 8 * i + fr;
        if (r >= rows) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int c = 8 * j + 2 * fk + h;
                if (c < cols) C[(long long)r * c_rs + (long long)c * c_cs] = acc[i][j][h];
            }
    }
}

int allow_product_memory() {
    static int allowed[64] = {};
    int device = 0;
    OB_CUDA(cudaGetDevice(&device));
    if (device >= 0 && device < 64 && allowed[device]) return OB_OK;
    OB_CUDA(cudaFuncSetAttribute(front_product_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem));
    OB_CUDA(cudaFuncSetAttribute(front_product_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileSmem));
    if (device >= 0 && device < 64) allowed[device] = 1;
    return OB_OK;
}

}  // namespace

int device_factor(CholAnalysis& A, const double* values, double sign, int pin_mode, double* vals, char* pinned,
                  const FactorTables& tables, const std::function<int()>& meanwhile, cudaStream_t stream) {
    if (int st = allow_product_memory()) return st;
    FactorPlan* P = nullptr;
    {
        std::lock_guard<std::mutex> guard(A.plan_mutex);
        int device = 0;
        OB_CUDA(cudaGetDevice(&device));
        if (A.plan != nullptr && A.plan->device != device) {
            release_plan(A.plan);
            A.plan = nullptr;
        }
        if (A.plan == nullptr) {
            FactorPlan* fresh = new FactorPlan();
            fresh->device = device;
            int st = build_plan(A, fresh, stream);
            if (st) {
                release_plan(fresh);
                return st;
            }
            A.plan = fresh;
        }
        P = A.plan;
    }
    const int n = A.n;
    const long long vals_count = tables.n_vals;
    const int ns = P->n_nodes;
    Scratch scratch(stream);
    double* fronts = scratch.take<double>((size_t)P->front_total);
    int* bad = scratch.take<int>((size_t)std::max(A.n_components, 1));
    int* status = scratch.take<int>(1);
    if (int st = scratch.commit()) return st;
    OB_CUDA(cudaMemsetAsync(fronts, 0, sizeof(double) * (size_t)std::max<long long>(P->front_total, 1), stream));
    OB_CUDA(cudaMemsetAsync(vals, 0, sizeof(double) * (size_t)std::max<long long>(vals_count, 1), stream));
    OB_CUDA(cudaMemsetAsync(bad, 0, sizeof(int) * (size_t)std::max(A.n_components, 1), stream));
    OB_CUDA(cudaMemsetAsync(status, 0, sizeof(int), stream));
    const int threads = 256;
    if (ns > 0) {
        factor_tables_kernel<<<ceil_div(32LL * ns, threads), threads, 0, stream>>>(
            ns, n, P->start, P->nc, P->rel_at, P->rows, P->rows_at, P->perm, P->parent, tables);
        OB_CHECK_LAUNCH("chol factor tables");
    }
    if (pin_mode == kPinZeroSum) {
        zero_sum_rows_kernel<<<ceil_div(n, threads), threads, 0, stream>>>(n, P->offsets, values, P->diag_pos,
                                                                           P->component, bad);
        OB_CHECK_LAUNCH("chol zero-sum rows");
    }
    pin_rows_kernel<<<ceil_div(n, threads), threads, 0, stream>>>(n, P->perm, values, P->diag_pos, P->component,
                                                                  P->component_last, bad, pin_mode, P->diag_dest,
                                                                  pinned, fronts);
    OB_CHECK_LAUNCH("chol pin rows");
    if (P->n_entries > 0) {
        scatter_entries_kernel<<<ceil_div(P->n_entries, threads), threads, 0, stream>>>(
            P->n_entries, values, P->entry_dest, P->entry_rc, pinned, sign, fronts);
        OB_CHECK_LAUNCH("chol scatter entries");
    }
    auto launch_early = [stream](auto kernel, int blocks, int block, int smem, auto... args) {
        cudaLaunchAttribute early;
        early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        early.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3((unsigned)blocks);
        config.blockDim = dim3((unsigned)block);
        config.dynamicSmemBytes = (size_t)smem;
        config.stream = stream;
        config.attrs = &early;
        config.numAttrs = 1;
        cudaLaunchKernelEx(&config, kernel, args...);
    };
    for (const FactorPlan::Launch& L : P->launches) {
        const ExtendTask* extend = static_cast<const ExtendTask*>(L.tasks);
        const StepTask* steps = static_cast<const StepTask*>(L.tasks);
        switch (L.kind) {
            case kExtend:
                launch_early(extend_add_kernel, L.count, kExtendThreads, 0, extend, (const long long*)P->front_at,
                             (const int*)P->fld, (const int*)P->nc, (const int*)P->noff, (const int*)P->rel_at,
                             (const int*)P->rel, fronts);
                OB_CHECK_LAUNCH("chol extend-add");
                break;
            case kDiag:
                launch_early(diag_block_kernel, L.count, kDiagThreads, 0, steps, (const double*)fronts, vals, status);
                OB_CHECK_LAUNCH("chol diagonal blocks");
                break;
            case kPanelProduct:
                launch_early(front_product_kernel<false>, L.count, kTileThreads, kTileSmem, steps, L.owner, fronts, vals);
                OB_CHECK_LAUNCH("chol panel products");
                break;
            default:
                launch_early(front_product_kernel<true>, L.count, kTileThreads, kTileSmem, steps, L.owner, fronts, vals);
                OB_CHECK_LAUNCH("chol trailing products");
        }
    }
    // The launches above run while the host goes on.
    const int beside = meanwhile();
    int host_status = 0;
    OB_CUDA(cudaMemcpyAsync(&host_status, status, sizeof(int), cudaMemcpyDeviceToHost, stream));
    OB_CUDA(cudaStreamSynchronize(stream));
    if (beside) return beside;
    return host_status ? OB_ERR_INDEFINITE : OB_OK;
}

}  // namespace ob
