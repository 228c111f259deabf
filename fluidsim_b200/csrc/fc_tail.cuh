// Coarse tail of the V-cycle: every level from GridDesc::tail to the coarsest cycled by one CTA
// per grid (PressureMultigrid.cpp:386-434), and the explicit inverse of the coarsest level.
//
// What bounds it. The tail is one SM's serial chain (pre-smooth, restrict, ... , coarsest solve,
// prolong, post-smooth), so only its latency counts; no unit is busy. Everything that is not part
// of the chain is moved in front of it or dropped:
//  * Every smoothed level has warps of its own that hold the level's weights, inverse diagonals
//    and values in registers from before the dependency wait to the end: nothing is reloaded
//    between the pre- and the post-smoothing, and the loads overlap the kernel before.
//  * A row group of kTailK rows takes 8, 16 or 32 lanes (a column pair per lane), as many as the
//    level is wide, so a warp holds 4, 2 or 1 row groups: a 32 x 32 level is 4 warps and a 16 x 16
//    level one warp, whose half-sweeps need no CTA barrier at all.
//  * The restriction's sums along x come from the residual registers; the coarse level's lanes
//    sum them along y straight into their right-hand side registers.
//  * The coarsest solve is one matrix product: its mean removals are folded into the inverse when
//    it is built (k_rebuild_tail), unless obstacles seal off a part of the level.
//  * The layout and the transfer weights come in one host-built block (TailTable).
//
// Measured with fc_time_kernel on a 512 x 512 grid (levels 32 x 32, 16 x 16, 8 x 8), before this
// form (levels in shared memory, reloaded per leg, 16 warps behind every barrier of the 32 x 32
// level) and with it: FP32 22.8 -> 11.9 us, FP64 31.0 -> 13.8 us, launch included. From the
// dependency wait on a form at 12.6 us took 11,500 cycles: 225 a half-sweep of the 32 x 32 level and 180 of the
// 16 x 16 one (118 to 144 in a loop of nothing else), 1,050 for the coarsest product, and 350 to
// 450 for each restriction and prolongation.
#pragma once

#include "fc_device.cuh"
#include "fc_smooth.cuh"
#include "fc_tma.cuh"

namespace fc
{

constexpr int kMaxCoarse = 64; // cells of the coarsest level
constexpr int kTailK = 4;      // rows of a row group
constexpr int kTailMaxSide = 64;
// Smoothed levels of a tail: 64 cells a side halve to 32, 16 and 8 a side, and a level of at most
// 64 cells is solved directly (thinner levels reach 64 cells sooner).
constexpr int kTailMaxSmoothed = 3;
// Block sizes. A strip, what goes with it and the code around it need about 125 registers in FP32
// and 168 in FP64 (at fewer, what spills sits in the sweeps: 270 cycles a half-sweep instead of
// 228), so FP32 runs 512 threads, which also cover the coarsest product (eight per row), and FP64,
// whose tail takes at most 1024 cells (8 + 2 + 1 warps), 384. Only a 64 x 64 level needs more
// (16 + 4 + 1 warps), at 80 registers.
template <typename T> constexpr int kTailThreads = sizeof(T) == 4 ? 512 : 384;
constexpr int kTailWideThreads = 32 * 21;

// Elements from one plane of edge rows to the next: a constant, so that a lane's slots are one
// register and immediate offsets. It holds the groups of any level and one more at each end (FP32:
// 16 groups of 32 lanes; FP64: 8).
template <typename T> constexpr int kTailPlane = (sizeof(T) == 4 ? 18 : 10) * 32;

// Where a tail level lives: its sides, the lanes of its row groups, its warps, element offsets into
// the tail's shared memory (the restriction's weights, four for each coarse row and column, the
// prolongation's weights of the level's columns and rows, the two edge rows of every row group, the
// restriction's x sums, and the solution its finer neighbour prolongs), and its arrays.
struct TailPlace
{
    int w, h, S, lanes, warps;
    int rows, cols, px, py, edges, lines, sol, sol_stride;
    const void* right;
    const void* down;
    const void* inv;
};

// Everything about a grid's tail that no projection changes, built by the host in one block so that
// the kernel's prologue is one descriptor load and one bulk copy: this header, then from
// kTailHeader on the transfer weights (`tables` elements, at the offsets in `place`).
struct TailTable
{
    int smoothed, first, tables;
    int zeroed;   // elements of edges and lines, which start at zero, behind the tables
    int elements; // all elements
    const void* rhs; // right-hand side and solution of the first level
    void* out;
    TailPlace place[kTailMaxSmoothed + 1]; // smoothed levels, then the coarsest at [smoothed]
};
constexpr int kTailHeader = 512;
static_assert(sizeof(TailTable) <= kTailHeader && kTailHeader % 16 == 0, "tail header");
constexpr size_t kTailTableBytes = 8192; // room for the header and any tail's tables

__host__ __device__ inline int tail_lanes(int w) { return w <= 16 ? 8 : (w <= 32 ? 16 : 32); }
__host__ __device__ inline int tail_warps(int w, int h)
{
    return (((h + kTailK - 1) / kTailK) * tail_lanes(w) + 31) / 32;
}

// Lays out the levels of a tail whose sides are in t.place (smoothed levels 0 .. smoothed - 1, then
// the coarsest).
inline void tail_layout(TailTable& t, int plane)
{
    int cursor = 0;
    auto take = [&](int n)
    {
        const int at = cursor;
        cursor += (n + 3) / 4 * 4;
        return at;
    };
    for (int i = 0; i < t.smoothed; ++i)
    {
        TailPlace& p = t.place[i];
        const TailPlace& c = t.place[i + 1];
        p.lanes = tail_lanes(p.w);
        p.warps = tail_warps(p.w, p.h);
        p.rows = take(4 * c.h);
        p.cols = take(4 * c.w);
        p.px = take(2 * p.lanes);
        p.py = take(p.warps * 32 / p.lanes * kTailK);
    }
    t.tables = cursor;
    for (int i = 0; i < t.smoothed; ++i)
    {
        TailPlace& p = t.place[i];
        // Four planes (the top and the bottom row of every group, in each colour) with a zero group
        // at each end; only the last one is cut short.
        p.edges = take(3 * plane + (p.warps * 32 / p.lanes + 2) * p.lanes);
        p.lines = take((p.h + 3) * p.lanes); // rows -1 .. h + 1, those outside the level zero
    }
    t.zeroed = cursor - t.tables;
    for (int i = t.smoothed > 0 ? 1 : 0; i <= t.smoothed; ++i)
    {
        TailPlace& p = t.place[i];
        p.sol_stride = i < t.smoothed ? 2 * p.lanes : p.w;
        p.sol = take(p.sol_stride * p.h);
    }
    t.elements = cursor;
}

// The coarsest inverse's rows are 72 doubles apart, in global and in shared memory: the four rows
// that a warp reads then cover every bank twice. It is copied whole; rows and columns beyond the
// level's cells are zero. One more row and column serve an inverse without folded means (TailMeans).
constexpr int kTailInverseStride = 72;
constexpr size_t kTailInverseBytes = size_t(kMaxCoarse + 1) * kTailInverseStride * sizeof(double);

// Elements of the inverse that say how the solve takes its means: the column sums (row kMaxCoarse),
// one for each open cell and zero for another (column kMaxCoarse), and the share of a cell in a
// mean, zero where the solve takes none (folded, or Dirichlet air).
struct TailMeans
{
    static __host__ __device__ constexpr int sums(int cell) { return kMaxCoarse * kTailInverseStride + cell; }
    static __host__ __device__ constexpr int open(int cell) { return cell * kTailInverseStride + kMaxCoarse; }
    static constexpr int share = kMaxCoarse * kTailInverseStride + kMaxCoarse;
};

// Dynamic shared memory: the coarsest inverse, its right-hand side in FP64, the table's header, and
// the levels' elements (at most 10840 in FP32 and 5912 in FP64 over every level shape a tail
// takes). Everything is addressed by element offsets, so that every access is a shared-memory one.
// A launch has what its plan's largest table needs, which the plan follows (plan_current in the engine):
// the largest any table needs in every launch cost 64 x 64 projections 1.4 % (933 -> 946 us), and a
// check of it in the kernel delayed the copies by 0.3 us.
constexpr size_t kTailSolveBytes = kTailInverseBytes + kMaxCoarse * sizeof(double);
inline size_t tail_bytes(int elements, size_t elem) { return kTailSolveBytes + kTailHeader + size_t(elements) * elem; }
constexpr size_t kTailMaxBytes = kTailSolveBytes + kTailHeader + 5912 * sizeof(double);
extern __shared__ __align__(16) unsigned char tail_smem[];
template <typename T> __device__ __forceinline__ T* tail_elements()
{
    return reinterpret_cast<T*>(tail_smem + kTailSolveBytes + kTailHeader);
}

// One level's view for one lane of its warps.
struct TailLane
{
    int w, h, lanes, warps;
    int j, y0;     // column pair and the row group's first row
    int top;       // element offset of this lane's slot in its group, first plane
    int barrier;   // named barrier of the level's warps
};

__device__ __forceinline__ void tail_barrier(const TailLane& t)
{
    if (t.warps == 1)
        __syncwarp();
    else
        asm volatile("bar.sync %0, %1;" ::"r"(t.barrier), "r"(t.warps * 32) : "memory");
}

// Publishes the strip's edge cells of colour c: its top row in plane c, its bottom row in plane
// 2 + c. Row 0 is even: colour c sits in a when c == 0; row kTailK - 1 is odd.
template <typename T, int c> __device__ __forceinline__ void tail_publish(const Strip<T, kTailK>& s, const TailLane& t)
{
    T* const m = tail_elements<T>();
    m[t.top + c * kTailPlane<T>] = c == 0 ? s.a[0] : s.b[0];
    m[t.top + (2 + c) * kTailPlane<T>] = c == 1 ? s.a[kTailK - 1] : s.b[kTailK - 1];
    tail_barrier(t);
}

// One red-black half-sweep of colour c over row groups of t.lanes lanes (strip_sweep's arithmetic,
// fc_smooth.cuh).
template <typename T, int c> __device__ __forceinline__ void tail_sweep(Strip<T, kTailK>& s, const TailLane& t)
{
    T* const m = tail_elements<T>();
    const T above = m[t.top - t.lanes + (3 - c) * kTailPlane<T>];
    const T below = m[t.top + t.lanes + (1 - c) * kTailPlane<T>];
#pragma unroll
    for (int k = 0; k < kTailK; ++k)
    {
        if ((k & 1) == c)
        {
            T left = __shfl_up_sync(0xffffffffu, s.wr[k] * s.b[k], 1, t.lanes);
            left = t.j == 0 ? T(0) : left;
            const T up = k == 0 ? above : s.a[k - 1];
            const T dn = k == kTailK - 1 ? below : s.a[k + 1];
            const T wu = k == 0 ? s.ua : s.da[k - 1];
            s.a[k] = (s.ra[k] + ((left + s.wm[k] * s.b[k]) + (wu * up + s.da[k] * dn))) * s.ia[k];
        }
        else
        {
            // The last lane's wr is zero: what the shuffle returns there does not count.
            const T right = __shfl_down_sync(0xffffffffu, s.a[k], 1, t.lanes);
            const T up = k == 0 ? above : s.b[k - 1];
            const T dn = k == kTailK - 1 ? below : s.b[k + 1];
            const T wu = k == 0 ? s.ub : s.db[k - 1];
            s.b[k] = (s.rb[k] + ((s.wm[k] * s.a[k] + s.wr[k] * right) + (wu * up + s.db[k] * dn))) * s.ib[k];
        }
    }
    tail_publish<T, c>(s, t);
}

// The residual after the sweeps, summed along x into the level's lines (PressureMultigrid.cpp:
// 398-402, 233-276). The last half-sweep solved the equations of its colour (1), so only cells of
// colour 0 have a residual: column 2j in even rows, column 2j + 1 in odd ones. Lanes beyond the
// last coarse column write lines that no one reads.
template <typename T>
__device__ __forceinline__ void tail_restrict(const Strip<T, kTailK>& s, const TailLane& t, const TailPlace& own,
    const TailPlace& coarser)
{
    T* const m = tail_elements<T>();
    constexpr int B = kTailPlane<T>;
    const int lanes = t.lanes;
    T along_x[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        along_x[e] = m[own.cols + 4 * min(t.j, coarser.w - 1) + e];
    const T above_a = m[t.top - lanes + 3 * B], below_b = m[t.top + lanes + B];
#pragma unroll
    for (int k = 0; k < kTailK; ++k)
    {
        const T a = s.a[k], b = s.b[k];
        T sum;
        // Cells without an open face pass no residual down.
        if (k % 2 == 0)
        {
            T left = __shfl_up_sync(0xffffffffu, b, 1, lanes);
            T wl = __shfl_up_sync(0xffffffffu, s.wr[k], 1, lanes);
            left = t.j == 0 ? T(0) : left;
            wl = t.j == 0 ? T(0) : wl;
            const T up = k == 0 ? above_a : s.a[k - 1];
            const T wu = k == 0 ? s.ua : s.da[k - 1];
            const T pa = (wl * (a - left) + s.wm[k] * (a - b)) + (wu * (a - up) + s.da[k] * (a - s.a[k + 1]));
            const T res = s.ia[k] > T(0) ? s.ra[k] - pa : T(0);
            T res_right = __shfl_down_sync(0xffffffffu, res, 1, lanes);
            res_right = t.j == lanes - 1 ? T(0) : res_right;
            sum = along_x[1] * res + along_x[3] * res_right;
        }
        else
        {
            const T right = __shfl_down_sync(0xffffffffu, a, 1, lanes);
            const T dn = k == kTailK - 1 ? below_b : s.b[k + 1];
            const T pb = (s.wm[k] * (b - a) + s.wr[k] * (b - right)) + (s.db[k - 1] * (b - s.b[k - 1]) + s.db[k] * (b - dn));
            const T res = s.ib[k] > T(0) ? s.rb[k] - pb : T(0);
            T res_left = __shfl_up_sync(0xffffffffu, res, 1, lanes);
            res_left = t.j == 0 ? T(0) : res_left;
            sum = along_x[0] * res_left + along_x[2] * res;
        }
        if (t.y0 + k < t.h)
            m[own.lines + (t.y0 + k + 1) * lanes + t.j] = sum;
    }
}

// The right-hand side of a level below the first: row y sums the finer level's lines 2y - 1 ..
// 2y + 2 (rows beyond the level's last one stay with what the finer level's last lines hold).
template <typename T>
__device__ __forceinline__ void tail_gather(Strip<T, kTailK>& s, const TailLane& t, const TailPlace& finer)
{
    using P = typename Pair<T>::type;
    T* const m = tail_elements<T>();
    const int column = finer.lines + min(2 * t.j, finer.lanes - 2);
    auto line = [&](int r) { return *reinterpret_cast<const P*>(m + column + min(2 * t.y0 + r, finer.h + 2) * finer.lanes); };
    P q0 = line(0), q1 = line(1);
#pragma unroll
    for (int k = 0; k < kTailK; ++k)
    {
        const P q2 = line(2 * k + 2), q3 = line(2 * k + 3);
        const T* w = m + finer.rows + 4 * min(t.y0 + k, t.h - 1);
        const T w0 = w[0], w1 = w[1], w2 = w[2], w3 = w[3];
        s.ra[k] = (w0 * q0.x + w1 * q1.x) + (w2 * q2.x + w3 * q3.x);
        s.rb[k] = (w0 * q0.y + w1 * q1.y) + (w2 * q2.y + w3 * q3.y);
        q0 = q2;
        q1 = q3;
    }
}

// The coarse solution prolonged onto the strip (bilinear; PressureMultigrid.cpp:278-298). Fine
// cells 2m and 2m + 1 read coarse cells m - 1, m and m, m + 1 (prolong_weights).
template <typename T>
__device__ __forceinline__ void tail_prolong(Strip<T, kTailK>& s, const TailLane& t, const TailPlace& own,
    const TailPlace& coarse)
{
    T* const m = tail_elements<T>();
    const T pa = m[own.px + 2 * t.j], pb = m[own.px + 2 * t.j + 1];
    // Lanes beyond the level read its last column and row; their cells stay zero.
    const int c0 = min(max(t.j - 1, 0), coarse.w - 1), c1 = min(t.j, coarse.w - 1), c2 = min(t.j + 1, coarse.w - 1);
    T xa[kTailK / 2 + 2], xb[kTailK / 2 + 2];
#pragma unroll
    for (int r = 0; r < kTailK / 2 + 2; ++r)
    {
        const int row = coarse.sol + min(max(t.y0 / 2 - 1 + r, 0), coarse.h - 1) * coarse.sol_stride;
        const T v0 = m[row + c0], v1 = m[row + c1], v2 = m[row + c2];
        xa[r] = fma(pa, v1, (T(1) - pa) * v0);
        xb[r] = fma(pb, v2, (T(1) - pb) * v1);
    }
#pragma unroll
    for (int k = 0; k < kTailK; ++k)
    {
        const int f = (k + 1) / 2;
        const T py = m[own.py + t.y0 + k];
        const T a = s.a[k] + fma(py, xa[f + 1], (T(1) - py) * xa[f]);
        const T b = s.b[k] + fma(py, xb[f + 1], (T(1) - py) * xb[f]);
        // A cell that is no unknown (and any beyond the level) keeps zero.
        s.a[k] = s.ia[k] > T(0) ? a : T(0);
        s.b[k] = s.ib[k] > T(0) ? b : T(0);
    }
}

// One thread's share of a product with a row of the coarsest inverse, and the sum of the eight.
__device__ __forceinline__ double coarse_dot(const double* row, const double* rhs, int part)
{
    const double* a = row + part;
    double z = 0.0, z1 = 0.0;
#pragma unroll
    for (int i = 0; i < kMaxCoarse / 16; ++i)
    {
        z += a[16 * i] * rhs[part + 16 * i];
        z1 += a[16 * i + 8] * rhs[part + 16 * i + 8];
    }
    return z + z1;
}

__device__ __forceinline__ double eight_lane_sum(double z)
{
    z += __shfl_xor_sync(0xffffffffu, z, 1);
    z += __shfl_xor_sync(0xffffffffu, z, 2);
    return z + __shfl_xor_sync(0xffffffffu, z, 4);
}

// The coarsest solve with an inverse that has no means folded in (k_rebuild_tail): the mean comes off
// the right-hand side in `rhs`, and the solution's, from the row of the column sums, off the solution.
// Returns the right-hand side's mean. Rare, and kept out of the cycle's code: inlined it cost every
// V-cycle 0.2 us.
template <typename T, int kThreads>
__device__ __noinline__ double tail_solve_means(const double* inverse, double* rhs, double share, int cells, int sol)
{
    double mean = 0.0;
    for (int i = threadIdx.x & 31; i < cells; i += 32)
        mean += inverse[TailMeans::open(i)] * rhs[i];
    mean = warp_sum(mean) * share;
    __syncthreads();
    if (int(threadIdx.x) < cells)
        rhs[threadIdx.x] -= mean;
    __syncthreads();
    const int part = threadIdx.x & 7;
    const double gauge = eight_lane_sum(coarse_dot(inverse + TailMeans::sums(0), rhs, part)) * share;
    T* const m = tail_elements<T>();
    for (int base = 0; base < kMaxCoarse; base += kThreads / 8)
    {
        const int row = base + int(threadIdx.x >> 3);
        const double z = eight_lane_sum(coarse_dot(inverse + min(row, kMaxCoarse - 1) * kTailInverseStride, rhs, part));
        if (row < cells && part == 0)
            m[sol + row] = inverse[TailMeans::open(row)] != 0.0 ? T(z - gauge) : T(0);
    }
    __syncthreads();
    return mean;
}

template <typename T, int kThreads> __global__ void __launch_bounds__(kThreads) k_mg_tail(const GridDesc* __restrict__ grids)
{
    using P = typename Pair<T>::type;
    allow_dependents();
    const GridDesc& g = grids[blockIdx.x];
    SolveState& state = *g.state;
    // In a batch (one CTA per grid), a grid whose solve is known to be done before the wait loads
    // nothing. A single grid skips the check: its load would delay the others.
    if (gridDim.x > 1 && done_before_wait(g.state))
        return;
    const TailTable* const table = static_cast<const TailTable*>(g.tail_table);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* const inverse = reinterpret_cast<double*>(tail_smem);
    double* const coarse_rhs = inverse + kTailInverseBytes / sizeof(double);
    const TailTable& shared_table = *reinterpret_cast<const TailTable*>(tail_smem + kTailSolveBytes);
    T* const m = tail_elements<T>();
    __shared__ uint64_t bar;
    // Everything read before the wait is written by no kernel of the projection. The header comes by
    // plain loads for the set-up, and with the tables and the coarsest inverse by bulk copy for the
    // cycle.
    const int smoothed = table->smoothed, first = table->first, tables = table->tables, zeroed = table->zeroed;
    // Bulk copies write 16-byte aligned shared addresses only: a misplaced buffer is reported.
    const bool aligned = (smem_address(tail_smem) & 15u) == 0;
    if (threadIdx.x == 0 && aligned)
    {
        mbarrier_init(&bar, 1);
        fence_async_shared();
        const unsigned bytes = kTailHeader + unsigned(tables) * sizeof(T);
        mbarrier_expect_tx(&bar, bytes + unsigned(kTailInverseBytes));
        bulk_load(tail_smem + kTailSolveBytes, table, bytes, &bar);
        bulk_load(inverse, g.coarse_inverse, unsigned(kTailInverseBytes), &bar);
    }
    // This warp's level (-1: none).
    int role = -1, level_warp = warp, warps_needed = 0;
#pragma unroll
    for (int i = 0; i < kTailMaxSmoothed; ++i)
    {
        const int warps = table->place[i].warps; // zero where there is no such level
        warps_needed += warps;
        if (role < 0)
        {
            if (level_warp < warps)
                role = i;
            else
                level_warp -= warps;
        }
    }
    const TailPlace& place = table->place[max(role, 0)];
    const int S = place.S;
    TailLane t{};
    Strip<T, kTailK> s{};
    if (role >= 0)
    {
        t.w = place.w;
        t.h = place.h;
        t.lanes = place.lanes;
        t.warps = place.warps;
        const int groups = 32 / t.lanes;
        t.j = lane & (t.lanes - 1);
        const int group = level_warp * groups + lane / t.lanes;
        t.y0 = kTailK * group;
        t.top = place.edges + (group + 1) * t.lanes + t.j;
        t.barrier = 1 + role;
        const T* right = static_cast<const T*>(place.right);
        const T* down = static_cast<const T*>(place.down);
        const T* inv = static_cast<const T*>(place.inv);
        // Columns beyond the level's last one are padding, which holds zeros.
        const bool column = 2 * t.j < t.w;
        if (column && t.y0 < t.h)
        {
            const P u = *reinterpret_cast<const P*>(down + padded_index32(S, 2 * t.j, t.y0 - 1));
            s.ua = u.x;
            s.ub = u.y;
        }
#pragma unroll
        for (int k = 0; k < kTailK; ++k)
        {
            if (!column || t.y0 + k >= t.h)
                continue;
            const int i = padded_index32(S, 2 * t.j, t.y0 + k);
            const P w2 = *reinterpret_cast<const P*>(right + i);
            const P d2 = *reinterpret_cast<const P*>(down + i);
            const P i2 = *reinterpret_cast<const P*>(inv + i);
            s.wm[k] = w2.x;
            s.wr[k] = w2.y;
            s.da[k] = d2.x;
            s.db[k] = d2.y;
            s.ia[k] = i2.x;
            s.ib[k] = i2.y;
        }
    }
    const T* const rhs = static_cast<const T*>(table->rhs);
    T* const out = static_cast<T*>(table->out);
    // Edges and lines start at zero: what lies outside a level is never written.
    for (int i = threadIdx.x; i < zeroed; i += blockDim.x)
        m[tables + i] = T(0);
    if (threadIdx.x < kMaxCoarse)
        coarse_rhs[threadIdx.x] = 0.0;
    __syncthreads();
    // A level's barrier waits for all its warps, so they must be in this launch.
    if (stage_failed(aligned && mbarrier_wait(&bar, 0) && 32 * warps_needed <= kThreads, g.state))
        return;
    const TailPlace& own = shared_table.place[max(role, 0)];
    const TailPlace& finer = shared_table.place[max(role - 1, 0)];
    const TailPlace& coarser = shared_table.place[max(role, 0) + (smoothed > 0 ? 1 : 0)];
    const TailPlace& last = shared_table.place[smoothed];
    const int cells = last.w * last.h;
    // The cell whose coarsest right-hand side this thread forms.
    const int cx = int(threadIdx.x) % last.w, cy = int(threadIdx.x) / last.w;

    // The right-hand side of the first tail level comes from the previous kernel.
    dependency_wait();
    const int done = state.done;
    const double mean_r = first == 0 ? state.mean_r : 0.0;
    // Only the fine level's right-hand side has a mean to take off: a coarser one is restricted from
    // a residual that has none of it left.
    const double level_mean = role == 0 ? mean_r : 0.0;
    if (role == 0)
    {
#pragma unroll
        for (int k = 0; k < kTailK; ++k)
            if (2 * t.j < t.w && t.y0 + k < t.h)
            {
                const P v = *reinterpret_cast<const P*>(rhs + padded_index32(S, 2 * t.j, t.y0 + k));
                s.ra[k] = v.x;
                s.rb[k] = v.y;
            }
    }
    if (done)
        return;

    // The coarsest level (at most 64 cells): mean-free, explicit inverse, mean-zero gauge
    // (PressureMultigrid.cpp:347-384), its solution to last.sol: one product with the means folded
    // into the inverse, or a solve that takes them itself (tail_solve_means) and returns the
    // right-hand side's. Eight threads per row, each with every eighth entry in two chains.
    auto solve_coarsest = [&](T value)
    {
        if (int(threadIdx.x) < cells)
            coarse_rhs[threadIdx.x] = double(value);
        __syncthreads();
        const double share = inverse[TailMeans::share];
        if (__builtin_expect(share != 0.0, 0))
            return tail_solve_means<T, kThreads>(inverse, coarse_rhs, share, cells, last.sol);
        const int part = threadIdx.x & 7;
#pragma unroll
        for (int base = 0; base < kMaxCoarse; base += kThreads / 8)
        {
            const int row = base + int(threadIdx.x >> 3);
            double z = 0.0;
            if (row < kMaxCoarse)
                z = coarse_dot(inverse + row * kTailInverseStride, coarse_rhs, part);
            z = eight_lane_sum(z);
            if (row < cells && part == 0)
                m[last.sol + row] = T(z);
        }
        __syncthreads();
        return 0.0;
    };
    if (smoothed == 0)
    {
        // A level of at most 64 cells is all the tail has: its right-hand side as it stands (less the
        // residual's mean on the fine level; closed cells have zero columns), and straight out.
        const double mean =
            mean_r + solve_coarsest(int(threadIdx.x) < cells ? minus_mean(rhs[padded_index32(S, cx, cy)], mean_r) : T(0));
        if (int(threadIdx.x) < cells)
            out[padded_index32(S, cx, cy)] = m[last.sol + threadIdx.x];
        if (first == 0 && threadIdx.x == 0)
        {
            double sz = 0.0, srz = 0.0;
            for (int i = 0; i < cells; ++i)
            {
                const double z = double(m[last.sol + i]);
                sz += z;
                srz += coarse_rhs[i] * z;
            }
            // coarse_rhs holds r - mean: sum r z = sum (r - mean) z + mean sum z.
            finish_preconditioner(state, sz, srz + mean * sz);
        }
        return;
    }

    // Both legs run through one copy of the code: on one SM, once per launch, the fetch of cold
    // instructions costs as much as their execution.
    constexpr int kDown = 0, kUp = 1;
#pragma unroll 1
    for (int leg = kDown; leg <= kUp; ++leg)
    {
        // Every warp passes one CTA barrier per smoothed level on the way down and one fewer on the
        // way up; a level's warps work between the barriers of its neighbours.
        if (leg == kDown)
        {
            for (int i = 0; i < role; ++i)
                __syncthreads();
            if (role > 0)
                tail_gather(s, t, finer);
#pragma unroll
            for (int k = 0; k < kTailK; ++k)
            {
                s.ra[k] = s.ia[k] > T(0) ? minus_mean(s.ra[k], level_mean) : T(0);
                s.rb[k] = s.ib[k] > T(0) ? minus_mean(s.rb[k], level_mean) : T(0);
                s.a[k] = s.b[k] = T(0);
            }
        }
        else
        {
            T value = T(0);
            if (int(threadIdx.x) < cells)
            {
                const TailPlace& f = shared_table.place[smoothed - 1];
                const int lanes = f.lanes;
                const T* l = m + f.lines + 2 * cy * lanes + cx;
                const T* w = m + f.rows + 4 * cy;
                value = (w[0] * l[0] + w[1] * l[lanes]) + (w[2] * l[2 * lanes] + w[3] * l[3 * lanes]);
            }
            solve_coarsest(value);
            for (int i = smoothed - 1; i > max(role, 0); --i)
                __syncthreads();
            if (role >= 0)
            {
                tail_prolong(s, t, own, coarser);
                tail_publish<T, 0>(s, t);
            }
        }
        // Four sweeps (PressureMultigrid.cpp:204-231): colours 0, 1 down, 1, 0 up. The first one of
        // the down leg starts from zero, as the edges do. The loop's body is a straight pair of
        // half-sweeps (with a branch on the colour in it the tail took 12.85 us instead of 11.94 in
        // FP32 and 14.6 instead of 13.8 in FP64).
        if (role >= 0)
        {
            __syncwarp();
            if (leg == kUp)
                tail_sweep<T, 1>(s, t);
#pragma unroll 1
            for (int i = leg; i < 4; ++i)
            {
                tail_sweep<T, 0>(s, t);
                tail_sweep<T, 1>(s, t);
            }
            if (leg == kUp)
                tail_sweep<T, 0>(s, t);
            if (leg == kDown)
                tail_restrict(s, t, own, coarser);
        }
        if (leg == kDown)
            for (int i = max(role, 0); i < smoothed; ++i)
                __syncthreads();
    }
    if (role > 0)
    {
#pragma unroll
        for (int k = 0; k < kTailK; ++k)
            if (t.y0 + k < t.h)
            {
                P ab;
                ab.x = s.a[k];
                ab.y = s.b[k];
                *reinterpret_cast<P*>(m + own.sol + (t.y0 + k) * own.sol_stride + 2 * t.j) = ab;
            }
    }
    else if (role == 0)
    {
        // The first tail level's solution goes to the finer post-smoothing (or to z).
#pragma unroll
        for (int k = 0; k < kTailK; ++k)
            if (2 * t.j < t.w && t.y0 + k < t.h)
            {
                // An odd last column leaves its pair in the padding, which stays zero.
                P ab;
                ab.x = s.a[k];
                ab.y = s.b[k];
                *reinterpret_cast<P*>(out + padded_index32(S, 2 * t.j, t.y0 + k)) = ab;
            }
    }
    for (int i = max(role, 0); i > 0; --i)
        __syncthreads();
    if (first != 0)
        return;
    // The fine level itself: sum z and r.z for the PCG scalars. Cells without an open face hold
    // z = 0 and add to neither sum.
    double sz = 0.0, srz = 0.0;
    if (role == 0)
    {
#pragma unroll
        for (int k = 0; k < kTailK; ++k)
        {
            sz += double(s.a[k]) + double(s.b[k]);
            srz += double(s.ra[k]) * double(s.a[k]) + double(s.rb[k]) * double(s.b[k]);
        }
    }
    __shared__ double2 warp_sums[32];
    sz = warp_sum(sz);
    srz = warp_sum(srz);
    if (lane == 0)
        warp_sums[warp] = make_double2(sz, srz);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        const int warps = shared_table.place[0].warps;
        sz = srz = 0.0;
        for (int i = 0; i < warps; ++i)
        {
            sz += warp_sums[i].x;
            srz += warp_sums[i].y;
        }
        // The strips hold r - mean r: sum r z = sum (r - mean r) z + mean r sum z.
        finish_preconditioner(state, sz, srz + mean_r * sz);
    }
}

// ------------------------------------------------------------------------------------------
// Rebuild of the tail's levels and of the coarsest level's explicit inverse
// ------------------------------------------------------------------------------------------

// One CTA per grid. The levels from the tail on hold a few thousand cells, less than a launch's worth
// of work each: they are rebuilt here, a barrier between levels, and the coarsest inverse after them.
//
// Dense pinned operator of the coarsest level and its inverse in FP64; one CTA per grid
// (PressureMultigrid.cpp:300-345, factorCoarsest). The first open cell is pinned (the reference
// pins cell 0; with no obstacle the two are the same), Dirichlet air pins none. A non-positive or
// non-finite pivot of the Cholesky factor marks the breakdown (:334-335). Rows and columns of cells
// that are no unknown are kept as those of the identity during the elimination and written as zeros.
//
// Gauss-Jordan elimination without pivoting: its pivots are the squares of the factor's diagonal, to
// rounding. A step publishes the pivot row and column in shared memory, double-buffered, so it costs
// one barrier and one division deep. The solve removes the mean of its right-hand side and gives
// its solution a mean-zero gauge (:347-384); both are linear, so the stored matrix is C inverse C
// with C = I - 1 1^T / open over the open cells (the pinned one included).
//
// Where obstacles seal off a part of the level the operator is singular: that part's last pivot is
// a rounding error, whose sign decides between breakdown and solve, and the inverse has entries of
// 1e16, in which folded means would drown every other part's. So if a pivot is not above kSealedPivot
// of the largest diagonal, the factor is formed again by the reference's column loop (invert_factor)
// and the means are left to the solve. (Gauss-Jordan pivots decided 26 of 96 sealed 8 x 8 and 7 x 9 scenes
// differently from the column loop.) Rounding moves either method's pivots by at most a few times
// 64 epsilon of the largest diagonal (the Schur complements of this diagonally dominant matrix do not
// grow), so above the limit both accept. Densities of 1000 : 1 leave pivots of 1e-5 and more.
// The whole kernel on a 64 x 64 grid in FP32: 40 us, 101 us where a wall across it needs the column loop.
constexpr double kSealedPivot = 1.0 / (1 << 24);

// Eight threads hold a row in registers (every eighth column).
constexpr int kCoarseThreads = 8 * kMaxCoarse;
constexpr int kCoarseColumns = kMaxCoarse / 8;
struct CoarseRow
{
    double a[kCoarseColumns]; // columns part, part + 8, ...
    int r, part;
};

// The inverse of the operator in `row` by its Cholesky factor, in the place of the operator; true
// if a pivot is not positive or not finite. `unknowns` has the bits of the unknowns' cells, and
// `factor` is global scratch of a row of kTailInverseStride a cell (in shared memory it made every
// rebuild's launch larger).
//
// The factor L is formed right-looking: every entry takes the reference's subtractions in the
// reference's order (PressureMultigrid.cpp:313-339), each product fused into its subtraction. Y = L^-1
// takes the place of the columns L is done with, and the inverse is Y^T Y. Step k publishes one
// vector: column k of L below the diagonal, and row k of Y up to it. Every warp carries the diagonal,
// two entries a lane, so its next pivot needs no other warp: one barrier a step, double-buffered.
static __device__ __noinline__ bool invert_factor(CoarseRow& row, const double* diagonal, unsigned long long unknowns, int cells,
    double* factor)
{
    constexpr int N = kMaxCoarse, E = kCoarseColumns;
    __shared__ double step[2][N];
    __shared__ int failed;
    const int r = row.r, part = row.part, lane = threadIdx.x & 31;
    const int first_row = r & ~3, last_row = first_row + 3; // of the warp
    double a[E];
#pragma unroll
    for (int i = 0; i < E; ++i)
        a[i] = row.a[i];
    double d0 = diagonal[lane], d1 = diagonal[lane + 32];
    int buf = 0;
    if (threadIdx.x == 0)
        failed = 0;
    __syncthreads();
#pragma unroll 1
    for (unsigned long long rest = unknowns; rest != 0; rest &= rest - 1, buf ^= 1)
    {
        const int k = __ffsll((long long)rest) - 1;
        if (last_row >= k)
        {
            const double value = __shfl_sync(0xffffffffu, k < 32 ? d0 : d1, k & 31);
            const double pivot = sqrt(value);
            double own = a[0];
#pragma unroll
            for (int i = 1; i < E; ++i)
                own = i == k >> 3 ? a[i] : own;
            // Row k's threads divide one, the others (those of column k count) their entry; a zero
            // stays zero without a division, which would take its slow path.
            const bool zero = own == 0.0;
            const double quotient = (r == k || zero ? 1.0 : own) / pivot;
            if (r == k)
            {
                if (!(value > 0.0) || !isfinite(value))
                    failed = 1;
#pragma unroll
                for (int i = 0; i < E; ++i)
                {
                    const int c = part + 8 * i;
                    if (c <= k)
                        step[buf][c] = a[i] = c == k ? quotient : a[i] * quotient;
                }
            }
            else if (r > k && part == (k & 7))
                step[buf][r] = zero ? 0.0 : quotient;
        }
        __syncthreads();
        if (last_row > k)
        {
            const double l0 = step[buf][lane], l1 = step[buf][lane + 32];
            if (lane > k)
                d0 = fma(-l0, l0, d0);
            if (lane + 32 > k)
                d1 = fma(-l1, l1, d1);
            if (r > k)
            {
                const double lr = step[buf][r];
#pragma unroll
                for (int i = 0; i < E; ++i)
                {
                    const int c = part + 8 * i;
                    a[i] = fma(-lr, step[buf][c], c == k ? 0.0 : a[i]);
                }
            }
        }
    }
    const bool mine = unknowns >> r & 1;
#pragma unroll
    for (int i = 0; i < E; ++i)
    {
        const int c = part + 8 * i;
        factor[r * kTailInverseStride + c] = mine && c <= r && (unknowns >> c & 1) ? a[i] : 0.0;
        a[i] = 0.0;
    }
    __threadfence_block();
    __syncthreads();
    // Entry (r, c) sums Y[k][r] Y[k][c] over k >= max(r, c): the terms before it are zero.
    for (int k = first_row; k < cells; ++k)
    {
        const double* const y = factor + k * kTailInverseStride;
        const double yr = __ldcg(y + r);
#pragma unroll
        for (int i = 0; i < E; ++i)
            a[i] = fma(yr, __ldcg(y + part + 8 * i), a[i]);
    }
    __syncthreads(); // the caller writes there
#pragma unroll
    for (int i = 0; i < E; ++i)
        row.a[i] = a[i];
    return failed != 0;
}

template <typename T> __global__ void __launch_bounds__(kCoarseThreads, 1) k_rebuild_tail(const GridDesc* __restrict__ grids)
{
    dependent_start();
    const GridDesc& g = grids[blockIdx.x];
    const int level = g.levels - 1;
    for (int i = g.tail; i < level; ++i)
    {
        const int w = g.lev[i + 1].w, cells = w * g.lev[i + 1].h;
        for (int q = threadIdx.x; q < cells; q += kCoarseThreads)
            rebuild_cell<T>(g, i, q % w, q / w);
        __syncthreads();
    }
    const LevelDesc& l = g.lev[level];
    const int cells = l.w * l.h;
    constexpr int N = kMaxCoarse, E = kCoarseColumns;
    __shared__ double pivot_row[2][N], pivot_col[2][N], row_mean[N], diagonal[N];
    __shared__ unsigned char open[N];
    __shared__ int sealed;
    const T* right = static_cast<const T*>(l.right);
    const T* down = static_cast<const T*>(l.down);
    const bool dirichlet = g.air != nullptr;
    const int r = threadIdx.x >> 3, part = threadIdx.x & 7, lane = threadIdx.x & 31;
    const int x = r % l.w, y = r / l.w;
    double diag = 0.0, wl = 0.0, wr = 0.0, wu = 0.0, wd = 0.0;
    if (r < cells)
    {
        const long long i = padded_index(l.S, x, y);
        wl = double(right[i - 1]);
        wr = double(right[i]);
        wu = double(down[i - l.S]);
        wd = double(down[i]);
        diag = ((wl + wr) + wu) + wd;
    }
    if (part == 0)
    {
        open[r] = r < cells && diag > 0.0 && !(dirichlet && held_cell<T>(g, level, x, y)) ? 1 : 0;
        diagonal[r] = diag;
    }
    if (threadIdx.x == 0)
        sealed = 0;
    __syncthreads();
    const unsigned low = __ballot_sync(0xffffffffu, open[lane] != 0);
    const unsigned high = __ballot_sync(0xffffffffu, open[lane + 32] != 0);
    const unsigned long long open_mask = (static_cast<unsigned long long>(high) << 32) | low;
    const unsigned long long unknowns = dirichlet ? open_mask : open_mask & (open_mask - 1); // less the first open cell
    auto unknown = [&](int c) { return (unknowns >> c & 1) != 0; };
    const bool mine = unknown(r);
    double largest = fmax(diagonal[lane], diagonal[lane + 32]);
    for (int offset = 16; offset > 0; offset >>= 1)
        largest = fmax(largest, __shfl_xor_sync(0xffffffffu, largest, offset));
    double a[E];
    auto form = [&]
    {
#pragma unroll
        for (int i = 0; i < E; ++i)
        {
            const int c = part + 8 * i;
            double value = c == r ? (mine ? diag : 1.0) : 0.0;
            if (mine && c != r && unknown(c))
            {
                if (x > 0 && c == r - 1)
                    value = -wl;
                if (x + 1 < l.w && c == r + 1)
                    value = -wr;
                if (c == r - l.w)
                    value = -wu;
                if (c == r + l.w)
                    value = -wd;
            }
            a[i] = value;
        }
    };
    form();
#pragma unroll
    for (int ki = 0; ki < E; ++ki)
    {
#pragma unroll 1
        for (int kp = 0; kp < 8; ++kp)
        {
            const int k = kp + 8 * ki, buf = kp & 1;
            if (k >= cells)
                break;
            if (r == k)
            {
#pragma unroll
                for (int i = 0; i < E; ++i)
                    pivot_row[buf][part + 8 * i] = a[i];
            }
            if (part == kp)
                pivot_col[buf][r] = a[ki];
            __syncthreads();
            const double pivot = pivot_row[buf][k];
            // (Rows that are no unknown have the pivot one.)
            if (r == k && mine && !(pivot > kSealedPivot * largest))
                sealed = 1;
            const double scale = 1.0 / pivot;
            if (r == k)
            {
#pragma unroll
                for (int i = 0; i < E; ++i)
                    a[i] *= scale;
                if (part == kp)
                    a[ki] = scale;
            }
            else
            {
                const double f = pivot_col[buf][r] * scale;
#pragma unroll
                for (int i = 0; i < E; ++i)
                    a[i] -= f * pivot_row[buf][part + 8 * i];
                if (part == kp)
                    a[ki] = -f;
            }
        }
    }
    __syncthreads();
    const bool exact = sealed != 0;
    bool failed = false;
    if (exact)
    {
        form();
        CoarseRow row{{}, r, part};
#pragma unroll
        for (int i = 0; i < E; ++i)
            row.a[i] = a[i];
        failed = invert_factor(row, diagonal, unknowns, cells, g.coarse_inverse);
#pragma unroll
        for (int i = 0; i < E; ++i)
            a[i] = row.a[i];
    }
    // Row sums (the matrix is symmetric: a column's is its row's).
    double sum = 0.0;
#pragma unroll
    for (int i = 0; i < E; ++i)
    {
        if (!mine || !unknown(part + 8 * i))
            a[i] = 0.0;
        sum += a[i];
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
    const double share = open_mask && !dirichlet ? 1.0 / __popcll(open_mask) : 0.0;
    // C a C over the open cells, unless the solve takes the means.
    const double fold = exact ? 0.0 : share;
    const double own_mean = sum * fold;
    if (part == 0)
        row_mean[r] = own_mean;
    __syncthreads();
    const double mean = fold * warp_sum(row_mean[lane] + row_mean[lane + 32]);
    if (r < cells)
    {
#pragma unroll
        for (int i = 0; i < E; ++i)
        {
            const int c = part + 8 * i;
            if (c >= cells)
                continue;
            g.coarse_inverse[r * kTailInverseStride + c] =
                open[r] && open[c] ? ((a[i] - own_mean) - row_mean[c]) + mean : 0.0;
        }
        if (part == 0)
        {
            g.coarse_inverse[TailMeans::sums(r)] = sum;
            g.coarse_inverse[TailMeans::open(r)] = open[r];
        }
    }
    if (threadIdx.x == 0)
    {
        g.coarse_inverse[TailMeans::share] = share - fold;
        g.state->mg_valid = failed ? 0 : 1;
    }
}

} // namespace fc
