// Multigrid preconditioner of the UniformCUDA projection: one fixed V-cycle, z = M r.
//
// Same preconditioner as the reference PressureMultigrid (PressureMultigrid.cpp): levels
// halve (rounding up) until at most 64 cells remain; conductances combine in series/parallel;
// four red-black Gauss-Seidel sweeps before (the first from zero) and after (colours reversed)
// the coarse correction; transpose-bilinear restriction, bilinear prolongation; the coarsest
// level is solved directly with one cell pinned, then given a mean-zero gauge.
//
// B200 mapping:
//  * k_smooth_pre / k_smooth_post (fc_stage.cuh): temporally blocked smoothing of one level per launch,
//    with the residual and restriction fused into the pre kernel and the prolongation and the
//    fine-level z reductions fused into the post kernel.
//  * k_mg_tail (fc_tail.cuh): the coarse levels of at most 64 x 64 cells are cycled by one CTA per
//    grid as register strips, including the coarsest direct solve (an explicit FP64 inverse).
//  * The rebuild: k_rebuild_level (one coarse cell per thread) down to the tail, then
//    k_rebuild_tail (fc_tail.cuh) for the rest and the coarsest inverse.
#pragma once

#include "fc_device.cuh"
#include "fc_smooth.cuh"
#include "fc_tma.cuh"

namespace fc
{

// Finishes a preconditioner application: z's mean, r.(z - mean z) and beta.
// FluidGridCPU.cpp:1712-1726 (applyPreconditioner) and :1806-1818 (beta, loop condition).
__device__ __forceinline__ void finish_preconditioner(SolveState& s, double sum_z, double sum_rz)
{
    const double mean_z = sum_z * s.inv_cells;
    const double rz = sum_rz - mean_z * s.sum_r;
    const double beta = s.restart ? 0.0 : rz / s.rz;
    s.mean_z = mean_z;
    s.beta = beta;
    s.restart = 0;
    s.rz = rz;
    if (!isfinite(beta) || !(rz > 0.0) || !isfinite(rz))
    {
        s.status = kStalled;
        s.done = 1;
    }
}

// Diagonal (Jacobi) preconditioner: z = (r - mean r) / diag. FluidGridCPU.cpp:1691-1698.
template <typename T, int CELLS, int SUM>
__global__ void __launch_bounds__(kVecThreads) k_precondition_diagonal(const GridDesc* grids, const Tile* tiles)
{
    allow_dependents();
    const Tile t = tiles[blockIdx.x];
    const GridDesc& g = grids[t.grid];
    SolveState& s = *g.state;
    dependency_wait();
    if (s.done)
        return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const T* right = static_cast<const T*>(g.lev[0].right);
    const T* down = static_cast<const T*>(g.lev[0].down);
    const T* r = static_cast<const T*>(g.r);
    T* z = static_cast<T*>(g.z);
    const double mean_r = s.mean_r;
    double4 acc[CELLS / SUM] = {};
#pragma unroll
    for (int k = 0; k < CELLS; ++k)
    {
        const int x = t.x0 + tx + 32 * (k & 1), y = t.y0 + ty + 8 * (k >> 1);
        if (x >= g.W || y >= g.H)
            continue;
        const long long i = padded_index(g.S, x, y);
        const double sum = ((double(right[i - 1]) + double(right[i])) + double(down[i - g.S])) + double(down[i]);
        const double inv = sum > 0.0 ? 1.0 / sum : 0.0;
        const T value = g.air && g.air[(long long)y * g.W + x] ? T(0) : T((double(r[i]) - mean_r) * inv);
        z[i] = value;
        if (g.solid && g.solid[(long long)y * g.W + x])
            continue;
        acc[k / SUM].x += double(value);
        acc[k / SUM].y += double(r[i]) * double(value);
    }
    __shared__ double4 total;
    if (arrive_tile<kVecThreads, 2>(g, t, acc, &total, 0))
    {
        if (threadIdx.x == 0)
            finish_preconditioner(s, total.x, total.y);
    }
}

// ------------------------------------------------------------------------------------------
// Rebuild: coarse conductances and the coarsest inverse
// ------------------------------------------------------------------------------------------

// Dirichlet air (no reference counterpart): a cell held at zero. On the fine level the air
// cells; on a coarse level the cells none of whose fine cells (2x .. 2x+1, 2y .. 2y+1 of the
// level above, whose inverse diagonal is final) is an unknown. A held cell keeps its face
// weights, so the unknowns beside it see the zero: the p = 0 boundary on every level.
template <typename T> __device__ __forceinline__ bool held_cell(const GridDesc& g, int level, int x, int y)
{
    if (level == 0)
        return g.air[(long long)y * g.W + x] != 0;
    const LevelDesc& F = g.lev[level - 1];
    const T* inv = static_cast<const T*>(F.inv);
    for (int dy = 0; dy < 2; ++dy)
        for (int dx = 0; dx < 2; ++dx)
        {
            const int fx = 2 * x + dx, fy = 2 * y + dy;
            if (fx < F.w && fy < F.h && inv[padded_index(F.S, fx, fy)] > T(0))
                return false;
        }
    return true;
}

// FP16 copy of a face weight of a mixed-precision coarse level, divided by the level's scale and
// saturated at the largest finite FP16 value; the smoothing kernels read it times the scale.
__device__ __forceinline__ __half half_weight(float w, float inv_scale) { return __float2half_rn(fminf(w * inv_scale, 65504.0f)); }

// Inverse diagonal of cell (x, y) of a smoothed level: 1 / (((left + right) + up) + down) over its
// face weights as the kernels decode them (`half`: the FP16 copies times the level scale), 0 where the
// sum is not positive (PressureMultigrid.cpp:104-117).
template <typename T>
__device__ __forceinline__ T inverse_diagonal(const GridDesc& g, const LevelDesc& L, int level, bool half, int x, int y)
{
    const long long i = padded_index(L.S, x, y);
    const T* right = static_cast<const T*>(L.right);
    const T* down = static_cast<const T*>(L.down);
    T wl = right[i - 1], wr = right[i], wu = down[i - L.S], wd = down[i];
    if constexpr (sizeof(T) == 4)
    {
        if (half)
        {
            const float inv = 1.0f / L.wscale;
            wl = __half2float(half_weight(wl, inv)) * L.wscale;
            wr = __half2float(half_weight(wr, inv)) * L.wscale;
            wu = __half2float(half_weight(wu, inv)) * L.wscale;
            wd = __half2float(half_weight(wd, inv)) * L.wscale;
        }
    }
    const T diag = ((wl + wr) + wu) + wd;
    if (g.air && held_cell<T>(g, level, x, y))
        return T(0);
    return diag > T(0) ? reciprocal(diag) : T(0);
}

// Everything that follows from level `level` around coarse cell (x, y) of the next one: the inverse
// diagonals of its up to four fine cells (and, in mixed precision, the FP16 copies of their weights),
// and the coarse cell's conductances (PressureMultigrid.cpp:142-202, coarsen).
template <typename T> __device__ __forceinline__ void rebuild_cell(const GridDesc& g, int level, int x, int y)
{
    const LevelDesc& f = g.lev[level];
    const LevelDesc& c = g.lev[level + 1];
    const T* fr = static_cast<const T*>(f.right);
    const T* fd = static_cast<const T*>(f.down);
    bool half = false;
    if constexpr (sizeof(T) == 4)
        half = f.right_h != nullptr && level >= 1 && level < g.tail;
    const int fy_end = min(2 * y + 2, f.h), fx_end = min(2 * x + 2, f.w);
    for (int fy = 2 * y; fy < fy_end; ++fy)
        for (int fx = 2 * x; fx < fx_end; ++fx)
        {
            const long long i = padded_index(f.S, fx, fy);
            static_cast<T*>(f.inv)[i] = inverse_diagonal<T>(g, f, level, half, fx, fy);
            if constexpr (sizeof(T) == 4)
            {
                if (half)
                {
                    const float inv = 1.0f / f.wscale;
                    static_cast<__half*>(const_cast<void*>(f.right_h))[i] = half_weight(fr[i], inv);
                    static_cast<__half*>(const_cast<void*>(f.down_h))[i] = half_weight(fd[i], inv);
                }
            }
        }
    double right = 0.0, down = 0.0;
    if (x + 1 < c.w)
    {
        const int e = 2 * x + 2;
        const double a = (f.cx[e - 1] - c.cx[x]) / (f.cx[e - 1] - f.cx[e - 2]);
        const double b = e + 1 < f.w ? (c.cx[x + 1] - f.cx[e]) / (f.cx[e + 1] - f.cx[e]) : 0.0;
        for (int fy = 2 * y; fy < fy_end; ++fy)
        {
            const long long i = padded_index(f.S, e - 1, fy); // fine cell 2x+1: its right face is the coarse face
            double resistance = a / double(fr[i - 1]) + 1.0 / double(fr[i]);
            if (b != 0.0)
                resistance += b / double(fr[i + 1]);
            right += 1.0 / resistance;
        }
    }
    if (y + 1 < c.h)
    {
        const int e = 2 * y + 2;
        const double a = (f.cy[e - 1] - c.cy[y]) / (f.cy[e - 1] - f.cy[e - 2]);
        const double b = e + 1 < f.h ? (c.cy[y + 1] - f.cy[e]) / (f.cy[e + 1] - f.cy[e]) : 0.0;
        for (int fx = 2 * x; fx < fx_end; ++fx)
        {
            const long long i = padded_index(f.S, fx, e - 1); // fine cell 2y+1: its lower face is the coarse face
            double resistance = a / double(fd[i - f.S]) + 1.0 / double(fd[i]);
            if (b != 0.0)
                resistance += b / double(fd[i + f.S]);
            down += 1.0 / resistance;
        }
    }
    const long long ci = padded_index(c.S, x, y);
    static_cast<T*>(c.right)[ci] = T(right);
    static_cast<T*>(c.down)[ci] = T(down);
}

// The rebuild of one level above the tail (blockIdx.y = grid), one thread per coarse cell: the FP64
// divisions of a cell form a long dependent chain, so the kernel needs many cells in flight rather
// than many cells per thread. The levels from the tail on are rebuilt by one CTA (k_rebuild_tail).
template <typename T> __global__ void k_rebuild_level(const GridDesc* __restrict__ grids, int level)
{
    dependent_start();
    const GridDesc& g = grids[blockIdx.y];
    if (level >= g.tail)
        return;
    const LevelDesc& c = g.lev[level + 1];
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < c.w * c.h)
        rebuild_cell<T>(g, level, q % c.w, q / c.w);
}

} // namespace fc
