// Implicit viscosity of the UniformCUDA step: backward Euler
//   m (v - v0) = -dt K v,   K = the Hessian of the strain energy sum mu (normal^2 + shear^2),
// solved by CG with a damped-Jacobi multigrid preconditioner.
//
// Follows the reference's GPU solver (FluidSim/UniformWebGPU/ViscosityKernels.h:8-400 and
// ViscositySolverGPU.cpp:61-294): the same operator, diagonal, smoother, transfers, V-cycle,
// CG recurrences and 4-iteration true-residual check. Vectors are in the working precision;
// every reduction and CG scalar is FP64.
//
// A pass is bound by instructions and launches more than by bytes (206 instructions a node and 41 %
// of DRAM peak in a sweep that formed its diagonal and mask; 2.5 to 3 us for a pass of a small
// level), so the V-cycle takes few of them: the sweep from zero is written by whatever writes its
// right-hand side, the residual is restricted where it is formed (k_visc_restrict), the prolongation
// is swept where it is formed (k_visc_prolong_smooth), and the small levels run in one CTA
// (k_visc_tail): 17 launches a CG iteration instead of 41 at 321 x 239. Measured, whole solves in
// FP32 from one pass per step of the method to this form, on one box: 321 x 239 6.72 -> 4.42 ms,
// 4096 x 4096 189 -> 164 ms.
//
// Layout: the (w+1) x (h+1) node lattice of a level, row-major; node p holds u face p (x) and v
// face p (y) as one 2-vector, and 4 coefficients (cell mu, vertex mu, u-face mass, v-face mass).
// Reads outside a field clamp to its edge, as the reference's field accessor does. One thread
// per node, 1D blocks of kViscThreads. The V-cycle and CG kernels are launched as programmatic
// dependents of their predecessor and wait for it (dependency_wait) before their first memory
// access, so only the launch itself overlaps the kernel before.
#pragma once

#include "fc_device.cuh"

namespace fc
{

constexpr int kViscThreads = 256;
// Nodes per thread of the kernels that end in a grid reduction: a block covers this many runs
// of kViscThreads consecutive nodes, so the per-block reduction, fence and atomic are paid a
// quarter as often.
constexpr int kViscReduceNodes = 4;

template <typename T> struct Vec;
template <> struct Vec<float>
{
    using two = float2;
    using four = float4;
};
template <> struct Vec<double>
{
    using two = double2;
    using four = double4;
};

// CG state of one solve (device). Written by the last block of each reduction.
struct ViscState
{
    double rz, alpha, beta;
    double target;     // tol^2 |x0|^2_M + 1e-12 total mass
    double rnorm;      // recurrence residual, sum r.r / m
    double truth;      // true residual of the last check
    double energy;     // |x0|^2_M (twice the initial kinetic energy)
    double total_mass;
    int count;         // alpha updates since the last (re)start
    int stopped;       // recurrence residual reached the target
    int breakdown;     // non-positive curvature or non-finite value
    int pad;
};

struct ViscLevel
{
    int w, h;
    double dx;
    const void* material; // 2 per cell (density, viscosity)
    const void* coeff;    // 4 per node
    const void* half;     // 2 per node: half the inverse diagonal, zero where there is no open face
    void* x;
    void* next;
    void* rhs;
};

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ bool valid_u_face(int w, int h, int x, int y) { return x > 0 && x < w && y < h; }
__device__ __forceinline__ bool valid_v_face(int w, int h, int x, int y) { return y > 0 && y < h && x < w; }

// Faces of obstacle cells are closed on the finest level (no reference counterpart: the
// reference has only the outer walls).
__device__ __forceinline__ bool solid_at(const unsigned char* solid, int w, int x, int y)
{
    return solid && solid[(long long)y * w + x];
}

// Deterministic two-level reduction. Blocks arrive in fixed groups of NT consecutive blocks:
// the last block of a group to arrive folds the group's partials (one per thread, then
// block_reduce4's fixed tree) into a group sum, and the last group to finish folds the group
// sums (each thread a contiguous run, in index order). No serial chain is longer than two
// loads per thread, and the order of every sum is set by the block indices, not by arrival.
// partial holds blocks + groups slots; counter[0] counts finished groups and counter[1 + g] the
// arrivals in group g (viscosity_layout sizes both).
template <int NT>
__device__ bool visc_arrive_last(double4* partial, unsigned int* counter, int index, int blocks, double4 mine,
    double4* total, int max_mask)
{
    __shared__ int is_last;
    const int group = index / NT, groups = (blocks + NT - 1) / NT;
    const int first = group * NT, members = min(NT, blocks - first);
    if (threadIdx.x == 0)
    {
        partial[index] = mine;
        __threadfence();
        is_last = atomicAdd(counter + 1 + group, 1u) == unsigned(members - 1);
    }
    __syncthreads();
    if (!is_last)
        return false;
    __threadfence();
    const double2* slots = reinterpret_cast<const double2*>(partial);
    double4 v = make_double4(0, 0, 0, 0);
    if (int(threadIdx.x) < members)
    {
        const double2 lo = __ldcg(slots + 2 * (first + threadIdx.x)), hi = __ldcg(slots + 2 * (first + threadIdx.x) + 1);
        v = make_double4(lo.x, lo.y, hi.x, hi.y);
    }
    const double4 group_total = block_reduce4<NT>(v, max_mask);
    if (threadIdx.x == 0)
    {
        partial[blocks + group] = group_total;
        counter[1 + group] = 0u;
        __threadfence();
        is_last = atomicAdd(counter, 1u) == unsigned(groups - 1);
    }
    __syncthreads();
    if (!is_last)
        return false;
    __threadfence();
    const int per = (groups + NT - 1) / NT;
    const int a = threadIdx.x * per, b = min(groups, a + per);
    double4 acc = make_double4(0, 0, 0, 0);
    for (int t = a; t < b; ++t)
    {
        const double2 lo = __ldcg(slots + 2 * (blocks + t)), hi = __ldcg(slots + 2 * (blocks + t) + 1);
        acc.x = (max_mask & 1) ? fmax(acc.x, lo.x) : acc.x + lo.x;
        acc.y = (max_mask & 2) ? fmax(acc.y, lo.y) : acc.y + lo.y;
        acc.z = (max_mask & 4) ? fmax(acc.z, hi.x) : acc.z + hi.x;
        acc.w = (max_mask & 8) ? fmax(acc.w, hi.y) : acc.w + hi.y;
    }
    const double4 out = block_reduce4<NT>(acc, max_mask);
    if (threadIdx.x == 0)
    {
        *total = out;
        *counter = 0u;
        __threadfence();
    }
    __syncthreads();
    return true;
}

// ---------------------------------------------------------------------------------------------
// Set-up: material, coarse material, coefficients
// ---------------------------------------------------------------------------------------------

// Cell density sum m / dx^2 and volume-weighted viscosity sum(m mu/rho) / sum(m / rho)
// (FluidGridGPU.cpp:172-217, 987-1037); comp[k] = (mu_k / rho_k, 1 / rho_k). A cell without
// mass gets viscosity 0.
template <typename T>
__global__ void k_visc_material(const double* const* masses, int components, const double2* comp, int cells,
    double inv_area, void* material)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cells)
        return;
    double total = 0.0, weighted = 0.0, volume = 0.0;
    for (int k = 0; k < components; ++k)
    {
        const double m = masses[k][i];
        total += m;
        weighted += m * comp[k].x;
        volume += m * comp[k].y;
    }
    using T2 = typename Vec<T>::two;
    T2 out;
    out.x = T(total * inv_area);
    out.y = T(volume > 0.0 ? weighted / volume : 0.0);
    static_cast<T2*>(material)[i] = out;
}

// Mean of the existing fine cells of each 2x2 block (ViscosityKernels.h "coarse material").
template <typename T>
__global__ void k_visc_coarsen(const void* fine, int fw, int fh, void* coarse, int cw, int ch)
{
    using T2 = typename Vec<T>::two;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cw * ch)
        return;
    const int x = i % cw, y = i / cw;
    T a = 0, b = 0, n = 0;
    for (int j = 0; j < 2; ++j)
        for (int k = 0; k < 2; ++k)
        {
            const int qx = 2 * x + k, qy = 2 * y + j;
            if (qx < fw && qy < fh)
            {
                const T2 m = static_cast<const T2*>(fine)[(long long)qy * fw + qx];
                a += m.x;
                b += m.y;
                n += T(1);
            }
        }
    T2 out;
    out.x = a / n;
    out.y = b / n;
    static_cast<T2*>(coarse)[i] = out;
}

// Node coefficients (ViscosityKernels.h "viscosity coefficients"): cell mu, the mean mu of the
// four cells around an interior vertex, and the face masses rho_face dx^2.
template <typename T>
__global__ void k_visc_coefficients(const void* material, int w, int h, double dx, void* coeff)
{
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (w + 1) * (h + 1))
        return;
    const int x = n % (w + 1), y = n / (w + 1);
    const T2* m = static_cast<const T2*>(material);
    auto at = [&](int cx, int cy) { return m[(long long)clampi(cy, 0, h - 1) * w + clampi(cx, 0, w - 1)]; };
    const T2 c = at(x, y);
    T mu = 0;
    if (x > 0 && y > 0 && x < w && y < h)
        mu = T(0.25) * (c.y + at(x - 1, y).y + at(x, y - 1).y + at(x - 1, y - 1).y);
    const T area = T(dx * dx);
    T4 out;
    out.x = c.y;
    out.y = mu;
    out.z = T(0.5) * area * (c.x + at(x - 1, y).x);
    out.w = T(0.5) * area * (c.x + at(x, y - 1).x);
    static_cast<T4*>(coeff)[n] = out;
}

// ---------------------------------------------------------------------------------------------
// Operator (ViscosityKernels.h:8-75)
// ---------------------------------------------------------------------------------------------

// Offsets of a node and its neighbours in a row-major lattice, with the reference's clamps: left,
// right, up, down, and the two diagonal ones that the shear terms read.
struct Around
{
    int own, left, right, up, down, down_left, up_right;
};

__device__ __forceinline__ Around around(int w, int h, int x, int y)
{
    const int row = y * (w + 1), above = max(y - 1, 0) * (w + 1), below = min(y + 1, h) * (w + 1);
    const int left = max(x - 1, 0), right = min(x + 1, w);
    return {row + x, row + left, row + right, above + x, below + x, below + left, above + right};
}

// mass f + dt stress(f) for both components of a node, before the valid-face mask: f at the offsets
// n, the node's own coefficients and those of its neighbours that the operator reads (the cell
// viscosities to the left and above, the vertex viscosities below and to the right).
template <typename T>
__device__ __forceinline__ void operator_terms(const typename Vec<T>::two* f, const Around& n, const typename Vec<T>::four& a,
    T mu_left, T mu_up, T vertex_down, T vertex_right, T dt, T& ax, T& ay)
{
    const auto c = f[n.own], fl = f[n.left], fr = f[n.right], fu = f[n.up], fd = f[n.down];
    const T down_left = f[n.down_left].y, up_right = f[n.up_right].x;
    const T t = a.y * ((c.x - fu.x) + (c.y - fl.y));
    const T below = vertex_down * ((fd.x - c.x) + (fd.y - down_left));
    const T beside = vertex_right * ((fr.x - up_right) + (fr.y - c.y));
    const T nx = T(2) * (mu_left * (c.x - fl.x) + a.x * (c.x - fr.x));
    const T ny = T(2) * (mu_up * (c.y - fu.y) + a.x * (c.y - fd.y));
    ax = a.z * c.x + dt * (nx + (t - below));
    ay = a.w * c.y + dt * (ny + (t - beside));
}

// The same with the coefficients at the offsets m.
template <typename T>
__device__ __forceinline__ void operator_at(const typename Vec<T>::two* f, const Around& n, const typename Vec<T>::four* coeff,
    const Around& m, T dt, T& ax, T& ay)
{
    operator_terms<T>(f, n, coeff[m.own], coeff[m.left].x, coeff[m.up].x, coeff[m.down].y, coeff[m.right].y, dt, ax, ay);
}

struct FaceMask
{
    bool u, v;
};

__device__ __forceinline__ FaceMask face_mask(int w, int h, int x, int y, const unsigned char* solid)
{
    FaceMask m{valid_u_face(w, h, x, y), valid_v_face(w, h, x, y)};
    if (solid)
    {
        if (m.u && (solid_at(solid, w, x - 1, y) || solid_at(solid, w, x, y)))
            m.u = false;
        if (m.v && (solid_at(solid, w, x, y - 1) || solid_at(solid, w, x, y)))
            m.v = false;
    }
    return m;
}

// Half the inverse of a face's diagonal, zero for a closed face. Of an infinite diagonal (a viscosity
// or a mass beyond the working precision) it is no number, not the zero that would close the face:
// such a solve ends as nonfinite.
template <typename T> __device__ __forceinline__ T half_inverse(bool open, T diagonal)
{
    if (!open)
        return T(0);
    return isinf(diagonal) ? T(NAN) : T(0.5) / diagonal;
}

// Half the inverse diagonal of a level's operator, once per solve: the damped Jacobi sweep is then a
// multiplication (the two divisions and the face mask were a quarter of its instructions).
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_diagonal(ViscLevel lv, double dt, const unsigned char* solid, void* half)
{
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (lv.w + 1) * (lv.h + 1))
        return;
    const int x = n % (lv.w + 1), y = n / (lv.w + 1);
    const FaceMask m = face_mask(lv.w, lv.h, x, y, solid);
    const Around o = around(lv.w, lv.h, x, y);
    const T4* coeff = static_cast<const T4*>(lv.coeff);
    const T4 c = coeff[o.own];
    const T dx = c.z + T(dt) * (T(2) * (c.x + coeff[o.left].x) + c.y + coeff[o.down].y);
    const T dy = c.w + T(dt) * (T(2) * (c.x + coeff[o.up].x) + c.y + coeff[o.right].y);
    static_cast<T2*>(half)[n] = T2{half_inverse(m.u, dx), half_inverse(m.v, dy)};
}

__device__ __forceinline__ bool visc_stopped(const ViscState* s) { return s->stopped || s->breakdown; }

// out = A f on valid faces (ViscosityKernels.h "apply"), and d.Ad reduced into the CG step length
// alpha (ViscosityKernels.h "scalar" mode 2).
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_apply(ViscLevel lv, double dt, const void* f, void* out,
    ViscState* state, double4* partial, unsigned int* counter)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    const bool stopped = visc_stopped(state);
    double dq = 0.0;
#pragma unroll 1
    for (int k = 0; k < kViscReduceNodes && !stopped; ++k)
    {
        const int n = (blockIdx.x * kViscReduceNodes + k) * blockDim.x + threadIdx.x;
        if (n >= (lv.w + 1) * (lv.h + 1))
            break;
        const Around o = around(lv.w, lv.h, n % (lv.w + 1), n / (lv.w + 1));
        const T2 half = static_cast<const T2*>(lv.half)[n];
        T ax, ay;
        operator_at<T>(static_cast<const T2*>(f), o, static_cast<const T4*>(lv.coeff), o, T(dt), ax, ay);
        T2 r;
        r.x = half.x != T(0) ? ax : T(0);
        r.y = half.y != T(0) ? ay : T(0);
        const T2 d = static_cast<const T2*>(f)[n];
        dq += double(d.x) * double(r.x) + double(d.y) * double(r.y);
        static_cast<T2*>(out)[n] = r;
    }
    double4 total;
    if (visc_arrive_last<kViscThreads>(partial, counter, blockIdx.x, gridDim.x,
            block_reduce4<kViscThreads>(make_double4(dq, 0, 0, 0), 0), &total, 0))
    {
        if (threadIdx.x == 0 && !stopped)
        {
            if (!(total.x > 0.0) || !isfinite(total.x))
                state->breakdown = 1;
            else
            {
                state->alpha = state->rz / total.x;
                state->count += 1;
            }
        }
    }
}

// Damped Jacobi (ViscosityKernels.h "smooth"): x + (b - A x) / (2 D). The sweep from zero, b / (2 D),
// has no kernel: whatever writes b writes it to x as well.
template <typename T>
__device__ __forceinline__ typename Vec<T>::two jacobi(const typename Vec<T>::two& c, const typename Vec<T>::two& b,
    const typename Vec<T>::two& half, T ax, T ay)
{
    typename Vec<T>::two out;
    out.x = half.x != T(0) ? c.x + (b.x - ax) * half.x : T(0);
    out.y = half.y != T(0) ? c.y + (b.y - ay) * half.y : T(0);
    return out;
}

template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_smooth(ViscLevel lv, double dt, const void* b, const ViscState* state)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (lv.w + 1) * (lv.h + 1) || visc_stopped(state))
        return;
    const Around o = around(lv.w, lv.h, n % (lv.w + 1), n / (lv.w + 1));
    const T2* x = static_cast<const T2*>(lv.x);
    T ax, ay;
    operator_at<T>(x, o, static_cast<const T4*>(lv.coeff), o, T(dt), ax, ay);
    static_cast<T2*>(lv.next)[n] =
        jacobi<T>(x[n], static_cast<const T2*>(b)[n], static_cast<const T2*>(lv.half)[n], ax, ay);
}

// Statistics a residual pass reduces (ViscosityKernels.h "first_reduce" modes 0 and 3).
enum ViscResidualMode
{
    kResidualInitial = 1, // |r|^2_M, |x|^2_M, total mass; sets the target
    kResidualTruth = 2    // |r|^2_M into state->truth
};

// out = b - A f on valid faces; the initial one also starts the V-cycle's sweep from zero (lv.x).
template <typename T, int kMode>
__global__ void __launch_bounds__(kViscThreads) k_visc_residual(ViscLevel lv, double dt, const void* f, const void* b,
    void* out, ViscState* state, double4* partial, unsigned int* counter, double tolerance)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    double4 mine = make_double4(0, 0, 0, 0);
#pragma unroll 1
    for (int k = 0; k < kViscReduceNodes; ++k)
    {
        const int n = (blockIdx.x * kViscReduceNodes + k) * blockDim.x + threadIdx.x;
        if (n >= (lv.w + 1) * (lv.h + 1))
            break;
        const Around o = around(lv.w, lv.h, n % (lv.w + 1), n / (lv.w + 1));
        const T2 half = static_cast<const T2*>(lv.half)[n];
        T ax, ay;
        operator_at<T>(static_cast<const T2*>(f), o, static_cast<const T4*>(lv.coeff), o, T(dt), ax, ay);
        const T2 bb = static_cast<const T2*>(b)[n];
        T2 r;
        r.x = half.x != T(0) ? bb.x - ax : T(0);
        r.y = half.y != T(0) ? bb.y - ay : T(0);
        static_cast<T2*>(out)[n] = r;
        const T4 c = static_cast<const T4*>(lv.coeff)[n];
        const double rx = r.x, ry = r.y;
        mine.x += rx / double(c.z) * rx + ry / double(c.w) * ry;
        if (kMode == kResidualInitial)
        {
            const T2 v = static_cast<const T2*>(f)[n];
            mine.y += double(c.z) * double(v.x) * double(v.x) + double(c.w) * double(v.y) * double(v.y);
            mine.z += double(c.z) + double(c.w);
            static_cast<T2*>(lv.x)[n] = T2{r.x * half.x, r.y * half.y};
        }
    }
    double4 total;
    if (visc_arrive_last<kViscThreads>(partial, counter, blockIdx.x, gridDim.x, block_reduce4<kViscThreads>(mine, 0),
            &total, 0))
    {
        if (threadIdx.x == 0)
        {
            const bool finite = isfinite(total.x) && isfinite(total.y) && isfinite(total.z);
            if (kMode == kResidualInitial)
            {
                // A new solve: earlier flags are cleared.
                state->breakdown = finite ? 0 : 1;
                state->rz = state->alpha = state->beta = 0.0;
                state->count = 0;
                state->stopped = 0;
                state->energy = total.y;
                state->total_mass = total.z;
                state->target = tolerance * tolerance * total.y + 1e-12 * total.z;
                state->rnorm = total.x;
                state->truth = total.x;
            }
            else
            {
                if (!finite)
                    state->breakdown = 1;
                state->truth = total.x;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Transfers (ViscosityKernels.h:290-400): bilinear interpolation at face locations and its
// exact transpose, with the reference's tangential clamps.
// ---------------------------------------------------------------------------------------------


__device__ __forceinline__ void transfer_clamp(int bx, int by, int component, int cw, int ch, int& cx, int& cy)
{
    cx = clampi(bx, 0, cw - (component == 1 ? 1 : 0));
    cy = clampi(by, 0, ch - (component == 1 ? 0 : 1));
}

// Coarse coordinate of fine index f along an axis with face offset `half` (0 or 1/2):
// l = (f + half) / 2 - half, returned as b = floor(l) and t = l - b. Both are exact in integer
// arithmetic: t is 0 or 1/2 without the offset, 3/4 or 1/4 with it.
__device__ __forceinline__ void transfer_axis(int f, bool half, int& b, double& t)
{
    if (half)
    {
        b = (f - 1) >> 1; // arithmetic shift: floor((f - 1) / 2)
        t = (f & 1) ? 0.25 : 0.75;
    }
    else
    {
        b = f >> 1;
        t = (f & 1) ? 0.5 : 0.0;
    }
}

// Weight of fine index f in coarse index p along one axis whose coarse indexes are clamped to
// [0, limit]. The clamps of the two axes are independent, so a stencil weight is the product of its
// axes' weights (all of them and their sums exact in binary).
__device__ __forceinline__ double transfer_weight(int f, bool half, int p, int limit)
{
    int b;
    double t;
    transfer_axis(f, half, b, t);
    return (clampi(b, 0, limit) == p ? 1.0 - t : 0.0) + (clampi(b + 1, 0, limit) == p ? t : 0.0);
}

// Coarse tile of a restriction block, and the fine nodes its stencils cover.
constexpr int kViscTileX = 32, kViscTileY = 8;
constexpr int kViscFineX = 2 * kViscTileX + 2, kViscFineY = 2 * kViscTileY + 2;

// Origin of a block's tile in a lattice of w + 1 columns. The tiles are counted in one grid dimension:
// a tall thin lattice has more rows of them than a second one holds.
__device__ __forceinline__ void visc_tile(int w, int& x0, int& y0)
{
    const int columns = w / kViscTileX + 1; // ceil((w + 1) / kViscTileX)
    x0 = int(blockIdx.x % columns) * kViscTileX;
    y0 = int(blockIdx.x / columns) * kViscTileY;
}

// The coarse right-hand side at node (px, py): the transpose of the prolongation applied to the 4 x 4
// fine residuals 2p - 1 .. 2p + 2, q(row, column), summed in the stencil's row order.
template <typename T, typename Q>
__device__ __forceinline__ typename Vec<T>::two restrict_node(int px, int py, int cw, int ch, int fw, int fh, Q&& q)
{
    double value[2] = {0.0, 0.0};
    if (px >= 2 && py >= 2 && px <= cw - 3 && py <= ch - 3)
    {
        // No clamp reaches a node two or more from every edge: each stencil weight is the
        // product of the 1D weights (1/2, 1, 1/2) along the face's own axis and
        // (1/4, 3/4, 3/4, 1/4) across it, exactly transfer_weight's value.
        constexpr double kNear[3] = {0.5, 1.0, 0.5};
        constexpr double kFar[4] = {0.25, 0.75, 0.75, 0.25};
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int x = 0; x < 3; ++x)
                value[0] += kNear[x] * kFar[y] * double(q(y, x).x);
#pragma unroll
        for (int y = 0; y < 3; ++y)
#pragma unroll
            for (int x = 0; x < 4; ++x)
                value[1] += kFar[x] * kNear[y] * double(q(y, x).y);
    }
    else
    {
        // Near an edge: each axis's weights with its clamps, zero for fine nodes outside the lattice
        // and for faces on the walls.
        double across_x[4], along_x[4], across_y[4], along_y[4];
        const bool u = px != 0 && px != cw && py != ch, v = py != 0 && py != ch && px != cw;
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const int fx = 2 * px + i - 1, fy = 2 * py + i - 1;
            const bool in_x = fx >= 0 && fx <= fw, in_y = fy >= 0 && fy <= fh;
            along_x[i] = in_x && u && i < 3 ? transfer_weight(fx, false, px, cw) : 0.0;
            across_y[i] = in_y ? transfer_weight(fy, true, py, ch - 1) : 0.0;
            across_x[i] = in_x ? transfer_weight(fx, true, px, cw - 1) : 0.0;
            along_y[i] = in_y && v && i < 3 ? transfer_weight(fy, false, py, ch) : 0.0;
        }
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int x = 0; x < 4; ++x)
            {
                const auto r = q(y, x);
                if (x < 3)
                    value[0] += along_x[x] * across_y[y] * double(r.x);
                if (y < 3)
                    value[1] += across_x[x] * along_y[y] * double(r.y);
            }
    }
    return {T(value[0]), T(value[1])};
}

// Residual of the fine level and its restriction in one kernel: a block forms the residuals under
// its coarse tile in shared memory (66 x 18 of them for 64 x 16 fine nodes of its own, 16 % more work
// than a pass of its own, against 16 bytes a node written and read back and a launch), then each
// thread restricts one coarse node, and starts the coarse level's sweep from zero (`start`: the
// level is smoothed by kernels of its own).
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_restrict(ViscLevel fine, ViscLevel coarse, double dt, const void* b,
    int start, const ViscState* state)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    __shared__ T2 res[kViscFineY][kViscFineX];
    if (visc_stopped(state))
        return;
    int X0, Y0;
    visc_tile(coarse.w, X0, Y0);
    for (int i = threadIdx.x; i < kViscFineX * kViscFineY; i += kViscThreads)
    {
        const int j = i / kViscFineX, k = i - j * kViscFineX;
        const int x = 2 * X0 - 1 + k, y = 2 * Y0 - 1 + j;
        T2 r{T(0), T(0)};
        if (x >= 0 && y >= 0 && x <= fine.w && y <= fine.h)
        {
            const Around o = around(fine.w, fine.h, x, y);
            T ax, ay;
            operator_at<T>(static_cast<const T2*>(fine.x), o, static_cast<const T4*>(fine.coeff), o, T(dt), ax, ay);
            const T2 bb = static_cast<const T2*>(b)[o.own], half = static_cast<const T2*>(fine.half)[o.own];
            r.x = half.x != T(0) ? bb.x - ax : T(0);
            r.y = half.y != T(0) ? bb.y - ay : T(0);
        }
        res[j][k] = r;
    }
    __syncthreads();
    const int lx = threadIdx.x % kViscTileX, ly = threadIdx.x / kViscTileX;
    const int px = X0 + lx, py = Y0 + ly;
    if (px > coarse.w || py > coarse.h)
        return;
    const T2 out = restrict_node<T>(px, py, coarse.w, coarse.h, fine.w, fine.h,
        [&](int j, int i) { return res[2 * ly + j][2 * lx + i]; });
    const int n = py * (coarse.w + 1) + px;
    static_cast<T2*>(coarse.rhs)[n] = out;
    if (start)
    {
        const T2 half = static_cast<const T2*>(coarse.half)[n];
        static_cast<T2*>(coarse.x)[n] = T2{out.x * half.x, out.y * half.y};
    }
}

// x plus the bilinear interpolation of the coarse correction at fine node (px, py), on valid faces;
// `coarse` is the correction's lattice, cw x ch cells.
template <typename T>
__device__ __forceinline__ typename Vec<T>::two prolong_node(const typename Vec<T>::two& own,
    const typename Vec<T>::two& half, const typename Vec<T>::two* coarse, int cw, int ch, int px, int py)
{
    T value[2] = {own.x, own.y};
#pragma unroll
    for (int component = 0; component < 2; ++component)
    {
        int bx, by;
        double tx, ty;
        transfer_axis(px, component == 1, bx, tx);
        transfer_axis(py, component == 0, by, ty);
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int x = 0; x < 2; ++x)
            {
                int cx, cy;
                transfer_clamp(bx + x, by + y, component, cw, ch, cx, cy);
                const auto v = coarse[cy * (cw + 1) + cx];
                value[component] += T((x == 1 ? tx : 1.0 - tx) * (y == 1 ? ty : 1.0 - ty)) * (component == 0 ? v.x : v.y);
            }
    }
    return {half.x != T(0) ? value[0] : T(0), half.y != T(0) ? value[1] : T(0)};
}

// The prolongation and the first post-smoothing sweep in one kernel: a block forms the prolonged
// solution of its 32 x 8 nodes and the ring around them in shared memory (1.33 times the nodes,
// against 16 bytes a node written and read back and a launch), then sweeps them (into fine.next).
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_prolong_smooth(ViscLevel fine, ViscLevel coarse, double dt,
    const void* b, const ViscState* state)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    constexpr int RX = kViscTileX + 2, RY = kViscTileY + 2;
    __shared__ T2 tile[RY * RX];
    if (visc_stopped(state))
        return;
    int X0, Y0;
    visc_tile(fine.w, X0, Y0);
    for (int i = threadIdx.x; i < RX * RY; i += kViscThreads)
    {
        // Clamped like the operator's reads: the ring beyond the lattice repeats its edge.
        const int j = i / RX, k = i - j * RX;
        const int x = clampi(X0 - 1 + k, 0, fine.w), y = clampi(Y0 - 1 + j, 0, fine.h);
        const int n = y * (fine.w + 1) + x;
        tile[i] = prolong_node<T>(static_cast<const T2*>(fine.x)[n], static_cast<const T2*>(fine.half)[n],
            static_cast<const T2*>(coarse.x), coarse.w, coarse.h, x, y);
    }
    __syncthreads();
    const int lx = threadIdx.x % kViscTileX, ly = threadIdx.x / kViscTileX;
    const int x = X0 + lx, y = Y0 + ly;
    if (x > fine.w || y > fine.h)
        return;
    const int at = (ly + 1) * RX + lx + 1;
    const Around t{at, at - 1, at + 1, at - RX, at + RX, at + RX - 1, at - RX + 1};
    const Around o = around(fine.w, fine.h, x, y);
    T ax, ay;
    operator_at<T>(tile, t, static_cast<const T4*>(fine.coeff), o, T(dt), ax, ay);
    static_cast<T2*>(fine.next)[o.own] =
        jacobi<T>(tile[at], static_cast<const T2*>(b)[o.own], static_cast<const T2*>(fine.half)[o.own], ax, ay);
}

// ---------------------------------------------------------------------------------------------
// Coarse tail: the small levels cycled by one CTA in shared memory
// ---------------------------------------------------------------------------------------------

// Below a few thousand nodes a pass is nothing but its launch (2.5 to 3 us each, five passes a level),
// so the V-cycle's last levels run in one CTA: coefficients, half inverse diagonals, right-hand sides
// and two solutions of every level in shared memory, a barrier between passes. Where a level has a
// thread for every node its sweeps keep all but the solution in registers, and stencil weights near
// the lattice's edges, which most nodes of these levels are, are products of their axes' weights
// (321 x 239, whole solve: 5.18 -> 4.11 ms with both). The coarsest level takes 16 damped-Jacobi
// sweeps from zero (ViscosityKernels.h "coarse_smooth").
constexpr int kViscTailThreads = 1024;
constexpr int kViscTailLevels = 8;

struct ViscTail
{
    int levels;
    ViscLevel lev[kViscTailLevels];
};

// Shared-memory bytes of one node of a tail level: four coefficients, two half inverse diagonals, the
// right-hand side and two solutions.
__host__ __device__ inline size_t visc_tail_bytes(int nodes, size_t elem) { return size_t(nodes) * 12 * elem; }

constexpr size_t kViscTailMaxBytes = 200 * 1024;
extern __shared__ __align__(16) unsigned char visc_smem[];

template <typename T>
__global__ void __launch_bounds__(kViscTailThreads) k_visc_tail(const ViscTail tail, double dt, const ViscState* state)
{
    allow_dependents();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    const T step = T(dt);
    // Level l's arrays: node counts add up, each array of all levels together.
    int base[kViscTailLevels + 1];
    base[0] = 0;
#pragma unroll
    for (int l = 0; l < kViscTailLevels; ++l)
        base[l + 1] = base[l] + (l < tail.levels ? (tail.lev[l].w + 1) * (tail.lev[l].h + 1) : 0);
    const int total = base[kViscTailLevels];
    T4* const coeff = reinterpret_cast<T4*>(visc_smem);
    T2* const half = reinterpret_cast<T2*>(coeff + total);
    T2* const rhs = half + total;
    T2* const xs = rhs + total;
    T2* const ys = xs + total;
    // Written once per solve, long before this launch: read ahead of the wait.
#pragma unroll
    for (int l = 0; l < kViscTailLevels; ++l)
        if (l < tail.levels)
            for (int n = threadIdx.x; n < base[l + 1] - base[l]; n += kViscTailThreads)
            {
                coeff[base[l] + n] = static_cast<const T4*>(tail.lev[l].coeff)[n];
                half[base[l] + n] = static_cast<const T2*>(tail.lev[l].half)[n];
            }
    dependency_wait();
    if (visc_stopped(state))
        return;
    for (int n = threadIdx.x; n < base[1]; n += kViscTailThreads)
        rhs[n] = static_cast<const T2*>(tail.lev[0].rhs)[n];
    __syncthreads();
    // `count` Jacobi sweeps of a level (its first node at o), from x to y, from y to x and so on. A level
    // of at most one node a thread keeps everything but x in registers; its idle warps wait at the end.
    auto sweeps = [&](int w, int h, int o, T2* x, T2* y, int count)
    {
        const int nodes = (w + 1) * (h + 1);
        if (nodes <= kViscTailThreads)
        {
            const int warps = (nodes + 31) / 32;
            const int n = min(int(threadIdx.x), nodes - 1);
            if (int(threadIdx.x) < 32 * warps)
            {
                const Around a = around(w, h, n % (w + 1), n / (w + 1));
                const T4* k = coeff + o;
                const T4 own = k[a.own];
                const T left = k[a.left].x, up = k[a.up].x, down = k[a.down].y, right = k[a.right].y;
                const T2 b = rhs[o + n], hd = half[o + n];
                for (int i = 0; i < count; ++i)
                {
                    const T2* f = (i & 1 ? y : x) + o;
                    T ax, ay;
                    operator_terms<T>(f, a, own, left, up, down, right, step, ax, ay);
                    (i & 1 ? x : y)[o + n] = jacobi<T>(f[n], b, hd, ax, ay);
                    if (i + 1 < count)
                        asm volatile("bar.sync 1, %0;" ::"r"(32 * warps) : "memory");
                }
            }
        }
        else
            for (int i = 0; i < count; ++i)
            {
                if (i > 0)
                    __syncthreads();
                const T2* f = (i & 1 ? y : x) + o;
                T2* g = (i & 1 ? x : y) + o;
                for (int n = threadIdx.x; n < nodes; n += kViscTailThreads)
                {
                    const Around a = around(w, h, n % (w + 1), n / (w + 1));
                    T ax, ay;
                    operator_at<T>(f, a, coeff + o, a, step, ax, ay);
                    g[n] = jacobi<T>(f[n], rhs[o + n], half[o + n], ax, ay);
                }
            }
        __syncthreads();
    };
#pragma unroll 1
    for (int l = 0; l < tail.levels; ++l)
    {
        const int w = tail.lev[l].w, h = tail.lev[l].h, o = base[l], nodes = (w + 1) * (h + 1);
        for (int n = threadIdx.x; n < nodes; n += kViscTailThreads)
            xs[o + n] = T2{rhs[o + n].x * half[o + n].x, rhs[o + n].y * half[o + n].y};
        __syncthreads();
        if (l + 1 == tail.levels)
        {
            // The first of the 16 sweeps is the one from zero.
            sweeps(w, h, o, xs, ys, 15);
            break;
        }
        sweeps(w, h, o, xs, ys, 1);
        // The residual of ys goes to xs, which the up leg's prolongation overwrites.
        for (int n = threadIdx.x; n < nodes; n += kViscTailThreads)
        {
            const Around a = around(w, h, n % (w + 1), n / (w + 1));
            T ax, ay;
            operator_at<T>(ys + o, a, coeff + o, a, step, ax, ay);
            xs[o + n] = T2{half[o + n].x != T(0) ? rhs[o + n].x - ax : T(0), half[o + n].y != T(0) ? rhs[o + n].y - ay : T(0)};
        }
        __syncthreads();
        const int cw = tail.lev[l + 1].w, ch = tail.lev[l + 1].h, co = base[l + 1];
        for (int n = threadIdx.x; n < (cw + 1) * (ch + 1); n += kViscTailThreads)
        {
            const int px = n % (cw + 1), py = n / (cw + 1);
            rhs[co + n] = restrict_node<T>(px, py, cw, ch, w, h,
                [&](int j, int i) { return xs[o + clampi(2 * py + j - 1, 0, h) * (w + 1) + clampi(2 * px + i - 1, 0, w)]; });
        }
        __syncthreads();
    }
    // Up: the solution of level l is in ys.
#pragma unroll 1
    for (int l = tail.levels - 2; l >= 0; --l)
    {
        const int w = tail.lev[l].w, h = tail.lev[l].h, o = base[l];
        const int cw = tail.lev[l + 1].w, ch = tail.lev[l + 1].h, co = base[l + 1];
        for (int n = threadIdx.x; n < (w + 1) * (h + 1); n += kViscTailThreads)
            ys[o + n] = prolong_node<T>(ys[o + n], half[o + n], ys + co, cw, ch, n % (w + 1), n / (w + 1));
        __syncthreads();
        sweeps(w, h, o, ys, xs, 2);
    }
    for (int n = threadIdx.x; n < base[1]; n += kViscTailThreads)
        static_cast<T2*>(tail.lev[0].x)[n] = ys[n];
}

// ---------------------------------------------------------------------------------------------
// CG on the finest level (ViscosityKernels.h "scalar", "direction", "update", "pack", "unpack")
// ---------------------------------------------------------------------------------------------

// r.z and |r|^2_M; sets beta, or stops when the recurrence residual reaches the target.
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_dot_rz(int nodes, const void* coeff, const void* r, const void* z,
    ViscState* state, double4* partial, unsigned int* counter)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    double4 mine = make_double4(0, 0, 0, 0);
    if (!visc_stopped(state))
    {
        T2 a[kViscReduceNodes], b[kViscReduceNodes];
        T4 c[kViscReduceNodes];
#pragma unroll
        for (int k = 0; k < kViscReduceNodes; ++k)
        {
            const int n = (blockIdx.x * kViscReduceNodes + k) * blockDim.x + threadIdx.x;
            if (n < nodes)
            {
                a[k] = static_cast<const T2*>(r)[n];
                b[k] = static_cast<const T2*>(z)[n];
                c[k] = static_cast<const T4*>(coeff)[n];
            }
        }
#pragma unroll
        for (int k = 0; k < kViscReduceNodes; ++k)
        {
            const int n = (blockIdx.x * kViscReduceNodes + k) * blockDim.x + threadIdx.x;
            if (n < nodes)
            {
                mine.x += double(a[k].x) * double(b[k].x) + double(a[k].y) * double(b[k].y);
                // r.x^2 / m.u + r.y^2 / m.v over one division.
                const double mu = double(c[k].z), mv = double(c[k].w), rx = double(a[k].x), ry = double(a[k].y);
                mine.y += (rx * rx * mv + ry * ry * mu) / (mu * mv);
            }
        }
    }
    double4 total;
    if (visc_arrive_last<kViscThreads>(partial, counter, blockIdx.x, gridDim.x, block_reduce4<kViscThreads>(mine, 0),
            &total, 0))
    {
        if (threadIdx.x == 0 && !visc_stopped(state))
        {
            state->rnorm = total.y;
            if (!isfinite(total.y))
                state->breakdown = 1;
            else if (total.y <= state->target)
                state->stopped = 1;
            else if (!(total.x > 0.0) || !isfinite(total.x))
                state->breakdown = 1;
            else
            {
                state->beta = state->count > 0 ? total.x / state->rz : 0.0;
                state->rz = total.x;
            }
        }
    }
}

// d = z + beta d.
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_direction(int nodes, const void* z, void* d, const ViscState* state)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nodes || visc_stopped(state))
        return;
    const T2 c = static_cast<const T2*>(z)[n];
    T2 out = c;
    if (state->count > 0)
    {
        const T beta = T(state->beta);
        const T2 p = static_cast<const T2*>(d)[n];
        out.x = c.x + beta * p.x;
        out.y = c.y + beta * p.y;
    }
    static_cast<T2*>(d)[n] = out;
}

// x += alpha d, r -= alpha q, and the next V-cycle's sweep from zero, r / (2 D), into `start`.
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_update(int nodes, void* x, void* r, const void* d, const void* q,
    const void* half, void* start, const ViscState* state)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nodes || visc_stopped(state))
        return;
    const T alpha = T(state->alpha);
    T2 a = static_cast<T2*>(x)[n], b = static_cast<T2*>(r)[n];
    const T2 dd = static_cast<const T2*>(d)[n], qq = static_cast<const T2*>(q)[n];
    a.x += alpha * dd.x;
    a.y += alpha * dd.y;
    b.x -= alpha * qq.x;
    b.y -= alpha * qq.y;
    static_cast<T2*>(x)[n] = a;
    static_cast<T2*>(r)[n] = b;
    const T2 hd = static_cast<const T2*>(half)[n];
    static_cast<T2*>(start)[n] = T2{b.x * hd.x, b.y * hd.y};
}

// solution = face velocities on valid faces, rhs = mass * solution.
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_pack(int w, int h, const void* u, const void* v, const void* coeff,
    const unsigned char* solid, void* solution, void* rhs)
{
    using T2 = typename Vec<T>::two;
    using T4 = typename Vec<T>::four;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (w + 1) * (h + 1))
        return;
    const int x = n % (w + 1), y = n / (w + 1);
    const FaceMask m = face_mask(w, h, x, y, solid);
    T2 s;
    s.x = m.u ? static_cast<const T*>(u)[(long long)y * (w + 1) + x] : T(0);
    s.y = m.v ? static_cast<const T*>(v)[(long long)y * w + x] : T(0);
    const T4 c = static_cast<const T4*>(coeff)[n];
    static_cast<T2*>(solution)[n] = s;
    static_cast<T2*>(rhs)[n] = T2{c.z * s.x, c.w * s.y};
}

// Every face velocity from the solution (walls and closed faces receive zero).
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_unpack(int w, int h, const void* solution, void* u, void* v)
{
    using T2 = typename Vec<T>::two;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (w + 1) * (h + 1))
        return;
    const int x = n % (w + 1), y = n / (w + 1);
    const T2 s = static_cast<const T2*>(solution)[n];
    if (y < h)
        static_cast<T*>(u)[(long long)y * (w + 1) + x] = s.x;
    if (x < w)
        static_cast<T*>(v)[(long long)y * w + x] = s.y;
}

// Restart from the true residual after the recurrence claimed convergence too early.
template <typename T>
__global__ void __launch_bounds__(kViscThreads) k_visc_refresh(int nodes, const void* truth, void* r, const void* half,
    void* start, ViscState* state)
{
    allow_dependents();
    dependency_wait();
    using T2 = typename Vec<T>::two;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < nodes)
    {
        const T2 b = static_cast<const T2*>(truth)[n], hd = static_cast<const T2*>(half)[n];
        static_cast<T2*>(r)[n] = b;
        static_cast<T2*>(start)[n] = T2{b.x * hd.x, b.y * hd.y};
    }
    if (n == 0)
    {
        state->rz = state->alpha = state->beta = 0.0;
        state->count = 0;
        state->stopped = 0;
        state->rnorm = state->truth;
    }
}

} // namespace fc
