// Block-scale Darcy pressure solve of the convergence accelerator.
//
// Given a mobility M per block of a periodic block grid (nz x ny x nx
// blocks of edge h voxels) and a body force g along +x, find the zero-mean
// pressure phi (over rho0) with a conserved block flux
//     F_f = M_f (g [f is an x face] - (phi_nb - phi) / h)
// across every block face, M_f the geometric mean of the two blocks'
// mobilities:   sum_f M_f (phi_nb - phi) / h^2 = g (Mx_{i+1/2} - Mx_{i-1/2}) / h.
//
// Conjugate gradients in FP64 preconditioned by one symmetric multigrid
// V-cycle in FP32: damped Jacobi (2 + 2 sweeps), trilinear prolongation,
// its adjoint / 8 as restriction, coarse face mobilities = mean of the four
// fine faces of each coarse interface, and a single-CTA Jacobi solve on the
// coarsest grid.  The solve is bound by launches: most grids are small, and a
// 96^3 solve of ten iterations took 485 launches with gaps as long as the
// kernels (3.2 ms, 2.2 ms of it kernels).  So every kernel is launched with
// programmatic dependent launch, the two coarsest levels run in one block from
// shared memory, a vector update and the dot product that follows it share a
// launch, and dot products finish in their last block (fixed order, so results
// do not vary).  The only host synchronisation per iteration is the residual
// norm.  96^3, 10 iterations: 3,500 -> 2,183 us; 48 x 80 x 96 and smaller grids
// 1.2 to 2.3 times faster.  The arithmetic of every cell is that of the separate
// kernels: same iterations, same pressure.
#include "../../include/lbflow.h"
#include "internal.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <utility>
#include <vector>

namespace {

constexpr int kT = 256;
constexpr int kCoarseSweeps = 120;   // Jacobi sweeps on the coarsest (<= 1024-cell) grid

struct Dims {
    int nz, ny, nx;
    __host__ __device__ size_t n() const { return (size_t)nz * ny * nx; }
};

__device__ __forceinline__ int wrapi(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

__device__ __forceinline__ void coords(const Dims& d, size_t i, int& z, int& y, int& x)
{
    x = (int)(i % d.nx);
    const size_t t = i / d.nx;
    y = (int)(t % d.ny);
    z = (int)(t / d.ny);
}

__device__ __forceinline__ size_t idx(const Dims& d, int z, int y, int x)
{
    return ((size_t)z * d.ny + y) * d.nx + x;
}

// First statement of every kernel: let the next one be scheduled, and wait for
// the previous ones' results, which are read by plain loads (see pdl_wait).
__device__ __forceinline__ void pdl_begin()
{
    lbf::pdl_trigger();
    lbf::pdl_wait();
}

// Face mobilities on the + faces (geometric mean) and the right-hand side.
__global__ void setup_fine(Dims d, const double* __restrict__ mob, double g, double h, float* __restrict__ mx,
                           float* __restrict__ my, float* __restrict__ mz, double* __restrict__ rhs)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= d.n()) return;
    int z, y, x;
    coords(d, i, z, y, x);
    const double m = fmax(mob[i], 1e-300);
    const double fx = sqrt(m * fmax(mob[idx(d, z, y, wrapi(x + 1, d.nx))], 1e-300));
    const double fxm = sqrt(fmax(mob[idx(d, z, y, wrapi(x - 1, d.nx))], 1e-300) * m);
    mx[i] = (float)fx;
    my[i] = (float)sqrt(m * fmax(mob[idx(d, z, wrapi(y + 1, d.ny), x)], 1e-300));
    mz[i] = (float)sqrt(m * fmax(mob[idx(d, wrapi(z + 1, d.nz), y, x)], 1e-300));
    rhs[i] = g * (fx - fxm) / h;
}

// sum_faces M_f (x_nb - x_i), and the diagonal -sum_faces M_f.
template <class T>
__device__ __forceinline__ T stencil(const Dims& d, const T* x, const float* mx,
                                     const float* my, const float* mz, size_t i, int z,
                                     int y, int xx, T& diag)
{
    const size_t xm = idx(d, z, y, wrapi(xx - 1, d.nx)), xp = idx(d, z, y, wrapi(xx + 1, d.nx));
    const size_t ym = idx(d, z, wrapi(y - 1, d.ny), xx), yp = idx(d, z, wrapi(y + 1, d.ny), xx);
    const size_t zm = idx(d, wrapi(z - 1, d.nz), y, xx), zp = idx(d, wrapi(z + 1, d.nz), y, xx);
    const T c = x[i];
    const T a = (T)mx[i], b = (T)mx[xm], e = (T)my[i], f = (T)my[ym], gg = (T)mz[i], k = (T)mz[zm];
    diag = -(a + b + e + f + gg + k);
    return a * (x[xp] - c) - b * (c - x[xm]) + e * (x[yp] - c) - f * (c - x[ym]) + gg * (x[zp] - c) -
           k * (c - x[zm]);
}

// The diagonal alone, as stencil() forms it.
__device__ __forceinline__ float diagonal(const Dims& d, const float* mx, const float* my,
                                          const float* mz, size_t i, int z, int y, int xx)
{
    const float a = mx[i], b = mx[idx(d, z, y, wrapi(xx - 1, d.nx))], e = my[i],
                f = my[idx(d, z, wrapi(y - 1, d.ny), xx)], gg = mz[i], k = mz[idx(d, wrapi(z - 1, d.nz), y, xx)];
    return -(a + b + e + f + gg + k);
}

// One damped Jacobi sweep: xo = xi + omega (r - A xi) / diag   (FP32)
__global__ void jacobi(Dims d, float h2inv, float omega, const float* xi, const float* r,
                       const float* mx, const float* my, const float* mz,
                       float* __restrict__ xo)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= d.n()) return;
    int z, y, xx;
    coords(d, i, z, y, xx);
    float dg;
    const float ax = stencil<float>(d, xi, mx, my, mz, i, z, y, xx, dg) * h2inv;
    xo[i] = dg != 0.f ? xi[i] + omega * (r[i] - ax) / (dg * h2inv) : xi[i];
}

// The first sweep, from x = 0.
__global__ void jacobi_first(Dims d, float h2inv, float omega, const float* r,
                             const float* mx, const float* my, const float* mz,
                             float* __restrict__ xo)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= d.n()) return;
    int z, y, xx;
    coords(d, i, z, y, xx);
    const float dg = diagonal(d, mx, my, mz, i, z, y, xx);
    xo[i] = dg != 0.f ? omega * r[i] / (dg * h2inv) : 0.f;
}

// res = r - A x  (FP32)
__global__ void residual(Dims d, float h2inv, const float* x, const float* r,
                         const float* mx, const float* my, const float* mz,
                         float* __restrict__ res)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= d.n()) return;
    int z, y, xx;
    coords(d, i, z, y, xx);
    float dg;
    res[i] = r[i] - stencil<float>(d, x, mx, my, mz, i, z, y, xx, dg) * h2inv;
}

// Coarse face mobilities: mean of the four fine faces on each coarse interface.
__global__ void coarsen_faces(Dims c, Dims f, const float* fmx, const float* fmy,
                              const float* fmz, float* __restrict__ cmx, float* __restrict__ cmy,
                              float* __restrict__ cmz)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= c.n()) return;
    int z, y, x;
    coords(c, i, z, y, x);
    const int Z = 2 * z, Y = 2 * y, X = 2 * x;
    float sx = 0.f, sy = 0.f, sz = 0.f;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b) {
            sx += fmx[idx(f, Z + a, Y + b, X + 1)];
            sy += fmy[idx(f, Z + a, Y + 1, X + b)];
            sz += fmz[idx(f, Z + 1, Y + a, X + b)];
        }
    cmx[i] = 0.25f * sx;
    cmy[i] = 0.25f * sy;
    cmz[i] = 0.25f * sz;
}

// Restriction: adjoint of the trilinear prolongation / 8; weights
// 1/8, 3/8, 3/8, 1/8 over fine cells 2i-1 .. 2i+2 on each axis.
__device__ __forceinline__ float restricted(const Dims& c, const Dims& f, const float* rf, size_t i)
{
    int z, y, x;
    coords(c, i, z, y, x);
    const float w[4] = {0.125f, 0.375f, 0.375f, 0.125f};
    float s = 0.f;
    for (int a = 0; a < 4; ++a) {
        const int Z = wrapi(2 * z - 1 + a, f.nz);
        for (int b = 0; b < 4; ++b) {
            const int Y = wrapi(2 * y - 1 + b, f.ny);
            for (int e = 0; e < 4; ++e) {
                const int X = wrapi(2 * x - 1 + e, f.nx);
                s += w[a] * w[b] * w[e] * rf[idx(f, Z, Y, X)];
            }
        }
    }
    return s;
}
__global__ void restrict3(Dims c, Dims f, const float* rf, float* __restrict__ rc)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < c.n()) rc[i] = restricted(c, f, rf, i);
}

// Trilinear prolongation of ec at fine cell i, and xf += it.
__device__ __forceinline__ float prolonged(const Dims& f, const Dims& c, const float* ec, size_t i)
{
    int z, y, x;
    coords(f, i, z, y, x);
    const int cz0 = z >> 1, cy0 = y >> 1, cx0 = x >> 1;
    const int cz1 = wrapi(cz0 + ((z & 1) ? 1 : -1), c.nz);
    const int cy1 = wrapi(cy0 + ((y & 1) ? 1 : -1), c.ny);
    const int cx1 = wrapi(cx0 + ((x & 1) ? 1 : -1), c.nx);
    const int cz[2] = {cz0, cz1}, cy[2] = {cy0, cy1}, cx[2] = {cx0, cx1};
    const float w[2] = {0.75f, 0.25f};
    float s = 0.f;
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b)
            for (int e = 0; e < 2; ++e) s += w[a] * w[b] * w[e] * ec[idx(c, cz[a], cy[b], cx[e])];
    return s;
}
__global__ void prolong_add(Dims f, Dims c, const float* ec, float* __restrict__ xf)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < f.n()) xf[i] += prolonged(f, c, ec, i);
}

// Zero-mean damped Jacobi sweeps on the coarsest grid (n <= 1024 cells, one
// per thread) by the block's first warps; r: this thread's right-hand side.
// xs: 2 * 1024 floats of shared memory, red: 33.  Returns the thread's
// solution.  Faces and neighbour indices stay in registers and the two halves
// of xs alternate, one barrier a sweep, of the warps that hold cells only: 120
// sweeps on 6^3 cells took 36 us with 1,024 threads, two barriers and the
// faces read from memory in every sweep.
__device__ float coarse_sweeps(const Dims& d, float h2inv, int sweeps, float r, const float* mx,
                               const float* my, const float* mz, float* xs, float* red)
{
    const int n = (int)d.n(), t = threadIdx.x;
    const int nwarps = (n + 31) / 32;
    auto barrier = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(nwarps * 32) : "memory"); };
    auto mean = [&](float v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        barrier();
        if ((t & 31) == 0) red[t >> 5] = v;
        barrier();
        if (t == 0) {
            float s = 0.f;
            for (int w = 0; w < nwarps; ++w) s += red[w];
            red[32] = s / (float)n;
        }
        barrier();
        return red[32];
    };
    if (t >= nwarps * 32) return 0.f;
    const bool in = t < n;
    const float rs = r - mean(in ? r : 0.f);
    float a = 0.f, b = 0.f, e = 0.f, f = 0.f, gg = 0.f, k = 0.f, x = 0.f;
    int xm = 0, xp = 0, ym = 0, yp = 0, zm = 0, zp = 0;
    if (in) {
        int z, y, xx;
        coords(d, (size_t)t, z, y, xx);
        xm = (int)idx(d, z, y, wrapi(xx - 1, d.nx)); xp = (int)idx(d, z, y, wrapi(xx + 1, d.nx));
        ym = (int)idx(d, z, wrapi(y - 1, d.ny), xx); yp = (int)idx(d, z, wrapi(y + 1, d.ny), xx);
        zm = (int)idx(d, wrapi(z - 1, d.nz), y, xx); zp = (int)idx(d, wrapi(z + 1, d.nz), y, xx);
        a = mx[t]; b = mx[xm]; e = my[t]; f = my[ym]; gg = mz[t]; k = mz[zm];
        xs[t] = 0.f;
    }
    const float dg = -(a + b + e + f + gg + k);
    barrier();
    for (int s = 0; s < sweeps; ++s) {
        const float* cur = xs + (s & 1) * 1024;
        if (in) {
            const float c = x;
            const float ax = (a * (cur[xp] - c) - b * (c - cur[xm]) + e * (cur[yp] - c) - f * (c - cur[ym]) +
                              gg * (cur[zp] - c) - k * (c - cur[zm])) * h2inv;
            x = dg != 0.f ? c + 0.8f * (rs - ax) / (dg * h2inv) : c;
            xs[((s + 1) & 1) * 1024 + t] = x;
        }
        barrier();
    }
    return x - mean(in ? x : 0.f);
}

__global__ void __launch_bounds__(1024) coarse_solve(Dims d, float h2inv, int sweeps, const float* r,
                                                     const float* mx, const float* my,
                                                     const float* mz, float* __restrict__ x)
{
    pdl_begin();
    __shared__ float xs[2048], red[33];
    const int t = threadIdx.x, n = (int)d.n();
    const float v = coarse_sweeps(d, h2inv, sweeps, t < n ? r[t] : 0.f, mx, my, mz, xs, red);
    if (t < n) x[t] = v;
}

// The V-cycle of the two coarsest levels in one block, the finer one of at
// most kBottomCells cells: the sweeps and transfers of the kernels above on
// shared-memory arrays.  As launches these were 9 of 46 per iteration.
constexpr int kBottomCells = 4096;
constexpr size_t kBottomShared = (3 * kBottomCells + 1024) * sizeof(float);

__global__ void __launch_bounds__(1024)
bottom_cycle(Dims d, float h2inv, float omega, const float* r, const float* mx,
             const float* my, const float* mz, float* __restrict__ x, Dims c, float ch2inv,
             int sweeps, const float* cmx, const float* cmy, const float* cmz)
{
    pdl_begin();
    extern __shared__ float sm[];
    __shared__ float xs[2048], red[33];
    float *A = sm, *B = sm + kBottomCells, *R = sm + 2 * kBottomCells, *C = sm + 3 * kBottomCells;
    const int n = (int)d.n(), t = threadIdx.x;
    auto sweep = [&](const float* xi, float* xo) {
        for (int i = t; i < n; i += 1024) {
            int z, y, xx;
            coords(d, (size_t)i, z, y, xx);
            float dg;
            const float ax = stencil<float>(d, xi, mx, my, mz, (size_t)i, z, y, xx, dg) * h2inv;
            xo[i] = dg != 0.f ? xi[i] + omega * (R[i] - ax) / (dg * h2inv) : xi[i];
        }
        __syncthreads();
    };
    for (int i = t; i < n; i += 1024) {
        int z, y, xx;
        coords(d, (size_t)i, z, y, xx);
        const float dg = diagonal(d, mx, my, mz, (size_t)i, z, y, xx);
        R[i] = r[i];
        A[i] = dg != 0.f ? omega * R[i] / (dg * h2inv) : 0.f;
    }
    __syncthreads();
    sweep(A, B);
    for (int i = t; i < n; i += 1024) {
        int z, y, xx;
        coords(d, (size_t)i, z, y, xx);
        float dg;
        A[i] = R[i] - stencil<float>(d, B, mx, my, mz, (size_t)i, z, y, xx, dg) * h2inv;
    }
    __syncthreads();
    const int cn = (int)c.n();
    const float v = coarse_sweeps(c, ch2inv, sweeps, t < cn ? restricted(c, d, A, (size_t)t) : 0.f, cmx, cmy, cmz, xs, red);
    if (t < cn) C[t] = v;
    __syncthreads();
    for (int i = t; i < n; i += 1024) B[i] += prolonged(d, c, C, (size_t)i);
    __syncthreads();
    sweep(B, A);
    sweep(A, B);
    for (int i = t; i < n; i += 1024) x[i] = B[i];
}

// p = the V-cycle's result (the first search direction).
__global__ void to_f64(size_t n, const float* a, double* __restrict__ b)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) b[i] = (double)a[i];
}
// p = z + (num / den) p
__global__ void xpby_ratio(size_t n, const float* z, const double* num,
                           const double* den, double* __restrict__ p)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) p[i] = (double)z[i] + (num[0] / den[0]) * p[i];
}

// Deterministic reductions in one launch: per-block sums of v(i) over a
// grid-stride range, then the last block to finish adds them in a fixed tree
// order (part: per-block sums; done: blocks finished, left at 0).
template <class V>
__device__ __forceinline__ void reduce_sum(size_t n, V&& value, double* __restrict__ part, uint32_t* __restrict__ done,
                                           double* __restrict__ out)
{
    __shared__ double s[kT];
    __shared__ bool last;
    double v = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        v += value(i);
    auto tree = [&](double a) {
        s[threadIdx.x] = a;
        __syncthreads();
        for (int o = kT / 2; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
            __syncthreads();
        }
    };
    tree(v);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s[0];
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double a = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kT) a += __ldcg(&part[i]);
    tree(a);
    if (threadIdx.x == 0) {
        out[0] = s[0];
        *done = 0;
    }
}

// sum a (b null), or a . b with b the FP32 vector's values.
__global__ void __launch_bounds__(kT) dot(size_t n, const double* a, const float* b,
                                          double* __restrict__ part, uint32_t* __restrict__ done,
                                          double* __restrict__ out)
{
    pdl_begin();
    reduce_sum(n, [&](size_t i) { return b ? a[i] * (double)b[i] : a[i]; }, part, done, out);
}

// r = rhs - mean (phi = 0), its FP32 copy and r . r
__global__ void __launch_bounds__(kT) start_dot(size_t n, const double* sum,
                                                const double* rhs, double* __restrict__ r,
                                                float* __restrict__ r32, double* __restrict__ part,
                                                uint32_t* __restrict__ done, double* __restrict__ rr)
{
    pdl_begin();
    const double mean = sum[0] / (double)n;
    reduce_sum(n, [&](size_t i) {
        const double v = rhs[i] - mean;
        r[i] = v;
        r32[i] = (float)v;
        return v * v;
    }, part, done, rr);
}

// out = A p  (FP64, the CG operator) and p . out
__global__ void __launch_bounds__(kT) apply_dot(Dims d, double h2inv, const double* p,
                                                const float* mx, const float* my,
                                                const float* mz, double* __restrict__ out,
                                                double* __restrict__ part, uint32_t* __restrict__ done,
                                                double* __restrict__ pap)
{
    pdl_begin();
    reduce_sum(d.n(), [&](size_t i) {
        int z, y, xx;
        coords(d, i, z, y, xx);
        double dg;
        const double v = stencil<double>(d, p, mx, my, mz, i, z, y, xx, dg) * h2inv;
        out[i] = v;
        return p[i] * v;
    }, part, done, pap);
}

// phi += (rz / pap) p, r -= (rz / pap) Ap, r's FP32 copy and r . r
__global__ void __launch_bounds__(kT) update_dot(size_t n, const double* rz,
                                                 const double* pap, const double* p,
                                                 const double* Ap, double* __restrict__ phi,
                                                 double* __restrict__ r, float* __restrict__ r32,
                                                 double* __restrict__ part, uint32_t* __restrict__ done,
                                                 double* __restrict__ rr)
{
    pdl_begin();
    const double alpha = rz[0] / pap[0];
    reduce_sum(n, [&](size_t i) {
        phi[i] += alpha * p[i];
        const double v = r[i] + -alpha * Ap[i];
        r[i] = v;
        r32[i] = (float)v;
        return v * v;
    }, part, done, rr);
}

__global__ void sub_mean(size_t n, const double* sum, double* __restrict__ a)
{
    pdl_begin();
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) a[i] -= sum[0] / (double)n;
}

unsigned nblk(size_t n) { return (unsigned)((n + kT - 1) / kT); }

struct Level {
    Dims d;
    float h2inv;
    float *mx, *my, *mz, *x, *r, *t;
};

struct Solver {
    cudaStream_t s = nullptr;
    std::vector<Level> L;
    double* part = nullptr;
    uint32_t* done = nullptr;     // blocks finished in the running reduction
    unsigned nb_dot = 0;
    cudaError_t err = cudaSuccess;
    // One device allocation carved into 256-byte-aligned arrays: a first
    // pass (base == nullptr) only adds up the size.
    char* base = nullptr;
    size_t used = 0;

    template <class T> T* alloc(size_t n)
    {
        T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
        used += (n * sizeof(T) + 255) / 256 * 256;
        return p;
    }
    ~Solver() { if (base) cudaFreeAsync(base, s); }

    void sweep(Level& v)
    {
        lbf::launch_pdl(jacobi, nblk(v.d.n()), kT, s, v.d, v.h2inv, 0.7f, v.x, v.r, v.mx, v.my, v.mz, v.t);
        std::swap(v.x, v.t);
    }

    // L[l].x = V-cycle applied to L[l].r.
    void vcycle(int l)
    {
        Level& v = L[l];
        if (l + 1 == (int)L.size()) {
            lbf::launch_pdl(coarse_solve, 1, 1024, s, v.d, v.h2inv, kCoarseSweeps, v.r, v.mx, v.my, v.mz, v.x);
            return;
        }
        Level& c = L[l + 1];
        if (l + 2 == (int)L.size() && v.d.n() <= (size_t)kBottomCells) {
            lbf::launch_pdl_shared(bottom_cycle, 1, 1024, kBottomShared, s, v.d, v.h2inv, 0.7f, v.r, v.mx, v.my, v.mz,
                                   v.x, c.d, c.h2inv, kCoarseSweeps, c.mx, c.my, c.mz);
            return;
        }
        lbf::launch_pdl(jacobi_first, nblk(v.d.n()), kT, s, v.d, v.h2inv, 0.7f, v.r, v.mx, v.my, v.mz, v.x);
        sweep(v);
        lbf::launch_pdl(residual, nblk(v.d.n()), kT, s, v.d, v.h2inv, v.x, v.r, v.mx, v.my, v.mz, v.t);
        lbf::launch_pdl(restrict3, nblk(c.d.n()), kT, s, c.d, v.d, v.t, c.r);
        vcycle(l + 1);
        lbf::launch_pdl(prolong_add, nblk(v.d.n()), kT, s, v.d, c.d, c.x, v.x);
        sweep(v);
        sweep(v);
    }

    void sum(size_t n, const double* a, const float* b, double* out)
    {
        lbf::launch_pdl(dot, nb_dot, kT, s, n, a, b, part, done, out);
    }
};

int fail(const std::string& m, int code = LBF_EINVAL)
{
    lbf::set_global_error(m);
    return code;
}

}  // namespace

extern "C" int lbf_darcy_pressure(const double* mob, uint32_t nz, uint32_t ny, uint32_t nx, double h, double g,
                                  double rtol, uint32_t max_iter, double* phi, uint32_t* iterations, void* stream)
{
    if (!mob || !phi || !nz || !ny || !nx || !(h > 0)) return fail("lbf_darcy_pressure: bad arguments");
    const Dims d0{(int)nz, (int)ny, (int)nx};
    const size_t n = d0.n();
    if (n > ((size_t)1 << 30)) return fail("lbf_darcy_pressure: grid too large");
    // Level hierarchy: halve while every extent is even and the grid has > 512 cells.
    std::vector<Dims> dims{d0};
    while (dims.back().n() > 512 && !((dims.back().nz | dims.back().ny | dims.back().nx) & 1))
        dims.push_back(Dims{dims.back().nz / 2, dims.back().ny / 2, dims.back().nx / 2});
    if (dims.back().n() > 1024)
        return fail("lbf_darcy_pressure: grid extents must halve down to at most 1024 cells");
    cudaPointerAttributes pa{};
    if (cudaPointerGetAttributes(&pa, mob) != cudaSuccess || pa.type != cudaMemoryTypeDevice ||
        cudaPointerGetAttributes(&pa, phi) != cudaSuccess || pa.type != cudaMemoryTypeDevice) {
        cudaGetLastError();
        return fail("lbf_darcy_pressure: mob and phi must be device memory");
    }
    Solver S;
    S.s = static_cast<cudaStream_t>(stream);
    S.nb_dot = (unsigned)std::min<size_t>(nblk(n), 1184);
    double *rhs = nullptr, *r = nullptr, *p = nullptr, *Ap = nullptr, *sc = nullptr;
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
            // The workspace comes from the library's device pool on the
            // solve's stream: a correction inside a timed run reuses memory
            // reserved by earlier solves instead of calling the driver.
            void* mem = nullptr;
            int dev = 0;
            cudaMemPool_t pool = nullptr;
            S.err = cudaGetDevice(&dev);
            if (S.err == cudaSuccess) S.err = lbf::device_pool(dev, &pool);
            if (S.err == cudaSuccess) S.err = cudaMallocFromPoolAsync(&mem, S.used, pool, S.s);
            if (S.err != cudaSuccess)
                return fail(std::string("lbf_darcy_pressure: ") + cudaGetErrorString(S.err), LBF_ENOMEM);
            S.base = static_cast<char*>(mem);
            S.used = 0;
            S.L.clear();
        }
        float hh = (float)h;
        for (const Dims& d : dims) {
            Level v{};
            v.d = d;
            v.h2inv = 1.0f / (hh * hh);
            const size_t m = d.n();
            v.mx = S.alloc<float>(m); v.my = S.alloc<float>(m); v.mz = S.alloc<float>(m);
            v.x = S.alloc<float>(m); v.r = S.alloc<float>(m); v.t = S.alloc<float>(m);
            S.L.push_back(v);
            hh *= 2.f;
        }
        rhs = S.alloc<double>(n);
        r = S.alloc<double>(n);
        p = S.alloc<double>(n);
        Ap = S.alloc<double>(n);
        sc = S.alloc<double>(8);          // scalars: rz, pAp, rz_new, rr, sum
        S.part = S.alloc<double>(S.nb_dot);
        S.done = S.alloc<uint32_t>(1);
    }
    cudaStream_t s = S.s;
    const double h2inv = 1.0 / (h * h);
    cudaError_t e = cudaFuncSetAttribute(bottom_cycle, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBottomShared);
    if (e != cudaSuccess) return fail(std::string("lbf_darcy_pressure: ") + cudaGetErrorString(e), LBF_ECUDA);
    cudaMemsetAsync(S.done, 0, sizeof(uint32_t), s);
    lbf::launch_pdl(setup_fine, nblk(n), kT, s, d0, mob, g, h, S.L[0].mx, S.L[0].my, S.L[0].mz, rhs);
    for (size_t l = 1; l < S.L.size(); ++l)
        lbf::launch_pdl(coarsen_faces, nblk(S.L[l].d.n()), kT, s, S.L[l].d, S.L[l - 1].d, S.L[l - 1].mx, S.L[l - 1].my,
                        S.L[l - 1].mz, S.L[l].mx, S.L[l].my, S.L[l].mz);
    // phi = 0, once mob has been read (the caller may pass one array as both);
    // zero-mean right-hand side; r = rhs.
    cudaMemsetAsync(phi, 0, n * sizeof(double), s);
    S.sum(n, rhs, nullptr, sc + 4);
    double hr = 0.0;
    lbf::launch_pdl(start_dot, S.nb_dot, kT, s, n, sc + 4, rhs, r, S.L[0].r, S.part, S.done, sc + 3);
    cudaMemcpyAsync(&hr, sc + 3, sizeof(double), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail(std::string("lbf_darcy_pressure: ") + cudaGetErrorString(e), LBF_ECUDA);
    const double nrm0 = std::sqrt(hr);
    uint32_t it = 0;
    if (nrm0 > 0) {
        // z is the V-cycle's FP32 result, L[0].x, read in FP64.
        double *rz = sc + 0, *rz_new = sc + 2;
        S.vcycle(0);
        lbf::launch_pdl(to_f64, nblk(n), kT, s, n, S.L[0].x, p);
        S.sum(n, r, S.L[0].x, rz);
        while (it < max_iter) {
            lbf::launch_pdl(apply_dot, S.nb_dot, kT, s, d0, h2inv, p, S.L[0].mx, S.L[0].my, S.L[0].mz, Ap, S.part, S.done,
                            sc + 1);
            lbf::launch_pdl(update_dot, S.nb_dot, kT, s, n, rz, sc + 1, p, Ap, phi, r, S.L[0].r, S.part, S.done, sc + 3);
            ++it;
            cudaMemcpyAsync(&hr, sc + 3, sizeof(double), cudaMemcpyDeviceToHost, s);
            e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return fail(std::string("lbf_darcy_pressure: ") + cudaGetErrorString(e), LBF_ECUDA);
            if (!(std::sqrt(hr) > rtol * nrm0)) break;
            S.vcycle(0);
            S.sum(n, r, S.L[0].x, rz_new);
            lbf::launch_pdl(xpby_ratio, nblk(n), kT, s, n, S.L[0].x, rz_new, rz, p);
            std::swap(rz, rz_new);
        }
    }
    // Zero mean.
    S.sum(n, phi, nullptr, sc + 4);
    lbf::launch_pdl(sub_mean, nblk(n), kT, s, n, sc + 4, phi);
    e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return fail(std::string("lbf_darcy_pressure: ") + cudaGetErrorString(e), LBF_ECUDA);
    if (iterations) *iterations = it;
    return LBF_OK;
}
