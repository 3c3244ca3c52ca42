// vb_gravity.cu -- self-gravity on uniform grids (src/gravity.jl): the
// Poisson solve nabla^2 phi = 4 pi G rho by matrix-free conjugate gradients on
// the device, and the field g = -grad phi that the stage kernels add as a
// source (gravity_source in vb_common.cuh) while the grid has gravity enabled.
//
// Compiled with -fmad=false: the operator row, the field and the CG vector
// updates round every product and sum separately, like the reference's Julia
// loops.  The operator row is summed in the reference's CSR order
// (_assemble_poisson_struct, src/gravity.jl:514-545), so A x is bit-identical
// to the reference's _lap_csr_cpu! (325-334); the passes of periodic cubes sum the
// same differences axis by axis.  The CG inner products are
// deterministic block-tree sums (fixed partial count and order) rather than
// the reference's serial sums, so a solve matches the reference's to the
// solver tolerance, not bit for bit.
//
// Periodic cubes (n^3, n <= 1024) have their own passes, below, plain or
// preconditioned.  On other grids every pass streams the CG vectors from HBM
// over a fixed grid of GP blocks (the stencil's neighbours come from L1/L2); the
// stencil passes walk rows of x so that a cell's coordinates cost no division.
// One CG iteration is then five launches (matvec + p.Ap partials, alpha, vector
// update + r.r partials, beta, direction update); groups of iterations replay as
// one CUDA graph, each launch returning at once after convergence, and the host
// reads the stop flag between groups.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "vb_internal.h"
#include "vb_physics.cuh"

namespace vb {
namespace {

constexpr int GB = 256;  // threads per block
constexpr int GP = 592;  // blocks (= partial sums) per reduction pass: 4 per SM, fixed
constexpr int GP_SM = 4;  // the GP blocks fit in one wave only at <= 64 registers a thread
constexpr int GRAPH_ITERS = 8;
// Iterations of a cube's loop between looks by the host: a solve of no more (the
// default limit is 500) needs none, a longer one cannot hold the device for the
// whole of a large maxiter (a residual of NaN never meets the tolerance).
constexpr long long CUBE_RUN = 512;

struct GravCtrl {
    double rhobar, rsold, pAp, alpha, beta, bnorm, relres, mu, mgmu;
    long long iters, maxiter;
    long long pause;  // iterations after which a cube's loop returns to the host
    int done;
    unsigned int ticket, ticket2;  // blocks past a grid_sum; zero between launches
    double tol;
};

// phi's boundary codes and the operator's per-axis coefficient area / distance
struct GravP {
    int per_lo[3], per_hi[3];  // 1: periodic side
    double coef[3];
    double G;
    int project_mean;
};

// neighbour of `lin` (coordinate c on axis d) across its lo or hi face under
// phi's codes; -1 at a wall (homogeneous Neumann)
__device__ __forceinline__ int64_t gnb(const Geom &g, const GravP &P, int64_t lin, int64_t c,
                                       int d, bool hi)
{
    const int64_t n = g.n[d];
    const int64_t j = hi ? c + 1 : c - 1;
    if (j >= 0 && j < n) return hi ? lin + g.stride[d] : lin - g.stride[d];
    if (hi ? P.per_hi[d] : P.per_lo[d]) return lin + ((j < 0 ? n - 1 : 0) - c) * g.stride[d];
    return -1;
}

// Visit this block's cells: rows of x (coordinates derived once per row), rows
// strided over the GP blocks and x over the block's threads; a row shorter
// than half the block is shared with the next rows (thread t takes x = t % n0
// of row t / n0 of each group of GB / n0 rows), so no thread idles on a short
// row.  1D grids stride cells directly.  A fixed order per thread, so the
// partial sums are deterministic.
template <int ND, typename F>
__device__ __forceinline__ void for_cells(const Geom &g, F &&f)
{
    if constexpr (ND == 1) {
        for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < g.ncell; i += (int64_t)GP * GB) {
            const int64_t cc[3] = {i, 0, 0};
            f(i, cc);
        }
    } else {
        const int64_t n0 = g.n[0], nrow = g.ncell / n0;
        const int rpg = n0 >= GB / 2 ? 1 : GB / (int)n0;  // rows per group
        const int rsub = rpg == 1 ? 0 : (int)threadIdx.x / (int)n0;
        const int64_t cx0 = rpg == 1 ? threadIdx.x : (int)threadIdx.x - rsub * (int)n0;
        if (rsub >= rpg) return;
        // row = cz * n1 + cy, advanced by `step` rows without a division per row
        const int64_t n1 = g.n[1], step = (int64_t)GP * rpg, sy = step % n1, sz = step / n1;
        int64_t row = (int64_t)blockIdx.x * rpg + rsub, cy = row % n1, cz = row / n1;
        if (n0 <= GB) {
            // one cell per row and thread: two rows per pass, in the same
            // order, so that the loads of both are in flight together
            if (cx0 >= n0) return;
            for (; row + step < nrow; row += 2 * step) {
                int64_t cy2 = cy + sy, cz2 = cz + sz;
                if (cy2 >= n1) {
                    cy2 -= n1;
                    ++cz2;
                }
                const int64_t c1[3] = {cx0, cy, cz}, c2[3] = {cx0, cy2, cz2};
                f(row * n0 + cx0, c1);
                f((row + step) * n0 + cx0, c2);
                cy = cy2 + sy;
                cz = cz2 + sz;
                if (cy >= n1) {
                    cy -= n1;
                    ++cz;
                }
            }
            if (row < nrow) {
                const int64_t c1[3] = {cx0, cy, cz};
                f(row * n0 + cx0, c1);
            }
            return;
        }
        for (; row < nrow; row += step) {
            for (int64_t cx = cx0; cx < n0; cx += GB) {
                const int64_t cc[3] = {cx, cy, cz};
                f(row * n0 + cx, cc);
            }
            cy += sy;
            cz += sz;
            if (cy >= n1) {
                cy -= n1;
                ++cz;
            }
        }
    }
}

// (A x)[lin], A = -nabla^2 V: sum over the row's faces of coef * (x_c - x_nb),
// in the order the reference's CSR row lists them: lo faces emitted by a lower
// cell (z, y, x), the cell's own hi faces (x, y, z; a 1-cell periodic axis
// lists its self face twice), lo faces emitted by a periodic partner above
// (x, y, z).
template <int ND>
__device__ __forceinline__ double lap_row(const Geom &g, const GravP &P, const double *__restrict__ x,
                                          int64_t lin, const int64_t cc[3])
{
    const double xc = x[lin];
    double s = 0.0;
    bool inner = true;  // every neighbour inside the grid: the row lists the lo
#pragma unroll          // faces z, y, x, then the hi faces x, y, z
    for (int d = 0; d < ND; ++d) inner = inner && cc[d] >= 1 && cc[d] + 1 < g.n[d];
    if (inner) {
#pragma unroll
        for (int d = ND - 1; d >= 0; --d) s = s + P.coef[d] * (xc - x[lin - g.stride[d]]);
#pragma unroll
        for (int d = 0; d < ND; ++d) s = s + P.coef[d] * (xc - x[lin + g.stride[d]]);
        return s;
    }
#pragma unroll
    for (int d = ND - 1; d >= 0; --d) {
        const int64_t nb = gnb(g, P, lin, cc[d], d, false);
        if (nb >= 0 && nb < lin) s = s + P.coef[d] * (xc - x[nb]);
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int64_t nb = gnb(g, P, lin, cc[d], d, true);
        if (nb < 0) continue;
        s = s + P.coef[d] * (xc - x[nb]);
        if (nb == lin) s = s + P.coef[d] * (xc - x[nb]);
    }
#pragma unroll
    for (int d = 0; d < ND; ++d) {
        const int64_t nb = gnb(g, P, lin, cc[d], d, false);
        if (nb > lin) s = s + P.coef[d] * (xc - x[nb]);
    }
    return s;
}

// (x, y, z) of cell i of a periodic n^3 cube, x fastest: masks and shifts
// when n is a power of two, else two unsigned divisions
__device__ __forceinline__ void cube_coords(int n, int i, int c[3])
{
    const unsigned u = (unsigned)i, un = (unsigned)n;
    if ((un & (un - 1u)) == 0u) {
        const int sh = __ffs(n) - 1;
        c[0] = (int)(u & (un - 1u));
        c[1] = (int)((u >> sh) & (un - 1u));
        c[2] = (int)(u >> (2 * sh));
    } else {
        const unsigned q = u / un, r = q / un;
        c[0] = (int)(u - q * un);
        c[1] = (int)(q - r * un);
        c[2] = (int)r;
    }
}

// Deterministic sum over the block's threads (fixed tree: a shuffle tree in
// each warp, then one over the warp sums), returned to every thread.  `sh`
// holds at least NW + 1 doubles.
template <int NTH>
__device__ __forceinline__ double tree_sum(double v, double *sh)
{
    constexpr int NW = NTH / 32;
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, o);
    if (l == 0) sh[w] = v;
    __syncthreads();
    if (w == 0) {
        double r = l < NW ? sh[l] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r = r + __shfl_down_sync(0xffffffffu, r, o);
        if (l == 0) sh[NW] = r;
    }
    __syncthreads();
    const double r = sh[NW];
    __syncthreads();  // sh is free for the next sum
    return r;
}

__device__ __forceinline__ double block_sum(double v, double *sh) { return tree_sum<GB>(v, sh); }

// Sum of the GP partials part[0..GP) by one block of 1024 threads (fixed tree).
__device__ __forceinline__ double final_sum(const double *part, double *sh)
{
    const int t = threadIdx.x;
    return tree_sum<1024>(t < GP ? part[t] : 0.0, sh);
}

// partials of sum(x * V) and sum(V) (the volume-weighted mean of a field)
__global__ void __launch_bounds__(GB, GP_SM) k_meanpart(Geom g, const double *__restrict__ x, double *part)
{
    __shared__ double sh[GB];
    double s = 0.0, v = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < g.ncell; i += (int64_t)GP * GB) {
        s = s + x[i] * g.vol;
        v = v + g.vol;
    }
    s = block_sum(s, sh);
    v = block_sum(v, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s;
        part[GP + blockIdx.x] = v;
    }
}

// which = 0: rhobar; 1: mu (the potential's mean)
__global__ void __launch_bounds__(1024) k_mean_final(const double *part, GravCtrl *gc, int which)
{
    __shared__ double sh[1024];
    const double s = final_sum(part, sh);
    const double v = final_sum(part + GP, sh);
    if (threadIdx.x == 0) {
        if (which == 0) gc->rhobar = s / v;
        else gc->mu = s / v;
    }
}

// _rhs_flat_kernel!, src/gravity.jl:215-231: b = -4 pi G (rho - rhobar) V
__global__ void __launch_bounds__(GB, GP_SM) k_rhs(Geom g, GravP P, const double *__restrict__ U, double *b,
                                           const GravCtrl *gc)
{
    const double rhobar = P.project_mean ? gc->rhobar : 0.0;
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < g.ncell; i += (int64_t)GP * GB)
        b[i] = -VB_FOURPI * P.G * (U[i] - rhobar) * g.vol * 1.0;
}

// CG start, src/gravity.jl:272-279: r = b - A phi, p = r; partials of r.r and b.b
template <int ND>
__global__ void __launch_bounds__(GB, GP_SM) k_cg_init(Geom g, GravP P, const double *__restrict__ phi,
                                               const double *__restrict__ b, double *r, double *p,
                                               double *part)
{
    __shared__ double sh[GB];
    double rr = 0.0, bb = 0.0;
    for_cells<ND>(g, [&](int64_t i, const int64_t cc[3]) {
        const double ri = b[i] - lap_row<ND>(g, P, phi, i, cc);
        r[i] = ri;
        p[i] = ri;
        rr = rr + ri * ri;
        bb = bb + b[i] * b[i];
    });
    rr = block_sum(rr, sh);
    bb = block_sum(bb, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = rr;
        part[GP + blockIdx.x] = bb;
    }
}

__global__ void __launch_bounds__(1024) k_cg_init_final(const double *part, GravCtrl *gc)
{
    __shared__ double sh[1024];
    const double rr = final_sum(part, sh);
    const double bb = final_sum(part + GP, sh);
    if (threadIdx.x == 0) {
        double bnorm = sqrt(bb);
        if (bnorm == 0.0) bnorm = 1.0;
        gc->rsold = rr;
        gc->bnorm = bnorm;
        gc->relres = sqrt(rr) / bnorm;
        gc->iters = 0;
        gc->done = gc->maxiter <= 0 ? 1 : 0;
    }
}

// Ap = A p; partials of p.Ap
template <int ND>
__global__ void __launch_bounds__(GB, GP_SM) k_cg_matvec(Geom g, GravP P, const double *__restrict__ p,
                                                 double *__restrict__ Ap, double *part, const GravCtrl *gc)
{
    __shared__ double sh[GB];
    if (gc->done) return;
    double s = 0.0;
    for_cells<ND>(g, [&](int64_t i, const int64_t cc[3]) {
        const double a = lap_row<ND>(g, P, p, i, cc);
        Ap[i] = a;
        s = s + p[i] * a;
    });
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// iters = k; stop when p.Ap <= 0, else alpha = rsold / p.Ap
__global__ void __launch_bounds__(1024) k_cg_alpha(const double *part, GravCtrl *gc)
{
    __shared__ double sh[1024];
    if (gc->done) return;
    const double pAp = final_sum(part, sh);
    if (threadIdx.x == 0) {
        gc->iters += 1;
        gc->pAp = pAp;
        if (pAp <= 0.0) gc->done = 1;
        else gc->alpha = gc->rsold / pAp;
    }
}

// phi += alpha p; r -= alpha Ap; partials of r.r
__global__ void __launch_bounds__(GB, GP_SM) k_cg_update(Geom g, double *phi, const double *__restrict__ p,
                                                 double *r, const double *__restrict__ Ap,
                                                 double *part, const GravCtrl *gc)
{
    __shared__ double sh[GB];
    if (gc->done) return;
    const double alpha = gc->alpha;
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < g.ncell; i += (int64_t)GP * GB) {
        phi[i] = phi[i] + alpha * p[i];
        const double ri = r[i] - alpha * Ap[i];
        r[i] = ri;
        s = s + ri * ri;
    }
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// relres; stop at tol, else beta = rsnew / rsold; stop after maxiter
__global__ void __launch_bounds__(1024) k_cg_beta(const double *part, GravCtrl *gc)
{
    __shared__ double sh[1024];
    if (gc->done) return;
    const double rsnew = final_sum(part, sh);
    if (threadIdx.x == 0) {
        gc->relres = sqrt(rsnew) / gc->bnorm;
        if (gc->relres <= gc->tol) {
            gc->done = 1;
            return;
        }
        gc->beta = rsnew / gc->rsold;
        gc->rsold = rsnew;
        if (gc->iters >= gc->maxiter) gc->done = 1;
    }
}

// p = r + beta p
__global__ void __launch_bounds__(GB, GP_SM) k_cg_dir(Geom g, double *p, const double *__restrict__ r,
                                              const GravCtrl *gc)
{
    if (gc->done) return;
    const double beta = gc->beta;
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < g.ncell; i += (int64_t)GP * GB)
        p[i] = r[i] + beta * p[i];
}

__global__ void __launch_bounds__(GB, GP_SM) k_sub_mean(Geom g, double *phi, const GravCtrl *gc)
{
    const double mu = gc->mu;
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < g.ncell; i += (int64_t)GP * GB)
        phi[i] = phi[i] - mu;
}

// g = -grad phi, _gax (src/gravity.jl:387-394): central difference over the two
// face distances; across a wall the neighbour value is the cell's own and the
// distance half a width
template <int ND>
__global__ void __launch_bounds__(GB, GP_SM) k_accel(Geom g, GravP P, const double *__restrict__ phi,
                                             double *gacc)
{
    for_cells<ND>(g, [&](int64_t i, const int64_t cc[3]) {
        const double pc = phi[i];
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            const int64_t lo = gnb(g, P, i, cc[d], d, false), hi = gnb(g, P, i, cc[d], d, true);
            const double wlo = lo < 0 ? pc : phi[lo], whi = hi < 0 ? pc : phi[hi];
            const double fd = 0.5 * (g.w[d] + g.w[d]);  // _face_distance
            const double dlo = lo < 0 ? 0.5 * g.w[d] : fd, dhi = hi < 0 ? 0.5 * g.w[d] : fd;
            gacc[d * g.ncell + i] = -(whi - wlo) / (dlo + dhi);
        }
    });
}

template <int ND>
__global__ void __launch_bounds__(GB, GP_SM) k_lap(Geom g, GravP P, const double *__restrict__ x, double *out)
{
    for_cells<ND>(g, [&](int64_t i, const int64_t cc[3]) { out[i] = lap_row<ND>(g, P, x, i, cc); });
}

// ---------------------------------------------------------------------------
// The solver on a periodic n^3 cube: plain CG (the recurrence above) and CG
// preconditioned after the reference's ext/mg_pcg.jl (precond =
// VB_GRAV_PRECOND_MG): z = M^-1 r is one composite-smoothed two-level cycle
// (_amg_cycle!, mg_pcg.jl:152-174): two damped-Jacobi sweeps on A from z = 0,
// the residual moved to the base grid (on a uniform mesh the cells
// themselves), one periodic cell-centred V-cycle of -lap there (_mg_vcycle!,
// 123-145: damped Jacobi 2 + 2, full-weighting restriction, trilinear
// prolongation, 30 sweeps on the coarsest level), the correction de-meaned,
// scaled by 1/V and added, two more Jacobi sweeps on A.
//
// Every pass streams arrays of the fine grid, so passes are merged where one's
// values can be formed from another's inputs:
//   - the direction p = z + beta p and A p are one pass (p in two buffers);
//   - a smoother's two sweeps from zero are one pass over its right-hand side
//     (the first sweep is a multiple of it), on A and on every level;
//   - residual and restriction are one pass; the correction's (e - mean) / V
//     is formed where the first post-smoothing sweep reads it;
//   - diag(A) is one number here (every row lists the same six coefficients);
//   - each inner product is finished by the last block of the pass that forms
//     it (fixed-order sums of the block partials: the same bits every run),
//     which also sets the step's scalars.
// That is 275 B of fine-grid traffic an iteration against 456 B as separate
// passes, and about 25 launches against 90.  Levels of 16^3 and below run in
// one block, in shared memory.  The iterations run as one graph with a WHILE
// node on the stop flag, so the host reads nothing in between.
//
// A thread owns an (x, y) column of cells, two side by side where n is even, and
// marches z over a chunk with the values below and above in registers; the y
// neighbours come from L1, the x neighbours of a pair from the lanes beside it.
// What bounds the passes is the loads in flight: with one cell a thread they ran
// at 2.4-3.6 TB/s at 256^3, with pairs (and 5 blocks an SM, which the sweeps have
// to be held to) at 4.0-5.8 TB/s, 1.48 -> 1.2 ms an iteration.  Tried and slower:
// two passes chained through shared memory (half the traffic, but the barrier a
// plane leaves 2.4 TB/s of it), loads a plane further ahead, passes running
// alternately up and down through the planes.

constexpr double MG_OMEGA = 0.8;
constexpr int MG_BLOCK = 16;  // levels of at most MG_BLOCK^3 cells run in one block

struct CubeP {
    int n;
    double c[3];  // the operator's coefficients
    double w;     // MG_OMEGA / diag(A)
};

// planes of a thread's chunk: long ones re-read fewer planes, short ones keep
// the chip full (and the chain of dependent planes short) on small levels.  Odd
// cubes, one cell a thread, want longer ones before even ones do (CG, us an
// iteration with 2, 5 and 8 planes: 71^3 20.4, 16.8, 19.6; 95^3 25.8, 21.3, 21.7).
__host__ __device__ inline int cube_kz(int n)
{
    if ((n & 1) && n >= 64 && n < 96) return 5;
    return n >= 512 ? 64 : n >= 192 ? 16 : n >= 96 ? 8 : n >= 48 ? 2 : 1;
}

// Two neighbouring cells of a row: the passes below run on D2 when n is even
// (one 16-byte access for both) and on double otherwise, with the same
// operations per cell.
struct alignas(16) D2 {
    double x, y;
};
__device__ __forceinline__ D2 operator+(D2 a, D2 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ D2 operator-(D2 a, D2 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ D2 operator-(D2 a, double b) { return {a.x - b, a.y - b}; }
__device__ __forceinline__ D2 operator*(D2 a, D2 b) { return {a.x * b.x, a.y * b.y}; }
__device__ __forceinline__ D2 operator*(double a, D2 b) { return {a * b.x, a * b.y}; }
__device__ __forceinline__ double scaled(double a, double b, double c) { return a * b * c; }
__device__ __forceinline__ D2 scaled(double a, D2 b, double c) { return {a * b.x * c, a * b.y * c}; }
__device__ __forceinline__ double total(double a) { return a; }
__device__ __forceinline__ double total(D2 a) { return a.x + a.y; }

// the cells at i: load from and store to an array
template <class T>
struct At {
    int i;
    __device__ __forceinline__ T operator()(const double *p) const { return *reinterpret_cast<const T *>(p + i); }
    __device__ __forceinline__ void put(double *p, T v) const { *reinterpret_cast<T *>(p + i) = v; }
};

// what f gets of a cell's two neighbours on an axis: their sum, or (DIFF) the
// sum of the cell's differences to them.  The operator of CG takes differences:
// each is exact where v varies slowly, while 2 c - (a + b) is rounded to a part
// in 2^53 of v itself, n / 2 pi times more on the longest mode and without bound
// under a constant offset of v.
template <bool DIFF, class T>
__device__ __forceinline__ T cube_axis(T c, T a, T b)
{
    if constexpr (DIFF) return (c - a) + (c - b);
    else return a + b;
}

// f(at, v, sx, sy, sz) for this thread's cells, s* cube_axis per axis; v(at)
// forms the operand.  Blocks of 32 x 8 cells (D2: 32 x 16).
template <class T, bool DIFF = false, class V, class F>
__device__ __forceinline__ void cube_cells(int n, V &&v, F &&f)
{
    constexpr bool PAIR = sizeof(T) == 16;
    const int kz = cube_kz(n), z0 = blockIdx.z * kz, z1 = min(n, z0 + kz), nn = n * n;
    if constexpr (PAIR) {
        // x neighbours of a pair come from the lanes beside it (16 lanes a row),
        // at the ends of the segment from memory; lanes beyond the cube repeat
        // its last cells and store nothing
        const int lane = threadIdx.x & 15, xr = blockIdx.x * 32 + 2 * lane, yr = blockIdx.y * 16 + (threadIdx.x >> 4);
        const int x = min(xr, n - 2), y = min(yr, n - 1);
        const bool in = xr < n && yr < n;
        const int base = x + n * y, ym = (y > 0 ? -1 : n - 1) * n, yp = (y + 1 < n ? 1 : 1 - n) * n;
        const bool first = lane == 0, last = lane == 15 || x + 2 >= n;
        const int xe = first ? (x > 0 ? -1 : n - 1) : x + 2 < n ? 2 : 2 - n;
        D2 lo = v(At<D2>{base + (z0 > 0 ? z0 - 1 : n - 1) * nn}), c = v(At<D2>{base + z0 * nn});
        for (int z = z0; z < z1; ++z) {
            const int i = base + z * nn;
            const D2 hi = v(At<D2>{base + (z + 1 < n ? z + 1 : 0) * nn});
            // check build only: every cell read and written lies in the cube
            const bool ok = VB_DCHECK(i >= 0 && i + 1 < n * nn && i + ym >= 0 && i + ym + 1 < n * nn && i + yp >= 0 &&
                                      i + yp + 1 < n * nn && i + xe >= 0 && i + xe < n * nn);
            const D2 sy = ok ? cube_axis<DIFF>(c, v(At<D2>{i + ym}), v(At<D2>{i + yp})) : c;
            double l = __shfl_up_sync(0xffffffffu, c.y, 1, 16), r = __shfl_down_sync(0xffffffffu, c.x, 1, 16);
            if ((first || last) && ok) {
                const double e = v(At<double>{i + xe});
                if (first) l = e;
                else r = e;
                if (first && last) r = v(At<double>{i + (x + 2 < n ? 2 : 2 - n)});
            }
            if (in && ok) f(At<D2>{i}, c, cube_axis<DIFF>(c, D2{l, c.x}, D2{c.y, r}), sy, cube_axis<DIFF>(c, lo, hi));
            lo = c;
            c = hi;
        }
    } else {
        const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
        if (x >= n || y >= n) return;
        const int base = x + n * y;
        const int xm = x > 0 ? -1 : n - 1, xp = x + 1 < n ? 1 : 1 - n;
        const int ym = (y > 0 ? -1 : n - 1) * n, yp = (y + 1 < n ? 1 : 1 - n) * n;
        double lo = v(At<double>{base + (z0 > 0 ? z0 - 1 : n - 1) * nn}), c = v(At<double>{base + z0 * nn});
        for (int z = z0; z < z1; ++z) {
            const int i = base + z * nn;
            if (!VB_DCHECK(i >= 0 && i < n * nn && i + xm >= 0 && i + xp < n * nn && i + ym >= 0 && i + yp < n * nn))
                return;  // check build only
            const double hi = v(At<double>{base + (z + 1 < n ? z + 1 : 0) * nn});
            f(At<double>{i}, c, cube_axis<DIFF>(c, v(At<double>{i + xm}), v(At<double>{i + xp})),
              cube_axis<DIFF>(c, v(At<double>{i + ym}), v(At<double>{i + yp})), cube_axis<DIFF>(c, lo, hi));
            lo = c;
            c = hi;
        }
    }
}

// A v at a cell from cube_cells' sums of differences.  The reference's row sums
// the same six differences face by face (lap_row); the order differs.
template <class T>
__device__ __forceinline__ T cube_lap(const CubeP &P, T dx, T dy, T dz)
{
    return P.c[0] * dx + P.c[1] * dy + P.c[2] * dz;
}

// The grid's sum of s over its threads: true in thread 0 of the last block to
// get here, with the total of the block partials summed in block order strides.
__device__ __forceinline__ bool grid_sum(double s, double *part, unsigned int *ticket, double &total)
{
    __shared__ double sh[GB / 32 + 1];
    __shared__ bool last;
    const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
    s = block_sum(s, sh);
    if (threadIdx.x == 0) {
        part[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = s;
        __threadfence();
        last = atomicAdd(ticket, 1u) == nb - 1;
        if (last) *ticket = 0u;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    double r = 0.0;
    for (unsigned j = threadIdx.x; j < nb; j += GB) r = r + __ldcg(part + j);
    total = block_sum(r, sh);
    return threadIdx.x == 0;
}

// CG start on the cube: r = b - A phi with b = -4 pi G (rho - rhobar) V
// (k_rhs), and the scalars of k_cg_init_final
template <class T>
__global__ void __launch_bounds__(GB) k_cube_init(CubeP P, GravP Q, double vol, const double *__restrict__ rho,
                                                 const double *__restrict__ phi,
                                                 double *__restrict__ r, double *part, GravCtrl *gc)
{
    const double rhobar = Q.project_mean ? gc->rhobar : 0.0;
    double rr = 0.0, bb = 0.0;
    cube_cells<T, true>(
        P.n, [&](auto at) { return at(phi); },
        [&](auto at, T c, T dx, T dy, T dz) {
            const T b = scaled(-VB_FOURPI * Q.G, at(rho) - rhobar, vol);
            const T ri = b - cube_lap(P, dx, dy, dz);
            at.put(r, ri);
            rr = rr + total(ri * ri);
            bb = bb + total(b * b);
        });
    // two sums: the first one's total waits in gc for the second's last block
    double t;
    if (grid_sum(rr, part, &gc->ticket, t)) gc->rsold = t;
    const unsigned nb = gridDim.x * gridDim.y * gridDim.z;
    if (grid_sum(bb, part + nb, &gc->ticket2, t)) {
        double bnorm = sqrt(t);
        if (bnorm == 0.0) bnorm = 1.0;
        gc->bnorm = bnorm;
    }
}
// the scalars that need both sums
__global__ void k_cube_init_final(GravCtrl *gc)
{
    gc->relres = sqrt(gc->rsold) / gc->bnorm;
    gc->iters = 0;
    gc->done = gc->maxiter <= 0 ? 1 : 0;
    gc->pause = CUBE_RUN;
    gc->beta = 0.0;  // the first direction is z (mg_pcg.jl:188-191) or r
}

__global__ void k_cube_resume(GravCtrl *gc) { gc->pause = gc->iters + CUBE_RUN; }

// the loop's condition after an iteration
__device__ __forceinline__ unsigned cube_more(const GravCtrl *gc) { return !gc->done && gc->iters < gc->pause; }

// k_accel on the cube: the same differences and quotients
__global__ void __launch_bounds__(GB) k_cube_accel(const __grid_constant__ Geom g, int n,
                                                  const double *__restrict__ phi,
                                                  double *__restrict__ gacc)
{
    const int x = blockIdx.x * 32 + (threadIdx.x & 31), y = blockIdx.y * 8 + (threadIdx.x >> 5);
    const int kz = cube_kz(n), z0 = blockIdx.z * kz, z1 = min(n, z0 + kz);
    if (x >= n || y >= n) return;
    const int nn = n * n, base = x + n * y;
    const int xm = x > 0 ? -1 : n - 1, xp = x + 1 < n ? 1 : 1 - n;
    const int ym = (y > 0 ? -1 : n - 1) * n, yp = (y + 1 < n ? 1 : 1 - n) * n;
    double d[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double fd = 0.5 * (g.w[a] + g.w[a]);
        d[a] = fd + fd;
    }
    double lo = phi[base + (z0 > 0 ? z0 - 1 : n - 1) * nn], c = phi[base + z0 * nn];
    for (int z = z0; z < z1; ++z) {
        const int i = base + z * nn;
        const double hi = phi[base + (z + 1 < n ? z + 1 : 0) * nn];
        gacc[i] = -(phi[i + xp] - phi[i + xm]) / d[0];
        gacc[g.ncell + i] = -(phi[i + yp] - phi[i + ym]) / d[1];
        gacc[2 * g.ncell + i] = -(hi - lo) / d[2];
        lo = c;
        c = hi;
    }
}

// p = z + beta p (beta 0: z) into the other of the two direction buffers,
// Ap = A p, alpha = rsold / p.Ap; stop when p.Ap <= 0
template <class T>
__global__ void __launch_bounds__(GB) k_cube_dir(CubeP P, const double *__restrict__ z, double *pa,
                                                double *pb, double *__restrict__ Ap, double *part,
                                                GravCtrl *gc)
{
    if (gc->done) return;
    const bool odd = gc->iters & 1;
    const double *__restrict__ po = odd ? pb : pa;
    double *__restrict__ pn = odd ? pa : pb;
    const double beta = gc->beta;
    double s = 0.0;
    cube_cells<T, true>(
        P.n, [&](auto at) { return beta != 0.0 ? at(z) + beta * at(po) : at(z); },
        [&](auto at, T c, T dx, T dy, T dz) {
            const T a = cube_lap(P, dx, dy, dz);
            at.put(pn, c);
            at.put(Ap, a);
            s = s + total(c * a);
        });
    double pAp;
    if (grid_sum(s, part, &gc->ticket, pAp)) {
        gc->iters += 1;
        gc->pAp = pAp;
        if (pAp <= 0.0) gc->done = 1;
        else gc->alpha = gc->rsold / pAp;
    }
}

// phi += alpha p; r -= alpha Ap; relres, stop at tol.  CG (no preconditioner):
// also beta = r.r / rsold and the iteration limit; `more`: the loop's condition.
__global__ void __launch_bounds__(GB) k_cube_update(int n, double *__restrict__ phi, const double *pa,
                                                   const double *pb, double *__restrict__ r,
                                                   const double *__restrict__ Ap, double *part,
                                                   GravCtrl *gc, int cg, cudaGraphConditionalHandle more)
{
    if (gc->done) {
        if (cg && blockIdx.x == 0 && threadIdx.x == 0) cudaGraphSetConditional(more, 0);
        return;
    }
    const double *__restrict__ p = (gc->iters & 1) ? pb : pa;
    const double alpha = gc->alpha;
    const int64_t N = (int64_t)n * n * n;
    double s = 0.0;
#pragma unroll 4
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < N; i += (int64_t)gridDim.x * GB) {
        phi[i] = phi[i] + alpha * p[i];
        const double ri = r[i] - alpha * Ap[i];
        r[i] = ri;
        s = s + ri * ri;
    }
    double rr;
    if (grid_sum(s, part, &gc->ticket, rr)) {
        gc->relres = sqrt(rr) / gc->bnorm;
        if (gc->relres <= gc->tol) {
            gc->done = 1;
        } else if (cg) {
            gc->beta = rr / gc->rsold;
            gc->rsold = rr;
            if (gc->iters >= gc->maxiter) gc->done = 1;
        }
        if (cg) cudaGraphSetConditional(more, cube_more(gc));
    }
}

// two damped-Jacobi sweeps on A from zero: z1 = w r, z = z1 + w (r - A z1)
template <class T>
__global__ void __launch_bounds__(GB) k_cube_pre(CubeP P, const double *__restrict__ r,
                                                double *__restrict__ z, const GravCtrl *gc)
{
    if (gc->done) return;
    cube_cells<T, true>(
        P.n, [&](auto at) { return at(r); },
        [&](auto at, T c, T dx, T dy, T dz) {
            at.put(z, P.w * c + P.w * (c - P.w * cube_lap(P, dx, dy, dz)));
        });
}

// the base grid's right-hand side: b = r - A z
template <class T>
__global__ void __launch_bounds__(GB) k_cube_resid(CubeP P, const double *__restrict__ z,
                                                  const double *__restrict__ r,
                                                  double *__restrict__ b, const GravCtrl *gc)
{
    if (gc->done) return;
    cube_cells<T, true>(
        P.n, [&](auto at) { return at(z); },
        [&](auto at, T c, T dx, T dy, T dz) { at.put(b, at(r) - cube_lap(P, dx, dy, dz)); });
}

// first post-smoothing sweep on A of z + (e - mean e) / V
template <class T>
__global__ void __launch_bounds__(GB) k_cube_post1(CubeP P, const double *__restrict__ z,
                                                  const double *__restrict__ e,
                                                  const double *__restrict__ r, double iV,
                                                  double *__restrict__ z2, const GravCtrl *gc)
{
    if (gc->done) return;
    const double mu = gc->mgmu;
    cube_cells<T, true>(
        P.n, [&](auto at) { return at(z) + iV * (at(e) - mu); },
        [&](auto at, T c, T dx, T dy, T dz) {
            at.put(z2, c + P.w * (at(r) - cube_lap(P, dx, dy, dz)));
        });
}

// second one, and r.z: at the solve's start (start) rsold = r.z and beta = 0,
// then beta = r.z / rsold and the iteration limit; `more`: the loop's condition
template <class T>
__global__ void __launch_bounds__(GB) k_cube_post2(CubeP P, const double *__restrict__ z2,
                                                  const double *__restrict__ r,
                                                  double *__restrict__ z, double *part, GravCtrl *gc,
                                                  int start, cudaGraphConditionalHandle more)
{
    if (gc->done) {
        if (!start && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0)
            cudaGraphSetConditional(more, 0);
        return;
    }
    double s = 0.0;
    cube_cells<T, true>(
        P.n, [&](auto at) { return at(z2); },
        [&](auto at, T c, T dx, T dy, T dz) {
            const T ri = at(r), v = c + P.w * (ri - cube_lap(P, dx, dy, dz));
            at.put(z, v);
            s = s + total(ri * v);
        });
    double rz;
    if (grid_sum(s, part, &gc->ticket, rz)) {
        gc->beta = start ? 0.0 : rz / gc->rsold;
        gc->rsold = rz;
        if (!start) {
            if (gc->iters >= gc->maxiter) gc->done = 1;
            cudaGraphSetConditional(more, cube_more(gc));
        }
    }
}

__device__ __forceinline__ int mg_wrap(int a, int n) { return a < 0 ? n - 1 : (a >= n ? 0 : a); }

// a / 6: the reciprocal's product corrected by its residual rounds as the
// division does unless a step of it leaves the normal numbers
__device__ __forceinline__ double sixth(double a)
{
    const unsigned h = (unsigned)__double2hiint(a) & 0x7fffffffu;
    return h - 0x06000000u < 0x79000000u ? quot64(a, 6.0, 1.0 / 6.0) : a / 6.0;
}

// _mgk_jacobi! (mg_pcg.jl:21-31): phi = (1 - w) phiold + w (sum_nb + h^2 b) / 6
__device__ __forceinline__ double mg_jacobi(double c, double nb, double h2b)
{
    return (1.0 - MG_OMEGA) * c + sixth(MG_OMEGA * (nb + h2b));
}
__device__ __forceinline__ D2 mg_jacobi(D2 c, D2 nb, D2 h2b)
{
    return {mg_jacobi(c.x, nb.x, h2b.x), mg_jacobi(c.y, nb.y, h2b.y)};
}

// a level's two sweeps from zero: e1 = w h^2 b / 6, then one sweep of it
template <class T>
__global__ void __launch_bounds__(GB, 5) k_mg_first(int n, double h2, const double *__restrict__ b,
                                                double *__restrict__ e, const GravCtrl *gc)
{
    if (gc->done) return;
    const double k = MG_OMEGA * h2 / 6.0;
    cube_cells<T>(
        n, [&](auto at) { return at(b); },
        [&](auto at, T c, T sx, T sy, T sz) {
            at.put(e, mg_jacobi(k * c, k * (sx + sy + sz), h2 * c));
        });
}

// one sweep; mean: also the mean of the result (the base grid's last sweep)
template <class T>
__global__ void __launch_bounds__(GB, 5) k_mg_sweep(int n, double h2, const double *__restrict__ old,
                                                const double *__restrict__ b, double *__restrict__ e,
                                                int mean, double *part, GravCtrl *gc)
{
    if (gc->done) return;
    double s = 0.0;
    cube_cells<T>(
        n, [&](auto at) { return at(old); },
        [&](auto at, T c, T sx, T sy, T sz) {
            const T v = mg_jacobi(c, sx + sy + sz, h2 * at(b));
            at.put(e, v);
            if (mean) s = s + total(v);
        });
    double all;
    if (mean && grid_sum(s, part, &gc->ticket, all)) gc->mgmu = all / ((double)n * n * n);
}

// _mgk_residual! (33-43) and _mgk_restrict! (45-53): the coarse right-hand side
// is the mean of the 8 children's b - (6 e - sum_nb) / h^2
__device__ __forceinline__ double mg_coarse_rhs(int n, double invh2, const double *e, const double *b,
                                                int X, int Y, int Z)
{
    const int nn = n * n, x[4] = {mg_wrap(2 * X - 1, n), 2 * X, 2 * X + 1, mg_wrap(2 * X + 2, n)};
    const int y[4] = {mg_wrap(2 * Y - 1, n) * n, 2 * Y * n, (2 * Y + 1) * n, mg_wrap(2 * Y + 2, n) * n};
    const int z[4] = {mg_wrap(2 * Z - 1, n) * nn, 2 * Z * nn, (2 * Z + 1) * nn, mg_wrap(2 * Z + 2, n) * nn};
    double sb = 0.0, in = 0.0, out = 0.0;
#pragma unroll
    for (int k = 1; k < 3; ++k)
#pragma unroll
        for (int j = 1; j < 3; ++j) {
#pragma unroll
            for (int i = 1; i < 3; ++i) {
                sb = sb + b[x[i] + y[j] + z[k]];
                in = in + e[x[i] + y[j] + z[k]];
            }
            out = out + (e[x[0] + y[j] + z[k]] + e[x[3] + y[j] + z[k]]);
            out = out + (e[x[j] + y[0] + z[k]] + e[x[j] + y[3] + z[k]]);
            out = out + (e[x[j] + y[k] + z[0]] + e[x[j] + y[k] + z[3]]);
        }
    // each child has three of its siblings and three outer cells as neighbours
    return 0.125 * (sb - (3.0 * in - out) * invh2);
}

__global__ void __launch_bounds__(GB) k_mg_down(int nc, double invh2, const double *__restrict__ e,
                                               const double *__restrict__ b, double *__restrict__ bc,
                                               const GravCtrl *gc)
{
    if (gc->done) return;
    const int I = blockIdx.x * GB + threadIdx.x;
    if (I >= nc * nc * nc) return;
    int C[3];
    cube_coords(nc, I, C);
    bc[I] = mg_coarse_rhs(2 * nc, invh2, e, b, C[0], C[1], C[2]);
}

// _mgk_prolong_add! (55-66): trilinear cell-centred prolongation (weights 3/4,
// 1/4, periodic) at fine cell (x, y, z)
__device__ __forceinline__ double mg_prolong(int nc, const double *ec, int x, int y, int z)
{
    const int i0 = x >> 1, i1 = mg_wrap(i0 + ((x & 1) ? 1 : -1), nc);
    const int j0 = (y >> 1) * nc, j1 = mg_wrap((y >> 1) + ((y & 1) ? 1 : -1), nc) * nc;
    const int k0 = (z >> 1) * nc * nc, k1 = mg_wrap((z >> 1) + ((z & 1) ? 1 : -1), nc) * nc * nc;
    auto line = [&](int o) { return 0.75 * ec[i0 + o] + 0.25 * ec[i1 + o]; };
    auto face = [&](int o) { return 0.75 * line(j0 + o) + 0.25 * line(j1 + o); };
    return 0.75 * face(k0) + 0.25 * face(k1);
}

// The same for a whole level, added to e: a thread takes the 8 children of a
// coarse cell from the 27 coarse values around it, interpolated along x, then
// y, then z as above.
__global__ void __launch_bounds__(GB) k_mg_up(int nc, const double *__restrict__ ec,
                                             double *__restrict__ e, const GravCtrl *gc)
{
    if (gc->done) return;
    const int I = blockIdx.x * GB + threadIdx.x;
    if (I >= nc * nc * nc) return;
    int C[3];
    cube_coords(nc, I, C);
    const int n = 2 * nc;
    const int x[3] = {mg_wrap(C[0] - 1, nc), C[0], mg_wrap(C[0] + 1, nc)};
    D2 f[3][2];  // the children's x pair: by coarse z and child y
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        D2 l[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double *p = ec + (mg_wrap(C[2] + k - 1, nc) * nc + mg_wrap(C[1] + j - 1, nc)) * nc;
            const double m = 0.75 * p[x[1]];
            l[j] = {m + 0.25 * p[x[0]], m + 0.25 * p[x[2]]};
        }
        f[k][0] = 0.75 * l[1] + 0.25 * l[0];
        f[k][1] = 0.75 * l[1] + 0.25 * l[2];
    }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const At<D2> at{((2 * C[2] + k) * n + 2 * C[1] + j) * n + 2 * C[0]};
            at.put(e, at(e) + (0.75 * f[1][j] + 0.25 * f[2 * k][j]));
        }
}

// The V-cycle from a level of n <= MG_BLOCK down, in one block: b in, e out.
// Shared memory per level: e, t, b.
__global__ void __launch_bounds__(1024) k_mg_bottom(int n, double h, const double *__restrict__ b,
                                                   double *__restrict__ e, const GravCtrl *gc)
{
    extern __shared__ double sm[];
    if (gc->done) return;
    const int t = threadIdx.x;
    auto sweep = [&](int m, double h2, const double *old, const double *rhs, double *out) {
        for (int i = t; i < m * m * m; i += blockDim.x) {
            int c[3];
            cube_coords(m, i, c);
            const int mm = m * m;
            const double s = old[i - c[0] + mg_wrap(c[0] - 1, m)] + old[i - c[0] + mg_wrap(c[0] + 1, m)] +
                             old[i + (mg_wrap(c[1] - 1, m) - c[1]) * m] + old[i + (mg_wrap(c[1] + 1, m) - c[1]) * m] +
                             old[i + (mg_wrap(c[2] - 1, m) - c[2]) * mm] + old[i + (mg_wrap(c[2] + 1, m) - c[2]) * mm];
            out[i] = mg_jacobi(old[i], s, h2 * rhs[i]);
        }
        __syncthreads();
    };
    for (int i = t; i < n * n * n; i += blockDim.x) sm[2 * n * n * n + i] = b[i];
    __syncthreads();
    double *base = sm;
    int m = n;
    double hm = h;
    for (;;) {  // down: two sweeps from zero, then the coarse right-hand side
        const int mc = m * m * m;
        double *E = base, *T = base + mc, *B = base + 2 * mc;
        const double h2 = hm * hm, k = MG_OMEGA * h2 / 6.0;
        for (int i = t; i < mc; i += blockDim.x) T[i] = k * B[i];
        __syncthreads();
        sweep(m, h2, T, B, E);
        if (!(m > 4 && m % 2 == 0)) {  // coarsest: 30 more sweeps
            for (int q = 0; q < 30; q += 2) {
                sweep(m, h2, E, B, T);
                sweep(m, h2, T, B, E);
            }
            break;
        }
        double *next = base + 3 * mc;
        const int c = m / 2, cc = c * c * c;
        for (int I = t; I < cc; I += blockDim.x) {
            int C[3];
            cube_coords(c, I, C);
            next[2 * cc + I] = mg_coarse_rhs(m, 1.0 / h2, E, B, C[0], C[1], C[2]);
        }
        __syncthreads();
        base = next;
        m = c;
        hm = 2.0 * hm;
    }
    while (m < n) {  // up: the coarse correction, then two sweeps
        const double *ec = base;
        const int f = 2 * m, fc = f * f * f;
        base -= 3 * fc;
        hm = 0.5 * hm;
        double *E = base, *T = base + fc, *B = base + 2 * fc;
        for (int i = t; i < fc; i += blockDim.x) {
            int c[3];
            cube_coords(f, i, c);
            E[i] = E[i] + mg_prolong(m, ec, c[0], c[1], c[2]);
        }
        __syncthreads();
        sweep(f, hm * hm, E, B, T);
        sweep(f, hm * hm, T, B, E);
        m = f;
    }
    for (int i = t; i < n * n * n; i += blockDim.x) e[i] = base[i];
}

// shared memory of k_mg_bottom
inline size_t mg_bottom_smem(int n)
{
    size_t d = 0;
    for (;;) {
        d += 3 * (size_t)n * n * n;
        if (!(n > 4 && n % 2 == 0)) break;
        n /= 2;
    }
    return d * sizeof(double);
}

// partials of sum(e) over the base grid (the correction's mean)
__global__ void __launch_bounds__(GB, GP_SM) k_sumpart(int64_t n, const double *__restrict__ e, double *part,
                                               const GravCtrl *gc)
{
    __shared__ double sh[GB];
    if (gc->done) return;
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * GB + threadIdx.x; i < n; i += (int64_t)GP * GB) s = s + e[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void __launch_bounds__(1024) k_sum_final(const double *part, int64_t n, GravCtrl *gc)
{
    __shared__ double sh[1024];
    if (gc->done) return;
    const double s = final_sum(part, sh);
    if (threadIdx.x == 0) gc->mgmu = s / (double)n;
}

}  // namespace
}  // namespace vb

using vb::detail::fail;
using vb::detail::use;

struct vb_gravity {
    vb::GravP P{};
    double *phi = nullptr, *b = nullptr, *r = nullptr, *p = nullptr, *Ap = nullptr;
    double *gacc = nullptr, *part = nullptr;
    // periodic cube (n^3, n <= 1024, phi periodic on every side): its solver's
    // second direction buffer and block partials
    int cube_n = 0;
    double *p2 = nullptr, *cpart = nullptr;
    vb::GravCtrl *gc = nullptr;   // device
    vb::GravCtrl *hgc = nullptr;  // pinned host mirror
    cudaGraphExec_t gexec = nullptr;
    long long maxiter = 500;
    double tol = 1e-8;
    bool limits_set = false;      // maxiter and tol are in the device block
    // multigrid preconditioner (precond = VB_GRAV_PRECOND_MG)
    int precond = VB_GRAV_PRECOND_NONE;
    double *z = nullptr, *z2 = nullptr;
    struct Level {
        int n;
        double h;
        double *e, *b, *t;
    };
    std::vector<Level> lev;  // base grid first, then each coarsening
    double vbase = 0.0;
    int64_t graph_launches = 0;  // kernels per replay of the iteration graph
};

namespace {

// launch kern<ND> on the grid-stride grid; evaluates to 1 (one launch)
#define ND_DISPATCH(nd, kern, ...)                                        \
    ((nd) == 1   ? (kern<1><<<vb::GP, vb::GB, 0, s>>>(__VA_ARGS__), 1)   \
     : (nd) == 2 ? (kern<2><<<vb::GP, vb::GB, 0, s>>>(__VA_ARGS__), 1)   \
                 : (kern<3><<<vb::GP, vb::GB, 0, s>>>(__VA_ARGS__), 1))

// One CG iteration (five launches; each returns at once after convergence).
inline unsigned mg_blocks(int64_t n) { return (unsigned)((n + vb::GB - 1) / vb::GB); }

int queue_iteration(vb_grid *gr, vb_gravity *gv)
{
    cudaStream_t s = gr->ctx->stream;
    const vb::Geom &g = gr->g;
    VB_CHECK_LAUNCH(gr->ctx, ND_DISPATCH(g.nd, vb::k_cg_matvec, g, gv->P, gv->p, gv->Ap, gv->part, gv->gc));
    vb::k_cg_alpha<<<1, 1024, 0, s>>>(gv->part, gv->gc);
    VB_CHECK_LAUNCH(gr->ctx, 1);
    vb::k_cg_update<<<vb::GP, vb::GB, 0, s>>>(g, gv->phi, gv->p, gv->r, gv->Ap, gv->part, gv->gc);
    VB_CHECK_LAUNCH(gr->ctx, 1);
    vb::k_cg_beta<<<1, 1024, 0, s>>>(gv->part, gv->gc);
    VB_CHECK_LAUNCH(gr->ctx, 1);
    vb::k_cg_dir<<<vb::GP, vb::GB, 0, s>>>(g, gv->p, gv->r, gv->gc);
    VB_CHECK_LAUNCH(gr->ctx, 1);
    return VB_OK;
}

dim3 cube_grid(int n)
{
    const int kz = vb::cube_kz(n);
    return dim3((unsigned)((n + 31) / 32), (unsigned)((n + 7) / 8), (unsigned)((n + kz - 1) / kz));
}
// launch kern on the cells of an n^3 cube, in pairs where n is even
#define CUBE_LAUNCH(kern, n, ...)                                                        \
    do {                                                                                 \
        dim3 cg_ = cube_grid(n);                                                         \
        if ((n) % 2 == 0) {                                                              \
            cg_.y = ((unsigned)(n) + 15) / 16;                                           \
            vb::kern<vb::D2><<<cg_, vb::GB, 0, s>>>(__VA_ARGS__);                        \
        } else {                                                                         \
            vb::kern<double><<<cg_, vb::GB, 0, s>>>(__VA_ARGS__);                        \
        }                                                                                \
    } while (0)
constexpr unsigned CUBE_UPDATE_BLOCKS = 1184;  // k_cube_update: 8 per SM

vb::CubeP cube_params(const vb_gravity *gv)
{
    vb::CubeP P;
    P.n = gv->cube_n;
    double diag = 0.0;
    for (int d = 2; d >= 0; --d) diag += gv->P.coef[d];
    for (int d = 0; d < 3; ++d) diag += gv->P.coef[d];
    for (int d = 0; d < 3; ++d) P.c[d] = gv->P.coef[d];
    P.w = vb::MG_OMEGA / diag;
    return P;
}

// z = M^-1 r (one composite-smoothed two-level cycle), then r.z and its scalars
int queue_precond(vb_grid *gr, vb_gravity *gv, bool start, cudaGraphConditionalHandle more)
{
    cudaStream_t s = gr->ctx->stream;
    const vb::CubeP P = cube_params(gv);
    CUBE_LAUNCH(k_cube_pre, P.n, P, gv->r, gv->z, gv->gc);
    auto &top = gv->lev[0];
    CUBE_LAUNCH(k_cube_resid, P.n, P, gv->z, gv->r, top.b, gv->gc);
    VB_CHECK_LAUNCH(gr->ctx, 2);
    const int L = (int)gv->lev.size();
    // the first level that k_mg_bottom takes, or the coarsest one
    int bot = 0;
    while (bot < L - 1 && gv->lev[bot].n > vb::MG_BLOCK) ++bot;
    auto sweep = [&](const vb_gravity::Level &l, const double *old, double *out, bool mean) {
        CUBE_LAUNCH(k_mg_sweep, l.n, l.n, l.h * l.h, old, l.b, out, mean ? 1 : 0, gv->cpart, gv->gc);
        return 1;
    };
    for (int k = 0; k < bot; ++k) {
        const auto &l = gv->lev[k], &c = gv->lev[k + 1];
        CUBE_LAUNCH(k_mg_first, l.n, l.n, l.h * l.h, l.b, l.e, gv->gc);
        vb::k_mg_down<<<mg_blocks((int64_t)c.n * c.n * c.n), vb::GB, 0, s>>>(
            c.n, 1.0 / (l.h * l.h), l.e, l.b, c.b, gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 2);
    }
    {
        const auto &l = gv->lev[bot];
        if (l.n <= vb::MG_BLOCK) {
            vb::k_mg_bottom<<<1, 1024, vb::mg_bottom_smem(l.n), s>>>(l.n, l.h, l.b, l.e, gv->gc);
            VB_CHECK_LAUNCH(gr->ctx, 1);
        } else {  // a coarsest level too large for one block (odd side)
            CUBE_LAUNCH(k_mg_first, l.n, l.n, l.h * l.h, l.b, l.e, gv->gc);
            VB_CHECK_LAUNCH(gr->ctx, 1);
            for (int q = 0; q < 30; q += 2)
                VB_CHECK_LAUNCH(gr->ctx, sweep(l, l.e, l.t, false) + sweep(l, l.t, l.e, false));
        }
    }
    for (int k = bot - 1; k >= 0; --k) {
        const auto &l = gv->lev[k], &c = gv->lev[k + 1];
        vb::k_mg_up<<<mg_blocks((int64_t)c.n * c.n * c.n), vb::GB, 0, s>>>(c.n, c.e, l.e, gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 1);
        VB_CHECK_LAUNCH(gr->ctx, sweep(l, l.e, l.t, false) + sweep(l, l.t, l.e, k == 0));
    }
    if (bot == 0) {  // the base grid itself was the bottom: its correction's mean
        vb::k_sumpart<<<vb::GP, vb::GB, 0, s>>>((int64_t)P.n * P.n * P.n, top.e, gv->part + 2 * vb::GP, gv->gc);
        vb::k_sum_final<<<1, 1024, 0, s>>>(gv->part + 2 * vb::GP, (int64_t)P.n * P.n * P.n, gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 2);
    }
    CUBE_LAUNCH(k_cube_post1, P.n, P, gv->z, top.e, gv->r, 1.0 / gv->vbase, gv->z2, gv->gc);
    CUBE_LAUNCH(k_cube_post2, P.n, P, gv->z2, gv->r, gv->z, gv->cpart, gv->gc, start ? 1 : 0, more);
    VB_CHECK_LAUNCH(gr->ctx, 2);
    return VB_OK;
}

// One iteration on the cube (mg_pcg.jl:194-209, or CG).
int queue_cube_iteration(vb_grid *gr, vb_gravity *gv, cudaGraphConditionalHandle more)
{
    cudaStream_t s = gr->ctx->stream;
    const bool mg = gv->precond == VB_GRAV_PRECOND_MG;
    const vb::CubeP P = cube_params(gv);
    CUBE_LAUNCH(k_cube_dir, P.n, P, mg ? gv->z : gv->r, gv->p, gv->p2, gv->Ap, gv->cpart, gv->gc);
    vb::k_cube_update<<<CUBE_UPDATE_BLOCKS, vb::GB, 0, s>>>(P.n, gv->phi, gv->p, gv->p2, gv->r, gv->Ap,
                                                           gv->cpart, gv->gc, mg ? 0 : 1, more);
    VB_CHECK_LAUNCH(gr->ctx, 2);
    return mg ? queue_precond(gr, gv, false, more) : VB_OK;
}

// The cube's iterations as one graph: a WHILE node whose body is one iteration
// (CG: 8, each of which returns at once after the stop) and whose condition the
// last reduction of each sets from the stop flag.  Going round the loop takes 4
// us, which the two launches of a CG iteration on a small cube show: 19.1, 17.0,
// 15.9, 15.4 and 15.1 us an iteration at 48^3 with 1, 2, 4, 8 and 16 in the body
// (five plain launches: 16.0), 245 and 242 at 256^3 with 1 and 8.
constexpr int CG_BODY = 8;
int capture_cube(vb_grid *gr, vb_gravity *gv)
{
    cudaStream_t s = gr->ctx->stream;
    cudaGraph_t root = nullptr;
    VB_CUDA(cudaGraphCreate(&root, 0));
    cudaGraphConditionalHandle h;
    cudaGraphNodeParams cp = {};
    cudaGraphNode_t node;
    cudaError_t e = cudaGraphConditionalHandleCreate(&h, root, 1, cudaGraphCondAssignDefault);
    if (e == cudaSuccess) {
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        e = cudaGraphAddNode(&node, root, nullptr, 0, &cp);
    }
    if (e == cudaSuccess)
        e = cudaStreamBeginCaptureToGraph(s, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                          cudaStreamCaptureModeThreadLocal);
    int rc = VB_OK;
    if (e == cudaSuccess) {
        const int64_t before = gr->ctx->launches;
        const int body = gv->precond == VB_GRAV_PRECOND_MG ? 1 : CG_BODY;
        for (int k = 0; k < body && !rc; ++k) rc = queue_cube_iteration(gr, gv, h);
        cudaGraph_t out = nullptr;
        e = cudaStreamEndCapture(s, &out);
        gv->graph_launches = gr->ctx->launches - before;
        gr->ctx->launches = before;  // counted when the graph runs
    }
    if (!rc && e == cudaSuccess) e = cudaGraphInstantiate(&gv->gexec, root, 0);
    cudaGraphDestroy(root);
    if (!rc && e != cudaSuccess) {
        gv->gexec = nullptr;
        rc = fail(VB_ECUDA, std::string("gravity graph: ") + cudaGetErrorString(e));
    }
    return rc;
}

int capture_iterations(vb_grid *gr, vb_gravity *gv)
{
    cudaStream_t s = gr->ctx->stream;
    VB_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int64_t before = gr->ctx->launches;
    int rc = VB_OK;
    gv->graph_launches = 0;
    for (int k = 0; k < vb::GRAPH_ITERS && !rc; ++k)
        rc = queue_iteration(gr, gv);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(s, &graph);
    gv->graph_launches = gr->ctx->launches - before;
    gr->ctx->launches = before;  // counted per replay
    if (rc) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    if (e != cudaSuccess) return fail(VB_ECUDA, std::string("graph capture: ") + cudaGetErrorString(e));
    e = cudaGraphInstantiate(&gv->gexec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) {
        gv->gexec = nullptr;
        return fail(VB_ECUDA, std::string("graph instantiate: ") + cudaGetErrorString(e));
    }
    return VB_OK;
}

int refresh_accel(vb_grid *gr, vb_gravity *gv)
{
    cudaStream_t s = gr->ctx->stream;
    const vb::Geom &g = gr->g;
    if (gv->cube_n) {
        vb::k_cube_accel<<<cube_grid(gv->cube_n), vb::GB, 0, s>>>(g, gv->cube_n, gv->phi, gv->gacc);
        VB_CHECK_LAUNCH(gr->ctx, 1);
        return VB_OK;
    }
    VB_CHECK_LAUNCH(gr->ctx, ND_DISPATCH(g.nd, vb::k_accel, g, gv->P, gv->phi, gv->gacc));
    return VB_OK;
}

void free_gravity(vb_gravity *gv)
{
    if (!gv) return;
    if (gv->gexec) cudaGraphExecDestroy(gv->gexec);
    cudaFree(gv->phi);
    cudaFree(gv->b);
    cudaFree(gv->r);
    cudaFree(gv->p);
    cudaFree(gv->Ap);
    cudaFree(gv->gacc);
    cudaFree(gv->part);
    cudaFree(gv->cpart);
    cudaFree(gv->gc);
    cudaFreeHost(gv->hgc);
    cudaFree(gv->z);
    cudaFree(gv->z2);
    cudaFree(gv->p2);
    for (auto &l : gv->lev) {
        cudaFree(l.e);
        cudaFree(l.b);
        cudaFree(l.t);
    }
    delete gv;
}

int check_grid(vb_grid *gr)
{
    if (!gr) return fail(VB_EINVAL, "null grid");
    if (!gr->grav) return fail(VB_EINVAL, "gravity is not enabled on this grid");
    return use(gr->ctx);
}

}  // namespace

// solve_poisson! (src/gravity.jl:251-300) for the grid's current density,
// warm-started from the stored potential; then g = -grad phi for the stages.
int vb::detail::gravity_solve(vb_grid *gr, int64_t *iters, double *relres)
{
    vb_gravity *gv = gr->grav;
    cudaStream_t s = gr->ctx->stream;
    const Geom &g = gr->g;
    if (!gv->limits_set) {  // the stop criteria, once per configuration
        VB_CUDA(cudaMemcpyAsync(&gv->gc->maxiter, &gv->maxiter, sizeof(long long), cudaMemcpyHostToDevice, s));
        VB_CUDA(cudaMemcpyAsync(&gv->gc->tol, &gv->tol, sizeof(double), cudaMemcpyHostToDevice, s));
        gv->limits_set = true;
    }
    if (gv->P.project_mean) {
        k_meanpart<<<GP, GB, 0, s>>>(g, gr->U, gv->part);
        VB_CHECK_LAUNCH(gr->ctx, 1);
        k_mean_final<<<1, 1024, 0, s>>>(gv->part, gv->gc, 0);
        VB_CHECK_LAUNCH(gr->ctx, 1);
    }
    if (gv->cube_n) {
        const CubeP P = cube_params(gv);
        CUBE_LAUNCH(k_cube_init, P.n, P, gv->P, g.vol, gr->U, gv->phi, gv->r, gv->cpart, gv->gc);
        k_cube_init_final<<<1, 1, 0, s>>>(gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 2);
    } else {
        k_rhs<<<GP, GB, 0, s>>>(g, gv->P, gr->U, gv->b, gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 1);
        VB_CHECK_LAUNCH(gr->ctx, ND_DISPATCH(g.nd, k_cg_init, g, gv->P, gv->phi, gv->b, gv->r, gv->p, gv->part));
        k_cg_init_final<<<1, 1024, 0, s>>>(gv->part, gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 1);
    }
    if (!gv->gexec) {
        int rc = gv->cube_n ? capture_cube(gr, gv) : capture_iterations(gr, gv);
        if (rc) return rc;
    }
    if (gv->cube_n) {
        if (gv->precond == VB_GRAV_PRECOND_MG) {
            int rc = queue_precond(gr, gv, true, 0);
            if (rc) return rc;
        }
    }
    // the stop flag is set by convergence, p.Ap <= 0 or maxiter, so this ends
    for (;;) {
        VB_CUDA(cudaGraphLaunch(gv->gexec, s));
        gr->ctx->launches += gv->graph_launches;  // a cube's: of one iteration, the count stays on the device
        VB_CUDA(cudaMemcpyAsync(gv->hgc, gv->gc, sizeof(GravCtrl), cudaMemcpyDeviceToHost, s));
        if (gv->cube_n && gv->maxiter <= CUBE_RUN) break;
        VB_CUDA(cudaStreamSynchronize(s));
        if (gv->hgc->done) break;
        if (gv->cube_n) {
            k_cube_resume<<<1, 1, 0, s>>>(gv->gc);
            VB_CHECK_LAUNCH(gr->ctx, 1);
        }
    }
    if (gv->P.project_mean) {
        k_meanpart<<<GP, GB, 0, s>>>(g, gv->phi, gv->part);
        VB_CHECK_LAUNCH(gr->ctx, 1);
        k_mean_final<<<1, 1024, 0, s>>>(gv->part, gv->gc, 1);
        VB_CHECK_LAUNCH(gr->ctx, 1);
        k_sub_mean<<<GP, GB, 0, s>>>(g, gv->phi, gv->gc);
        VB_CHECK_LAUNCH(gr->ctx, 1);
    }
    int rc = refresh_accel(gr, gv);
    if (rc) return rc;
    if (gv->cube_n && (iters || relres)) VB_CUDA(cudaStreamSynchronize(s));
    if (iters) *iters = gv->hgc->iters;
    if (relres) *relres = gv->hgc->relres;
    return VB_OK;
}

void vb::detail::gravity_free(vb_gravity *gv) { free_gravity(gv); }

extern "C" {

int vb_gravity_enable(vb_grid *gr, const vb_gravity_desc *d)
{
    if (!gr || !d) return fail(VB_EINVAL, "null argument");
    if (d->flags != 0) return fail(VB_EINVAL, "flags must be 0");
    if (!(d->tol >= 0.0) || d->maxiter < 0) return fail(VB_EINVAL, "tol and maxiter must be non-negative");
    if (!std::isfinite(d->G)) return fail(VB_EINVAL, "G must be finite");
    int rc = use(gr->ctx);
    if (rc) return rc;
    const vb::Geom &g = gr->g;
    vb::GravP P{};
    for (int a = 0; a < 3; ++a) {
        if (a < g.nd) {
            for (int side = 0; side < 2; ++side) {
                const int bc = side ? d->bc_hi[a] : d->bc_lo[a];
                if (bc < VB_BC_OUTFLOW || bc > VB_BC_REFLECTING)
                    return fail(VB_EINVAL, "unknown boundary condition");
            }
            if ((d->bc_lo[a] == VB_BC_PERIODIC) != (d->bc_hi[a] == VB_BC_PERIODIC))
                return fail(VB_EINVAL, "a periodic axis must be periodic on both sides");
            P.per_lo[a] = d->bc_lo[a] == VB_BC_PERIODIC;
            P.per_hi[a] = d->bc_hi[a] == VB_BC_PERIODIC;
            P.coef[a] = g.area[a] / (0.5 * (g.w[a] + g.w[a]));  // area / _face_distance
        } else {
            P.per_lo[a] = P.per_hi[a] = 1;
            P.coef[a] = 0.0;
        }
    }
    P.G = d->G;
    P.project_mean = d->project_mean ? 1 : 0;
    if (d->precond != VB_GRAV_PRECOND_NONE && d->precond != VB_GRAV_PRECOND_MG)
        return fail(VB_EINVAL, "unknown preconditioner");
    if (d->precond == VB_GRAV_PRECOND_MG) {
        // the base-grid V-cycle is periodic and cubic (mg_pcg.jl:88-89)
        bool ok = g.nd == 3 && g.n[0] == g.n[1] && g.n[1] == g.n[2] && g.n[0] <= 1024;
        for (int a = 0; a < 3; ++a) ok = ok && P.per_lo[a] && P.per_hi[a];
        if (!ok)
            return fail(VB_ENOTSUP, "the multigrid preconditioner needs a 3D cubic grid (n <= 1024) "
                                    "with periodic phi on every side");
    }
    bool cube = g.nd == 3 && g.n[0] == g.n[1] && g.n[1] == g.n[2] && g.n[0] <= 1024;
    for (int a = 0; a < 3; ++a) cube = cube && P.per_lo[a] && P.per_hi[a];
    const bool mg = d->precond == VB_GRAV_PRECOND_MG;
    // Everything that can fail comes first: a grid that has gravity keeps it, with
    // its settings, when it does.  Each buffer is guarded by its own pointer (a
    // failed call's are taken up by the next one, or freed with the rest).
    vb_gravity *gv = gr->grav ? gr->grav : new (std::nothrow) vb_gravity;
    if (!gv) return fail(VB_ENOMEM, "host allocation failed");
    cudaError_t e = cudaSuccess;
    auto need = [&](auto **p, size_t bytes) {
        if (e == cudaSuccess && !*p) e = cudaMalloc(p, bytes);
    };
    const size_t n = (size_t)g.ncell * sizeof(double);
    for (double **buf : {&gv->phi, &gv->r, &gv->p, &gv->Ap}) need(buf, n);
    if (!cube) need(&gv->b, n);  // a cube's first pass forms its right-hand side where it reads it
    need(&gv->gacc, n * g.nd);
    need(&gv->part, sizeof(double) * 3 * vb::GP);
    need(&gv->gc, sizeof(vb::GravCtrl));
    if (e == cudaSuccess && !gv->hgc) e = cudaMallocHost(&gv->hgc, sizeof(vb::GravCtrl));
    if (cube) {
        const dim3 b = cube_grid((int)g.n[0]);
        need(&gv->cpart, sizeof(double) * std::max<size_t>(2 * (size_t)b.x * b.y * b.z, CUBE_UPDATE_BLOCKS));
        need(&gv->p2, n);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(vb::k_mg_bottom, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)vb::mg_bottom_smem(vb::MG_BLOCK));
    }
    if (mg) {
        for (double **buf : {&gv->z, &gv->z2}) need(buf, n);
        if (gv->lev.empty()) {  // levels: coarsen while even and > 4 (mg_pcg.jl:111-116)
            int nl = (int)g.n[0];
            double h = g.w[0];
            gv->vbase = h * h * h;
            for (;;) {
                gv->lev.push_back({nl, h, nullptr, nullptr, nullptr});
                if (!(nl > 4 && nl % 2 == 0)) break;
                nl /= 2;
                h *= 2.0;
            }
        }
        for (auto &l : gv->lev) {
            const size_t bytes = sizeof(double) * (size_t)l.n * l.n * l.n;
            need(&l.e, bytes);
            need(&l.b, bytes);
            if (l.n > vb::MG_BLOCK) need(&l.t, bytes);  // k_mg_bottom's levels sweep in shared memory
        }
    }
    if (e == cudaSuccess && !gr->grav) {
        std::memset(gv->hgc, 0, sizeof(vb::GravCtrl));
        e = cudaMemsetAsync(gv->phi, 0, n, gr->ctx->stream);  // phi starts at 0
        if (e == cudaSuccess) e = cudaMemsetAsync(gv->gacc, 0, n * g.nd, gr->ctx->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(gv->gc, 0, sizeof(vb::GravCtrl), gr->ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(gr->ctx->stream);
    }
    if (e != cudaSuccess) {
        if (!gr->grav) free_gravity(gv);
        cudaGetLastError();
        return fail(e == cudaErrorMemoryAllocation ? VB_ENOMEM : VB_ECUDA,
                    std::string("gravity allocation: ") + cudaGetErrorString(e));
    }
    gv->P = P;
    gv->cube_n = cube ? (int)g.n[0] : 0;
    gv->maxiter = d->maxiter;
    gv->tol = d->tol;
    gv->limits_set = false;
    gv->precond = d->precond;
    if (gv->gexec) {  // the iteration graph depends on all of these
        cudaGraphExecDestroy(gv->gexec);
        gv->gexec = nullptr;
    }
    gr->grav = gv;
    gr->g.grav_g = gv->gacc;
    gr->g.grav_G = d->G;
    gr->box_kz = -1;          // the tiled kernels' box descriptor carries the geometry
    gr->invdt_valid = false;  // the free-fall limiter joins the CFL maximum
    return VB_OK;
}

int vb_gravity_disable(vb_grid *gr)
{
    if (!gr) return fail(VB_EINVAL, "null grid");
    if (!gr->grav) return VB_OK;
    int rc = use(gr->ctx);
    if (rc) return rc;
    cudaStreamSynchronize(gr->ctx->stream);
    free_gravity(gr->grav);
    gr->grav = nullptr;
    gr->g.grav_g = nullptr;
    gr->g.grav_G = 0.0;
    gr->box_kz = -1;
    gr->invdt_valid = false;
    return VB_OK;
}

int vb_gravity_solve(vb_grid *gr, int64_t *iters, double *relres)
{
    VB_RANGE("vb_gravity_solve");
    int rc = check_grid(gr);
    if (rc) return rc;
    return vb::detail::gravity_solve(gr, iters, relres);
}

int vb_gravity_phi(vb_grid *gr, double *phi)
{
    int rc = check_grid(gr);
    if (rc) return rc;
    if (!phi) return fail(VB_EINVAL, "null output");
    VB_CUDA(cudaMemcpyAsync(phi, gr->grav->phi, sizeof(double) * gr->g.ncell, cudaMemcpyDeviceToHost,
                            gr->ctx->stream));
    VB_CUDA(cudaStreamSynchronize(gr->ctx->stream));
    return VB_OK;
}

int vb_gravity_set_phi(vb_grid *gr, const double *phi)
{
    int rc = check_grid(gr);
    if (rc) return rc;
    if (!phi) return fail(VB_EINVAL, "null input");
    VB_CUDA(cudaMemcpyAsync(gr->grav->phi, phi, sizeof(double) * gr->g.ncell, cudaMemcpyHostToDevice,
                            gr->ctx->stream));
    rc = refresh_accel(gr, gr->grav);
    if (rc) return rc;
    VB_CUDA(cudaStreamSynchronize(gr->ctx->stream));
    return VB_OK;
}

int vb_gravity_accel(vb_grid *gr, double *gout)
{
    int rc = check_grid(gr);
    if (rc) return rc;
    if (!gout) return fail(VB_EINVAL, "null output");
    VB_CUDA(cudaMemcpyAsync(gout, gr->grav->gacc, sizeof(double) * gr->g.ncell * gr->g.nd,
                            cudaMemcpyDeviceToHost, gr->ctx->stream));
    VB_CUDA(cudaStreamSynchronize(gr->ctx->stream));
    return VB_OK;
}

int vb_gravity_laplacian(vb_grid *gr, const double *x, double *Ax)
{
    VB_RANGE("vb_gravity_laplacian");
    int rc = check_grid(gr);
    if (rc) return rc;
    if (!x || !Ax) return fail(VB_EINVAL, "null argument");
    vb_gravity *gv = gr->grav;
    cudaStream_t s = gr->ctx->stream;
    const size_t n = sizeof(double) * gr->g.ncell;
    // the CG scratch r (input) and Ap (output) are free between solves
    VB_CUDA(cudaMemcpyAsync(gv->r, x, n, cudaMemcpyHostToDevice, s));
    VB_CHECK_LAUNCH(gr->ctx, ND_DISPATCH(gr->g.nd, vb::k_lap, gr->g, gv->P, gv->r, gv->Ap));
    VB_CUDA(cudaMemcpyAsync(Ax, gv->Ap, n, cudaMemcpyDeviceToHost, s));
    VB_CUDA(cudaStreamSynchronize(s));
    return VB_OK;
}

}  // extern "C"
