// vb_march.cu -- whole runs of small float64 1D and 2D grids in one launch.
//
// A step of such a grid is latency: as separate kernels (dt, stage 1, stage 2,
// clock) it cost 17 us at 128 cells and 26 us at 64 x 64 (a whole run over its
// steps), nearly all of it launches, loads from L2 and the serial chain of one
// flux.  Here one cluster of up to 16 blocks keeps the state in shared memory
// and runs the steps in a loop: 3.6 us and 8.7 us a step.  Of 17 k cycles at
// 64 x 64 the face solves take 7.5 k (the float64 pipes of 16 SMs), the cluster
// barriers 3.6 k, both updates 3.6 k.  Each block owns a slab of rows (1D: of
// cells), about 256 cells; two cluster barriers a step (a grid of one block: two
// block barriers) separate the stages, the two rows of halo on each side are read
// from the neighbours' shared memory, and the CFL maximum rides on the first
// barrier.  One thread solves each face once (hllc_frame with its quotients side
// by side).
//
// Same operations and per-cell accumulation order as the cell-centric kernel,
// compiled with -fmad=false: bit-identical to it and to the oracle.
#include <cooperative_groups.h>

#include "vb_launch.h"
#include "vb_physics.cuh"
#include "vb_stage_generic.cuh"
#include "vb_stage_tiled3d.cuh"

namespace cg = cooperative_groups;

namespace vb {

namespace {

constexpr int MARCH_CLUSTER = 16;      // blocks of a cluster at most
constexpr int MARCH_THREADS = 640;     // threads of a block at most (96 registers)
constexpr int MARCH_CELLS = 256;       // cells of a block while the cluster can still grow
constexpr size_t MARCH_SMEM = 225 * 1024;

// the row axis is the last; a row of a 1D grid is one cell
struct MarchPlan {
    int blocks, rows, threads;  // cluster size, rows of a block at most, threads of a block
    size_t smem;
};

__host__ __device__ inline int march_doubles(int rows, int L, bool two)
{
    int n = 2 * 5 * (rows + 4) * L;           // primitives of both stages, with halo rows
    if (two) n += 5 * rows * (L + 1);         // faces within rows
    n += 5 * (rows + 1) * L;                  // faces between rows
    return n + 2 * 5 * rows * L;              // step-start and stage state
}

bool march_plan(const Geom &g, MarchPlan *p)
{
    if (g.nd > 2) return false;
    for (int d = 0; d < g.nd; ++d)
        if (g.n[d] < 4) return false;
    if (g.ncell > 32768) return false;
    const int L = g.nd == 1 ? 1 : (int)g.n[0], nr = (int)g.n[g.nd - 1];
    int c = (int)((g.ncell + MARCH_CELLS - 1) / MARCH_CELLS);
    c = c > MARCH_CLUSTER ? MARCH_CLUSTER : c;
    c = c > nr ? nr : c;
    p->blocks = c;
    p->rows = (nr + c - 1) / c;
    p->smem = sizeof(double) * (size_t)march_doubles(p->rows, L, g.nd == 2);
    const int tasks = (g.nd == 2 ? p->rows * (L + 1) : 0) + (p->rows + 1) * L;
    p->threads = (tasks + 31) / 32 * 32;
    if (p->threads > MARCH_THREADS) p->threads = MARCH_THREADS;
    return p->smem <= MARCH_SMEM;
}

template <int ND>
__global__ void __launch_bounds__(MARCH_THREADS, 1)
k_march(const __grid_constant__ Geom g, double *__restrict__ U, Ctrl *ctrl, long long nsteps, int rmax)
{
    extern __shared__ __align__(16) double sm[];
    __shared__ double red[32];
    __shared__ double slot[2][MARCH_CLUSTER];  // every block's CFL maximum, by step parity
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int t = threadIdx.x, T = blockDim.x;
    const int L = ND == 1 ? 1 : (int)g.n[0], NR = (int)g.n[ND - 1];
    auto row0 = [&](int r) { return r * NR / C; };  // r < 16, NR <= 32768
    const int ra = row0(rank), R = row0(rank + 1) - ra, own = R * L;
    const int ws = (rmax + 4) * L;                  // field stride of a primitive buffer
    const int xs = rmax * (L + 1), ys = (rmax + 1) * L, us = rmax * L;
    double *const wb[2] = {sm, sm + 5 * ws};
    double *const fx = sm + 10 * ws;                // ND 2 only
    double *const fy = ND == 2 ? fx + 5 * xs : fx;
    double *const u0 = fy + 5 * ys, *const uc = u0 + 5 * us;
    const double gamma = g.gamma, ig1 = inv_gamma1(gamma);
    double yw[ND];  // 1 / w_d
#pragma unroll
    for (int d = 0; d < ND; ++d) yw[d] = rcp64(g.w[d]);
    const double avol = g.aexp * g.vol;
    const int bcl = g.bc_lo[ND - 1], bch = g.bc_hi[ND - 1];
    auto barrier = [&] {
        if (C > 1) cl.sync();
        else __syncthreads();
    };

    // primitives of a new state of own cell c into buffer w, and its CFL terms
    // (|v_d| + c): the largest is divided by the width once (a division by a
    // constant keeps the order, so the maximum has the same bits)
    auto prim = [&](const double u[5], int c, double *w, double m[ND], bool cfl) {
        double W[5];
        cons2prim(u, gamma, W);
#pragma unroll
        for (int f = 0; f < 5; ++f) w[f * ws + 2 * L + c] = W[f];
        if (cfl) {
            const double gp = gamma * W[4], q = gp > 1e-30 && gp < 1e30 && W[0] > 1e-30 && W[0] < 1e30
                                                    ? quot64(gp, W[0], rcp64(W[0]))
                                                    : gp / W[0];
            const double cs = q > 1e-30 && q < 1e30 ? root64(q) : sqrt(q);
#pragma unroll
            for (int d = 0; d < ND; ++d) m[d] = nan_max(m[d], fabs(W[1 + d]) + cs);
        }
    };
    // the block's maximum into every block's slot; the next barrier publishes it
    auto publish = [&](const double m[ND], int par) {
        double q = 0.0;
#pragma unroll
        for (int d = 0; d < ND; ++d)
            q = nan_max(q, m[d] > 1e-30 && m[d] < 1e30 && g.w[d] > 1e-30 && g.w[d] < 1e30
                               ? quot64(m[d], g.w[d], yw[d])
                               : m[d] / g.w[d]);
        q = warp_max(q);
        if ((t & 31) == 0) red[t >> 5] = q;
        __syncthreads();
        if (t < 32) {
            q = warp_max(t < (T >> 5) ? red[t] : 0.0);
            if (t < C) *cl.map_shared_rank(&slot[par][rank], t) = q;
        }
    };
    // rows -2, -1, R, R+1 of buffer w: the neighbours' rows, wrapped on a
    // periodic axis, else mirrored, a reflecting wall negating the normal
    // velocity.  A thread's elements are the same every time: the first one's
    // place is worked out once.
    auto halo_place = [&](int i, int &o, int &src, int &dst, bool &flip) {
        const int h = i / L, x = i - h * L, lr = h < 2 ? h - 2 : R + h - 2;
        int r = ra + lr;
        flip = false;
        if (r < 0) {
            flip = bcl == BC_REFLECTING;
            r = bcl == BC_PERIODIC ? r + NR : -1 - r;
        } else if (r >= NR) {
            flip = bch == BC_REFLECTING;
            r = bch == BC_PERIODIC ? r - NR : 2 * NR - 1 - r;
        }
        o = ((r + 1) * C - 1) / NR;
        src = (r - row0(o) + 2) * L + x;
        dst = (lr + 2) * L + x;
    };
    int ho = 0, hsrc = 0, hdst = 0;
    bool hflip = false;
    if (t < 4 * L) halo_place(t, ho, hsrc, hdst, hflip);
    auto halo = [&](double *w) {
        for (int i = t; i < 4 * L; i += T) {
            int o = ho, is = hsrc, id = hdst;
            bool flip = hflip;
            if (i != t) halo_place(i, o, is, id, flip);
            if (!VB_DCHECK(o >= 0 && o < C && is >= 0 && is < ws && id >= 0 && id < ws)) continue;  // check build only
            const double *src = (C > 1 ? cl.map_shared_rank(w, o) : w) + is;
            double v[5];
#pragma unroll
            for (int f = 0; f < 5; ++f) v[f] = src[f * ws];
            if (flip) v[ND] = -v[ND];
#pragma unroll
            for (int f = 0; f < 5; ++f) w[f * ws + id] = v[f];
        }
        __syncthreads();
    };
    // Face j of the block, one body for both axes: the four cells across it
    // (o[]), where its flux goes, and which of the four a reflecting x wall
    // mirrors (bits 0..3 of flags; bit 4: an x face).  A thread's first face is
    // the same every time and is worked out once.
    const int nxf = ND == 2 ? R * (L + 1) : 0, nf = nxf + (R + 1) * L;
    struct Face {
        int o[4], out, flags;
    };
    auto face_place = [&](int j) {
        Face f;
        if (ND == 2 && j < nxf) {
            const int lr = j / (L + 1), x = j - lr * (L + 1);
            f.out = j;
            f.flags = 16;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                int c = x - 2 + k;
                if (c < 0) {
                    if (g.bc_lo[0] == BC_REFLECTING) f.flags |= 1 << k;
                    c = g.bc_lo[0] == BC_PERIODIC ? c + L : -1 - c;
                } else if (c >= L) {
                    if (g.bc_hi[0] == BC_REFLECTING) f.flags |= 1 << k;
                    c = g.bc_hi[0] == BC_PERIODIC ? c - L : 2 * L - 1 - c;
                }
                f.o[k] = (lr + 2) * L + c;
            }
        } else {  // below row i / L: rows -2 .. 1 of it
            const int i = j - nxf;
            f.out = i;
            f.flags = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) f.o[k] = i + k * L;
        }
        return f;
    };
    const Face face0 = face_place(t < nf ? t : 0);
    // every face of the block's cells, area * flux
    auto faces = [&](const double *w) {
        for (int j = t; j < nf; j += T) {
            const Face f = j == t ? face0 : face_place(j);
            const bool isx = ND == 1 || (f.flags & 16);
            if (!VB_DCHECK(f.o[0] >= 0 && f.o[1] >= 0 && f.o[2] >= 0 && f.o[3] >= 0 && f.o[0] < ws && f.o[1] < ws &&
                           f.o[2] < ws && f.o[3] < ws && f.out >= 0 && f.out < (ND == 2 && isx ? xs : ys)))
                continue;  // check build only
            // normal and first tangential velocity: fields 1, 2 along x, 2, 1 along y
            const int fn = isx ? 1 : 2, ft = isx ? 2 : 1;
            double Lw[5], Rw[5], F[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const double *p = w + (k == 1 ? fn : k == 2 ? ft : k) * ws;
                double a0 = p[f.o[0]], a1 = p[f.o[1]], a2 = p[f.o[2]], a3 = p[f.o[3]];
                if (ND == 2 && k == 1 && (f.flags & 15)) {
                    if (f.flags & 1) a0 = -a0;
                    if (f.flags & 2) a1 = -a1;
                    if (f.flags & 4) a2 = -a2;
                    if (f.flags & 8) a3 = -a3;
                }
                const double d = a2 - a1;
                Lw[k] = face_val(a1, 0.5, minmod<double>(a1 - a0, d));
                Rw[k] = face_val(a2, -0.5, minmod<double>(d, a3 - a2));
            }
            hllc_frame<false>(Lw, Rw, gamma, ig1, F);
            const bool rowface = ND == 1 || !(f.flags & 16);
            double *q = (rowface ? fy : fx) + f.out;
            const int qs = rowface ? ys : xs;
            const double ar = rowface ? g.area[ND - 1] : g.area[0];
#pragma unroll
            for (int k = 0; k < 5; ++k) q[(k == 1 ? fn : k == 2 ? ft : k) * qs] = ar * F[k];
        }
        __syncthreads();
    };
    // flux divergence of own cell (row lr, column x), in the reference's order
    const int lr0 = ND == 2 ? t / L : t;  // of the thread's first cell
    auto divergence = [&](int c, double acc[5]) {
        const int lr = c == t ? lr0 : ND == 2 ? c / L : c, x = ND == 2 ? c - lr * L : 0;
        const int cr = lo_class(ra + lr, NR, bcl == BC_PERIODIC);
        const int cx = ND == 2 ? lo_class(x, L, g.bc_lo[0] == BC_PERIODIC) : LO_BEFORE;
        const int i = lr * (L + 1) + x;
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const double yl = fy[c + f * ys], yh = fy[c + L + f * ys];
            double a = 0.0;
            if (cr == LO_BEFORE) a -= yl;
            if constexpr (ND == 2) {
                const double xl = fx[i + f * xs], xh = fx[i + 1 + f * xs];
                if (cx == LO_BEFORE) a -= xl;
                a += xh;
                if (cx == LO_SELF) a -= xl;
                a += yh;
                if (cr == LO_SELF) a -= yl;
                if (cx == LO_AFTER) a -= xl;
            } else {
                a += yh;
                if (cr == LO_SELF) a -= yl;
            }
            if (cr == LO_AFTER) a -= yl;
            acc[f] = a;
        }
    };

    double m[ND] = {};
    for (int c = t; c < own; c += T) {
        double u[5];
        if (!VB_DCHECK((int64_t)ra * L + c < g.ncell && c < us)) continue;  // check build only
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            u[f] = U[f * g.ncell + (int64_t)ra * L + c];
            u0[f * us + c] = u[f];
        }
        prim(u, c, wb[0], m, true);
    }
    if (C > 1) cl.sync();  // every block runs before its shared memory is written
    int par = 0;
    publish(m, par);
    double time = ctrl->t, dt = ctrl->dt, invV = ctrl->invV, invdt = 0.0;
    const double tend = ctrl->tfinal;
    long long step = ctrl->step;
    const long long limit = ctrl->step_limit;
    int active = ctrl->active, flags = 0;
    for (long long done = 0;; ++done) {
        barrier();
        invdt = warp_max((t & 31) < C ? slot[par][t & 31] : 0.0);
        // evolve!'s loop head (k_finalize_cfl); the same on every thread of
        // the cluster
        if (done == nsteps) break;
        active = 0;
        if (!(time < tend * (1.0 - 1e-12)) || step >= limit) break;
        double h = invdt == 0.0 ? (double)INFINITY : div64(g.cfl, invdt);
        h = fmin(h, tend - time);
        if (invdt != invdt || !(h < (double)INFINITY)) {
            flags = CTRL_F_NONFINITE;
            break;
        }
        active = 1;
        dt = h;
        invV = div64(dt, avol);
        // stage 1
        halo(wb[0]);
        faces(wb[0]);
        for (int c = t; c < own; c += T) {
            double acc[5], u[5];
            divergence(c, acc);
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                u[f] = u0[f * us + c] - invV * acc[f];
                uc[f * us + c] = u[f];
            }
            prim(u, c, wb[1], m, false);
        }
        barrier();
        // stage 2
        halo(wb[1]);
        faces(wb[1]);
#pragma unroll
        for (int d = 0; d < ND; ++d) m[d] = 0.0;
        for (int c = t; c < own; c += T) {
            double acc[5], u[5];
            divergence(c, acc);
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                u[f] = 0.5 * u0[f * us + c] + 0.5 * (uc[f * us + c] - invV * acc[f]);
                u0[f * us + c] = u[f];
            }
            prim(u, c, wb[0], m, true);
        }
        par ^= 1;
        publish(m, par);
        time = time + dt;
        step = step + 1;
    }
    for (int c = t; c < own && VB_DCHECK((int64_t)ra * L + c < g.ncell); c += T)
#pragma unroll
        for (int f = 0; f < 5; ++f) U[f * g.ncell + (int64_t)ra * L + c] = u0[f * us + c];
    if (rank == 0 && t == 0) {
        ctrl->t = time;
        ctrl->dt = dt;
        ctrl->invV = invV;
        ctrl->step = step;
        ctrl->active = active;
        ctrl->flags |= flags;
        ctrl->invdt_bits = order_bits(invdt);
    }
    if (C > 1) cl.sync();  // no block leaves while another reads its shared memory
}

// the opt-ins of k_march on the current device
template <int ND>
bool opted()
{
    static PerDevice set;
    return set.get([] {
        cudaError_t e = cudaFuncSetAttribute(k_march<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)MARCH_SMEM);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_march<ND>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return e == cudaSuccess ? 1 : -1;
    }) > 0;
}

// f(configuration) of the plan's launch
template <typename F>
cudaError_t configured(const MarchPlan &p, cudaStream_t s, F &&f)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.blocks);
    cfg.blockDim = dim3((unsigned)p.threads);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)p.blocks;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return f(cfg);
}

template <int ND>
bool fits(const MarchPlan &p)
{
    int n = 0;
    const bool ok = opted<ND>() && configured(p, nullptr, [&](const cudaLaunchConfig_t &cfg) {
                        return cudaOccupancyMaxActiveClusters(&n, k_march<ND>, &cfg);
                    }) == cudaSuccess;
    cudaGetLastError();
    return ok && n > 0;
}

template <int ND>
int go(const Geom &g, const MarchPlan &p, double *U, Ctrl *ctrl, int64_t nsteps, cudaStream_t s)
{
    if (!opted<ND>()) return -1;
    return configured(p, s, [&](const cudaLaunchConfig_t &cfg) {
               return cudaLaunchKernelEx(&cfg, k_march<ND>, g, U, ctrl, (long long)nsteps, p.rows);
           }) == cudaSuccess ? 1 : -1;
}

}  // namespace

bool march_supported(const Geom &g)
{
    MarchPlan p;
    return march_plan(g, &p) && (g.nd == 1 ? fits<1>(p) : fits<2>(p));
}

int launch_march(const Geom &g, double *U, Ctrl *ctrl, int64_t nsteps, cudaStream_t s)
{
    MarchPlan p;
    if (!march_plan(g, &p) || nsteps < 0) return -1;
    return g.nd == 1 ? go<1>(g, p, U, ctrl, nsteps, s) : go<2>(g, p, U, ctrl, nsteps, s);
}

}  // namespace vb
