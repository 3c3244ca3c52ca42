// vb_stage_tiled3d_f64.cuh -- VB_FP64 tiled 3D stage kernel.
//
// A block of 12 warps owns a 16 x 16 column tile of any 3D grid with nx, ny >=
// 16 and marches it along z.  When a side is no multiple of 16 the last tile
// is shifted back inside the grid; cells it shares with the tile before it
// are computed and not written.  Warps 0..7 are one thread per column, warps
// 8..11 one thread per halo cell of the plane (4 strips of 32).
//
// Primitives live in a ring of three planes in shared memory; beyond a wall a
// halo thread fetches the mirror cell.  Raw conserved values arrive in the slot
// itself (8-byte cp.async, each element fetched by the thread that converts it
// in place, so no alignment of the rows is needed and no thread waits for
// another's copy).
// One barrier per plane separates iterations; iteration k
//   - solves the x and y faces of plane k+1 into one of two flux buffers: 17
//     warp tasks (8 of x, 8 of y, one of both hi edges), one on each column
//     warp and two or three on each halo warp, all through one body with the
//     states in the face-normal frame;
//   - converts plane k+2 and solves the z face k+1/2 down the column;
//   - updates plane k from the fluxes of the last iteration.
// Iteration k0-1 is the prologue: the same code without the update.
//
// Every operation is the reference's, rounded separately (-fmad=false), in the
// reference's per-cell accumulation order, so the result is bit-identical to
// the cell-centric kernel and to the oracle.
//
// What bounds it: issue slots and dependency waits of 24 warps per SM (2050
// instructions a cell and stage, 61 % of the issue slots, the float64 pipe 43 %
// busy; its floor at 256^3 would be 1.5 ms a step).  256^3: 3.63 -> 3.05 ms a
// step against 8 warps of 128 registers with two barriers a plane; 150 x 90 x
// 75, which the cell-centric kernel ran: 0.68 -> 0.28 ms.  Divisions without
// range branches (hllc_frame) spill at 80 registers: 3.1-3.35 ms.
#pragma once

#include "vb_stage_tiled3d_mixed.cuh"

namespace vb {

namespace t3d {

using t3::NH;
using t3::TX;
using t3::TY;
using t3m::PC;
using t3m::PSLOT;
using t3m::wrow;
using t3m::wxs;

constexpr int NC = TX * TY;           // column threads (one per cell of a plane)
constexpr int NTH = NC + NH;          // and one thread per halo cell
constexpr int FX = TY * (TX + 1);     // x faces of a plane
constexpr int FY = (TY + 1) * TX;     // y faces

struct Smem {
    double w[3][PSLOT];          // plane ring (t3m layout): raw state, then primitives in place
    double g[2][5 * (FX + FY)];  // area * flux of a plane: [5][FX] of x, then [5][FY] of y
    double hz[5][NC];            // hi z face value of the plane in work, per column
    double fz[5][NC];            // area * flux through its lower z face
};

// face_val(w, h, minmod(a, b))
__device__ __forceinline__ double face_mm(double w, double h, double a, double b)
{
    return face_val(w, h, minmod<double>(a, b));
}

// cfl_bound keeps its digits above this maximum, with widths whose inverses are
// normal float32 numbers
constexpr float CFL_FLOOR = 1e-30f;
__device__ __forceinline__ bool cfl_widths(const Geom &g)
{
    return g.invw[0] > 1.2e-38 && g.invw[1] > 1.2e-38 && (g.nd < 3 || g.invw[2] > 1.2e-38);
}

// An upper bound, in float32, of the cell's compute_dt term max_d (|v_d| + c) /
// w_d (and of the free-fall rate, GRAV).  Relative slack 4e-6 on the pressure
// (measured against E + kinetic, which its difference cancels; with what the
// squares may lose below the normal numbers) and on the result covers the
// float32 roundings.  Operands out of float32's normal range, and any negative
// density or pressure, come out NaN or Inf, which asks for the exact term: above
// p c = 1e-30 the pressure has all its digits (the reciprocal of a density below
// the normal range is Inf).
template <bool GRAV>
__device__ __forceinline__ float cfl_bound(const double un[5], const Geom &g, float gf, float iw0,
                                           float iw1, float iw2)
{
    const float rho = (float)un[0], ir = rcp_approx(rho), E = (float)un[4];
    const float vx = (float)un[1] * ir, vy = (float)un[2] * ir, vz = (float)un[3] * ir;
    const float ke = 0.5f * rho * (vx * vx + vy * vy + vz * vz);
    const float p = (gf - 1.0f) * (E - ke) + 4e-6f * (fabsf(E) + fmaf(1.2e-38f, rho, ke));
    const float c = sqrt_approx(gf * p * ir);
    float b = fmaxf(fmaxf((fabsf(vx) + c) * iw0, (fabsf(vy) + c) * iw1), (fabsf(vz) + c) * iw2);
    if (!(p * c > 1e-30f)) b = __int_as_float(0x7fc00000);  // NaN operands too, which fmaxf drops
    if constexpr (GRAV) {
        const float q = 12.566371f * (float)g.grav_G * rho;
        const float f = q > 1e-30f || g.grav_G == 0.0 ? 2.0f * sqrt_approx(q) : __int_as_float(0x7fc00000);
        if (!(f <= b)) b = f;
    }
    return b * (1.0f + 4e-6f);
}

}  // namespace t3d

template <int STAGE, bool BATCH, bool GRAV = false, bool BF = false>
__global__ void __launch_bounds__(t3d::NTH, 2)
k_stage_tiled3d_f64(const __grid_constant__ BoxDesc box0, const BoxDesc *__restrict__ boxes,
                    const int *__restrict__ item_box, int nitems, unsigned int *work)
{
    using namespace t3d;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    t3d::Smem &S = *reinterpret_cast<t3d::Smem *>(smem_raw);
    __shared__ double red[32];
    __shared__ int item_sh;
    // float bits: a lower bound of the item's CFL maximum so far; -1: none above
    // CFL_FLOOR, NaN: every cell takes the exact term
    __shared__ int cfl_sh;

    const int t = threadIdx.x;
    const bool col = t < NC;  // column thread, else halo thread
    const int tx = t & (TX - 1), ty = (t >> 4) & (TY - 1);
    // ring offset of the element this thread fetches and converts
    const int h = t - NC;  // halo thread: strip cell
    const int o_c = col      ? wrow(tx, ty)
                    : h < 32 ? wxs(-2 + (h & 1), h >> 1)
                    : h < 64 ? wxs(TX + (h & 1), (h - 32) >> 1)
                    : h < 96 ? wrow((h - 64) & 15, -2 + ((h - 64) >> 4))
                             : wrow((h - 96) & 15, TY + ((h - 96) >> 4));
    // its cell relative to the tile's corner
    const int dx = col      ? tx
                   : h < 32 ? -2 + (h & 1)
                   : h < 64 ? TX + (h & 1)
                            : (h & 15);
    const int dy = col      ? ty
                   : h < 64 ? (h & 31) >> 1
                   : h < 96 ? -2 + ((h - 64) >> 4)
                            : TY + ((h - 96) >> 4);
    // face tasks: column warps the own lo x face; halo warp i the lo y faces of
    // rows 4 i .. 4 i + 3 (two tasks), the last one also the hi-edge faces
    const int ntask = col ? 1 : (t < NTH - 32 ? 2 : 3);
    const int fr = col ? ty : 4 * (h >> 5) + ((h >> 4) & 1);  // row of the first task
    const int f_c = wrow(tx, fr);

    for (;;) {
    if (t == 0) item_sh = (int)atomicAdd(&work[STAGE - 1], 1u);
    __syncthreads();
    const int item = item_sh;
    if (item >= nitems) break;
    const BoxDesc &B = box_of<BATCH>(box0, boxes, item_box, item);
    Ctrl *ctrl = B.ctrl;
    if (!ctrl->active) {  // uniform: the box is not stepping
        __syncthreads();  // everyone has read item_sh before thread 0 rewrites it
        continue;
    }
    const Geom &g = B.g;
    const double *__restrict__ Uin = STAGE == 1 ? B.U : B.U1;
    const double *U0 = B.U;
    double *Uout = STAGE == 1 ? B.U1 : B.U;
    const int nx = (int)g.n[0], ny = (int)g.n[1], nz = (int)g.n[2];
    const bool perx = g.bc_lo[0] == BC_PERIODIC, pery = g.bc_lo[1] == BC_PERIODIC;
    const bool perz = g.bc_lo[2] == BC_PERIODIC;
    const double gamma = g.gamma;
    const double bscale = BF ? 0.5 * ctrl->dt : 0.0;  // boundary-flux stage weight
    if (STAGE == 2 && t == 0) cfl_sh = cfl_widths(g) ? __float_as_int(-1.0f) : 0x7fc00000;
    const int local = item - B.item0;
    const int tile = local % B.ntiles;
    // the last tile of a side that is no multiple of 16 is shifted back; the
    // cells left of (below) the nominal corner belong to the tile before it
    const int xn = (tile % B.ntx) * TX, yn = (tile / B.ntx) * TY;
    const int x0 = min(xn, nx - TX), y0 = min(yn, ny - TY);
    int k0, k1;
    chunk_span(nz, B.kz, B.nchu, local / B.ntiles, k0, k1);
    const int64_t plane = (int64_t)nx * ny;
    // this thread's element: its column in the state.  Beyond the grid that is
    // the wrapped cell on a periodic axis, else the mirror cell, whose normal
    // velocity (field `flip`) a reflecting wall negates (ghost_state)
    int ex = x0 + dx, ey = y0 + dy, flip = 0;
    if (!col) {
        auto mirror = [&](int &c, int n, bool per, int bl, int bh, int nrm) {
            if (c < 0) {
                if (!per && bl == BC_REFLECTING) flip = nrm;
                c = per ? c + n : -1 - c;
            } else if (c >= n) {
                if (!per && bh == BC_REFLECTING) flip = nrm;
                c = per ? c - n : 2 * n - 1 - c;
            }
        };
        mirror(ex, nx, perx, g.bc_lo[0], g.bc_hi[0], 1);
        mirror(ey, ny, pery, g.bc_lo[1], g.bc_hi[1], 2);
    }
    const int64_t ecol = (int64_t)ex + (int64_t)nx * ey;
    const bool own = col && ex >= xn && ey >= yn;  // this thread updates its column
    double cflm = 0.0;

    // cp.async of plane p's element into ring slot ws (periodic planes wrap;
    // planes beyond a wall are left out, the z face formulas do not read them)
    auto fetch_plane = [&](int p, double *ws) {
        int z = p;
        if (perz) {
            z = p < 0 ? p + nz : (p >= nz ? p - nz : p);
            if (z < 0 || z >= nz) z = ((p % nz) + nz) % nz;  // nz < 3 only
        }
        if (z >= 0 && z < nz) {
            const double *src = Uin + ecol + plane * z;
            if (VB_DCHECK(ecol >= 0 && ecol < plane))
#pragma unroll
                for (int f = 0; f < 5; ++f) cp_async8(ws + o_c + f * PC, src + f * g.ncell);
        }
    };
    // in-place conversion of this thread's element of a landed plane
    auto convert = [&](double *ws, double W[5]) {
        double u[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) u[f] = ws[o_c + f * PC];
        cons2prim(u, gamma, W);
        if (flip == 1) W[1] = -W[1];
        if (flip == 2) W[2] = -W[2];
#pragma unroll
        for (int f = 0; f < 5; ++f) ws[o_c + f * PC] = W[f];
    };

    // ring slots of planes k, k+1, k+2 at the loop's start (k = k0 - 1)
    double *r0 = S.w[0], *r1 = S.w[1], *r2 = S.w[2];
    // plane k0-2 passes through slot r2 on its way to the column's hi z face
    // value of plane k0-1
    const bool gl = !perz && k0 == 0;  // the chunk's lower z face is a wall
    if (col) {
        if (!gl) {
            fetch_plane(k0 - 2, r2);
            fetch_plane(k0 - 1, r0);
        }
    }
    fetch_plane(k0, r1);
    cp_async_commit();
    cp_async_wait_all();
    {
        double Wa[5], Wb[5], Wc[5];
        convert(r1, Wc);
        if (col && !gl) {
            const bool gll = !perz && k0 - 2 < 0;
            if (!gll) {
                double u[5];
#pragma unroll
                for (int f = 0; f < 5; ++f) u[f] = r2[o_c + f * PC];
                cons2prim(u, gamma, Wa);
            }
            {
                double u[5];
#pragma unroll
                for (int f = 0; f < 5; ++f) u[f] = r0[o_c + f * PC];
                cons2prim(u, gamma, Wb);
            }
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                r0[o_c + f * PC] = Wb[f];
                const double wl = gll ? ((g.bc_lo[2] == BC_REFLECTING && f == 3) ? -Wb[f] : Wb[f]) : Wa[f];
                S.hz[f][t] = face_val(Wb[f], 0.5, limited_slope<double>(wl, Wb[f], Wc[f]));
            }
        }
    }
    if (col || k0 + 1 < k1) fetch_plane(k0 + 1, r2);
    cp_async_commit();
    __syncthreads();

    const int cx = lo_class(ex, nx, perx), cy = lo_class(ey, ny, pery);
    const float gf = (float)gamma;
    const float iw0 = (float)g.invw[0], iw1 = (float)g.invw[1], iw2 = (float)g.invw[2];

    for (int k = k0 - 1; k < k1; ++k) {
        // warm L1 for the update's own-cell loads (a 16-cell row spans at most
        // two 128-byte lines)
        if (STAGE == 2 && col && k >= k0 && (tx == 0 || tx == TX - 1)) {
            const int64_t l = ecol + plane * k;
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                prefetch_l1(Uin + l + f * g.ncell);
            }
        }
        // halo elements of plane k are free (its faces are solved): fetch k+3's
        if (!col) {
            if (k + 3 < k1) fetch_plane(k + 3, r0);
            cp_async_commit();
        }
        // ---- x and y faces of plane k+1 ----
        if (k + 1 < k1) {
            double *gw = S.g[(k + 1) & 1];
            const double *w1 = r1;
            const double ax = g.area[0], ay = g.area[1];
            for (int it = 0; it < ntask; ++it) {
                // the four cells across the face; x: cells tx-2 .. tx+1, y: rows
                int o0, o1, o2, o3, out;
                bool isy;
                if (it < 2) {
                    isy = !col;
                    const int c = f_c + 32 * it;  // the second task is two rows up
                    if (isy) {
                        o0 = c - 32; o1 = c - 16; o2 = c; o3 = c + 16;
                        out = 5 * FX + (fr + 2 * it) * TX + tx;
                    } else {
                        o0 = tx >= 2 ? c - 2 : wxs(tx - 2, fr);
                        o1 = tx >= 1 ? c - 1 : wxs(-1, fr);
                        o2 = c;
                        o3 = tx <= TX - 2 ? c + 1 : wxs(TX, fr);
                        out = fr * (TX + 1) + tx;
                    }
                } else {  // hi edges: lanes 0..15 of x (row tx), 16..31 of y (column tx)
                    isy = (t & 16) != 0;
                    if (isy) {
                        o2 = wrow(tx, TY);
                        o0 = o2 - 32; o1 = o2 - 16; o3 = o2 + 16;
                        out = 5 * FX + TY * TX + tx;
                    } else {
                        o1 = wrow(TX - 1, tx);
                        o0 = o1 - 1; o2 = wxs(TX, tx); o3 = wxs(TX + 1, tx);
                        out = tx * (TX + 1) + TX;
                    }
                }
                // normal and first tangential velocity are fields 1, 2 (x) or 2, 1 (y)
                const int fn = isy ? 2 * PC : PC, ft = isy ? PC : 2 * PC;
                double L[5], R[5], F[5];
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    const double *p = w1 + (f == 1 ? fn : f == 2 ? ft : f * PC);
                    const double a0 = p[o0], a1 = p[o1], a2 = p[o2], a3 = p[o3];
                    const double d = a2 - a1;
                    L[f] = face_mm(a1, 0.5, a1 - a0, d);
                    R[f] = face_mm(a2, -0.5, d, a3 - a2);
                }
                hllc_frame_any<false>(L, R, gamma, F);
                const int os = isy ? FY : FX;
                const double ar = isy ? ay : ax;
                double *o = gw + out;
                o[0] = ar * F[0];
                o[(isy ? 2 : 1) * os] = ar * F[1];
                o[(isy ? 1 : 2) * os] = ar * F[2];
                o[3 * os] = ar * F[3];
                o[4 * os] = ar * F[4];
                if constexpr (BF) {  // domain faces of cells this tile updates
                    const double Fd[5] = {F[0], isy ? F[2] : F[1], isy ? F[1] : F[2], F[3], F[4]};
                    const int kk = k + 1;
                    if (!isy) {
                        const int fy = y0 + (it < 2 ? fr : tx), side = it < 2 ? 0 : 1;
                        if (fy >= yn && !perx && (side ? x0 + TX == nx : x0 + tx == 0))
                            bflux_add(g, B.bflux, 0, side, (int64_t)fy + (int64_t)ny * kk, bscale, ax, Fd);
                    } else {
                        const int fx = x0 + tx, side = it < 2 ? 0 : 1;
                        if (fx >= xn && !pery && (side ? y0 + TY == ny : y0 + fr + 2 * it == 0))
                            bflux_add(g, B.bflux, 1, side, (int64_t)fx + (int64_t)nx * kk, bscale, ay, Fd);
                    }
                }
            }
        }
        if (!col) {
            cp_async_wait_group<1>();  // plane k+2's element (k+3's is in flight)
            double W[5];
            if (k + 2 < k1) convert(r2, W);
        } else {
            // ---- plane k+2 of the column, and the z face k+1/2 ----
            cp_async_wait_all();
            const bool below = perz || k >= 0;       // plane k exists
            const bool above = perz || k + 1 < nz;   // plane k+1 exists
            const bool top = !perz && k + 2 >= nz;   // plane k+2 does not
            double zl[5], zr[5], F[5];
            {
                double W2[5];
                if (!top) convert(r2, W2);
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    zl[f] = S.hz[f][t];
                    if (above) {
                        const double c = r1[o_c + f * PC];
                        const double lo = below ? r0[o_c + f * PC]
                                                : ((g.bc_lo[2] == BC_REFLECTING && f == 3) ? -c : c);
                        const double hi = top ? ((g.bc_hi[2] == BC_REFLECTING && f == 3) ? -c : c) : W2[f];
                        zr[f] = face_mm(c, -0.5, c - lo, hi - c);
                        S.hz[f][t] = face_mm(c, 0.5, c - lo, hi - c);
                    }
                }
                if (!above) ghost_state<double>(zl, g.bc_hi[2], 2, zr);
                if (!below) ghost_state<double>(zr, g.bc_lo[2], 2, zl);
            }
            // the column's entries of plane k have been read: until plane k+3
            // lands there they hold the update's input (U^n in stage 2)
            const bool write = own && k >= k0;
            const int64_t lin = ecol + plane * k;
            const bool inb = write && VB_DCHECK(lin >= 0 && lin < g.ncell);  // check build only
            if (inb)
#pragma unroll
                for (int f = 0; f < 5; ++f)
                    cp_async8(r0 + o_c + f * PC, (STAGE == 1 ? Uin : U0) + lin + f * g.ncell);
            cp_async_commit();
            {
                const double L[5] = {zl[0], zl[3], zl[1], zl[2], zl[4]};
                const double R[5] = {zr[0], zr[3], zr[1], zr[2], zr[4]};
                hllc_frame_any<true>(L, R, gamma, F);
            }
            const double Fz[5] = {F[0], F[2], F[3], F[1], F[4]};
            if constexpr (BF) {
                if (own && (!below || !above))
                    bflux_add(g, B.bflux, 2, below ? 1 : 0, ecol, bscale, g.area[2], Fz);
            }
            // ---- flux divergence in the reference's order, then the update ----
            const double az = g.area[2];
            const int cz = (k == g.zw0 && g.zcls0 >= 0) ? g.zcls0 : lo_class(k, nz, perz);
            const bool interior = cx == LO_BEFORE && cy == LO_BEFORE && cz == LO_BEFORE;
            const double invV = ctrl->invV;
            const double *gr = S.g[k & 1] + ty * (TX + 1) + tx;
            const double *gq = S.g[k & 1] + 5 * FX + ty * TX + tx;
            double un[5], acc[5];
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const double gzh = az * Fz[f], gzl = S.fz[f][t];
                S.fz[f][t] = gzh;
                const double gxl = gr[f * FX], gxh = gr[f * FX + 1];
                const double gyl = gq[f * FY], gyh = gq[f * FY + TX];
                double a = 0.0;
                if (interior) {
                    a = a - gzl - gyl - gxl + gxh + gyh + gzh;
                } else {
                    if (cz == LO_BEFORE) a -= gzl;
                    if (cy == LO_BEFORE) a -= gyl;
                    if (cx == LO_BEFORE) a -= gxl;
                    a += gxh;
                    if (cx == LO_SELF) a -= gxl;
                    a += gyh;
                    if (cy == LO_SELF) a -= gyl;
                    a += gzh;
                    if (cz == LO_SELF) a -= gzl;
                    if (cx == LO_AFTER) a -= gxl;
                    if (cy == LO_AFTER) a -= gyl;
                    if (cz == LO_AFTER) a -= gzl;
                }
                acc[f] = a;
            }
            cp_async_wait_all();
            if (inb) {
                if constexpr (GRAV) {  // the source from the stage state, after the fluxes
                    double u[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f)
                        u[f] = STAGE == 1 ? r0[o_c + f * PC] : __ldg(Uin + lin + f * g.ncell);
                    gravity_source<3>(g, lin, u, acc);
                }
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    const double ep = r0[o_c + f * PC];
                    if constexpr (STAGE == 1) un[f] = ep - invV * acc[f];
                    else un[f] = 0.5 * ep + 0.5 * (__ldg(Uin + lin + f * g.ncell) - invV * acc[f]);
                    Uout[lin + f * g.ncell] = un[f];
                }
                if constexpr (STAGE == 2) {
                    // the exact CFL term only of cells whose bound exceeds the
                    // item's maximum so far (the slab's own planes)
                    if (k >= g.zw0 && k < g.zw1) {
                        const float b = cfl_bound<GRAV>(un, g, gf, iw0, iw1, iw2);
                        if (!(b <= __int_as_float(*(volatile int *)&cfl_sh))) {
                            cflm = cfl_term_exact<GRAV>(un, g, cflm);
                            const float m = __double2float_rd(cflm);
                            if (m > CFL_FLOOR) atomicMax(&cfl_sh, __float_as_int(m));
                        }
                    }
                }
            }
            if (k + 3 <= k1 + 1) fetch_plane(k + 3, r0);
            cp_async_commit();
        }
        __syncthreads();  // faces of plane k+1 and primitives of plane k+2 are ready
        double *rt = r0;
        r0 = r1;
        r1 = r2;
        r2 = rt;
    }
    cp_async_wait_all();
    if constexpr (STAGE == 2) block_max_to(&ctrl->invdt_bits, cflm, red);  // this box's CFL max
    }  // work items
}

// Boxes the kernel takes: 16 x 16 tiles, the last one shifted back.
inline int launch_tiled3d_f64(const BoxDesc *hbox, const BoxDesc *boxes, const int *item_box,
                              int nitems, unsigned int *work, int stage, cudaStream_t s, bool grav,
                              bool bf)
{
    const size_t smem = sizeof(t3d::Smem);
    static PerDevice res1, resb, resg, resf;
    if ((grav || bf) && !hbox) return -1;  // gravity, boundary fluxes: single boxes only
    if (grav && bf) return -1;
    if (bf && !hbox->bflux) return -1;
    auto fits = [&](auto k1, auto k2) { return persistent_blocks(k1, k2, smem, t3d::NTH); };
    const int resident =
        grav   ? resg.get([&] { return fits(k_stage_tiled3d_f64<1, false, true>, k_stage_tiled3d_f64<2, false, true>); })
        : bf   ? resf.get([&] {
              return fits(k_stage_tiled3d_f64<1, false, false, true>, k_stage_tiled3d_f64<2, false, false, true>);
          })
        : hbox ? res1.get([&] { return fits(k_stage_tiled3d_f64<1, false>, k_stage_tiled3d_f64<2, false>); })
               : resb.get([&] { return fits(k_stage_tiled3d_f64<1, true>, k_stage_tiled3d_f64<2, true>); });
    if (resident <= 0 || nitems <= 0) return -1;
    const unsigned grid = (unsigned)(nitems < resident ? nitems : resident);
    BoxDesc box0;
    if (hbox) box0 = *hbox;
    else std::memset(&box0, 0, sizeof box0);
    auto go = [&](auto k1, auto k2, const BoxDesc *tab, const int *ib) {
        if (stage == 1) k1<<<grid, t3d::NTH, smem, s>>>(box0, tab, ib, nitems, work);
        else k2<<<grid, t3d::NTH, smem, s>>>(box0, tab, ib, nitems, work);
    };
    if (grav) go(k_stage_tiled3d_f64<1, false, true>, k_stage_tiled3d_f64<2, false, true>, nullptr, nullptr);
    else if (bf)
        go(k_stage_tiled3d_f64<1, false, false, true>, k_stage_tiled3d_f64<2, false, false, true>, nullptr, nullptr);
    else if (hbox) go(k_stage_tiled3d_f64<1, false>, k_stage_tiled3d_f64<2, false>, nullptr, nullptr);
    else go(k_stage_tiled3d_f64<1, true>, k_stage_tiled3d_f64<2, true>, boxes, item_box);
    return 1;
}

}  // namespace vb
