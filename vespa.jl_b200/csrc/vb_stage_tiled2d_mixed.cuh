// vb_stage_tiled2d_mixed.cuh -- VB_MIXED tiled 2D stage kernel: 256-cell row
// segments marching y (the plan of k_stage_tiled2d, its row loads by TMA and
// persistent queue) with the plane structure of k_stage_tiled3d_mixed.
//
// Float32 primitives live in a ring of two rows with the x halo (mirror ghosts
// at walls) beside them, so every thread rebuilds both states of its lo x face
// from the four cells across it.  Iteration r solves, as one packed HLLC, the x
// face of row r+1 and the y face r+1/2 of the thread's column, converts row
// r+2, and updates row r from the x fluxes of the last iteration: one barrier a
// row, where exchanging face values took three.
//
// The last segment of a row whose length is even and no multiple of 256 is
// shifted back inside the grid (its loads stay 16-byte aligned); cells it shares
// with the segment before it are not written.
//
// What bounds it: issue slots (24 warps per SM).  4096^2: 1.18 -> 0.92 ms a step,
// of which HBM takes 0.51.
#pragma once

#include "vb_hllc_x2.cuh"
#include "vb_stage_tiled2d.cuh"
#include "vb_stage_tiled3d_mixed.cuh"

namespace vb {

namespace t2m {

using t2::NT;
using t2::ROW_BYTES;
using t2::TX;
using t2::U_XHI;
using t2::U_XLO;
using t2::UROW;

constexpr int WR = TX + 4;  // a ring row: cells -2 .. TX + 1, cell c at c + 2

template <int NS>
struct Smem {
    alignas(128) double u[NS][UROW];  // TMA stage buffers (raw conserved state)
    double ep[2][5][NT];     // own-cell epilogue inputs (Uin, U0), fetched by cp.async
    float w[2][5][WR];       // primitive rows, by the row's parity within the chunk
    float gx[2][5][TX + 1];  // x-face fluxes of a row, by the same parity
    uint64_t bar[NS];
};

}  // namespace t2m

template <int NS, int STAGE, bool BF = false>
__global__ void __launch_bounds__(256, 3)
k_stage_tiled2d_mixed(const __grid_constant__ BoxDesc B, int nitems, unsigned int *work)
{
    using namespace t2m;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // check build only: TMA destinations need a 128-byte aligned base (uniform)
    if (!VB_DCHECK(((uintptr_t)smem_raw & 127) == 0)) return;
    t2m::Smem<NS> &S = *reinterpret_cast<t2m::Smem<NS> *>(smem_raw);
    __shared__ double red[32];
    __shared__ int item_sh;
    __shared__ int stall_sh;  // a stage load's bounded wait gave up
    const int t = threadIdx.x;

    if (t == 0) {
        for (int s = 0; s < NS; ++s) mbar_init(&S.bar[s], 1);
        fence_mbar_init();
        stall_sh = 0;
    }
    __syncthreads();

    const Geom &g = B.g;
    Ctrl *ctrl = B.ctrl;
    const CUtensorMap *tm = B.map[STAGE - 1];
    if (!VB_DCHECK(((uintptr_t)tm & 63) == 0)) return;  // check build only (uniform)
    const double *__restrict__ Uin = STAGE == 1 ? B.U : B.U1;
    const double *U0 = B.U;
    double *Uout = STAGE == 1 ? B.U1 : B.U;
    const int nx = (int)g.n[0], ny = (int)g.n[1];
    const bool perx = g.bc_lo[0] == BC_PERIODIC, pery = g.bc_lo[1] == BC_PERIODIC;
    const double gamma = g.gamma;
    const float gf = (float)gamma, ig1 = 1.0f / ((float)gamma - 1.0f);
    const double bscale = BF ? 0.5 * ctrl->dt : 0.0;  // boundary-flux stage weight
    auto ghostc = [](float w, int f, int bc, int axis) {
        return (bc == BC_REFLECTING && f == 1 + axis) ? -w : w;
    };

    int qb = 0;
    double invdt = 0.0;
    for (;;) {
    if (t == 0) item_sh = (int)atomicAdd(&work[STAGE - 1], 1u);
    __syncthreads();
    const int item = item_sh;
    if (item >= nitems) break;
    if (!ctrl->active) {  // uniform: the grid is not stepping
        __syncthreads();
        continue;
    }
    const int xn = (item % B.ntx) * TX, x0 = min(xn, nx - TX);
    const bool own = x0 + t >= xn;  // this thread updates its column
    const int r0 = (item / B.ntx) * B.kz, r1 = min(ny, r0 + B.kz);
    const int nrows = (r1 - r0) + 4;  // rows r0-2 .. r1+1
    const bool xlo_bnd = !perx && x0 == 0, xhi_bnd = !perx && x0 + TX == nx;
    const double invV = ctrl->invV;
    const double sx = __dmul_rn(invV, g.area[0]), sy = __dmul_rn(invV, g.area[1]);

    auto issue = [&](int q) {
        const int p = r0 - 2 + q;
        const int y = pery ? ((p % ny) + ny) % ny : p;  // out-of-range rows read the zero fill
        double *dst = S.u[(unsigned)(qb + q) % NS];
        uint64_t *bar = &S.bar[(unsigned)(qb + q) % NS];
        const int xl = (perx && x0 == 0) ? nx - 2 : x0 - 2;
        const int xh = (perx && x0 + TX == nx) ? 0 : x0 + TX;
        mbar_expect_tx(bar, ROW_BYTES);
        tma_load_4d(dst, &tm[0], x0, y, 0, 0, bar);
        tma_load_4d(dst + U_XLO, &tm[1], xl, y, 0, 0, bar);
        tma_load_4d(dst + U_XHI, &tm[1], xh, y, 0, 0, bar);
    };
    if (t == 0) {
        fence_proxy_async_smem();
        for (int q = 0; q < NS && q < nrows; ++q) issue(q);
    }
    // wait for staged row q and convert the own cell; keep: also into ring row
    // ws, with the halo cells (mirrored at a wall)
    auto consume = [&](int q, float W[5], bool keep, float (*ws)[WR]) {
        const int b = (unsigned)(qb + q) % NS;
        if (!mbar_wait(&S.bar[b], ((unsigned)(qb + q) / NS) & 1, WAIT_LIMIT_NS)) stall_sh = 1;
        const double *u = S.u[b];
        double uu[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) uu[f] = u[f * TX + t];
        t3m::cons2prim_mixed(uu, gamma, W);
        if (!keep) return;
#pragma unroll
        for (int f = 0; f < 5; ++f) ws[f][t + 2] = W[f];
        if (xlo_bnd && t < 2)
#pragma unroll
            for (int f = 0; f < 5; ++f) ws[f][1 - t] = ghostc(W[f], f, g.bc_lo[0], 0);
        if (xhi_bnd && t >= TX - 2)
#pragma unroll
            for (int f = 0; f < 5; ++f) ws[f][2 * TX + 1 - t] = ghostc(W[f], f, g.bc_hi[0], 0);
        // halo cells -2, -1, TX, TX+1 on four threads of a warp without an edge face
        const int h = t - 64;
        if (h >= 0 && h < 4 && !(h < 2 ? xlo_bnd : xhi_bnd)) {
            float w[5];
            const int base = h < 2 ? U_XLO + h : U_XHI + (h - 2);
#pragma unroll
            for (int f = 0; f < 5; ++f) uu[f] = u[base + 2 * f];
            t3m::cons2prim_mixed(uu, gamma, w);
#pragma unroll
            for (int f = 0; f < 5; ++f) ws[f][h < 2 ? h : TX + h] = w[f];
        }
    };
    auto release = [&](int q) {
        if (t == 0 && q + NS < nrows) {
            fence_proxy_async_smem();
            issue(q + NS);
        }
    };
    // after the barrier that follows consume(q): uniform across the block
    auto stalled = [&](int q) -> bool {
        if (!stall_sh) return false;
        stage_abandon<NS>(S.bar, qb, q, nrows, ctrl);
        return true;
    };
    // float32 states of x face i (between cells i-1 and i of the segment)
    auto x_states = [&](const float (*w)[WR], int i, float L[5], float R[5]) {
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const float *p = w[f] + i;
            const float a1 = p[1], a2 = p[2], d = a2 - a1;
            const float lo = fminf(0.f, d), hi = fmaxf(0.f, d);
            L[f] = fmaf(0.5f, fminf(fmaxf(a1 - p[0], lo), hi), a1);
            R[f] = fmaf(-0.5f, fminf(fmaxf(p[3] - a2, lo), hi), a2);
        }
    };
    auto capture = [&](int d, int side, int64_t idx, const float F[5]) {
        const double Fd[5] = {(double)F[0], (double)F[1], (double)F[2], (double)F[3], (double)F[4]};
        bflux_add(g, B.bflux, d, side, idx, bscale, g.area[d], Fd);
    };
    // x face t of row `row` (ring row w) and the y face (yl, yr) as one packed
    // solve; the segment's hi edge face by the last thread, through the x lane
    auto solve = [&](const float (*w)[WR], int row, bool xon, const float yl[5], const float yr[5],
                     float Fy[5]) {
        float L[5] = {1.f, 0.f, 0.f, 0.f, 1.f}, R[5] = {1.f, 0.f, 0.f, 0.f, 1.f};
        if (xon) x_states(w, t, L, R);
        // x face in (rho, vx, vy, vz, p), y face rotated to (rho, vy, vx, vz, p)
        const Face2 l{f2(L[0], yl[0]), f2(L[1], yl[2]), f2(L[2], yl[1]), f2(L[3], yl[3]), f2(L[4], yl[4])};
        const Face2 r{f2(R[0], yr[0]), f2(R[1], yr[2]), f2(R[2], yr[1]), f2(R[3], yr[3]), f2(R[4], yr[4])};
        f2 F[5];
        hllc_x2(l, r, gf, ig1, F);
        Fy[0] = F[0].v.y;
        Fy[1] = F[2].v.y;
        Fy[2] = F[1].v.y;
        Fy[3] = F[3].v.y;
        Fy[4] = F[4].v.y;
        if (!xon) return;
        float (*gx)[TX + 1] = S.gx[(row - r0) & 1];
#pragma unroll
        for (int f = 0; f < 5; ++f) gx[f][t] = F[f].v.x;
        if constexpr (BF) {
            const float Fx[5] = {F[0].v.x, F[1].v.x, F[2].v.x, F[3].v.x, F[4].v.x};
            if (own && t == 0 && xlo_bnd) capture(0, 0, row, Fx);
        }
        if (t == TX - 1) {
            float L2[5], R2[5];
            x_states(w, TX, L2, R2);
            const Face2 le{f2::splat(L2[0]), f2::splat(L2[1]), f2::splat(L2[2]), f2::splat(L2[3]), f2::splat(L2[4])};
            const Face2 re{f2::splat(R2[0]), f2::splat(R2[1]), f2::splat(R2[2]), f2::splat(R2[3]), f2::splat(R2[4])};
            hllc_x2(le, re, gf, ig1, F);
#pragma unroll
            for (int f = 0; f < 5; ++f) gx[f][TX] = F[f].v.x;
            if constexpr (BF) {
                const float Fx[5] = {F[0].v.x, F[1].v.x, F[2].v.x, F[3].v.x, F[4].v.x};
                if (xhi_bnd) capture(0, 1, row, Fx);
            }
        }
    };

    float Wa[5], Wb[5], Wy0[5], Wy1[5], Wy2[5];
    consume(0, Wa, false, nullptr);
    __syncthreads();
    if (stalled(0)) return;
    release(0);
    consume(1, Wb, false, nullptr);
    __syncthreads();
    if (stalled(1)) return;
    release(1);
    consume(2, Wy0, true, S.w[0]);
    __syncthreads();
    if (stalled(2)) return;
    release(2);
    consume(3, Wy1, true, S.w[1]);

    // y state entering row r0: hi face value of r0 and, with row r0's x faces,
    // the flux through r0-1/2
    float hy[5], Fylo[5];
    {
        const bool gl = !pery && r0 == 0;
        const bool gh = !pery && r0 + 1 >= ny;
        float loy[5], yl[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const float wl = gl ? ghostc(Wy0[f], f, g.bc_lo[1], 1) : Wb[f];
            const float wr = gh ? ghostc(Wy0[f], f, g.bc_hi[1], 1) : Wy1[f];
            const float s = t3m::mm(wl, Wy0[f], wr);
            hy[f] = face_val(Wy0[f], 0.5f, s);
            loy[f] = face_val(Wy0[f], -0.5f, s);
        }
        if (gl) {
            ghost_state<float>(loy, g.bc_lo[1], 1, yl);
        } else {
            const bool gll = !pery && r0 - 2 < 0;
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const float wl = gll ? ghostc(Wb[f], f, g.bc_lo[1], 1) : Wa[f];
                yl[f] = face_val(Wb[f], 0.5f, t3m::mm(wl, Wb[f], Wy0[f]));
            }
        }
        solve(S.w[0], r0, true, yl, loy, Fylo);
        if constexpr (BF) {
            if (own && gl) capture(1, 0, x0 + t, Fylo);  // y-lo domain face of cell (x, 0)
        }
    }
    __syncthreads();
    if (stalled(3)) return;
    release(3);

    double unp[5];
    for (int r = r0; r < r1; ++r) {
        const int q = r - r0 + 4, par = (r - r0) & 1;
        const int64_t lin = (int64_t)(x0 + t) + (int64_t)nx * r;
        const bool inb = own && VB_DCHECK(lin >= 0 && lin < g.ncell);  // check build only
        if (inb)
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                cp_async8(&S.ep[0][f][t], Uin + (int64_t)f * g.ncell + lin);
                if constexpr (STAGE == 2) cp_async8(&S.ep[1][f][t], U0 + (int64_t)f * g.ncell + lin);
            }
        cp_async_commit();
        // row r+2 into the ring slot of row r, whose x faces are solved
        consume(q, Wy2, r + 2 < r1, S.w[par]);
        if constexpr (STAGE == 2)
            if (r > r0 && own) invdt = t3m::cfl_term2d(unp, g, invdt);
        // ---- the y face r+1/2 down the own column, with row r+1's x face ----
        float yr[5], hy1[5], Fyhi[5];
        if (pery || r + 1 < ny) {
            const bool gh = !pery && r + 2 >= ny;
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                const float wr = gh ? ghostc(Wy1[f], f, g.bc_hi[1], 1) : Wy2[f];
                const float s = t3m::mm(Wy0[f], Wy1[f], wr);
                yr[f] = face_val(Wy1[f], -0.5f, s);
                hy1[f] = face_val(Wy1[f], 0.5f, s);
            }
        } else {
            ghost_state<float>(hy, g.bc_hi[1], 1, yr);
#pragma unroll
            for (int f = 0; f < 5; ++f) hy1[f] = hy[f];
        }
        solve(S.w[par ^ 1], r + 1, r + 1 < r1, hy, yr, Fyhi);
        if constexpr (BF) {
            if (own && !pery && r + 1 >= ny) capture(1, 1, x0 + t, Fyhi);  // y-hi face of (x, ny-1)
        }
        // ---- the stage update from row r's fluxes (float64 differences) ----
        const float (*gx)[TX + 1] = S.gx[par];
        double un[5];
        cp_async_wait_all();
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const double dx = (double)gx[f][t + 1] - (double)gx[f][t];
            const double dy = (double)Fyhi[f] - (double)Fylo[f];
            const double u = __fma_rn(-sy, dy, __fma_rn(-sx, dx, S.ep[0][f][t]));
            un[f] = STAGE == 1 ? u : __dmul_rn(0.5, __dadd_rn(S.ep[1][f][t], u));
            if (inb) Uout[(int64_t)f * g.ncell + lin] = un[f];
            Fylo[f] = Fyhi[f];
            hy[f] = hy1[f];
            Wy0[f] = Wy1[f];
            Wy1[f] = Wy2[f];
        }
        if constexpr (STAGE == 2) {
#pragma unroll
            for (int f = 0; f < 5; ++f) unp[f] = un[f];
        }
        __syncthreads();  // row r+2 converted, x faces of row r+1 solved, those of r read
        if (stalled(q)) return;
        release(q);
    }
    if constexpr (STAGE == 2)
        if (own) invdt = t3m::cfl_term2d(unp, g, invdt);  // the item's last row
    qb += nrows;
    }  // work items
    if constexpr (STAGE == 2) block_max_to(&ctrl->invdt_bits, invdt, red);
}

template <int NS>
int launch_tiled2d_mixed(const BoxDesc *hbox, int nitems, unsigned int *work, int stage,
                         cudaStream_t s, bool bf)
{
    if (!hbox || nitems <= 0 || (bf && !hbox->bflux)) return -1;
    const size_t smem = sizeof(t2m::Smem<NS>);
    static PerDevice res, resf;
    const int resident =
        bf ? resf.get([&] {
            return persistent_blocks(k_stage_tiled2d_mixed<NS, 1, true>, k_stage_tiled2d_mixed<NS, 2, true>, smem);
        })
           : res.get([&] { return persistent_blocks(k_stage_tiled2d_mixed<NS, 1>, k_stage_tiled2d_mixed<NS, 2>, smem); });
    if (resident <= 0) return -1;
    const unsigned grid = (unsigned)(nitems < resident ? nitems : resident);
    auto k = bf ? (stage == 1 ? k_stage_tiled2d_mixed<NS, 1, true> : k_stage_tiled2d_mixed<NS, 2, true>)
                : (stage == 1 ? k_stage_tiled2d_mixed<NS, 1> : k_stage_tiled2d_mixed<NS, 2>);
    k<<<grid, 256, smem, s>>>(*hbox, nitems, work);
    return 1;
}

}  // namespace vb
