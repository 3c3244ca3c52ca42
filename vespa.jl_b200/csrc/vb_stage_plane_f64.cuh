// vb_stage_plane_f64.cuh -- VB_FP64 stage kernel of 2D grids of any size from
// 16 x 16: one block of 9 warps per 16 x 16 tile, no marching.
//
// The counterpart of k_stage_tiled3d_f64 for a single plane (tile geometry,
// shifted last tiles, mirrored or wrapped halo cells, face tasks in the
// face-normal frame: see that file).  Warps 0..7 hold one cell per thread and
// keep its state in registers for the update, the halo cells are converted by
// warp 8 and, as second cells, warps 0..2; after the conversion 17 warp tasks (8
// of x faces, 8 of y, one of both hi edges) are dealt to the 9 warps in two
// rounds.  Against the row-marching kernel a tile loads 1.5 times its cells, but
// every tile runs at once, 27 warps an SM instead of 16, and no thread waits for
// a row: 136 against 170 ps a cell and step at 1024 x 2048, 134 against 158 at
// 2048^2, 132 against 143 at 4096^2.  What bounds it: dependency waits, the
// tile's loads and the two barriers (issue slots 59 % used).
//
// Same operations, roundings and accumulation order as the cell-centric
// kernel: bit-identical to it.
#pragma once

#include "vb_stage_tiled3d_f64.cuh"

namespace vb {

namespace t3d {

constexpr int NTP = 288;

struct PlaneSmem {
    double w[PSLOT];           // primitives (t3m layout)
    double g[5 * (FX + FY)];   // area * flux: [5][FX] of x, then [5][FY] of y
};

}  // namespace t3d

template <int STAGE, int OCC>
__global__ void __launch_bounds__(t3d::NTP, OCC)
k_stage_plane_f64(const __grid_constant__ Geom g, const double *__restrict__ Uin, const double *U0,
                  double *Uout, Ctrl *ctrl, int ntx)
{
    using namespace t3d;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    PlaneSmem &S = *reinterpret_cast<PlaneSmem *>(smem_raw);
    __shared__ double red[32];
    if (!ctrl->active) return;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const bool col = t < NC;
    const int tx = t & (TX - 1), ty = (t >> 4) & (TY - 1);
    const int nx = (int)g.n[0], ny = (int)g.n[1];
    const bool perx = g.bc_lo[0] == BC_PERIODIC, pery = g.bc_lo[1] == BC_PERIODIC;
    const double gamma = g.gamma;
    const int xn = (int)(blockIdx.x % ntx) * TX, yn = (int)(blockIdx.x / ntx) * TY;
    const int x0 = min(xn, nx - TX), y0 = min(yn, ny - TY);
    // halo cells: 0..31 on the ninth warp, the others as second cells of warps 0..2
    const int h = col ? t + 32 : t - NC;
    int64_t hlin = 0;
    int o_h = 0, flip = 0;
    if (h < NH) {
        o_h = h < 32   ? wxs(-2 + (h & 1), h >> 1)
              : h < 64 ? wxs(TX + (h & 1), (h - 32) >> 1)
              : h < 96 ? wrow((h - 64) & 15, -2 + ((h - 64) >> 4))
                       : wrow((h - 96) & 15, TY + ((h - 96) >> 4));
        int hx = x0 + (h < 32 ? -2 + (h & 1) : h < 64 ? TX + (h & 1) : (h & 15));
        int hy = y0 + (h < 64 ? (h & 31) >> 1 : h < 96 ? -2 + ((h - 64) >> 4) : TY + ((h - 96) >> 4));
        auto mirror = [&](int &c, int n, bool per, int bl, int bh, int nrm) {
            if (c < 0) {
                if (!per && bl == BC_REFLECTING) flip = nrm;
                c = per ? c + n : -1 - c;
            } else if (c >= n) {
                if (!per && bh == BC_REFLECTING) flip = nrm;
                c = per ? c - n : 2 * n - 1 - c;
            }
        };
        mirror(hx, nx, perx, g.bc_lo[0], g.bc_hi[0], 1);
        mirror(hy, ny, pery, g.bc_lo[1], g.bc_hi[1], 2);
        hlin = hx + (int64_t)nx * hy;
    }
    const int ex = x0 + tx, ey = y0 + ty;
    const int64_t lin = ex + (int64_t)nx * ey;
    const bool own = col && ex >= xn && ey >= yn && VB_DCHECK(lin >= 0 && lin < g.ncell);
    // the grid's CFL maximum so far: a lower bound of the final one (-1: none)
    float sofar = 0.0f;
    if constexpr (STAGE == 2) {
        sofar = __double2float_rd(__longlong_as_double((long long)__ldcg(&ctrl->invdt_bits)));
        if (!(sofar > CFL_FLOOR) || !cfl_widths(g)) sofar = -1.0f;
    }
    double u[5], v[5], uh[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) u[f] = col ? __ldg(Uin + lin + f * g.ncell) : 0.0;
    if (h < NH)
#pragma unroll
        for (int f = 0; f < 5; ++f) uh[f] = __ldg(Uin + hlin + f * g.ncell);
    if constexpr (STAGE == 2)
#pragma unroll
        for (int f = 0; f < 5; ++f) v[f] = own ? U0[lin + f * g.ncell] : 0.0;
    double W[5];
    if (h < NH) {
        cons2prim(uh, gamma, W);
        if (flip == 1) W[1] = -W[1];
        if (flip == 2) W[2] = -W[2];
#pragma unroll
        for (int f = 0; f < 5; ++f) S.w[o_h + f * PC] = W[f];
    }
    if (col) {
        cons2prim(u, gamma, W);
#pragma unroll
        for (int f = 0; f < 5; ++f) S.w[wrow(tx, ty) + f * PC] = W[f];
    }
    __syncthreads();
    for (int j = warp; j < 17; j += NTP / 32) {
        int o0, o1, o2, o3, out;
        bool isy;
        const int lx = lane & 15, ly = lane >> 4;
        if (j < 8) {  // lo x faces of rows 2j, 2j + 1
            const int r = 2 * j + ly;
            isy = false;
            o2 = wrow(lx, r);
            o0 = lx >= 2 ? o2 - 2 : wxs(lx - 2, r);
            o1 = lx >= 1 ? o2 - 1 : wxs(-1, r);
            o3 = lx <= TX - 2 ? o2 + 1 : wxs(TX, r);
            out = r * (TX + 1) + lx;
        } else if (j < 16) {  // lo y faces of those rows
            const int r = 2 * (j - 8) + ly;
            isy = true;
            o2 = wrow(lx, r);
            o0 = o2 - 32; o1 = o2 - 16; o3 = o2 + 16;
            out = 5 * FX + r * TX + lx;
        } else {  // hi edges: lanes 0..15 of x (row lx), 16..31 of y (column lx)
            isy = ly != 0;
            if (isy) {
                o2 = wrow(lx, TY);
                o0 = o2 - 32; o1 = o2 - 16; o3 = o2 + 16;
                out = 5 * FX + TY * TX + lx;
            } else {
                o1 = wrow(TX - 1, lx);
                o0 = o1 - 1; o2 = wxs(TX, lx); o3 = wxs(TX + 1, lx);
                out = lx * (TX + 1) + TX;
            }
        }
        const int fn = isy ? 2 * PC : PC, ft = isy ? PC : 2 * PC;
        double L[5], R[5], F[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const double *p = S.w + (f == 1 ? fn : f == 2 ? ft : f * PC);
            const double a0 = p[o0], a1 = p[o1], a2 = p[o2], a3 = p[o3];
            const double d = a2 - a1;
            L[f] = face_mm(a1, 0.5, a1 - a0, d);
            R[f] = face_mm(a2, -0.5, d, a3 - a2);
        }
        hllc_frame_any<false>(L, R, gamma, F);
        const int os = isy ? FY : FX;
        const double ar = isy ? g.area[1] : g.area[0];
        double *o = S.g + out;
        o[0] = ar * F[0];
        o[(isy ? 2 : 1) * os] = ar * F[1];
        o[(isy ? 1 : 2) * os] = ar * F[2];
        o[3 * os] = ar * F[3];
        o[4 * os] = ar * F[4];
    }
    __syncthreads();
    double m = 0.0;
    if (own) {
        const int cx = lo_class(ex, nx, perx), cy = lo_class(ey, ny, pery);
        const double invV = ctrl->invV;
        const double *gr = S.g + ty * (TX + 1) + tx;
        const double *gq = S.g + 5 * FX + ty * TX + tx;
        double un[5];
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            const double gxl = gr[f * FX], gxh = gr[f * FX + 1];
            const double gyl = gq[f * FY], gyh = gq[f * FY + TX];
            double a = 0.0;
            if (cy == LO_BEFORE) a -= gyl;
            if (cx == LO_BEFORE) a -= gxl;
            a += gxh;
            if (cx == LO_SELF) a -= gxl;
            a += gyh;
            if (cy == LO_SELF) a -= gyl;
            if (cx == LO_AFTER) a -= gxl;
            if (cy == LO_AFTER) a -= gyl;
            if constexpr (STAGE == 1) un[f] = u[f] - invV * a;
            else un[f] = 0.5 * v[f] + 0.5 * (u[f] - invV * a);
            Uout[lin + f * g.ncell] = un[f];
        }
        if constexpr (STAGE == 2) {
            // the exact CFL term only of cells whose bound exceeds that
            const float b = cfl_bound<false>(un, g, (float)gamma, (float)g.invw[0], (float)g.invw[1], 0.0f);
            if (!(b <= sofar)) m = cfl_term2d_exact(un, g, 0.0);
        }
    }
    if constexpr (STAGE == 2) block_max_to(&ctrl->invdt_bits, m, red);
}

inline int launch_plane_f64(const Geom &g, int stage, const double *Uin, const double *U0,
                            double *Uout, Ctrl *ctrl, cudaStream_t s)
{
    if (!plane_f64_supported(g)) return -1;
    const int ntx = (int)((g.n[0] + 15) / 16);
    const int64_t nt = ntx * ((g.n[1] + 15) / 16);
    if (nt > 0x7fffffffLL) return -1;
    const size_t smem = sizeof(t3d::PlaneSmem);
    static_assert(sizeof(t3d::PlaneSmem) <= 48 * 1024, "within the default shared memory");
    // two blocks an SM hold everything in registers, three (72 registers) spill a
    // little: two where the tiles are done in two rounds of 2 x 148 blocks (384^2:
    // 27.6 us a step against 30.1), three beyond (512^2: 43.4 against 46.4,
    // 1000 x 999: 143 against 162)
    const bool three = nt > 4 * 148;
    auto k = stage == 1 ? three ? k_stage_plane_f64<1, 3> : k_stage_plane_f64<1, 2>
                        : three ? k_stage_plane_f64<2, 3> : k_stage_plane_f64<2, 2>;
    k<<<(unsigned)nt, t3d::NTP, smem, s>>>(g, Uin, U0, Uout, ctrl, ntx);
    return 1;
}

}  // namespace vb
