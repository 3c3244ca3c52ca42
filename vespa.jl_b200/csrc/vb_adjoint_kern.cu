// vb_adjoint_kern.cu -- adjoint (reverse-mode) kernels of one SSP-RK2 stage
// on a periodic uniform mesh, float64, built with -fmad=false so the
// recomputed forward quantities (and hence every frozen branch) are the
// forward step's own bits.
//
// A stage is Uout = base - invV * D(U) with D(U)_i = sum over the faces of
// cell i of +-area * F(WL, WR) (src/driver.jl:236-281, 297-321).  Its
// transpose applied to an adjoint mu is, face by face,
//   Fb = area * (mu_L - mu_R)  ->  HLLC reverse  ->  WLb, WRb
// then through the PLM face values WL = W_i + s_i/2, WR = W_{i+1} - s_{i+1}/2
// (src/driver.jl:227-233) and minmod slopes into the cell primitives, and
// through cons2prim into the conserved adjoint.
//
// Two passes, no atomics (the result does not depend on scheduling):
//   k_adj_face: one thread per (cell i, axis): face i+1/2 of that axis; writes
//     WLb, WRb of the face and the minmod branch codes of s_i.
//   k_adj_cell: one thread per cell: gathers the face adjoints that depend on
//     its primitives, applies the cons2prim reverse and the RK2 combination.
#include "vb_adjoint.cuh"
#include "vb_launch.h"
#include "vb_stage_generic.cuh"

namespace vb {

namespace {

// the cell `off` cells away along ax (periodic); the modulo only at the wrap
__device__ __forceinline__ int64_t wrap_lin(const Geom &g, int ax, int64_t lin, int64_t c, int off)
{
    const int64_t n = g.n[ax];
    int64_t j = c + off;
    if (j < 0 || j >= n) {
        j %= n;
        if (j < 0) j += n;
    }
    return lin + (j - c) * g.stride[ax];
}

__device__ __forceinline__ int64_t coord(const Geom &g, int ax, int64_t lin)
{
    int64_t cc[3];
    cell_coords(g, lin, cc);
    return cc[ax];
}

template <int AX>
__device__ __forceinline__ void adj_face_axis(const Geom &g, const double *__restrict__ U,
                                              const double *__restrict__ M, double ms, int64_t lin,
                                              double *__restrict__ gL, double *__restrict__ gR,
                                              uint16_t *__restrict__ code)
{
    const int64_t nc = g.ncell;
    const int64_t c = coord(g, AX, lin);
    const int64_t lm1 = wrap_lin(g, AX, lin, c, -1);
    const int64_t lp1 = wrap_lin(g, AX, lin, c, 1);
    const int64_t lp2 = wrap_lin(g, AX, lin, c, 2);
    double Wm1[5], W0[5], Wp1[5], Wp2[5];
    load_prim<double>(g, U, lm1, Wm1);
    load_prim<double>(g, U, lin, W0);
    load_prim<double>(g, U, lp1, Wp1);
    load_prim<double>(g, U, lp2, Wp2);
    double WL[5], WR[5], Fb[5];
    unsigned cd = 0;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const double a0 = W0[k] - Wm1[k], b0 = Wp1[k] - W0[k];
        cd |= minmod_code(a0, b0) << (2 * k);
        WL[k] = face_val(W0[k], 0.5, minmod<double>(a0, b0));
        WR[k] = face_val(Wp1[k], -0.5, limited_slope<double>(W0[k], Wp1[k], Wp2[k]));
        Fb[k] = g.area[AX] * (ms * __ldg(M + k * nc + lin) - ms * __ldg(M + k * nc + lp1));
    }
    double WLb[5] = {0, 0, 0, 0, 0}, WRb[5] = {0, 0, 0, 0, 0};
    hllc_vjp<AX + 1>(WL, WR, g.gamma, Fb, WLb, WRb);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        gL[(AX * 5 + k) * nc + lin] = WLb[k];
        gR[(AX * 5 + k) * nc + lin] = WRb[k];
    }
    code[AX * nc + lin] = (uint16_t)cd;
}

template <int ND>
__global__ void __launch_bounds__(128)
k_adj_face(Geom g, const double *__restrict__ U, const double *__restrict__ M, double ms,
           double *__restrict__ gL, double *__restrict__ gR, uint16_t *__restrict__ code)
{
    const int64_t lin = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= g.ncell) return;
    const int ax = blockIdx.y;
    if (ax == 0) adj_face_axis<0>(g, U, M, ms, lin, gL, gR, code);
    if constexpr (ND > 1) if (ax == 1) adj_face_axis<1>(g, U, M, ms, lin, gL, gR, code);
    if constexpr (ND > 2) if (ax == 2) adj_face_axis<2>(g, U, M, ms, lin, gL, gR, code);
}

// out = 0.5*lam + (M ? M : 0) - invV * (dD/dU)^T mu   (per cell)
template <int ND>
__global__ void __launch_bounds__(256)
k_adj_cell(Geom g, const double *__restrict__ U, const double *__restrict__ gL,
           const double *__restrict__ gR, const uint16_t *__restrict__ code,
           const double *lam, const double *M, double invV, double *out)
{
    const int64_t nc = g.ncell;
    const int64_t lin = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= nc) return;
    double Wb[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int ax = 0; ax < ND; ++ax) {
        const int64_t c = coord(g, ax, lin);
        const int64_t km1 = wrap_lin(g, ax, lin, c, -1);
        const int64_t km2 = wrap_lin(g, ax, lin, c, -2);
        const int64_t kp1 = wrap_lin(g, ax, lin, c, 1);
        const unsigned ck = code[ax * nc + lin];
        const unsigned cp = code[ax * nc + kp1];
        const unsigned cm = code[ax * nc + km1];
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int64_t o = (int64_t)(ax * 5 + k) * nc;
            const double fl = gL[o + lin], fr = gR[o + km1];
            // own value in both faces' states
            double w = fl + fr;
            // own slope s_k (hi face +1/2, lo face -1/2)
            const double sb = 0.5 * fl - 0.5 * fr;
            const unsigned bk = (ck >> (2 * k)) & 3u;
            if (bk == 1u) w += sb;
            else if (bk == 2u) w -= sb;
            // s_{k+1} = W_{k+1} - W_k when its branch is the left difference
            if (((cp >> (2 * k)) & 3u) == 1u) w -= 0.5 * gL[o + kp1] - 0.5 * gR[o + lin];
            // s_{k-1} = W_k - W_{k-1} when its branch is the right difference
            if (((cm >> (2 * k)) & 3u) == 2u) w += 0.5 * gL[o + km1] - 0.5 * gR[o + km2];
            Wb[k] += w;
        }
    }
    double u[5], Ub[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) u[k] = __ldg(U + k * nc + lin);
    cons2prim_vjp(u, g.gamma, Wb, Ub);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int64_t i = k * nc + lin;
        double v = 0.5 * lam[i];
        if (M) v = v + M[i];
        out[i] = v - invV * Ub[k];
    }
}

// Both passes of a 2D stage in one kernel: a block owns a 16 x 16 tile.  The
// primitives of the tile and of the three cells around it along each axis come
// into shared memory (each converted once, not four times per face and axis);
// the 19 faces per row and per column that the tile's cells depend on are
// solved there (1.19 times the faces, against writing and gathering ten
// values a face through memory), then each cell gathers its own.
namespace adj2 {

constexpr int T = 16, H = 3, S = T + 2 * H;  // tile, halo, extended side
constexpr int NW = T * S;                     // cells of one extended strip
constexpr int NF = T * (T + 3);               // faces of one axis: 19 per line
constexpr int NTH = 320;

struct Smem {
    double w[2][5][NW];   // primitives: x strip [row][22], y strip [column][22]
    double mu[2][5][NW];  // the adjoint state that the face fluxes meet, the same way
    double gl[2][5][NF], gr[2][5][NF];  // face adjoints WLb, WRb, line-major
    uint16_t code[2][NF]; // minmod codes of the cell behind each face
};

}  // namespace adj2

__global__ void __launch_bounds__(adj2::NTH, 2)
k_adj_plane(const __grid_constant__ Geom g, const double *__restrict__ U, const double *lam,
            const double *M, double invV, double *out, int ntx)
{
    using namespace adj2;
    extern __shared__ __align__(16) unsigned char raw[];
    adj2::Smem &S_ = *reinterpret_cast<adj2::Smem *>(raw);
    const int t = threadIdx.x;
    const int nx = (int)g.n[0], ny = (int)g.n[1];
    const int x0 = (int)(blockIdx.x % ntx) * T, y0 = (int)(blockIdx.x / ntx) * T;
    const int64_t nc = g.ncell;
    const double gamma = g.gamma, ig1 = 1.0 / (gamma - 1.0);
    auto wrap = [](int c, int n) {
        c %= n;
        return c < 0 ? c + n : c;
    };
    // strip a's cell (line, pos): along x position pos - 3 of row `line`, along
    // y of column `line`
    auto cell = [&](int a, int line, int pos) {
        const int x = a == 0 ? x0 + pos - H : x0 + line, y = a == 0 ? y0 + line : y0 + pos - H;
        return (int64_t)wrap(x, nx) + (int64_t)nx * wrap(y, ny);
    };
    const double *mu = M ? M : lam;  // mu = 0.5 lam (stage 2) or M (stage 1)
    const double ms = M ? 1.0 : 0.5;
    // the tile's cells go into both strips, the halo cells into their own
    for (int i = t; i < T * T + 4 * H * T; i += NTH) {
        int a = 0, line, pos, pos2 = -1, line2 = 0;
        if (i < T * T) {
            line = i / T;
            pos = (i & (T - 1)) + H;
            line2 = i & (T - 1);
            pos2 = line + H;
        } else {
            const int h = i - T * T;
            a = h / (2 * H * T);
            const int r = h - a * 2 * H * T, k = r / T;  // halo position 0 .. 5
            // along y consecutive threads take consecutive columns
            line = r - k * T;
            pos = k < H ? k : k + T;
        }
        const int64_t l = cell(a, line, pos);
        if (!VB_DCHECK(l >= 0 && l < nc && line * S + pos < NW && line2 * S + pos2 < NW)) continue;  // check build only
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            cp_async8(&S_.mu[a][k][line * S + pos], mu + k * nc + l);
            if (pos2 >= 0) cp_async8(&S_.mu[1][k][line2 * S + pos2], mu + k * nc + l);
        }
        double u[5], W[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) u[k] = __ldg(U + k * nc + l);
        cons2prim(u, gamma, W);
#pragma unroll
        for (int k = 0; k < 5; ++k) S_.w[a][k][line * S + pos] = W[k];
        if (pos2 >= 0)
#pragma unroll
            for (int k = 0; k < 5; ++k) S_.w[1][k][line2 * S + pos2] = W[k];
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    for (int i = t; i < 2 * NF; i += NTH) {
        const int a = i >= NF, j = i - a * NF, line = j / (T + 3), f = j - line * (T + 3);
        // face f lies between cells f + 1 and f + 2 of the strip
        const int c = line * S + f + 1;
        double L[5], R[5], Fb[5], Lb[5], Rb[5];
        unsigned cd = 0;
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            // component k of the frame is field kf: normal and first tangential
            // velocity swap on y faces
            const int kf = a == 1 && (k == 1 || k == 2) ? 3 - k : k;
            const double *p = S_.w[a][kf] + c;
            const double m1 = p[-1], q0 = p[0], q1 = p[1], q2 = p[2], b = q1 - q0;
            cd |= minmod_code(q0 - m1, b) << (2 * kf);
            L[k] = face_val(q0, 0.5, minmod<double>(q0 - m1, b));
            R[k] = face_val(q1, -0.5, minmod<double>(b, q2 - q1));
            const double *q = S_.mu[a][kf] + c;
            Fb[k] = g.area[a] * (ms * q[0] - ms * q[1]);
        }
        hllc_vjp_frame(L, R, gamma, ig1, Fb, Lb, Rb);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            const int kf = a == 1 && (k == 1 || k == 2) ? 3 - k : k;
            S_.gl[a][kf][j] = Lb[k];
            S_.gr[a][kf][j] = Rb[k];
        }
        S_.code[a][j] = (uint16_t)cd;
    }
    // the own cell's inputs of the last part arrive while others solve faces
    static_assert(T * T <= NTH, "one cell a thread");
    const int lx = t & (T - 1), ly = t / T, x = x0 + lx, y = y0 + ly;
    const int64_t lin = (int64_t)x + (int64_t)nx * y;
    const bool own = t < T * T && x < nx && y < ny && VB_DCHECK(lin >= 0 && lin < nc);
    double u[5], v[5];
    if (own)
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            u[k] = __ldg(U + k * nc + lin);
            v[k] = lam[k * nc + lin];
        }
    __syncthreads();
    if (own) {
        double Wb[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            // the cell's hi face is face pos + 2 of its line: cell pos + 3 of the
            // strip is behind it
            const int o = (a == 0 ? ly * (T + 3) + lx : lx * (T + 3) + ly) + 2;
            const unsigned ck = S_.code[a][o], cp = S_.code[a][o + 1], cm = S_.code[a][o - 1];
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const double *gl = S_.gl[a][k] + o, *gr = S_.gr[a][k] + o;
                const double fl = gl[0], fr = gr[-1];
                double w = fl + fr;
                const double sb = 0.5 * fl - 0.5 * fr;
                const unsigned bk = (ck >> (2 * k)) & 3u;
                if (bk == 1u) w += sb;
                else if (bk == 2u) w -= sb;
                if (((cp >> (2 * k)) & 3u) == 1u) w -= 0.5 * gl[1] - 0.5 * gr[0];
                if (((cm >> (2 * k)) & 3u) == 2u) w += 0.5 * gl[-1] - 0.5 * gr[-2];
                Wb[k] += w;
            }
        }
        double Ub[5];
        cons2prim_vjp(u, gamma, Wb, Ub);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
            double b = 0.5 * v[k];
            if (M) b = b + S_.mu[0][k][ly * S + lx + H];
            out[k * nc + lin] = b - invV * Ub[k];
        }
    }
}

__global__ void k_record_dt(const Ctrl *ctrl, double *dts, long long step0, long long cap)
{
    if (!ctrl->active) return;
    const long long i = ctrl->step - step0;
    if (i >= 0 && i < cap) dts[i] = ctrl->dt;
}

}  // namespace

int launch_adj_stage(const Geom &g, const double *U, const double *lam, const double *M,
                     double invV, double *gL, double *gR, uint16_t *code, double *out,
                     cudaStream_t s)
{
    if (adj_on_chip(g)) {
        const int ntx = (int)((g.n[0] + adj2::T - 1) / adj2::T);
        const int64_t nt = ntx * ((g.n[1] + adj2::T - 1) / adj2::T);
        static PerDevice opted;
        const int set = opted.get([] {
            return cudaFuncSetAttribute(k_adj_plane, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)sizeof(adj2::Smem)) == cudaSuccess
                       ? 1
                       : -1;
        });
        if (set < 0 || nt > 0x7fffffffLL) return -1;
        k_adj_plane<<<(unsigned)nt, adj2::NTH, sizeof(adj2::Smem), s>>>(g, U, lam, M, invV, out, ntx);
        return 1;
    }
    const int64_t nb_f = (g.ncell + 127) / 128;
    if (g.ncell <= 0 || nb_f > 0x7fffffffLL) return -1;
    // mu = 0.5*lam (adjoint of stage 2) or M (adjoint of stage 1)
    const double *mu = M ? M : lam;
    const double ms = M ? 1.0 : 0.5;
    const dim3 gf((unsigned)nb_f, (unsigned)g.nd);
    const unsigned gc = (unsigned)((g.ncell + 255) / 256);
    switch (g.nd) {
    case 1:
        k_adj_face<1><<<gf, 128, 0, s>>>(g, U, mu, ms, gL, gR, code);
        k_adj_cell<1><<<gc, 256, 0, s>>>(g, U, gL, gR, code, lam, M, invV, out);
        break;
    case 2:
        k_adj_face<2><<<gf, 128, 0, s>>>(g, U, mu, ms, gL, gR, code);
        k_adj_cell<2><<<gc, 256, 0, s>>>(g, U, gL, gR, code, lam, M, invV, out);
        break;
    case 3:
        k_adj_face<3><<<gf, 128, 0, s>>>(g, U, mu, ms, gL, gR, code);
        k_adj_cell<3><<<gc, 256, 0, s>>>(g, U, gL, gR, code, lam, M, invV, out);
        break;
    default: return -1;
    }
    return 2;
}

int launch_record_dt(const Ctrl *ctrl, double *dts, int64_t step0, int64_t cap, cudaStream_t s)
{
    k_record_dt<<<1, 1, 0, s>>>(ctrl, dts, (long long)step0, (long long)cap);
    return 1;
}

}  // namespace vb
