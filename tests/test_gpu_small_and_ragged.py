"""Grids that fit no 16-cell tile, small grids marched in one launch, and the
general paths behind the float64 fast forms: each against the oracle, bit for
bit, at the sizes where a new branch begins or ends."""
import math

import numpy as np
import pytest

import vespa_b200 as vb
from vespa_b200 import muscl as M
from vespa_b200 import problem as P

from test_gpu_parity import assert_bit_identical, make_sim, problem_from

pytestmark = pytest.mark.gpu

WALLS = [((1, 1, 1), (1, 1, 1)), ((0, 2, 0), (2, 0, 2)), ((1, 2, 1), (1, 0, 1)), ((0, 1, 2), (0, 1, 0))]


def run_pair(oracle, dims, lo, hi, steps, kz=None, tfinal=math.inf, sharp=True):
    nd = len(dims)
    prob = problem_from(dims, [(0.0, 1.0), (0.0, 1.3), (0.0, 0.9)][:nd], lo[:nd], hi[:nd], 1.4, 0.4)
    U0 = P.initial_state(P.smooth_random_problem(dims, seed=sum(dims)))
    if sharp:
        U0[0] *= 1 + 10 * (np.arange(U0.shape[1]) % 7 == 0)
    sim = make_sim(prob, U0)
    if kz:
        sim.set_kernel("auto", kz=kz)
    vb.evolve(sim, tfinal=tfinal, max_steps=steps)
    U = U0.copy()
    t, n = oracle.evolve(oracle.grid_from_problem(prob), U, tfinal, max_steps=steps, mode=1)
    assert sim.step == n and sim.t == t
    assert_bit_identical(sim.state(), U)
    return sim


# 3D boxes around the float64 tile kernel's choice.  Below 148 blocks of cells the
# cell kernel: one tile, 2 planes, odd sides.  Above it the tile kernel: a shifted
# last tile that leaves 1 or 15 cells of its own along x, along y or both, one
# tile along y, 2 planes, chunks shorter than the box
CELL_BOXES = [(16, 16, 2), (17, 19, 7), (31, 33, 20), (18, 17, 6), (35, 16, 16)]
TILE_BOXES = [(33, 47, 31), (31, 33, 40), (17, 31, 80), (35, 16, 70), (49, 63, 17), (160, 161, 2), (48, 32, 26)]


@pytest.mark.parametrize("dims", CELL_BOXES + TILE_BOXES)
@pytest.mark.parametrize("lo,hi", WALLS)
@pytest.mark.parametrize("kz", [None, 3])
def test_ragged_boxes_bit_identical(vb, oracle, dims, lo, hi, kz):
    sim = run_pair(oracle, dims, lo, hi, 3, kz if kz and kz < dims[2] else None)
    assert sim.kernel == ("tiled" if dims in TILE_BOXES else "cell")


@pytest.mark.parametrize("dims", [(19, 33, 9), (33, 47, 31), (17, 31, 80), (49, 34, 25)])
@pytest.mark.parametrize("lo,hi", WALLS[1:])
def test_ragged_box_records_boundary_fluxes_and_gravity(vb, oracle, dims, lo, hi):
    prob = problem_from(dims, [(0.0, 1.0)] * 3, lo, hi, 1.4, 0.4)
    U0 = P.initial_state(P.smooth_random_problem(dims, seed=3))
    out = []
    for kind in ("auto", "cell"):
        sim = make_sim(prob, U0)
        sim.set_kernel(kind)
        sim.bflux_enable()
        assert sim.kernel == ("tiled" if kind == "auto" and dims[2] > 9 else "cell")
        vb.evolve(sim, max_steps=3)
        out.append((sim.state(), sim.bflux_read()))
        sim.bflux_enable(False)
        vb.enable_gravity(sim, G=0.3, bcs=P.Outflow, tol=1e-10, project_mean=True)
        assert sim.kernel == ("tiled" if kind == "auto" and dims[2] > 9 else "cell")
        vb.evolve(sim, max_steps=2)
        out[-1] += (sim.state(),)
    for a, b in zip(*out):
        assert_bit_identical(a, b)


# 1D and 2D grids marched by one cluster: 4 cells, one block, the largest
# cluster, uneven slabs, thin slabs (halo rows from two blocks away), slabs that
# just fit in shared memory; 112 x 113 does not and takes the plane kernel
@pytest.mark.parametrize("dims", [(4,), (5,), (255,), (257,), (3000,), (18000,), (4, 4), (17, 33), (100, 31),
                                  (31, 100), (8, 300), (300, 8), (112, 112), (112, 113)])
@pytest.mark.parametrize("lo,hi", WALLS)
def test_marched_grids_bit_identical(vb, oracle, dims, lo, hi):
    assert run_pair(oracle, dims, lo, hi, 7).kernel == ("plane" if dims == (112, 113) else "march")


def test_march_stops_resumes_and_reports(vb, oracle):
    sim = run_pair(oracle, (40,), (0,), (0,), -1, tfinal=0.1, sharp=False)
    n, t = sim.step, sim.t
    vb.evolve(sim, tfinal=0.1)  # already there
    assert (sim.step, sim.t) == (n, t)
    ref = make_sim(sim.problem, sim.state())
    ref.set_kernel("cell")
    vb.run_steps_async(sim, 5)  # queued steps continue, as the cell kernel's do
    vb.run_steps_async(ref, 5)
    assert_bit_identical(sim.state(), ref.state())
    assert vb.compute_dt(sim) == vb.compute_dt(ref)
    U = sim.state()
    U[0, 7] = -1.0
    sim.upload(U)
    with pytest.raises(vb.VespaB200Error) as e:
        vb.evolve(sim, max_steps=3)
    assert "VB_ENONFINITE" in str(e.value)


# 2D grids of the plane kernel (beyond the march's size, all but 16 x 900): ragged
# both ways, one tile across
@pytest.mark.parametrize("dims", [(129, 145), (256, 128), (1000, 17), (16, 900), (16, 2500), (2500, 31), (400, 401),
                                  (512, 512)])
@pytest.mark.parametrize("lo,hi", WALLS)
def test_plane_grids_bit_identical(vb, oracle, dims, lo, hi):
    assert run_pair(oracle, dims, lo, hi, 3).kernel == ("march" if dims == (16, 900) else "plane")


# operands outside the range of the divisions' fast form, zeros among them
@pytest.mark.parametrize("scale", [1e-200, 1e-38, 1.0, 1e38, 1e150])
def test_extreme_magnitudes_bit_identical(vb, oracle, scale):
    dims = (48,)
    prob = problem_from(dims, [(0.0, 1.0)], (2,), (0,), 1.4, 0.4)
    U0 = P.initial_state(P.smooth_random_problem(dims, seed=5))
    U0[1:4, :20] = 0.0
    U0[0] *= scale
    U0[1:4] *= scale
    U0[4] *= scale
    U0[:, 30:] *= 1e-3
    sim = make_sim(prob, U0)
    vb.evolve(sim, max_steps=4)
    U = U0.copy()
    oracle.evolve(oracle.grid_from_problem(prob), U, math.inf, max_steps=4, mode=1)
    assert_bit_identical(sim.state(), U)


@pytest.mark.parametrize("case", ["plain", "tiny", "huge", "nan", "inf"])
def test_muscl_general_forms_bit_identical(vb, oracle, case):
    dims, ng = (39, 13, 11), 3
    prob = P.smooth_random_problem(dims, seed=8)
    U = P.initial_state(prob)
    if case == "tiny":
        U *= 1e-45
    elif case == "huge":
        U *= 1e60
    elif case in ("nan", "inf"):
        U[0, 39 * 13 * 5 + 39 * 6 + 20] = math.nan if case == "nan" else math.inf
    g = M.MusclGrid(dims, ng)
    g.upload(U)
    kw = dict(dt=1e-3, gamma=1.4, theta=1.5, dx=1.0 / 39, small_rho=1e-60)
    for _ in range(2):
        g.step(**kw)
        U = oracle.muscl_step(dims, ng, U, kw["dt"], kw["gamma"], kw["theta"], kw["dx"], kw["small_rho"])
    assert np.array_equal(g.state(), U, equal_nan=True)


# the mixed kernels on shifted tiles and segments: near the float64 result, and
# conserving as on whole tiles (each updated cell takes both fluxes of a face
# from one solve)
MIXED_TILED = [(48, 47, 60), (34, 18, 80), (18, 31, 80), (50, 62, 17), (258, 1200), (510, 1190), (766, 800)]


@pytest.mark.parametrize("dims", [(18, 34, 9), (258, 20), (510, 130), (20, 18, 130)] + MIXED_TILED)
@pytest.mark.parametrize("per", [True, False])
def test_ragged_mixed_grids(vb, dims, per):
    nd = len(dims)
    bc = (1, 1, 1) if per else (2, 0, 2)
    prob = problem_from(dims, [(0.0, 1.0)] * nd, bc[:nd], bc[:nd], 1.4, 0.4)
    U0 = P.initial_state(P.smooth_random_problem(dims, seed=4))
    a, b = make_sim(prob, U0), make_sim(prob, U0, "mixed")
    t0 = np.array(vb.conserved_totals(b))
    assert b.kernel == ("tiled" if dims in MIXED_TILED else "cell")
    for s in (a, b):
        vb.evolve(s, max_steps=10)
    l1 = np.sum(np.abs(a.state()[0] - b.state()[0])) / np.sum(np.abs(a.state()[0]))
    assert l1 <= 1e-6, l1
    if per:
        assert np.allclose(np.array(vb.conserved_totals(b)), t0, rtol=1e-12, atol=1e-12 * np.abs(t0).max())


def test_large_face_batches_bit_identical(vb, oracle):
    from tests.golden.make_golden import random_faces
    for nf in (32767, 32768, 8192 * 9 + 1):  # below and at the staged path, a last piece of one face
        WL, WR, axis = random_faces(nf, seed=nf)
        F = np.zeros_like(WL)
        for _ in range(2):
            vb.compute_face_fluxes(vb.B200Flux(), 1.4, F, WL, WR, axis)
        assert_bit_identical(F, oracle.compute_face_fluxes(WL, WR, axis, 1.4))
    bad = axis.copy()
    bad[-1] = 4
    G = np.full_like(F, 7.0)
    with pytest.raises(vb.VespaB200Error):
        vb.compute_face_fluxes(vb.B200Flux(), 1.4, G, WL, WR, bad)
    assert np.all(G == 7.0)


# cubes whose coarsest level is the base grid, odd and too large for one block,
# or reached through levels in one block; cubes whose neighbours are the cell
# itself or one another; plain CG through the same graph
@pytest.mark.parametrize("n,precond", [(1, "none"), (1, "mg"), (2, "none"), (2, "mg"), (3, "mg"), (6, "none"),
                                       (4, "mg"), (7, "mg"), (16, "mg"), (17, "mg"), (34, "mg"), (20, "mg"),
                                       (40, "mg"), (5, "none"), (33, "none")])
def test_cube_solves_reach_the_oracle(vb, oracle, n, precond):
    prob = P.smooth_random_problem((n, n, n), seed=n)
    U0 = P.initial_state(prob)
    sim = make_sim(prob, U0)
    grav = vb.enable_gravity(sim, G=1.0, tol=1e-10, maxiter=400, precond=precond)
    iters, relres = vb.solve_poisson(sim)
    assert 0 < iters < 400 and relres <= 1e-10
    first = grav.phi
    o = oracle.make_gravity(1.0, (1, 1, 1), (1, 1, 1), maxiter=400, tol=1e-10, project_mean=True)
    phi = np.zeros(n ** 3)
    oracle.grav_solve(oracle.grid_from_problem(prob), o, U0, phi)
    # both residuals are below 1e-10 of the right-hand side; the inverse of the
    # smallest mode amplifies that by at most (n / 2)^2
    assert np.max(np.abs(first - phi)) <= 1e-10 * (n / 2 + 1) ** 2 * np.max(np.abs(phi))
    grav.phi = np.zeros(n ** 3)
    vb.solve_poisson(sim)
    assert np.array_equal(grav.phi, first)  # fixed-order sums: the same bits again
