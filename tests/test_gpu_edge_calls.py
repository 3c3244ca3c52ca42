"""Calls at the edge of what they do: no step to take, refused options, states
and coefficients at the end of a fast form's range.  Each against the oracle or
against the same run without the edge call."""
import math

import numpy as np
import pytest

import vespa_b200 as vb
from vespa_b200 import problem as P

from test_gpu_parity import assert_bit_identical, make_sim, problem_from

pytestmark = pytest.mark.gpu


def box(dims, bc=(0, 2, 1), gamma=1.4):
    nd = len(dims)
    return problem_from(dims, [(0.0, 1.0), (0.0, 1.3), (0.0, 0.9)][:nd], bc[:nd], bc[:nd], gamma, 0.4)


# cell-centric, plane, row-marching and cluster-marched grids
@pytest.mark.parametrize("dims,kind", [((20, 12, 9), "auto"), ((48, 47, 40), "auto"), ((129, 145), "auto"),
                                       ((256, 40), "tiled"), ((64, 32), "auto"), ((64, 32), "cell")])
def test_evolve_without_steps_changes_nothing(vb, oracle, dims, kind):
    prob = box(dims)
    g = oracle.grid_from_problem(prob)
    sim = make_sim(prob, np.ones((5, int(np.prod(dims)))))
    sim.set_kernel(kind)
    for seed, scale in ((1, 1.0), (2, 40.0)):  # the second state's dt differs from the first's
        U0 = P.initial_state(P.smooth_random_problem(dims, seed=seed))
        U0[4] *= scale
        sim.upload(U0)
        sim.set_time(0.0)
        for tfinal in (math.inf, 0.05):
            vb.evolve(sim, tfinal=tfinal, max_steps=0)
            assert (sim.t, sim.step) == (0.0, 0)
        assert_bit_identical(sim.state(), U0)
        vb.evolve(sim, tfinal=0.05, max_steps=3)
        U = U0.copy()
        t, n = oracle.evolve(g, U, 0.05, max_steps=3, mode=1)
        assert (sim.t, sim.step) == (t, n)
        assert_bit_identical(sim.state(), U)
        vb.evolve(sim, tfinal=0.05, max_steps=0)  # and after steps: the folded maximum stays good
        vb.evolve(sim, tfinal=0.05, max_steps=2)
        t2, n2 = oracle.evolve(g, U, 0.05, max_steps=2, t0=t, mode=1)
        assert (sim.t, sim.step) == (t2, n + n2)
        assert_bit_identical(sim.state(), U)


def test_staged_face_batches_bit_identical(vb, oracle):
    """Batches and copies before and after the staging lanes come in (256 MiB of
    them), a last piece of one face, fluxes over the left states, pinned arrays."""
    from tests.golden.make_golden import random_faces
    torch = pytest.importorskip("torch")
    ctx = vb.Context(0)
    backend = vb.B200Flux(ctx)
    for nf in (32768, 8192 * 9 + 1):
        WL, WR, axis = random_faces(nf, seed=nf)
        ref = oracle.compute_face_fluxes(WL, WR, axis, 1.4)
        for k in range(36 if nf > 32768 else 2):
            F = np.zeros_like(WL)
            vb.compute_face_fluxes(backend, 1.4, F, WL, WR, axis)
            assert_bit_identical(F, ref)
    pin = [torch.from_numpy(a.copy()).pin_memory().numpy() for a in (WL, WR, F)]
    vb.compute_face_fluxes(backend, 1.4, pin[2], pin[0], pin[1], axis)
    assert_bit_identical(pin[2], ref)
    both = np.vstack([WL, np.zeros((7, 5))])
    vb.compute_face_fluxes(backend, 1.4, both[7:], both[:-7], WR, axis)
    assert_bit_identical(both[7:], ref)
    prob = box((64, 64, 33))
    U0 = P.initial_state(P.smooth_random_problem((64, 64, 33), seed=2))
    sim = vb.Simulation(vb.B200Mesh(prob.dims, prob.domain), prob, initial=U0, ctx=ctx)
    assert_bit_identical(sim.state(), U0)


# the stage kernels fold the exact CFL term only of cells whose float32 bound
# exceeds the maximum so far: gammas next to 1, speeds and pressures that float32
# cannot hold, very wide and very narrow cells, a free-fall rate below its range
@pytest.mark.parametrize("dims", [(48, 48, 40), (129, 145)])
@pytest.mark.parametrize("case", [dict(gamma=1.0005), dict(gamma=1.00001), dict(speed=1e-25), dict(speed=1e-18),
                                  dict(speed=1e18), dict(mass=1e-60), dict(mass=1e60), dict(width=1e43),
                                  dict(width=1e-43), dict(speed=1e-25, G=1e-46), dict(G=0.0), dict(G=0.5)])
def test_time_step_matches_the_cell_kernel_bit_for_bit(vb, dims, case):
    if "G" in case and len(dims) != 3:
        pytest.skip("gravity steps 2D grids with the cell kernel")
    gamma, v, m, w = (case.get(k, d) for k, d in (("gamma", 1.4), ("speed", 1.0), ("mass", 1.0), ("width", 1.0)))
    prob = problem_from(dims, [(0.0, w)] * len(dims), (1, 1, 1)[:len(dims)], (1, 1, 1)[:len(dims)], gamma, 0.4)
    U0 = P.initial_state(P.smooth_random_problem(dims, seed=12, gamma=gamma))
    U0[1:4] *= v
    U0[4] *= v * v
    U0 *= m
    out = []
    for kind in ("auto", "cell"):
        sim = make_sim(prob, U0)
        sim.set_kernel(kind)
        if "G" in case:
            vb.enable_gravity(sim, G=case["G"], tol=1e-6, maxiter=50)
        vb.evolve(sim, tfinal=math.inf, max_steps=8)
        assert sim.step == 8
        out.append((sim.t, sim.state()))
    assert out[0][0] == out[1][0]
    assert_bit_identical(out[0][1], out[1][1])
