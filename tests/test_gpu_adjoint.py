"""CUDA adjoint of the float64 step (vb_adjoint_*) against the torch
autograd restatement (oracle/adjoint_ref.py) and against central finite
differences of the CUDA forward path."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _sim(vb, prob):
    mesh = vb.B200Mesh(prob.dims, prob.domain)
    return vb.Simulation(mesh, prob, precision="fp64")


def _grid(prob):
    from oracle import adjoint_ref as R
    return R.PeriodicGrid(prob.dims, prob.domain, prob.gamma)


def _close(got, ref, rtol):
    scale = np.abs(ref).max(axis=1, keepdims=True) + 1e-300
    err = (np.abs(got - ref) / scale).max()
    assert err <= rtol, err


CASES = {
    "kh16": lambda vb: vb.kelvin_helmholtz_problem(n=16),
    "kh24_textured": lambda vb: vb.kelvin_helmholtz_problem(n=24, texture=1e-2),
    "smooth2d_24x20": lambda vb: vb.smooth_random_problem((24, 20)),
    "smooth3d_8x6x5": lambda vb: vb.smooth_random_problem((8, 6, 5)),
    "smooth1d_40": lambda vb: vb.smooth_random_problem((40,)),
    "smooth2d_3x2": lambda vb: vb.smooth_random_problem((3, 2)),
    "smooth2d_2x4737": lambda vb: vb.smooth_random_problem((2, 4737)),  # too thin for the tiles
    "smooth2d_9x4737": lambda vb: vb.smooth_random_problem((9, 4737)),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_adjoint_step_matches_autograd(vb, case):
    from oracle import adjoint_ref as R
    prob = CASES[case](vb)
    sim = _sim(vb, prob)
    U0 = sim.state()
    dt = vb.compute_dt(sim)
    lam = np.random.default_rng(11).standard_normal(U0.shape)
    adj = vb.Adjoint(sim, 1, 1)
    got = adj.step(dt, lam)
    UT, ref = R.vjp(_grid(prob), U0, [dt], lam)
    _close(got, ref, 1e-10)
    # the grid is not advanced by the single-step adjoint
    assert np.array_equal(sim.state(), U0)
    adj.close()
    sim.close()


def test_checkpointed_run_matches_autograd(vb):
    """12 steps with checkpoints every 5: equals torch autograd over the same
    dts, and equals the runs checkpointed every step / once (bitwise)."""
    from oracle import adjoint_ref as R
    prob = vb.kelvin_helmholtz_problem(n=24, texture=1e-2)
    U0 = vb.initial_state(prob)
    lam = None
    results = []
    for every in (5, 1, 12):
        sim = _sim(vb, prob)
        adj = vb.Adjoint(sim, 12, every)
        t, n = adj.forward(max_steps=12)
        assert n == 12
        UT = sim.state()
        if lam is None:
            lam = vb.rho2_seed(sim, UT)
            dts = adj.dts()
        else:
            assert np.array_equal(adj.dts(), dts)
        results.append(adj.backward(lam))
        adj.close()
        sim.close()
    assert np.array_equal(results[0], results[1])
    assert np.array_equal(results[0], results[2])
    UT_ref, ref = R.vjp(_grid(prob), U0, dts, lam)
    _close(results[0], ref, 1e-9)


def test_forward_run_matches_plain_evolve(vb):
    """The recording forward run advances the grid exactly like evolve!."""
    prob = vb.kelvin_helmholtz_problem(n=32)
    a = _sim(vb, prob)
    b = _sim(vb, prob)
    adj = vb.Adjoint(a, 30, 7)
    adj.forward(max_steps=30)
    vb.evolve(b, max_steps=30)
    assert np.array_equal(a.state(), b.state())
    assert a.step == b.step == 30
    adj.close()
    a.close()
    b.close()


def test_tfinal_stops_recording(vb):
    prob = vb.kelvin_helmholtz_problem(n=32)
    sim = _sim(vb, prob)
    adj = vb.Adjoint(sim, 100, 8)
    t, n = adj.forward(tfinal=0.01)
    assert 0 < n < 100 and abs(t - 0.01) < 1e-15
    dts = adj.dts()
    assert len(dts) == n and abs(float(np.sum(dts)) - t) < 1e-14
    lam = np.ones((5, sim.ncell))
    out = adj.backward(lam)
    assert np.all(np.isfinite(out))
    adj.close()
    sim.close()


def _run_fixed(vb, sim, U0, dts):
    sim.upload(U0)
    for dt in dts:
        vb.step(sim, float(dt))
    return sim.state()


def _fd_errors(vb, prob, nsteps, every, ncells, h_rel, seed=3):
    sim = _sim(vb, prob)
    U0 = sim.state()
    adj = vb.Adjoint(sim, nsteps, every)
    adj.forward(max_steps=nsteps)
    UT = sim.state()
    dts = adj.dts()
    grad = adj.backward(vb.rho2_seed(sim, UT))
    V = sim.backend.cell_volume()
    errs = []
    for cell in np.random.default_rng(seed).choice(sim.ncell, size=ncells, replace=False):
        h = h_rel * U0[0, cell]
        Up = U0.copy(); Up[0, cell] += h
        Um = U0.copy(); Um[0, cell] -= h
        rp = _run_fixed(vb, sim, Up, dts)[0]
        rm = _run_fixed(vb, sim, Um, dts)[0]
        fd = float(np.sum((rp - rm) * (rp + rm)) * V) / (2.0 * h)
        errs.append(abs(fd - grad[0, cell]) / abs(grad[0, cell]))
    adj.close()
    sim.close()
    return np.array(errs)


def test_kh512_short_run_matches_finite_differences(vb):
    """d(int rho^2)/d rho_0 after 20 steps of KH 512^2 (checkpoints every 5)
    at 32 random cells against central differences (h = 1e-6 relative) with
    the dt sequence held fixed: every cell within 1e-6.  The KH state gets a
    1e-2 texture so no limiter starts on a tie."""
    prob = vb.kelvin_helmholtz_problem(n=512, texture=1e-2)
    errs = _fd_errors(vb, prob, 20, 5, 32, 1e-6)
    assert errs.max() <= 1e-6, errs


def test_kh512_200_steps_matches_finite_differences(vb):
    """The full KH 512^2 adjoint run (200 steps, checkpoints every 20) against
    central differences at 32 random cells, h = 1e-6 relative.

    After 200 steps two things bound how well central differences can
    resolve a 1e-6 agreement: rounding noise of the two perturbed runs (every
    one of the 262,144 cells differs in its last bits, ~1e-6 of the signal at
    h = 1e-7, ~2e-7 at h = 1e-6) and perturbations that carry a minmod or
    HLLC decision somewhere in the flow across its switch point (more likely
    the larger h is).  The median cell must agree to 1e-6, 90 % of cells
    within 1e-6 and every cell within 1e-5."""
    prob = vb.kelvin_helmholtz_problem(n=512, texture=1e-2)
    errs = _fd_errors(vb, prob, 200, 20, 32, 1e-6)
    assert np.median(errs) <= 1e-6, errs
    assert np.mean(errs <= 1e-6) >= 0.9, errs
    assert errs.max() <= 1e-5, errs


def test_evolve_function_backpropagates_through_the_device_run(vb):
    """The torch.autograd bridge (rrule shape): a torch objective of the final
    state differentiates to the same gradient as the adjoint's backward."""
    prob = vb.kelvin_helmholtz_problem(n=32, texture=1e-2)
    sim = _sim(vb, prob)
    U0 = torch.tensor(sim.state(), requires_grad=True)
    UT = vb.EvolveFunction.apply(U0, sim, 6, 2)
    V = sim.backend.cell_volume()
    J = (UT[0] * UT[0]).sum() * V
    J.backward()
    # the same through the explicit API
    sim2 = _sim(vb, prob)
    adj = vb.Adjoint(sim2, 6, 2)
    adj.forward(max_steps=6)
    ref = adj.backward(vb.rho2_seed(sim2, sim2.state()))
    assert np.array_equal(UT.detach().numpy(), sim2.state())
    np.testing.assert_allclose(U0.grad.numpy(), ref, rtol=0, atol=1e-15 * np.abs(ref).max())
    adj.close()
    sim.close()
    sim2.close()


def _frozen_fd_errors(vb, prob, nsteps, every, ncells, h_rel, seed=3):
    """The device adjoint's gradient of int rho^2 against central differences
    of the step map with the branch choices of the unperturbed device run
    frozen: the torch float64 restatement (oracle/adjoint_ref.py) runs on the
    GPU, records its branch conditions while reproducing the device forward
    bit for bit, and replays them for the perturbed runs."""
    from oracle import adjoint_ref as R
    sim = _sim(vb, prob)
    U0 = sim.state()
    adj = vb.Adjoint(sim, nsteps, every)
    adj.forward(max_steps=nsteps)
    UT = sim.state()
    dts = adj.dts()
    grad = adj.backward(vb.rho2_seed(sim, UT))
    V = sim.backend.cell_volume()
    adj.close()
    sim.close()
    grid = _grid(prob)
    dev = torch.device("cuda")
    tape = R.Tape(record=True)
    with torch.no_grad():
        UT_t = R.evolve(grid, torch.tensor(U0, device=dev), dts, tape=tape)
        assert np.array_equal(UT_t.cpu().numpy(), UT)  # the device run's branches
        del UT_t
        errs = []
        for cell in np.random.default_rng(seed).choice(U0.shape[1], size=ncells, replace=False):
            h = h_rel * U0[0, cell]
            Up = U0.copy(); Up[0, cell] += h
            Um = U0.copy(); Um[0, cell] -= h
            rp = R.evolve(grid, torch.tensor(Up, device=dev), dts, tape=tape.replay())[0]
            rm = R.evolve(grid, torch.tensor(Um, device=dev), dts, tape=tape.replay())[0]
            fd = float(((rp - rm) * (rp + rm)).sum().item()) * V / (2.0 * h)
            errs.append(abs(fd - grad[0, cell]) / abs(grad[0, cell]))
    del tape
    torch.cuda.empty_cache()
    return np.array(errs)


def test_kh512_as_specified_matches_frozen_map_differences(vb):
    """The KH 512^2 configuration exactly as specified (no texture), 200
    steps with checkpoints every 20: at 32 random cells the adjoint agrees
    with central differences of the frozen-branch map to 1e-6 relative,
    every cell."""
    prob = vb.kelvin_helmholtz_problem(n=512)
    errs = _frozen_fd_errors(vb, prob, 200, 20, 32, 1e-6)
    assert errs.max() <= 1e-6, errs


@pytest.mark.xfail(reason="the KH state as specified starts on minmod kinks (a = b = 0 in "
                          "every uniform band), where the step map has only one-sided "
                          "derivatives: central differences of the plain map measured max "
                          "1.1e-4 and 53 % of 32 cells within 1e-6 over 200 steps; the "
                          "frozen-branch check above is the one that reaches 1e-6",
                   strict=False)
def test_kh512_as_specified_plain_differences_every_cell(vb):
    """The strict form of the plain check on the configuration as specified:
    every one of 32 cells within 1e-6 (expected to fail, see the marker)."""
    prob = vb.kelvin_helmholtz_problem(n=512)
    errs = _fd_errors(vb, prob, 200, 20, 32, 1e-6)
    assert errs.max() <= 1e-6, errs


def test_long_side_matches_its_period(vb):
    """A side beyond the on-chip stage's 2^24 cells: a state that repeats every
    64 cells has the adjoint of one period.  The wrapped cells add their faces
    in another order (a few roundings of the largest term)."""
    period, copies = 64, 2 ** 18 + 1
    small, lam_s = None, np.random.default_rng(5).standard_normal((5, 2, period))
    for reps in (1, copies):
        n = period * reps
        prob = vb.smooth_random_problem((period, 2), seed=9)
        U0 = np.tile(vb.initial_state(prob).reshape(5, 2, period), (1, 1, reps)).reshape(5, -1)
        prob.dims, prob.domain = (n, 2), ((0.0, float(n)), (0.0, 2.0))
        sim = vb.Simulation(vb.B200Mesh(prob.dims, prob.domain), prob, initial=U0)
        adj = vb.Adjoint(sim, 1, 1)
        got = adj.step(0.2, np.ascontiguousarray(np.tile(lam_s, (1, 1, reps)).reshape(5, -1)))
        adj.close()
        sim.close()
        got = got.reshape(5, 2, n)
        if small is None:
            small = got
    assert n > 2 ** 24
    scale = np.abs(small).max()
    for k in (0, 1, reps // 2, reps - 1):
        assert np.abs(got[:, :, k * period:(k + 1) * period] - small).max() <= 1e-13 * scale
