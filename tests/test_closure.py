"""The learned subgrid closure: the oracle's own consistency on the CPU; on the
GPU the tensor-core inference, the gradients and an Adam step against the
oracle, the training data against the oracle's restatement, the untrained
network against plain Smagorinsky, and what training gains over c = 0 on
held-out data."""
import numpy as np
import pytest

from oracle import closure as OC


def _rand_params(seed, scale=0.5):
    r = np.random.default_rng(seed)
    w = r.uniform(-scale, scale, OC.N_PARAMS)
    return w.astype(np.float32).astype(np.float64)


# ---------------------------------------------------------------- oracle, CPU
def test_oracle_backward_is_the_chain_rule(monkeypatch):
    """With the bfloat16 roundings switched off the oracle's gradients equal
    central finite differences of its loss."""
    monkeypatch.setattr(OC, "bf16", lambda a: np.asarray(a, np.float64))
    r = np.random.default_rng(2)
    w = r.uniform(-0.4, 0.4, OC.N_PARAMS)
    x = r.uniform(-1, 1, (7, OC.N_IN))
    y = r.uniform(-1, 1, 7)
    _, g = OC.gradients(w, x, y)
    for q in list(range(0, OC.N_PARAMS, 97)) + [OC.B3, OC.W3 + 5, OC.B1 + 3]:
        e = np.zeros(OC.N_PARAMS)
        e[q] = 1e-6
        fd = (OC.gradients(w + e, x, y)[0] - OC.gradients(w - e, x, y)[0]) / 2e-6
        assert abs(fd - g[q]) < 1e-7 + 1e-5 * abs(fd), q


def test_oracle_inputs_known_answers():
    s = np.array([[0, 0, 0, 1e-3, 0, 0], [2e-3, -1e-3, -1e-3, 0, 0, 0]])
    x = OC.features(s, np.array([1.0, 1.002]), np.array([0.05, 0.0]), np.zeros(2), np.zeros(2),
                    np.array([3.0, 20.0]), 0.004, np.array([1e-5, 2e-5]), 0.05)
    # pure shear: all of S:S off the diagonal, tr(S^3) = 0; |S| = sqrt(2 * 2 d^2) = 2d
    assert x[0, 2] == pytest.approx(1.0) and abs(x[0, 1]) < 1e-12 and x[0, 0] == pytest.approx(100 * 2e-3)
    # axisymmetric extension: no off-diagonal part, tr(S^3) > 0
    assert x[1, 2] == 0.0 and x[1, 1] > 0
    assert x[0, 3] == pytest.approx(1.0) and x[0, 4] == pytest.approx(1.0)
    assert x[1, 5] == pytest.approx(0.1 * 0.002 / 0.0025)
    assert x[0, 6] == pytest.approx(3 / 8) and x[1, 6] == 1.0
    assert x[0, 7] == pytest.approx(10 * 1e-5 / 0.004) and x[0, 8] == pytest.approx(0.8)


def test_oracle_wall_distance():
    solid = np.zeros((6, 7, 9), bool)
    solid[3, 3, 4] = True
    d = OC.wall_distance(solid)
    z, y, x = np.indices(solid.shape)
    manhattan = np.abs(x - 4) + np.minimum(np.abs(y - 3), 7 - np.abs(y - 3)) + np.minimum(np.abs(z - 3), 6 - np.abs(z - 3))
    assert np.array_equal(d, np.where(manhattan <= 8, manhattan, 255))


def test_bf16_rounding_ties_to_even():
    vals = np.array([1.0, 1.0 + 2 ** -8, 1.0 + 3 * 2 ** -8, -2.5, 1e-40], np.float32)
    r = OC.bf16(vals)
    assert r[0] == 1.0 and r[1] == 1.0 and r[2] == 1.0 + 2 ** -6 and r[3] == -2.5


# ---------------------------------------------------------------- GPU
pytest_gpu = pytest.mark.gpu


def _closure(w=None, seed=1):
    from pocketwind_gb300.closure import Closure
    c = Closure(seed)
    if w is not None:
        c.params = w
    return c


@pytest_gpu
def test_tensor_core_inference_matches_oracle():
    w = _rand_params(3)
    c = _closure(w)
    x = np.random.default_rng(4).uniform(-1.5, 1.5, (1000, OC.N_IN)).astype(np.float32)
    got = c.eval(x)
    ref, _ = OC.forward(w, x)
    assert np.abs(got - ref).max() < 3e-2 * max(1.0, np.abs(ref).max())
    assert np.corrcoef(got, ref)[0, 1] > 0.999
    c.destroy()


@pytest_gpu
def test_untrained_network_outputs_zero():
    c = _closure(seed=9)
    x = np.random.default_rng(5).uniform(-1, 1, (300, OC.N_IN)).astype(np.float32)
    assert np.all(c.eval(x) == 0.0)
    c.destroy()


@pytest_gpu
def test_gradients_match_oracle():
    w = _rand_params(6, 0.3)
    c = _closure(w)
    r = np.random.default_rng(7)
    x = r.uniform(-1, 1, (512, OC.N_IN)).astype(np.float32)
    y = r.uniform(-1, 1, 512).astype(np.float32)
    loss, g = c.gradients(x, y)
    rl, rg = OC.gradients(w, x, y)
    assert loss == pytest.approx(rl, rel=2e-2)
    assert np.linalg.norm(g - rg) / np.linalg.norm(rg) < 2e-2
    c.destroy()


@pytest_gpu
@pytest.mark.parametrize("count", [1, 31, 33, 4863, 4865, 77825])
def test_gradients_match_oracle_at_group_edges(count):
    """Counts around a warp's 32 samples, a block's first warp (152 blocks) and the
    whole grid (a warp's second group).  The last sample's target outweighs all
    others, so leaving it out shows; the tolerance is that of the network's
    rounding (one bfloat16 step of an activation is 0.4%)."""
    w = _rand_params(6, 0.3)
    c = _closure(w)
    r = np.random.default_rng(count)
    x = r.uniform(-1, 1, (count, OC.N_IN)).astype(np.float32)
    y = r.uniform(-1, 1, count).astype(np.float32)
    y[-1] = 30.0 * np.sqrt(count)
    loss, g = c.gradients(x, y)
    rl, rg = OC.gradients(w, x, y)
    assert loss == pytest.approx(rl, rel=2e-2)
    assert np.linalg.norm(g - rg) / np.linalg.norm(rg) < 2e-2
    c.destroy()


@pytest_gpu
def test_one_adam_step_matches_oracle():
    """A dataset of one repeated sample makes every drawn batch the same, so one
    training step is one Adam step on that sample's gradient."""
    w = _rand_params(8, 0.3)
    c = _closure(w)
    x = np.tile(np.random.default_rng(9).uniform(-1, 1, (1, OC.N_IN)), (256, 1)).astype(np.float32)
    y = np.full(256, 0.7, np.float32)
    c.set_dataset(x, y)
    c.train(1, batch=256, lr=1e-2)
    _, g = OC.gradients(w, x, y)
    ref, _, _ = OC.adam(w, np.zeros_like(w), np.zeros_like(w), g, 1, 1e-2)
    got = c.params.astype(np.float64)
    moved = np.abs(ref - w) > 1e-4
    assert moved.sum() > 100
    assert np.abs(got - ref)[moved].max() < 2e-3
    c.destroy()


@pytest_gpu
def test_training_fits_a_smooth_target():
    r = np.random.default_rng(10)
    x = r.uniform(-1, 1, (20000, OC.N_IN)).astype(np.float32)
    y = (0.5 * np.tanh(2 * x[:, 0]) - 0.3 * x[:, 3] * x[:, 4]).astype(np.float32)
    c = _closure(seed=3)
    c.set_dataset(x, y)
    first, last = c.train(400, batch=4096, lr=3e-3)
    assert last < 0.1 * first
    c.destroy()


def _fine_run(steps=300):
    from pocketwind_gb300 import cases, solver
    v = cases.vehicle_case(64)
    grid = v.grid()
    s = solver.GpuSolver.create(v.layout, grid, solver.SolverParams(tau0=v.tau0, u_in=0.05, les=True,
                                                                     operator="reg"))
    s.step(steps, True)
    return v, grid, s


@pytest_gpu
def test_training_data_match_oracle():
    from pocketwind_gb300.closure import Closure
    v, grid, s = _fine_run()
    c = Closure(1)
    nu0 = 0.5 * (v.tau0 - 0.5) / 3
    n = c.add_samples(s, nu0)
    x, y = c.dataset()
    walls = np.isin(grid.flags & 7, [1, 2, 3])
    q, solid = OC.coarsen(s.macros(), walls, v.layout)
    d = OC.wall_distance(solid)
    rx, ry = OC.samples(q, d, nu0, 0.05)
    assert n == len(rx) > 1000
    assert np.abs(y - ry).max() < 1e-3 * max(1.0, np.abs(ry).max()) + 1e-3
    assert np.abs(x - rx).max() < 1e-3 * np.abs(rx).max(axis=0).max()
    c.destroy()
    s.destroy()


@pytest_gpu
@pytest.mark.parametrize("walls,lateral", [("bb", "periodic"), ("bouzidi", "periodic"), ("bb", "free-slip")])
def test_untrained_closure_is_plain_smagorinsky(walls, lateral):
    """An untrained network (c = 0) attached to a domain reproduces plain
    Smagorinsky, with halfway walls and with interpolated (Bouzidi) walls, whose
    wall cells run in the same edge kernel with or without the closure
    (walls.wgsl:6-21), and with free-slip faces, where the one-cell closure
    kernel runs."""
    from pocketwind_gb300 import cases, solver
    from pocketwind_gb300.closure import Closure
    v = cases.vehicle_case(64)
    v.walls = walls
    grid = v.grid()
    mk = lambda: solver.GpuSolver.create(v.layout, grid, solver.SolverParams(tau0=v.tau0, u_in=0.05, les=True,
                                                                             operator="reg", walls=walls,
                                                                             lateral=lateral))
    plain, closed = mk(), mk()
    c = Closure(5)
    c.attach(closed)
    # With c = 0 the closure's relaxation time tau0 + (tau_s - tau0) can differ
    # from tau_s in the last bit, and this flow at tau0 = 0.509 amplifies
    # rounding differences about tenfold every ten steps, so the comparison is
    # made at step 20.
    plain.step(20, True)
    closed.step(20, True)
    a, b = closed.populations().astype(np.float64), plain.populations().astype(np.float64)
    assert np.linalg.norm(a - b) / np.linalg.norm(b) < 1e-5
    ua, ub = closed.macros()[:, 1:].astype(np.float64), plain.macros()[:, 1:].astype(np.float64)
    assert np.linalg.norm(ua - ub) / np.linalg.norm(ub) < 1e-5
    closed.encode_force()
    plain.encode_force()
    fa, fb = closed.read_force(), plain.read_force()
    assert abs(fa.fx - fb.fx) < 1e-4 * abs(fb.fx)
    c.destroy()


@pytest_gpu
@pytest.mark.parametrize("precision", ["f16", "bf16"])
def test_untrained_closure_16bit_within_storage_noise(precision):
    """With 16-bit storage the closure's kernel pairs cells x and x + 32 of a
    row, the plain step's cell-pair kernel x and x + 1, so the two round each
    code with another dither realization (same probabilities); the floor
    layer runs in the floor kernel beside both.  An untrained network then
    stays within the storage's rounding noise of plain Smagorinsky: after 40
    steps of the 64x32x32 vehicle, velocity within relative L2 2e-3 (f16) and
    1e-2 (bf16), the tolerances of the floor kernel's own check."""
    from pocketwind_gb300 import cases, solver
    from pocketwind_gb300.closure import Closure
    v = cases.vehicle_case(64)
    grid = v.grid()
    mk = lambda: solver.GpuSolver.create(v.layout, grid, solver.SolverParams(tau0=v.tau0, u_in=0.05, les=True,
                                                                             operator="reg", precision=precision))
    plain, closed = mk(), mk()
    c = Closure(5)
    c.attach(closed)
    plain.step(40, True)
    closed.step(40, True)
    ua, ub = closed.macros()[:, 1:].astype(np.float64), plain.macros()[:, 1:].astype(np.float64)
    assert np.isfinite(ua).all()
    assert np.linalg.norm(ua - ub) / np.linalg.norm(ub) < (2e-3 if precision == "f16" else 1e-2)
    c.destroy()


@pytest_gpu
def test_closure_step_is_deterministic():
    """With a network whose output is not zero, two runs of the closure step
    (the tensor-core kernel with the edge and floor kernels beside it) give the
    same stored codes bit for bit after 40 steps."""
    from pocketwind_gb300 import cases, solver
    v = cases.vehicle_case(64)
    grid = v.grid()
    net = _closure(_rand_params(9))
    runs = []
    for _ in range(2):
        s = solver.GpuSolver.create(v.layout, grid, solver.SolverParams(tau0=v.tau0, u_in=0.05, les=True,
                                                                         operator="reg", precision="f16"))
        net.attach(s)
        s.step(40, True)
        runs.append(s.populations_raw().view(np.uint8).copy())
        s.destroy()
    net.destroy()
    assert np.array_equal(runs[0], runs[1])


@pytest_gpu
@pytest.mark.parametrize("nx", [32, 128])
def test_closure_step_hands_out_every_tile(nx):
    """Tiles handed out beyond the blocks' first ones (128) and none (32): steps one by
    one and in one call, and steps from a state loaded at once and after an odd number
    of further steps, give the same stored codes bit for bit."""
    from pocketwind_gb300 import cases, solver
    v = cases.vehicle_case(nx)
    net = _closure(_rand_params(9))

    def codes(single, more=None):
        s = solver.GpuSolver.create(v.layout, v.grid(), solver.SolverParams(tau0=v.tau0, u_in=0.05, les=True,
                                                                             operator="reg", precision="f16"))
        net.attach(s)
        s.step(2, True)
        if more is not None:
            blob = s.save_checkpoint()
            s.step(more)
            s.load_checkpoint(blob)
        for n in [1] * 71 if single else [71]:
            s.step(n)
        out = s.populations_raw().view(np.uint8).copy()
        s.destroy()
        return out

    assert np.array_equal(codes(True), codes(False))
    assert np.array_equal(codes(False, more=0), codes(False, more=1))
    net.destroy()


@pytest_gpu
def test_trained_closure_beats_smagorinsky_on_held_out_data():
    """What the network gains over the method without it: after training on
    filtered fine-grid samples its a-priori error on held-out samples is below
    that of c = 0 (plain Smagorinsky), and a coarse run with it attached stays
    finite and differs from Smagorinsky."""
    from pocketwind_gb300 import cases, solver
    from pocketwind_gb300.closure import Closure
    v, grid, s = _fine_run(400)
    c = Closure(2)
    nu0 = 0.5 * (v.tau0 - 0.5) / 3
    c.add_samples(s, nu0)
    s.step(100, True)
    c.add_samples(s, nu0)
    x, y = c.dataset()
    r = np.random.default_rng(11)
    perm = r.permutation(len(x))
    hold, train = perm[: len(x) // 5], perm[len(x) // 5:]
    c.set_dataset(x[train], y[train])
    c.train(600, batch=8192, lr=2e-3)
    mse_net = float(np.mean((c.eval(x[hold]) - y[hold]) ** 2))
    mse_smag = float(np.mean(y[hold] ** 2))
    assert mse_net < 0.8 * mse_smag
    coarse = cases.vehicle_case(32)
    cg = coarse.grid()
    cs = solver.GpuSolver.create(coarse.layout, cg, solver.SolverParams(tau0=coarse.tau0, u_in=0.05, les=True,
                                                                         operator="reg"))
    c.attach(cs)
    cs.step(200, True)
    assert np.isfinite(cs.macros()).all()
    c.destroy()
    s.destroy()


# sizes whose long runs are captured (64 steps a graph) and, the last, one past the line;
# 65 and 129 steps leave one step behind the graphs; with 1,352 tiles the captured blocks
# take theirs from the counter
@pytest_gpu
@pytest.mark.parametrize("precision,operator,layout", [
    ("f32", "reg", (64, 32, 32)), ("f16", "reg", (33, 17, 17)), ("f32", "trt", (104, 52, 52)),
    ("f32", "reg", (72, 36, 36))])
@pytest.mark.parametrize("count", [64, 65, 129])
def test_long_closure_runs_equal_single_steps(precision, operator, layout, count):
    from pocketwind_gb300 import geometry, meshes, solver
    net = _closure(_rand_params(9))
    grid = geometry.voxelize(meshes.icosphere([n / 2.2 for n in layout], min(layout) / 5, 3), None, layout, True)
    got = []
    for calls in ([1] * count, [count]):
        s = solver.GpuSolver.create(layout, grid, solver.SolverParams(tau0=0.56, u_in=0.05, les=True,
                                                                      operator=operator, precision=precision))
        net.attach(s)
        s.inject_nan()
        s.step(1, True)
        assert s.guard_unstable()
        s.reset()
        for k, n in enumerate(calls):
            s.step(n, k + 1 == len(calls))
        assert not s.guard_unstable()
        s.encode_force()
        f = s.read_force()
        got.append((s.populations_raw().view(np.uint8), s.macros(), (f.fx, f.fy, f.fz)))
        s.destroy()
    net.destroy()
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2]


@pytest_gpu
def test_long_closure_runs_of_small_domains_are_captured():
    """A step of 256 in a call costs less than one of 8 in calls of 8 (64x32x32: 12.4 and 14.3
    us; launched early 13.7)."""
    import time
    from pocketwind_gb300 import cases, solver
    v = cases.vehicle_case(64)
    s = solver.GpuSolver.create(v.layout, v.grid(), v.params("f32"))
    net = _closure(_rand_params(9))
    net.attach(s)
    best = []
    for count in (8, 256):
        times = []
        for _ in range(40):
            t = time.perf_counter()
            for _ in range(256 // count):
                s.step(count)
            s.guard_unstable()
            times.append(time.perf_counter() - t)
        best.append(min(times))
    s.destroy()
    net.destroy()
    assert best[1] < 0.95 * best[0], best
