"""Solver iterations recorded as one CUDA graph (conditional while node) against the host
loop: same kernels in the same order, so the same discrepancy traces, steps and outputs
(up to the order of FP64 atomic additions), for every solver, single and batched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def D():
    import dda_fft_b200
    return dda_fft_b200


def problem(oracle, n=16, x=4.0):
    occ, _ = oracle.gen_ellipsoid(n, n, n, 0.8, 0.6)
    kd = 2 * x / n
    m = complex(1.6, 0.002)
    a = kd ** 3 * (0.75 / np.pi) * (m * m - 1) / (m * m + 2)
    alpha = np.array([0, a], np.complex64)
    th = np.deg2rad(np.arange(19) * 10.0)
    ksc = np.stack([np.sin(th), np.zeros_like(th), np.cos(th)], 1)[None]
    return occ, kd, alpha, ksc


@pytest.mark.parametrize("solver", [0, 1, 2, 3])
def test_graph_equals_host_loop(D, oracle, solver):
    occ, kd, alpha, ksc = problem(oracle)
    tau = 0.6 if solver == 3 else 0.0
    out = {}
    with D.Context(occ.shape, kd) as ctx:
        for g in (False, True):
            ctx.set_solver_graph(g)
            runs0 = ctx.solver_graph_runs
            out[g] = ctx.dda_fft(occ, alpha, [0, 1], kd, (0, 0, 1), (1, 0, 0), ksc, solver=solver,
                                 tau=tau, max_step=40, err_max=1e-6)
            out[g, "runs"] = ctx.solver_graph_runs - runs0
    a, b = out[False], out[True]
    assert a["steps"] == b["steps"] and a["steps"] >= 2
    for q in ("step_min", "rolled_back", "matvecs"):
        assert a[q] == b[q], q
    assert out[True, "runs"] == 1 and out[False, "runs"] == 0
    n = a["steps"] + 1
    np.testing.assert_allclose(b["trace"][:n], a["trace"][:n], rtol=1e-9)
    for q in ("cext", "cabs"):
        assert abs(b[q] - a[q]) <= 1e-6 * abs(a[q])
    np.testing.assert_allclose(b["esc"], a["esc"], rtol=1e-5, atol=1e-7 * np.abs(a["esc"]).max())


def test_graph_batched_and_rebuilt(D, oracle):
    """Orientation batches with the graph: equal to the host loop; a different Max_Step
    rebuilds the graph and still stops where the host loop stops."""
    n, x = 16, 4.0
    occ, _ = oracle.gen_ellipsoid(n, n, n, 0.7, 0.5)
    rot = D.mc_rotations(7, 3)
    res = {}
    with D.Context(n, 2 * x / n, max_rhs=6) as ctx:
        for ms in (30, 7):
            for g in (False, True):
                ctx.set_solver_graph(g)
                cfg = D.BatchConfig(occ=occ, materials=[(1.6, 0.002)], err_max=1e-6, max_step=ms)
                res[ms, g] = ctx.orientation_solves(cfg, rot)
        assert ctx.solver_graph_runs == 2
    for ms in (30, 7):
        a, b = res[ms, False], res[ms, True]
        assert a["max_steps"] == b["max_steps"]
        np.testing.assert_allclose(b["cext"], a["cext"], rtol=1e-6)
        np.testing.assert_allclose(b["mueller"], a["mueller"], rtol=1e-5,
                                   atol=1e-7 * np.abs(a["mueller"]).max())
    assert res[7, True]["max_steps"] == 7


def test_graph_in_refinement(D, oracle):
    """Inner solves of the FP64-residual refinement run through the graph too."""
    occ, kd, alpha, ksc = problem(oracle)
    with D.Context(occ.shape, kd) as ctx:
        out = {}
        for g in (False, True):
            ctx.set_solver_graph(g)
            out[g] = ctx.dda_fft_refined(occ, alpha, [0, 1], kd, (0, 0, 1), (0, 1, 0), ksc,
                                         solver=2, err_max=1e-8, max_outer=20)
    assert out[True]["err"] <= 1e-8 and out[False]["err"] <= 1e-8
    assert abs(out[True]["cext"] - out[False]["cext"]) <= 1e-6 * abs(out[False]["cext"])


@pytest.mark.parametrize("max_step", [1, 2, 3])
@pytest.mark.parametrize("solver", [0, 2])
def test_graph_short_runs(D, oracle, solver, max_step):
    """Max_Step at the edges of the graph (1: no graph; 2: one pass; 3): the same stopping
    step, best iterate and rollback as the host loop."""
    occ, kd, alpha, ksc = problem(oracle)
    out = {}
    with D.Context(occ.shape, kd) as ctx:
        for g in (False, True):
            ctx.set_solver_graph(g)
            out[g] = ctx.dda_fft(occ, alpha, [0, 1], kd, (0, 0, 1), (1, 0, 0), ksc, solver=solver,
                                 max_step=max_step, err_max=1e-9)
    a, b = out[False], out[True]
    for q in ("steps", "step_min", "rolled_back", "matvecs"):
        assert a[q] == b[q], q
    assert a["steps"] == max_step
    np.testing.assert_allclose(b["trace"], a["trace"], rtol=1e-9)
    assert abs(b["cext"] - a["cext"]) <= 1e-6 * abs(a["cext"])


@pytest.mark.parametrize("xv", [3, 9])
def test_bounded_wait_reports_and_recovers(D, oracle, xv):
    """The x pass's bounded wait on its bulk copies (xv 3) and TMA tensor tiles (xv 9): a
    wait made to run out (self-test: after the copies have landed, a barrier phase nothing
    completes) fails the call with DDAGPU_ECUDA instead of hanging, and the context
    computes correctly again afterwards."""
    occ, kd, alpha, ksc = problem(oracle)
    rng = np.random.default_rng(2)
    p = (rng.standard_normal(occ.shape + (3,)) + 1j * rng.standard_normal(occ.shape + (3,))).astype(np.complex64)
    with D.Context(occ.shape, kd) as ctx:
        ctx.set_fast_variant(xv, 0)
        ref = ctx.convolution(p)
        ctx.selftest_wait_timeout(True)
        with pytest.raises(D.DDAGPUError, match="wait ran out"):
            ctx.convolution(p)
        with pytest.raises(D.DDAGPUError, match="wait ran out"):
            ctx.dda_fft(occ, alpha, [0, 1], kd, (0, 0, 1), (1, 0, 0), ksc, max_step=5)
        ctx.selftest_wait_timeout(False)
        again = ctx.convolution(p)
        np.testing.assert_array_equal(again, ref)
        r = ctx.dda_fft(occ, alpha, [0, 1], kd, (0, 0, 1), (1, 0, 0), ksc, max_step=5)
        assert r["steps"] >= 1


@pytest.mark.parametrize("grid,solver", [((8, 8, 8), 0), ((16, 16, 16), 2), ((4, 8, 16), 1)])
def test_recorded_single_solves_follow_their_arguments(D, oracle, grid, solver):
    """From its third call on a single solve of one shape is replayed.  Between replays everything a
    call passes changes -- occupancy, polarisabilities, activity list, incident field, directions,
    their number (the pinned staging is laid out anew) -- and each call equals the unrecorded
    solve on a context of its own (same kernels on the same inputs; 1e-6 for the order of the
    atomic sums)."""
    rng = np.random.default_rng(7)
    kd = 0.3
    base = dict(occ=(rng.random(grid) < 0.7).astype(np.int8), alpha=np.array([0, 0.02 + 0.002j], np.complex64),
                mv=[0, 1], kinc=(0, 0, 1), einc=(1, 0, 0), ksc=oracle.scattering_geometry(2, 7, 0.0, 30.0)[1])
    other = (rng.random(grid) < 0.4).astype(np.int8)
    changes = [{}, {}, {}, {}, dict(occ=other), dict(alpha=np.array([0, 0.03 + 0.001j], np.complex64)),
               dict(kinc=(1, 0, 0), einc=(0, 1, 0)), dict(ksc=oracle.scattering_geometry(4, 37, 0.0, 5.0)[1]),
               dict(ksc=base["ksc"]), {}, {}]

    def run(ctx, s):
        return ctx.dda_fft(s["occ"], s["alpha"], s["mv"], kd, s["kinc"], s["einc"], s["ksc"], solver=solver,
                           max_step=12, err_max=1e-5, trace=False)

    state = dict(base)
    with D.Context(grid, kd) as ctx:
        for ch in changes:
            state.update(ch)
            got = run(ctx, state)
            with D.Context(grid, kd) as plain:
                plain.set_solver_graph(False)
                ref = run(plain, state)
            assert np.abs(got["esc"] - ref["esc"]).max() <= 1e-6 * np.abs(ref["esc"]).max()
            for q in ("cabs", "cext"):
                assert abs(got[q] - ref[q]) <= 1e-6 * abs(ref[q])


@pytest.mark.parametrize("xv", [None, 3, 9])
def test_device_products_that_gave_up_are_reported(D, xv):
    """convolution_dev only enqueues its passes.  Where a wait ran out (the variant a context starts
    with, bulk copies, TMA tiles) the product is not a number everywhere, and synchronize() reports
    it and clears the report: the calls after it are their own."""
    import torch
    grid = (16, 16, 16)
    rng = np.random.default_rng(13)
    p = (rng.standard_normal((1, 3) + grid) + 1j * rng.standard_normal((1, 3) + grid)).astype(np.complex64)
    x = torch.from_numpy(p).cuda()
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    with D.Context(grid, 0.4) as ctx:
        if xv is not None:
            ctx.set_fast_variant(xv, 0)
        assert ctx.fast_variant[0] in (3, 9)
        ctx.convolution_dev(x, y, 1)
        ctx.synchronize()
        ref = y.cpu().numpy()
        assert np.isfinite(ref).all()
        ctx.selftest_wait_timeout(True)
        ctx.convolution_dev(x, y, 1)
        with pytest.raises(D.DDAGPUError, match="wait ran out"):
            ctx.synchronize()
        assert np.isnan(y.cpu().numpy()).all()
        ctx.selftest_wait_timeout(False)
        ctx.synchronize()
        ctx.convolution_dev(x, y, 1)
        ctx.synchronize()
        np.testing.assert_array_equal(y.cpu().numpy(), ref)


def test_autotune_takes_no_variant_that_gives_up(D, oracle):
    """Variants whose wait runs out while they are timed are not picked, and leave no error."""
    grid = (16, 16, 16)
    rng = np.random.default_rng(14)
    p = (rng.standard_normal(grid + (3,)) + 1j * rng.standard_normal(grid + (3,))).astype(np.complex64)
    ref = oracle.convolution(oracle.green_hat(*grid, 0.4), p.astype(np.complex128))
    with D.Context(grid, 0.4) as ctx:
        ctx.selftest_wait_timeout(True)
        ctx.autotune(1)
        out = ctx.convolution(p)   # (the pick does not wait)
        assert not ctx.fast_kernels or ctx.fast_variant[0] in (0, 1, 2, 6, 7, 8)
        ctx.selftest_wait_timeout(False)
        again = ctx.convolution(p)
    for o in (out, again):
        assert np.abs(o - ref).max() < 2e-5 * np.abs(ref).max()


def test_refinement_reports_its_last_product(D, oracle):
    """The product behind the last true residual of a refinement is checked like the others."""
    occ, kd, alpha, ksc = problem(oracle)
    rhs = np.ones(occ.shape + (3,), np.complex64)
    with D.Context(occ.shape, kd) as ctx:
        ctx.set_fast_variant(9, 0)
        ctx.selftest_wait_timeout(True)
        with pytest.raises(D.DDAGPUError, match="wait ran out"):
            ctx.solve_linear(occ, alpha, [0, 1], rhs, solver=2, max_step=0, refine=True)
        with pytest.raises(D.DDAGPUError, match="wait ran out"):
            ctx.dda_fft_refined(occ, alpha, [0, 1], kd, (0, 0, 1), (1, 0, 0), ksc, solver=2, max_outer=0)
        ctx.selftest_wait_timeout(False)
        ctx.solve_linear(occ, alpha, [0, 1], rhs, solver=2, max_step=0, refine=True)


def test_mueller_between_recorded_solves_keeps_the_recording(D, oracle):
    """The drop-in sample loop: solves of both polarisations, then their Mueller matrix.  The first
    mueller() after a recorded solve finds the pinned block wide enough: it does not release the
    block that the recording writes to and allocate another (milliseconds against the 40 us of a
    call; the medians of nine contexts, a factor of five between the first call and the second).
    A wider one goes by the pageable copies.  All give what a context without a recording gives,
    and the solves around them what they gave."""
    import time
    occ, kd, alpha, ksc = problem(oracle, 8)
    nrm, ksc = oracle.scattering_geometry(4, 37, 0.0, 5.0)
    wide, wksc = oracle.scattering_geometry(9, 37, 0.0, 5.0)
    k, E = (0, 0, 1), ((1, 0, 0), (0, 1, 0))
    rng = np.random.default_rng(15)
    wesc = (rng.standard_normal(wksc.shape) + 1j * rng.standard_normal(wksc.shape)).astype(np.complex64)
    times = []
    for _ in range(9):
        with D.Context(occ.shape, kd, max_rhs=2) as ctx, D.Context(occ.shape, kd, max_rhs=2) as fresh:
            def solve():
                return ctx.dda_fft(occ, alpha, [0, 1], kd, k, E[0], ksc, max_step=20, err_max=1e-3, trace=False)["esc"]

            def mueller():
                t = time.perf_counter()
                M = ctx.mueller(k, *E, ksc, nrm, esc, wesc[:4])
                return time.perf_counter() - t, M
            for _ in range(4):
                esc = solve()
            (t0, M0), (t1, M1) = mueller(), mueller()
            times.append((t0, t1))
            Mw = ctx.mueller(k, *E, wksc, wide, wesc, wesc[::-1])
            np.testing.assert_array_equal(M0, fresh.mueller(k, *E, ksc, nrm, esc, wesc[:4]))
            np.testing.assert_array_equal(M1, M0)
            np.testing.assert_array_equal(Mw, fresh.mueller(k, *E, wksc, wide, wesc, wesc[::-1]))
            again = solve()
            assert np.abs(again - esc).max() <= 1e-6 * np.abs(esc).max()
    first, second = np.median(np.array(times), axis=0)
    assert first < 5 * second


def test_pinned_blocks_go_from_context_to_context(D, oracle):
    """The third solve of a shape pins its staging.  A context gives its block back when it is closed
    and the next one takes it: its third solve does not wait for an allocation of the driver
    (1.4 to 4 ms; the medians of nine contexts, a factor of 2.5 between the third call and the
    fourth).  Contexts of several threads at once do not share a block: every call gives what an
    unrecorded one gives (1e-6: the order of the atomic sums)."""
    import threading
    import time
    occ, kd, alpha, ksc = problem(oracle, 8)

    def solve(ctx, a):
        t = time.perf_counter()
        r = ctx.dda_fft(occ, alpha * np.float32(a), [0, 1], kd, (0, 0, 1), (1, 0, 0), ksc, max_step=20, err_max=1e-3,
                        trace=False)
        return time.perf_counter() - t, r["esc"]
    scale = (1.0, 1.1, 0.9, 1.2, 1.05)
    with D.Context(occ.shape, kd) as ctx:
        ctx.set_solver_graph(False)
        ref = [solve(ctx, a)[1] for a in scale]
    times = []
    for _ in range(10):
        with D.Context(occ.shape, kd) as ctx:
            times.append([solve(ctx, a)[0] for a in scale])
    third, fourth = np.median(np.array(times[1:]), axis=0)[2:4]
    assert third < 2.5 * fourth
    worst = []

    def worker():
        for _ in range(4):
            with D.Context(occ.shape, kd) as ctx:
                for _ in range(3):
                    for a, e in zip(scale, ref):
                        worst.append(np.abs(solve(ctx, a)[1] - e).max() / np.abs(e).max())
    threads = [threading.Thread(target=worker) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(worst) == 4 * 4 * 3 * len(scale) and max(worst) <= 1e-6


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("grid,solver", [((8, 8, 8), 0), ((16, 8, 4), 2)])
def test_replayed_solves_take_every_value_of_their_call(D, oracle, grid, solver, mode):
    """Replays of one recording with new values of the same shape -- the activity list (a material
    switched off and on), directions of the same number (with mode 2 by kz groups, one plan after
    the other and the first again), an incident field -- then recordings for a second and again
    the first number of directions, whose pinned layouts differ, with Mueller averages in between.
    Each call equals the unrecorded one on a context of its own (1e-6: the order of the atomic
    sums, at discrepancies near 1e-3)."""
    rng = np.random.default_rng(17)
    kd = 0.3
    geom = lambda step, na: oracle.scattering_geometry(3, na, 0.0, step)
    nrm, a = geom(30.0, 7)
    b, c, many = geom(25.0, 7)[1], geom(12.0, 7)[1], geom(5.0, 37)[1]
    base = dict(mv=[0, 1, 1], kinc=(0, 0, 1), einc=(1, 0, 0), ksc=a)
    occ = (rng.integers(0, 3, grid) * (rng.random(grid) < 0.8)).astype(np.int8)
    alpha = np.array([0, 0.02 + 0.002j, 0.03 + 0.001j], np.complex64)
    changes = [{}, {}, {}, dict(mv=[0, 1, 0]), dict(mv=[0, 0, 1]), dict(mv=[0, 1, 1]), dict(ksc=b), dict(ksc=a),
               dict(ksc=c, einc=(0, 1, 0)), dict(ksc=a), dict(ksc=many), {}, {}, {}, dict(einc=(1, 0, 0)),
               dict(ksc=b), {}, {}, dict(ksc=a)]

    def run(ctx, s):
        return ctx.dda_fft(occ, alpha, s["mv"], kd, s["kinc"], s["einc"], s["ksc"], solver=solver, max_step=6,
                           err_max=1e-5, trace=False)
    state = dict(base)
    with D.Context(grid, kd, max_rhs=2) as ctx, D.Context(grid, kd, max_rhs=2) as plain:
        ctx.set_farfield_mode(mode)
        plain.set_farfield_mode(mode)
        plain.set_solver_graph(False)
        runs = ctx.solver_graph_runs
        for ch in changes:
            state.update(ch)
            got, ref = run(ctx, state), run(plain, state)
            assert np.abs(got["esc"] - ref["esc"]).max() <= 1e-6 * np.abs(ref["esc"]).max()
            for q in ("cabs", "cext"):
                assert abs(got[q] - ref[q]) <= 1e-6 * abs(ref[q])
            if state["ksc"].shape == a.shape:
                args = ((0, 0, 1), (1, 0, 0), (0, 1, 0), state["ksc"], nrm, got["esc"], got["esc"][::-1])
                np.testing.assert_array_equal(ctx.mueller(*args), plain.mueller(*args))
        assert ctx.solver_graph_runs - runs >= 13
