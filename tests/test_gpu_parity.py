"""GPU parity: libddagpu (through its C ABI) against the FP64 oracle and the reference's
golden outputs.  Tolerances are written per test: the kernels compute in float32 with
FP64 reductions, so a single convolution agrees with the FP64 oracle to ~1e-6 of its
largest element; solver outputs are compared under the float-noise gate
max(1e-4 relative, 2 x |float reference - FP64 reference|)."""
import numpy as np
import pytest

from pyoracle import orientation_solves

pytestmark = pytest.mark.gpu

CONV_TOL = 2e-5     # max |gpu - fp64| / max |fp64| for one convolution


def rel(a, b):
    a, b = np.asarray(a), np.asarray(b)
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def crand(rng, shape):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)


@pytest.fixture(scope="module")
def D():
    import dda_fft_b200
    return dda_fft_b200


FAST = {16, 32, 64, 128}


@pytest.mark.parametrize("grid", [(2, 2, 2), (4, 4, 4), (8, 8, 8), (16, 16, 16), (32, 32, 32),
                                  (8, 16, 8), (16, 4, 32), (64, 64, 64), (16, 64, 32),
                                  (64, 16, 16), (32, 16, 64), (128, 16, 16), (16, 128, 32),
                                  (32, 16, 128)])
@pytest.mark.parametrize("conj", [False, True])
@pytest.mark.parametrize("fast", [False, True])
def test_convolution_vs_oracle(D, oracle, grid, conj, fast):
    if fast and not set(grid) <= FAST:
        pytest.skip("specialised passes cover edges 16..128")
    rng = np.random.default_rng(sum(grid) + conj)
    kd = 2 * 3.0 / grid[0]
    p = crand(rng, grid + (3,))
    with D.Context(grid, kd) as ctx:
        ctx.set_kernels(fast)
        out = ctx.convolution(p, conj=conj)
    ref = oracle.convolution(oracle.green_hat(*grid, kd), p.astype(np.complex128), conj=conj)
    assert rel(out, ref) < CONV_TOL


@pytest.mark.parametrize("n", [8, 16])
def test_convolution_vs_reference_golden(D, golden, n):
    """Against the reference's own float Convolution (CT) on the golden inputs."""
    kd = float(golden[f"conv{n}_kd"])
    p = golden[f"conv{n}_p"]
    with D.Context(n, kd) as ctx:
        out = ctx.convolution(p)
        outc = ctx.convolution(p, conj=True)
    assert rel(out, golden[f"conv{n}_out"]) < CONV_TOL
    assert rel(outc, golden[f"conv{n}_out_conj"]) < CONV_TOL


def test_set_green_from_reference_cmA(D, golden):
    """Uploading the reference's own cmA (its float Green tensor FFT) gives its output."""
    kd = float(golden["conv8_kd"])
    with D.Context(8, kd) as ctx:
        ctx.set_green(golden["green8_hat"])
        out = ctx.convolution(golden["conv8_p"])
    assert rel(out, golden["conv8_out"]) < 2e-6


def test_convolution_rectangular_golden(D, golden):
    p = golden["convrect_p"]
    with D.Context(p.shape[:3], float(golden["convrect_kd"])) as ctx:
        out = ctx.convolution(p)
    assert rel(out, golden["convrect_out"]) < CONV_TOL


def _green_point(r):
    """G(r) of CreateAMatrix (dda_func.cpp:110-141) in FP64, as a 3x3 matrix."""
    r = np.asarray(r, float)
    r2 = r @ r
    r1 = np.sqrt(r2)
    c2 = np.exp(1j * r1) / (r1 * r2)
    return c2 * (r2 - 1 + 1j * r1) * np.eye(3) + c2 * (3 - r2 - 3j * r1) / r2 * np.outer(r, r)


def test_convolution_128_impulse(D):
    """Size-independent check at 128^3: the response to a point dipole is the Green tensor
    itself, G(r - r0) e, sampled at scattered lattice points."""
    n, kd = 128, 2 * 16.0 / 128
    p = np.zeros((n, n, n, 3), np.complex64)
    r0 = (37, 90, 64)
    e = np.array([0.3 + 0.1j, -0.7, 0.2j])
    p[r0] = e
    with D.Context(n, kd) as ctx:
        out = ctx.convolution(p)
    rng = np.random.default_rng(5)
    pts = [tuple(rng.integers(0, n, 3)) for _ in range(64)] + [(0, 0, 0), (127, 127, 127)]
    worst, scale = 0.0, 0.0
    for q in pts:
        if q == r0:
            continue
        g = _green_point((np.array(q) - np.array(r0)) * kd) @ e
        worst = max(worst, np.abs(out[q] - g).max())
        scale = max(scale, np.abs(g).max())
    assert worst < 1e-4 * scale + 1e-7
    assert np.abs(out[r0]).max() < 1e-4 * scale + 1e-7     # G(0) = 0


@pytest.mark.parametrize("grid", [(128, 128, 128), (128, 64, 128), (64, 128, 32)])
def test_fast_and_generic_agree_128(D, grid):
    """The specialised 128-edge passes against the generic passes on the same random
    fields (both float32; two right-hand sides, plain and conjugate)."""
    import torch
    rng = np.random.default_rng(5)
    p = crand(rng, (2, 3) + grid)
    with D.Context(grid, 0.2, max_rhs=2) as ctx:
        assert ctx.fast_kernels
        x = torch.from_numpy(p).cuda()
        outs = {}
        for fast in (True, False):
            for conj in (False, True):
                ctx.set_kernels(fast)
                y = torch.empty_like(x)
                ctx.convolution_dev(x, y, 2, conj=conj)
                torch.cuda.synchronize()
                outs[fast, conj] = y.cpu().numpy()
    for conj in (False, True):
        assert rel(outs[True, conj], outs[False, conj]) < 2e-6


@pytest.mark.parametrize("grid", [(16, 16, 16), (64, 64, 64), (128, 64, 32), (32, 128, 16)])
def test_fast_launch_variants_agree(D, oracle, grid):
    """Every launch variant of the specialised passes -- tiles, bulk copies, TMA tensor
    tiles and both line factorisations of the x pass (the radix schedules) -- gives the
    oracle's convolution, and the autotuner's pick does too."""
    import torch
    rng = np.random.default_rng(9)
    p = crand(rng, (2, 3) + grid)
    kd = 2 * 3.0 / grid[0]
    ref = [oracle.convolution(oracle.green_hat(*grid, kd), p[r].transpose(1, 2, 3, 0).astype(np.complex128))
           for r in range(2)] if max(grid) <= 64 else None
    with D.Context(grid, kd, max_rhs=2) as ctx:
        x = torch.from_numpy(p).cuda()
        outs = []
        for vx in range(12):         # 3..5: bulk copies; 6..8: second factorisation; 9..11: TMA tiles
            for vyz in (0, 1, 2):
                ctx.set_fast_variant(vx, vyz)
                assert ctx.fast_variant == (vx, vyz)
                y = torch.empty_like(x)
                ctx.convolution_dev(x, y, 2)
                torch.cuda.synchronize()
                outs.append(y.cpu().numpy())
        ctx.autotune(2)
        y = torch.empty_like(x)
        ctx.convolution_dev(x, y, 2)
        torch.cuda.synchronize()
        outs.append(y.cpu().numpy())
    for o in outs[1:]:
        assert rel(o, outs[0]) < 2e-6
    if ref is not None:
        for r in range(2):
            assert rel(outs[0][r].transpose(1, 2, 3, 0), ref[r]) < CONV_TOL


def test_generic_tiling_of_one_context_keeps_another_working(D, oracle):
    """The generic passes' shared-memory limits are per process: tuning a second context
    on a smaller generic lattice must not lower what the first one launches with."""
    rng = np.random.default_rng(21)
    g1, g2 = (128, 8, 128), (8, 4, 8)
    p1 = crand(rng, g1 + (3,))
    with D.Context(g1, 0.05) as big:
        big.set_kernels(False)
        before = big.convolution(p1)
        with D.Context(g2, 0.5) as small:
            small.set_kernels(False)
            small.set_tiling(4, 2)
            small.autotune(1)
            small.convolution(crand(rng, g2 + (3,)))
        after = big.convolution(p1)
    assert np.array_equal(before, after)


def test_convolution_linearity_128(D):
    n, kd = 128, 0.25
    rng = np.random.default_rng(9)
    x = crand(rng, (n, n, n, 3))
    y = crand(rng, (n, n, n, 3))
    with D.Context(n, kd) as ctx:
        a, b, c = ctx.convolution(x), ctx.convolution(y), ctx.convolution(x + 2 * y)
    assert rel(c, a + 2 * b) < 1e-5


@pytest.mark.parametrize("name", ["cg", "aa", "bicgstab", "simple", "simple_div"])
def test_solver_vs_oracle_and_reference(D, golden, oracle, name):
    g = golden
    solver, tau, model, *einc = g[f"solve_{name}_cfg"]
    kd = float(g["solve_kd"])
    occ = g["solve_occ"]
    n = occ.shape[0]
    ksc = g["solve_ksc"]
    alpha = g[f"solve_{name}_alpha"]
    mv = np.array([0, 1])
    with D.Context(n, kd) as ctx:
        r = ctx.dda_fft(occ, alpha, mv, kd, (0, 0, 1), einc, ksc, solver=int(solver), tau=tau,
                        max_step=8, err_max=1e-9)
    o = oracle.dda_fft(occ, alpha.astype(np.complex128), mv, kd, (0, 0, 1), einc,
                       oracle.green_hat(n, n, n, kd), ksc.astype(np.float64), solver=int(solver),
                       tau=tau, max_step=8, err_max=1e-9)
    assert len(r["trace"]) == len(o["trace"])
    # per-step discrepancy: float solver vs FP64 oracle
    assert np.abs(r["trace"] - o["trace"]).max() <= 2e-3 * np.abs(o["trace"]).max()
    assert r["step_min"] == o["step_min"]
    for q in ("cext", "cabs"):
        ref32, ref64 = float(g[f"solve_{name}_{q}"]), float(g[f"solve_{name}64_{q}"])
        gate = max(1e-4 * abs(ref64), 2 * abs(ref32 - ref64))
        assert abs(r[q] - ref64) <= gate, (q, r[q], ref32, ref64)
    assert rel(r["esc"], o["esc"]) < 2e-3


def test_farfield_cabscext_mueller_vs_oracle(D, oracle):
    rng = np.random.default_rng(3)
    n, kd = 16, 0.4
    occ, _ = oracle.gen_ellipsoid(n, n, n, 0.7, 0.5)
    occ[occ == 1] = rng.integers(1, 3, size=int((occ == 1).sum()))
    alpha = np.array([0, 0.01 + 0.001j, 0.02 + 0.004j], np.complex64)
    mv = np.array([0, 1, 1])
    p = crand(rng, (n, n, n, 3))
    p[occ == 0] = 0
    nrm, ksc = oracle.scattering_geometry(3, 19, 0.0, 10.0)
    kinc = np.array([0.0, 0.6, 0.8])
    e0 = np.array([1.0, 0, 0], complex)
    e1 = np.array([0, 0.8, -0.6], complex)
    with D.Context(n, kd, max_rhs=2) as ctx:
        esc = ctx.farfield(occ, mv, kd, p, ksc)
        ca, ce = ctx.cabscext(occ, alpha, kd, kinc, e0, p)
        escb = ctx.farfield(occ, mv, kd, p * (0.3 - 0.2j), ksc)
        M = ctx.mueller(kinc, e0, e1, ksc, nrm, esc.reshape(3, 19, 3), escb.reshape(3, 19, 3))
    ref = np.array([oracle.farfield(occ, mv, kd, p, k) for k in ksc.reshape(-1, 3)])
    assert rel(esc, ref) < 1e-5
    oca, oce = oracle.cabscext(occ, alpha, kd, kinc, e0, p)
    assert abs(ca - oca) < 1e-5 * abs(oca) and abs(ce - oce) < 1e-5 * max(abs(oce), 1e-3)
    Mo = np.zeros((19, 4, 4))
    for a in range(19):
        for pl in range(3):
            Mo[a] += oracle.jones_mueller(kinc, ksc[pl, a], nrm[pl], e0, e1, esc.reshape(3, 19, 3)[pl, a],
                                          escb.reshape(3, 19, 3)[pl, a])[1] / 3
    assert rel(M, Mo) < 1e-5


def test_monte_carlo_batch_vs_reference(D, golden, oracle):
    """4 MC orientations (seed 7) of a 16^3 ellipsoid, batched: vs the FP64 reference."""
    n, x = 16, 3.0
    occ, _ = oracle.gen_ellipsoid(n, n, n, 0.7, 0.5)
    rot = D.mc_rotations(7, 4)
    cfg = D.BatchConfig(occ=occ, materials=[(1.55, 0.005)], nplanes=2, err_max=1e-3)
    with D.Context(n, 2 * x / n, max_rhs=8) as ctx:
        r = ctx.orientation_solves(cfg, rot)
    ref64, ref32 = golden["mc16_n4_64"], golden["mc16_n4"]
    for k, q in ((0, "cabs"), (1, "cext")):
        gate = max(1e-4 * abs(ref64[k]), 2 * abs(ref32[k] - ref64[k]))
        assert abs(r[q].sum() - ref64[k]) <= gate, (q, r[q].sum(), ref32[k], ref64[k])
    M = r["mueller"].sum(axis=0).ravel()
    scale = np.abs(ref64[2:]).max()
    sig = np.abs(ref64[2:]) > 1e-3 * scale
    err = np.abs(M - ref64[2:])[sig] / np.abs(ref64[2:])[sig]
    assert err.max() < 1e-3


def test_config1_end_to_end(D, golden, oracle):
    """Config 1 (32^3 sphere, x=2, CM, CG, 19 angles, fixed orientation) against the
    reference executable's .dat."""
    txt = bytes(golden["c1_dat"]).decode().strip().split("\n")
    head = txt[0].replace("\t", " ").split()
    ca, ce = float(head[0].split("=")[1]), float(head[1].split("=")[1])
    rows = np.array([[float(v) for v in ln.split()] for ln in txt[1:]])[:, 1:]
    occ, _ = oracle.gen_ellipsoid(32, 32, 32)
    cfg = D.BatchConfig(occ=occ, materials=[(1.5, 0.01)])
    with D.Context(32, 2 * 2.0 / 32, max_rhs=2) as ctx:
        r = ctx.orientation_solves(cfg, D.fixed_rotation(0, 0, 0)[None])
    o = orientation_solves(oracle, 32, 2.0, [(1.5, 0.01)], 1)
    assert abs(r["cabs"][0] - o["cabs"]) < 1e-4 * o["cabs"]
    assert abs(r["cext"][0] - o["cext"]) < 1e-4 * o["cext"]
    assert abs(r["cabs"][0] - ca) < 1e-4 * ca
    assert abs(r["cext"][0] - ce) < 3e-4 * ce
    M = r["mueller"][0].reshape(-1, 16)
    scale = np.abs(rows).max()
    sig = np.abs(rows) > 1e-3 * scale
    assert (np.abs(M - rows) / np.maximum(np.abs(rows), 1e-30))[sig].max() < 1e-3
    Mo = o["mueller"].reshape(-1, 16)
    sig = np.abs(Mo) > 1e-3 * np.abs(Mo).max()
    assert (np.abs(M - Mo) / np.maximum(np.abs(Mo), 1e-30))[sig].max() < 1e-4


def test_ldr_bicgstab_batch(D, golden, oracle):
    """LDR (per-polarisation alpha) + BiCGStab + 3 planes at 16^3 vs the FP64 reference."""
    occ, _ = oracle.gen_ellipsoid(16, 16, 16)
    cfg = D.BatchConfig(occ=occ, materials=[(1.5, 0.01)], polarizability=5, solver=2,
                        nplanes=3, theta_step=5.0, max_step=100)
    with D.Context(16, 2 * 4.0 / 16, max_rhs=2) as ctx:
        r = ctx.orientation_solves(cfg, D.fixed_rotation(0, 0, 0)[None])
    ref64, ref32 = golden["ldr16_64"], golden["ldr16"]
    for k, q in ((0, "cabs"), (1, "cext")):
        gate = max(1e-4 * abs(ref64[k]), 2 * abs(ref32[k] - ref64[k]))
        assert abs(r[q][0] - ref64[k]) <= gate
    M = r["mueller"][0].ravel()
    sig = np.abs(ref64[2:]) > 1e-3 * np.abs(ref64[2:]).max()
    assert (np.abs(M - ref64[2:])[sig] / np.abs(ref64[2:])[sig]).max() < 1e-3


def test_workspace_mismatch_and_bad_material(D):
    """A lattice that differs from the context is rejected like the reference's workspace
    check (dda_func.cpp:1091-1094); so is an occupancy index outside the material table."""
    import ctypes as C
    L = D.lib()
    n = 8
    occ = np.ones((n, n, n), np.int8)
    alpha = np.array([0, 0, 0.01, 0.0], np.float32)
    mv = np.array([0, 1], np.int32)
    k = np.array([0, 0, 1], np.float32)
    e = np.array([1, 0, 0, 0, 0, 0], np.float32)
    ksc = np.array([0, 0, 1], np.float32)
    esc = np.zeros(6, np.float32)
    ca, ce = C.c_float(), C.c_float()
    P = lambda a: C.c_void_p(a.ctypes.data)
    with D.Context(n, 0.5) as ctx:
        rc = L.ddagpu_dda_fft(ctx.handle, 0, 0, 0.0, 16, n, n, P(alpha), P(mv), 1, P(occ), 2,
                              1e-3, 0.5, P(k), P(e), 0, 1, 1, P(ksc), P(esc), C.byref(ca),
                              C.byref(ce), None, None)
        assert rc == -4
        bad = occ.copy()
        bad[0, 0, 0] = 5
        rc = L.ddagpu_dda_fft(ctx.handle, 0, 0, 0.0, n, n, n, P(alpha), P(mv), 1, P(bad), 2,
                              1e-3, 0.5, P(k), P(e), 0, 1, 1, P(ksc), P(esc), C.byref(ca),
                              C.byref(ce), None, None)
        assert rc == -1
        rc = L.ddagpu_dda_fft(ctx.handle, 0, 7, 0.0, n, n, n, P(alpha), P(mv), 1, P(occ), 2,
                              1e-3, 0.5, P(k), P(e), 0, 1, 1, P(ksc), P(esc), C.byref(ca),
                              C.byref(ce), None, None)
        assert rc == -1
        # the context stays usable after rejected calls
        rc = L.ddagpu_dda_fft(ctx.handle, 0, 0, 0.0, n, n, n, P(alpha), P(mv), 1, P(occ), 2,
                              1e-3, 0.5, P(k), P(e), 0, 1, 1, P(ksc), P(esc), C.byref(ca),
                              C.byref(ce), None, None)
        assert rc == 0 and np.isfinite(ce.value) and ce.value != 0.0


def test_occupancy_changes_between_calls(D, oracle):
    """A context keeps the last occupancy it uploaded and skips the upload when the next
    call's occupancy is the same; a changed occupancy (or material flags), even in the same
    host buffer, must still be used."""
    n, kd = 16, 0.4
    a, _ = oracle.gen_ellipsoid(n, n, n, 1.0, 1.0)
    b, _ = oracle.gen_ellipsoid(n, n, n, 0.6, 0.5)
    alpha = np.array([0, 0.02 + 0.001j], np.complex64)
    ksc = np.array([[[0.0, 0.0, 1.0], [1.0, 0.0, 0.0]]])

    def run(ctx, occ, mv=(0, 1)):
        return ctx.dda_fft(occ, alpha, list(mv), kd, (0, 0, 1), (1, 0, 0), ksc, max_step=30,
                           err_max=1e-6)["cext"]

    with D.Context(n, kd) as fresh:
        ref_a, ref_b = run(fresh, a), None
    with D.Context(n, kd) as fresh:
        ref_b = run(fresh, b)
    with D.Context(n, kd) as ctx:
        buf = a.copy()
        got = [run(ctx, buf), run(ctx, buf)]
        buf[...] = b                       # same host buffer, new contents
        got.append(run(ctx, buf))
        buf[...] = a
        got.append(run(ctx, buf))
        with pytest.raises(D.DDAGPUError):  # all materials inactive: no dipoles
            run(ctx, buf, mv=(0, 0))
        got.append(run(ctx, buf))
    for g, r in zip(got, (ref_a, ref_a, ref_b, ref_a, ref_a)):
        assert abs(g - r) <= 1e-6 * abs(r)


def test_material_switched_off_with_polarisability(D, oracle):
    """A material listed inactive (iListMV = 0) but given a nonzero polarisability: its
    cells carry no dipoles, the far field skips them, and CabsCext still visits them (it
    tests the polarisability, dda_func.cpp:1696) -- the fused far-field pass reads such
    cells from global memory.  Results equal the FP64 oracle's."""
    rng = np.random.default_rng(21)
    n, kd = 16, 0.4
    occ, _ = oracle.gen_ellipsoid(n, n, n, 0.8, 0.6)
    occ[occ == 1] = rng.integers(1, 3, size=int((occ == 1).sum()))
    alpha = np.array([0, 0.02 + 0.001j, 0.015 + 0.002j], np.complex64)
    mv = np.array([0, 1, 0])
    ksc = oracle.scattering_geometry(2, 19, 0.0, 10.0)[1]
    einc = (1.0, 0.0, 0.0)
    with D.Context(n, kd) as ctx:
        # the residual crosses 1.5e-2 at step 3 (1.23e-2; 1.73e-2 at step 2)
        r = ctx.dda_fft(occ, alpha, mv, kd, (0, 0, 1), einc, ksc, max_step=30, err_max=1.5e-2)
    o = oracle.dda_fft(occ, alpha.astype(np.complex128), mv, kd, (0, 0, 1), einc,
                       oracle.green_hat(n, n, n, kd), ksc.astype(np.float64), solver=0, tau=1.0,
                       max_step=30, err_max=1.5e-2)
    assert r["steps"] == 3
    for q in ("cext", "cabs"):
        assert abs(r[q] - o[q]) <= 1e-4 * abs(o[q]), (q, r[q], o[q])
    assert rel(r["esc"], o["esc"]) < 1e-3


@pytest.mark.parametrize("model", [2, 3, 4])
@pytest.mark.parametrize("err_max,solver", [(1e-3, 0), (1e-6, 0), (1e-6, 2)])
def test_batched_polarizability_models_vs_oracle(D, oracle, model, err_max, solver):
    """CMRR, CMNR and ILDR (dda_func.cpp:1639-1665), computed by the library's batched path,
    against the FP64 oracle's sample loop: at Error_max 1e-3 the solve stops at step 0, so
    the cross sections carry alpha itself (Cabs explicitly, dda_func.cpp:1709-1719); at 1e-6
    the solvers iterate.  Two materials, two planes, fixed orientation (30, 45, 60 deg)."""
    n, x = 16, 3.0
    rng = np.random.default_rng(model)
    occ, _ = oracle.gen_ellipsoid(n, n, n)
    occ = np.where(occ > 0, rng.integers(1, 3, occ.shape), 0).astype(np.int8)
    mats = [(1.5, 0.01), (1.3, 0.2)]
    cfg = D.BatchConfig(occ=occ, materials=mats, polarizability=model, solver=solver, err_max=err_max,
                        max_step=200, nplanes=2)
    rot = D.fixed_rotation(30.0, 45.0, 60.0)[None]
    with D.Context(n, 2 * x / n, max_rhs=2) as ctx:
        r = ctx.orientation_solves(cfg, rot)
    o = orientation_solves(oracle, n, x, mats, 1, polarizability=model, solver=solver, err_max=err_max,
                           max_step=200, nplanes=2, psi=30.0, iota=45.0, kappa=60.0, occ=occ)
    for q in ("cabs", "cext"):
        assert abs(r[q][0] - o[q]) < 1e-4 * abs(o[q]), (q, r[q][0], o[q])
    M, Mo = r["mueller"][0].reshape(-1, 16), o["mueller"].reshape(-1, 16)
    sig = np.abs(Mo) > 1e-3 * np.abs(Mo).max()
    assert (np.abs(M - Mo)[sig] / np.abs(Mo)[sig]).max() < 1e-4


@pytest.mark.parametrize("grid,nrhs", [((4, 4, 4), 1), ((16, 16, 16), 2), ((8, 128, 64), 1), ((64, 64, 64), 2)])
def test_products_in_flight_do_not_overtake(D, grid, nrhs):
    """Products launched one into the other's end without a wait in between, each reading what the
    one before wrote, equal the same chain with a synchronisation after every product (the same
    kernels on the same inputs: bit for bit)."""
    import torch
    with D.Context(grid, 0.3, max_rhs=nrhs) as ctx:
        x = torch.randn((nrhs, 3) + grid, dtype=torch.complex64, generator=torch.Generator().manual_seed(3)).cuda()
        runs = []
        for wait in (True, False):
            f = [x.clone(), torch.empty_like(x), torch.empty_like(x)]
            torch.cuda.synchronize()
            for k in range(12):
                ctx.convolution_dev(f[k % 3], f[(k + 1) % 3], nrhs, conj=k % 4 == 3)
                if wait:
                    torch.cuda.synchronize()
            torch.cuda.synchronize()
            runs.append([g.cpu().numpy() for g in f])
    for a, b in zip(*runs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("grid", [(4, 128, 64), (4, 128, 128), (16, 32, 8), (4, 4, 32)])
def test_split_and_permuted_planes_vs_generic(D, grid):
    """Sized y/z passes on planes split over two and four CTAs and on rows whose shared-memory order
    depends on the row: products (three right-hand sides, both operators) and the incident-field
    start of paired solves equal the run-time-sized passes (2e-6 of the field, two FP32 transforms;
    1e-5 of the cross sections after three steps)."""
    import torch
    rng = np.random.default_rng(11)
    x = torch.from_numpy(crand(rng, (3, 3) + grid)).cuda()
    occ = rng.integers(0, 3, grid).astype(np.int8)
    cfg = D.BatchConfig(occ=occ, materials=[(1.3, 0.01), (1.5, 0.1)], err_max=1e-12, max_step=3)
    rot = D.mc_rotations(2, 2)
    outs = []
    for fast in (True, False):
        with D.Context(grid, 0.2, max_rhs=4) as ctx:
            ctx.set_kernels(fast)
            y = [torch.empty_like(x) for _ in range(2)]
            for k in range(2):
                ctx.convolution_dev(x, y[k], 3, conj=k == 1)
            torch.cuda.synchronize()
            r = ctx.orientation_solves(cfg, rot)
            outs.append(([v.cpu().numpy() for v in y], r))
    for a, b in zip(outs[0][0], outs[1][0]):
        assert rel(a, b) < 2e-6
    for q in ("cabs", "cext"):
        np.testing.assert_allclose(outs[0][1][q], outs[1][1][q], rtol=1e-5)


def test_a_refused_product_leaves_no_error_behind(D, oracle):
    """More right-hand sides than a launch grid holds (65535) are refused by the CUDA runtime when the
    product is launched.  The next calls, of this context and of another one, are not affected."""
    import torch
    g, kd, n = (4, 4, 4), 0.4, 65536
    p = crand(np.random.default_rng(3), g + (3,))
    ref = oracle.convolution(oracle.green_hat(*g, kd), p.astype(np.complex128))
    with D.Context(g, kd, max_rhs=n) as big, D.Context(g, kd) as other:
        x = torch.zeros((n, 3) + g, dtype=torch.complex64, device="cuda")
        y = torch.empty_like(x)
        with pytest.raises(D.DDAGPUError):
            big.convolution_dev(x, y, n)
        for ctx in (other, big):
            assert rel(ctx.convolution(p), ref) < CONV_TOL


@pytest.mark.parametrize("grid", [(4, 4, 4), (8, 8, 8), (4, 8, 16), (16, 4, 32), (8, 16, 4), (64, 4, 4), (64, 8, 8),
                                  (128, 4, 8), (4, 128, 64), (8, 64, 128), (32, 16, 4)])
def test_sized_passes_at_small_edges_vs_oracle(D, oracle, grid):
    """The sized passes at edges 4 and 8 on every axis, both operators: every kernel that the variant
    numbers stand for (rows shorter than a tile of the x pass in its register and bulk-copy forms;
    planes split over two CTAs with both block sizes at 64 x 128 and 128 x 64), against the oracle.  Numbers that
    stand for the same kernel are accepted; TMA tiles are refused where a row is shorter than one."""
    import torch
    rng = np.random.default_rng(sum(grid))
    kd = 0.5
    p = crand(rng, (2, 3) + grid)
    A = oracle.green_hat(*grid, kd)
    ref = {conj: np.stack([oracle.convolution(A, q.transpose(1, 2, 3, 0).astype(np.complex128), conj=conj)
                           for q in p]) for conj in (False, True)}
    with D.Context(grid, kd, max_rhs=2) as ctx:
        assert ctx.fast_kernels
        x = torch.from_numpy(p).cuda()
        kernels = [3, 6] + ([0, 1, 2] if grid[0] == 64 else [])
        if grid[2] >= 8:
            kernels += [9]
            for alias in (10, 11):
                ctx.set_fast_variant(alias, 2)
        else:
            with pytest.raises(D.DDAGPUError):
                ctx.set_fast_variant(9, 0)
        for alias in (0, 1, 2, 4, 5, 7, 8):
            ctx.set_fast_variant(alias, 2)
        for vx in kernels:
            for vyz in (0, 1):
                ctx.set_fast_variant(vx, vyz)
                for conj in (False, True):
                    y = torch.empty_like(x)
                    ctx.convolution_dev(x, y, 2, conj=conj)
                    ctx.synchronize()
                    assert rel(y.cpu().numpy().transpose(0, 2, 3, 4, 1), ref[conj]) < CONV_TOL, (vx, vyz, conj)


@pytest.mark.parametrize("grid", [(4, 4, 4), (8, 8, 4), (16, 4, 8), (64, 4, 4), (128, 4, 4), (4, 64, 128)])
@pytest.mark.parametrize("model", [1, 5])
def test_sized_solves_at_small_edges_equal_generic(D, grid, model):
    """Step 0 from the incident field at edges 4 and 8, of polarisation pairs (CM) and of single
    right-hand sides (LDR), and two CG steps: the sized passes against the generic ones.  Both round
    at 2^-24 in 2 log2(8 N) butterflies a product, below 1e-6 of the largest value; three products
    and the sums after them: 1e-5."""
    rng = np.random.default_rng(sum(grid))
    occ = (rng.random(grid) < 0.8).astype(np.int8)
    rot = D.mc_rotations(5, 2)
    cfg = D.BatchConfig(occ=occ, materials=[(1.5, 0.02)], polarizability=model, max_step=2, err_max=1e-9)
    out = {}
    with D.Context(grid, 0.3, max_rhs=4) as ctx:
        for fast in (True, False):
            ctx.set_kernels(fast)
            out[fast] = ctx.orientation_solves(cfg, rot)
    for q in ("cabs", "cext"):
        np.testing.assert_allclose(out[True][q], out[False][q], rtol=1e-5)
    M, G = out[True]["mueller"], out[False]["mueller"]
    assert np.abs(M - G).max() <= 1e-5 * np.abs(G).max()
