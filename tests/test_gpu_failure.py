"""Failure handling on the device, made without faulting the GPU.

The reference has no failure handling of its own on this path: a fatal module
error ends the process (src/core/module.cpp:141) and a solve that does not
converge returns silently after MaxIterations
(local/include/pcgsolver/pcg_solver.h:267-295). The B200 library reports each
failure as a status code instead, and the context stays usable:

* a bounded device wait that runs out returns SHKZ_B200_ERR_TIMEOUT. The test
  makes it run out on purpose: B200.FaultSkipPublish stops one tile of the
  forward MIC(0) sweep from publishing its faces (a flag that nothing sets),
  and B200.SpinLimit shortens the waits;
* the same for the generic CSR solve's MIC(0) triangular solves: there
  B200.FaultSkipPublish stops one row of the forward solve from storing its
  value, and the rows that wait on it give up;
* a device-memory cap that the tile pool does not fit under returns
  SHKZ_B200_ERR_NOMEM before cudaMalloc is asked;
* a learned preconditioner that breaks down (a network of zeros) falls back to
  MIC(0) and the solve still reaches the MIC(0) answer.
After each, the next call on the same context succeeds.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_NOMEM, ERR_TIMEOUT = -3, -4


def _run(s, sc):
    from shiokaze_b200.projection import grids_from_scene
    vel, solid, svel, fluid = grids_from_scene(sc)
    res = s.project(sc.dt, vel, solid, svel, fluid)
    return res, s.get_pressure().values.copy(), [v.copy() for v in vel.values]


def _reference_solution(sc):
    from shiokaze_b200.projection import MacPressureSolver3
    s = MacPressureSolver3({"Residual": sc.tol})
    s.initialize((sc.nx, sc.ny, sc.nz), sc.dx)
    res, p, v = _run(s, sc)
    assert res["status"] == 0, res
    return res, p, v


def test_sweep_wait_timeout_returns_error_and_context_recovers():
    from shiokaze_b200 import scenes
    from shiokaze_b200.projection import MacPressureSolver3
    sc = scenes.dambreak_sphere(n=64, seed=1, tol=1e-6)
    res0, p0, v0 = _reference_solution(sc)
    # the first tile of the forward sweep's wavefront never publishes; its
    # consumers give up after 20000 polling rounds (milliseconds)
    s = MacPressureSolver3({"Residual": sc.tol, "B200.SpinLimit": 20000, "B200.FaultSkipPublish": 1})
    s.initialize((sc.nx, sc.ny, sc.nz), sc.dx)
    res, _, _ = _run(s, sc)
    assert res["status"] == ERR_TIMEOUT, res
    # the same context, fault off: a normal projection, identical to a fresh context's
    s.configure({"B200.SpinLimit": 0, "B200.FaultSkipPublish": 0})
    res1, p1, v1 = _run(s, sc)
    assert res1["status"] == 0, res1
    assert res1["iterations"] == res0["iterations"]
    assert np.array_equal(p1, p0)
    for d in range(3):
        assert np.array_equal(v1[d], v0[d])


def test_csr_solve_wait_timeout_returns_error_and_context_recovers():
    import ctypes
    from conftest import golden_names, load_golden
    from shiokaze_b200 import native
    g = load_golden(golden_names()[0])
    n = int(g["rhs"].size)
    indptr = np.ascontiguousarray(g["indptr"], np.int64)
    indices = np.ascontiguousarray(g["indices"], np.int64)
    data = np.ascontiguousarray(g["data"], np.float64)
    b = np.ascontiguousarray(g["rhs"], np.float64)
    L = native.load()

    def solve(ctx):
        x = np.zeros(n, np.float64)
        res = native.Result()
        rc = L.shkz_b200_solve_csr(ctx.handle, n, indptr.ctypes.data, indices.ctypes.data, data.ctypes.data,
                                   b.ctypes.data, x.ctypes.data, ctypes.byref(res))
        return rc, res, x

    cfg = native.default_config()
    cfg.residual = float(g["tol"])
    cfg.csr_preconditioner = native.PRECOND_MIC0
    rc0, res0, x0 = solve(native.Context(cfg))
    assert rc0 == 0 and res0.iterations > 0
    # the first row of the forward triangular solve never stores its value;
    # the rows that depend on it give up after 20000 polling rounds
    cfg.spin_limit, cfg.fault_skip_publish = 20000, 1
    ctx = native.Context(cfg)
    rc, _, _ = solve(ctx)
    assert rc == ERR_TIMEOUT, rc
    # the same context, fault off: the same solve as a fresh context's
    cfg.spin_limit, cfg.fault_skip_publish = 0, 0
    ctx.set_config(cfg)
    rc1, res1, x1 = solve(ctx)
    assert rc1 == 0 and res1.iterations == res0.iterations
    assert np.array_equal(x1, x0)


def test_device_memory_cap_returns_nomem_and_context_recovers():
    from shiokaze_b200 import native, scenes
    from shiokaze_b200.projection import MacPressureSolver3
    sc = scenes.dambreak_sphere(n=48, seed=2, tol=1e-6)
    res0, p0, _ = _reference_solution(sc)
    # 6 MiB holds the 48^3 grid and host-staging buffers (about 5 MB) but not
    # the tile pool (about 80 KB per tile for 100+ tiles)
    s = MacPressureSolver3({"Residual": sc.tol, "B200.DeviceMemoryLimitMB": 6})
    s.initialize((sc.nx, sc.ny, sc.nz), sc.dx)
    with pytest.raises(native.ShkzError) as e:
        _run(s, sc)
    assert e.value.code == ERR_NOMEM
    msg = str(e.value)
    assert "device memory cap of 6 MiB" in msg, msg
    pool_buffers = ("pool_tile", "nbr", "sched", "diag", "offx", "offy", "offz", "d32", "diag64", "offx64",
                    "offy64", "offz64", "rhs64", "colsum", "dmic64", "x64", "r64", "xref64", "p64", "q64", "z64")
    assert msg.split(" for ")[-1].split()[0] in pool_buffers, msg
    s.configure({"B200.DeviceMemoryLimitMB": 0})
    res1, p1, _ = _run(s, sc)
    assert res1["status"] == 0, res1
    assert np.array_equal(p1, p0)


def test_zero_network_falls_back_to_mic0_and_reaches_its_answer():
    from shiokaze_b200 import scenes
    from shiokaze_b200.projection import MacPressureSolver3
    sc = scenes.dambreak_sphere(n=32, seed=2, tol=1e-6)
    res0, p0, _ = _reference_solution(sc)
    s = MacPressureSolver3({"Residual": sc.tol})
    s.initialize((sc.nx, sc.ny, sc.nz), sc.dx)
    res, _, _ = _run(s, sc)
    assert res["status"] == 0
    s.learned_init(seed=3)
    s.learned_set_params(np.zeros_like(s.learned_params()))
    s.configure({"B200.Preconditioner": "learned"})
    res1, p1, _ = _run(s, sc)
    assert res1["status"] == 0, res1
    assert res1["fallbacks"] == 1, res1
    assert res1["reresid"] <= sc.tol
    assert np.abs(p1.astype(np.float64) - p0).max() / np.abs(p0).max() < 1e-4


@pytest.mark.parametrize("block", [16, 8])
@pytest.mark.parametrize("refine", [1, 0])
def test_breakdown_leaves_the_last_finite_iterate(block, refine):
    """A cell at minus infinity beside one outside the liquid gives a NaN
    weight and a finite right-hand side, so the solve breaks down in its first
    iteration. The call says so; the pressure it hands back is the iterate
    before that (zero) and only the face between the two cells has no value."""
    from shiokaze_b200.projection import Grid, MacGrid, MacPressureSolver3
    nx, ny, nz = 40, 33, 50
    rng = np.random.default_rng(5)
    dx = 1.0 / nz
    phi = np.where(rng.random((4, 3, 3)) < 0.6, -0.7, 0.7).repeat(16, 0).repeat(16, 1).repeat(16, 2)[:nz, :ny, :nx] * dx
    k, j, i = np.argwhere((phi[:, :, :-1] < 0) & (phi[:, :, 1:] > 0))[100]
    phi[k, j, i] = -np.inf
    vel = [rng.standard_normal((nz + (d == 2), ny + (d == 1), nx + (d == 0))).astype(np.float32) for d in range(3)]
    s = MacPressureSolver3({"Residual": 1e-6, "B200.MICBlock": block, "B200.Refine": refine})
    s.initialize((nx, ny, nz), dx)
    grid = MacGrid([v.copy() for v in vel], [np.ones(v.shape, np.uint8) for v in vel])
    res = s.project(0.01, grid, None, None, Grid(phi.astype(np.float32), np.ones(phi.shape, np.uint8)))
    assert res["status"] == -5 and res["iterations"] == 0
    assert not s.get_pressure().values.any()
    bad = [np.argwhere(np.isnan(v)) for v in grid.values]
    assert bad[0].tolist() == [[k, j, i + 1]] and not len(bad[1]) and not len(bad[2])


def test_csr_factor_wait_timeout_returns_error_and_context_recovers():
    """A column of the MIC(0) factorisation that never says it is done: the
    columns that wait on it give up after the configured rounds (the default,
    2^22, takes seconds)."""
    import ctypes
    import time
    from conftest import golden_names, load_golden
    from shiokaze_b200 import native
    g = load_golden(golden_names()[0])
    n = int(g["rhs"].size)
    arrays = [np.ascontiguousarray(g[k], t) for k, t in
              (("indptr", np.int64), ("indices", np.int64), ("data", np.float64), ("rhs", np.float64))]

    def solve(ctx):
        x = np.zeros(n, np.float64)
        res = native.Result()
        t0 = time.perf_counter()
        rc = native.load().shkz_b200_solve_csr(ctx.handle, n, *[a.ctypes.data for a in arrays], x.ctypes.data,
                                               ctypes.byref(res))
        return rc, time.perf_counter() - t0, res.iterations, x

    cfg = native.default_config()
    cfg.residual = float(g["tol"])
    cfg.csr_preconditioner = native.PRECOND_MIC0
    ctx = native.Context(cfg)
    rc0, _, it0, x0 = solve(ctx)
    assert rc0 == 0 and it0 > 0
    cfg.spin_limit, cfg.fault_skip_publish = 20000, -1
    ctx.set_config(cfg)
    tries = [solve(ctx)[:2] for _ in range(3)]
    assert all(rc == ERR_TIMEOUT for rc, _ in tries), tries
    assert min(seconds for _, seconds in tries) < 1.0, tries  # (a host may stall in an allocation)
    cfg.spin_limit, cfg.fault_skip_publish = 0, 0
    ctx.set_config(cfg)
    rc1, _, it1, x1 = solve(ctx)
    assert rc1 == 0 and it1 == it0
    assert np.array_equal(x1, x0)


def test_a_longer_wait_limit_is_not_cut_short():
    """Waits inside a CTA of the pencil sweeps end with an error after 4 s at
    the earliest, but not before a longer configured limit of the waits they
    depend on has run out: 2^25 rounds, 6 to 8 s."""
    import time
    from shiokaze_b200 import scenes
    from shiokaze_b200.projection import MacPressureSolver3
    sc = scenes.dambreak_sphere(n=48, seed=1, tol=1e-6)
    res0, p0, _ = _reference_solution(sc)
    s = MacPressureSolver3({"Residual": sc.tol, "B200.SpinLimit": 1 << 25, "B200.FaultSkipPublish": 1})
    s.initialize((sc.nx, sc.ny, sc.nz), sc.dx)
    t0 = time.perf_counter()
    res, _, _ = _run(s, sc)
    assert res["status"] == ERR_TIMEOUT
    assert time.perf_counter() - t0 > 5.2
    s.configure({"B200.SpinLimit": 0, "B200.FaultSkipPublish": 0})
    res1, p1, _ = _run(s, sc)
    assert res1["status"] == 0 and res1["iterations"] == res0["iterations"]
    assert np.array_equal(p1, p0)
