"""The solve loop's host side: iterations queued ahead of the device's reports,
and the pool's counts it reports. What is queued beyond the last iteration must
not show in the results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(sc, **config):
    from shiokaze_b200.projection import MacGrid, MacPressureSolver3
    s = MacPressureSolver3(config)
    s.initialize(sc.shape, sc.dx)
    vel = MacGrid([v.copy() for v in sc.velocity], [a.copy() for a in sc.velocity_active])
    res = s.project(sc.dt, vel, sc.solid, sc.solid_velocity, sc.fluid)
    return res, s.get_pressure().values, vel.values


class _Scene:
    def __init__(self, shape, filled, seed, block):
        from shiokaze_b200.projection import Grid
        nx, ny, nz = self.shape = shape
        self.dx, self.dt = 1.0 / max(shape), 0.01
        self.solid = self.solid_velocity = None
        rng = np.random.default_rng(seed)
        n = [(m + block - 1) // block for m in (nz, ny, nx)]
        inside = (rng.random(n) < filled).repeat(block, 0).repeat(block, 1).repeat(block, 2)[:nz, :ny, :nx]
        phi = np.where(inside, -0.7, 0.7).astype(np.float32) * np.float32(self.dx)
        self.fluid = Grid(phi, np.ones(phi.shape, np.uint8))
        self.velocity = [rng.standard_normal((nz + (d == 2), ny + (d == 1), nx + (d == 0)), dtype=np.float32)
                         for d in range(3)]
        self.velocity_active = [np.ones(v.shape, np.uint8) for v in self.velocity]


@pytest.mark.parametrize("precond,block", [("mic0", 16), ("mic0", 8), ("none", 16)])
@pytest.mark.parametrize("limit", [1, 2, 7, 30000])
def test_queue_depth_does_not_show(precond, block, limit):
    sc = _Scene((40, 33, 50), 0.6, 5, 16)
    config = {"Residual": 1e-5, "MaxIterations": limit, "B200.Preconditioner": precond, "B200.MICBlock": block}
    res, p, vel = _solve(sc, **config, **{"B200.CheckInterval": 1})
    assert res["iterations"] <= limit
    if limit <= 7:
        assert res["iterations"] == limit
    else:
        assert res["reresid"] <= 1e-5
    for depth in (2, 16):
        other, po, velo = _solve(sc, **config, **{"B200.CheckInterval": depth})
        assert other["iterations"] == res["iterations"] and other["reresid"] == res["reresid"]
        np.testing.assert_array_equal(p, po)
        for a, b in zip(vel, velo):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("shape,filled", [
    ((24, 16, 49152), 0.02),   # 36864 tiles: 37 block sums, levels by the thousand
    ((264, 32, 16), 0.5),
    ((8, 8, 8), 1.0),
])
@pytest.mark.parametrize("block", [16, 8])
def test_pool_counts(shape, filled, block):
    from shiokaze_b200.projection import MacGrid, MacPressureSolver3
    sc = _Scene(shape, filled, 7, 8)
    s = MacPressureSolver3({"Residual": 1e-2, "MaxIterations": 2, "B200.MICBlock": block})
    s.initialize(sc.shape, sc.dx)
    res = s.project(sc.dt, MacGrid(sc.velocity, sc.velocity_active), None, None, sc.fluid)
    act = s.get_pressure().active.astype(bool)
    pad = np.zeros([(m + 7) // 8 * 8 for m in act.shape], bool)
    pad[:act.shape[0], :act.shape[1], :act.shape[2]] = act
    nz, ny, nx = (m // 8 for m in pad.shape)
    assert act.any()
    assert res["unknowns"] == int(act.sum())
    assert res["tiles"] == int(pad.reshape(nz, 8, ny, 8, nx, 8).any(axis=(1, 3, 5)).sum())


@pytest.mark.parametrize("zero", [True, False])   # breakdown of the network at once, and a stall after some iterations
@pytest.mark.parametrize("limit", [12, 30000])
def test_queue_depth_does_not_show_after_the_fallback(zero, limit):
    """The learned solver's MIC(0) iterations are queued ahead, the network's
    are not: the answer is that of one iteration at a time."""
    from shiokaze_b200.projection import MacGrid, MacPressureSolver3
    sc = _Scene((40, 33, 50), 0.6, 5, 16)
    runs = []
    for depth in (1, 2, 16):
        s = MacPressureSolver3({"Residual": 1e-6, "B200.CheckInterval": depth})
        s.initialize(sc.shape, sc.dx)
        vel = lambda: MacGrid([v.copy() for v in sc.velocity], [a.copy() for a in sc.velocity_active])
        s.project(sc.dt, vel(), None, None, sc.fluid)
        s.learned_init(seed=3)
        if zero:
            s.learned_set_params(np.zeros_like(s.learned_params()))
        s.configure({"B200.Preconditioner": "learned", "MaxIterations": limit})
        v = vel()
        runs.append((s.project(sc.dt, v, None, None, sc.fluid), s.get_pressure().values, v.values))
    first, p, vel0 = runs[0]
    assert first["fallbacks"] == 1
    assert first["iterations"] == limit if limit == 12 else first["reresid"] <= 1e-6
    for res, q, v in runs[1:]:
        assert (res["iterations"], res["reresid"], res["fallbacks"]) == (first["iterations"], first["reresid"], 1)
        np.testing.assert_array_equal(p, q)
        for a, b in zip(vel0, v):
            np.testing.assert_array_equal(a, b)


_BLOCKING = r"""
import ctypes, sys, time
cu = ctypes.CDLL("libcuda.so.1")
dev = ctypes.c_int()
assert cu.cuInit(0) == 0 and cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
assert cu.cuDevicePrimaryCtxSetFlags_v2(dev, 4) == 0  # CU_CTX_SCHED_BLOCKING_SYNC
import torch
from shiokaze_b200 import native
n = 192
T = lambda shape, fill, dtype=torch.float32: torch.full(shape, fill, dtype=dtype, device="cuda")
g = torch.Generator(device="cuda").manual_seed(3)
phi, phia = T((n, n, n), -0.7 / n), T((n, n, n), 1, torch.uint8)
vel = [torch.randn((n + (d == 2), n + (d == 1), n + (d == 0)), device="cuda", generator=g) for d in range(3)]
act = [T(tuple(v.shape), 1, torch.uint8) for v in vel]
phi[n // 2:] = 0.7 / n
cfg = native.default_config()
cfg.residual = 1e-9
ctx = native.Context(cfg)
a = native.ProjectArgs()
a.nx = a.ny = a.nz = n
a.dx, a.dt, a.fluid, a.fluid_active = 1.0 / n, 0.01, phi.data_ptr(), phia.data_ptr()
torch.cuda.synchronize()
for _ in range(4):
    work = [v.clone() for v in vel]
    for d in range(3):
        a.velocity[d], a.velocity_active[d] = work[d].data_ptr(), act[d].data_ptr()
    torch.cuda.synchronize()
    res = native.Result()
    t, c = time.perf_counter(), time.thread_time()
    assert native.load().shkz_b200_project_device(ctx.handle, ctypes.byref(a), ctypes.byref(res)) == 0
    wall, cpu = time.perf_counter() - t, time.thread_time() - c
    assert res.ms_solve > 5
print(cpu / wall)
"""


def test_waits_sleep_under_blocking_synchronisation():
    """An application that has asked for cudaDeviceScheduleBlockingSync gets its
    core back while the solve runs: launches and looks are a small part of an
    iteration's 0.1 ms and more here, so well under half of the call is CPU time."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", _BLOCKING], cwd=root, env=dict(os.environ, PYTHONPATH=root),
                         capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    assert float(out.stdout.split()[-1]) < 0.5, out.stdout


def test_two_contexts_solve_at_once():
    """Two threads, a context and a scene each, project at the same time: their
    sweeps share the SMs, wait only for their own, and give what they give
    alone."""
    import threading
    scenes = [_Scene((40, 33, 50), 0.6, 5, 16), _Scene((96, 80, 64), 0.5, 9, 16)]
    config = {"Residual": 1e-5}
    alone = [_solve(sc, **config) for sc in scenes]
    got = [[], []]

    def work(i):
        for _ in range(6):
            got[i].append(_solve(scenes[i], **config))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        assert len(got[i]) == 6
        for res, p, vel in got[i]:
            assert (res["status"], res["iterations"], res["reresid"]) == (0, alone[i][0]["iterations"], alone[i][0]["reresid"])
            np.testing.assert_array_equal(p, alone[i][1])
            for a, b in zip(vel, alone[i][2]):
                np.testing.assert_array_equal(a, b)
