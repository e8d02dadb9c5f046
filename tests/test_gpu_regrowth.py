"""A call refused for device memory partway through growing a group of buffers
leaves nothing behind that a later, smaller call on the same context would
take for allocated: it allocates anew and gives a fresh context's answer."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_NOMEM = -3


def _project(ctx_holder, n):
    from shiokaze_b200 import scenes
    from shiokaze_b200.projection import grids_from_scene
    sc = scenes.dambreak_sphere(n=n, seed=3, tol=1e-5)
    vel, solid, svel, fluid = grids_from_scene(sc)
    ctx_holder.initialize((n, n, n), sc.dx)
    ctx_holder.project(sc.dt, vel, solid, svel, fluid)
    return [ctx_holder.get_pressure().values] + vel.values


def _faces(n, seed):
    rng = np.random.default_rng(seed)
    vel = [rng.standard_normal((n + (d == 2), n + (d == 1), n + (d == 0))).astype(np.float32) for d in range(3)]
    return vel, [(rng.random(v.shape) < 0.4).astype(np.uint8) for v in vel]


def _extend(ctx, n):
    from shiokaze_b200 import native
    vel, act = _faces(n, 1)
    z, y, x = np.meshgrid(*[np.arange(n + 1)] * 3, indexing="ij")
    solid = (np.sqrt((x - n / 2) ** 2 + (y - n / 2) ** 2 + (z - n / 2) ** 2) / n - 0.25).astype(np.float32)
    got = native.extend_velocity(ctx, vel, act, solid, np.ones(solid.shape, np.uint8), 1.0 / n, 3)
    return [a for part in got for a in part]


def _splat(ctx, n):
    from shiokaze_b200 import native, scenes
    vel, act = _faces(n, 1)
    P = np.zeros(n ** 3, scenes.PARTICLE_DTYPE)
    rng = np.random.default_rng(2)
    P["p"] = rng.random((len(P), 3))
    P["velocity"] = rng.standard_normal((len(P), 3))
    P["mass"] = 0.125
    return [a for part in native.splat(ctx, n, n, n, 1.0 / n, P, vel, act) for a in part]


@pytest.mark.parametrize("kind,large,limits", [
    ("project", 64, range(3, 60, 4)),
    ("extend", 64, range(1, 12)),
    ("splat", 64, range(1, 120, 7)),
])
def test_small_call_after_a_refused_large_one(kind, large, limits):
    from shiokaze_b200 import native
    from shiokaze_b200.projection import MacPressureSolver3
    small = 24

    def make():
        return MacPressureSolver3({"Residual": 1e-5}) if kind == "project" else native.Context(native.default_config())

    def limit(c, mib):
        if kind == "project":
            c.configure({"B200.DeviceMemoryLimitMB": mib})
        else:
            cfg = native.default_config()
            cfg.device_mem_limit_mb = mib
            c.set_config(cfg)

    call = {"project": _project, "extend": _extend, "splat": _splat}[kind]
    want = call(make(), small)
    refused = set()
    for mib in limits:
        c = make()
        call(c, small)
        limit(c, mib)
        try:
            call(c, large)
        except native.ShkzError as e:
            assert e.code == ERR_NOMEM
            refused.add(str(e).split(" for ")[-1].split()[0])
        limit(c, 0)
        for a, b in zip(call(c, small), want):
            np.testing.assert_array_equal(a, b)
    assert len(refused) >= 3, refused  # refusals at several buffers
