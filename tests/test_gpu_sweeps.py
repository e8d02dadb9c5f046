"""The MIC(0) sweeps on x-pencils (csrc/mic_pencil.cu) against the 8^3-tile
sweeps, which test_gpu_parity.py holds to the CPU oracle: the same cells in the
same dependency order with the same roundings, so the results are equal bit
for bit, whatever the shape of the grid and the gaps in its pencils."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _z(shape, blocks, block, seed):
    """One MIC(0) application on a system whose liquid fills the chosen 16^3
    blocks (all of them for blocks = 1.0), from a fresh context."""
    from shiokaze_b200.projection import Grid, MacGrid, MacPressureSolver3
    nx, ny, nz = shape
    dx = 1.0 / max(shape)
    rng = np.random.default_rng(seed)
    pick = rng.random(((nz + 15) // 16, (ny + 15) // 16, (nx + 15) // 16)) < blocks
    inside = pick.repeat(16, 0).repeat(16, 1).repeat(16, 2)[:nz, :ny, :nx]
    phi = np.where(inside, -1.0, 1.0) * rng.uniform(0.2, 1.7, (nz, ny, nx)) * dx
    vel = [rng.standard_normal((nz + (d == 2), ny + (d == 1), nx + (d == 0))).astype(np.float32) for d in range(3)]
    s = MacPressureSolver3({"Residual": 1e-2, "MaxIterations": 2, "B200.MICBlock": block})
    s.initialize(shape, dx)
    s.project(0.01, MacGrid(vel, [np.ones(v.shape, np.uint8) for v in vel]), None, None,
              Grid(phi.astype(np.float32), np.ones(phi.shape, np.uint8)))
    mask = s.get_pressure().active.astype(bool)
    assert mask.any()
    r = np.where(mask, rng.standard_normal((nz, ny, nx)), 0).astype(np.float32)
    return s.apply_preconditioner(r)


@pytest.mark.parametrize("shape,blocks", [
    ((8, 8, 8), 1.0),          # less than one macro tile
    ((16, 16, 16), 1.0),       # one macro tile: the shortest pencil
    ((17, 33, 15), 1.0),       # remainders on every side
    ((150, 20, 50), 1.0),      # long pencils, the ring wraps
    ((96, 80, 64), 0.5),       # gaps along x: several pencils in a row, missing neighbours
    ((64, 208, 224), 0.8),     # more pencils than SMs
])
def test_pencil_sweeps_equal_tile_sweeps(shape, blocks):
    np.testing.assert_array_equal(_z(shape, blocks, 16, 3), _z(shape, blocks, 8, 3))


@pytest.mark.parametrize("shape,blocks", [
    ((8, 8, 8), 1.0),
    ((16, 16, 16), 1.0),
    ((17, 33, 15), 1.0),
    ((150, 20, 50), 1.0),
    ((96, 80, 64), 0.5),
    ((64, 208, 224), 0.8),
])
@pytest.mark.parametrize("limit", [1, 2, 3, 30000])
def test_fused_iteration_equals_the_separate_kernels(shape, blocks, limit):
    """The loop every projection runs (r update, norms, z.r, rho and beta inside
    the pencil sweeps, x and p updates in the next stencil) against the loop of
    separate kernels on 8^3 tiles, at the shapes above and stopped after one,
    two and three iterations, where an update is pending and the direction is in
    either buffer. Per cell the FP32 arithmetic is the same; alpha and beta
    differ by the order in which FP64 sums are added, some 1e-13."""
    from shiokaze_b200.projection import Grid, MacGrid, MacPressureSolver3
    nx, ny, nz = shape
    dx = 1.0 / max(shape)
    rng = np.random.default_rng(3)
    pick = rng.random(((nz + 15) // 16, (ny + 15) // 16, (nx + 15) // 16)) < blocks
    inside = pick.repeat(16, 0).repeat(16, 1).repeat(16, 2)[:nz, :ny, :nx]
    inside[-1] = False  # a free surface
    phi = (np.where(inside, -1.0, 1.0) * rng.uniform(0.2, 1.7, (nz, ny, nx)) * dx).astype(np.float32)
    vel = [rng.standard_normal((nz + (d == 2), ny + (d == 1), nx + (d == 0))).astype(np.float32) for d in range(3)]
    runs = []
    for block in (16, 8):
        s = MacPressureSolver3({"Residual": 1e-6, "MaxIterations": limit, "B200.MICBlock": block})
        s.initialize(shape, dx)
        grid = MacGrid([v.copy() for v in vel], [np.ones(v.shape, np.uint8) for v in vel])
        res = s.project(0.01, grid, None, None, Grid(phi, np.ones(phi.shape, np.uint8)))
        runs.append((res, s.get_pressure().values.astype(np.float64)))
    (res, p), (other, want) = runs
    assert res["status"] == 0 and res["iterations"] == other["iterations"]
    assert res["iterations"] == limit if limit < 4 else res["reresid"] <= 1e-6
    # FP32 vectors of the same cells: a last bit of alpha or beta is 6e-8, a few
    # of them an iteration, summed over the iterations done
    tol = 5e-7 * (res["iterations"] + 1)
    assert np.abs(p - want).max() <= tol * np.abs(want).max()
    assert abs(res["reresid"] - other["reresid"]) <= max(tol * other["reresid"], 1e-8)
