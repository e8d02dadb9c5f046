"""The generic path's MIC(0) over patterns: those the device analyses (sorted
rows, symmetric) and those the host does, against the oracle's factor and
sweeps."""
import ctypes

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def _matrix(kind, rng):
    """(indptr, indices, data): diagonally dominant, symmetric values."""
    edges = set()
    n = {"chain": 3000, "one": 1, "pair": 2, "grid": 24 * 24 * 24}.get(kind, 700)
    if kind in ("random", "one_sided", "island"):
        span = n // 2 if kind == "island" else n  # the rest of the rows hold a diagonal only
        while len(edges) < 4 * span:
            i, j = sorted(int(v) for v in rng.integers(0, span, 2))
            if i < j:
                edges.add((i, j))
    elif kind in ("chain", "pair"):
        edges = {(i, i + 1) for i in range(n - 1)}
    elif kind == "first_dense":
        edges = {(0, j) for j in range(1, n)} | {(i, i + 1) for i in range(n - 1)}
    elif kind == "last_dense":
        edges = {(i, n - 1) for i in range(n - 1)}
    elif kind == "grid":
        idx = np.arange(n).reshape(24, 24, 24)
        for a in range(3):
            edges |= set(zip(np.take(idx, range(23), a).ravel().tolist(), np.take(idx, range(1, 24), a).ravel().tolist()))
    rows = [dict() for _ in range(n)]
    for i, j in edges:
        rows[i][j] = rows[j][i] = -float(rng.uniform(0.2, 1.0))
    for i in range(n):
        rows[i][i] = -sum(rows[i].values()) + float(rng.uniform(0.01, 0.1))
    if kind == "one_sided":  # stored zeros that the other triangle does not have
        for i, j in rng.integers(0, n, (200, 2)).tolist():
            rows[i].setdefault(j, 0.0)
    indptr = np.zeros(n + 1, np.int64)
    indptr[1:] = np.cumsum([len(r) for r in rows])
    indices = np.array([j for r in rows for j in sorted(r)], np.int64)
    data = np.array([r[j] for r in rows for j in sorted(r)], np.float64)
    return indptr, indices, data


@pytest.mark.parametrize("kind", ["one", "pair", "random", "island", "chain", "first_dense", "last_dense", "grid",
                                  "one_sided"])
def test_csr_mic0_over_patterns(kind):
    from shiokaze_b200 import native
    rng = np.random.default_rng(23)
    indptr, indices, data = _matrix(kind, rng)
    n = len(indptr) - 1
    b = rng.standard_normal(n)
    S = oracle.System(index=None, n=n, indptr=indptr, indices=indices, data=data, rhs=b)
    z, _ = oracle.mic0_apply(S, b)
    cfg = native.default_config()
    cfg.residual = 1e30  # stops after the first step: x = alpha z
    cfg.csr_preconditioner = native.PRECOND_MIC0
    ctx = native.Context(cfg)
    x = np.zeros(n)
    res = native.Result()
    rc = native.load().shkz_b200_solve_csr(ctx.handle, n, indptr.ctypes.data, indices.ctypes.data, data.ctypes.data,
                                           b.ctypes.data, x.ctypes.data, ctypes.byref(res))
    assert rc == 0 and res.iterations == 1
    alpha = float(z @ b) / float(z @ oracle.spmv(S, z))
    assert np.abs(x - alpha * z).max() <= 1e-12 * np.abs(alpha * z).max()
    # levels of the dependencies through the upper triangle's entries
    level = np.zeros(n, np.int64)
    for i in range(n):
        for j in indices[indptr[i]:indptr[i + 1]]:
            if j > i:
                level[j] = max(level[j], level[i] + 1)
    assert res.outer_steps == level.max() + 1
