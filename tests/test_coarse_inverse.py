"""Dense inverse of a symmetric dominant coarsest level in nested-dissection
order (csrc/coarse_inverse.cu), as exact one-level solves against numpy.

The graphs cover what the order decides on: long and compact meshes, parts
at the limit below which nothing is split (256 rows), many independent
components, rows without neighbours, and graphs without a useful separator.
Tolerance: rows are dominant with a margin of a tenth of their off-diagonal
sum, so |A^-1| |A| is below about 100 times the spread of the row sums; a
converged residual of 1e-10 then bounds the error by 1e-8, and in FP64 one
cycle (an exact solve up to n * eps) must reach that residual.
"""
import numpy as np
import pytest

from fvm_b200 import fvmbaseExt

pytestmark = pytest.mark.gpu


def _grid(shape):
    idx = np.arange(int(np.prod(shape))).reshape(shape)
    pairs = []
    for ax in range(len(shape)):
        a = np.take(idx, range(shape[ax] - 1), axis=ax).ravel()
        b = np.take(idx, range(1, shape[ax]), axis=ax).ravel()
        pairs.append(np.stack([a, b], 1))
    return idx.size, np.concatenate(pairs)


def _random(n, degree, seed=1):
    rng = np.random.default_rng(seed)
    e = rng.integers(0, n, (n * degree // 2, 2))
    e = e[e[:, 0] != e[:, 1]]
    return n, np.unique(np.sort(e, 1), axis=0)


def _shuffled(g, seed=3):
    n, e = g
    p = np.random.default_rng(seed).permutation(n)
    return n, p[e]


def _union(*gs):
    off, out = 0, []
    for n, e in gs:
        out.append(e + off)
        off += n
    return off, np.concatenate(out) if out else np.zeros((0, 2), int)


GRAPHS = {
    "chain-129": _grid((129,)),
    "chain-4096": _grid((4096,)),
    "grid-256": _grid((16, 16)),
    "grid-257": _union(_grid((16, 16)), _grid((1,))),
    "grid-45x40": _grid((45, 40)),
    "grid-64x64": _grid((64, 64)),
    "long-9x300": _grid((9, 300)),
    "cube-15": _grid((15, 15, 15)),
    "cube-13-shuffled": _shuffled(_grid((13, 13, 13))),
    "components": _union(*[_grid((k, k + 1)) for k in range(2, 20)]),
    "many-components": _union(*[_grid((3, 2))] * 300),
    "no-neighbours": (700, np.zeros((0, 2), int)),
    "random-2000": _random(2000, 9),
    "random-4096": _random(4096, 3),
    "dense-200": (200, np.stack(np.triu_indices(200, 1), 1)),
    "star-1500": (1500, np.stack([np.zeros(1499, int), np.arange(1, 1500)], 1)),
}


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("precision", [fvmbaseExt.AMG.FP64, fvmbaseExt.AMG.MIXED], ids=["fp64", "mixed"])
def test_one_level_solve(name, precision):
    n, e = GRAPHS[name]
    rng = np.random.default_rng(n)
    v = rng.uniform(0.1, 1.0, len(e)) * rng.choice([-1.0, 1.0], len(e))
    i, j = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    w = np.concatenate([v, v])
    o = np.lexsort((j, i))
    row = np.zeros(n + 1, np.int32)
    row[1:] = np.cumsum(np.bincount(i, minlength=n))
    diag = -(1.1 * np.bincount(i, weights=np.abs(w), minlength=n) + 0.05)
    diag[rng.uniform(size=n) < 0.2] *= -1.0
    b = rng.standard_normal(n)
    A = np.diag(diag)
    A[i, j] = w
    xref = np.linalg.solve(A, -b)
    amg = fvmbaseExt.AMG()
    amg.maxCoarseLevels = 0
    amg.coarseSolver = fvmbaseExt.AMG.COARSE_DIRECT
    amg.precision = precision
    amg.relativeTolerance = 1e-10
    amg.nMaxIterations = 20
    x, info = amg.solve_csr(row, j[o].astype(np.int32), diag, w[o], b)
    assert info["converged"]
    if precision == fvmbaseExt.AMG.FP64:
        assert info["iterations"] == 1
    assert np.linalg.norm(x - xref) <= 1e-8 * np.linalg.norm(xref)
    # the same bits again
    y, _ = amg.solve_csr(row, j[o].astype(np.int32), diag, w[o], b)
    np.testing.assert_array_equal(x, y)
