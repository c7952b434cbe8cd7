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

from fvm_b200 import fvmbaseExt, meshgen
from helpers import gpu_model

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


def _system(name):
    """The systems of test_one_level_solve."""
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
    return row, j[o].astype(np.int32), diag, w[o], rng.standard_normal(n)


@pytest.mark.parametrize("name", list(GRAPHS))
def test_fp32_inverse_refines_by_its_rounding_alone(name):
    """The FP32 inverse and its product, per refinement step. With A = D (I + N)
    and |N| <= 1 / 1.1 in every row, | |A| |A^-1| |_1 <= (1 + 1/1.1) / (1 - 1/1.1)
    = 21. An inverse rounded once to FP32 and a product whose sums are at most 45
    additions deep leave at most 21 (1 + 45 + 1) 2^-24 < 6e-5 of the residual's L1
    norm (one for the right-hand side's rounding); three steps reach 1e-10."""
    amg = fvmbaseExt.AMG()
    amg.maxCoarseLevels = 0
    amg.coarseSolver = fvmbaseExt.AMG.COARSE_DIRECT
    amg.precision = fvmbaseExt.AMG.MIXED
    amg.relativeTolerance = 1e-10
    amg.nMaxIterations = 20
    _, info = amg.solve_csr(*_system(name))
    h = np.asarray(info["history"])
    assert h[1] <= 6e-5 * h[0]
    assert info["converged"] and info["iterations"] <= 3


@pytest.mark.parametrize("precision", [fvmbaseExt.AMG.FP64, fvmbaseExt.AMG.MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["quad", "tet", "hex"])
def test_second_level_ordered_by_cell_centroids(kind, precision):
    """A device-built coarse level, whose elimination order comes from the cells'
    centroids: one cycle without smoothing is x = -P Ac^-1 P^T b, compared with
    numpy's solve of the exported level. FP64: the solves of both sides lose at
    most n eps cond(Ac) each. FP32: a rounding of the inverse and a product 45
    additions deep, against |Ac^-1| |P^T b|."""
    mesh, f = {"quad": lambda: meshgen.config0(n=60, seed=0), "tet": lambda: meshgen.config1(m=10, seed=1),
               "hex": lambda: meshgen.config3(n=16, seed=3)}[kind]()
    fields = {"conductivity": f["k"], "source": f["s"]}

    def amg(device):
        a = fvmbaseExt.AMG()
        a.precision = precision
        a.coarseSolver = fvmbaseExt.AMG.COARSE_DIRECT
        a.maxCoarseLevels = 1
        a.nPreSweeps = a.nPostSweeps = 0
        a.nMaxIterations = 2  # one cycle
        a.setupOnDevice = device
        return a

    b = gpu_model(mesh, f["bc"], solver=amg(False), fields=fields)[0].getLinearSystem()[-1]
    tm, tf, m = gpu_model(mesh, f["bc"], solver=amg(True), fields=fields)
    before = tf.temperature[m.getCells()][: mesh["nCells"]].copy()
    sizes, (ci,) = tm.getHierarchy()
    n = sizes[0]
    assert 256 < n <= 4096
    tm.advance(1)
    delta = tf.temperature[m.getCells()][: mesh["nCells"]] - before
    A = tm.getLevelMatrix(1)
    Ac = np.diag(A["diag"])
    Ac[np.repeat(np.arange(n), np.diff(A["row"])), A["col"]] = A["val"]
    bc = np.bincount(ci, weights=b, minlength=n)
    inv = np.linalg.inv(Ac)
    xc = -inv @ bc
    if precision == fvmbaseExt.AMG.FP64:
        bound = np.full(n, 2 * n * 2.0 ** -52 * np.linalg.cond(Ac) * np.abs(xc).max())
    else:
        bound = 47 * 2.0 ** -24 * (np.abs(inv) @ np.abs(bc))
    # (the field itself holds before + delta)
    bound = bound[ci] + 2.0 ** -52 * np.abs(before + delta).max()
    assert np.all(np.abs(delta - xc[ci]) <= bound)
    assert np.abs(xc).max() > 1e3 * bound.max()
