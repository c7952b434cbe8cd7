"""The coarse levels of a cycle as one cluster kernel (csrc/cycle_tail.cu)
against the same cycle as separate launches: the rows are summed in the same
order and divided with the same rounding, so iterates, residual histories and
solutions are bitwise the same. A forced launch plan (planThreadsPerRow)
keeps every level on separate launches, which the parity tests check against
the reference.
"""
import numpy as np
import pytest

from fvm_b200 import fvmbaseExt

pytestmark = pytest.mark.gpu


def _grid(nx, ny, seed=1):
    """Five-point diffusion with lognormal conductivities, delta form."""
    rng = np.random.default_rng(seed)
    k = rng.lognormal(0.0, 1.0, (ny, nx))
    idx = np.arange(nx * ny).reshape(ny, nx)
    cx = 2.0 * k[:, :-1] * k[:, 1:] / (k[:, :-1] + k[:, 1:])
    cy = 2.0 * k[:-1] * k[1:] / (k[:-1] + k[1:])
    i = np.concatenate([idx[:, :-1].ravel(), idx[:, 1:].ravel(), idx[:-1].ravel(), idx[1:].ravel()])
    j = np.concatenate([idx[:, 1:].ravel(), idx[:, :-1].ravel(), idx[1:].ravel(), idx[:-1].ravel()])
    v = np.concatenate([cx.ravel(), cx.ravel(), cy.ravel(), cy.ravel()])
    return _csr(nx * ny, i, j, v, rng, idx[:, 0], 2.0 * k[:, 0])


def _wide(n, width, seed=2):
    """Symmetric random pattern of up to about 2 width entries per row at
    distances up to 4 width: rows wider than the registers hold."""
    rng = np.random.default_rng(seed)
    a = np.repeat(np.arange(n), width)
    b = a + rng.integers(1, 4 * width, len(a))
    ok = b < n
    e = np.unique(np.stack([a[ok], b[ok]], 1), axis=0)
    v = rng.uniform(0.1, 1.0, len(e))
    i = np.concatenate([e[:, 0], e[:, 1]])
    j = np.concatenate([e[:, 1], e[:, 0]])
    return _csr(n, i, j, np.concatenate([v, v]), rng, np.arange(0, n, 7), 1.0)


def _csr(n, i, j, v, rng, where, extra):
    o = np.lexsort((j, i))
    row = np.zeros(n + 1, np.int32)
    row[1:] = np.cumsum(np.bincount(i, minlength=n))
    diag = -np.bincount(i, weights=v, minlength=n)
    diag[where] -= extra
    return row, j[o].astype(np.int32), diag, v[o], rng.standard_normal(n)


def _both(system, kind=fvmbaseExt.AMG, iterations=4, **knobs):
    out = []
    for launches in (False, True):
        amg = fvmbaseExt.AMG()
        amg.nMaxIterations = iterations
        amg.relativeTolerance = 1e-30
        for name, value in knobs.items():
            setattr(amg, name, value)
        if launches:
            amg.planThreadsPerRow = 1
        solver = amg
        if kind is not fvmbaseExt.AMG:
            solver = kind()
            solver.preconditioner = amg
            solver.nMaxIterations = iterations
            solver.relativeTolerance = 1e-30
        out.append(solver.solve_csr(*system))
    (x0, i0), (x1, i1) = out
    np.testing.assert_array_equal(i0["history"], i1["history"])
    np.testing.assert_array_equal(x0, x1)
    assert np.all(np.isfinite(x0)) and i0["history"][-1] < i0["history"][0]
    assert i0["launches"] < i1["launches"]


# one CTA's rows (512), the cluster's (8192, 16384) and a row more or less
@pytest.mark.parametrize("shape", [(3, 2), (8, 4), (31, 16), (32, 16), (27, 19), (64, 128), (89, 93), (128, 128),
                                   (131, 126), (211, 190)])
def test_sizes(shape):
    _both(_grid(*shape), nPreSweeps=1)


@pytest.mark.parametrize("n,width", [(300, 3), (500, 7), (3000, 12), (700, 20), (9000, 5)])
def test_wide_rows(n, width):
    _both(_wide(n, width), nPreSweeps=1)


@pytest.mark.parametrize("cycle", [0, 1, 2])
@pytest.mark.parametrize("sweeps", [(0, 1), (1, 1), (2, 3)])
def test_cycles_and_sweeps(cycle, sweeps):
    _both(_grid(60, 41), cycleType=cycle, nPreSweeps=sweeps[0], nPostSweeps=sweeps[1])


@pytest.mark.parametrize("knobs", [dict(smootherType=1), dict(coarseJacobiRows=1 << 30), dict(coarseJacobiRows=200),
                                   dict(gsReverse=False, nPostSweeps=2), dict(coarsePostSweeps=2),
                                   dict(coarsestSize=100), dict(maxCoarseLevels=0), dict(maxCoarseLevels=2)],
                         ids=lambda d: "-".join("%s%s" % kv for kv in d.items()))
@pytest.mark.parametrize("precision", [fvmbaseExt.AMG.FP64, fvmbaseExt.AMG.MIXED], ids=["fp64", "mixed"])
def test_smoothers(knobs, precision):
    _both(_grid(90, 77), precision=precision, **dict(dict(nPreSweeps=1), **knobs))


@pytest.mark.parametrize("kind", [fvmbaseExt.CG, fvmbaseExt.BCGStab])
@pytest.mark.parametrize("pre", [0, 1])
def test_as_preconditioner(kind, pre):
    _both(_grid(100, 67), kind, nPreSweeps=pre)
