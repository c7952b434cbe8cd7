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


def _scaled(scales, precision, kind):
    """Histories and solutions of both paths, matrix and right-hand side
    scaled: neither the place nor the size of a rounding may differ. Row by
    row the scale of the matrix varies by 2^20 in the last of them."""
    row, col, diag, off, b = _grid(60, 41)
    matrix, rhs, vary = scales
    s = np.full(len(diag), matrix)
    if vary:
        # symmetric: couplings take the smaller scale of their two rows
        s = matrix * 2.0 ** np.random.default_rng(5).integers(-10, 11, len(diag))
    rows = np.repeat(np.arange(len(diag)), np.diff(row))
    out = []
    for launches in (False, True):
        amg = fvmbaseExt.AMG()
        amg.precision = precision
        amg.nPreSweeps = 1
        amg.smootherType = kind
        amg.nMaxIterations = 3
        amg.relativeTolerance = 1e-30
        amg.absoluteTolerance = 0.0
        if launches:
            amg.planThreadsPerRow = 1
        x, info = amg.solve_csr(row, col, diag * s, off * np.minimum(s[rows], s[col]), b * rhs)
        out.append((x, info["history"], info["launches"]))
    (x0, h0, l0), (x1, h1, l1) = out
    assert np.all(np.isfinite(x1)) and len(h1) > 1 and l0 < l1
    np.testing.assert_array_equal(h0, h1)
    np.testing.assert_array_equal(x0, x1)
    np.testing.assert_array_equal(np.signbit(x0), np.signbit(x1))


# FP64: subnormal and nearly so (reciprocals that overflow), at both ends,
# quotients near the ends of the format
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("scales", [(1.0, 1e-305, False), (1.0, 1e290, False), (1e-310, 1e-310, False),
                                    (1e-305, 1e-290, False), (1e290, 1e290, False), (1e-150, 1e150, False),
                                    (1e200, 1e-100, False), (2.0 ** -300, 1.0, True), (2.0 ** 300, 1.0, True)], ids=str)
def test_scales_fp64(scales, kind):
    _scaled(scales, fvmbaseExt.AMG.FP64, kind)


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("scales", [(1.0, 1e-33, False), (1.0, 1e-42, False), (1.0, 1e33, False),
                                    (1e-42, 1e-42, False), (1e-38, 1e-33, False), (1e33, 1e33, False),
                                    (1e-15, 1e15, False), (1e20, 1e-20, False), (2.0 ** -30, 1.0, True),
                                    (2.0 ** 60, 1.0, True)], ids=str)
def test_scales_mixed(scales, kind):
    _scaled(scales, fvmbaseExt.AMG.MIXED, kind)
