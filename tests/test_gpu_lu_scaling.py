"""LU fronts whose unknowns and equations have different units: the updates by
8-bit slices share an exponent per row of L21 and per column of U12, so the
factor columns have to be balanced before they are cut, and what no balance
serves has to be left to plain multiply-adds.

Two leaf fronts (fs own rows, ss shared rows) below a root, as in
test_gpu_large_fronts.  The Schur complements are compared with exact ones in
more bits, each entry relative to its row's and column's units.
Tolerance: 16 times the error that numpy's own elimination of the same matrix in the
front's precision makes (the same pivots, the same error bound)."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from tests.test_gpu_large_fronts import _matrix, _mesh, _solutions
from uhm_gb300 import api, hpfem

pytestmark = pytest.mark.gpu

FP = {"fp64": np.float64, "fp32": np.float32}


def _eliminate(a, fs, pivoting):
    """The Schur complement of a's first fs rows, in a's type: 64 columns at a time,
    each update's product formed before it is subtracted."""
    a = a.copy()
    n = a.shape[0]
    for k0 in range(0, fs, 64):
        k1 = min(k0 + 64, fs)
        for k in range(k0, k1):
            if pivoting:
                p = k + int(np.argmax(np.abs(a[k:fs, k])))
                if p != k:
                    a[[k, p]] = a[[p, k]]
            a[k + 1:, k] = a[k + 1:, k] / a[k, k]
            a[k + 1:, k + 1:k1] -= np.outer(a[k + 1:, k], a[k, k + 1:k1])
        for k in range(k0, k1):
            a[k + 1:k1, k1:] -= np.outer(a[k + 1:k1, k], a[k, k1:])
        a[k1:, k1:] -= a[k1:, k0:k1] @ a[k0:k1, k1:]
    return a[fs:, fs:]


def _exact_columns(a, fs, cols):
    """Columns cols of the Schur complement, in numpy's widest type (FP32: a is in 64
    bits and all columns are as quick)."""
    if a.dtype == np.float32:
        return _eliminate(a.astype(np.float64), fs, True)[:, cols]
    a = a.astype(np.longdouble)
    lu, x = a[:fs, :fs].copy(), a[:fs, fs + cols].copy()
    for k in range(fs):
        p = k + int(np.argmax(np.abs(lu[k:, k])))
        for v in (lu, x):
            v[[k, p]] = v[[p, k]]
        f = lu[k + 1:, k] / lu[k, k]
        lu[k + 1:, k + 1:] -= np.outer(f, lu[k, k + 1:])
        x[k + 1:] -= np.outer(f, x[k])
    for k in range(fs - 1, -1, -1):
        x[k] /= lu[k, k]
        x[:k] -= np.outer(lu[:k, k], x[k])
    return a[fs:, fs + cols] - a[fs:, :fs] @ x


def _check_front(method, prec, fs, ss, mats, r, c):
    """mats: the leaves' matrices, r and c: units of their rows and columns (powers of
    two)."""
    m, leaves, mats, rhs = _mesh(fs, ss, False, 5, mats=mats)
    if prec == "fp32":
        m.set_mode(1, api.PREC_FP32, 1e-12, 10)
    m.factor(method)
    a = mats[0].astype(FP[prec])
    cols = np.sort(np.random.default_rng(3).choice(ss, min(ss, 40), replace=False))
    exact = _exact_columns(a, fs, cols)
    units = np.outer(r[fs:], c[fs + cols])
    if method == uo.CHOL:                       # lower triangle only
        units[np.arange(ss)[:, None] < cols[None, :]] = np.inf
    plain = float((np.abs(_eliminate(a, fs, method == uo.LU_PIV)[:, cols] - exact) / units).max())
    got = float((np.abs(m.front_block(int(m.fronts()[0][0]), "ABR")[:, cols] - exact) / units).max())
    assert got <= 16 * plain, (got, plain)
    return m, mats, rhs


def _units(kind, step, n, rng):
    """Units of rows and of columns: a factor of 2^step between neighbours (rows,
    columns, both alike), or any of 2^-step .. 2^step at random for both."""
    if kind == "random":
        return 2.0 ** rng.integers(-step, step + 1, n), 2.0 ** rng.integers(-step, step + 1, n)
    d = 2.0 ** (step * (np.arange(n) % 2))
    one = np.ones(n)
    return {"rows": (d, one), "columns": (one, d), "both": (d, d)}[kind]


@pytest.mark.parametrize("kind,step", [("rows", 20), ("rows", 33), ("columns", 33), ("both", 20), ("both", 27),
                                       ("random", 12)])
@pytest.mark.parametrize("method", [uo.LU_PIV, uo.LU_NOPIV])
@pytest.mark.parametrize("prec,fs,ss", [("fp64", 300, 129), ("fp32", 320, 200)])
def test_units(native_lib, prec, fs, ss, method, kind, step):
    """Steps of 64 columns, an outer panel's update and a remainder; FP32 with units
    within its range."""
    if prec == "fp32":
        step = min(step, 20)
    rng = np.random.default_rng(1000 + step)
    r, c = _units(kind, step, fs + ss, rng)
    base = [_matrix(fs + ss, False, rng) for _ in range(2)]
    if prec == "fp32":
        base = [b.astype(np.float32).astype(np.float64) for b in base]
    m, mats, rhs = _check_front(method, prec, fs, ss, [r[:, None] * b * c[None, :] for b in base], r, c)
    # the solution, in the columns' units: condition number of the equilibrated matrix
    # below 40, and pivots of the scaled one (growth as above): FP64, 10^4 n u
    m.solve(method)
    n = 2 * fs + ss
    i = [np.concatenate([np.arange(fs) + k * fs, np.arange(2 * fs, n)]) for k in range(2)]
    rr, cc = np.empty(n), np.empty(n)
    full, b = np.zeros((n, n)), np.zeros((n, 1))
    for k in range(2):
        rr[i[k]], cc[i[k]] = r, c
        full[np.ix_(i[k], i[k])] += base[k]
        b[i[k]] += rhs[k]
    x = m.node_solution(np.arange(3, dtype=np.int32), np.array([fs, fs, ss]), 1)
    z = np.linalg.solve(full, b / rr[:, None])
    err = np.abs(x * cc[:, None] - z).max()
    if prec == "fp64":
        assert err <= 1e4 * n * 2.0 ** -53 * np.abs(z).max()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_units_large_tiles(native_lib, prec):
    """Enough tiles for those of 128 x 128."""
    fs, ss = 260, 1300
    rng = np.random.default_rng(7)
    r, c = _units("both", 20, fs + ss, rng)
    base = [_matrix(fs + ss, False, rng) for _ in range(2)]
    _check_front(uo.LU_NOPIV, prec, fs, ss, [r[:, None] * b * c[None, :] for b in base], r, c)


@pytest.mark.parametrize("prec,weak,fs,ss", [("fp64", 30, 300, 129), ("fp64", 30, 260, 1300), ("fp32", 16, 320, 200),
                                             ("fp32", 16, 260, 1300)])
@pytest.mark.parametrize("side", ["rows", "columns"])
@pytest.mark.parametrize("method", [uo.LU_PIV, uo.LU_NOPIV])
def test_rows_that_no_balance_serves(native_lib, method, side, prec, weak, fs, ss):
    """Every seventh shared row couples to the odd own unknowns only, whose rows of U
    are 2^-weak of the others, and is of that size itself: its products are 2^-weak
    of the product of the two maxima whatever the columns are multiplied by.
    side columns: the same of the transpose."""
    rng = np.random.default_rng(40)
    w = 2.0 ** -weak
    odd, seventh = np.arange(fs) % 2 == 1, np.arange(ss) % 7 == 3
    mats = []
    for _ in range(2):
        a11 = 3.0 * np.eye(fs)
        a11[np.ix_(~odd, ~odd)] += 0.5 * rng.standard_normal((int((~odd).sum()),) * 2) / np.sqrt(fs)
        a11[np.ix_(odd, odd)] += 0.5 * rng.standard_normal((int(odd.sum()),) * 2) / np.sqrt(fs)
        a12, a21 = rng.standard_normal((fs, ss)), rng.standard_normal((ss, fs))
        a12[odd] *= w
        a21[np.ix_(seventh, ~odd)] = 0.0
        a21[np.ix_(~seventh, odd)] = 0.0
        a22 = rng.standard_normal((ss, ss)) + 2 * np.sqrt(ss) * np.eye(ss)
        a22[seventh] *= w
        a = np.block([[a11, a12], [a21, a22]])
        mats.append(np.ascontiguousarray(a.T if side == "columns" else a))
    u = np.ones(fs + ss)
    s = np.r_[np.ones(fs), np.where(seventh, w, 1.0)]
    r, c = (u, s) if side == "columns" else (s, u)
    _check_front(method, prec, fs, ss, mats, r, c)


def test_lookahead_changes_no_bit_with_units(native_lib):
    """Plain multiply-adds beside the next panel's steps read the panel's rows of L
    before its row interchanges reach them."""
    fs, ss, n0 = 2500, 500, 256
    rng = np.random.default_rng(50)
    w = 2.0 ** -30
    a = rng.standard_normal((fs + ss, fs + ss)) / np.sqrt(fs) + 0.1 * np.eye(fs + ss)
    odd = np.arange(n0) % 2 == 1
    seventh = np.arange(fs + ss) % 7 == 3
    seventh[:n0] = False
    first, others = a[:n0], a[n0:]
    first[:, :n0][np.ix_(odd, ~odd)] = 0.0
    first[:, :n0][np.ix_(~odd, odd)] = 0.0
    first[odd, n0:] *= w
    others[:, :n0][np.ix_(seventh[n0:], ~odd)] = 0.0
    others[:, :n0][np.ix_(~seventh[n0:], odd)] = 0.0
    others[seventh[n0:], n0:] *= w
    m, leaves, mats, rhs = _mesh(fs, ss, False, 51, mats=[a, a])
    got = []
    for la in (0, 1):
        m.set_tunables(lookahead=la)
        m.factor(uo.LU_PIV)
        eid = m.fronts()[0]
        got.append([m.front_block(int(e), q) for e in eid[:2] for q in ("ATL", "ATR", "ABL", "ABR")])
    assert all((x == y).all() for x, y in zip(*got))


def test_strong_coefficients(native_lib):
    """Convection-diffusion with coefficients of 1 to 10^4 and no units of its own: errors
    have to stay small in proportion to each column, or soft regions' large solutions see
    them.  Backward error at most 4 times that of the oracle's FP64 elimination of the
    same fronts."""
    spec = hpfem.convdiff3d(16, 3, seed=0)
    m = api.load_spec(spec)
    m.factor(uo.LU_PIV)
    m.solve(uo.LU_PIV)
    assert m.backward_error() <= 4 * uo.backward_error(spec, uo.solve_mesh(spec, uo.LU_PIV).x)


@pytest.mark.parametrize("kind,step", [("both", 20), ("both", 27), ("random", 12)])
@pytest.mark.parametrize("prec,fs,ss", [("fp64", 300, 129), ("fp32", 320, 200), ("fp64", 260, 1300)])
def test_cholesky_units(native_lib, prec, fs, ss, kind, step):
    """Symmetric fronts with units: a row of L is bounded by its diagonal entry's root, so
    that a shared exponent needs no scaling."""
    step = min(step, 20) if prec == "fp32" else step
    rng = np.random.default_rng(2000 + step)
    d = _units(kind, step, fs + ss, rng)[0] if kind == "random" else _units(kind, step, fs + ss, rng)[1]
    base = [_matrix(fs + ss, True, rng) for _ in range(2)]
    _check_front(uo.CHOL, prec, fs, ss, [d[:, None] * b * d[None, :] for b in base], d, d)
