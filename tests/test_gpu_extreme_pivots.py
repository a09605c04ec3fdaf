"""Pivots at the ends of a type's range: infinite ones, and those whose reciprocal
overflows while the quotients by them are ordinary numbers."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from tests.test_gpu_large_fronts import _matrix, _mesh, _solutions
from tests.test_gpu_lu_scaling import _check_front
from uhm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ss,at", [(30, 29), (30, 13), (29, 28), (1, 0)])
def test_infinite_pivot_of_a_small_front(native_lib, ss, at):
    """A root front of ss rows, one CTA, the pivot in row `at` infinite: its root is
    infinite, its column zero and so is that unknown; the others solve the system without
    it.  Tolerance: 3 n u times a condition number of 4."""
    fs = 5
    m, leaves, mats, rhs = _mesh(fs, ss, True, 60 + at)
    mats[0][fs + at, fs + at] = np.inf
    m.copy_in(leaves[0], [0, 2], api.UHM_LHS, mats[0])
    m.factor(uo.CHOL)
    m.solve(uo.CHOL)
    mats[0][fs + at, fs + at] = 1.0
    mats[0] *= 2                                # (copied in twice: copy_in adds)
    x, _ = _solutions(m, fs, ss, mats, rhs)
    n = 2 * fs + ss
    full, b = np.zeros((n, n)), np.zeros((n, 1))
    for k in range(2):
        i = np.concatenate([np.arange(fs) + k * fs, np.arange(2 * fs, n)])
        full[np.ix_(i, i)] += mats[k]
        b[i] += rhs[k]
    keep = np.arange(n) != 2 * fs + at
    ref = np.zeros((n, 1))
    ref[keep] = np.linalg.solve(full[np.ix_(keep, keep)], b[keep])
    assert np.abs(x - ref).max() <= 12 * n * 2.0 ** -53 * np.abs(ref).max()


@pytest.mark.parametrize("prec,unit,fs,ss", [("fp64", 513, 130, 140), ("fp32", 65, 130, 140), ("fp64", 513, 300, 2000)])
@pytest.mark.parametrize("method", [uo.LU_NOPIV, uo.CHOL])
def test_subnormal_pivots(native_lib, method, prec, unit, fs, ss):
    """Unknowns in units of 2^-unit: their pivots are subnormal, their reciprocals beyond
    the range, the multipliers near 2^unit.  Panels of a cluster and of many CTAs; the
    tolerance of _check_front."""
    if method == uo.CHOL and prec == "fp32":
        pytest.skip("an FP32 Cholesky step takes reciprocal square roots, which do not overflow")
    rng = np.random.default_rng(80)
    d = np.ones(fs + ss)
    d[[10, 63, 64, 70, fs - 1]] = 2.0 ** -unit
    base = [_matrix(fs + ss, method == uo.CHOL, rng) for _ in range(2)]
    mats = [d[:, None] * b * d[None, :] for b in base]
    if prec == "fp32":
        mats = [a.astype(np.float32).astype(np.float64) for a in mats]
    _check_front(method, prec, fs, ss, mats, d, d)
