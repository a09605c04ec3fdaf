"""The kernels' own reciprocals, square roots, quotients and scalings of integer sums
against numpy's, entry by entry, through fronts whose factors are single operations."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from tests.test_gpu_large_fronts import _mesh
from uhm_gb300 import api

pytestmark = pytest.mark.gpu


def _leaf(fs, ss, a, c, method, prec="fp64"):
    """The mesh of test_gpu_large_fronts with a as its first leaf's matrix; the second
    leaf adds c to the root's diagonal, which makes it regular."""
    other = np.diag(np.r_[np.ones(fs), np.full(ss, c)])
    m, leaves, mats, _ = _mesh(fs, ss, method == uo.CHOL, 1, mats=[a, other])
    if prec == "fp32":
        m.set_mode(1, api.PREC_FP32, 1e-12, 10)
    m.factor(method)
    e = int(m.fronts()[0][0])
    return lambda block: m.front_block(e, block)


def _values(n, lo, hi, rng):
    """Mantissas of every kind in [1, 2), exponents lo .. hi."""
    m = 1.0 + rng.random(n)
    m[: n // 8] = np.float64(2.0) - 2.0 ** -52 * rng.integers(1, 9, n // 8)
    m[n // 8: n // 4] = 1.0 + 2.0 ** -52 * rng.integers(0, 9, n // 4 - n // 8)
    return np.ldexp(m, rng.integers(lo, hi + 1, n))


@pytest.mark.parametrize("lo,hi", [(-3, 3), (-950, 950)])
def test_reciprocals(native_lib, lo, hi):
    """LU of a diagonal with ones below: the multipliers are the pivots' reciprocals, within an
    ulp of numpy's (correctly rounded but for near ties)."""
    fs, ss = 2048, 96
    rng = np.random.default_rng(lo + 5000)
    v = _values(fs, lo, hi, rng) * rng.choice([-1.0, 1.0], fs)
    a = np.zeros((fs + ss, fs + ss))
    a[np.arange(fs), np.arange(fs)] = v
    a[fs:, :fs] = 1.0
    got = _leaf(fs, ss, a, 1.0, uo.LU_NOPIV)("ABL")
    ref = 1.0 / v
    assert (np.abs(got - ref[None, :]) <= np.spacing(np.abs(ref))[None, :]).all()
    assert (got == ref[None, :]).mean() >= 0.999


@pytest.mark.parametrize("lo,hi", [(-3, 3), (-400, 400)])
def test_roots_and_quotients(native_lib, lo, hi):
    """A small FP64 Cholesky front with a diagonal block: roots and quotients as numpy's
    (rounded as the operations but for rare ties)."""
    fs, ss = 120, 40
    rng = np.random.default_rng(lo + 6000)
    v, w = _values(fs, lo, hi, rng), _values(ss * fs, -20, 20, rng).reshape(ss, fs)
    a = np.zeros((fs + ss, fs + ss))
    a[np.arange(fs), np.arange(fs)] = v
    a[fs:, :fs] = w
    a[:fs, fs:] = w.T
    block = _leaf(fs, ss, a, 4.0 * (w * w / v).sum(), uo.CHOL)
    root, quot = np.diag(block("ATL")), block("ABL")
    ref = w / np.sqrt(v)[None, :]
    assert (np.abs(root - np.sqrt(v)) <= np.spacing(np.sqrt(v))).all() and (root == np.sqrt(v)).mean() >= 0.98
    assert (np.abs(quot - ref) <= np.spacing(np.abs(ref))).all() and (quot == ref).mean() >= 0.98


@pytest.mark.parametrize("prec,lo,hi,c,tol,tiny", [
    ("fp64", -20, 19, 2.0 ** 50, 2.0 ** -51, 2.0 ** -1074), ("fp64", -535, 505, 2.0 ** 1020, 2.0 ** -51, 2.0 ** -1074),
    ("fp32", -10, 9, 2.0 ** 30, 2.0 ** -23, 2.0 ** -149), ("fp32", -72, 58, 2.0 ** 124, 2.0 ** -23, 2.0 ** -149)])
def test_scaled_sums(native_lib, prec, lo, hi, c, tol, tiny):
    """One product per entry of the Schur complement, -l u, of operands with exponents lo .. hi
    (results from subnormal to near the largest): the integers' last place is at most
    2^-52 (FP32 2^-30) of the product, and one rounding."""
    fs, ss = 64, 256
    rng = np.random.default_rng(hi)
    l, u = (_values(ss, lo, hi, rng) * rng.choice([-1.0, 1.0], ss) for _ in range(2))
    if prec == "fp32":
        l, u = (v.astype(np.float32).astype(np.float64) for v in (l, u))
    a = np.zeros((fs + ss, fs + ss))
    a[:fs, :fs] = np.eye(fs)
    k = np.arange(ss) % fs
    a[fs + np.arange(ss), k] = l
    a[k, fs + np.arange(ss)] = u
    got = _leaf(fs, ss, a, c, uo.LU_NOPIV, prec)("ABR")
    ref = np.where(k[:, None] == k[None, :], -np.outer(l, u), 0.0)
    assert (np.abs(got - ref) <= tol * np.abs(ref) + tiny).all()
