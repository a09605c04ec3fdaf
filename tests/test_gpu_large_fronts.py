"""Schur complements and solutions of blocked fronts (too large for one CTA's
shared memory), and of small ones, against 64-bit numpy, at sizes around the kernels' edges:
64-column steps, 256-column outer panels, 128 x 128 update tiles, 16-column
row blocks.

Two leaf fronts (fs own rows, ss shared rows) below a root of the ss shared
rows.  The element matrices are random symmetric positive definite (LU:
plus a random skew part) with eigenvalues in [1, 4], so the Schur complement
is well conditioned.  Tolerance, elementwise: the factorisation's backward
error is at most (fs + 8) u sqrt(a_ii a_jj) for the front's unit roundoff u, and it
reaches ABR multiplied by at most (1 + ||A21 A11^-1||)^2 <= 25 for this
spectrum."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from uhm_gb300 import api

pytestmark = pytest.mark.gpu

U = {"fp64": 2.0 ** -53, "fp32": 2.0 ** -24}


def _matrix(n, symmetric, rng):
    q, _ = np.linalg.qr(rng.standard_normal((n, n)))
    a = (q * rng.uniform(1.0, 4.0, n)) @ q.T
    a = 0.5 * (a + a.T)
    if not symmetric:
        s = rng.standard_normal((n, n)) / np.sqrt(n)
        a = a + 0.5 * (s - s.T)
    return a


def _mesh(fs, ss, symmetric, seed, n_rhs=1, mats=None):
    rng = np.random.default_rng(seed)
    m = api.Mesh()
    nodes = [m.add_node(0, fs), m.add_node(1, fs), m.add_node(2, ss)]
    leaves = [m.add_element(0), m.add_element(0)]
    root = m.add_element(-1)
    for k, e in enumerate(leaves):
        m.element_add_node(e, nodes[k])
        m.element_add_node(e, nodes[2])
        m.set_parent(e, root)
        m.add_child(root, e)
    m.lock()
    m.create_matrix_without_buffer(api.UHM_REAL, n_rhs)
    mats = mats or [_matrix(fs + ss, symmetric, rng) for _ in leaves]
    rhs = [rng.standard_normal((fs + ss, n_rhs)) for _ in leaves]
    for k, e in enumerate(leaves):
        m.copy_in(e, [k, 2], api.UHM_LHS, mats[k])
        m.copy_in(e, [k, 2], api.UHM_RHS, rhs[k])
    return m, leaves, mats, rhs


def _check(method, prec, fs, ss, seed, mats=None):
    m, leaves, mats, rhs = _mesh(fs, ss, method == uo.CHOL, seed, mats=mats)
    if prec == "fp32":
        m.set_mode(1, api.PREC_FP32, 1e-12, 10)
    m.factor(method)
    eid = m.fronts()[0]
    tol = 25 * (fs + 8) * U[prec]
    for k in range(2):
        a = mats[k]
        exact = a[fs:, fs:] - a[fs:, :fs] @ np.linalg.solve(a[:fs, :fs], a[:fs, fs:])
        got = m.front_block(int(eid[k]), "ABR")
        if method == uo.CHOL:
            exact = np.tril(exact)
        d = np.abs(np.diag(a)[fs:])
        assert (np.abs(got - exact) <= tol * np.sqrt(np.outer(d, d))).all(), (k, np.abs(got - exact).max())
    m.solve(method)
    x, ref = _solutions(m, fs, ss, mats, rhs)
    assert np.abs(x - ref).max() <= 3e-10 * np.abs(ref).max()   # 1e-12 times the condition number


def _solutions(m, fs, ss, mats, rhs):
    n, nr = 2 * fs + ss, rhs[0].shape[1]
    full, b = np.zeros((n, n)), np.zeros((n, nr))
    for k in range(2):
        i = np.concatenate([np.arange(fs) + k * fs, np.arange(2 * fs, n)])
        full[np.ix_(i, i)] += mats[k]
        b[i] += rhs[k]
    return m.node_solution(np.arange(3, dtype=np.int32), np.array([fs, fs, ss]), nr), np.linalg.solve(full, b)


# (fs, ss): one step; a step and one column; the outer panel's edge; one column past
# it; two panels with a remainder; one column
SIZES = [(64, 165), (65, 200), (256, 1), (257, 128), (300, 129), (449, 255), (1, 240)]


@pytest.mark.parametrize("fs,ss", SIZES)
@pytest.mark.parametrize("method,prec", [(uo.LU_PIV, "fp64"), (uo.LU_NOPIV, "fp32")])
def test_lu_front(native_lib, method, prec, fs, ss):
    _check(method, prec, fs, ss, 100 + fs)


@pytest.mark.parametrize("n_rhs", [2, 3, 5, 16])
@pytest.mark.parametrize("method", [uo.LU_PIV, uo.LU_NOPIV])
def test_lu_right_hand_sides(native_lib, method, n_rhs):
    """Groups of four, two and one right-hand sides through the flag-driven LU
    solves of blocked fronts (a ragged last block); tolerance 3 n u times a
    condition number of 40."""
    m, leaves, mats, rhs = _mesh(300, 129, False, 31, n_rhs)
    m.factor(method)
    m.solve(method)
    x, ref = _solutions(m, 300, 129, mats, rhs)
    assert np.abs(x - ref).max() <= 3 * 729 * U["fp64"] * 40 * np.abs(ref).max()


@pytest.mark.parametrize("n_rhs", [2, 3, 5, 16])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_cholesky_right_hand_sides(native_lib, prec, n_rhs):
    """Groups of one, two and four right-hand sides (the last one ragged) through
    the flag-driven Cholesky solves, ragged last blocks; the tolerance of _check."""
    m, leaves, mats, rhs = _mesh(300, 129, True, 32, n_rhs)
    if prec == "fp32":
        m.set_mode(1, api.PREC_FP32, 1e-12, 10)
    m.factor(uo.CHOL)
    m.solve(uo.CHOL)
    x, ref = _solutions(m, 300, 129, mats, rhs)
    assert np.abs(x - ref).max() <= 3e-10 * np.abs(ref).max()


@pytest.mark.parametrize("method,prec", [(uo.CHOL, api.PREC_FP64), (uo.CHOL, api.PREC_FP32),
                                         (uo.LU_PIV, api.PREC_FP64), (uo.LU_NOPIV, api.PREC_BF16X3)])
def test_lookahead_changes_no_bit(native_lib, method, prec):
    """Fronts of several outer panels whose updates run beside the next panel's
    steps (more launches): every entry meets the same operations in the same order."""
    got = []
    m, leaves, mats, rhs = _mesh(2500, 500, method == uo.CHOL, 33)
    for la in (0, 1):
        if prec != api.PREC_FP64:
            m.set_mode(1, prec, 1e-12, 10)
        m.set_tunables(lookahead=la)
        m.factor(method)
        launches = m.timing()["kernel_launches"]
        m.solve(method)
        eid = m.fronts()[0]
        got.append((launches, [m.front_block(int(e), "ABR") for e in eid[:2]],
                    m.node_solution(np.arange(3, dtype=np.int32), np.array([2500, 2500, 500]), 1)))
    assert got[1][0] > got[0][0]
    assert all((a == b).all() for a, b in zip(got[0][1], got[1][1])) and (got[0][2] == got[1][2]).all()


@pytest.mark.parametrize("fs,ss", SIZES)
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_cholesky_front(native_lib, prec, fs, ss):
    _check(uo.CHOL, prec, fs, ss, 200 + fs)


@pytest.mark.parametrize("prec,digits", [("fp32", (63, 127, 127, 64)), ("fp64", (63, 127, 127, 127, 127, 127, 64))])
def test_largest_digits(native_lib, prec, digits):
    """Panels whose 8-bit digits are all near their largest: the sums of 256 products
    pass 2^22 (and 2^24 between diagonals), beyond what a typical tile meets."""
    fs, ss = 256, 129
    v = sum(d * 256.0 ** -(k + 1) for k, d in enumerate(digits)) * 4
    a = np.diag(np.r_[np.full(fs, 256.0), np.full(ss, 3.0)])     # L11 = 16 I, L21 = v / 16; condition number 200
    a[fs:, :fs] = a[:fs, fs:] = v
    a[fs:, fs:] += v * v
    _check(uo.CHOL, prec, fs, ss, 35, mats=[a, a])


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_front_reports_status(native_lib, value):
    """A NaN or an infinity reaches the root's pivots through the leaf's Schur
    complement as NaN (an infinity becomes one in the panel's TRSM)."""
    m, leaves, mats, _ = _mesh(130, 140, True, 7)
    bad = np.zeros_like(mats[0])
    bad[40, 200] = bad[200, 40] = value
    m.copy_in(leaves[0], [0, 2], api.UHM_LHS, bad)
    with pytest.raises(api.UHMError) as ei:
        m.chol_with_free()
    assert ei.value.code == 13


@pytest.mark.parametrize("n_rhs", [1, 3, 4, 9])
@pytest.mark.parametrize("prec,fs,ss", [("fp64", 1, 5), ("fp64", 5, 3), ("fp64", 62, 98), ("fp64", 97, 30),
                                        ("fp32", 30, 1), ("fp32", 131, 93)])
def test_small_cholesky_front(native_lib, prec, fs, ss, n_rhs):
    """Fronts that fit one CTA: four-column steps with remainders, and the solves
    by whole blocks (up to three right-hand sides) or a warp each."""
    m, leaves, mats, rhs = _mesh(fs, ss, True, 300 + fs, n_rhs)
    if prec == "fp32":
        m.set_mode(1, api.PREC_FP32, 1e-12, 10)
    m.factor(uo.CHOL)
    eid = m.fronts()[0]
    for k in range(2):
        a = mats[k]
        exact = np.tril(a[fs:, fs:] - a[fs:, :fs] @ np.linalg.solve(a[:fs, :fs], a[:fs, fs:]))
        d = np.abs(np.diag(a)[fs:])
        got = m.front_block(int(eid[k]), "ABR")
        assert (np.abs(got - exact) <= 25 * (fs + 8) * U[prec] * np.sqrt(np.outer(d, d))).all(), k
    m.solve(uo.CHOL)
    x, ref = _solutions(m, fs, ss, mats, rhs)
    assert np.abs(x - ref).max() <= 3e-10 * np.abs(ref).max()
