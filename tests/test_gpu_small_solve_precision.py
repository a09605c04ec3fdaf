"""Solves of small FP32 Cholesky fronts whose panel passes 96 KB: FP64 arithmetic
on the FP32 factor."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from uhm_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_rhs", [(158, 1), (200, 1), (224, 1), (200, 3), (200, 5)])
def test_large_panels_are_solved_in_fp64(native_lib, n, n_rhs):
    """One front, A = L L^T with integers that every step keeps exact in FP32, so that the
    solution shows the solve's arithmetic alone.  Tolerance: 8 n u times A's condition
    number (u of FP64)."""
    rng = np.random.default_rng(n + n_rhs)
    low = 2.0 * np.eye(n)
    for i in range(1, n):
        k = rng.choice(i, min(i, 2), replace=False)
        low[i, k] = rng.choice([-1.0, 1.0], len(k))
    a = low @ low.T
    m = api.Mesh()
    nod = m.add_node(0, n)
    e = m.add_element(0)
    m.element_add_node(e, nod)
    m.lock()
    m.create_matrix_without_buffer(api.UHM_REAL, n_rhs)
    m.copy_in(e, [0], api.UHM_LHS, a)
    x = rng.standard_normal((n, n_rhs))
    b = a @ x
    m.copy_in(e, [0], api.UHM_RHS, b)
    m.set_mode(1, api.PREC_FP32, 1e-3, 10)      # accepted without a refinement step
    m.factor(uo.CHOL)
    m.solve(uo.CHOL)
    got = m.node_solution(np.array([0], dtype=np.int32), np.array([n]), n_rhs)
    assert np.abs(got - x).max() <= 8 * n * 2.0 ** -53 * np.linalg.cond(a) * np.abs(x).max()
