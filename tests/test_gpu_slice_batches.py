"""A level whose operand slices would pass the workspace: its fronts go in batches."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from uhm_gb300 import api

pytestmark = pytest.mark.gpu

N, COUNT = 400, 2400         # fronts of one level: 4.1 MB of LU slices each, 9.8 GB


@pytest.mark.parametrize("method", [uo.LU_PIV, uo.CHOL])
def test_a_wide_level_goes_in_batches(native_lib, method):
    """Trees of one front each, LU with 9.8 GB of slices (Cholesky 4.9), so three (two)
    batches.  The device holds the fronts, the elements, the inverses of the 64 x 64
    diagonal blocks (LU: of L and U) and at most 4 GiB of slices, and 5 % for the rest.  Solutions: 3 n u times a condition number of 40 (Cholesky 4)."""
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    rng = np.random.default_rng(8)
    q, _ = np.linalg.qr(rng.standard_normal((N, N)))
    sym = (q * rng.uniform(1.0, 4.0, N)) @ q.T
    skew = rng.standard_normal((N, N)) / np.sqrt(N)
    a = 0.5 * (sym + sym.T) + (0 if method == uo.CHOL else 0.5 * (skew - skew.T))
    m = api.Mesh()
    elems = []
    for k in range(COUNT):
        e = m.add_element(0)
        m.element_add_node(e, m.add_node(k, N))
        elems.append(e)
    m.lock()
    m.create_matrix_without_buffer(api.UHM_REAL, 1)
    scale = 1.0 + np.arange(COUNT) / COUNT
    b = rng.standard_normal((N, 1))
    for k, e in enumerate(elems):
        m.copy_in(e, [k], api.UHM_LHS, scale[k] * a)
        m.copy_in(e, [k], api.UHM_RHS, b)
    free = torch.cuda.mem_get_info()[0]
    m.factor(method)
    used = free - torch.cuda.mem_get_info()[0]
    m.solve(method)
    x = m.node_solution(np.arange(COUNT, dtype=np.int32), np.full(COUNT, N), 1).reshape(COUNT, N)
    ref = np.linalg.solve(a, b)[:, 0][None, :] / scale[:, None]
    cond = 4 if method == uo.CHOL else 40
    assert (np.abs(x - ref).max(axis=1) <= 3 * N * 2.0 ** -53 * cond * np.abs(ref).max(axis=1)).all()
    inverses = COUNT * -(-N // 64) * 64 * 64 * 8 * (1 if method == uo.CHOL else 2)
    assert used <= 1.05 * (2 * COUNT * N * N * 8 + inverses + (4 << 30)), used
