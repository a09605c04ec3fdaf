"""Solutions of plain FP64 fronts against numpy's, within 3 n u times the condition
number (at most 4 for the symmetric matrices, 40 with the skew part), u = 2^-53."""
import numpy as np
import pytest

from oracle import uhm_oracle as uo
from tests.test_gpu_large_fronts import SIZES, _mesh, _solutions

pytestmark = pytest.mark.gpu

SMALL = [(1, 5), (5, 3), (62, 98), (97, 30)]


@pytest.mark.parametrize("n_rhs", [1, 3, 4])
@pytest.mark.parametrize("fs,ss", SIZES + SMALL + [(1200, 300)])
@pytest.mark.parametrize("method", [uo.CHOL, uo.LU_PIV, uo.LU_NOPIV])
def test_solution(native_lib, method, fs, ss, n_rhs):
    m, leaves, mats, rhs = _mesh(fs, ss, method == uo.CHOL, 400 + fs, n_rhs)
    m.factor(method)
    m.solve(method)
    x, ref = _solutions(m, fs, ss, mats, rhs)
    cond = 4 if method == uo.CHOL else 40
    assert np.abs(x - ref).max() <= 3 * (2 * fs + ss) * 2.0 ** -53 * cond * np.abs(ref).max()
