"""The tuner sees every choice of the LU programs."""
import pytest

from oracle import uhm_oracle as uo
from tests.test_gpu_large_fronts import _mesh

pytestmark = pytest.mark.gpu


def test_lookahead_is_timed_for_lu(native_lib):
    """Fronts of 3,000 and 500 rows in plain FP64: of the candidates only the lookahead
    changes the programs, so that one is timed beside the defaults (not the one-CTA
    panels in global memory)."""
    m, leaves, mats, rhs = _mesh(2500, 500, False, 90)
    assert m.autotune(uo.LU_PIV, reps=1)["timed"] == 2
