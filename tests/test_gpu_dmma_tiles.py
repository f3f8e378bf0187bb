"""Which tiles the DMMA planner takes for C padded by the default ones, told by the
splits of k in its workspace (times of the small tiles beside those of the default)."""
import pytest

import spla_b200 as spla

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,opA,opB,m,n,k,splits", [
    ("float64", 1, 0, 2000, 140, 30621, 6),   # default tiles (small: 7 splits, 1.16)
    ("float64", 1, 0, 2000, 140, 30620, 6),   # default (small: 7, 1.12)
    ("float64", 1, 0, 2000, 140, 30608, 7),   # small tiles (default: 6 splits, 0.93)
    ("float64", 1, 0, 600, 140, 20001, 19),   # default (small: 15, 1.06)
    ("float64", 1, 0, 300, 1500, 20001, 11),  # small (default: 4, 0.95)
    ("float64", 1, 0, 350, 350, 9001, 6),     # small (default: 16, 0.96)
    ("float64", 0, 1, 350, 350, 9001, 16),    # default (small: 7, 1.09)
    ("float64", 0, 1, 103, 155, 7872, 41),    # small (default: 55, 0.81)
    ("float64", 0, 1, 800, 800, 30621, 13),   # default (small: 7, 1.08)
    ("float64", 0, 1, 140, 2000, 30621, 14)]) # small (default: 9, 0.76)
def test_small_tiles_only_where_they_pay(dt, opA, opB, m, n, k, splits):
    nbytes = spla.splab_gemm_workspace_size(dt, spla.PATH_DMMA, opA, opB, m, n, k)
    assert nbytes == splits * m * n * 8
