"""AUTO for tall products of modest k, where the row norms of a k-major A (one block
per row) decide: measured times (us) of DMMA and the Ozaki path beside each shape."""
import pytest

import spla_b200 as spla

pytestmark = pytest.mark.gpu

R64, C64 = 1, 3


@pytest.mark.parametrize("dt,opA,m,n,k,want", [
    (C64, 2, 200000, 256, 256, spla.PATH_DMMA),   # 3236, 3627
    (C64, 2, 500000, 256, 256, spla.PATH_DMMA),   # 8111, 8925
    (C64, 2, 60000, 512, 200, spla.PATH_DMMA),    # 1547, 1706
    (R64, 1, 200000, 512, 384, spla.PATH_DMMA),   # 2676, 3235
    (R64, 1, 200000, 256, 700, spla.PATH_DMMA),   # 2505, 2880
    (C64, 0, 500000, 256, 256, spla.PATH_OZAKI),  # 7898, 6510
    (C64, 0, 100000, 512, 512, spla.PATH_OZAKI),
    (C64, 2, 100000, 512, 512, spla.PATH_OZAKI)])
def test_auto_counts_the_norms_of_short_rows(dt, opA, m, n, k, want):
    assert spla.lib().splab_gemm_path(dt, spla.PATH_AUTO, opA, 0, m, n, k) == want
