"""Device scratch of the Ozaki path (splab_gemm_workspace_size; no GPU needed)."""
import pytest

import spla_b200 as spla


@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
@pytest.mark.parametrize("m,n,k", [(1000, 900, 4000), (64, 30000, 2048), (17, 33, 100000)])
def test_operands_read_in_place_need_no_more_than_k_major_ones(dt, m, n, k):
    """The partial sums of their row norms lie where their residues go next."""
    size = [spla.splab_gemm_workspace_size(dt, spla.PATH_OZAKI, opA, opB, m, n, k)
            for opA, opB in ((1, 0), (0, 0), (1, 1), (0, 1))]
    assert size == size[:1] * 4
