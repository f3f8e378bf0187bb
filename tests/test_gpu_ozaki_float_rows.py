"""Float rows sliced in FP32: rows near the ends of the exponent range (subnormal rows are
scaled by more than 2^127), rows whose reals span 2^60, k-major and read in place, ragged
lengths, against the device double-double product of the same numbers."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["float32", "complex64"])
@pytest.mark.parametrize("opA", [0, 1, 2])
@pytest.mark.parametrize("m,n,k", [(1, 1, 7), (37, 65, 515), (130, 96, 2051), (65, 130, 40009),
                                   (13, 20, 140003)])  # the last scales in one pass
def test_float_row_exponents(dt, opA, m, n, k):
    """|C - R| <= |a_i| |b_j| sqrt(K) 2^-32 + |R| 2^-23 + 2^-148, K reals per row: each
    real is rounded by half a unit at a scaled norm of at least 2^33, C to a float (by
    half a subnormal unit per part at least)."""
    import torch
    import spla_b200 as spla
    cplx = dt.startswith("complex")
    wide = torch.complex128 if cplx else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(m + 7 * n + opA)
    A = torch.randn((m, k), dtype=getattr(torch, dt), device="cuda", generator=g)
    B = torch.randn((n, k), dtype=getattr(torch, dt), device="cuda", generator=g)
    # powers of two: exact, but for the rows that become subnormal (their rounded reals
    # are the inputs)
    exps = torch.tensor([0, -140, 96, -126, -60, 1], device="cuda")
    e = exps[torch.arange(m, device="cuda") % len(exps)]
    half = e // 2
    A *= torch.ldexp(torch.ones_like(half, dtype=torch.float32), half)[:, None]
    A *= torch.ldexp(torch.ones_like(half, dtype=torch.float32), e - half)[:, None]
    B[:, ::3] *= 2.0 ** -60
    X = A.t().contiguous() if opA == 0 else A  # column-major m x k, or k x m
    ldx = m if opA == 0 else k
    nbytes = spla.splab_gemm_workspace_size(dt, spla.PATH_OZAKI, opA, 0, m, n, k)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    C = torch.zeros((n, m), dtype=A.dtype, device="cuda")
    assert spla.splab_gemm(dt, spla.PATH_OZAKI, opA, 0, m, n, k, 1.0, X, ldx, B, k, 0.0, C, m,
                           workspace=ws, workspace_bytes=nbytes) == 0
    torch.cuda.synchronize()
    assert spla.splab_gemm_check(dt, spla.PATH_OZAKI, opA, 0, m, n, k, workspace=ws) == 0
    R = torch.zeros((n, m), dtype=wide, device="cuda")
    assert spla.gemm_dd("complex128" if cplx else "float64", opA, 0, m, n, k, X.to(wide), ldx,
                        B.to(wide), k, R, m) == 0
    torch.cuda.synchronize()
    norms = (torch.linalg.vector_norm(B.to(wide), dim=1)[:, None] *
             torch.linalg.vector_norm(A.to(wide), dim=1)[None, :])
    K = (2 if cplx else 1) * k
    bound = norms * (K ** 0.5 * 2.0 ** -32) + R.abs() * 2.0 ** -23 + 2.0 ** -148
    assert bool(((C.to(wide) - R).abs() <= bound).all())
