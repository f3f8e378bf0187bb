"""The 32 x 32 tiles of the FP64 path (few CTAs, or default tiles that pad C): edges of
the tile, the k-step and the split, every operand layout, against the device
double-double product."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", ["float32", "float64", "complex64", "complex128"])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (31, 33, 7), (32, 32, 64), (33, 65, 129),
                                   (100, 80, 5000), (129, 129, 300), (5, 700, 90)])
def test_small_tiles(dt, m, n, k):
    """|C - R| <= k 2^-52 sum |a| |b| <= k 2^-52 |a_i| |b_j| for the FP64 sums (float adds
    the rounding of C), beta and a padded C included."""
    import torch
    import spla_b200 as spla
    cplx = dt.startswith("complex")
    tdt = getattr(torch, dt)
    wide = torch.complex128 if cplx else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(m + 10 * n + 100 * k)
    ctx = spla.Context(spla.PU_GPU)
    ctx.set_fp64_path(spla.PATH_DMMA)
    rows = torch.randn((m, k), dtype=tdt, device="cuda", generator=g)  # rows of op(A)
    cols = torch.randn((n, k), dtype=tdt, device="cuda", generator=g)  # columns of op(B)
    C0 = torch.randn((n, m + 2), dtype=tdt, device="cuda", generator=g)
    norms = (torch.linalg.vector_norm(cols.to(wide), dim=1)[:, None] *
             torch.linalg.vector_norm(rows.to(wide), dim=1)[None, :])
    for opA, opB in ((0, 0), (1, 0), (2, 2), (0, 1)):
        a = rows.T.contiguous() if opA == 0 else rows
        b = cols if opB == 0 else cols.T.contiguous()
        lda, ldb = (m if opA == 0 else k), (k if opB == 0 else n)
        C = C0.clone()
        spla.gemm(opA, opB, m, n, k, 1.0, a, lda, b, ldb, -1.0, C, m + 2, ctx)
        R = torch.zeros((n, m), dtype=wide, device="cuda")
        assert spla.gemm_dd("complex128" if cplx else "float64", opA, opB, m, n, k, a.to(wide),
                            lda, b.to(wide), ldb, R, m) == 0
        torch.cuda.synchronize()
        R -= C0[:, :m].to(wide)
        bound = (k + 4) * 2.0 ** -52 * (norms + C0[:, :m].abs().double())
        if dt in ("float32", "complex64"):
            bound = bound + 2.0 ** -23 * R.abs()
        assert bool(((C[:, :m].to(wide) - R).abs() <= bound).all()), (opA, opB)
        assert torch.equal(C[:, m:], C0[:, m:])
