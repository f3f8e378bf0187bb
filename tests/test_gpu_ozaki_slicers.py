"""The Ozaki path's two slicers of complex double rows against each other: k-major
rows go through the INT8 digit sums (oz_slice_mma), operands read in place through
the FP32 ones (oz_slice_mn). Both round the same scaled integers, and their residues
agree modulo every modulus, so C is bit-identical."""
import pytest

pytestmark = pytest.mark.gpu


def _gemm(opA, opB, m, n, k, A, lda, B, ldb):
    import torch
    import spla_b200 as spla
    nbytes = spla.splab_gemm_workspace_size("complex128", spla.PATH_OZAKI, opA, opB, m, n, k)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    C = torch.full((n, m), 7.0, dtype=torch.complex128, device="cuda")
    assert spla.splab_gemm("complex128", spla.PATH_OZAKI, opA, opB, m, n, k, 0.5 - 0.25j, A, lda,
                           B, ldb, 0.0, C, m, workspace=ws, workspace_bytes=nbytes) == 0
    torch.cuda.synchronize()
    return C


def _stored(X, pad, offset):
    """Rows of X k-major with `pad` elements between them, starting `offset` doubles
    into a buffer (one: 8 bytes off the 16-byte boundary); and their leading dimension."""
    import torch
    ld = X.shape[1] + pad
    buf = torch.full((2 * ld * X.shape[0] + 1,), float("nan"), dtype=torch.float64, device="cuda")
    view = buf[offset:offset + 2 * ld * X.shape[0]].view(X.shape[0], ld, 2)
    view[:, :X.shape[1]] = torch.view_as_real(X)
    return view, ld


@pytest.mark.parametrize("k", [1, 63, 64, 65, 128, 129, 300, 384, 640, 4100, 20000])
@pytest.mark.parametrize("m,n,pad,offset", [(1, 1, 0, 0), (3, 17, 0, 1), (130, 66, 3, 0),
                                            (33, 259, 1, 1)])
def test_k_major_and_in_place_rows_give_the_same_product(m, n, pad, offset, k):
    """Rows of 2, 4, 6, 10 and more steps of 128 reals, with ragged ends, one warp
    and several per row, rows on and off 16-byte boundaries, and rows of very
    different magnitude (what lies between the rows is NaN and not read)."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 * m + k)
    X = torch.randn((m, k), dtype=torch.complex128, device="cuda", generator=g)  # op(A)
    Y = torch.randn((n, k), dtype=torch.complex128, device="cuda", generator=g)  # op(B)^T
    X[m // 2] *= 1e-200
    Y[n // 2] *= 1e150
    Y[:, : k // 2] *= torch.logspace(-12, 0, n, dtype=torch.float64, device="cuda")[:, None]
    (a, lda), (b, ldb) = _stored(X, pad, offset), _stored(Y, pad, offset)
    (ah, ldah) = _stored(X.conj().resolve_conj(), pad, offset)
    (at, ldat), (bt, ldbt) = (_stored(Z.T.contiguous(), pad, offset) for Z in (X, Y))
    C = _gemm(1, 0, m, n, k, a, lda, b, ldb)
    assert bool(torch.isfinite(torch.view_as_real(C)).all())
    assert torch.equal(C, _gemm(2, 0, m, n, k, ah, ldah, b, ldb))
    assert torch.equal(C, _gemm(0, 0, m, n, k, at, ldat, b, ldb))
    assert torch.equal(C, _gemm(1, 1, m, n, k, a, lda, bt, ldbt))
    assert torch.equal(C, _gemm(0, 1, m, n, k, at, ldat, bt, ldbt))
