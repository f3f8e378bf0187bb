"""Byte residues of any number of rows (columns padded to 16 bytes) and of several
k-chunks: the tensor-core reconstruction takes all planes of all chunks and gives the
bits of the CUDA-core one (SPLAB_OZAKI_RECON_TC=0, which adds the chunks' residues),
and both match the device double-double product."""
import os

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,m,n,k", [
    ("float64", 1, 1, 600),            # one row, one column
    ("float64", 15, 40, 4096),         # fewer rows than a 16-byte line
    ("float64", 129, 33, 20000),       # four k-chunks, a ragged block of rows
    ("float32", 250, 256, 30000),      # seven
    ("complex64", 77, 300, 9000),      # three
    ("complex128", 127, 65, 10000),    # two: all 64 planes
    ("complex128", 257, 70, 145000),   # two from the INT32 bound, m just past a block
    ("complex128", 40, 24, 300000),    # three: int32 sums
    ("float64", 300, 200, 130000),     # two chunks at least, real
])
def test_any_rows_and_chunks(dt, m, n, k):
    """|C - R| <= |a_i| |b_j| (sqrt(K) 2^-55 + 2^-51), K reals per row: each real is
    rounded by half a unit at a scaled norm of at least 2^56 (float: 2^33, plus its own
    rounding of C)."""
    import torch
    import spla_b200 as spla
    cplx = dt.startswith("complex")
    wide = torch.complex128 if cplx else torch.float64
    g = torch.Generator(device="cuda")
    g.manual_seed(m * 31 + n)
    A = torch.randn((m, k), dtype=getattr(torch, dt), device="cuda", generator=g)
    B = torch.randn((n, k), dtype=getattr(torch, dt), device="cuda", generator=g)
    op = 2 if cplx else 1
    nbytes = spla.splab_gemm_workspace_size(dt, spla.PATH_OZAKI, op, 0, m, n, k)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    out = []
    for tc in ("1", "0"):
        os.environ["SPLAB_OZAKI_RECON_TC"] = tc
        try:
            C = torch.zeros((n, m), dtype=A.dtype, device="cuda")
            ws.fill_(255)  # nothing of an earlier call is relied on
            assert spla.splab_gemm(dt, spla.PATH_OZAKI, op, 0, m, n, k, 1.0, A, k, B, k, 0.0, C, m,
                                   workspace=ws, workspace_bytes=nbytes) == 0
            torch.cuda.synchronize()
            assert spla.splab_gemm_check(dt, spla.PATH_OZAKI, op, 0, m, n, k, workspace=ws) == 0
            out.append(C)
        finally:
            os.environ.pop("SPLAB_OZAKI_RECON_TC", None)
    assert torch.equal(torch.view_as_real(out[0]) if cplx else out[0],
                       torch.view_as_real(out[1]) if cplx else out[1])
    R = torch.zeros((n, m), dtype=wide, device="cuda")
    assert spla.gemm_dd("complex128" if cplx else "float64", op, 0, m, n, k, A.to(wide), k,
                        B.to(wide), k, R, m) == 0
    torch.cuda.synchronize()
    norms = (torch.linalg.vector_norm(B.to(wide), dim=1)[:, None] *
             torch.linalg.vector_norm(A.to(wide), dim=1)[None, :])
    K = (2 if cplx else 1) * k
    if dt in ("complex128", "float64"):
        bound = norms * (K ** 0.5 * 2.0 ** -55 + 2.0 ** -51)
    else:
        bound = norms * (K ** 0.5 * 2.0 ** -32 + 2.0 ** -51) + R.abs() * 2.0 ** -23
    assert bool(((out[0].to(wide) - R).abs() <= bound).all())
