"""splab_gemm_dmma_noalloc where the 32 x 32 tiles' plan does not fit its static
array: the default tiles' plan, with one k-split, does."""
import ctypes as ct

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,opA,opB,m,n,k", [("complex64", 2, 0, 68, 36925, 301),
                                              ("complex64", 0, 0, 56268, 94, 1027),
                                              ("float32", 1, 0, 534, 10934, 3317)])
def test_default_tiles_where_small_ones_do_not_fit(dt, opA, opB, m, n, k):
    """FP64 sums, rounded to float once: |C - R| <= 2^-23 |R| + k 2^-50 |a_i| |b_j|."""
    import torch
    import spla_b200 as spla
    code = {"float32": 0, "complex64": 2}[dt]
    per_split = m * n * (16 if code == 2 else 8)
    assert 2 * per_split > 64 << 20  # not two splits fit
    L = spla.lib()
    vp, i, i64 = ct.c_void_p, ct.c_int, ct.c_int64
    L.splab_gemm_dmma_noalloc.argtypes = [i, i, i, i64, i64, i64, vp, vp, i64, vp, i64, vp, vp,
                                          i64, i, i64, i64, vp]
    L.splab_gemm_dmma_noalloc.restype = i
    g = torch.Generator(device="cuda")
    g.manual_seed(m)
    tdt = getattr(torch, dt)
    a = torch.randn((m, k) if opA else (k, m), dtype=tdt, device="cuda", generator=g)
    b = torch.randn((n, k), dtype=tdt, device="cuda", generator=g)
    C = torch.zeros((n, m), dtype=tdt, device="cuda")
    one, zero = (ct.c_float * 2)(1.0, 0.0), (ct.c_float * 2)(0.0, 0.0)
    lda = k if opA else m
    torch.cuda.synchronize()
    assert L.splab_gemm_dmma_noalloc(code, opA, opB, m, n, k, ct.cast(one, vp), a.data_ptr(), lda,
                                     b.data_ptr(), k, ct.cast(zero, vp), C.data_ptr(), m, 0, 0, 0,
                                     None) == 0
    wide = torch.complex128 if code == 2 else torch.float64
    R = torch.zeros((n, m), dtype=wide, device="cuda")
    a2, b2 = a.to(wide), b.to(wide)
    assert spla.gemm_dd("complex128" if code == 2 else "float64", opA, opB, m, n, k, a2, lda, b2, k,
                        R, m) == 0
    torch.cuda.synchronize()
    na = torch.linalg.vector_norm(a2, dim=1 if opA else 0)
    nb = torch.linalg.vector_norm(b2, dim=1)
    bound = R.abs() * 2.0 ** -23 + nb[:, None] * na[None, :] * (k * 2.0 ** -50)
    assert bool(((C.to(wide) - R).abs() <= bound).all())
