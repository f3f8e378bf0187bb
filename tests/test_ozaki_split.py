"""The split moduli of the Ozaki path's complex products (two real products per
modulus): the CRT side (tests/cpp/test_crt_split.cu) and the slicer's residue
step on the CPU, and the whole path on the GPU at the edges of its tiles."""
import re
import shutil
import subprocess

import numpy as np
import pytest

from test_ozaki_crt import HERE
from test_ozaki_slice_arith import HDR, _centred, _quotient


@pytest.mark.parametrize("source", ["test_crt_split.cu", "test_slice_rows.cu"])
def test_split_arithmetic_on_the_cpu(tmp_path, source):
    """The reconstruction's weights (test_crt_split.cu) and the slicer's digit
    weights and reduction (test_slice_rows.cu), compiled for the host."""
    nvcc = shutil.which("nvcc") or shutil.which("/usr/local/cuda/bin/nvcc")
    if nvcc is None:
        pytest.skip("nvcc not available")
    exe = tmp_path / "check"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-o",
                    str(exe), str(HERE / "cpp" / source)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr


# digit base and largest |d_j| per digit, as in test_ozaki_slice_arith
@pytest.mark.parametrize("count,base,dmax", [
    ("kSplitCount", 1 << 15, [1 << 14, 1 << 14, 1 << 14, 1 << 13]),
    ("kSplitCountFloat", 1 << 13, [(1 << 13) - 1, (1 << 12) + 1, (1 << 12) + 1])])
def test_split_digit_sums_give_byte_residues(count, base, dmax):
    """u = sr + si with the digit sums of both parts: every intermediate is
    exact in FP32, and for every value the sum can take (the rounding is
    symmetric: the positive ones) u - q p is congruent and one signed byte."""
    text = HDR.read_text()
    table = [int(v) for v in re.search(r"kSplitModuli\[kSplitCount\]\s*=\s*\{([^}]*)\}",
                                       text).group(1).split(",")]
    n = int(re.search(r"\b" + count + r"\s*=\s*(\d+)", text).group(1))
    for p in table[:n]:
        j = next(j for j in range(1, p) if (j * j + 1) % p == 0)
        c = [1] + [_centred(pow(base, i, p), p) for i in range(1, len(dmax))]
        cj = [_centred(j * pow(base, i, p) % p, p) for i in range(len(dmax))]
        sr = sum(abs(w) * d for w, d in zip(c, dmax))
        smax = sr + sum(abs(w) * d for w, d in zip(cj, dmax))
        assert smax < (1 << 24) and 2 * sr + smax < (1 << 25)
        for lo in range(0, smax + 1, 1 << 22):
            s = np.arange(lo, min(lo + (1 << 22), smax + 1), dtype=np.int64)
            r = s - _quotient(s, p) * p
            assert np.abs(r).max() <= 127, p


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["complex128", "complex64"])
@pytest.mark.parametrize("opA,opB,m,n,k", [
    (2, 0, 1, 1, 1), (1, 0, 127, 3, 127), (2, 0, 128, 257, 129), (0, 0, 129, 64, 700),
    (2, 2, 257, 33, 260), (0, 1, 16, 300, 128), (2, 0, 144, 20, 125000), (1, 0, 50, 40, 250001)])
def test_split_products_match_double_double(dt, opA, opB, m, n, k):
    """|C - R| <= |a_i| |b_j| (sqrt(2 k) 2^-55 + 2^-51) for double: each real is
    rounded by half a unit at a scaled norm of at least 2^56 (2^-56 sqrt(2 k)
    per operand at most), and the result by 1.5 ulp; float adds its own
    rounding of C and has norms of at least 2^36."""
    import torch
    import spla_b200 as spla
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 * m + n)
    tdt = getattr(torch, dt)
    A = torch.randn((m, k), dtype=tdt, device="cuda", generator=g)  # rows of op(A)
    B = torch.randn((n, k), dtype=tdt, device="cuda", generator=g)  # columns of op(B)
    A[m // 2] *= 1e-3
    a = A.T.contiguous() if opA == 0 else A  # as stored (column-major)
    b = B.T.contiguous() if opB != 0 else B
    lda, ldb = (m if opA == 0 else k), (k if opB == 0 else n)
    C = torch.zeros((n, m), dtype=tdt, device="cuda")
    nbytes = spla.splab_gemm_workspace_size(dt, spla.PATH_OZAKI, opA, opB, m, n, k)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    assert spla.splab_gemm(dt, spla.PATH_OZAKI, opA, opB, m, n, k, 1.0, a, lda, b, ldb, 0.0, C, m,
                           workspace=ws, workspace_bytes=nbytes) == 0
    R = torch.zeros((n, m), dtype=torch.complex128, device="cuda")
    a2, b2 = a.to(torch.complex128), b.to(torch.complex128)
    assert spla.gemm_dd("complex128", opA, opB, m, n, k, a2, lda, b2, ldb, R, m) == 0
    torch.cuda.synchronize()
    na = torch.linalg.vector_norm(A.to(torch.complex128), dim=1)
    nb = torch.linalg.vector_norm(B.to(torch.complex128), dim=1)
    norms = nb[:, None] * na[None, :]
    if dt == "complex128":
        bound = norms * ((2 * k) ** 0.5 * 2.0 ** -55 + 2.0 ** -51)
    else:
        bound = norms * ((2 * k) ** 0.5 * 2.0 ** -35 + 2.0 ** -51) + R.abs() * 2.0 ** -23
    assert bool(((C.to(torch.complex128) - R).abs() <= bound).all())
