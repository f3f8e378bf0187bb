"""Host-resident operands, streamed in k-chunks: the chunk rule on the CPU
(tests/cpp/test_stream_chunks.cpp), and what the chunks may not change in the
result on the GPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_chunk_rule_on_the_cpu(tmp_path):
    exe = tmp_path / "check"
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    subprocess.run([gxx, "-std=c++17", "-O1", "-o", str(exe),
                    str(HERE / "cpp" / "test_stream_chunks.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout


def _cancelling(dt, rows, k, ld, seed):
    """(A, B) as stored for op(A) = A^H, op(B) = B, leading dimension ld: the
    products of the two halves of k cancel but for a small rest."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    A = torch.randn((rows, ld), dtype=getattr(torch, dt), device="cuda", generator=g)
    h = k // 2
    A[:, h:2 * h] = A[:, :h]
    B = A.clone()
    B[:, h:2 * h].neg_()
    return A, B + 1e-3 * torch.randn(B.shape, dtype=A.dtype, device="cuda", generator=g)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["float32", "complex64"])
@pytest.mark.parametrize("path", [0, 1, 2, 3], ids=["auto", "dmma", "ozaki", "tf32x3"])
@pytest.mark.parametrize("m,k,pad", [(128, 40000, 0), (70, 20001, 3)])
def test_float_results_of_host_operands_are_those_of_device_operands(dt, path, m, k, pad):
    """One chunk holds all of k: the same kernels on the same values, so C is
    bit-identical to the call on device operands (rounded to float once)."""
    import torch
    import spla_b200 as spla
    A, B = _cancelling(dt, m, k, k + pad, m)
    op = 2 if A.is_complex() else 1
    ctx = spla.Context(spla.PU_GPU)
    ctx.set_fp64_path(path)
    out = []
    for host in (False, True):
        a, b, C = A, B, torch.zeros((m, m), dtype=A.dtype, device="cuda")
        if host:
            a, b, C = (x.cpu().pin_memory() for x in (a, b, C))
        spla.gemm(op, 0, m, m, k, 1.0, a, k + pad, b, k + pad, 0.0, C, m, ctx)
        torch.cuda.synchronize()
        out.append(C.cpu())
    assert torch.equal(*out)
