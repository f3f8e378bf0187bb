"""Host-resident operands, streamed in k-chunks: the chunk rule on the CPU
(tests/cpp/test_stream_chunks.cpp), and what the chunks may not change in the
result on the GPU."""
import os
import shutil
import subprocess
import sys
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


def _host_and_device_results(dt, path, m, k, pad):
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
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["float32", "complex64"])
@pytest.mark.parametrize("path", [0, 1, 2, 3], ids=["auto", "dmma", "ozaki", "tf32x3"])
@pytest.mark.parametrize("m,k,pad", [(128, 40000, 0), (70, 20001, 3)])
def test_float_results_of_host_operands_are_those_of_device_operands(dt, path, m, k, pad):
    """One chunk holds all of k: the same kernels on the same values, so C is
    bit-identical to the call on device operands (rounded to float once)."""
    import torch
    assert torch.equal(*_host_and_device_results(dt, path, m, k, pad))


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["float64", "complex128"])
@pytest.mark.parametrize("m,k,pad", [(64, 40000, 0), (130, 30001, 3)])
def test_ozaki_results_of_host_operands_are_those_of_device_operands(dt, m, k, pad):
    """The same for the Ozaki path with the double types (rounded at C's last
    bit once, not once per chunk)."""
    import torch
    assert torch.equal(*_host_and_device_results(dt, 2, m, k, pad))


@pytest.mark.gpu
@pytest.mark.parametrize("dt,m,n,k", [("complex128", 320, 320, 40960), ("complex128", 400, 300, 40000),
                                      ("float64", 700, 700, 22000)])
def test_host_operands_take_the_path_of_device_operands(dt, m, n, k):
    """AUTO resolves on all of k, not on the chunks it is cut into: the Ozaki path's
    slicing events (17) are recorded after a marker set before the call."""
    import ctypes as ct
    import torch
    import spla_b200 as spla
    code = {"float64": 1, "complex128": 3}[dt]
    op = 2 if dt == "complex128" else 1
    L = spla.lib()
    assert L.splab_gemm_path(code, spla.PATH_AUTO, op, 0, m, n, k) == spla.PATH_OZAKI
    A = torch.randn((m, k), dtype=getattr(torch, dt)).pin_memory()
    B = torch.randn((n, k), dtype=A.dtype).pin_memory()
    C = torch.zeros((n, m), dtype=A.dtype).pin_memory()
    nphase = 20
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2 * nphase + 1)]
    for e in ev:
        e.record()
    torch.cuda.synchronize()
    ctx = spla.Context(spla.PU_GPU)
    L.splab_set_phase_events((ct.c_void_p * (2 * nphase))(*[e.cuda_event for e in ev[:-1]]), nphase)
    try:
        spla.gemm(op, 0, m, n, k, 1.0, A, k, B, k, 0.0, C, m, ctx)
    finally:
        L.splab_set_phase_events(None, 0)
    assert ev[-1].elapsed_time(ev[35]) > 0.0


@pytest.mark.gpu
def test_a_wait_that_gives_up_in_an_early_chunk_is_reported():
    """The test hook lets the bounded waits of the first of eight chunks run out
    (50 ms; no copies are issued): the call reports it although the later chunks,
    whose contractions clear the status word, succeed."""
    code = r"""
import sys, torch
sys.path.insert(0, %r)
import spla_b200 as spla
m, n, k = 64, 64, 2000
A = torch.randn(m * k, dtype=torch.complex128).pin_memory()
B = torch.randn(n * k, dtype=torch.complex128).pin_memory()
C = torch.zeros(m * n, dtype=torch.complex128, device='cuda')
ctx = spla.Context(spla.PU_GPU)
ctx.set_fp64_path(spla.PATH_OZAKI)
ctx.set_tile_size_gpu(64)  # chunks of 256
try:
    spla.gemm(2, 0, m, n, k, 1.0, A, k, B, k, 0.0, C, m, ctx)
    print('NO_ERROR')
except spla.GPULaunchError:
    print('TIMEOUT_REPORTED')
spla.gemm(2, 0, m, n, k, 1.0, A, k, B, k, 1.0, C, m, ctx)  # no stall with beta = 1
print('CONTEXT_OK')
""" % str(HERE.parent)
    env = dict(os.environ, SPLAB_OZAKI_STALL_TEST="2")
    out = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True,
                         timeout=300)
    assert "TIMEOUT_REPORTED" in out.stdout and "CONTEXT_OK" in out.stdout, out.stdout + out.stderr
