"""One-pass row scaling of the Ozaki path: which rows take their exponent from the
sample, which take their exact norm, and which are sliced a second time."""
import os

import pytest

pytestmark = pytest.mark.gpu


def _run(dt, A, B, onepass):
    """(C, rows listed for a second slicing, rows with an exact norm) of op(A) B,
    op(A) = A^H or A^T; A, B: rows of op(A) and columns of B. The lists, exact
    flags and the two counts are the last 2 R + 2 ints of the workspace."""
    import torch
    import spla_b200 as spla
    (m, k), n = A.shape, B.shape[0]
    op = 2 if A.is_complex() else 1
    nbytes = spla.splab_gemm_workspace_size(dt, spla.PATH_OZAKI, op, 0, m, n, k)
    ws = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    C = torch.zeros((n, m), dtype=A.dtype, device="cuda")
    os.environ["SPLAB_OZAKI_ONEPASS"] = "1" if onepass else "0"
    try:
        assert spla.splab_gemm(dt, spla.PATH_OZAKI, op, 0, m, n, k, 1.0, A, k, B, k, 0.0, C, m,
                               workspace=ws, workspace_bytes=nbytes) == 0
        torch.cuda.synchronize()
    finally:
        os.environ.pop("SPLAB_OZAKI_ONEPASS", None)
    rows = m + n
    size = 4 * (2 * rows + 2)
    off = nbytes - (size + 255) // 256 * 256
    ints = ws[off:off + size].view(torch.int32)
    return C, int(ints[2 * rows:].sum()), int(ints[rows:2 * rows].sum())


def _rows(dt, rows, k, profile, seed):
    """Rows with the profile's weight along k and norms spread over an octave."""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    X = torch.randn((rows, k), dtype=getattr(torch, dt), device="cuda", generator=g)
    x = torch.arange(k, device="cuda", dtype=torch.float64) / k
    w = {"even": torch.ones_like(x), "falling": torch.exp(-8 * x), "start": torch.exp(-400 * x),
         "middle": torch.exp(-((x - 0.53) / 0.005) ** 2 / 2),
         "few": (torch.rand(k, device="cuda", dtype=torch.float64, generator=g) < 30 / k).double()}
    X *= w[profile].to(X.real.dtype)
    X /= torch.linalg.vector_norm(X, dim=1, keepdim=True)
    return X * 2 ** torch.rand((rows, 1), device="cuda", dtype=X.real.dtype, generator=g)


@pytest.mark.parametrize("dt,m,n,k", [("complex128", 64, 40, 70000), ("float64", 64, 40, 140000),
                                      ("float32", 64, 40, 140000), ("complex64", 33, 70, 66000),
                                      ("complex128", 900, 820, 10016)])
@pytest.mark.parametrize("profile", ["even", "falling", "start", "middle", "few"])
def test_rows_of_uneven_weight_are_sliced_once(dt, m, n, k, profile):
    """A sample of 16 runs whose sums differ widely does not decide a row: it takes
    its exact norm at once, where an estimate would fail the check and cost a third
    read and a second slicing. Rows of even weight keep their estimates: their
    estimate's standard error is 0.8 % of the norm at 140000 reals and 2.3 % at
    20032, against a distance of 3.1 % and two standard errors (2 in 1000 rows at
    most beyond it; a fifth of the octave within it). C is that of the two-pass order
    in any case."""
    import torch
    A, B = _rows(dt, m, k, profile, 1), _rows(dt, n, k, profile, 2)
    C, again, exact = _run(dt, A, B, True)
    assert torch.equal(C, _run(dt, A, B, False)[0])
    if profile == "even":
        assert again <= 0.02 * (m + n) and exact <= 0.3 * (m + n)
    else:
        assert again == 0 and exact == m + n


def _threshold(dt):
    """thr of a type's default moduli, as ozaki_crt.cuh makes it: the exponents change at
    row norms thr 2^e."""
    import math
    import re
    from pathlib import Path
    text = (Path(__file__).resolve().parent.parent / "spla_b200" / "csrc" / "kernels" /
            "ozaki_crt.cuh").read_text()
    cplx = dt.startswith("complex")
    name, count = ("kSplitModuli", {"complex128": 16, "complex64": 10}) if cplx else \
                  ("kModuli", {"float64": 15, "float32": 9})
    table = [int(v) for v in re.search(name + r"\[\w+\]\s*=\s*\{([^}]*)\}",
                                       text).group(1).split(",")]
    half = (math.log2(math.prod(table[:count[dt]])) - 2.0) / 2.0
    f = 2.0 ** (half - math.floor(half)) / 2.0 * (1.0 - 1.0 / 64)
    return 0.75 if dt == "complex64" else 0.5 if f < 0.6 else f


@pytest.mark.parametrize("dt", ["complex128", "float64", "complex64", "float32"])
def test_norms_where_the_exponents_change(dt):
    """Rows of even weight at, next to and off the norms thr 2^e (an estimate counts
    from 3.1 % off: exact norms within 2 %, none beyond 6 %), and rows whose sample
    gives 0.8 or 1.25 of a norm next to such a step, which only the check of the sums
    of squares can send back, at either end of its range. All end with the two-pass
    exponents: C is bit-identical."""
    import torch
    thr = _threshold(dt)
    cplx = dt.startswith("complex")
    k = 70000 if cplx else 140000
    K2 = 140000
    steps = torch.tensor([0.0] + [s * d for d in (1e-12, 1e-9, 3e-7, 1e-6, 1e-5, 1e-3)
                                  for s in (1, -1)], dtype=torch.float64, device="cuda")
    near = torch.cat([steps, torch.tensor([0.02, -0.02], device="cuda", dtype=torch.float64)])
    off = torch.tensor([0.06, 0.2, 0.5, 0.85, -0.06, -0.2, -0.4, -0.47], device="cuda",
                       dtype=torch.float64)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    # the sample: 16 runs of `run` reals, `gap` apart
    run, gap = (K2 // 256 + 7) // 8 * 8, K2 // 16
    sampled = torch.zeros(K2, dtype=torch.bool, device="cuda")
    for c in range(16):
        sampled[c * gap:c * gap + run] = True
    even = torch.randn((len(near) + len(off), K2), dtype=torch.float64, device="cuda", generator=g)
    even *= (thr * (1.0 + torch.cat([near, off])) /
             torch.linalg.vector_norm(even, dim=1))[:, None]
    parts = [even]
    for est in (0.8, 1.25):
        X = torch.randn((len(steps), K2), dtype=torch.float64, device="cuda", generator=g)
        ins = torch.where(sampled, X, torch.zeros_like(X))
        rest = X - ins
        share = est * est * 16.0 * run / K2  # of the sum of squares, in the sample
        ins *= (share ** 0.5 / torch.linalg.vector_norm(ins, dim=1))[:, None]
        rest *= ((1.0 - share) ** 0.5 / torch.linalg.vector_norm(rest, dim=1))[:, None]
        parts.append((ins + rest) * (thr * (1.0 + steps))[:, None])
    rows = torch.cat(parts)
    rows[::2] *= 2.0 ** 20  # other octaves
    rows = rows.to(torch.float64 if dt in ("complex128", "float64") else torch.float32)
    A = torch.view_as_complex(rows.view(len(rows), k, 2).contiguous()) if cplx else rows
    B = A.flip(0).contiguous()
    C, again, exact = _run(dt, A, B, True)
    assert torch.equal(C, _run(dt, A, B, False)[0])
    # A's and B's rows: exact norms for those within 2 % of a step, an estimate for the
    # others; sent back: at least the rows on the wrong side (six steps of either sign)
    assert exact == 2 * len(near)
    assert 2 * 12 <= again <= 2 * 2 * len(steps)
