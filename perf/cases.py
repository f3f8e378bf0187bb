"""Performance cases of the local contraction path, through the public Python
interface (spla_b200, spla_b200.autograd).

A case is a dict of plain values:

  kind   "gemm" | "ssb" | "ssbtr" | "sbs" | "batch" | "adjoint"
  dtype  float32 | float64 | complex64 | complex128
  m, n, k                   as in the entry point (sbs: m is mLocal)
  opA, opB                  gemm only: 0 = N, 1 = T, 2 = C
  beta                      0 or 1
  pad                       extra elements in every leading dimension
  host                      operands in pinned host memory
  count, path               batch only: instances, contraction path

All operands are seeded: Gaussian entries scaled by 1/sqrt(k) (near-unit-norm
columns of wavefunctions), uniform ones for the real-double stripe, a random
unitary as the rotation of sbs. Matrices are column-major; a column-major
rows x cols matrix with leading dimension ld is held as a (cols, ld) tensor.
"""
import math

import torch

import spla_b200 as spla
from spla_b200.autograd import ssb_autograd

_COMPLEX = ("complex64", "complex128")


def _case(name, kind, dtype, m, n, k, **more):
    c = {"name": name, "kind": kind, "dtype": dtype, "m": m, "n": n, "k": k, "opA": 0, "opB": 0,
         "beta": 0, "pad": 0, "host": False, "count": 0, "path": 0}
    c.update(more)
    return c


def listed():
    return [
        # subspace-sized Hermitian product of a few bands: latency of one call
        _case("zgemm_small", "gemm", "complex128", 64, 64, 64, opA=2),
        # an ordinary local product with ragged sizes and a transposed operand
        _case("dgemm_ragged_nt", "gemm", "float64", 1501, 2003, 1207, opB=1, pad=3),
        # real-double overlap of a small system (m = n = 256, k = 20000)
        _case("dssb_256", "ssb", "float64", 256, 256, 20000),
        # wavefunction overlap, the headline workload (m = n = 1024, k = 250000)
        _case("zssb_1024", "ssb", "complex128", 1024, 1024, 250000),
        # overlap of an odd number of bands on a ragged plane-wave count,
        # accumulated into C
        _case("zssb_ragged", "ssb", "complex128", 387, 515, 60013, beta=1, pad=3),
        # subspace rotation of 2048 bands (n = k = 2048), accumulated into C
        _case("zsbs_2048", "sbs", "complex128", 200000, 2048, 2048, beta=1),
        # lower triangle of a real-float Gram-like product (long k)
        _case("ssbtr_float", "ssbtr", "float32", 1536, 1536, 400000),
        # single-precision overlap of a small system
        _case("cssb_256", "ssb", "complex64", 256, 256, 16384),
        # single-precision overlap, large and ragged
        _case("cssb_ragged", "ssb", "complex64", 771, 1003, 130001, pad=1),
        # k-points of one self-consistency step: instances of uneven k, m = n
        _case("zbatch_kpoints", "batch", "complex128", 512, 1024, 30000, count=8, path=2),
        # differentiable overlap: forward and backward of ||A^H B - I||^2
        _case("zadjoint_512", "adjoint", "complex128", 512, 512, 100000),
        # overlap with the wavefunctions in pinned host memory
        _case("zssb_host", "ssb", "complex128", 256, 256, 50000, host=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "ssb", "ssb", "ssb", "ssbtr", "sbs", "batch", "adjoint"])
    dtype = rng.choice(["complex128", "complex128", "float64", "complex64", "float32"])
    more = {"beta": rng.choice([0, 0, 1]), "pad": rng.choice([0, 0, 1, 3])}
    if kind == "gemm":
        m, n, k = (_log(rng, 32, 3000) for _ in range(3))
        more.update(opA=rng.randrange(3), opB=rng.randrange(3))
    elif kind in ("ssb", "ssbtr"):
        m, n, k = _log(rng, 32, 1024), _log(rng, 32, 1024), _log(rng, 1000, 250000)
        if kind == "ssbtr":
            n = m
        elif rng.random() < 0.15:
            m, n, k, more["host"] = min(m, 400), min(n, 400), min(k, 60000), True
    elif kind == "sbs":
        m, n = _log(rng, 1000, 100000), _log(rng, 32, 2048)
        k = n
    elif kind == "batch":
        dtype = rng.choice(["complex128", "complex64"])
        path = rng.choice([1, 2] if dtype == "complex128" else [1, 2, 3])
        hi = _log(rng, 64, 1024)
        m, n, k = max(32, hi // 2), hi, _log(rng, 4000, 40000)
        more = {"count": rng.randrange(4, 13), "path": path}
    else:
        dtype = rng.choice(["complex128", "complex128", "float64"])
        m, n, k, more = _log(rng, 32, 512), _log(rng, 32, 512), _log(rng, 2000, 100000), {}
    c = _case("", kind, dtype, m, n, k, **more)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs

_KEPT = {}


def _context():
    """The Context and C distribution a program creates once and keeps."""
    if not _KEPT:
        _KEPT["ctx"] = spla.Context(spla.PU_GPU)
        _KEPT["dist"] = spla.MatrixDistribution.create_blacs_block_cyclic(
            spla.MPI_COMM_SELF, "R", 1, 1, 128, 128)
    return _KEPT["ctx"], _KEPT["dist"]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _matrix(g, case, rows, cols, pad, scale):
    """A column-major rows x cols matrix as a (cols, rows + pad) tensor."""
    dt = getattr(torch, case["dtype"])
    shape = (cols, rows + pad)
    if case["kind"] == "ssb" and case["dtype"] == "float64":
        return torch.rand(shape, dtype=dt, device="cuda", generator=g) * 2 - 1
    return torch.randn(shape, dtype=dt, device="cuda", generator=g).mul_(scale)


def _unitary(g, case, rows, cols, pad):
    """A column-major rows x cols matrix with orthonormal columns."""
    dt = torch.complex128 if case["dtype"] in _COMPLEX else torch.float64
    q = torch.linalg.qr(torch.randn((rows, cols), dtype=dt, device="cuda", generator=g)).Q
    out = torch.zeros((cols, rows + pad), dtype=getattr(torch, case["dtype"]), device="cuda")
    out[:, :rows] = q.T
    return out


def _batch_shapes(case):
    """(m, n, k) of every instance: m = n between the case's m and n, k
    between 1 and 1.5 times the case's k."""
    sizes = sorted({case["m"], (case["m"] + case["n"]) // 2, case["n"]})
    return [(sizes[i % len(sizes)],) * 2 + (case["k"] + (case["k"] * (37 * i % 100)) // 200,)
            for i in range(case["count"])]


def _op(case):
    """op(A) of the stripe products: conjugate transpose (complex) / transpose."""
    return spla.OP_CONJ_TRANSPOSE if case["dtype"] in _COMPLEX else spla.OP_TRANSPOSE


def _operands(case, seed):
    """A, B, C (column-major) with their leading dimensions."""
    g = _generator(seed)
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    scale = k ** -0.5
    a_n = case["kind"] == "sbs" or (case["kind"] == "gemm" and case["opA"] == 0)
    b_n = case["kind"] != "gemm" or case["opB"] == 0
    A = _matrix(g, case, *((m, k) if a_n else (k, m)), pad, scale)
    if case["kind"] == "sbs":
        B = _unitary(g, case, k, n, pad)
    else:
        B = _matrix(g, case, *((k, n) if b_n else (n, k)), pad, scale)
    if case["beta"]:
        C = _matrix(g, case, m, n, pad, scale)
    else:
        C = torch.zeros((n, m + pad), dtype=A.dtype, device="cuda")
    return A, B, C


def prepare(case, seed):
    ctx, dist = _context()
    s = {"case": case, "ctx": ctx, "dist": dist}
    if case["kind"] == "batch":
        g = _generator(seed)
        problems, keep = [], []
        for m, n, k in _batch_shapes(case):
            A = _matrix(g, case, k, m, 0, k ** -0.5)
            B = _matrix(g, case, k, n, 0, k ** -0.5)
            C = torch.zeros((n, m), dtype=A.dtype, device="cuda")
            keep.append((A, B, C))
            problems.append(dict(opA=_op(case), opB=0, m=m, n=n, k=k, A=A, lda=k, B=B, ldb=k, C=C,
                                 ldc=m, alpha=1.0, beta=0.0))
        s["batch"] = spla.Batch(case["dtype"], problems, path=case["path"])
        s["ws"] = torch.empty(s["batch"].workspace_bytes, dtype=torch.uint8, device="cuda")
        s["keep"] = keep
        return s
    if case["kind"] == "adjoint":
        g = _generator(seed)
        s["A"] = _matrix(g, case, case["k"], case["m"], 0, case["k"] ** -0.5).requires_grad_(True)
        s["B"] = _matrix(g, case, case["k"], case["n"], 0, case["k"] ** -0.5).requires_grad_(True)
        s["eye"] = torch.eye(case["m"], case["n"], dtype=s["A"].dtype, device="cuda")
        return s
    s["A"], s["B"], s["C"] = _operands(case, seed)
    if case["host"]:
        for x in "ABC":
            s[x] = s[x].cpu().pin_memory()
    return s


def _loss(C, eye):
    return (C - eye).abs().square().sum()


def run(s):
    c, ctx, dist = s["case"], s["ctx"], s["dist"]
    kind, m, n, k = c["kind"], c["m"], c["n"], c["k"]
    if kind == "batch":
        s["batch"].run(s["ws"])
        return [C for _, _, C in s["keep"]]
    if kind == "adjoint":
        C = ssb_autograd(s["A"], s["B"], ctx)
        dA, dB = torch.autograd.grad(_loss(C, s["eye"]), (s["A"], s["B"]))
        return {"C": C.detach(), "dA": dA, "dB": dB}
    A, B, C = s["A"], s["B"], s["C"]
    lda, ldb, ldc = A.shape[1], B.shape[1], C.shape[1]
    if kind == "gemm":
        spla.gemm(c["opA"], c["opB"], m, n, k, 1.0, A, lda, B, ldb, c["beta"], C, ldc, ctx)
    elif kind == "ssb":
        spla.pgemm_ssb(m, n, k, _op(c), 1.0, A, lda, B, ldb, c["beta"], C, ldc, 0, 0, dist, ctx)
    elif kind == "sbs":
        spla.pgemm_sbs(m, n, k, 1.0, A, lda, B, ldb, 0, 0, dist, c["beta"], C, ldc, ctx)
    else:
        spla.pgemm_ssbtr(m, n, k, _op(c), 1.0, A, lda, B, ldb, c["beta"], C, ldc, 0, 0,
                         spla.FILL_MODE_LOWER, dist, ctx)
        # elements above the diagonal may be computed or left alone; the (n, m)
        # view of the column-major C has its lower triangle above its diagonal
        return C[:, :m].triu()
    return C


# ---------------------------------------------------------------------------
# what a pass cannot do without, and the result in 64 bits

_BYTES = {"float32": 4, "float64": 8, "complex64": 8, "complex128": 16}


def work(case):
    es, per = _BYTES[case["dtype"]], 8 if case["dtype"] in _COMPLEX else 2
    if case["kind"] == "batch":
        shapes = _batch_shapes(case)
        return {"bytes": sum(es * (k * (m + n) + m * n) for m, n, k in shapes),
                "flops": sum(per * m * n * k for m, n, k in shapes)}
    m, n, k = case["m"], case["n"], case["k"]
    if case["kind"] == "adjoint":  # A and B read, C, dA and dB written
        return {"bytes": es * (2 * k * (m + n) + m * n), "flops": 3 * per * m * n * k}
    share = 0.5 if case["kind"] == "ssbtr" else 1.0
    return {"bytes": es * (k * (m + n) + share * m * n * (1 + case["beta"])),
            "flops": share * per * m * n * k}


def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _product(A, B):
    """A (m x k) times B (k x n) in 64 bits, summed over pieces of k."""
    C = torch.zeros((A.shape[0], B.shape[1]), dtype=_wide(A[:1, :1]).dtype, device=A.device)
    step = 4096
    for k0 in range(0, A.shape[1], step):
        C += _wide(A[:, k0:k0 + step]) @ _wide(B[k0:k0 + step])
    return C


def _apply(op, x):
    return x if op == 0 else x.T if op == 1 else x.mH


def exact(case, seed):
    if case["kind"] == "batch":
        g = _generator(seed)
        out = []
        for m, n, k in _batch_shapes(case):
            A = _matrix(g, case, k, m, 0, k ** -0.5)
            B = _matrix(g, case, k, n, 0, k ** -0.5)
            out.append(_product(A.conj(), B.T).T.contiguous())
        return out
    if case["kind"] == "adjoint":
        g = _generator(seed)
        A = _matrix(g, case, case["k"], case["m"], 0, case["k"] ** -0.5)
        B = _matrix(g, case, case["k"], case["n"], 0, case["k"] ** -0.5)
        C = _product(A.conj(), B.T)
        G = 2 * (C - torch.eye(case["m"], case["n"], dtype=C.dtype, device="cuda"))
        return {"C": C, "dA": G.conj() @ B, "dB": G.T @ A}
    m, n, k, pad = case["m"], case["n"], case["k"], case["pad"]
    A, B, C = _operands(case, seed)
    kind = case["kind"]
    op_a = case["opA"] if kind == "gemm" else 0 if kind == "sbs" else _op(case)
    op_b = case["opB"] if kind == "gemm" else 0
    a = A[:, :A.shape[1] - pad].T
    b = B[:, :B.shape[1] - pad].T
    P = _product(_apply(op_a, a), _apply(op_b, b)).T
    R = _wide(C)
    R[:, :m] = P + case["beta"] * R[:, :m] if case["beta"] else P
    if kind == "ssbtr":
        return R[:, :m].triu()
    return R
