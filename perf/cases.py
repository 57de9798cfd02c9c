"""Workloads this library is timed on, through its public Python entry points.

listed() names the workloads, draw(rng) gives another one of the same ranges,
prepare() makes what a program holds before the call, run() is one call,
work() the bytes and operations it cannot do without, and exact() the result in
64-bit torch arithmetic.  All matrices are column-major: a tensor of shape
(columns, leading dimension).
"""
import math

import numpy as np
import torch

from zynum_b200 import autograd, blas

DTYPES = {"f64": torch.float64, "f32": torch.float32, "z": torch.complex128, "c": torch.complex64}
BYTES = {"f64": 8, "f32": 4, "z": 16, "c": 8}


def listed():
    return [
        # A small product inside a larger program: latency and launches count.
        dict(name="dgemm_256", kind="gemm", dtype="f64", ta="N", tb="N", m=256, n=256, k=256, pad=0,
             alpha=1.0, beta=0.0),
        # The reference's plain DGEMM: padded, odd leading dimensions, alpha and beta both in use.
        dict(name="dgemm_1024_padded", kind="gemm", dtype="f64", ta="T", tb="N", m=1024, n=1024, k=1024, pad=7,
             alpha=1.5, beta=0.5),
        # A large FP64 product, accumulated into C.
        dict(name="dgemm_4096", kind="gemm", dtype="f64", ta="N", tb="T", m=4096, n=4096, k=4096, pad=0,
             alpha=1.0, beta=1.0),
        # The headline: FP64 product emulated on the INT8 tensor cores.
        dict(name="dgemm_emulated_8192", kind="emulated", dtype="f64", ta="N", tb="N", m=8192, n=8192, k=8192, pad=0,
             alpha=1.0, beta=0.0, phi=0.0),
        # Tall-skinny product (a block of vectors against a small matrix): memory-bound.
        dict(name="dgemm_tall", kind="gemm", dtype="f64", ta="N", tb="N", m=131072, n=64, k=64, pad=0,
             alpha=1.0, beta=1.0),
        # A large FP32 product.
        dict(name="sgemm_4096", kind="gemm", dtype="f32", ta="N", tb="N", m=4096, n=4096, k=4096, pad=0,
             alpha=1.0, beta=0.0),
        # An ordinary complex product.
        dict(name="zgemm_2048", kind="gemm", dtype="z", ta="N", tb="C", m=2048, n=2048, k=2048, pad=0,
             alpha=1.0, beta=0.0),
        # A triangular solve with several hundred right-hand sides.
        dict(name="dtrsm_4096x512", kind="trsm", side="L", uplo="L", ta="N", diag="N", n=4096, nrhs=512, pad=0),
        # Forward and backward of solve -> rank-k update -> scalar loss.
        dict(name="chain_4096x512", kind="chain", n=4096, nrhs=512),
        # Many independent products of varied sizes in one call.
        dict(name="dgemm_batch_20000", kind="gemm_batch", dtype="f64", ta="N", tb="N", count=20000, layout=1),
        # Many independent triangular solves of varied sizes in one call.
        dict(name="dtrsm_batch_5000", kind="trsm_batch", dtype="f64", count=5000, layout=2),
        # The drop-in Fortran call on host arrays (pageable memory, as an unchanged caller has it).
        dict(name="dgemm_host_2048", kind="host", dtype="f64", ta="N", tb="N", m=2048, n=2048, k=2048,
             alpha=1.0, beta=0.0),
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of lo .. hi."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "tall", "emulated", "complex", "trsm", "chain", "gemm_batch",
                       "trsm_batch", "host"])
    trans = rng.choice("NT"), rng.choice("NT")
    beta = rng.choice([0.0, 1.0, 0.5])
    if kind == "gemm":
        return dict(kind="gemm", dtype=rng.choice(["f64", "f32"]), ta=trans[0], tb=trans[1],
                    m=_log_int(rng, 64, 4096), n=_log_int(rng, 64, 4096), k=_log_int(rng, 64, 4096),
                    pad=rng.choice([0, 0, 1, 7, 8]), alpha=1.5, beta=beta)
    if kind == "tall":
        return dict(kind="gemm", dtype=rng.choice(["f64", "f32"]), ta="N", tb=trans[1],
                    m=_log_int(rng, 8192, 131072), n=rng.randint(17, 64), k=rng.randint(17, 64),
                    pad=rng.choice([0, 0, 2]), alpha=1.0, beta=beta)
    if kind == "emulated":
        return dict(kind="emulated", dtype="f64", ta=trans[0], tb=trans[1], m=_log_int(rng, 1024, 6144),
                    n=_log_int(rng, 1024, 6144), k=_log_int(rng, 1024, 6144), pad=rng.choice([0, 1, 8]), alpha=1.0,
                    beta=beta, phi=rng.choice([0.0, 4.0, 8.0]))
    if kind == "complex":
        return dict(kind="gemm", dtype=rng.choice(["z", "c"]), ta=rng.choice("NTC"), tb=rng.choice("NTC"),
                    m=_log_int(rng, 128, 2048), n=_log_int(rng, 128, 2048), k=_log_int(rng, 128, 2048),
                    pad=rng.choice([0, 1]), alpha=1.0, beta=beta)
    if kind == "trsm":
        return dict(kind="trsm", side=rng.choice("LR"), uplo=rng.choice("LU"), ta=trans[0], diag=rng.choice("NNU"),
                    n=_log_int(rng, 256, 4096), nrhs=_log_int(rng, 16, 512), pad=rng.choice([0, 0, 1]))
    if kind == "chain":
        return dict(kind="chain", n=_log_int(rng, 512, 4096), nrhs=_log_int(rng, 64, 512))
    if kind == "gemm_batch":
        return dict(kind="gemm_batch", dtype=rng.choice(["f64", "f32"]), ta=trans[0], tb=trans[1],
                    count=_log_int(rng, 500, 16000), layout=rng.randint(3, 1 << 20))
    if kind == "trsm_batch":
        return dict(kind="trsm_batch", dtype=rng.choice(["f64", "f32"]), count=_log_int(rng, 500, 5000),
                    layout=rng.randint(3, 1 << 20))
    return dict(kind="host", dtype=rng.choice(["f64", "f32"]), ta=trans[0], tb=trans[1], m=_log_int(rng, 128, 2048),
                n=_log_int(rng, 128, 2048), k=_log_int(rng, 128, 2048), alpha=1.0, beta=beta)


# ------------------------------------------------------------------ inputs
class _Random:
    """Seeded inputs on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def uniform(self, shape, dtype):
        """Entries (real and imaginary parts) uniform in [-1, 1]."""
        if dtype.is_complex:
            real = torch.float64 if dtype == torch.complex128 else torch.float32
            return torch.view_as_complex(self.uniform(tuple(shape) + (2,), real))
        return torch.rand(shape, generator=self.g, dtype=dtype, device="cuda").mul_(2).sub_(1)

    def normal(self, shape, dtype):
        return torch.randn(shape, generator=self.g, dtype=dtype, device="cuda")


def _log_sizes(rs, lo, hi, count):
    return np.exp(rs.uniform(math.log(lo), math.log(hi + 1), count)).astype(np.int64).clip(lo, hi)


def _batch_sizes(case):
    """Problem sizes of a batch: m, n, k in [8, 512], or n in [16, 1024] with 1 .. 64 right-hand sides."""
    rs = np.random.RandomState(case["layout"])
    if case["kind"] == "gemm_batch":
        return [_log_sizes(rs, 8, 512, case["count"]) for _ in range(3)]
    return [_log_sizes(rs, 16, 1024, case["count"]), _log_sizes(rs, 1, 64, case["count"])]


def _offsets(elements):
    return np.concatenate([[0], np.cumsum(elements)]).astype(np.int64)


def _stored(case):
    """Stored rows and columns of A and B."""
    m, n, k = case["m"], case["n"], case["k"]
    return ((m, k) if case["ta"] == "N" else (k, m)), ((k, n) if case["tb"] == "N" else (n, k))


def _triangular(r, n, ld, uplo, dtype=torch.float64):
    """A well-conditioned triangle: N(0, 1/n) off the diagonal, 1 + |N(0, 1)| on it; zeros elsewhere."""
    a = r.normal((n, ld), dtype).mul_(1.0 / math.sqrt(n))
    a[:, :n] = torch.triu(a[:, :n]) if uplo == "L" else torch.tril(a[:, :n])  # row j of the tensor is column j
    a[:, :n].diagonal().copy_(1.0 + r.normal((n,), dtype).abs())
    return a


def prepare(case, seed):
    r, kind = _Random(seed), case["kind"]
    s = {"case": case}
    if kind in ("gemm", "emulated"):
        dt, pad = DTYPES[case["dtype"]], case["pad"]
        (ra, ca), (rb, cb) = _stored(case)
        s["a"], s["b"] = r.uniform((ca, ra + pad), dt), r.uniform((cb, rb + pad), dt)
        if case.get("phi"):  # entries u 10^e, e uniform in [-phi, phi]
            for x in (s["a"], s["b"]):
                x.mul_(torch.pow(10.0, r.uniform(x.shape, dt).mul_(case["phi"])))
        s["c"] = r.uniform((case["n"], case["m"] + pad), dt)
    elif kind == "trsm":
        n, nr, pad = case["n"], case["nrhs"], case["pad"]
        s["a"] = _triangular(r, n, n + pad, case["uplo"])
        if case["diag"] == "U":
            s["a"][:, :n].mul_(0.5)
        rows, cols = (n, nr) if case["side"] == "L" else (nr, n)
        s["b"] = r.normal((cols, rows + pad), torch.float64)
        s["x"] = torch.empty_like(s["b"])
    elif kind == "chain":
        n = case["n"]
        s["l"] = _triangular(r, n, n, "L").t().contiguous().requires_grad_()  # row-major lower triangle
        s["b"] = r.normal((n, case["nrhs"]), torch.float64).requires_grad_()
    elif kind == "gemm_batch":
        dt, w = DTYPES[case["dtype"]], BYTES[case["dtype"]]
        m, n, k = _batch_sizes(case)
        s["plan"] = blas.GemmBatch(m, n, k, dtype=case["dtype"], transa=case["ta"], transb=case["tb"])
        s["a_at"], s["b_at"], s["c_at"] = _offsets(m * k), _offsets(k * n), _offsets(m * n)
        for x in "abc":
            at = s[x + "_at"]
            s[x] = r.uniform((int(at[-1]),), dt)
            s[x + "_ptr"] = torch.from_numpy(s[x].data_ptr() + w * at[:-1]).cuda()
        for x, ld in (("lda", m if case["ta"] == "N" else k), ("ldb", k if case["tb"] == "N" else n), ("ldc", m)):
            s[x] = torch.from_numpy(ld.astype(np.int32)).cuda()
    elif kind == "trsm_batch":
        dt, w = DTYPES[case["dtype"]], BYTES[case["dtype"]]
        n, nr = _batch_sizes(case)
        s["plan"] = blas.TrsmBatch(n, nr, dtype=case["dtype"])
        a_at, b_at = _offsets(n * n), _offsets(n * nr)
        # off-diagonal entries N(0, 1), diagonals 2 + |N(0, 1)|, scaled by the order to keep X of ordinary size
        s["a"] = r.normal((int(a_at[-1]),), dt)
        order = torch.repeat_interleave(torch.from_numpy(n).cuda(), torch.from_numpy(n * n).cuda())
        s["a"].mul_(torch.rsqrt(order.to(dt)))
        del order
        diag = torch.from_numpy(np.concatenate([o + np.arange(q) * (q + 1) for o, q in zip(a_at[:-1], n)])).cuda()
        s["a"][diag] = 2.0 + r.normal((diag.numel(),), dt).abs()
        s["b"] = r.normal((int(b_at[-1]),), dt)
        s["x"] = torch.empty_like(s["b"])
        s["a_ptr"] = torch.from_numpy(s["a"].data_ptr() + w * a_at[:-1]).cuda()
        s["x_ptr"] = torch.from_numpy(s["x"].data_ptr() + w * b_at[:-1]).cuda()
        s["lda"] = s["ldb"] = torch.from_numpy(n.astype(np.int32)).cuda()
        s["a_at"], s["b_at"] = a_at, b_at
    else:  # host arrays
        dt = DTYPES[case["dtype"]]
        (ra, ca), (rb, cb) = _stored(case)
        shapes = {"a": (ca, ra), "b": (cb, rb), "c": (case["n"], case["m"])}
        for x, shape in shapes.items():
            s[x] = np.array(r.uniform(shape, dt).cpu().numpy()).T  # column-major, this array's own memory
    return s


# -------------------------------------------------------------------- calls
_GEMM = {"f64": blas.dgemm_device, "f32": blas.sgemm_device, "z": blas.zgemm_device, "c": blas.cgemm_device}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "gemm":
        return _GEMM[case["dtype"]](case["ta"], case["tb"], case["m"], case["n"], case["k"], case["alpha"], s["a"],
                                    s["a"].shape[1], s["b"], s["b"].shape[1], case["beta"], s["c"], s["c"].shape[1])
    if kind == "emulated":
        blas.set_dgemm_method(1)
        try:
            return blas.dgemm_device(case["ta"], case["tb"], case["m"], case["n"], case["k"], case["alpha"], s["a"],
                                     s["a"].shape[1], s["b"], s["b"].shape[1], case["beta"], s["c"], s["c"].shape[1])
        finally:
            blas.set_dgemm_method(0)
    if kind == "trsm":
        s["x"].copy_(s["b"])  # the solve works in place
        rows, cols = (case["n"], case["nrhs"]) if case["side"] == "L" else (case["nrhs"], case["n"])
        return blas.dtrsm_device(case["side"], case["uplo"], case["ta"], case["diag"], rows, cols, 1.0, s["a"],
                                 s["a"].shape[1], s["x"], s["x"].shape[1])
    if kind == "chain":
        loss = autograd.chain_loss(s["l"], s["b"])
        dl, db = torch.autograd.grad(loss, (s["l"], s["b"]))
        return {"loss": loss, "dl": dl, "db": db}
    if kind == "gemm_batch":
        s["plan"].run(1.0, s["a_ptr"], s["lda"], s["b_ptr"], s["ldb"], 0.0, s["c_ptr"], s["ldc"])
        return s["c"]
    if kind == "trsm_batch":
        s["x"].copy_(s["b"])
        s["plan"].run(1.0, s["a_ptr"], s["lda"], s["x_ptr"], s["ldb"])
        return s["x"]
    (ra, _), (rb, _) = _stored(case)
    fn = blas.dgemm if case["dtype"] == "f64" else blas.sgemm
    fn(case["ta"], case["tb"], case["m"], case["n"], case["k"], case["alpha"], s["a"], ra, s["b"], rb, case["beta"],
       s["c"], case["m"])
    return s["c"]


# ----------------------------------------------------------------- the work
def work(case):
    kind = case["kind"]
    if kind in ("gemm", "emulated", "host"):
        m, n, k, w = case["m"], case["n"], case["k"], BYTES[case["dtype"]]
        flops = (8 if case["dtype"] in "zc" else 2) * m * n * k
        return {"bytes": w * (m * k + k * n + m * n * (2 if case["beta"] else 1)), "flops": flops}
    if kind == "trsm":
        n, nr = case["n"], case["nrhs"]
        return {"bytes": 8 * (n * (n + 1) // 2 + 2 * n * nr), "flops": n * n * nr}
    if kind == "chain":
        n, nr = case["n"], case["nrhs"]
        # two solves and the masked product of dL (n^2 r each), the symmetric update (n r^2), its adjoint (2 n r^2)
        return {"bytes": 8 * (n * (n + 1) // 2 + n * nr + n * n + n * nr), "flops": 3 * n * n * nr + 3 * n * nr * nr}
    w = BYTES[case["dtype"]]
    if kind == "gemm_batch":
        m, n, k = _batch_sizes(case)
        return {"bytes": int(w * (m * k + k * n + m * n).sum()), "flops": int((2 * m * n * k).sum())}
    n, nr = _batch_sizes(case)
    return {"bytes": int(w * (n * (n + 1) // 2 + 2 * n * nr).sum()), "flops": int((n * n * nr).sum())}


# ------------------------------------------------------- the result in 64 bits
def _wide(x):
    return x.to(torch.complex128 if x.is_complex() else torch.float64)


def _op(stored, rows, trans):
    """op(X) from the column-major tensor (columns, ld) holding `rows` rows."""
    x = stored[:, :rows].t()
    return x if trans == "N" else x.t() if trans == "T" else x.t().conj()


def exact(case, seed):
    s, kind = prepare(case, seed), case["kind"]
    if kind in ("gemm", "emulated", "host"):
        a, b, c = s["a"], s["b"], s["c"]
        if kind == "host":
            a, b, c = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (a, b, c))
        (ra, _), (rb, _) = _stored(case)
        out = _wide(c).clone()
        ab = torch.matmul(_op(_wide(a), ra, case["ta"]), _op(_wide(b), rb, case["tb"]))
        window = out[:, :case["m"]]
        window.copy_((case["alpha"] * ab + case["beta"] * window.t()).t() if case["beta"] else case["alpha"] * ab.t())
        return out.cpu().numpy().T if kind == "host" else out
    if kind == "trsm":
        n = case["n"]
        left, upper = case["side"] == "L", (case["uplo"] == "U") != (case["ta"] == "T")
        rows = n if left else case["nrhs"]
        x = torch.linalg.solve_triangular(_op(s["a"], n, case["ta"]), s["b"][:, :rows].t(), upper=upper, left=left,
                                          unitriangular=case["diag"] == "U")
        out = s["b"].clone()
        out[:, :rows] = x.t()
        return out
    if kind == "chain":
        x = torch.linalg.solve_triangular(s["l"], s["b"], upper=False)
        loss = torch.sin(x.t() @ x).sum()
        dl, db = torch.autograd.grad(loss, (s["l"], s["b"]))
        return {"loss": loss.detach(), "dl": dl, "db": db}
    if kind == "gemm_batch":
        out = torch.empty(s["c"].shape, dtype=torch.float64, device="cuda")
        for m, n, k, i, j, q in zip(*_batch_sizes(case), s["a_at"], s["b_at"], s["c_at"]):
            m, n, k = int(m), int(n), int(k)
            ra, rb = (m if case["ta"] == "N" else k), (k if case["tb"] == "N" else n)
            a, b = s["a"][i:i + m * k].view(-1, ra).double(), s["b"][j:j + k * n].view(-1, rb).double()
            torch.matmul(_op(b, rb, case["tb"]).t(), _op(a, ra, case["ta"]).t(), out=out[q:q + m * n].view(n, m))
        return out
    out = torch.empty(s["b"].shape, dtype=torch.float64, device="cuda")
    for n, r, i, j in zip(*_batch_sizes(case), s["a_at"], s["b_at"]):
        n, r = int(n), int(r)
        a, b = s["a"][i:i + n * n].view(n, n).double(), s["b"][j:j + n * r].view(r, n).double()
        out[j:j + n * r] = torch.linalg.solve_triangular(a.t(), b.t(), upper=False).t().reshape(-1)
    return out
