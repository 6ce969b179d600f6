"""Performance cases of atlas_b200: what users have the library do, one pass per call of run().

Each case is one workload through the public C ABI (atlas_b200's ctypes
mirror) on device data, on a stream shared with torch as a GPU program would
share it.  The factorizations overwrite their input, so a pass first restores
it from a copy, as the callers that keep their matrix do.  Column-major
matrices live in torch tensors as their transposes: a tensor of shape
(cols, rows) is the rows x cols matrix with leading dimension rows.
"""
import ctypes
import math

import numpy as np
import torch

import atlas_b200 as AB

F64, F32, I32 = torch.float64, torch.float32, torch.int32
DEV = "cuda"
NOTRANS, TRANS = AB.CblasNoTrans, AB.CblasTrans
LOWER, UPPER = AB.CblasLower, AB.CblasUpper

_stream = None


def _use_stream():
    """One stream for torch's work and the library's (bench.py does the same)."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
        torch.cuda.set_stream(_stream)
        AB.atlb_set_stream(_stream.cuda_stream)
    return _stream


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call of a program that links the BLAS: one blocking
        # cblas_dgemm of a few tiles, where launch and call overhead count
        dict(name="dgemm_small", kind="gemm", dtype="f64", api="cblas", m=96, n=80, k=112, ta=False, tb=False, beta=0.0),
        # an ordinary product inside a user's algorithm: odd sizes (unaligned
        # columns), a transposed operand, accumulation into C
        dict(name="dgemm_ragged", kind="gemm", dtype="f64", api="dev", m=1501, n=1203, k=999, ta=True, tb=False, beta=0.5),
        # the benchmark's plain DGEMM
        dict(name="dgemm_8192", kind="gemm", dtype="f64", api="dev", m=8192, n=8192, k=8192, ta=False, tb=False, beta=0.0),
        # single precision through the drop-in call
        dict(name="sgemm_4096", kind="gemm", dtype="f32", api="cblas", m=4096, n=4096, k=4096, ta=False, tb=False, beta=0.0),
        # the small dense solve of an application: one blocking clapack_dgesv
        dict(name="dgesv_500", kind="lu", api="clapack", n=500, nrhs=1),
        # the benchmark's LU configuration: getrf + getrs, 16 right-hand sides
        dict(name="dgetrf_dgetrs_8192", kind="lu", api="dev", n=8192, nrhs=16),
        # the benchmark's Cholesky configuration
        dict(name="dpotrf_dpotrs_8192", kind="chol", uplo="L", n=8192, nrhs=16),
        # the benchmark's QR configuration
        dict(name="dgeqrf_16384x8192", kind="qr", m=16384, n=8192),
        # the headline: mixed-precision dgesv (split-TF32 factors, FP64
        # refinement) on the benchmark's matrix class
        dict(name="dsgesv_8192", kind="mixed", n=8192, nrhs=1, prec=3, kappa=1e2),
        # the benchmark's batches: 10,000 systems of orders 8..256
        dict(name="batched_posv_10k", kind="batch_posv", count=10000, lo=8, hi=256, nrhs=4, mix=2024),
        dict(name="batched_gesv_10k", kind="batch_gesv", count=10000, lo=8, hi=256, nrhs=1, mix=2024),
        # training through a Gaussian likelihood: Cholesky, solve, and the
        # reverse-mode derivatives of both
        dict(name="gaussian_grad_4096", kind="grad", n=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "lu", "chol", "qr", "mixed", "batch_posv", "batch_gesv", "grad"])
    if kind == "gemm":
        dtype = rng.choice(["f64", "f64", "f32"])
        m, n, k = (_log_int(rng, 16, 8192) for _ in range(3))
        return dict(kind=kind, dtype=dtype, api=rng.choice(["cblas", "dev"]), m=m, n=n, k=k, ta=rng.random() < 0.5,
                    tb=rng.random() < 0.5, beta=rng.choice([0.0, 1.0, 0.5]))
    if kind == "lu":
        return dict(kind=kind, api=rng.choice(["clapack", "dev"]), n=_log_int(rng, 32, 8192), nrhs=rng.choice([1, 3, 16, 64]))
    if kind == "chol":
        return dict(kind=kind, uplo=rng.choice(["L", "U"]), n=_log_int(rng, 32, 8192), nrhs=rng.choice([1, 3, 16, 64]))
    if kind == "qr":
        n = _log_int(rng, 32, 4096)
        return dict(kind=kind, m=n + _log_int(rng, 1, 8192), n=n)
    if kind == "mixed":
        return dict(kind=kind, n=_log_int(rng, 256, 8192), nrhs=rng.choice([1, 2, 4]), prec=rng.choice([0, 3]), kappa=1e2)
    if kind == "grad":
        return dict(kind=kind, n=_log_int(rng, 64, 4096))
    lo = rng.choice([8, 16, 40])
    return dict(kind=kind, count=_log_int(rng, 100, 10000), lo=lo, hi=rng.randint(lo + 1, 256), nrhs=rng.randint(1, 4),
                mix=rng.randint(1, 10 ** 6))


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _randn(g, *shape, dtype=F64):
    return torch.randn(*shape, dtype=dtype, device=DEV, generator=g)


def _uniform(g, *shape, dtype=F64):
    return torch.rand(*shape, dtype=dtype, device=DEV, generator=g) * 2 - 1


def _spd(g, n):
    b = _randn(g, n, n)
    a = torch.mm(b, b.T)
    a /= n
    a.diagonal().add_(1.0)
    return a


def _general(g, a):
    """Scale the normal entries of a (matrices in the last two dimensions) and
    add 2 along one random permutation: interchanges at nearly every column,
    and a condition number that does not grow with the order."""
    n = a.shape[-1]
    a /= math.sqrt(n)
    a[..., torch.arange(n, device=DEV), torch.randperm(n, device=DEV, generator=g)] += 2.0
    return a


def _sizes(case):
    return np.random.default_rng(case["mix"]).integers(case["lo"], case["hi"] + 1, case["count"]).astype(np.int32)


def _batch_layout(case):
    """Sizes, and each problem's offset in one packed buffer of n*n matrices
    (problems of one size side by side), and the groups (size, offset, count)."""
    ns = _sizes(case)
    off = np.zeros(case["count"], dtype=np.int64)
    boff = np.zeros(case["count"], dtype=np.int64)
    groups, at, bat = [], 0, 0
    for n in np.unique(ns):
        idx = np.nonzero(ns == n)[0]
        n = int(n)
        off[idx] = at + np.arange(len(idx)) * n * n
        boff[idx] = bat + np.arange(len(idx)) * n
        groups.append((n, at, bat, len(idx)))
        at += len(idx) * n * n
        bat += len(idx) * n
    return ns, off, boff, groups, at, bat


def _pointers(base, offsets, size):
    return (ctypes.c_void_p * len(offsets))(*[int(base + size * int(o)) for o in offsets])


def _prepare_batch(case, g, spd):
    ns, off, boff, groups, total, rows = _batch_layout(case)
    nrhs, count = case["nrhs"], case["count"]
    a0 = _randn(g, total)
    for n, at, _, cnt in groups:
        v = a0[at:at + cnt * n * n].view(cnt, n, n)
        if spd:
            v.copy_(torch.bmm(v, v.transpose(1, 2)))
            v.diagonal(dim1=1, dim2=2).add_(float(n))
        else:
            _general(g, v)
    b0 = _uniform(g, rows * nrhs)
    a, b = torch.empty_like(a0), torch.empty_like(b0)
    ipiv = torch.zeros(rows, dtype=I32, device=DEV)
    return dict(case=case, ns=ns, a0=a0, b0=b0, a=a, b=b, ipiv=ipiv, info=np.zeros(count, dtype=np.int32),
                nr=np.full(count, nrhs, dtype=np.int32), pa=_pointers(a.data_ptr(), off, 8),
                pb=_pointers(b.data_ptr(), boff * nrhs, 8), pi=_pointers(ipiv.data_ptr(), boff, 4))


def prepare(case, seed):
    _use_stream()
    g = _gen(seed)
    kind = case["kind"]
    if kind == "gemm":
        dt = F64 if case["dtype"] == "f64" else F32
        m, n, k = case["m"], case["n"], case["k"]
        # row-major operands for the cblas form, column-major (transposed
        # tensors) for the device form: op(A) is m x k, op(B) k x n
        col = case["api"] == "dev"
        ash = (k, m) if case["ta"] != col else (m, k)
        bsh = (n, k) if case["tb"] != col else (k, n)
        csh = (n, m) if col else (m, n)
        s = dict(case=case, a=_uniform(g, *ash, dtype=dt), b=_uniform(g, *bsh, dtype=dt), c=torch.zeros(*csh, dtype=dt, device=DEV))
        if case["beta"] != 0.0:
            s["c0"] = _uniform(g, *csh, dtype=dt)
        return s
    if kind == "lu":
        n = case["n"]
        a0, b0 = _general(g, _randn(g, n, n)), _uniform(g, case["nrhs"], n)
        return dict(case=case, a0=a0, b0=b0, a=torch.empty_like(a0), b=torch.empty_like(b0),
                    ipiv=torch.zeros(n, dtype=I32, device=DEV), info=torch.zeros(1, dtype=I32, device=DEV))
    if kind == "chol":
        n = case["n"]
        a0, b0 = _spd(g, n), _uniform(g, case["nrhs"], n)
        return dict(case=case, a0=a0, b0=b0, a=torch.empty_like(a0), b=torch.empty_like(b0),
                    info=torch.zeros(1, dtype=I32, device=DEV))
    if kind == "qr":
        a0 = _uniform(g, case["n"], case["m"])
        return dict(case=case, a0=a0, a=torch.empty_like(a0), tau=torch.zeros(min(case["m"], case["n"]), dtype=F64, device=DEV))
    if kind == "mixed":
        n = case["n"]
        q1, _ = torch.linalg.qr(_randn(g, n, n))
        q2, _ = torch.linalg.qr(_randn(g, n, n))
        sv = torch.logspace(0, -math.log10(case["kappa"]), n, dtype=F64, device=DEV)
        a = torch.mm(q2 * sv, q1.T)  # the transpose of Q1 diag(s) Q2^T: its column-major storage
        del q1, q2
        b = _uniform(g, case["nrhs"], n)
        return dict(case=case, a=a, b=b, x=torch.empty_like(b), ipiv=torch.zeros(n, dtype=I32, device=DEV), it=np.zeros(1, dtype=np.int32))
    if kind == "grad":
        n = case["n"]
        a0 = _spd(g, n)
        y = _uniform(g, n)
        z = lambda: torch.zeros(n, n, dtype=F64, device=DEV)  # noqa: E731
        return dict(case=case, a0=a0, y=y, l=z(), x=torch.empty_like(y), lbar=z(), abar=z(), ybar=torch.empty_like(y),
                    info=torch.zeros(1, dtype=I32, device=DEV))
    return _prepare_batch(case, g, kind == "batch_posv")


# ---------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "gemm":
        m, n, k, beta = case["m"], case["n"], case["k"], case["beta"]
        a, b, c = s["a"], s["b"], s["c"]
        if beta != 0.0:
            c.copy_(s["c0"])
        ta, tb = (TRANS if case["ta"] else NOTRANS), (TRANS if case["tb"] else NOTRANS)
        lda, ldb, ldc = a.shape[1], b.shape[1], c.shape[1]
        f64 = case["dtype"] == "f64"
        if case["api"] == "cblas":
            (AB.cblas_dgemm if f64 else AB.cblas_sgemm)(AB.CblasRowMajor, ta, tb, m, n, k, 1.0, a, lda, b, ldb, beta, c, ldc)
        else:
            (AB.atlb_dgemm_dev if f64 else AB.atlb_sgemm_dev)(ta, tb, m, n, k, 1.0, a, lda, b, ldb, beta, c, ldc)
        return c
    if kind == "lu":
        n, nrhs, a, b, ipiv = case["n"], case["nrhs"], s["a"], s["b"], s["ipiv"]
        a.copy_(s["a0"])
        b.copy_(s["b0"])
        if case["api"] == "clapack":
            info = AB.clapack_dgesv(AB.CblasColMajor, n, nrhs, a, n, ipiv, b, n)
        else:
            info = s["info"]
            AB.atlb_dgetrf_dev(n, n, a, n, ipiv, info)
            AB.atlb_dgetrs_dev(NOTRANS, n, nrhs, a, n, ipiv, b, n)
        return dict(x=b, lu=a, ipiv=ipiv, info=info)
    if kind == "chol":
        n, nrhs, a, b = case["n"], case["nrhs"], s["a"], s["b"]
        uplo = LOWER if case["uplo"] == "L" else UPPER
        a.copy_(s["a0"])
        b.copy_(s["b0"])
        AB.atlb_dpotrf_dev(uplo, n, a, n, s["info"])
        AB.atlb_dpotrs_dev(uplo, n, nrhs, a, n, b, n)
        return dict(x=b, factor=a, info=s["info"])
    if kind == "qr":
        s["a"].copy_(s["a0"])
        AB.atlb_dgeqrf_dev(case["m"], case["n"], s["a"], case["m"], s["tau"])
        return dict(qr=s["a"], tau=s["tau"])
    if kind == "mixed":
        n, nrhs = case["n"], case["nrhs"]
        info = AB.atlb_dsgesv(n, nrhs, s["a"], n, s["ipiv"], s["b"], n, s["x"], n, case["prec"], s["it"])
        return dict(x=s["x"], info=info)
    if kind == "grad":
        # loss = log det A + y^T A^-1 y
        n, l, x, lbar, abar = case["n"], s["l"], s["x"], s["lbar"], s["abar"]
        l.copy_(s["a0"])
        x.copy_(s["y"])
        AB.atlb_dpotrf_dev(LOWER, n, l, n, s["info"])
        AB.atlb_dpotrs_dev(LOWER, n, 1, l, n, x, n)
        lbar.zero_()
        lbar.view(-1)[:: n + 1] = 2.0 / l.view(-1)[:: n + 1]
        AB.atlb_dpotrf_adjoint_dev(n, l, n, lbar, n, abar, n)
        AB.atlb_dpotrs_adjoint_dev(n, 1, l, n, x, n, s["y"], n, s["ybar"], n, abar, n)
        return dict(x=x, factor=l, abar=abar, ybar=s["ybar"], info=s["info"])
    a, b, ns, count = s["a"], s["b"], s["ns"], case["count"]
    a.copy_(s["a0"])
    b.copy_(s["b0"])
    if kind == "batch_posv":
        AB.atlb_dposv_batched(count, ns, s["pa"], ns, s["pb"], ns, s["nr"], s["info"])
        return dict(x=b, factor=a, info=s["info"])
    AB.atlb_dgesv_batched(count, ns, s["pa"], ns, s["pi"], s["pb"], ns, s["nr"], s["info"])
    return dict(x=b, lu=a, ipiv=s["ipiv"], info=s["info"])


# ---------------------------------------------------------------- floors

def work(case):
    """Bytes (each input read once, each output written once) and flops of one pass."""
    kind = case["kind"]
    if kind == "gemm":
        m, n, k, e = case["m"], case["n"], case["k"], 8 if case["dtype"] == "f64" else 4
        return {"bytes": e * (m * k + k * n + m * n * (2 if case["beta"] != 0.0 else 1)), "flops": 2.0 * m * n * k}
    if kind == "lu":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 16 * n * n + 16 * n * r + 4 * n, "flops": 2 / 3 * n ** 3 + 2.0 * n * n * r}
    if kind == "chol":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8 * n * n + 16 * n * r, "flops": n ** 3 / 3 + 2.0 * n * n * r}
    if kind == "qr":
        m, n = case["m"], case["n"]
        return {"bytes": 16 * m * n, "flops": 2.0 * m * n * n - 2 / 3 * n ** 3}
    if kind == "mixed":
        n, r = case["n"], case["nrhs"]
        return {"bytes": 8 * n * n + 16 * n * r, "flops": 2 / 3 * n ** 3 + 2.0 * n * n * r}
    if kind == "grad":
        n = case["n"]
        return {"bytes": 8 * n * n * 2 + 24 * n, "flops": n ** 3 / 3 + 2.0 * n ** 3 + 4.0 * n * n}
    ns, r = _sizes(case).astype(np.float64), case["nrhs"]
    if kind == "batch_posv":
        return {"bytes": float((8 * ns ** 2 + 16 * ns * r).sum()), "flops": float((ns ** 3 / 3 + 2 * ns ** 2 * r).sum())}
    return {"bytes": float((16 * ns ** 2 + 16 * ns * r + 4 * ns).sum()), "flops": float((2 / 3 * ns ** 3 + 2 * ns ** 2 * r).sum())}


# ---------------------------------------------------------------- in 64 bits

def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "gemm":
        col = case["api"] == "dev"
        a, b = s["a"].double(), s["b"].double()
        a, b = (a.T if col else a), (b.T if col else b)
        r = torch.mm(a.T if case["ta"] else a, b.T if case["tb"] else b)
        if case["beta"] != 0.0:
            r += case["beta"] * (s["c0"].T if col else s["c0"]).double()
        return r.T.contiguous() if col else r
    if kind == "lu":
        a = s["a0"].T.contiguous()
        lu, piv = torch.linalg.lu_factor(a)
        return dict(x=torch.linalg.lu_solve(lu, piv, s["b0"].T).T.contiguous(), lu=lu.T.contiguous(), ipiv=None, info=None)
    if kind == "chol":
        low = torch.linalg.cholesky(s["a0"])
        x = torch.cholesky_solve(s["b0"].T.contiguous(), low).T.contiguous()
        # the other triangle keeps the input; the tensor holds the transpose
        if case["uplo"] == "L":
            f = torch.tril(s["a0"], -1) + low.T
        else:
            f = torch.triu(s["a0"], 1) + low
        return dict(x=x, factor=f.contiguous(), info=None)
    if kind == "qr":
        a, tau = torch.geqrf(s["a0"].T)
        return dict(qr=a.T.contiguous(), tau=tau)
    if kind == "mixed":
        return dict(x=torch.linalg.solve(s["a"].T, s["b"].T).T.contiguous(), info=None)
    if kind == "grad":
        low = torch.linalg.cholesky(s["a0"])
        inv = torch.cholesky_inverse(low)
        x = torch.mv(inv, s["y"])
        # the tensor holds the transpose: L in its upper triangle, the rest is the input's
        f = torch.tril(s["a0"], -1) + low.T
        return dict(x=x, factor=f.contiguous(), abar=inv - torch.outer(x, x), ybar=x.clone(), info=None)
    _, _, _, groups, _, _ = _batch_layout(case)
    a, b, r = s["a0"], s["b0"], case["nrhs"]
    for n, at, bat, cnt in groups:
        v = a[at:at + cnt * n * n].view(cnt, n, n)  # transposes of the matrices
        w = b[bat * r:(bat + cnt * n) * r].view(cnt, r, n)
        rhs = w.transpose(1, 2).contiguous()
        if kind == "batch_posv":
            low = torch.linalg.cholesky(v)
            w.copy_(torch.cholesky_solve(rhs, low).transpose(1, 2))
            v.copy_(torch.tril(v, -1) + low.transpose(1, 2))
        else:
            lu, piv = torch.linalg.lu_factor(v.transpose(1, 2).contiguous())
            w.copy_(torch.linalg.lu_solve(lu, piv, rhs).transpose(1, 2))
            v.copy_(lu.transpose(1, 2))
    if kind == "batch_posv":
        return dict(x=b, factor=a, info=None)
    return dict(x=b, lu=a, ipiv=None, info=None)
