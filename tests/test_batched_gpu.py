"""Batched uneven-size problems (one persistent launch per batch) against a
per-instance loop of the oracle / numpy: batched Cholesky solve, batched LU
(ipiv identical to the oracle's getrf on each instance) with solve, and the
grouped DGEMM (l3blastst residual per instance)."""
import ctypes

import numpy as np
import pytest

import atlas_b200 as AB
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _ptr_array(ts, ctype=ctypes.c_void_p):
    return (ctype * len(ts))(*[t.data_ptr() for t in ts])


def _int_array(v):
    return np.ascontiguousarray(v, dtype=np.int32)


def test_batched_posv(gpu):
    import torch
    rng = np.random.default_rng(0)
    count = 300
    ns = rng.integers(8, 257, count)
    ns[:3] = [8, 96, 97]          # the size-bucket edges
    nr = 4
    As, Bs, a0s, b0s = [], [], [], []
    for n in ns:
        g = rng.standard_normal((n, n))
        a = g @ g.T + n * np.eye(n)           # A = B B^T + n I
        b = rng.uniform(-1, 1, (n, nr))
        a0s.append(a); b0s.append(b)
        As.append(torch.tensor(np.asfortranarray(a).T.copy(), device="cuda"))   # column-major storage
        Bs.append(torch.tensor(np.asfortranarray(b).T.copy(), device="cuda"))
    info = np.zeros(count, dtype=np.int32)
    r = AB.atlb_dposv_batched(count, _int_array(ns), _ptr_array(As), _int_array(ns), _ptr_array(Bs),
                              _int_array(ns), _int_array([nr] * count), info)
    assert r == 0 and np.all(info == 0)
    for i in range(count):
        x = Bs[i].cpu().numpy().T
        res = np.abs(a0s[i] @ x - b0s[i]).max() / (np.abs(a0s[i]).sum(1).max() * np.abs(x).max())
        assert res < 1e-14, (i, ns[i], res)
        L = np.tril(As[i].cpu().numpy().T)
        np.testing.assert_allclose(L, np.linalg.cholesky(a0s[i]), rtol=1e-10, atol=1e-12)


@pytest.mark.parametrize("nrhs", [0, 1, 8, 9, 20])
def test_batched_posv_tile_edges(gpu, nrhs):
    """Orders at the edges of the 16 x 16 tiles and of the size buckets, leading
    dimensions above the order, right-hand sides across the block rows of
    eight; nothing outside the lower triangle and B's n rows is written.
    Bounds: |A - L L^T| <= (n + 1) u |L||L^T| and the solve's residual
    (3 n + 1) u |L||L^T||x| componentwise (Higham, Accuracy and Stability,
    theorems 10.3 and 10.4), u = 2^-53, doubled for the reciprocal diagonal."""
    import torch
    rng = np.random.default_rng(nrhs)
    ns = [1, 2, 15, 16, 17, 33, 48, 49, 112, 113, 176, 177, 240, 255, 256, 0]
    u = 2.0 ** -53
    As, Bs, a0s, b0s, lda, ldb = [], [], [], [], [], []
    for n in ns:
        la, lb = n + 3, n + 5
        g = rng.standard_normal((n, n))
        a = np.full((max(n, 1), la), 7.0)             # row = column of the matrix
        a[:n, :n] = g @ g.T + n * np.eye(n)
        b = np.full((max(nrhs, 1), lb), 9.0)
        b[:, :n] = rng.uniform(-1, 1, (max(nrhs, 1), n))
        a0s.append(a)
        b0s.append(b)
        lda.append(la)
        ldb.append(lb)
        As.append(torch.tensor(a, device="cuda"))
        Bs.append(torch.tensor(b, device="cuda"))
    count = len(ns)
    info = np.full(count, -1, dtype=np.int32)
    assert AB.atlb_dposv_batched(count, _int_array(ns), _ptr_array(As), _int_array(lda), _ptr_array(Bs),
                                 _int_array(ldb), _int_array([nrhs] * count), info) == 0
    assert np.all(info == 0)
    for i, n in enumerate(ns):
        a, b = As[i].cpu().numpy(), Bs[i].cpu().numpy()
        assert np.array_equal(a[:, n:], a0s[i][:, n:]) and np.array_equal(b[:, n:], b0s[i][:, n:])
        if n == 0:
            continue
        low = np.triu(a[:n, :n]).T                    # rows of `a` are columns of L
        assert np.array_equal(np.tril(a[:n, :n], -1), np.tril(a0s[i][:n, :n], -1))
        mag = np.abs(low) @ np.abs(low.T)
        assert np.all(np.abs(low @ low.T - a0s[i][:n, :n]) <= 2 * (n + 2) * u * mag)
        for r in range(nrhs):
            x = b[r, :n]
            assert np.all(np.abs(a0s[i][:n, :n] @ x - b0s[i][r, :n]) <= 2 * (3 * n + 2) * u * (mag @ np.abs(x)))
        if nrhs == 0:
            assert np.array_equal(b, b0s[i])


def test_batched_posv_reports_indefinite(gpu):
    import torch
    ns = np.array([20, 150], dtype=np.int32)
    As, Bs = [], []
    for n in ns:
        a = np.eye(n) * 2.0
        a[n // 2, n // 2] = -1.0
        As.append(torch.tensor(a, device="cuda"))
        Bs.append(torch.ones(1, n, dtype=torch.float64, device="cuda"))
    info = np.zeros(2, dtype=np.int32)
    assert AB.atlb_dposv_batched(2, ns, _ptr_array(As), ns, _ptr_array(Bs), ns, _int_array([1, 1]), info) == 0
    assert list(info) == [n // 2 + 1 for n in ns]


def test_batched_gesv_matches_oracle(gpu, orc):
    import torch
    rng = np.random.default_rng(1)
    count = 120
    ns = rng.integers(8, 257, count)
    ns[:4] = [8, 160, 161, 256]   # shared-memory / global-memory edge
    As, Bs, Ps, a0s, b0s = [], [], [], [], []
    for k, n in enumerate(ns):
        a = O.gegen(int(n), int(n), int(n), 7 + k)[:n, :n].copy(order="F")   # random pivots
        b = rng.uniform(-1, 1, (n, 2))
        a0s.append(a); b0s.append(b)
        As.append(torch.tensor(a.T.copy(), device="cuda"))
        Bs.append(torch.tensor(np.asfortranarray(b).T.copy(), device="cuda"))
        Ps.append(torch.zeros(n, dtype=torch.int32, device="cuda"))
    info = np.zeros(count, dtype=np.int32)
    r = AB.atlb_dgesv_batched(count, _int_array(ns), _ptr_array(As), _int_array(ns), _ptr_array(Ps),
                              _ptr_array(Bs), _int_array(ns), _int_array([2] * count), info)
    assert r == 0 and np.all(info == 0)
    for i in range(count):
        lu, rpiv, _ = orc.dgetrf(a0s[i].copy(order="F"))
        np.testing.assert_array_equal(Ps[i].cpu().numpy(), rpiv)
        assert np.max(np.abs(As[i].cpu().numpy().T - lu)) < 1e-10
        x = Bs[i].cpu().numpy().T
        xt = np.asfortranarray(np.linalg.solve(a0s[i], b0s[i]))   # the oracle reads column-major
        assert orc.resid_slv(a0s[i], np.asfortranarray(x), xt) <= 100


@pytest.mark.parametrize("nrhs", [0, 1, 8, 9, 20])
def test_batched_gesv_panel_edges(gpu, orc, nrhs):
    """Orders at the edges of the 16-column panels and of the size buckets,
    leading dimensions above the order, right-hand sides across the eight that
    ride along, random pivots; ipiv equal to the oracle's, nothing outside A and
    B's n rows written, |P A - L U| <= (n + 1) u |L||U| and the solve's residual
    <= (3 n + 2) u |L||U||x| componentwise (Higham, theorems 9.3 and 9.4),
    u = 2^-53, doubled for the reciprocal pivots."""
    import torch
    rng = np.random.default_rng(100 + nrhs)
    ns = [1, 2, 15, 16, 17, 48, 63, 64, 65, 127, 128, 129, 255, 256, 0]
    u = 2.0 ** -53
    As, Bs, Ps, a0s, b0s, lda, ldb = [], [], [], [], [], [], []
    for n in ns:
        la, lb = n + 3, n + 5
        a = np.full((max(n, 1), la), 7.0)             # row = column of the matrix
        a[:n, :n] = rng.uniform(-1, 1, (n, n))
        b = np.full((max(nrhs, 1), lb), 9.0)
        b[:, :n] = rng.uniform(-1, 1, (max(nrhs, 1), n))
        a0s.append(a)
        b0s.append(b)
        lda.append(la)
        ldb.append(lb)
        As.append(torch.tensor(a, device="cuda"))
        Bs.append(torch.tensor(b, device="cuda"))
        Ps.append(torch.full((n + 1,), -7, dtype=torch.int32, device="cuda"))
    count = len(ns)
    info = np.full(count, -1, dtype=np.int32)
    assert AB.atlb_dgesv_batched(count, _int_array(ns), _ptr_array(As), _int_array(lda), _ptr_array(Ps),
                                 _ptr_array(Bs), _int_array(ldb), _int_array([nrhs] * count), info) == 0
    assert np.all(info == 0)
    for i, n in enumerate(ns):
        a, b, piv = As[i].cpu().numpy(), Bs[i].cpu().numpy(), Ps[i].cpu().numpy()
        assert np.array_equal(a[:, n:], a0s[i][:, n:]) and np.array_equal(b[:, n:], b0s[i][:, n:])
        assert piv[n] == -7
        if n == 0:
            continue
        a0 = np.asfortranarray(a0s[i][:n, :n].T)
        _, rpiv, _ = orc.dgetrf(a0.copy(order="F"))
        np.testing.assert_array_equal(piv[:n], rpiv)
        lu = a[:n, :n].T
        low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
        pa = a0.copy()
        for k in range(n):
            pa[[k, piv[k]]] = pa[[piv[k], k]]
        mag = np.abs(low) @ np.abs(up)
        assert np.all(np.abs(low @ up - pa) <= 2 * (n + 2) * u * mag)
        for r in range(nrhs):
            pb = b0s[i][r, :n].copy()
            for k in range(n):
                pb[[k, piv[k]]] = pb[[piv[k], k]]
            x = b[r, :n]
            assert np.all(np.abs(pa @ x - pb) <= 2 * (3 * n + 3) * u * (mag @ np.abs(x)))


def test_batched_gesv_singular(gpu):
    """A zero column, a zero matrix and a row repeated in a matrix whose elimination
    is exact (entries 0 and +-1, pivots of +-1): the first zero pivot's position, the
    factorization completed, the right-hand side untouched."""
    import torch
    n = 40
    rng = np.random.default_rng(3)
    a = [rng.uniform(-1, 1, (n, n)), np.zeros((n, n)), None]
    a[0][17] = 0.0                                     # column 17 (stored as a row)
    rep = np.triu(rng.integers(-1, 2, (n, n)).astype(np.float64), 1) + np.eye(n)
    rep[25] = rep[7]
    a[2] = np.ascontiguousarray(rep.T)
    As = [torch.tensor(m, device="cuda") for m in a] + [torch.eye(n, dtype=torch.float64, device="cuda")]
    Bs = [torch.ones(1, n, dtype=torch.float64, device="cuda") for _ in As]
    Ps = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in As]
    ns, one = _int_array([n] * 4), _int_array([1] * 4)
    info = np.zeros(4, dtype=np.int32)
    assert AB.atlb_dgesv_batched(4, ns, _ptr_array(As), ns, _ptr_array(Ps), _ptr_array(Bs), ns, one, info) == 0
    _, _, rinfo = O.dgetrf(np.asfortranarray(rep))
    assert list(info) == [18, 1, rinfo, 0] and rinfo == 26
    assert np.array_equal(Ps[1].cpu().numpy(), np.arange(n)) and np.array_equal(Ps[3].cpu().numpy(), np.arange(n))
    for k in (0, 1, 2):
        assert np.all(Bs[k].cpu().numpy() == 1.0)
    assert np.all(np.isfinite(As[0].cpu().numpy()))


@pytest.mark.parametrize("scale", [0, 490, 1020])
@pytest.mark.parametrize("nrhs", [1, 10])
def test_batched_gesv_divides_by_its_pivots(gpu, nrhs, scale):
    """Diagonal systems, subnormal pivots among them, whose reciprocals are
    infinite, and pivots and right-hand sides over 2^-scale .. 2^scale: every solution
    is the one correctly rounded quotient, zero where the right-hand side is zero."""
    import torch
    rng = np.random.default_rng(nrhs + scale)
    ns = [1, 5, 17, 40, 64, 100, 129, 256]
    As, Bs, Ps, want = [], [], [], []
    for n in ns:
        d = rng.uniform(-2, 2, n) * 2.0 ** rng.integers(-scale, scale + 1, n)
        d[::3] = rng.integers(1, 9, d[::3].size) * 2.0 ** -1070
        x = rng.integers(-3, 4, (nrhs, n)).astype(np.float64)
        b = rng.uniform(-1, 1, (nrhs, n)) * 2.0 ** rng.integers(-scale, scale + 1, (nrhs, n))
        b = np.where(np.abs(d) < 1e-300, x * d, b)
        b[:, 1::7] = 0.0
        with np.errstate(all="ignore"):
            want.append(b / d)
        As.append(torch.tensor(np.diag(d), device="cuda"))
        Bs.append(torch.tensor(b, device="cuda"))
        Ps.append(torch.zeros(n, dtype=torch.int32, device="cuda"))
    info = np.full(len(ns), -1, dtype=np.int32)
    assert AB.atlb_dgesv_batched(len(ns), _int_array(ns), _ptr_array(As), _int_array(ns), _ptr_array(Ps),
                                 _ptr_array(Bs), _int_array(ns), _int_array([nrhs] * len(ns)), info) == 0
    assert np.all(info == 0)
    for b, w in zip(Bs, want):
        # an overflowed solution times a zero of U is NaN in the rows above it
        b, ok = b.cpu().numpy(), np.cumprod(np.isfinite(w)[:, ::-1], axis=1)[:, ::-1].astype(bool)
        np.testing.assert_array_equal(b[ok], w[ok])


def test_batched_dgemm_uneven(gpu, orc):
    import torch
    rng = np.random.default_rng(2)
    count = 200
    M, N, K = (rng.integers(16, 513, count) for _ in range(3))
    As = [torch.rand(k, m, dtype=torch.float64, device="cuda") * 2 - 1 for m, k in zip(M, K)]   # col-major m x k
    Bs = [torch.rand(n, k, dtype=torch.float64, device="cuda") * 2 - 1 for k, n in zip(K, N)]
    Cs = [torch.rand(n, m, dtype=torch.float64, device="cuda") for m, n in zip(M, N)]
    C0 = [c.clone() for c in Cs]
    r = AB.atlb_dgemm_batched_dev(111, 111, count, _int_array(M), _int_array(N), _int_array(K), 1.5,
                                  _ptr_array(As), _int_array(M), _ptr_array(Bs), _int_array(K), -0.5,
                                  _ptr_array(Cs), _int_array(M))
    assert r == 0
    AB.atlb_sync()
    for i in range(count):
        a = np.asfortranarray(As[i].cpu().numpy().T)
        b = np.asfortranarray(Bs[i].cpu().numpy().T)
        c0 = np.asfortranarray(C0[i].cpu().numpy().T)
        c = np.asfortranarray(Cs[i].cpu().numpy().T)
        assert orc.resid_gemm(111, 111, int(M[i]), int(N[i]), int(K[i]), 1.5, a, b, -0.5, c0, c) < 50


@pytest.mark.parametrize("edges", [(48, 49), (112, 113), (176, 177)])
def test_batched_posv_graph_replays(gpu, edges):
    """Batches with orders on both sides of a size bucket's edge: the third and
    later calls of one batch shape (replayed from a CUDA graph) solve the new data
    each call carries."""
    import torch
    rng = np.random.default_rng(edges[1])
    count, nr = 64, 2
    ns = rng.integers(8, 257, count)
    ns[:4] = [*edges, 8, 256]
    for call in range(4):
        As, Bs, a0s, b0s = [], [], [], []
        for n in ns:
            g = rng.standard_normal((n, n))
            a = g @ g.T + n * np.eye(n)
            b = rng.uniform(-1, 1, (n, nr))
            a0s.append(a)
            b0s.append(b)
            As.append(torch.tensor(a, device="cuda"))            # symmetric: either order
            Bs.append(torch.tensor(np.ascontiguousarray(b.T), device="cuda"))
        info = np.zeros(count, dtype=np.int32)
        assert AB.atlb_dposv_batched(count, _int_array(ns), _ptr_array(As), _int_array(ns), _ptr_array(Bs),
                                     _int_array(ns), _int_array([nr] * count), info) == 0
        assert np.all(info == 0)
        for i in range(count):
            x = Bs[i].cpu().numpy().T
            res = np.abs(a0s[i] @ x - b0s[i]).max() / (np.abs(a0s[i]).sum(1).max() * np.abs(x).max())
            assert res < 1e-14, (call, i, ns[i], res)


def test_batched_getrf_only_matches_oracle(gpu):
    import torch
    rng = np.random.default_rng(21)
    count = 40
    ns = rng.integers(8, 257, count)
    As, Ps, a0s = [], [], []
    for n in ns:
        a = O.lu_matrix(int(n), int(n) + 1)
        a0s.append(a)
        As.append(torch.tensor(np.ascontiguousarray(a.T), device="cuda"))
        Ps.append(torch.zeros(int(n), dtype=torch.int32, device="cuda"))
    info = np.zeros(count, dtype=np.int32)
    for _ in range(3):  # replays from the graph on the later calls
        for i, a in enumerate(a0s):
            As[i].copy_(torch.tensor(np.ascontiguousarray(a.T), device="cuda"))
        assert AB.atlb_dgetrf_batched(count, _int_array(ns), _ptr_array(As), _int_array(ns), _ptr_array(Ps),
                                      info) == 0
        assert np.all(info == 0)
        for i in range(count):
            ref, rpiv, _ = O.dgetrf(a0s[i].copy(order="F"))
            np.testing.assert_array_equal(Ps[i].cpu().numpy(), rpiv)
            assert np.abs(As[i].cpu().numpy().T - ref).max() < 1e-12


def test_batched_getrf_ties_and_zero_columns_match_oracle(gpu):
    """Pivot ties (entries in {-2..2}: many equal |values| per column, the
    first maximum wins) and exactly-zero columns (info = first zero pivot,
    1-based; the factorization completes, as ATL_getf2 does), on sizes that
    cross the 16-column panels of the batched LU."""
    import torch
    ns = [8, 17, 33, 64, 100, 130, 200, 256]
    As, Ps, a0s, zero_col = [], [], [], []
    for k, n in enumerate(ns):
        a = np.asfortranarray(np.round(4.0 * O.gegen(n, n, n, 40 + k)[:n, :n]))
        zc = -1
        if k % 2:          # an exactly-zero column past the first panel
            zc = min(n - 1, 16 + 3 * k)
            a[:, zc] = 0.0
        zero_col.append(zc)
        a0s.append(a)
        As.append(torch.tensor(np.ascontiguousarray(a.T), device="cuda"))
        Ps.append(torch.zeros(n, dtype=torch.int32, device="cuda"))
    info = np.zeros(len(ns), dtype=np.int32)
    assert AB.atlb_dgetrf_batched(len(ns), _int_array(ns), _ptr_array(As), _int_array(ns), _ptr_array(Ps),
                                  info) == 0
    for i, n in enumerate(ns):
        ref, rpiv, rinfo = O.dgetrf(a0s[i].copy(order="F"))
        assert info[i] == rinfo, (n, info[i], rinfo)
        if zero_col[i] >= 0:
            assert rinfo > 0
        np.testing.assert_array_equal(Ps[i].cpu().numpy(), rpiv)
        assert np.abs(As[i].cpu().numpy().T - ref).max() <= 1e-12 * max(1.0, np.abs(ref).max())
