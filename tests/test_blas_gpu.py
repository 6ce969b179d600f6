"""Parity of the GPU level-3 BLAS with the reference: the reference's own C
BLAS outputs (tests/golden/ref_blas.npz) and the oracle, through the C ABI
with host buffers (the drop-in path), checked by bin/l3blastst.c's residual
(< 50) plus an elementwise tolerance, with the lda gaps checked for stray
writes (ATL_gechkgap)."""
import os

import numpy as np
import pytest

import atlas_b200 as AB
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "ref_blas.npz")
CM, RM = AB.CblasColMajor, AB.CblasRowMajor
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def gold():
    return np.load(GOLD)


def test_dgemm_golden_cases(gpu, orc, gold):
    for i in range(int(gold["counts"][0])):
        m, n, k, ta, tb, alpha, beta = gold[f"gemm{i}"]
        m, n, k, ta, tb = int(m), int(n), int(k), int(ta), int(tb)
        a, b = gold[f"gemm{i}_A"], gold[f"gemm{i}_B"]
        c0 = gold[f"gemm{i}_C0"]
        c = np.array(c0, order="F")
        AB.cblas_dgemm(CM, ta, tb, m, n, k, alpha, a, a.shape[0], b, b.shape[0], beta, c, c.shape[0])
        ref = gold[f"gemm{i}_C"]
        r = orc.resid_gemm(ta, tb, m, n, k, alpha, a, b, beta, c0, c)
        assert r < 50.0, f"case {i}: l3blastst residual {r}"
        assert np.max(np.abs(c[:m, :n] - ref[:m, :n])) <= 1e-13 * max(1, k), f"case {i}"
        assert orc.gechkgap(c, m, n) == 0


@pytest.mark.parametrize("ta", [111, 112])
@pytest.mark.parametrize("tb", [111, 112])
@pytest.mark.parametrize("m,n,k", [(129, 257, 95), (300, 200, 513), (1, 130, 17), (128, 128, 16)])
def test_dgemm_vs_oracle(gpu, orc, ta, tb, m, n, k):
    ma, na = (m, k) if ta == 111 else (k, m)
    mb, nb = (k, n) if tb == 111 else (n, k)
    a = orc.gegen(ma, na, ma + 1, 3 + m)     # odd lda: 8-byte staging path on the host side
    b = orc.gegen(mb, nb, mb + 2, 5 + n)
    c0 = orc.gegen(m, n, m + 3, 7 + k)
    c = np.array(c0, order="F")
    AB.cblas_dgemm(CM, ta, tb, m, n, k, 0.75, a, a.shape[0], b, b.shape[0], -1.25, c, c.shape[0])
    r = orc.resid_gemm(ta, tb, m, n, k, 0.75, a, b, -1.25, c0, c)
    assert r < 50.0
    assert orc.gechkgap(c, m, n) == 0


def test_dgemm_device_pointers_unaligned_lda(gpu, orc):
    import torch
    m, n, k = 77, 65, 91
    A = torch.randn(81, k, dtype=torch.float64, device="cuda")  # lda = 81 (odd)
    B = torch.randn(k, n, dtype=torch.float64, device="cuda")
    C = torch.zeros(m, n, dtype=torch.float64, device="cuda")
    # column-major views: pass the transposed storage of row-major torch tensors
    At, Bt, Ct = A.t().contiguous(), B.t().contiguous(), C.t().contiguous()
    assert AB.atlb_dgemm_dev(111, 111, m, n, k, 1.0, At, 81, Bt, k, 0.0, Ct, m) == 0
    AB.atlb_sync()
    ref = A[:m].double() @ B
    assert torch.allclose(Ct.t(), ref, rtol=1e-12, atol=1e-12)


def test_dgemm_row_major_and_syrk_shortcut(gpu, orc):
    m, n, k = 70, 50, 40
    a = orc.uniform((m, k), 1)  # row-major M x K == col-major K x M storage
    b = orc.uniform((k, n), 2)
    A = np.ascontiguousarray(a)
    B = np.ascontiguousarray(b)
    C = np.zeros((m, n))
    AB.cblas_dgemm(RM, 111, 111, m, n, k, 1.0, A, k, B, n, 0.0, C, n)
    np.testing.assert_allclose(C, a @ b, rtol=1e-12, atol=1e-12)
    # A == B, TA != TB, beta == 0: the reference calls SYRK + reflect (cblas_dgemm.c:123-129)
    S = np.zeros((m, m), order="F")
    af = np.asfortranarray(a)
    AB.cblas_dgemm(CM, 111, 112, m, m, k, 1.0, af, m, af, m, 0.0, S, m)
    np.testing.assert_allclose(S, a @ a.T, rtol=1e-12, atol=1e-12)
    assert np.array_equal(S, S.T)


def test_dgemm_beta_zero_ignores_nan(gpu):
    c = np.full((9, 9), np.nan, order="F")
    a = np.ones((9, 9), order="F")
    AB.cblas_dgemm(CM, 111, 111, 9, 9, 9, 1.0, a, 9, a, 9, 0.0, c, 9)
    assert np.all(c == 9.0)


@pytest.mark.parametrize("ta", [111, 112])
@pytest.mark.parametrize("tb", [111, 112])
def test_sgemm_vs_oracle(gpu, orc, ta, tb):
    m, n, k = 190, 133, 257
    ma, na = (m, k) if ta == 111 else (k, m)
    mb, nb = (k, n) if tb == 111 else (n, k)
    a = np.asfortranarray(orc.uniform((ma, na), 4), dtype=np.float32)
    b = np.asfortranarray(orc.uniform((mb, nb), 5), dtype=np.float32)
    c0 = np.asfortranarray(orc.uniform((m, n), 6), dtype=np.float32)
    c = c0.copy(order="F")
    AB.cblas_sgemm(CM, ta, tb, m, n, k, 1.5, a, ma, b, mb, 0.5, c, m)
    cr = c0.copy(order="F")
    orc.sgemm(ta, tb, m, n, k, 1.5, a, b, 0.5, cr)
    # FP32 with K=257: |error| <= ~K * eps32 * sum|a||b|
    tol = 4 * k * np.finfo(np.float32).eps * (np.abs(a).max() * np.abs(b).max() * k + 1)
    assert np.max(np.abs(c - cr)) <= tol


@pytest.mark.parametrize("ta,tb", [(111, 111), (112, 112), (111, 112)])
@pytest.mark.parametrize("m,n,k", [(200, 150, 5000), (128, 128, 4096)])
def test_sgemm_split_k_vs_fp64(gpu, ta, tb, m, n, k):
    """A few output tiles with a long K: the SIMT FP32 GEMM splits K over the
    grid (partial products summed by a second pass) -- alpha, beta and the
    transposes still apply, to FP32 accuracy against an FP64 product."""
    rng = np.random.default_rng(m + n + k + ta + tb)
    ma, na = (m, k) if ta == 111 else (k, m)
    mb, nb = (k, n) if tb == 111 else (n, k)
    a = np.asfortranarray(rng.uniform(-1, 1, (ma, na)), dtype=np.float32)
    b = np.asfortranarray(rng.uniform(-1, 1, (mb, nb)), dtype=np.float32)
    c0 = np.asfortranarray(rng.uniform(-1, 1, (m, n)), dtype=np.float32)
    c = c0.copy(order="F")
    AB.cblas_sgemm(CM, ta, tb, m, n, k, -0.75, a, ma, b, mb, 0.5, c, m)
    opa = a.astype(np.float64) if ta == 111 else a.astype(np.float64).T
    opb = b.astype(np.float64) if tb == 111 else b.astype(np.float64).T
    ref = -0.75 * (opa @ opb) + 0.5 * c0.astype(np.float64)
    tol = 4 * k * np.finfo(np.float32).eps * (np.abs(opa) @ np.abs(opb)).max()
    assert np.max(np.abs(c - ref)) <= tol


def test_trsm_trmm_golden_cases(gpu, orc, gold):
    for i in range(int(gold["counts"][1])):
        m, n, side, uplo, ta, diag, alpha = gold[f"trsm{i}"]
        m, n, side, uplo, ta, diag = map(int, (m, n, side, uplo, ta, diag))
        a = gold[f"trsm{i}_A"]
        b = np.array(gold[f"trsm{i}_B0"], order="F")
        AB.cblas_dtrsm(CM, side, uplo, ta, diag, m, n, alpha, a, a.shape[0], b, b.shape[0])
        x = gold[f"trsm{i}_X"]
        assert np.max(np.abs(b[:m, :n] - x[:m, :n])) <= 1e-12 * max(m, n), f"trsm case {i}"
        assert orc.gechkgap(b, m, n) == 0
        bm = np.array(gold[f"trsm{i}_B0"], order="F")
        AB.cblas_dtrmm(CM, side, uplo, ta, diag, m, n, alpha, a, a.shape[0], bm, bm.shape[0])
        assert np.max(np.abs(bm[:m, :n] - gold[f"trsm{i}_TB"][:m, :n])) <= 1e-12 * max(m, n), f"trmm {i}"


@pytest.mark.parametrize("side", [141, 142])
@pytest.mark.parametrize("uplo", [121, 122])
@pytest.mark.parametrize("ta", [111, 112])
def test_trsm_large_vs_oracle(gpu, orc, side, uplo, ta):
    m, n = (300, 45) if side == 141 else (45, 300)
    na = m if side == 141 else n
    a = orc.gegen(na, na, na, 17)
    orc.trddom(uplo, a, na)
    b0 = orc.gegen(m, n, m, 19)
    b = b0.copy(order="F")
    AB.cblas_dtrsm(CM, side, uplo, ta, 131, m, n, 2.0, a, na, b, m)
    x = orc.dtrsm(side, uplo, ta, 131, m, n, 2.0, a, b0.copy(order="F"))
    assert np.max(np.abs(b - x)) <= 1e-12 * max(m, n) * max(1, np.abs(x).max())


def test_trsm_row_major(gpu, orc):
    m, n = 40, 30
    a = orc.gegen(m, m, m, 3)
    orc.trddom(122, a, m)
    b = orc.uniform((m, n), 4)
    # row-major B (m x n) with ldb = n; A row-major lower
    Ar = np.ascontiguousarray(a)
    Br = np.ascontiguousarray(b)
    AB.cblas_dtrsm(RM, 141, 122, 111, 131, m, n, 1.0, Ar, m, Br, n)
    L = np.tril(a)
    np.testing.assert_allclose(L @ Br, b, rtol=1e-11, atol=1e-11)


def test_syrk_golden_cases(gpu, orc, gold):
    for i in range(int(gold["counts"][2])):
        n, k, uplo, tr, alpha, beta = gold[f"syrk{i}"]
        n, k, uplo, tr = map(int, (n, k, uplo, tr))
        a = gold[f"syrk{i}_A"]
        c = np.array(gold[f"syrk{i}_C0"], order="F")
        AB.cblas_dsyrk(CM, uplo, tr, n, k, alpha, a, a.shape[0], beta, c, c.shape[0])
        ref = gold[f"syrk{i}_C"]
        assert np.max(np.abs(c[:n, :n] - ref[:n, :n])) <= 1e-13 * max(1, k), f"syrk case {i}"
        # the other triangle is untouched
        c0 = gold[f"syrk{i}_C0"]
        mask = np.tril(np.ones((n, n), bool), -1) if uplo == 121 else np.triu(np.ones((n, n), bool), 1)
        assert np.array_equal(c[:n, :n][mask], c0[:n, :n][mask])
        assert orc.gechkgap(c, n, n) == 0


@pytest.mark.parametrize("ta,tb", [(111, 111), (111, 112), (112, 111), (112, 112)])
@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 1, 0), (31, 33, 7, 1), (32, 32, 16, 0), (33, 31, 17, 0), (64, 96, 48, 1),
                                       (96, 80, 112, 0), (700, 640, 512, 0), (700, 640, 513, 1), (513, 65, 300, 1),
                                       (1665, 1700, 529, 1), (1664, 1666, 528, 0), (250, 300, 480, 0), (250, 300, 481, 0),
                                       (250, 301, 400, 1), (250, 301, 401, 1), (1000, 1000, 60, 0), (999, 1000, 60, 1)])
def test_dgemm_few_tiles(gpu, ta, tb, m, n, k, pad):
    """Products with few output tiles (32 x 32 and 64 x 64 tiles up to K = 512, 400 or
    480 with one tile an SM or less, split K above; 128 x 64 where 128 x 128 ones leave much of the last wave idle): sizes around the tiles and the K steps, aligned and
    unaligned leading dimensions; |C - C_ref| <= (k + 3) u (|alpha||A||B| + |beta||C|)
    componentwise, doubled for the reference's own rounding."""
    rng = np.random.default_rng(m + n + k)
    mat = lambda r, c: np.asfortranarray(rng.uniform(-1, 1, (r + pad, c)))
    a, b = mat(*((m, k) if ta == 111 else (k, m))), mat(*((k, n) if tb == 111 else (n, k)))
    c0 = mat(m, n)
    opa = (a[:m] if ta == 111 else a[:k].T)
    opb = (b[:k] if tb == 111 else b[:n].T)
    for beta in (0.0, -0.5):
        c = c0.copy(order="F")
        AB.cblas_dgemm(102, ta, tb, m, n, k, 1.5, a, a.shape[0], b, b.shape[0], beta, c, c.shape[0])
        ref = 1.5 * (opa @ opb) + beta * c0[:m]
        mag = 1.5 * (np.abs(opa) @ np.abs(opb)) + abs(beta) * np.abs(c0[:m])
        assert np.all(np.abs(c[:m] - ref) <= 2 * (k + 3) * 2.0 ** -53 * mag)
        assert np.array_equal(c[m:], c0[m:])


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("m,n,k", [(1280, 1024, 1), (1281, 1087, 40), (1282, 1088, 256), (1408, 1408, 512), (1280, 1024, 514)])
@pytest.mark.parametrize("pinned", [False, True])
def test_dgemm_whole_tiles_by_bulk_copy(gpu, m, n, k, beta, pinned):
    """beta = 0 and 1, whose whole tiles leave by bulk copies that add in L2: on
    device memory, next to tiles at the edges, and on pinned host memory, which
    keeps loads and stores.  |C - C_ref| <= (k + 3) u (|A||B| + |beta||C|)
    componentwise, doubled for the reference's own rounding; the padding rows of
    C stay as they are."""
    import torch
    g = torch.Generator().manual_seed(m + k)
    ldc = m + 2 + m % 2
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64) * 2 - 1
    a, b, c0 = rnd(k, m + m % 2), rnd(n, k + k % 2), rnd(n, ldc)
    c = c0.clone().pin_memory() if pinned else c0.cuda()
    AB.atlb_dgemm_dev(111, 111, m, n, k, -1.0, a.cuda(), m + m % 2, b.cuda(), k + k % 2, beta, c, ldc)
    torch.cuda.synchronize()
    c = c.cpu()
    ref = beta * c0[:, :m] - b[:, :k] @ a[:, :m]
    mag = beta * c0[:, :m].abs() + b[:, :k].abs() @ a[:, :m].abs()
    assert bool(((c[:, :m] - ref).abs() <= 2 * (k + 3) * 2.0 ** -53 * mag).all())
    assert torch.equal(c[:, m:], c0[:, m:])


@pytest.mark.parametrize("ta,tb", [(111, 111), (111, 112), (112, 111), (112, 112)])
@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 1, 0), (63, 65, 17, 1), (64, 64, 16, 0), (65, 132, 33, 3), (128, 256, 128, 0),
                                       (500, 708, 300, 0), (1500, 1200, 40, 0), (1664, 1537, 20, 1),
                                       (4730, 300, 130, 0), (4737, 300, 130, 1), (1400, 1290, 128, 0), (1400, 1290, 129, 0)])
def test_sgemm_few_tiles(gpu, ta, tb, m, n, k, pad):
    """64 x 64 tiles (up to 111 tiles of 128 x 128, 147 up to K = 128) and the first
    sizes beyond: sizes around the tiles, aligned and unaligned columns; |C - C_ref| <=
    (k + 3) u (|alpha||A||B| + |beta||C|) componentwise with FP32's u, against
    FP64."""
    rng = np.random.default_rng(m + n + k)
    mat = lambda r, c: np.asfortranarray(rng.uniform(-1, 1, (r + pad, c)).astype(np.float32))
    a, b = mat(*((m, k) if ta == 111 else (k, m))), mat(*((k, n) if tb == 111 else (n, k)))
    c0 = mat(m, n)
    opa = (a[:m] if ta == 111 else a[:k].T).astype(np.float64)
    opb = (b[:k] if tb == 111 else b[:n].T).astype(np.float64)
    for beta in (0.0, -0.5):
        c = c0.copy(order="F")
        AB.cblas_sgemm(102, ta, tb, m, n, k, 1.5, a, a.shape[0], b, b.shape[0], beta, c, c.shape[0])
        ref = 1.5 * (opa @ opb) + beta * c0[:m]
        mag = 1.5 * (np.abs(opa) @ np.abs(opb)) + abs(beta) * np.abs(c0[:m])
        assert np.all(np.abs(c[:m] - ref) <= (k + 3) * 2.0 ** -24 * mag)
        assert np.array_equal(c[m:], c0[m:])


@pytest.mark.parametrize("uplo", [121, 122])
@pytest.mark.parametrize("n,k", [(1, 1), (33, 20), (64, 130), (200, 64), (640, 300)])
def test_dsyrk_few_tiles(gpu, uplo, n, k):
    """The triangle mask of the small tiles: the other triangle is not written."""
    rng = np.random.default_rng(n + k)
    a = np.asfortranarray(rng.uniform(-1, 1, (n, k)))
    c0 = np.asfortranarray(rng.uniform(-1, 1, (n, n)))
    c = c0.copy(order="F")
    AB.cblas_dsyrk(102, uplo, 111, n, k, -1.0, a, n, 1.0, c, n)
    part = np.triu(np.ones((n, n), bool)) if uplo == 121 else np.tril(np.ones((n, n), bool))
    mag = np.abs(a) @ np.abs(a.T) + np.abs(c0)
    assert np.all((np.abs(c - (c0 - a @ a.T)) <= 2 * (k + 3) * 2.0 ** -53 * mag)[part])
    assert np.array_equal(c[~part], c0[~part])


@pytest.mark.parametrize("m", [18944, 18945, 19100])
@pytest.mark.parametrize("n", [16, 64, 65, 100, 128, 129, 200, 256, 300])
def test_dtrsm_many_columns(gpu, n, m):
    """Solves around the number of columns from which CTAs of 32 columns and an
    order of at most 128 take over, all sides and triangles: |T X - B| <= 2 (n + 64) u
    (|T||T^-1||T||X| + |T||X|) componentwise, for the inverted 64 x 64 diagonal tiles
    and the check's own product."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + m)
    u = 2.0 ** -53
    t = (torch.rand(n, n, generator=g, dtype=torch.float64, device="cuda") * 2 - 1) / n ** 0.5
    t += 2 * torch.eye(n, dtype=torch.float64, device="cuda")
    for side in (141, 142):
        b0 = torch.rand(*((m, n) if side == 141 else (n, m)), generator=g, dtype=torch.float64, device="cuda") * 2 - 1
        for uplo in (121, 122):
            for trans in (111, 112):
                b = b0.clone()
                assert AB.atlb_dtrsm_dev(side, uplo, trans, 131, *((n, m) if side == 141 else (m, n)), 1.0, t, n, b,
                                         n if side == 141 else m) == 0
                T = torch.triu(t.T) if uplo == 121 else torch.tril(t.T)
                T = T if trans == 111 else T.T
                X, B = (b.T, b0.T) if side == 141 else (b, b0)      # T X = B or X^T T = B^T
                T = T if side == 141 else T.T
                aT, aX = T.abs(), X.abs()
                mag = aT @ (torch.linalg.inv(T).abs() @ (aT @ aX) + aX)
                assert bool(((T @ X - B).abs() <= 2 * (n + 64) * u * mag).all()), (side, uplo, trans)
