"""Parity of the GPU LAPACK path with the oracle (the restatement of ATLAS's
recursive getrf/potrf and blocked geqrf): ipiv identical, factors within
rounding, the reference testers' residuals (bin/lutst.c, bin/llttst.c,
bin/qrtst.c, bin/slvtst.c: <= 100), info codes for singular / indefinite
inputs, and lda gaps untouched -- all through the drop-in C ABI."""
import numpy as np
import pytest

import atlas_b200 as AB
from oracle import oracle as O

pytestmark = pytest.mark.gpu
CM, RM = AB.CblasColMajor, AB.CblasRowMajor


def _getrf_gpu(a, m, n, order=CM):
    ipiv = np.zeros(max(min(m, n), 1), dtype=np.int32)
    info = AB.clapack_dgetrf(order, m, n, a, a.shape[0] if order == CM else a.shape[1], ipiv)
    return ipiv[:min(m, n)], info


@pytest.mark.parametrize("m,n", [(1, 1), (2, 2), (5, 5), (31, 31), (32, 32), (33, 33), (100, 100),
                                 (257, 257), (600, 600), (700, 300), (300, 700), (1500, 40)])
def test_getrf_vs_oracle_gegen(gpu, orc, m, n):
    lda = m + 3
    a0 = orc.gegen(m, n, lda, m * n + lda)           # the lutst input (random pivots)
    a = a0.copy(order="F")
    ipiv, info = _getrf_gpu(a, m, n)
    ref, rpiv, rinfo = orc.dgetrf(a0.copy(order="F"), m, n)
    assert info == rinfo == 0
    np.testing.assert_array_equal(ipiv, rpiv)
    assert np.max(np.abs(a[:m, :n] - ref[:m, :n])) <= 1e-9
    assert orc.resid_lu(a0[:m, :n].copy(order="F"), a[:m, :n].copy(order="F"), ipiv) <= 100.0
    assert orc.gechkgap(a, m, n) == 0


@pytest.mark.parametrize("n", [64, 513, 1024])
def test_getrf_benchmark_matrix_identity_pivots(gpu, orc, n):
    a0 = orc.lu_matrix(n, 42)
    a = a0.copy(order="F")
    ipiv, info = _getrf_gpu(a, n, n)
    ref, rpiv, _ = orc.dgetrf(a0.copy(order="F"))
    assert info == 0
    np.testing.assert_array_equal(ipiv, rpiv)
    np.testing.assert_array_equal(ipiv, np.arange(n))
    assert orc.resid_lu(a0, a, ipiv) <= 100.0


def test_getrf_singular_info(gpu, orc):
    for col in (0, 6, 39):
        a0 = orc.lu_matrix(40, 5)
        a0[:, col] = 0.0
        a = a0.copy(order="F")
        ipiv, info = _getrf_gpu(a, 40, 40)
        _, rpiv, rinfo = orc.dgetrf(a0.copy(order="F"))
        assert info == rinfo == col + 1
        np.testing.assert_array_equal(ipiv, rpiv)


def test_getrf_row_major(gpu, orc):
    m, n = 60, 45
    a = orc.gegen(m, n, m, 77)[:m, :n]
    R = np.ascontiguousarray(a)              # row-major M x N, lda = N
    ipiv = np.zeros(min(m, n), dtype=np.int32)
    info = AB.clapack_dgetrf(RM, m, n, R, n, ipiv)
    assert info == 0
    # row-major A = L U P (unit U) == column-major factorization of A^T
    ref, rpiv, _ = orc.dgetrf(np.asfortranarray(a.T))
    np.testing.assert_array_equal(ipiv, rpiv)
    np.testing.assert_allclose(R.T, ref, rtol=1e-10, atol=1e-10)


@pytest.mark.parametrize("trans", [111, 112])
def test_getrs_and_gesv(gpu, orc, trans):
    n, r = 400, 5
    a0 = orc.gegen(n, n, n, 9)
    xt = orc.uniform((n, r), 10)
    b = (a0 if trans == 111 else a0.T) @ xt
    lu = a0.copy(order="F")
    ipiv, info = _getrf_gpu(lu, n, n)
    x = np.array(b, order="F")
    assert AB.clapack_dgetrs(CM, trans, n, r, lu, n, ipiv, x, n) == 0
    A = a0 if trans == 111 else np.asfortranarray(a0.T)
    assert orc.resid_slv(A, x, xt) <= 100.0
    # gesv: A overwritten with its factors, B with the solution
    a = a0.copy(order="F")
    x2 = np.array(a0 @ xt, order="F")
    ip2 = np.zeros(n, dtype=np.int32)
    assert AB.clapack_dgesv(CM, n, r, a, n, ip2, x2, n) == 0
    np.testing.assert_array_equal(ip2, ipiv)
    assert orc.resid_slv(a0, x2, xt) <= 100.0


def test_gesv_row_major(gpu, orc):
    n, r = 200, 3
    a = orc.gegen(n, n, n, 12)
    xt = orc.uniform((n, r), 13)
    rhs = a @ xt                              # each RHS is a column of a @ xt
    Ar = np.ascontiguousarray(a)
    Br = np.asfortranarray(rhs)               # row-major NRHS x N storage == column-major N x NRHS
    ip = np.zeros(n, dtype=np.int32)
    assert AB.clapack_dgesv(RM, n, r, Ar, n, ip, Br, n) == 0
    assert orc.resid_slv(np.asfortranarray(a), Br, xt) <= 100.0


@pytest.mark.parametrize("uplo", [121, 122])
@pytest.mark.parametrize("n", [1, 4, 5, 63, 64, 65, 200, 700])
def test_potrf_vs_oracle(gpu, orc, uplo, n):
    a0 = orc.spd_matrix(n, 3 + n)
    lda = n + 2
    a = np.zeros((lda, n), order="F")
    a[:n] = a0
    a[n:] = -2560000000.0  # ATL_gegen FILLCONST in the lda gap
    assert AB.clapack_dpotrf(CM, uplo, n, a, lda) == 0
    f = a0.copy(order="F")
    assert orc.dpotrf(uplo, f) == 0
    tri = np.tril if uplo == 122 else np.triu
    assert np.max(np.abs(tri(a[:n]) - tri(f))) <= 1e-11
    assert orc.resid_llt(uplo, a0, a[:n].copy(order="F")) <= 100.0
    assert orc.gechkgap(a, n, n) == 0
    # the other triangle is not touched
    other = np.triu(np.ones((n, n), bool), 1) if uplo == 122 else np.tril(np.ones((n, n), bool), -1)
    assert np.array_equal(a[:n][other], a0[other])


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 100])
@pytest.mark.parametrize("m", [1, 16, 17, 33, 127, 128, 129, 255, 256, 257, 300])
def test_getrf_panels_of_one_cta(gpu, m, n):
    """LU of few rows, whose panels one CTA factors: |PA - LU| <= gamma |L||U|
    componentwise with gamma = min(m, n) u, doubled for the product's own
    rounding; multipliers of at most 1; a zero column in each half of a panel is
    reported and the factorization completes."""
    rng = np.random.default_rng(m * 1000 + n)
    mn, u = min(m, n), 2.0 ** -53
    for zero in ((), (mn // 2,), (mn - 1, mn // 3)):
        a0 = np.asfortranarray(rng.uniform(-1, 1, (m + 1, n)))
        a0[:, list(zero)] = 0.0
        a, ipiv = a0.copy(order="F"), np.full(mn, -1, dtype=np.int32)
        info = AB.clapack_dgetrf(CM, m, n, a, m + 1, ipiv)
        assert info == (min(zero) + 1 if zero else 0)
        assert np.array_equal(a[m], a0[m])
        p = a0[:m].copy()
        for k in range(mn):
            assert k <= ipiv[k] < m
            p[[k, ipiv[k]]] = p[[ipiv[k], k]]
        low, up = np.tril(a[:m, :mn], -1) + np.eye(m, mn), np.triu(a[:mn])
        assert np.max(np.abs(low)) <= 1.0
        assert np.all(np.abs(p - low @ up) <= 2 * (mn + 1) * u * (np.abs(low) @ np.abs(up)))


@pytest.mark.parametrize("m,n,nb", [(193, 193, 192), (300, 300, 192), (500, 500, 192), (400, 1100, 192),
                                    (250, 1000, 64), (500, 500, 256), (300, 1000, 256)])
def test_getrf_of_ill_conditioned_multipliers(gpu, m, n, nb):
    """A = L U with every multiplier the same: the diagonal tiles of L11 are then
    far worse conditioned than the matrix, and |PA - LU| <= gamma |L||U| has to
    hold all the same, through the U12 solve between block columns of nb.  gamma =
    (m + 2) u (Higham, theorem 9.3, with multipliers by the reciprocal pivot) and m u
    for the check's own product."""
    rng = np.random.default_rng(m + n)
    u = 2.0 ** -53
    old = AB.atlb_tune_get("getrf_nb")
    try:
        assert AB.atlb_tune_set("getrf_nb", nb) == nb
        for mult in (-0.5, -0.9, -1.0):
            low = np.eye(m) + mult * np.tril(np.ones((m, m)), -1)
            up = np.triu(rng.uniform(-1, 1, (m, n)))
            up[np.arange(m), np.arange(m)] = 1.0
            a0 = np.asfortranarray(low @ up)
            a = a0.copy(order="F")
            ipiv, info = _getrf_gpu(a, m, n)
            assert info == 0
            for k in range(m):
                a0[[k, ipiv[k]]] = a0[[ipiv[k], k]]
            low, up = np.tril(a[:, :m], -1) + np.eye(m), np.triu(a)
            assert np.max(np.abs(low)) <= 1.0
            assert np.all(np.abs(a0 - low @ up) <= 2 * (m + 1) * u * (np.abs(low) @ np.abs(up))), mult
    finally:
        AB.atlb_tune_set("getrf_nb", old)


@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 256, 257, 300, 520])
def test_few_rhs_solves_at_block_edges(gpu, n, nrhs):
    """potrs and getrs across the right-hand sides one launch takes and the
    128-row blocks: each solve's residual <= gamma |L||U||x| componentwise, with
    gamma = 4 (n + 128) u for the inverted 128 x 128 diagonal blocks times their
    largest condition number here (diagonally dominant factors: < 8)."""
    rng = np.random.default_rng(n * 100 + nrhs)
    u, ldb = 2.0 ** -53, n + 3
    g = rng.uniform(-1, 1, (n, n))
    sym = np.asfortranarray(g @ g.T / n + 4 * np.eye(n))
    gen = np.asfortranarray(g / np.sqrt(n) + 4 * np.eye(n))
    b0 = np.full((ldb, nrhs), 3.0, order="F")
    b0[:n] = rng.uniform(-1, 1, (n, nrhs))
    for uplo in (121, 122):
        f = sym.copy(order="F")
        b = b0.copy(order="F")
        assert AB.clapack_dpotrf(CM, uplo, n, f, n) == 0
        assert AB.clapack_dpotrs(CM, uplo, n, nrhs, f, n, b, ldb) == 0
        low = np.abs(np.tril(f) if uplo == 122 else np.triu(f).T)
        assert np.array_equal(b[n:], b0[n:])
        bound = 8 * 4 * (n + 128) * u * (low @ (low.T @ np.abs(b[:n])))
        assert np.all(np.abs(sym @ b[:n] - b0[:n]) <= bound)
    lu = gen.copy(order="F")
    ipiv = np.zeros(n, dtype=np.int32)
    assert AB.clapack_dgetrf(CM, n, n, lu, n, ipiv) == 0
    low, up = np.abs(np.tril(lu, -1) + np.eye(n)), np.abs(np.triu(lu))
    perm = np.arange(n)
    for k in range(n):
        perm[[k, ipiv[k]]] = perm[[ipiv[k], k]]
    for trans in (111, 112):
        b = b0.copy(order="F")
        assert AB.clapack_dgetrs(CM, trans, n, nrhs, lu, n, ipiv, b, ldb) == 0
        assert np.array_equal(b[n:], b0[n:])
        x = np.abs(b[:n])
        if trans == 111:
            mag = np.zeros_like(x)
            mag[perm] = low @ (up @ x)
            res = np.abs(gen @ b[:n] - b0[:n])
        else:
            mag, res = up.T @ (low.T @ x[perm]), np.abs(gen.T @ b[:n] - b0[:n])
        assert np.all(res <= 8 * 4 * (n + 128) * u * mag)


@pytest.mark.parametrize("uplo", [121, 122])
@pytest.mark.parametrize("n,bad", [(1, 0), (15, 0), (16, 0), (17, 17), (129, 0), (240, 200), (255, 0), (256, 0),
                                   (256, 241), (256, 256), (257, 0)])
def test_potrf_one_launch_orders(gpu, uplo, n, bad):
    """Orders around the tiles of the one-launch factorization, and a negative
    minor in the first, middle and last tile.  |A - L L^T| <= (n + 1) u |L||L^T|
    componentwise (Higham, theorem 10.3), doubled for the reciprocal diagonal;
    the other triangle and the rows below the matrix are not written."""
    rng = np.random.default_rng(n + bad)
    lda = n + 2
    g = rng.standard_normal((n, n))
    sym = g @ g.T + n * np.eye(n)
    if bad:
        sym[bad - 1, bad - 1] = -1.0
    a = np.full((lda, n), 5.0, order="F")
    a[:n] = sym
    a0 = a.copy(order="F")
    assert AB.clapack_dpotrf(CM, uplo, n, a, lda) == bad
    assert np.array_equal(a[n:], a0[n:])
    other = np.triu(np.ones((n, n), bool), 1) if uplo == 122 else np.tril(np.ones((n, n), bool), -1)
    assert np.array_equal(a[:n][other], a0[:n][other])
    if not bad:
        low = np.tril(a[:n]) if uplo == 122 else np.triu(a[:n]).T
        assert np.all(np.abs(low @ low.T - sym) <= 2 * (n + 2) * 2.0 ** -53 * (np.abs(low) @ np.abs(low.T)))


@pytest.mark.parametrize("bad", [0, 37, 64, 150])
def test_potrf_not_spd_info(gpu, orc, bad):
    n = 200
    a0 = orc.spd_matrix(n, 8)
    a0[bad, bad] = -5.0
    a = a0.copy(order="F")
    info = AB.clapack_dpotrf(CM, 122, n, a, n)
    rinfo = orc.dpotrf(122, a0.copy(order="F"))
    assert info == rinfo == bad + 1


@pytest.mark.parametrize("uplo", [121, 122])
@pytest.mark.parametrize("r", [13, 32, 40])
def test_potrs_many_rhs(gpu, orc, uplo, r):
    """13 and 32 right-hand sides take the one-launch solves in chunks of 8
    columns, 40 the recursive TRSM: the same solution either way."""
    n = 700
    a0 = orc.spd_matrix(n, 31)
    xt = orc.uniform((n, r), 32)
    f = a0.copy(order="F")
    assert AB.clapack_dpotrf(CM, uplo, n, f, n) == 0
    x = np.array(a0 @ xt, order="F")
    assert AB.clapack_dpotrs(CM, uplo, n, r, f, n, x, n) == 0
    assert orc.resid_slv(a0, x, xt) <= 100.0
    np.testing.assert_allclose(x, xt, rtol=1e-9, atol=1e-9)


@pytest.mark.parametrize("uplo", [121, 122])
def test_potrs_posv(gpu, orc, uplo):
    n, r = 300, 4
    a0 = orc.spd_matrix(n, 21)
    xt = orc.uniform((n, r), 22)
    a = a0.copy(order="F")
    x = np.array(a0 @ xt, order="F")
    assert AB.clapack_dposv(CM, uplo, n, r, a, n, x, n) == 0
    assert orc.resid_slv(a0, x, xt) <= 100.0
    x2 = np.array(a0 @ xt, order="F")
    assert AB.clapack_dpotrs(CM, uplo, n, r, a, n, x2, n) == 0
    np.testing.assert_allclose(x2, x, rtol=1e-12, atol=1e-12)
    # row-major Upper == column-major Lower on the same buffer
    ar = a0.copy(order="F")
    assert AB.clapack_dpotrf(RM, 121 if uplo == 122 else 122, n, ar, n) == 0
    tri = np.tril if uplo == 122 else np.triu
    np.testing.assert_allclose(tri(ar), tri(a), rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("m,n", [(1, 1), (5, 3), (3, 5), (64, 64), (100, 37), (300, 200), (200, 300),
                                 (1000, 130), (700, 700)])
def test_geqrf_vs_oracle(gpu, orc, m, n):
    a0 = orc.normal((m, n), 5 * m + n)
    lda = m + 1
    a = np.full((lda, n), -2560000000.0, order="F")
    a[:m] = a0
    tau = np.zeros(min(m, n))
    assert AB.clapack_dgeqrf(CM, m, n, a, lda, tau) == 0
    qr, rtau = orc.dgeqrf(a0.copy(order="F"))
    k = min(m, n)
    np.testing.assert_allclose(tau, rtau, rtol=1e-9, atol=1e-11)
    np.testing.assert_allclose(np.triu(a[:m]), np.triu(qr), rtol=1e-9, atol=1e-10)
    np.testing.assert_allclose(np.tril(a[:m], -1), np.tril(qr, -1), rtol=1e-8, atol=1e-10)
    assert orc.resid_qr(a0, a[:m].copy(order="F"), tau) <= 100.0
    assert orc.gechkgap(a, m, n) == 0
    assert np.all((tau == 0) | ((tau >= 1) & (tau <= 2)))


def test_geqrf_row_major_is_lq_of_the_view(gpu, orc):
    m, n = 90, 60
    a = orc.normal((m, n), 31)
    R = np.ascontiguousarray(a)               # row-major M x N
    tau = np.zeros(min(m, n))
    assert AB.clapack_dgeqrf(RM, m, n, R, n, tau) == 0
    qr, rtau = orc.dgeqrf(np.asfortranarray(a))
    np.testing.assert_allclose(tau, rtau, rtol=1e-9, atol=1e-11)
    np.testing.assert_allclose(R, qr, rtol=1e-8, atol=1e-10)


def test_device_api_getrf_potrf(gpu, orc):
    import torch
    n = 256
    a0 = orc.lu_matrix(n, 3)
    A = torch.tensor(a0.T.copy(), device="cuda")   # storage == column-major a0
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert AB.atlb_dgetrf_dev(n, n, A, n, ipiv, info) == 0
    AB.atlb_sync()
    ref, rpiv, _ = orc.dgetrf(a0.copy(order="F"))
    assert int(info.item()) == 0
    np.testing.assert_array_equal(ipiv.cpu().numpy(), rpiv)
    np.testing.assert_allclose(A.cpu().numpy().T, ref, rtol=1e-10, atol=1e-10)


# ------------------------------------------------- pinned to the reference's own LAPACK
import golden_lapack as GL  # noqa: E402


def test_getrf_vs_reference_lapack_golden(gpu):
    """ipiv and info identical to the reference's ATL_getrf (getrfC / getrfR) on
    the testers' sizes, ties in the pivot search, zero columns, row-major and
    1 x n / m x 1 edges; the factors agree to rounding."""
    for i, a, order, lu_ref, ipiv_ref, info_ref in GL.getrf_cases():
        m, n = a.shape
        ipiv = np.zeros(max(min(m, n), 1), dtype=np.int32)
        if order == RM:
            buf = np.ascontiguousarray(a)
            info = AB.clapack_dgetrf(RM, m, n, buf, max(n, 1), ipiv)
            lu = buf
        else:
            lu = a.copy(order="F")
            info = AB.clapack_dgetrf(CM, m, n, lu, max(m, 1), ipiv)
        assert info == info_ref, f"getrf case {i}"
        np.testing.assert_array_equal(ipiv[:min(m, n)], ipiv_ref, err_msg=f"getrf case {i}")
        assert GL.close(lu, lu_ref, 1e-10), f"getrf case {i}"


def test_getrs_vs_reference_lapack_golden(gpu):
    cases = GL.getrf_cases()
    for i, fi, trans, b, x_ref in GL.getrs_cases():
        _, _, _, lu, ipiv, _ = cases[fi]
        n = lu.shape[0]
        x = np.array(b, order="F")
        lu = np.asfortranarray(lu)
        AB.clapack_dgetrs(CM, trans, n, x.shape[1], lu, n, np.ascontiguousarray(ipiv, np.int32), x, n)
        assert GL.close(x, x_ref, 1e-9), f"getrs case {i}"


def test_potrf_potrs_vs_reference_lapack_golden(gpu):
    facs = []
    for i, a, uplo, f_ref, info_ref in GL.potrf_cases():
        n = a.shape[0]
        f = a.copy(order="F")
        info = AB.clapack_dpotrf(CM, uplo, n, f, n)
        facs.append((f, uplo))
        assert info == info_ref, f"potrf case {i}"
        k = n if info == 0 else info - 1
        assert GL.close(GL.tri(f, uplo)[:k, :k], f_ref[:k, :k], 1e-11), f"potrf case {i}"
    for i, fi, b, x_ref in GL.potrs_cases():
        f, uplo = facs[fi]
        n = f.shape[0]
        x = np.array(b, order="F")
        AB.clapack_dpotrs(CM, uplo, n, x.shape[1], f, n, x, n)
        assert GL.close(x, x_ref, 1e-9), f"potrs case {i}"


def test_geqrf_vs_reference_lapack_golden(gpu):
    """R, the Householder vectors and tau of the reference's ATL_geqrf
    (ATLAS's larfg sign and tau conventions)."""
    for i, a, qr_ref, tau_ref, info_ref in GL.geqrf_cases():
        m, n = a.shape
        qr = a.copy(order="F")
        tau = np.zeros(max(min(m, n), 1))
        info = AB.clapack_dgeqrf(CM, m, n, qr, max(m, 1), tau)
        assert info == info_ref == 0, f"geqrf case {i}"
        assert GL.close(qr, qr_ref, 1e-10), f"geqrf case {i}"
        assert GL.close(tau[:min(m, n)], tau_ref, 1e-10), f"geqrf case {i}"


@pytest.mark.parametrize("m,n", [(300, 900), (900, 300), (257, 385), (129, 129), (640, 129)])
def test_geqrf_lookahead_shapes_vs_oracle(gpu, orc, m, n):
    """Wide, tall and ragged shapes through the look-ahead driver: the last
    panel narrower than the others, a wide matrix whose columns beyond
    min(m, n) get only the block reflectors, a single extra column."""
    a0 = orc.normal((m, n), 3 * m + n)
    a = a0.copy(order="F")
    tau = np.zeros(min(m, n))
    assert AB.clapack_dgeqrf(CM, m, n, a, m, tau) == 0
    qr, rtau = orc.dgeqrf(a0.copy(order="F"))
    np.testing.assert_allclose(tau, rtau, rtol=1e-9, atol=1e-11)
    np.testing.assert_allclose(np.triu(a), np.triu(qr), rtol=1e-9, atol=1e-10)
    np.testing.assert_allclose(np.tril(a, -1), np.tril(qr, -1), rtol=1e-8, atol=1e-10)
    assert orc.resid_qr(a0, a.copy(order="F"), tau) <= 100.0


@pytest.mark.parametrize("m,n", [(300, 70), (2048, 70), (2049, 70), (4097, 33), (8193, 40), (16384, 20),
                                 (16385, 20), (40000, 10)])
def test_geqrf_panel_rows_and_reflectors_that_vanish(gpu, orc, m, n):
    """Rows around the limits of a panel's CTAs and of its rows a thread; random
    columns, zero columns at the start, in the middle and at the end of a leaf, and
    leading columns that are triangular already: tau = 0 there, R, V and tau the
    oracle's, and |A - QR| <= m n u |A| (Higham, theorem 19.4)."""
    for kind in ("random", "zero", "triangular"):
        a0 = orc.normal((m, n), 5 * m + n)
        if kind == "zero":
            a0[:, [c for c in (0, 7, 15, 16, 31, 32, 47, n - 1) if c < n]] = 0.0
        if kind == "triangular":
            a0[:, :n // 2] = np.triu(a0[:, :n // 2])
        a = a0.copy(order="F")
        tau = np.zeros(n)
        assert AB.clapack_dgeqrf(CM, m, n, a, m, tau) == 0
        qr, rtau = orc.dgeqrf(a0.copy(order="F"))
        np.testing.assert_array_equal(tau == 0.0, rtau == 0.0)
        np.testing.assert_allclose(tau, rtau, rtol=1e-9, atol=1e-11)
        np.testing.assert_allclose(np.triu(a), np.triu(qr), rtol=1e-9, atol=1e-10)
        np.testing.assert_allclose(np.tril(a, -1), np.tril(qr, -1), rtol=1e-8, atol=1e-10)
        back = np.triu(a)
        for c in range(n - 1, -1, -1):
            v = np.concatenate([[1.0], a[c + 1:, c]])
            back[c:] -= tau[c] * np.outer(v, v @ back[c:])
        assert np.linalg.norm(back - a0) <= m * n * 2.0 ** -53 * np.linalg.norm(a0)


@pytest.mark.parametrize("n", [129, 300, 513])
@pytest.mark.parametrize("uplo", [121, 122])
def test_potrf_lookahead_sizes_vs_oracle(gpu, orc, n, uplo):
    """Orders just past one, two and four 128-column blocks through the
    Cholesky look-ahead (the last block narrow), both triangles."""
    a0 = orc.spd_matrix(n, 7 * n)
    a = a0.copy(order="F")
    assert AB.clapack_dpotrf(CM, uplo, n, a, n) == 0
    f = a0.copy(order="F")
    assert orc.dpotrf(uplo, f) == 0
    tri = np.triu if uplo == 121 else np.tril
    np.testing.assert_allclose(tri(a), tri(f), rtol=1e-10, atol=1e-11)


@pytest.mark.parametrize("nb", [64, 256])
@pytest.mark.parametrize("la", [0, 1])
def test_geqrf_panel_widths_vs_oracle(gpu, orc, nb, la):
    """qr_nb = 256 factors each panel as two 128-column halves (the left
    half's block reflector applied to the right half in between, T built
    from the two halves' T); with and without look-ahead the result matches
    the oracle as with the default width, and so does Q applied by dormqr."""
    m, n = 1100, 700
    a0 = orc.normal((m, n), 97)
    try:
        assert AB.atlb_tune_set("qr_nb", nb) == nb
        assert AB.atlb_tune_set("lookahead", la) == la
        a = a0.copy(order="F")
        tau = np.zeros(n)
        assert AB.clapack_dgeqrf(CM, m, n, a, m, tau) == 0
        qr, rtau = orc.dgeqrf(a0.copy(order="F"))
        np.testing.assert_allclose(tau, rtau, rtol=1e-9, atol=1e-11)
        np.testing.assert_allclose(np.triu(a), np.triu(qr), rtol=1e-9, atol=1e-10)
        np.testing.assert_allclose(np.tril(a, -1), np.tril(qr, -1), rtol=1e-8, atol=1e-10)
        assert orc.resid_qr(a0, a.copy(order="F"), tau) <= 100.0
        # Q^T A = R through the blocked apply at the same width
        c = a0.copy(order="F")
        assert AB.ATL_dormqr(AB.CblasLeft, AB.CblasTrans, m, n, n, a, m, tau, c, m, None, 0) == 0
        r = np.triu(a)[:n]
        np.testing.assert_allclose(c[:n], r, rtol=1e-9, atol=1e-9 * np.abs(r).max())
        assert np.abs(c[n:]).max() <= 1e-9 * np.abs(r).max()
    finally:
        AB.atlb_tune_set("qr_nb", 128)
        AB.atlb_tune_set("lookahead", 1)


def _ok(result):
    assert result[0] == 0, result[0]
    return result[1] if len(result) > 1 else None


@pytest.mark.parametrize("kind", ["getrf", "potrf"])
def test_replayed_factorizations_follow_the_memory_behind_an_address(gpu, kind):
    """The factorizations' graphs are kept by address.  Here the same address is
    device memory for the calls that record and replay one, and host memory for
    the call after: the updates are then not those that add in the device's own L2.
    |PA - LU| or |A - LL^T| <= gamma |L||U| with gamma = (n + 2) u, doubled for the
    check's own product."""
    import torch
    from cuda.bindings import driver as d
    from cuda.bindings import runtime as rt
    dev = _ok(d.cuDeviceGet(0))
    host_vmm = d.CUdevice_attribute.CU_DEVICE_ATTRIBUTE_HOST_NUMA_VIRTUAL_MEMORY_MANAGEMENT_SUPPORTED
    if not _ok(d.cuDeviceGetAttribute(host_vmm, dev)):
        pytest.skip("no host memory in the driver's virtual memory management here")
    numa = _ok(d.cuDeviceGetAttribute(d.CUdevice_attribute.CU_DEVICE_ATTRIBUTE_HOST_NUMA_ID, dev))
    n, u = 1536, 2.0 ** -53
    rng = np.random.default_rng(9)
    a0 = rng.uniform(-1, 1, (n, n))
    if kind == "potrf":
        a0 = a0 @ a0.T + n * np.eye(n)
    src = torch.tensor(np.ascontiguousarray(a0.T), device="cuda")
    out, ipiv, info = torch.empty_like(src), torch.zeros(n, dtype=torch.int32, device="cuda"), \
        torch.zeros(1, dtype=torch.int32, device="cuda")

    loc = d.CUmemLocation()
    access = d.CUmemAccessDesc()
    access.location.type = d.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
    access.location.id = 0
    access.flags = d.CUmemAccess_flags.CU_MEM_ACCESS_FLAGS_PROT_READWRITE
    size, addr = 0, None

    def memory(where, index):
        nonlocal size, addr
        prop = d.CUmemAllocationProp()
        prop.type = d.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
        loc.type, loc.id = where, index
        prop.location = loc
        gran = _ok(d.cuMemGetAllocationGranularity(
            prop, d.CUmemAllocationGranularity_flags.CU_MEM_ALLOC_GRANULARITY_RECOMMENDED))
        if addr is None:
            size = (8 * n * n + gran - 1) // gran * gran
            addr = _ok(d.cuMemAddressReserve(size, 0, 0, 0))
        assert size % gran == 0
        return _ok(d.cuMemCreate(size, prop, 0))

    def factor():
        st = torch.cuda.current_stream().cuda_stream
        _ok(d.cuMemcpyAsync(addr, src.data_ptr(), 8 * n * n, st))
        if kind == "getrf":
            assert AB.atlb_dgetrf_dev(n, n, int(addr), n, ipiv, info) == 0
        else:
            assert AB.atlb_dpotrf_dev(122, n, int(addr), n, info) == 0
        _ok(d.cuMemcpyAsync(out.data_ptr(), addr, 8 * n * n, st))
        assert AB.atlb_sync() == 0 and int(info.item()) == 0
        f = out.cpu().numpy().T
        if kind == "getrf":
            want = a0.copy()
            for k, p in enumerate(ipiv.cpu().numpy()):
                want[[k, p]] = want[[p, k]]
            low, up = np.tril(f, -1) + np.eye(n), np.triu(f)
        else:
            want, low = a0, np.tril(f)
            up = low.T
        assert np.all(np.abs(want - low @ up) <= 2 * (n + 2) * u * (np.abs(low) @ np.abs(up)))

    for where, index, calls in ((d.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE, 0, 3),
                                (d.CUmemLocationType.CU_MEM_LOCATION_TYPE_HOST_NUMA, numa, 1)):
        handle = memory(where, index)
        _ok(d.cuMemMap(addr, size, 0, handle, 0))
        _ok(d.cuMemSetAccess(addr, size, [access], 1))
        own = _ok(rt.cudaPointerGetAttributes(int(addr))).type == rt.cudaMemoryType.cudaMemoryTypeDevice
        device = where == d.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
        if own == device:
            for _ in range(calls):
                factor()
        _ok(d.cuMemUnmap(addr, size))
        _ok(d.cuMemRelease(handle))
        assert own == device
    _ok(d.cuMemAddressFree(addr, size))


def test_a_wait_that_gave_up_is_reported_by_the_next_synchronization(gpu, orc):
    """The word that a kernel sets, set here: the synchronising call after it returns
    cudaErrorLaunchTimeout, unless it has an info value to return, and clears it."""
    import ctypes
    timeout = 702
    word = ctypes.cast(AB.atlb_wait_word(), ctypes.POINTER(ctypes.c_int))
    assert word[0] == 0 and AB.atlb_sync() == 0
    n = 40
    a, tau, ipiv = orc.lu_matrix(n, 3), np.zeros(n), np.zeros(n, dtype=np.int32)
    b = np.asfortranarray(np.ones((n, 1)))
    singular = np.zeros((n, n), order="F")
    calls = [(AB.atlb_sync, timeout),
             (lambda: AB.ATL_dgeqrf(n, n, a.copy(order="F"), n, tau, None, 0), timeout),
             (lambda: AB.clapack_dgesv(CM, n, 1, a.copy(order="F"), n, ipiv, b.copy(order="F"), n), timeout),
             (lambda: AB.clapack_dpotrf(CM, 122, n, np.asfortranarray(np.eye(n)), n), timeout),
             (lambda: AB.clapack_dgetrf(CM, n, n, singular, n, ipiv), 1)]
    for call, want in calls:
        word[0] = 1
        assert call() == want
        assert word[0] == 0 and AB.atlb_last_cuda_error() == timeout
        assert AB.atlb_sync() == 0
