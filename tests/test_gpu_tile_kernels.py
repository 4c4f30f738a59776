"""The blocked tile kernels at the edges of their blocks: Cholesky factorisation (32-column blocks), the panel
solve of the tile Cholesky (32 rows, 4 columns), the stack QR's clusters (their size follows the load), and
compression of dense tiles by the core alone."""
import ctypes as C

import numpy as np
import pytest

from oracle import hcore_oracle as O
from tests.helpers import rel_fro

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def T():
    import torch
    assert torch.cuda.is_available()
    from hcorepp_gb300 import tiles
    return tiles


def _potrf(T, a, uplo, lda=None):
    import torch
    n = a.shape[0]
    lda = lda or n
    buf = np.full((lda, n), 7.0, order="F")
    buf[:n] = a
    d = torch.from_numpy(buf.ravel(order="F").copy()).cuda()
    info = T.Blas.potrf(uplo, n, d, lda)
    out = d.cpu().numpy().reshape((lda, n), order="F")
    assert np.all(out[n:] == 7.0)
    return info, out[:n]


@pytest.mark.parametrize("uplo", [0, 1])
@pytest.mark.parametrize("n,lda", [(1, 1), (31, 31), (32, 40), (33, 33), (64, 64), (97, 101), (300, 300)])
def test_potrf_blocks(T, n, lda, uplo):
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n + 3))
    a = g @ g.T + n * np.eye(n)
    stored = np.tril(a) + np.triu(np.full((n, n), -3.0), 1) if uplo == 0 else np.triu(a) + np.tril(np.full((n, n), -3.0), -1)
    info, out = _potrf(T, stored, uplo, lda)
    assert info == 0
    f = np.tril(out) if uplo == 0 else np.triu(out).T
    # the other triangle is not touched; |A - L L^T| <= gamma_{n+1} |L| |L|^T (Higham, Theorem 10.3)
    other = np.triu(out, 1) if uplo == 0 else np.tril(out, -1)
    assert np.array_equal(other, np.triu(stored, 1) if uplo == 0 else np.tril(stored, -1))
    assert np.all(np.abs(f @ f.T - a) <= 2 * (n + 2) * EPS * (np.abs(f) @ np.abs(f).T))


@pytest.mark.parametrize("n,bad", [(5, 0), (40, 31), (40, 32), (70, 69), (70, 40)])
def test_potrf_reports_the_first_failing_minor(T, n, bad):
    a = np.eye(n)
    a[bad, bad] = -1.0
    assert _potrf(T, a, 0)[0] == bad + 1


@pytest.mark.parametrize("nb,nt", [(33, 3), (100, 4), (64, 3)])
def test_cholesky_panel_solve_matches_the_tile_loop(T, nb, nt):
    """The batched driver and the per-tile calls give the same bits."""
    import torch
    from hcorepp_gb300 import _lib as L
    from hcorepp_gb300.problems import KernelMatrix
    km = KernelMatrix(nb * nt, nb, 3, 0.2, 2, diag_shift=1e-2)
    kinds = [[L.DENSE if i == j else L.COMPRESSED if i > j else None for j in range(nt)] for i in range(nt)]
    params = T.CompressionParameters(1e-8, truncated_svd=True)
    out = []
    for batched in (True, False):
        tm = T.TileMatrix(nt, nt, nb, kinds, nb, vt=True)
        for j in range(nt):
            for i in range(j, nt):
                d = km.tile(i, j)
                if i == j:
                    tm.set_tile(i, j, dense=d)
                else:
                    t = O.CompressedTile.from_dense(d, O.CompressionParameters(1e-8, truncated_svd=True), max_rank=nb)
                    tm.set_tile(i, j, u=t.u, v=t.v)
        assert T.tile_cholesky(tm, params, batched=batched) == 0
        torch.cuda.synchronize()
        out.append((tm.rank_grid(), np.tril(tm.to_dense())))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    a = np.block([[km.tile(i, j) for j in range(nt)] for i in range(nt)])
    assert rel_fro(out[0][1] @ out[0][1].T, a) < 1e-7


@pytest.mark.parametrize("rc,ra", [(9, 8), (60, 45), (100, 90)])
def test_results_do_not_depend_on_the_number_of_updates(T, rc, ra):
    """One update, and the same one among 3, 12, 30 and 50: the QR's clusters have 8, 8, 4, 2 and 1 CTAs."""
    import torch
    from hcorepp_gb300 import _lib as L
    rng = np.random.default_rng([rc, ra])
    n, cap = 203, rc + ra
    q = lambda r: np.linalg.qr(rng.standard_normal((n, r)))[0]
    cu, cv = q(rc), np.logspace(0, -8, rc)[:, None] * q(rc).T
    au, av, bu, bv = q(ra), np.logspace(0, -8, ra)[:, None] * q(ra).T, q(ra), q(ra).T
    params = T.CompressionParameters(1e-8, truncated_svd=True)
    p, first = params.c(), None
    for count in (1, 3, 12, 30, 50):
        a, b = T.CompressedTile(n, n, au, av, max_rank=cap), T.CompressedTile(n, n, bu, bv, max_rank=cap)
        cs = [T.CompressedTile(n, n, cu, cv, max_rank=cap) for _ in range(count)]
        ups = (L.Update * count)(*[L.Update(a.c_tile(), b.c_tile(), c.c_tile()) for c in cs])
        ctx = T.run_context()
        ctx.check(L.lib().hcgb_gemm_batch(ctx.handle, 1.0, 1.0, count, ups, C.byref(p), None))
        torch.cuda.synchronize()
        got = [(c.rank, c.u(), c.v()) for c in cs]
        first = first or got[0]
        for r, u, v in got:
            assert r == first[0]
            np.testing.assert_array_equal(u, first[1])
            np.testing.assert_array_equal(v, first[2])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("close", [False, True])
@pytest.mark.parametrize("k", [113, 114, 115, 116, 117, 118, 165, 166, 167, 168])
def test_heavy_cores_do_not_depend_on_the_team(T, k, close, mode):
    """One update, alone and among 19, 20 and 40: heavy cores run on clusters up to 19 updates and on one SM each
    beyond, at widths around half an SM's shared memory and a whole one's.  With close, groups of nearly equal
    singular values; without, a core of full rank."""
    import torch
    from hcorepp_gb300 import _lib as L
    rng = np.random.default_rng([k, close, mode])
    n, ra = 203, k // 2
    rc = k - ra
    q = lambda r: np.linalg.qr(rng.standard_normal((n, r)))[0]
    sigma = lambda r: (np.repeat(np.logspace(0, -9, (r + 4) // 5), 5)[:r] * (1.0 + 1e-7 * np.arange(r)) if close
                       else np.logspace(0, -6, r))
    cu, cv = q(rc), sigma(rc)[:, None] * q(rc).T
    au, av, bu, bv = q(ra), sigma(ra)[:, None] * q(ra).T, q(ra), q(ra).T
    p, first = T.CompressionParameters(1e-8, truncated_svd=True, mode=mode).c(), None
    for count in (1, 19, 20, 40):
        a, b = T.CompressedTile(n, n, au, av, max_rank=k), T.CompressedTile(n, n, bu, bv, max_rank=k)
        cs = [T.CompressedTile(n, n, cu, cv, max_rank=k) for _ in range(count)]
        ups = (L.Update * count)(*[L.Update(a.c_tile(), b.c_tile(), c.c_tile()) for c in cs])
        ctx = T.run_context()
        ctx.check(L.lib().hcgb_gemm_batch(ctx.handle, 1.0, 1.0, count, ups, C.byref(p), None))
        torch.cuda.synchronize()
        got = [(c.rank, c.u(), c.v()) for c in cs]
        first = first or got[0]
        for r, u, v in got:
            assert r == first[0]
            np.testing.assert_array_equal(u, first[1])
            np.testing.assert_array_equal(v, first[2])
    d = cu @ cv + au @ (av @ bu) @ bv
    # at most k dropped singular values of up to 1e-8 of the largest, and the pivoted QR's share of 1e-2 of that
    assert rel_fro(first[1] @ first[2], d) <= 1.02e-8 * np.sqrt(k)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("m,n", [(1, 1), (5, 40), (40, 5), (100, 100), (131, 90), (90, 131), (300, 257)])
def test_compression_of_rectangular_tiles(T, m, n, mode):
    rng = np.random.default_rng([m, n])
    r = min(m, n)
    d = (np.linalg.qr(rng.standard_normal((m, r)))[0] * np.logspace(0, -12, r)) @ np.linalg.qr(
        rng.standard_normal((n, r)))[0].T
    g = T.CompressedTile.from_dense(d, T.CompressionParameters(1e-8, truncated_svd=True, mode=mode), max_rank=r)
    o = O.CompressedTile.from_dense(d, O.CompressionParameters(1e-8, truncated_svd=True), max_rank=r)
    assert abs(g.rank - o.rank) <= 1
    assert rel_fro(g.to_dense(), d) <= 2 * max(rel_fro(o.to_dense(), d), 1e-14)


@pytest.mark.parametrize("k", [16, 17, 33, 128, 129, 512])
@pytest.mark.parametrize("m,n", [(16, 16), (17, 31), (129, 8), (40, 70), (300, 24)])
def test_tensor_core_products_at_tile_edges(T, m, n, k):
    """One dense update C = A B + C on the tensor cores: 56-bit operands relative to the row and column maxima
    (rounding 2^-57 each, dropped digit pairs below 2^-56), one rounding of the sum and one of beta C."""
    rng = np.random.default_rng([m, n, k])
    a = rng.standard_normal((m, k)) * 2.0 ** rng.integers(-20, 20, (m, 1))
    b = rng.standard_normal((k, n)) * 2.0 ** rng.integers(-20, 20, (1, n))
    a[0], b[:, 0] = 0.0, -np.abs(b[:, 0])
    c = rng.standard_normal((m, n))
    g = T.DenseTile(m, n, c)
    T.HCore.Gemm(1.0, T.DenseTile(m, k, a), 0, T.DenseTile(k, n, b), 0, 1.0, g, T.CompressionParameters(1e-8))
    p = a.astype(np.longdouble) @ b.astype(np.longdouble)
    scale = np.abs(a).max(1)[:, None] * np.abs(b).max(0)[None, :]
    bound = 2 * k * 2.0 ** -56 * scale * 2 + EPS * np.abs(p) + EPS * (np.abs(c) + np.abs(p))
    assert np.all(np.abs(g.to_dense() - (p + c)) <= bound)


@pytest.mark.parametrize("m,n", [(16, 16), (17, 31), (45, 45), (129, 8)])
def test_dense_products_below_2048_outputs_are_componentwise(T, m, n):
    """C = A B + C of a small dense update: each output's error is relative to its own terms (an FP64 sum of k + 1
    terms), also where the row's and the column's largest entries meet a zero."""
    rng = np.random.default_rng([m, n])
    k = 40
    a, b = rng.standard_normal((m, k)), rng.standard_normal((k, n))
    a[:, k // 2:] *= 2.0 ** -80
    b[:k // 2] = 0.0
    c = rng.standard_normal((m, n)) * 2.0 ** -80
    g = T.DenseTile(m, n, c)
    T.HCore.Gemm(1.0, T.DenseTile(m, k, a), 0, T.DenseTile(k, n, b), 0, 1.0, g, T.CompressionParameters(1e-8))
    p = a.astype(np.longdouble) @ b.astype(np.longdouble) + c
    bound = (k + 2) * EPS * (np.abs(a) @ np.abs(b) + np.abs(c))
    assert np.all(np.abs(g.to_dense() - p) <= bound)


@pytest.mark.parametrize("uplo", [0, 1])
@pytest.mark.parametrize("n,bad", [(20, 7), (70, 0), (300, 31), (300, 32), (300, 45), (300, 150), (300, 299)])
def test_potrf_stops_at_the_failing_column(T, n, bad, uplo):
    """A matrix whose leading minor of order bad + 1 is not positive: the columns before are those of the factor, the
    rest is as given, in every run alike."""
    rng = np.random.default_rng([n, bad])
    g = rng.standard_normal((n, n + 3))
    a = g @ g.T + n * np.eye(n)
    a[bad, bad] = -1.0
    stored = np.tril(a) if uplo == 0 else np.triu(a)
    first = None
    for _ in range(4):
        info, out = _potrf(T, stored, uplo)
        assert info == bad + 1
        first = out if first is None else first
        np.testing.assert_array_equal(out, first)
    f = np.tril(first) if uplo == 0 else np.triu(first).T
    np.testing.assert_array_equal(f[:, bad:], np.tril(a)[:, bad:])
    l = f[:, :bad]
    low = np.tril(np.ones((n, bad), dtype=bool))
    err = np.abs(l @ l[:bad].T - a[:, :bad])
    assert np.all(err[low] <= 2 * (n + 2) * EPS * (np.abs(l) @ np.abs(l[:bad]).T)[low])


def test_potrf_of_a_large_matrix_stops_at_the_failing_column(T):
    """Beyond the copy that a context keeps (64 MiB): the same after a failure, and no memory is held afterwards."""
    import torch
    n, bad = 3100, 2500
    a = np.eye(n) * 4.0 + 1.0
    a[bad, bad] = -5.0
    _potrf(T, np.eye(8), 0)
    torch.cuda.synchronize()
    info, out = _potrf(T, np.tril(a), 0)
    assert info == bad + 1
    np.testing.assert_array_equal(out[:, bad:], np.tril(a)[:, bad:])
    l = np.tril(out[:, :bad])
    low = np.tril(np.ones((n, bad), dtype=bool))
    err = np.abs(l @ l[:bad].T - a[:, :bad])
    assert np.all(err[low] <= 2 * (n + 2) * EPS * (np.abs(l) @ np.abs(l[:bad]).T)[low])
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    _potrf(T, np.tril(a), 0)
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] >= free - (16 << 20)
