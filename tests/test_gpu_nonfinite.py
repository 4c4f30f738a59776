"""Inputs with a NaN or an infinity: a compressed result is a rank-1 tile of NaN, whatever the core's width and
form, and the other tiles of the batch do not notice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import torch
    assert torch.cuda.is_available()
    from hcorepp_gb300 import tiles
    return tiles


def _tile(rng, m, n):
    r = min(m, n)
    return (np.linalg.qr(rng.standard_normal((m, r)))[0] * np.logspace(0, -4, r)) @ np.linalg.qr(
        rng.standard_normal((n, r)))[0].T


def _compress(T, tiles, mode):
    import torch
    m, n = tiles[0].shape
    out = [T.CompressedTile(m, n, rank=0, max_rank=min(m, n)) for _ in tiles]
    ranks = T.CompressedTile.compress_batch([torch.from_numpy(t.ravel(order="F").copy()).cuda() for t in tiles], out,
                                            T.CompressionParameters(1e-8, truncated_svd=True, mode=mode))
    return [(r, t.u(), t.v()) for r, t in zip(ranks, out)]


# Teams of the core: FP64 sweeps alone (12), a quarter and half an SM (40, 100), an SM and a cluster (150 among 20 and
# among 3), clusters (200), both orders of a rectangle.
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("m,n,count", [(1, 1, 3), (12, 12, 3), (40, 40, 5), (100, 100, 3), (150, 150, 20), (150, 150, 3),
                                       (200, 200, 3), (60, 100, 3), (200, 130, 3)])
def test_compression_of_a_tile_with_a_nonfinite_entry(T, m, n, count, value, mode):
    rng = np.random.default_rng([m, n, count])
    tiles = [_tile(rng, m, n) for _ in range(count)]
    want = _compress(T, tiles, mode)
    tiles[1][(2 * m) // 3, n // 2] = value
    got = _compress(T, tiles, mode)
    assert got[1][0] == 1
    assert np.isnan(got[1][1] @ got[1][2]).all()
    for i in [0] + list(range(2, count)):
        assert got[i][0] == want[i][0]
        np.testing.assert_array_equal(got[i][1], want[i][1])
        np.testing.assert_array_equal(got[i][2], want[i][2])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,r", [(40, 6), (96, 20), (200, 55), (256, 90)])
def test_update_of_a_tile_with_a_nan(T, n, r, mode):
    rng = np.random.default_rng([n, r])
    q = lambda: np.linalg.qr(rng.standard_normal((n, r)))[0]
    sigma = np.logspace(0, -6, r)[:, None]
    cu = q()
    cu[n // 3, r // 2] = np.nan
    c = T.CompressedTile(n, n, cu, sigma * q().T, max_rank=n)
    a = T.CompressedTile(n, n, q(), sigma * q().T, max_rank=r)
    b = T.CompressedTile(n, n, q(), q().T, max_rank=r)
    T.HCore.Gemm(1.0, a, 0, b, 0, 1.0, c, T.CompressionParameters(1e-8, truncated_svd=True, mode=mode))
    assert c.rank == 1
    assert np.isnan(c.to_dense()).all()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [12, 40, 100, 200])
@pytest.mark.parametrize("e", [-505, -512, -530])
def test_compression_of_tiny_tiles_stays_finite(T, n, e, mode):
    """Squared column norms in the subnormal range.  Singular values of at most 1e-150 (2^-498) count as zero: such a
    tile is dropped, to the last bit."""
    d = _tile(np.random.default_rng([n, -e]), n, n) * 2.0 ** e
    t = T.CompressedTile.from_dense(d, T.CompressionParameters(1e-5, truncated_svd=True, mode=mode), max_rank=n)
    assert np.isfinite(t.u()).all() and np.isfinite(t.v()).all()
    assert not t.to_dense().any()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [5, 12, 15, 40, 100, 200])
@pytest.mark.parametrize("e", [-470, -300, -250, 300])
def test_compression_does_not_depend_on_the_scale(T, n, e, mode):
    """Far from 1 (the squares of squared norms leave the range) as near it: a power of two changes no digit of the
    sweeps.  Smaller squared norms than 2^-960 (e = -470, entries down to 1e-8 of the top) may lose digits in the
    subnormal range, which moves singular values by at most 1e-150 each."""
    d = _tile(np.random.default_rng([n, 1]), n, n)
    p = T.CompressionParameters(1e-5, truncated_svd=True, mode=mode)
    near = T.CompressedTile.from_dense(d, p, max_rank=n)
    far = T.CompressedTile.from_dense(d * 2.0 ** e, p, max_rank=n)
    assert far.rank == near.rank
    err = np.linalg.norm(far.to_dense() * 2.0 ** -e - d) / np.linalg.norm(d)
    assert err <= 1.02e-5 * np.sqrt(n) + n * max(1e-150 * 2.0 ** -e, 1e-13) / np.linalg.norm(d)


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("m,n,k", [(8, 8, 8), (16, 16, 16), (40, 30, 33), (45, 45, 200), (130, 70, 129)])
def test_products_carry_nonfinite_entries(T, m, n, k, ta, tb):
    """A NaN reaches its row and column of the product, an infinity too (NaN where it meets a zero); every other
    output is that of the same product without them."""
    import torch
    rng = np.random.default_rng([m, n, k])
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((k, n)), rng.standard_normal((m, n))
    b[k // 2, n // 3] = 0.0

    def gemm(a, b):
        ta_, tb_ = a.T if ta else a, b.T if tb else b
        g = T.DenseTile(m, n, c)
        T.HCore.Gemm(-1.5, T.DenseTile(*ta_.shape, ta_), ta, T.DenseTile(*tb_.shape, tb_), tb, 0.5, g,
                     T.CompressionParameters(1e-8))
        return g.to_dense()

    want = gemm(a, b)
    a2, b2 = a.copy(), b.copy()
    a2[m // 2, k // 2] = np.inf
    a2[0, k - 1] = np.nan
    b2[0, n - 1] = -np.inf
    with np.errstate(invalid="ignore"):
        special = -1.5 * (a2 @ b2) + 0.5 * c
    got = gemm(a2, b2)
    finite = np.isfinite(special)
    np.testing.assert_array_equal(got[finite], want[finite])
    np.testing.assert_array_equal(got[~finite], special[~finite])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n,r", [(64, 17), (128, 40)])
def test_update_with_a_nan_in_a_factor_of_a(T, n, r, mode):
    """The NaN enters by the factor products."""
    rng = np.random.default_rng([n, r])
    q = lambda: np.linalg.qr(rng.standard_normal((n, r)))[0]
    av = np.logspace(0, -6, r)[:, None] * q().T
    av[r // 2, n // 3] = np.nan
    a = T.CompressedTile(n, n, q(), av, max_rank=r)
    b = T.CompressedTile(n, n, q(), q().T, max_rank=r)
    c = T.CompressedTile(n, n, q(), q().T, max_rank=n)
    T.HCore.Gemm(1.0, a, 0, b, 0, 1.0, c, T.CompressionParameters(1e-8, truncated_svd=True, mode=mode))
    assert c.rank == 1
    assert np.isnan(c.to_dense()).all()
