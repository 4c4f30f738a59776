"""The recompression core at the edges of its classes: stack widths around the preconditioner's smallest core
(16 columns), the quarter- and half-CTA teams' shared memory (82 and 117 columns), the wide cores of a
thread-block cluster, odd sizes, slow and fast decay, nearly equal singular values."""
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


def _factor(rng, m, n, s):
    """A compressed tile with singular values s: U orthonormal, rows of V orthogonal."""
    r = len(s)
    u = np.linalg.qr(rng.standard_normal((m, r)))[0]
    v = np.linalg.qr(rng.standard_normal((n, r)))[0]
    return u, s[:, None] * v.T


def _spectrum(kind, r, top):
    if kind == "decay":      # the kernels' own: down to the accuracy
        return top * np.logspace(0, -8, r)
    if kind == "slow":       # nothing to truncate
        return top * np.linspace(1.0, 0.5, r)
    s = np.repeat(np.logspace(0, -7, (r + 2) // 3), 3)[:r]  # "triples": clusters of equal singular values
    return top * s


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind", ["decay", "slow", "triples"])
@pytest.mark.parametrize("n,rc,ra", [(40, 7, 8), (40, 8, 9), (75, 33, 31), (300, 41, 41), (301, 42, 41), (300, 60, 57),
                                     (301, 61, 57), (299, 80, 75), (320, 120, 105), (512, 170, 170)])
def test_recompression_at_class_edges(T, n, rc, ra, kind, mode):
    rng = np.random.default_rng([n, rc, ra, len(kind)])
    acc, k, cap = 1e-8, rc + ra, min(n, rc + ra)
    cu, cv = _factor(rng, n, n, _spectrum(kind, rc, 1.0))
    au, av = _factor(rng, n, n, _spectrum(kind, ra, 0.7))
    bu, bv = _factor(rng, n, n, np.ones(min(n, ra + 3)))
    oc = O.CompressedTile(cu, cv, cap)
    oa = O.CompressedTile(au, av, cap)
    ob = O.CompressedTile(bu, bv, max(cap, bu.shape[1]))
    gc, ga = (T.CompressedTile(n, n, t.u, t.v, max_rank=cap) for t in (oc, oa))
    gb = T.CompressedTile(n, n, bu, bv, max_rank=max(cap, bu.shape[1]))
    exact = oa.to_dense() @ ob.to_dense() + oc.to_dense()
    O.hcore_gemm(1.0, oa, ob, 1.0, oc, O.CompressionParameters(acc, truncated_svd=True))
    T.HCore.Gemm(1.0, ga, 0, gb, 0, 1.0, gc, T.CompressionParameters(acc, truncated_svd=True, mode=mode))
    assert abs(gc.rank - oc.rank) <= 1
    assert rel_fro(gc.to_dense(), exact) <= 2 * max(rel_fro(oc.to_dense(), exact), acc)
    # V's rows are singular vectors: orthogonal to the sweeps' tolerance (8 eps k) plus the rounding of the Q application, a few units of roundoff
    # (2^-48 in the float-float form) a reflector
    v = np.asarray(gc.v(), dtype=np.float64)
    norms = np.linalg.norm(v, axis=1)
    assert np.all(norms > 0)
    g = np.abs((v / norms[:, None]) @ (v / norms[:, None]).T - np.eye(len(norms)))
    unit = EPS / 2 if mode == 0 else 2.0 ** -48
    assert g.max() <= 64 * k * unit
    # U = M XV Sigma^-2: orthonormal up to rounding relative to the smallest kept singular value
    u = np.asarray(gc.u(), dtype=np.float64)
    assert np.abs(u.T @ u - np.eye(u.shape[1])).max() <= 64 * k * unit * norms.max() / norms.min()


def _update_in_capacities(T, k, kind, mode, extras):
    """(rank, U, V) of one update of stack width k in tiles of capacity sum k + extra.  A lies below the threshold but not
    below the pivoted QR's stop: all k columns are swept, C's own rank is the result's in every capacity."""
    rng = np.random.default_rng([k, len(kind)])
    n, ra = max(120, k), k // 2
    rc = k - ra
    sc = np.logspace(0, -6, rc) if kind == "decay" else np.repeat(np.logspace(0, -6, (rc + 2) // 3), 3)[:rc]
    cu, cv = _factor(rng, n, n, sc)
    au, av = _factor(rng, n, n, np.linspace(3e-9, 2e-9, ra))
    bv = np.linalg.qr(rng.standard_normal((n, ra)))[0].T
    bu = av.T / np.linalg.norm(av, axis=1)  # A B = Au Sigma Bv
    out = []
    for extra in extras:
        c = T.CompressedTile(n, n, cu, cv, max_rank=rc + extra)
        a = T.CompressedTile(n, n, au, av, max_rank=ra)
        b = T.CompressedTile(n, n, bu, bv, max_rank=ra)
        T.HCore.Gemm(1.0, a, 0, b, 0, 1.0, c, T.CompressionParameters(1e-8, truncated_svd=True, mode=mode))
        out.append((c.rank, c.u(), c.v()))
    return out


def _assert_same(results):
    for r, u, v in results[1:]:
        assert r == results[0][0]
        np.testing.assert_array_equal(u, results[0][1])
        np.testing.assert_array_equal(v, results[0][2])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind", ["decay", "triples"])
@pytest.mark.parametrize("k", [30, 41, 45, 73, 75, 76, 80, 81, 82])
def test_preconditioned_cores_in_every_team(T, k, kind, mode):
    """Widths around the quarter team's, in tiles whose capacities put them there and in the next larger team: a core
    is preconditioned in either, with the same bits."""
    _assert_same(_update_in_capacities(T, k, kind, mode, (4, 19, 30, 60, 200)))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind", ["decay", "triples"])
@pytest.mark.parametrize("k", [9, 10, 25, 26, 41, 58, 74, 90, 105, 106, 114, 115])
def test_results_do_not_depend_on_the_capacity(T, k, kind, mode):
    """A full stack of k columns, in tiles that hold no more and in larger ones."""
    _assert_same(_update_in_capacities(T, k, kind, mode, (0, 1, 16, 60, 200)))


def _full_rank_core(T, n, extras, mode):
    """An update whose core has full rank n = k and nothing to truncate before the threshold, in several capacities."""
    rng = np.random.default_rng(n)
    rc = n - n // 2
    orth = lambda m: np.linalg.qr(rng.standard_normal((m, m)))[0]
    qu, qv, gc, ga = orth(n), orth(n), orth(rc), orth(n - rc)  # gc, ga: the sweeps have something to turn
    sa = np.linspace(3e-9, 2e-9, n - rc)
    out = []
    for extra in extras:
        c = T.CompressedTile(n, n, (qu[:, :rc] * np.logspace(0, -6, rc)) @ gc, qv[:, :rc].T, max_rank=rc + extra)
        a = T.CompressedTile(n, n, (qu[:, rc:] * sa) @ ga, qv[:, rc:].T, max_rank=n - rc)
        b = T.CompressedTile(n, n, qv[:, rc:], qv[:, rc:].T, max_rank=n - rc)
        T.HCore.Gemm(1.0, a, 0, b, 0, 1.0, c, T.CompressionParameters(1e-8, truncated_svd=True, mode=mode))
        out.append((c.rank, c.u(), c.v()))
    return out


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [197, 199, 301, 302, 303, 304])
def test_wide_full_rank_cores_do_not_depend_on_the_capacity(T, n, mode):
    """As many rows as columns, and no multiple of 4: the padded columns of X and J at their longest."""
    _assert_same(_full_rank_core(T, n, (0, 1, 16, 100), mode))


def test_noalloc_shapes_at_the_limit_of_its_scratch(T):
    """A shape that fits the 8 MiB only without those columns' padding is still taken."""
    import ctypes as C
    import torch
    from hcorepp_gb300 import _lib as L
    rng = np.random.default_rng(1)
    n, rmax, rc = 400, 152, 245
    cu, cv = _factor(rng, n, n, np.logspace(0, -6, 12))
    au, av = _factor(rng, n, n, np.logspace(0, -6, 10))
    tiles = [T.CompressedTile(n, n, au, av, max_rank=rmax), T.CompressedTile(n, n, av.T, au.T, max_rank=rmax),
             T.CompressedTile(n, n, cu, cv, max_rank=rc)]
    a, b, c = (t.c_tile() for t in tiles)
    p = T.CompressionParameters(1e-8, truncated_svd=True).c()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.lib().hcgb_tile_gemm_noalloc(1.0, C.byref(a), C.byref(b), 1.0, C.byref(c), C.byref(p), stream,
                                          C.c_void_p(0)) == L.HCGB_OK
    torch.cuda.synchronize()
    exact = au @ av @ av.T @ au.T + cu @ cv
    assert rel_fro(tiles[2].to_dense(), exact) <= 1.02e-8 * np.sqrt(22)
