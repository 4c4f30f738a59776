"""The calls a user of this library makes, as timed cases.

Five kinds of work, each through the Python mirror of the public entry points (hcorepp_gb300.tiles):

  update     one tile update C <- alpha op(A) op(B) + beta C (HCore.Gemm), the call a task runtime makes
             for every task: latency and launches count
  multiply   C <- A B + C over tile grids (tlr_gemm): the main path, from a few tiles to 32 x 32
  compress   dense tiles -> U V with the rank rule of the constructor (CompressedTile.compress_batch)
  cholesky   tile Cholesky A = L L^T of a covariance matrix (tile_cholesky)
  transfer   the rank-trimmed transfer format out of one tile matrix and into another (pack, unpack)

Matrices are exponential kernels on Morton-sorted uniform points, the family tile-low-rank codes are built
for (hcorepp_gb300.problems): a_ij = exp(-|x_i - x_j| / ell), 2-D with ell = 0.1 for multiplies and
compression, 3-D with ell = 0.2 and 1e-2 on the diagonal for Cholesky.  Compressed input tiles hold what a
truncated factorisation of the block at the case's accuracy gives: U with orthonormal columns, the rows of V
graded like the singular values, the rank clamped at the capacity: the constructor's min(m, n) / 3, or nb in the
Cholesky cases (the 3-D kernel's neighbouring tiles need more than a third).

A compressed result has no unique factors (signs, rotations within clusters), so the passes return the
matrix its tiles stand for (TileMatrix.to_dense_device, the decoding a program that reads the result does)
and the ranks.
"""
import math

import numpy as np
import torch

from hcorepp_gb300 import _lib as L
from hcorepp_gb300 import tiles as T

PLAIN, MIXED = L.PLAIN_FP64, L.MIXED
MODES = {"plain": PLAIN, "mixed": MIXED}


def listed():
    return [
        # One task of a task runtime at a small tile size: all three tiles compressed.
        dict(name="update_nb256", kind="update", nb=256, combo="CCC", trans=False, accuracy=1e-8, mode="plain"),
        # The same call with a dense A and a transposed B, as the panels next to the diagonal need it.
        dict(name="update_nb512_dcc_t", kind="update", nb=512, combo="DCC", trans=True, accuracy=1e-8, mode="plain"),
        # A small multiply, every tile compressed (4 x 4 tiles): few updates in flight, the chain's latency.
        dict(name="multiply_n2048_nb512", kind="multiply", nt=4, nb=512, accuracy=1e-8, mode="plain", dense=False,
             cost_first=False),
        # Odd tile size and tile count at a looser accuracy (ragged panels, remainders everywhere).
        dict(name="multiply_11x11_nb301", kind="multiply", nt=11, nb=301, accuracy=1e-6, mode="plain", dense=True,
             cost_first=False),
        # The low accuracy that statistics codes run at: thin updates, many in flight.
        dict(name="multiply_n8192_nb512_1e-4", kind="multiply", nt=16, nb=512, accuracy=1e-4, mode="plain", dense=True,
             cost_first=False),
        # The float-float form on a middle-sized multiply.
        dict(name="multiply_n8192_nb512_mixed", kind="multiply", nt=16, nb=512, accuracy=1e-8, mode="mixed",
             dense=True, cost_first=True),
        # The benchmark's multiply (32 x 32 tiles, 32,768 updates), in the k order the benchmark uses.
        dict(name="multiply_n16384_nb512", kind="multiply", nt=32, nb=512, accuracy=1e-8, mode="plain", dense=True,
             cost_first=True),
        # Large tiles: wide stacks and cores.
        dict(name="multiply_n4096_nb1024", kind="multiply", nt=4, nb=1024, accuracy=1e-8, mode="plain", dense=True,
             cost_first=False),
        # Encoding input tiles: a batch of dense tiles of the benchmark's tile size.
        dict(name="compress_48x512", kind="compress", count=48, nb=512, accuracy=1e-8, mode="plain"),
        # Tile Cholesky of a 3-D covariance matrix.
        dict(name="cholesky_n2560_nb512", kind="cholesky", nt=5, nb=512, accuracy=1e-8, mode="plain"),
        # A smaller one in the float-float form with an odd tile size.
        dict(name="cholesky_9x9_nb200_mixed", kind="cholesky", nt=9, nb=200, accuracy=1e-8, mode="mixed"),
        # The transfer format of a 16 x 16-tile matrix, out and back in (the copies around an end-to-end run).
        dict(name="transfer_n8192_nb512", kind="transfer", nt=16, nb=512, accuracy=1e-8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update", "multiply", "multiply", "multiply", "compress", "cholesky", "transfer"])
    accuracy = 10.0 ** -rng.uniform(4.0, 9.0)
    mode = rng.choice(["plain", "plain", "mixed"])
    if kind == "update":
        return dict(kind=kind, nb=_log_int(rng, 64, 700), combo=rng.choice(["CCC", "DCC", "CDC", "CCD"]),
                    trans=rng.random() < 0.3, accuracy=accuracy, mode=mode)
    if kind == "multiply":
        nb = _log_int(rng, 128, 700)
        nt = _log_int(rng, 3, min(20, 9000 // nb))
        return dict(kind=kind, nt=nt, nb=nb, accuracy=accuracy, mode=mode, dense=rng.random() < 0.6,
                    cost_first=rng.random() < 0.5)
    if kind == "compress":
        return dict(kind=kind, count=_log_int(rng, 3, 90), nb=_log_int(rng, 100, 512), accuracy=accuracy, mode=mode)
    if kind == "cholesky":
        nb = _log_int(rng, 100, 400)
        return dict(kind=kind, nt=_log_int(rng, 3, 9), nb=nb, accuracy=min(accuracy, 1e-6), mode=mode)
    nb = _log_int(rng, 100, 700)
    return dict(kind=kind, nt=_log_int(rng, 3, min(24, 9000 // nb)), nb=nb, accuracy=accuracy)


# ---------------------------------------------------------------------------------------------------
# Inputs, in plain torch.
# ---------------------------------------------------------------------------------------------------

def _points(n, d, seed, which):
    """n uniform points in [0, 1]^d in Morton order, on the GPU."""
    x = np.random.default_rng([seed, which]).random((n, d))
    q = (x * 2.0 ** 20).astype(np.uint64)
    code = np.zeros(n, dtype=np.uint64)
    for b in range(20):
        for c in range(d):
            code |= ((q[:, c] >> np.uint64(b)) & np.uint64(1)) << np.uint64(b * d + c)
    return torch.from_numpy(x[np.argsort(code, kind="stable")]).cuda()


def _blocks(x, nb, pairs, ell, shift):
    """Kernel blocks (len(pairs), nb, nb) of the point set x."""
    xi = torch.stack([x[i * nb:(i + 1) * nb] for i, _ in pairs])
    xj = torch.stack([x[j * nb:(j + 1) * nb] for _, j in pairs])
    out = torch.zeros((len(pairs), nb, nb), dtype=torch.float64, device=x.device)
    for c in range(x.shape[1]):
        out += (xi[:, :, None, c] - xj[:, None, :, c]).square_()
    out.sqrt_().mul_(-1.0 / ell).exp_()
    for t, (i, j) in enumerate(pairs):
        if i == j and shift:
            out[t].diagonal().add_(shift)
    return out


def _pivoted(a, most, rel):
    """Batched column-pivoted Gram-Schmidt (with reorthogonalisation) of a (b, m, n), overwritten: Q
    (b, m, s) with orthonormal columns and R (b, s, n), a = Q R up to columns below rel * the first pivot."""
    b, m, n = a.shape
    most = min(most, m, n)
    q = torch.zeros((b, most, m), dtype=a.dtype, device=a.device)
    r = torch.zeros((b, most, n), dtype=a.dtype, device=a.device)
    rows = torch.arange(b, device=a.device)
    first = None
    for s in range(most):
        norms = a.square().sum(1)
        top, piv = norms.max(1)
        first = top if first is None else first
        live = top > first * rel * rel
        if s % 8 == 0 and not bool(live.any()):
            return q[:, :s].transpose(1, 2), r[:, :s]
        v = a[rows, :, piv]
        for _ in range(2):
            if s:
                v = v - torch.bmm(q[:, :s].transpose(1, 2), torch.bmm(q[:, :s], v[:, :, None]))[:, :, 0]
        v = torch.where(live[:, None], v / v.norm(dim=1, keepdim=True).clamp_min(1e-300), torch.zeros_like(v))
        q[:, s] = v
        r[:, s] = torch.bmm(v[:, None, :], a)[:, 0]
        a.baddbmm_(v[:, :, None], r[:, s:s + 1], alpha=-1.0)
    return q.transpose(1, 2), r


def _capacity(nb, kind):
    return nb if kind == "cholesky" else max(nb // 3, 1)


def _factors(blocks, accuracy, cap):
    """[(U, V)] of the blocks: U (nb, r) orthonormal, V (r, nb) with rows graded like the singular values (a
    pivoted QR of the pivoted R factor tracks them closely), r the first index below accuracy * the first,
    clamped at cap."""
    nb = blocks.shape[1]
    out = []
    for part in blocks.split(max(1, int(3.0e8 / (8.0 * nb * nb)))):
        q1, r1 = _pivoted(part.transpose(1, 2).contiguous(), cap + 32, 0.02 * accuracy)
        p, l = _pivoted(r1.transpose(1, 2).contiguous(), cap + 32, 0.02 * accuracy)
        # part^T = q1 r1, r1^T = p l: part = r1^T q1^T = p (l q1^T)
        v = torch.bmm(l, q1.transpose(1, 2))
        s = v.norm(dim=2)
        keep = (s < accuracy * s[:, :1])
        keep[:, 0] = False
        ranks = torch.where(keep.any(1), keep.to(torch.int32).argmax(1), s.shape[1]).clamp(1, cap).tolist()
        out += [(p[t, :, :r], v[t, :r]) for t, r in enumerate(ranks)]
    return out


def _matrix(nt, nb, d, ell, shift, accuracy, cap, dense_diagonal, seed, which, lower=False):
    """Tiles {(i, j): dense block or (U, V)} of a kernel matrix."""
    x = _points(nt * nb, d, seed, which)
    every = [(i, j) for j in range(nt) for i in range(nt) if i >= j or not lower]
    near = [p for p in every if dense_diagonal and p[0] == p[1]]
    far = [p for p in every if not (dense_diagonal and p[0] == p[1])]
    far.sort(key=lambda p: (abs(p[0] - p[1]), p))  # tiles of like ranks together: the factorisation stops sooner
    tiles = {}
    step = max(1, int(2.0e9 / (8.0 * nb * nb)))
    for o in range(0, len(far), step):
        tiles.update(zip(far[o:o + step], _factors(_blocks(x, nb, far[o:o + step], ell, shift), accuracy, cap)))
    if near:
        tiles.update(zip(near, _blocks(x, nb, near, ell, shift).unbind(0)))
    return tiles


def _tile_matrix(tiles, nt, nb, cap, vt=False):
    kinds = [[None if (i, j) not in tiles else L.COMPRESSED if isinstance(tiles[i, j], tuple) else L.DENSE
              for j in range(nt)] for i in range(nt)]
    tm = T.TileMatrix(nt, nt, nb, kinds, cap, vt=vt)
    ranks = [0] * (nt * nt)
    for (i, j), t in tiles.items():
        buf = tm.tile(i, j).buffer
        if not isinstance(t, tuple):
            buf.view(nb, nb).copy_(t.t())
            continue
        u, v = t
        r = u.shape[1]
        ranks[tm.index(i, j)] = r
        buf[:nb * r].view(r, nb).copy_(u.t())
        region = buf[nb * tm.max_rank:nb * tm.max_rank + nb * r]
        if vt:
            region.view(r, nb).copy_(v)
        else:
            region.view(nb, r).copy_(v.t())
    tm.ranks.copy_(torch.tensor(ranks, dtype=torch.int32))
    return tm


def _dense(tiles, nt, nb):
    out = torch.zeros((nt * nb, nt * nb), dtype=torch.float64, device="cuda")
    for (i, j), t in tiles.items():
        out[i * nb:(i + 1) * nb, j * nb:(j + 1) * nb] = t[0] @ t[1] if isinstance(t, tuple) else t
    return out


def _params(case):
    return T.CompressionParameters(case["accuracy"], truncated_svd=True, mode=MODES[case.get("mode", "plain")])


def _update_inputs(case, seed):
    """Blocks next to each other of two kernel matrices: A = (0, 1), B = (1, 2), C = (0, 2); a transposed B
    is handed over as its transpose."""
    nb, acc = case["nb"], case["accuracy"]
    xa, xc = _points(4 * nb, 2, seed, 0), _points(4 * nb, 2, seed, 1)
    blocks = [_blocks(xa, nb, [(0, 1)], 0.1, 0.0), _blocks(xa, nb, [(1, 2)], 0.1, 0.0), _blocks(xc, nb, [(0, 2)], 0.1, 0.0)]
    if case["trans"]:
        blocks[1] = blocks[1].transpose(1, 2).contiguous()
    cap = _capacity(nb, "update")
    return [b[0] if kind == "D" else _factors(b, acc, cap)[0] for b, kind in zip(blocks, case["combo"])]


def _multiply_inputs(case, seed):
    """B = A as in the benchmark; C from another point set."""
    nt, nb = case["nt"], case["nb"]
    return [_matrix(nt, nb, 2, 0.1, 0.0, case["accuracy"], _capacity(nb, "multiply"), case["dense"], seed, which)
            for which in (0, 1)]


def _compress_inputs(case, seed):
    """Off-diagonal blocks of a kernel matrix, column by column."""
    nb, count = case["nb"], case["count"]
    nt = 2
    while nt * (nt - 1) < count:
        nt += 1
    pairs = [(i, j) for j in range(nt) for i in range(nt) if i != j][:count]
    return _blocks(_points(nt * nb, 2, seed, 0), nb, pairs, 0.1, 0.0)


def _cholesky_inputs(case, seed):
    return _matrix(case["nt"], case["nb"], 3, 0.2, 1e-2, case["accuracy"], _capacity(case["nb"], "cholesky"), True, seed, 0,
                   lower=True)


# ---------------------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------------------

_CONTEXTS = {}


def _context(cost_first):
    """A program keeps one context per setting (its workspace grows to the largest call)."""
    if cost_first not in _CONTEXTS:
        ctx = L.Context(torch.cuda.current_device())
        ctx.set_k_order(1 if cost_first else 0)
        _CONTEXTS[cost_first] = ctx
    ctx = _CONTEXTS[cost_first]
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def prepare(case, seed):
    kind, nb, nt = case["kind"], case["nb"], case.get("nt", 1)
    cap = _capacity(nb, kind)
    if kind == "update":
        tms = [_tile_matrix({(0, 0): t}, 1, nb, cap) for t in _update_inputs(case, seed)]
        return dict(kind=kind, a=tms[0].tile(0, 0), b=tms[1].tile(0, 0), c=tms[2], ct=tms[2].tile(0, 0), keep=tms,
                    c0=tms[2].arena.clone(), r0=tms[2].ranks.clone(), op=L.TRANS if case["trans"] else L.NOTRANS,
                    params=_params(case))
    if kind == "multiply":
        a, c = [_tile_matrix(t, nt, nb, cap) for t in _multiply_inputs(case, seed)]
        return dict(kind=kind, a=a, c=c, c0=c.arena.clone(), r0=c.ranks.clone(), params=_params(case),
                    ctx=_context(case["cost_first"]))
    if kind == "compress":
        blocks = _compress_inputs(case, seed)
        dense = [t.reshape(-1) for t in blocks.transpose(1, 2).contiguous().unbind(0)]  # column-major
        out = T.TileMatrix(case["count"], 1, nb, [[L.COMPRESSED]] * case["count"], cap)
        return dict(kind=kind, dense=dense, out=out, tiles=[out.tile(i, 0) for i in range(case["count"])],
                    params=_params(case))
    if kind == "cholesky":
        a = _tile_matrix(_cholesky_inputs(case, seed), nt, nb, cap, vt=True)
        return dict(kind=kind, a=a, a0=a.arena.clone(), r0=a.ranks.clone(), params=_params(case))
    tiles = _matrix(nt, nb, 2, 0.1, 0.0, case["accuracy"], cap, True, seed, 0)
    src, dst = _tile_matrix(tiles, nt, nb, cap), _tile_matrix(tiles, nt, nb, cap)
    dst.arena.zero_()
    return dict(kind=kind, src=src, dst=dst, packed=torch.zeros_like(src.arena),
                offsets=torch.zeros(nt * nt + 1, dtype=torch.int64, device="cuda"))


def run(state):
    kind = state["kind"]
    if kind == "update":
        c = state["c"]
        c.arena.copy_(state["c0"])  # the update is in place: every pass starts from the same C
        c.ranks.copy_(state["r0"])
        T.HCore.Gemm(1.0, state["a"], L.NOTRANS, state["b"], state["op"], 1.0, state["ct"], state["params"])
        return dict(c=c.to_dense_device(), ranks=c.ranks)
    if kind == "multiply":
        c = state["c"]
        c.arena.copy_(state["c0"])
        c.ranks.copy_(state["r0"])
        T.tlr_gemm(1.0, state["a"], state["a"], 1.0, c, state["params"], ctx=state["ctx"])
        return dict(c=c.to_dense_device(), ranks=c.ranks)
    if kind == "compress":
        ranks = T.CompressedTile.compress_batch(state["dense"], state["tiles"], state["params"])
        return dict(tiles=state["out"].to_dense_device(), ranks=torch.tensor(ranks))
    if kind == "cholesky":
        a = state["a"]
        a.arena.copy_(state["a0"])
        a.ranks.copy_(state["r0"])
        info = T.tile_cholesky(a, state["params"])
        return dict(l=torch.tril(a.to_dense_device()), ranks=a.ranks, info=info)
    state["src"].pack(state["packed"], state["offsets"])
    state["dst"].unpack(state["packed"], state["offsets"])
    return dict(packed=state["packed"], offsets=state["offsets"], arena=state["dst"].arena)


# ---------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------------

def _rank(case):
    """Mean tile rank of these kernels at the case's accuracy (30 at 1e-8 and nb = 512, 3-D ranks ~2.5 times
    the 2-D ones), within the capacity."""
    digits = -math.log10(case["accuracy"])
    r = 3.7 * digits * (2.5 if case["kind"] == "cholesky" else 1.0)
    return min(r, 1.0 * _capacity(case["nb"], case["kind"]))


def _recompression(nb, r):
    """Flops of one recompressing update: products, two stack QRs, the core's SVD, two Q applications."""
    k = 1.5 * r
    return 4.0 * nb * r * r + 4.0 * nb * k * k + 22.0 * k ** 3 + 8.0 * nb * k * r


def work(case):
    kind, nb = case["kind"], case["nb"]
    r = _rank(case)
    tile = 16.0 * nb * r
    if kind == "update":
        dense = 8.0 * nb * nb
        return dict(bytes=sum(dense if k == "D" else tile for k in case["combo"] + case["combo"][2]) + dense,
                    flops=_recompression(nb, r) + (2.0 * nb * nb * r if "D" in case["combo"] else 0.0))
    if kind == "multiply":
        nt = case["nt"]
        n = nt * nt * tile
        return dict(bytes=4.0 * n + 8.0 * (nt * nb) ** 2, flops=nt ** 3 * _recompression(nb, r))
    if kind == "compress":
        return dict(bytes=case["count"] * (16.0 * nb * nb + tile), flops=case["count"] * 6.0 * nb * nb * r)
    if kind == "cholesky":
        nt = case["nt"]
        updates = nt * (nt * nt - 1) / 6.0
        return dict(bytes=nt * nt * tile + 8.0 * nt * nb * nb + 8.0 * (nt * nb) ** 2,
                    flops=updates * _recompression(nb, r) + nt * nb ** 3 / 3.0 + nt * nt / 2.0 * nb * nb * r)
    nt = case["nt"]
    used = nt * (nt - 1) * tile + 8.0 * nt * nb * nb
    return dict(bytes=4.0 * used, flops=0.0)


# ---------------------------------------------------------------------------------------------------
# The same results in 64 bits, in plain torch / numpy
# ---------------------------------------------------------------------------------------------------

def _truncate(u, s, vt, accuracy, cap):
    small = np.nonzero(s[1:] < accuracy * s[0])[0]
    r = min(max(int(small[0]) + 1 if small.size else s.size, 1), cap)
    return u[:, :r], s[:r, None] * vt[:r]


def _host(t):
    return tuple(x.cpu().numpy() for x in t) if isinstance(t, tuple) else t.cpu().numpy()


def _full(t):
    return t[0] @ t[1] if isinstance(t, tuple) else t


def _add_product(a, b, c, accuracy, cap):
    """C + A B as a tile of C's kind: truncated after the sum when C is compressed (LAPACK QR and SVD)."""
    if not isinstance(c, tuple):
        return c + _full(a) @ _full(b)
    if isinstance(a, tuple) and isinstance(b, tuple):
        w = a[1] @ b[0]
        pu, pv = (a[0], w @ b[1]) if a[0].shape[1] <= b[0].shape[1] else (a[0] @ w, b[1])
    elif isinstance(a, tuple):
        pu, pv = a[0], a[1] @ b
    else:
        pu, pv = a @ b[0], b[1]
    qu, ru = np.linalg.qr(np.hstack([c[0], pu]))
    qv, rv = np.linalg.qr(np.hstack([c[1].T, pv.T]))
    u, v = _truncate(*np.linalg.svd(ru @ rv.T, full_matrices=False), accuracy, cap)
    return qu @ u, v @ qv.T


def exact(case, seed):
    kind, nb, acc = case["kind"], case["nb"], case["accuracy"]
    cap = _capacity(nb, kind)
    if kind == "update":
        a, b, c = [_host(t) for t in _update_inputs(case, seed)]
        d = _full(a) @ (_full(b).T if case["trans"] else _full(b)) + _full(c)
        if isinstance(c, tuple):
            u, v = _truncate(*np.linalg.svd(d, full_matrices=False), acc, cap)
            d = u @ v
        return dict(c=d, ranks=None)
    if kind == "multiply":
        nt = case["nt"]
        a, c = _multiply_inputs(case, seed)
        if case["cost_first"] or nt ** 3 * nb > 500000:
            # the sum itself: no truncation (an order of the sums that is the library's own to choose, or
            # too many truncations to restate here)
            d = _dense(a, nt, nb)
            return dict(c=_dense(c, nt, nb).addmm_(d, d), ranks=None)
        a, c = ({k: _host(t) for k, t in x.items()} for x in (a, c))
        for (i, j) in c:
            for k in range(nt):
                c[i, j] = _add_product(a[i, k], a[k, j], c[i, j], acc, cap)
        return dict(c=np.block([[_full(c[i, j]) for j in range(nt)] for i in range(nt)]), ranks=None)
    if kind == "compress":
        out = []
        for d in _compress_inputs(case, seed).cpu().numpy():
            u, v = _truncate(*np.linalg.svd(d, full_matrices=False), acc, cap)
            out.append(u @ v)
        return dict(tiles=np.vstack(out), ranks=None)
    if kind == "cholesky":
        d = _dense(_cholesky_inputs(case, seed), case["nt"], nb)
        return dict(l=torch.linalg.cholesky(torch.tril(d) + torch.tril(d, -1).t()), ranks=None, info=None)
    return None
