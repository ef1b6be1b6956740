"""Rounding of the tiled sigma on flat vectors.

On a vector without decay a panel's largest |x| is the largest of all, so a product's rounding
is that of the tile's scale: the tile's largest column sum of |H| may be no larger than the
real one.  The bounds count that scale only: a product is rounded to 2^-51 (FP64 vectors) or
2^-30 (FP32) of its tile's largest column sum, itself at most the largest row sum of |H|, and
the errors of the m terms of a row add up like independent ones (5 sqrt(m) of the root mean
square, 2^-0.5 / sqrt(6) of a unit).
"""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


def system(norb, nel, eps):
    ints, _, dets, _, diag, _ = H.synthetic_hci(norb, nel, eps)
    n = len(dets)
    sp = O.Sparse().build(H.oracle_ham(ints), dets, diag, 0, builder=_capi.BUILDER_FAST)
    rp, cols, vals, _ = sp.export()
    rows = np.repeat(np.arange(n), np.diff(rp))
    order = np.lexsort((dets[:, 2], dets[:, 0]))  # internal order: by (up, dn)
    return ints, dets, diag, sp, rows, cols, vals, order


def column_sums(rows, cols, vals, order, rb, cb):
    """Largest column sum of |H| of every (panel, window) tile, per determinant: the mean
    square of those of the tiles that add to it from above (its columns)."""
    n = len(order)
    rank = np.argsort(order)
    p, q = np.minimum(rank[rows], rank[cols]), np.maximum(rank[rows], rank[cols])
    panel, window = p >> rb, q >> cb
    key = panel * n + q
    u, inv = np.unique(key, return_inverse=True)
    s = np.bincount(inv, weights=np.abs(vals))
    tile = (u // n) * (n + 1) + ((u % n) >> cb)
    t, tinv = np.unique(tile, return_inverse=True)
    big = np.zeros(len(t))
    np.maximum.at(big, tinv, s)
    per_pair = big[np.searchsorted(t, panel * (n + 1) + window)]
    return np.bincount(q, weights=per_pair ** 2, minlength=n)  # internal order


@pytest.mark.parametrize("norb,nel,eps", [(12, 6, 1e-3), (12, 6, 1e-4)])
def test_column_sums_round_at_the_tile_maximum(norb, nel, eps):
    ints, dets, diag, sp, rows, cols, vals, order = system(norb, nel, eps)
    n = len(dets)
    x = np.where(np.random.default_rng(1).random(n) < 0.5, -1.0, 1.0)
    ref = sp.mv(x)
    # FP32 tiles: windows of at most 4096 columns, fewer for small sets, panels of at most 2048
    # rows; a larger tile only makes its largest column sum larger
    var = column_sums(rows, cols, vals, order, 11, 12)
    mag = np.abs(diag * x)
    np.add.at(mag, rows, np.abs(vals))
    np.add.at(mag, cols, np.abs(vals))
    # the FP64 parts: every product and sum of at most 2^-52 of its size
    exact = 8 * 2.0 ** -52 * mag[order]
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        g.build(_capi.MIXED_UPPER, _capi.BUILDER_FAST)
        err = np.abs(g.matrix_vector_prod(x) - ref)[order]
    # one unit is at most 2^-51 of twice the tile's largest column sum (power-of-two scale)
    rms = 2.0 ** -50 * np.sqrt(var / 12.0)
    # remainders: a stored value is FP32 + FP32, 2^-48 of itself
    stored = 2.0 ** -48 * np.sqrt(np.bincount(np.concatenate([rows, cols]), weights=np.tile(vals ** 2, 2),
                                              minlength=n))[order]
    assert np.all(err <= exact + 5 * rms + 5 * stored)
    assert np.sqrt((err ** 2).mean()) <= np.sqrt(((0.125 * exact) ** 2 + rms ** 2 + stored ** 2).mean())


def test_row_sums_over_many_windows_round_once():
    """FP32 sigma, a row's sum without signs, from every window to the right of it: rounded to
    FP32 at the end (0.29 units of 2^-24 root mean square) and, for each slot of 64 elements,
    by up to 16 additions of a twentieth of it or less; products and values round by as much
    as the end, but each on its own small part.  Half a unit is the line."""
    ints, dets, diag, sp, rows, cols, vals, order = system(12, 6, 1e-3)
    n = len(dets)
    rank = np.argsort(order)
    p, q = np.minimum(rank[rows], rank[cols]), np.maximum(rank[rows], rank[cols])
    import torch

    errs = []
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        g.build(_capi.MIXED_UPPER, _capi.BUILDER_FAST)
        for p0 in range(0, 240, 5):
            at = p == p0
            x = np.zeros(n)
            x[q[at]] = np.sign(vals[at])
            total = np.abs(vals[at]).sum()
            xd = torch.tensor(x, dtype=torch.float32, device="cuda")
            yd = torch.empty_like(xd)
            torch.cuda.synchronize()
            g.sigma_device(xd.data_ptr(), yd.data_ptr(), 1)
            errs.append((float(yd[p0]) - total) / total)
    assert np.sqrt(np.mean(np.square(errs))) <= 0.5 * 2.0 ** -24
