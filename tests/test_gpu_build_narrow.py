"""Builds with strings in 32-bit registers (up to 32 orbitals) and at the first size past them.

Sets whose strings reach the highest orbital, with two alpha groups long enough to be probed
through the determinant table and many short ones that are scanned: the stored elements
against the oracle, bitwise, and the matrix-free product.
"""
import itertools

import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _set(norb):
    rng = np.random.default_rng(norb)
    orbs = [0, 1, 2, 15, 16, 17] + list(range(norb - 5, norb))  # both ends and the middle
    strings = [sum(1 << o for o in c) for c in itertools.combinations(orbs, 4)]  # 330
    pairs = {(strings[k], s) for k in (0, 1) for s in strings}
    while len(pairs) < 1200:
        pairs.add((strings[rng.integers(330)], strings[rng.integers(330)]))
    dets = np.zeros((len(pairs), 4), dtype=np.uint64)
    dets[:, [0, 2]] = np.array(sorted(pairs), dtype=np.uint64)
    return dets[rng.permutation(len(dets))]


@pytest.mark.parametrize("norb", [31, 32, 33])
def test_elements_bitwise_around_32_orbitals(norb):
    ints = synthetic_integrals(norb, 5)
    dets = _set(norb)
    oh = H.oracle_ham(ints)
    x = np.random.default_rng(1).standard_normal(len(dets))
    with GpuHam(ints) as g:
        g.set_dets(dets)
        g.build(_capi.FP64, _capi.BUILDER_FAST)
        rp, cols, vals, diag = g.export_upper()
        sp = O.Sparse().build(oh, dets, diag, 0, builder=_capi.BUILDER_FAST)
        orp, ocols, ovals, _ = sp.export()
        ref = sp.mv(x)
        np.testing.assert_array_equal(rp, orp)
        np.testing.assert_array_equal(cols, ocols)
        np.testing.assert_array_equal(vals, ovals)
        g.build(_capi.FP64_UPPER, _capi.BUILDER_FAST)
        rp, cols, vals, _ = g.export_upper()
        np.testing.assert_array_equal(rp, orp)
        np.testing.assert_array_equal(cols, ocols)
        np.testing.assert_array_equal(vals, ovals)
        for prec in (_capi.MIXED, _capi.MIXED_UPPER):
            g.build(prec, _capi.BUILDER_FAST)
            rp, cols, vals, _ = g.export_upper()
            np.testing.assert_array_equal(rp, orp)
            np.testing.assert_array_equal(cols, ocols)
            # FP32 value + FP32 remainder carries 48 bits of the FP64 element
            assert np.all(np.abs(vals - ovals) <= 2.0 ** -46 * np.abs(ovals) + 1e-300)
        g.build(_capi.MATRIX_FREE, _capi.BUILDER_FAST)
        y = g.matrix_vector_prod(x)
    assert np.max(np.abs(y - ref)) <= 1e-11 * np.max(np.abs(ref))
