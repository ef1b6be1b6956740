"""Calls after a determinant set was refused: an error or the general path, no stale groups."""
import numpy as np
import pytest

from risq_b200 import GpuHam, _capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [False, True])  # on a new handle, or after another set
@pytest.mark.parametrize("extra", ["duplicate", "electrons"])
def test_selection_after_a_refused_set(first, extra):
    ints, _, dets, coeffs, diag, _ = H.synthetic_hci(10, 4, 1e-3)
    dets, coeffs = dets[:301], coeffs[:301]
    # one more determinant, too small a coefficient to add any: twice the last one, or a
    # string with more up electrons than the first determinant has
    more = dets[-1:].copy()
    if extra == "electrons":
        more[0, 0] = 0b1111111110
    bad = np.concatenate([dets, more])
    c = np.append(coeffs, 1e-30)
    with GpuHam(ints) as g:
        g.set_dets(dets)
        want, want_diag = g.find_new_dets(coeffs, 1e-3, True)
        assert len(want) > 0
    with GpuHam(ints) as g:
        if first:
            g.set_dets(dets[:40])
            g.build(_capi.FP64, _capi.BUILDER_FAST)
        with pytest.raises(_capi.RisqGpuError):
            g.set_dets(bad)
        with pytest.raises(_capi.RisqGpuError, match="refused"):
            g.build(_capi.FP64)
        g.n = len(bad)  # the C interface takes as many coefficients as the refused set has
        got, got_diag = g.find_new_dets(c, 1e-3, True)
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(got_diag, want_diag)
        # the handle stays usable
        g.set_dets(dets)
        assert g.build(_capi.FP64)["nnz_upper"] > 0
        got, _ = g.find_new_dets(coeffs, 1e-3, True)
        np.testing.assert_array_equal(got, want)
