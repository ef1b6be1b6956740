"""Selection under a memory bound that holds the excitation lists but not their sorting."""
import numpy as np
import pytest

from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nel,ncore", [(12, 6, 0), (20, 8, 0), (20, 8, 3)])
def test_lists_sorted_on_the_host_are_the_same(norb, nel, ncore):
    ints, _, dets, coeffs, _, _ = H.synthetic_hci(norb, nel, 3e-3)
    dets, coeffs = dets[:900], coeffs[:900]
    nv = norb - ncore
    entries = nv * nv * (nv - 1) ** 2 + nv * (nv - 1) // 2 * ((nv - 2) * (nv - 3) // 2)
    with GpuHam(ints) as g:
        g.set_dets(dets)
        used, _ = g.memory_used()
        want, want_diag = g.find_new_dets(coeffs, 1e-3, True, ncore)
        assert len(want) > 0
        # 10 bytes an entry leave nothing for the step itself
        g.set_memory_limit(used + 10 * entries + 1)
        with pytest.raises(_capi.RisqGpuError) as e:
            g.find_new_dets(coeffs, 1e-3, True, ncore)
        assert e.value.code == _capi.ERR_OOM and g.memory_used()[0] < used + 10 * entries
        lo, hi = used, used + (1 << 28)
        while hi - lo > 4096:  # the smallest bound that is enough
            mid = (lo + hi) // 2
            g.set_memory_limit(mid)
            try:
                got, got_diag = g.find_new_dets(coeffs, 1e-3, True, ncore)
                np.testing.assert_array_equal(got, want)
                np.testing.assert_array_equal(got_diag, want_diag)
                hi = mid
            except _capi.RisqGpuError as err:
                assert err.code == _capi.ERR_OOM
                lo = mid


def test_a_bound_of_the_lists_is_enough():
    """64 orbitals, two determinants: the lists, 10 bytes an entry, are all but 2 MB of it."""
    norb = 64
    ints = synthetic_integrals(norb, 1)
    dets = np.zeros((2, 4), dtype=np.uint64)
    dets[:, 0], dets[:, 2] = [0b11, 0b101], [0b11, 0b101]
    coeffs = np.array([1.0, 0.1])
    entries = norb ** 2 * (norb - 1) ** 2 + norb * (norb - 1) // 2 * ((norb - 2) * (norb - 3) // 2)
    with GpuHam(ints) as g:
        g.set_dets(dets)
        want, want_diag = g.find_new_dets(coeffs, 1e-2, True)
        assert len(want) > 0
        used, _ = g.memory_used()
        g.set_memory_limit(used + 10 * entries + (2 << 20))
        got, got_diag = g.find_new_dets(coeffs, 1e-2, True)
        np.testing.assert_array_equal(got, want)
        np.testing.assert_array_equal(got_diag, want_diag)
