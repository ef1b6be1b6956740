"""One selection step at the edges of its lists, its caches and its determinant table.

Two orbitals (refused) and three, a valence space of one orbital below the core's edge,
strings of one and of two words (above 64 orbitals membership is a binary search), and
lists of more than 32 entries.
"""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nel,ncore,eps,steps", [
    (2, 1, 0, 1e-4, 3), (3, 1, 0, 1e-4, 3), (5, 2, 0, 1e-3, 4), (6, 3, 2, 1e-3, 4), (9, 4, 3, 1e-4, 4),
    (33, 3, 0, 2e-2, 3), (64, 2, 1, 3e-2, 2), (65, 2, 0, 3e-2, 2), (70, 2, 1, 3e-2, 2)])
def test_find_new_dets_matches_oracle(n, nel, ncore, eps, steps):
    ints = synthetic_integrals(n, n)
    hci = O.Hci(H.oracle_ham(ints, ncore), nel, nel, eps)
    states = [hci.export()]
    for _ in range(steps):
        done = hci.step()
        states.append(hci.export())
        if done:
            break
    log = hci.log()
    d_fin, _, g_fin = states[-1]
    with GpuHam(ints) as gpu:
        for k in range(min(len(log), len(states))):
            d, c, g = states[k]
            gpu.set_dets(d, 0, g)
            if nel > n - 2:  # no orbital left besides i and r for each other electron
                with pytest.raises(_capi.RisqGpuError):
                    gpu.find_new_dets(c, eps, True, ncore)
                return
            nd, ng = gpu.find_new_dets(c, log[k]["eps"], log[k]["eps"] == eps, ncore)
            # whole numbers and the diagonal's fixed order of sums: equal
            np.testing.assert_array_equal(nd, d_fin[len(d):log[k]["ndets"]])
            np.testing.assert_array_equal(ng, g_fin[len(d):log[k]["ndets"]])
