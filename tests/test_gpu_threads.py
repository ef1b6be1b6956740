"""Handles of very different sizes in threads of one process."""
import threading

import pytest

from risq_b200 import GpuHam, _capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


def test_kernels_of_different_shared_memory_in_two_threads():
    """A large set's FP64 sigma takes 64 KB of shared memory a CTA, a small one's 4 KB: the calls of
    one thread must not take the permission from the other."""
    import torch

    small = H.synthetic_hci(10, 4, 1e-3)
    large = H.synthetic_hci(12, 6, 1e-4)
    errors, stop = [], threading.Event()

    def work(sys, rounds):
        try:
            ints, _, dets, coeffs, diag, _ = sys
            with GpuHam(ints) as g:
                g.set_dets(dets, 0, diag)
                g.build(_capi.MIXED_UPPER)
                x = torch.tensor(coeffs, device="cuda")
                want, y = torch.empty_like(x), torch.empty_like(x)
                g.sigma_device(x.data_ptr(), want.data_ptr(), 0)
                for k in range(rounds):
                    g.sigma_device(x.data_ptr(), y.data_ptr(), 0)
                    if k % 100 == 0:
                        assert torch.equal(y, want)
                    if stop.is_set():
                        break
        except BaseException as e:  # noqa: BLE001
            errors.append(e)
        stop.set()

    threads = [threading.Thread(target=work, args=a) for a in ((small, 20000), (large, 4000))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
