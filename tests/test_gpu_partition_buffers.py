"""What a partitioned handle passes to the caller's reduce function."""
import numpy as np
import pytest

from risq_b200 import GpuHam, _capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [_capi.FP64_UPPER, _capi.MIXED_UPPER])
@pytest.mark.parametrize("lists", [False, True])
def test_reduced_buffers_can_be_shared(prec, lists, monkeypatch):
    """They are plain device allocations, which other processes and GPUs can open."""
    from cuda.bindings import driver

    attr = driver.CUpointer_attribute.CU_POINTER_ATTRIBUTE_IS_LEGACY_CUDA_IPC_CAPABLE
    seen = []

    def reduce(ptr, count, stream, user):
        err, ok = driver.cuPointerGetAttribute(attr, ptr)
        seen.append((int(count), int(err) == 0 and bool(ok)))
        return 0

    if lists:
        monkeypatch.setenv("RISQGPU_TEST_TILE_OOM", "1")
    ints, _, dets, coeffs, diag, _ = H.synthetic_hci(10, 4, 1e-3)
    fn = _capi.ALLREDUCE_FN(reduce)
    with GpuHam(ints) as g:
        g.set_partition(0, 2, fn)
        g.set_dets(dets, 0, diag)
        g.build(prec)
        builds = len(seen)
        g.matrix_vector_prod(coeffs)
    assert builds >= 2 and len(seen) == builds + 1
    assert seen[-1][0] == len(dets)
    assert all(ok for _, ok in seen), seen
