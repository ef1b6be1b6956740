"""Row sigma of sets with more rows than the chip holds warps and few elements a row."""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals
from tests import helpers as H
from tests.test_gpu_memory import full_space

pytestmark = pytest.mark.gpu


# elements a row, on average: 53, 61, 111, 168 and 214, on both sides of the lines between the
# kernels, or hardly any
@pytest.mark.parametrize("n,lo,hi", [(4737, 0, 96), (5401, 0, 96), (10003, 96, 192), (15007, 96, 192), (19001, 192, 400)])
@pytest.mark.parametrize("sparse", [False, True])
def test_short_rows_match_oracle(n, lo, hi, sparse):
    import torch

    rng = np.random.default_rng(n)
    if sparse:  # hardly any connections
        norb = 30
        dets = np.zeros((n, 4), dtype=np.uint64)
        orbs = np.argsort(rng.random((n, 2, norb)), axis=2)[:, :, :7].astype(np.uint64)
        dets[:, ::2] = (np.uint64(1) << orbs).sum(axis=2, dtype=np.uint64)
        dets = np.unique(dets, axis=0)
        n = len(dets)
    else:
        norb = 14
        s = full_space(norb, 3)
        dets = s[rng.permutation(len(s))[:n]]
    ints = synthetic_integrals(norb, 1)
    with GpuHam(ints) as g:
        diag = g.ham_diag(dets)
    sp = O.Sparse().build(H.oracle_ham(ints), dets, diag, 0, builder=_capi.BUILDER_FAST)
    rp, cols, vals, _ = sp.export()
    if not sparse:
        assert lo < 2 * len(vals) / n <= hi
    x = rng.standard_normal(n)
    ref = sp.mv(x)
    rows = np.repeat(np.arange(n), np.diff(rp))
    mag = np.abs(diag * x)
    np.add.at(mag, rows, np.abs(vals * x[cols]))
    np.add.at(mag, cols, np.abs(vals * x[rows]))
    terms = 2 + np.bincount(rows, minlength=n) + np.bincount(cols, minlength=n)
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        for prec in (_capi.FP64, _capi.MIXED):
            g.build(prec, _capi.BUILDER_FAST)
            y = g.matrix_vector_prod(x)
            # both sides sum in FP64 in some order; MIXED values carry at least 2^-46
            assert np.all(np.abs(y - ref) <= (2 * terms * 2.0 ** -53 + 2.0 ** -46) * mag)
        order = np.lexsort((dets[:, 2], dets[:, 0]))  # internal order: by (up, dn)
        xd = torch.tensor(x[order], dtype=torch.float32, device="cuda")
        yd = torch.full_like(xd, float("nan"))
        torch.cuda.synchronize()
        g.sigma_device(xd.data_ptr(), yd.data_ptr(), 1)
        bound = (terms + 3) * 2.0 ** -24 * mag[order]
        assert np.all(np.abs(yd.double().cpu().numpy() - ref[order]) <= bound)
