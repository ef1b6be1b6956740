"""Device memory between builds: what is kept, what is counted, and when it goes back."""
import itertools
import threading

import numpy as np
import pytest

from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def strings(norb, nel):
    return np.array([sum(1 << o for o in c) for c in itertools.combinations(range(norb), nel)], dtype=np.uint64)


def full_space(norb, nel):
    s = strings(norb, nel)
    d = np.zeros((len(s) ** 2, 4), dtype=np.uint64)
    d[:, 0], d[:, 2] = np.repeat(s, len(s)), np.tile(s, len(s))
    return d


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_a_large_matrix_stays_for_the_next_build_and_then_goes():
    """853,776 determinants, 18.6 GB of FP64 rows."""
    ints = synthetic_integrals(12, 1)
    dets = full_space(12, 6)
    small = dets[:2000]
    x = np.random.default_rng(0).standard_normal(len(dets))
    free_bytes()  # torch's own context
    with GpuHam(ints) as g:
        g.release_memory()
        f0 = free_bytes()
        g.set_dets(small)
        g.build(_capi.FP64)
        want = g.matrix_vector_prod(x[:2000])
        g.set_dets(dets)
        g.build(_capi.FP64)
        used, _ = g.memory_used()
        f1 = free_bytes()
        assert used > 18 * GIB * 0.9
        assert f0 - f1 < used + 8.5 * GIB  # buffers, and the idle memory that may be kept
        y = g.matrix_vector_prod(x)
        # dropped, but kept until the next build: nothing is unmapped here and mapped again there
        g.set_dets(dets[:-100])
        assert g.memory_used()[0] < used / 4
        assert free_bytes() - f1 < GIB
        g.build(_capi.FP64)
        assert free_bytes() - f1 < GIB
        # the next build returns what it did not use, down to what may be kept idle
        g.set_dets(small)
        g.build(_capi.FP64)
        assert f0 - free_bytes() < 8.5 * GIB
        np.testing.assert_array_equal(g.matrix_vector_prod(x[:2000]), want)
        g.release_memory()
        assert f0 - free_bytes() < GIB
        np.testing.assert_array_equal(g.matrix_vector_prod(x[:2000]), want)


def test_release_after_a_dropped_matrix():
    ints = synthetic_integrals(12, 1)
    dets = full_space(12, 6)
    free_bytes()
    with GpuHam(ints) as g:
        g.release_memory()
        f0 = free_bytes()
        g.set_dets(dets)
        g.build(_capi.FP64)
        g.set_dets(dets[:2000])
        g.release_memory()
        assert f0 - free_bytes() < GIB
        g.set_dets(dets)
        g.build(_capi.FP64)
        bad = np.concatenate([dets[:5], dets[:1]])
        with pytest.raises(_capi.RisqGpuError):
            g.set_dets(bad)  # refused: no build will follow
        assert f0 - free_bytes() < 8.5 * GIB


def test_handles_on_streams_and_threads_share_blocks():
    """Two threads with a handle each, rebuilding sets whose blocks fit one another's, on their
    own and on caller streams, one with a memory bound half of the time."""
    import torch

    ints = synthetic_integrals(12, 2)
    dets = full_space(12, 6)
    sets = [dets[:60001], dets[:62003], dets[20000:80001]]
    xs = [np.random.default_rng(k).standard_normal(len(d)) for k, d in enumerate(sets)]
    want = []
    with GpuHam(ints) as g:
        for d, x in zip(sets, xs):
            for prec in (_capi.FP64, _capi.MIXED_UPPER):
                g.set_dets(d)
                g.build(prec)
                want.append(g.matrix_vector_prod(x))
    errors = []

    def work(seed):
        try:
            rng = np.random.default_rng(seed)
            s = torch.cuda.Stream()
            with GpuHam(ints) as g:
                for _ in range(8):
                    k, p = int(rng.integers(3)), int(rng.integers(2))
                    if seed == 1:
                        g.set_memory_limit(int(rng.integers(2)) * 20 * GIB)
                    g.set_stream(s.cuda_stream if rng.integers(2) else None)
                    g.set_dets(sets[k])
                    g.build((_capi.FP64, _capi.MIXED_UPPER)[p])
                    g.set_stream(s.cuda_stream if rng.integers(2) else None)  # with a live matrix
                    np.testing.assert_array_equal(g.matrix_vector_prod(xs[k]), want[2 * k + p])
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]
