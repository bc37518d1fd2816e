"""Truncations by host threads with a context each, at the same time."""
import threading

import numpy as np
import pytest

from qcmaquis_b200 import dmrg, heff

pytestmark = pytest.mark.gpu


def test_threads_with_a_context_each():
    """Blocks of unlike sizes above 420 columns (whose rotations are logged, with shared memory by the block's size):
    each thread gets what it gets alone, to the bit."""
    sizes = [1000, 430, 560, 430]
    blocks = [np.random.default_rng(k).standard_normal((n, n)) for k, n in enumerate(sizes)]
    alone = [dmrg.truncate_svd(heff.Context(0), [b], 10 ** 6, 1e-30)[0][0] for b in blocks]
    start = threading.Barrier(len(sizes))
    wrong = []

    def work(k):
        try:
            ctx = heff.Context(0)
            start.wait(60)
            for _ in range(12 if sizes[k] == 1000 else 40):
                got = dmrg.truncate_svd(ctx, [blocks[k]], 10 ** 6, 1e-30)[0][0]
                if not all(np.array_equal(x, y) for x, y in zip(got, alone[k])):
                    wrong.append((k, "other values"))
        except Exception as e:  # reported by the test's own thread
            wrong.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
