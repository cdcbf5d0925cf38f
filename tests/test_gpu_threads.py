"""Calls of different sizes from several threads, each with its own context: the launches of one kernel with
different amounts of shared memory do not get in one another's way, and the results are those of a single thread.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["plain", "chosen"])
def test_sizes_side_by_side(mode):
    from powerspectra_gpu import Context, synthetic as syn
    sizes = [100, 230, 400, 500, 600]  # no limit, and one, two, three or four blocks per SM
    Ws = [syn.mask_spectrum(2 * L + 1, 0.5, L / 2.0, seed=L) for L in sizes]
    want = [Context(0).mcm_multi({2: W, 3: W}, 0, L, mode=mode) for L, W in zip(sizes, Ws)]
    errors = []

    def work(k):
        try:
            ctx = Context(0)
            for _ in range(40):
                got = ctx.mcm_multi({2: Ws[k], 3: Ws[k]}, 0, sizes[k], mode=mode)
                for s in (2, 3):
                    assert np.array_equal(got[s], want[k][s])
        except BaseException as e:  # reported by the test's own thread
            errors.append((sizes[k], repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
