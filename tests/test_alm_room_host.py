"""The room for the partial sums of a mask spectrum: never less than the sums a call cuts its work into, and growing with
both limits, so that a call fits after any larger one.  The two rules are read from the source."""
import os
import re

from conftest import PKG


def _rules():
    src = open(os.path.join(PKG, "csrc", "ps_window.cu")).read()
    threads = int(re.search(r"kAlmThreads = (\d+)", src).group(1))
    most = int(re.search(r"kAlmChunk = (\d+)", open(os.path.join(PKG, "csrc", "ps_internal.cuh")).read()).group(1))
    least, blocks = map(int, re.search(r"chunk > (\d+) && .* < (\d+)\) chunk /= 2", src).groups())
    fine = int(re.search(r"fine = \(size_t\)(\d+) \* kAlmThreads", src).group(1))
    return threads, most, least, blocks, fine


def test_room_for_every_size():
    threads, most, least, blocks, fine = _rules()

    def chunk(mmax, lout):
        c = most
        while c > least and (lout + threads) // threads * (mmax // c + 1) < blocks:
            c //= 2
        return c

    def room(mmax, lout):
        return max((mmax // most + 1) * (lout + 1), fine * threads)

    sizes = list(range(0, 300, 7)) + [255, 256, 257, 511, 512, 513, 1000, 1023, 1024, 1200, 2047, 2508, 4095, 8191, 65535]
    for lout in sizes:
        last = 0
        for mmax in sorted(sizes):
            r = room(mmax, lout)
            assert (mmax // chunk(mmax, lout) + 1) * (lout + 1) <= r
            assert r >= last
            last = r
