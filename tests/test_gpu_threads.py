"""Calls of several threads at once, whose launches ask for different amounts of shared memory."""
import threading

import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["dd", "dd-terms"])
def test_launches_of_different_shared_memory(precision):
    A, D = wl.complex_symmetric(10, seed=9), wl.complex_symmetric(10, seed=5)[0] * 0.5
    insts = [tw.prepare_loop_hafnian_batch(A[:m, :m], D[:m], [1] * (m - 1), cutoff)
             for m, cutoff in ((10, 15), (10, 9), (6, 12), (8, 15))]
    want = [nat.run([i], precision) for i in insts]
    start, wrong = threading.Barrier(len(insts)), []

    def calls(k):
        start.wait()
        for _ in range(400):
            try:
                if not np.array_equal(nat.run([insts[k]], precision), want[k]):
                    wrong.append(k)
            except RuntimeError as e:
                wrong.append(e)

    threads = [threading.Thread(target=calls, args=(k,)) for k in range(len(insts))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
