"""Magnitudes, partials and chunks of plans whose sums are taken by trees: asked for on another stream
than the plan was made on, from several threads, and again without an execution between."""
import threading
import time

import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def state_and_requests(count=12, modes=24):
    B = wl.complex_symmetric(modes, seed=1) * 0.05
    patterns = [[1] * (4 + k) + [0] * (modes - 4 - k) for k in range(count)]
    return nat.DeviceState(B, B[0] * 2), [tw.matched_reps(p) for p in patterns]


def test_queries_on_another_stream():
    """A plan made and executed on its own stream, its queries on the default one."""
    torch = pytest.importorskip("torch")
    state, triples = state_and_requests()
    terms = nat.Plan.from_requests(state, triples, "fp64-terms")
    terms.execute()
    want, parts = terms.read_magnitudes(), terms.partials()
    for order in range(3):
        s = torch.cuda.Stream()
        plan = nat.Plan.from_requests(state, triples, "fp64", stream=s.cuda_stream)
        plan.execute(s.cuda_stream)
        if order == 0:
            plan.read(s.cuda_stream)
        if order == 1:  # nothing waited for the plan's stream
            assert np.array_equal(plan.partials()[0], parts[0])
        assert np.array_equal(plan.read_magnitudes(), want)
        assert np.array_equal(plan.partials()[0], parts[0]) and plan.partials()[1] == parts[1]
        plan.read(s.cuda_stream)
        plan.close()


def test_queries_from_several_threads():
    insts = [tw.prepare_hafnian(wl.complex_symmetric(n, seed=n)) for n in (20, 24, 26)]
    terms = nat.Plan(insts, precision="fp64-terms")
    terms.execute()
    want, parts = terms.read_magnitudes(), terms.partials()
    for _ in range(5):
        plan = nat.Plan(insts)
        plan.execute()
        plan.read()
        wrong = []

        def ask(k):
            if k % 2:
                got = plan.partials()
                if not (np.array_equal(got[0], parts[0]) and got[1] == parts[1]):
                    wrong.append(k)
            elif not np.array_equal(plan.read_magnitudes(), want):
                wrong.append(k)

        threads = [threading.Thread(target=ask, args=(k,)) for k in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not wrong
        plan.close()


def test_asked_again_is_a_copy():
    """The terms are summed for an execution once: asking again costs a copy (some 20 us) and not the per-term
    sum (6 ms here)."""
    inst = tw.prepare_hafnian(wl.complex_symmetric(32, seed=1))
    plan = nat.Plan([inst])
    for _ in range(2):
        plan.execute()
        plan.read()
        t0 = time.perf_counter()
        first = plan.read_magnitudes()
        t1 = time.perf_counter()
        again = [time.perf_counter()]
        for _ in range(5):
            assert np.array_equal(plan.read_magnitudes(), first)
            again.append(time.perf_counter())
        assert min(np.diff(again)) < 0.1 * (t1 - t0)
