"""The device memory of the elimination trees' levels: a plan's option, the server's budget.

A tree within less memory walks smaller blocks, so that its sum is taken in another order: equal to
1e-12, a hundred roundings of these sums; one that does not fit is the per-term sum, bit for bit."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu


def run(insts, precision="fp64", **options):
    plan = nat.Plan(insts, precision=precision, **options)
    plan.execute()
    got, size = plan.read(), plan.device_bytes()
    plan.close()
    return got, size


@pytest.mark.parametrize("limit", [100e6, 20e6, 4e6])
def test_blocks_within_a_limit(limit):
    A, g, rpt = wl.gaussian_state_loop(modes=12, seed=2, photons=20, max_rep=3)
    insts = [tw.prepare_hafnian(wl.complex_symmetric(32, seed=1)), tw.prepare_hafnian(wl.real_nonneg(30, seed=1)),
             tw.prepare_hafnian(wl.complex_symmetric(20, seed=2)), tw.prepare_loop_hafnian(A, g, list(rpt)),
             tw.prepare_loop_hafnian(wl.complex_symmetric(25, seed=3), wl.complex_symmetric(25, seed=4)[0])]
    want, most = run(insts)
    got, size = run(insts, max_workspace=limit)
    assert most > limit and size < limit + 8e6  # programs, matrices and partials beside the levels
    assert np.all(np.abs(got - want) <= 1e-12 * np.abs(want))


def test_no_room_is_the_per_term_sum():
    insts = [tw.prepare_hafnian(wl.complex_symmetric(22, seed=1)), tw.prepare_hafnian(wl.real_nonneg(24, seed=1))]
    got, size = run(insts, max_workspace=1)
    assert size < 8e6 and np.array_equal(got, run(insts, "fp64-terms")[0])


@pytest.mark.parametrize("budget", [2e6, 30e6, 300e6])
def test_served_within_the_budget(budget, monkeypatch):
    """All plans that a server holds at a time, their trees included, stay within its budget."""
    pytest.importorskip("torch")
    from thewalrus_gb300.serving import GaussianState, ProbabilityServer, poisson_requests

    held = {"now": 0, "most": 0}

    class Counted(nat.Plan):
        @classmethod
        def from_requests(cls, *args, **options):
            plan = super().from_requests(*args, **options)
            held["now"] += plan.device_bytes()
            held["most"] = max(held["most"], held["now"])
            return plan

        def close(self):
            if self.handle:
                held["now"] -= self.device_bytes()
            super().close()

    states = [GaussianState.synthetic(modes=32, seed=3)]
    reqs = poisson_requests(states, rate=1e6, count=24, photons=(8, 28), seed=1, max_rep=1)
    want = [r["amplitude"] for r in ProbabilityServer(states).serve(reqs)]
    monkeypatch.setattr(nat, "Plan", Counted)
    got = [r["amplitude"] for r in ProbabilityServer(states, mem_budget=budget).serve(reqs)]
    assert 0 < held["most"] <= budget and held["now"] == 0
    assert np.all(np.abs(np.array(got) - want) <= 1e-10 * np.abs(want))


def test_estimate_of_a_request():
    """What the server counts for a request is at least what its per-term plan takes."""
    pytest.importorskip("torch")
    from thewalrus_gb300.serving import GaussianState, ProbabilityServer

    state = GaussianState.synthetic(modes=48, seed=3).to_device()
    for photons in (2, 5, 10, 16, 24, 27, 28, 33, 36, 40, 44, 47):
        for rep in (1, 2, 4):
            p = np.zeros(48, dtype=np.int64)
            p[:-(-photons // rep)] = rep
            p[0] -= p.sum() - photons
            plan = nat.Plan.from_requests(state, [tw.matched_reps(p)], "fp64-terms")
            assert plan.device_bytes() <= ProbabilityServer.estimate_bytes(photons), (photons, rep)
            plan.close()


@pytest.fixture
def small_pool():
    """A function that makes the device's stream-ordered allocations come from a pool of so many bytes."""
    import ctypes

    class Props(ctypes.Structure):  # CUmemPoolProps
        _fields_ = [("alloc_type", ctypes.c_int), ("handle_types", ctypes.c_int), ("location_type", ctypes.c_int),
                    ("location_id", ctypes.c_int), ("security", ctypes.c_void_p), ("max_size", ctypes.c_size_t),
                    ("usage", ctypes.c_ushort), ("reserved", ctypes.c_ubyte * 54)]

    nat.run([tw.prepare_hafnian(wl.real_nonneg(4, seed=1))])  # the library's context
    cuda = ctypes.CDLL("libcuda.so.1")
    dev, default, made = ctypes.c_int(), ctypes.c_void_p(), []
    assert cuda.cuCtxGetDevice(ctypes.byref(dev)) == 0
    assert cuda.cuDeviceGetDefaultMemPool(ctypes.byref(default), dev) == 0

    def use(size):
        pool, props = ctypes.c_void_p(), Props(1, 0, 1, dev.value, None, int(size))  # pinned, on the device
        if cuda.cuMemPoolCreate(ctypes.byref(pool), ctypes.byref(props)) != 0:
            pytest.skip("no memory pool of a bounded size")
        made.append(pool)
        assert cuda.cuDeviceSetMemPool(dev, pool) == 0

    yield use
    assert cuda.cuDeviceSetMemPool(dev, default) == 0
    for pool in made:
        cuda.cuMemPoolDestroy(pool)


def test_allocation_that_fails_is_tried_with_less(small_pool):
    insts = [tw.prepare_hafnian(wl.complex_symmetric(34, seed=1)), tw.prepare_hafnian(wl.complex_symmetric(20, seed=2))]
    want = nat.run(insts)
    small_pool(256e6)  # smaller blocks
    assert np.all(np.abs(nat.run(insts) - want) <= 1e-12 * np.abs(want))
    last = [tw.prepare_hafnian(wl.complex_symmetric(30, seed=3))]
    small_pool(32e6)  # no tree
    assert np.array_equal(nat.run(last), nat.run(last, "fp64-terms"))


@pytest.mark.parametrize("reps", [[2] * 21, [1] + [2] * 20, [3] * 14, [1] * 30])
def test_plan_of_a_small_and_a_huge_member(reps):
    """A member of hours beside one whose multiple edge may be taken as copies: the plan is made (its estimates
    had divided by zero) and not run."""
    huge = nat.Instance(nat.WG_KIND_PLAIN, wl.real_nonneg(2 * len(reps), seed=1) * 0.1, np.array(reps, dtype=np.int64))
    plan = nat.Plan([tw.prepare_hafnian(wl.real_nonneg(2, seed=1), [2, 2]), huge])
    assert plan.total_out == 2
    plan.close()
