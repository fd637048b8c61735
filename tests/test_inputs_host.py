"""CPU checks of what calls refuse and which route an input takes: counts, arrays, precisions."""
import ctypes

import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _hafnian as H
from thewalrus_gb300 import _native as nat
from thewalrus_gb300.serving import GaussianState


def test_negative_counts_are_refused():
    """A photon count below zero has no factorial, whatever the others are."""
    state = GaussianState.synthetic(modes=4, seed=1)
    for pattern in ([1, -1, 0, 0], [-1, 3, 0, 0], np.array([2, 2, -2, 0])):
        with pytest.raises(ValueError):
            state.norm(pattern)
    assert abs(state.norm([2, 0, 3, 1]) - state.vacuum / np.sqrt(12)) <= 1e-15 * abs(state.vacuum)


def test_pairing_of_counts_of_any_size():
    """Counts up to the largest of 64 bits pair as smaller ones do; larger ones are refused, not cut."""
    big = 2 ** 63 - 1
    for reps in ([big, big], [big, 2 ** 62], [2 ** 62, 2 ** 62 + 1, 3], [big, 1, 1], [big]):
        x, m, odd = tw.matched_reps(reps)
        used = np.zeros(len(reps), dtype=object)
        for e, r in enumerate(m.tolist()):
            used[x[e]] += r
            used[x[e + len(m)]] += r
        if odd is not None:
            used[odd] += 1
        assert used.tolist() == reps
    for reps in ([2 ** 64], [2 ** 64 + 2, 1, 1], [1, 2 ** 70], np.array([2 ** 64 - 1], dtype=np.uint64)):
        with pytest.raises(OverflowError):
            tw.matched_reps(reps)


def test_direct_route_leaves_balancing_and_copies_to_the_general_one(monkeypatch):
    """Rows that balancing would scale although the unpaired vertex's entries hide it, and arrays whose numbers
    do not lie on their own boundaries, are not the direct route's."""
    seen = []
    monkeypatch.setattr(nat, "run", lambda insts, precision="fp64", stream=0: seen.append(insts[0]) or np.zeros(1))
    rng = np.random.default_rng(3)
    S = rng.normal(size=(7, 7))
    S = S + S.T
    d = np.array([1, 1e3, 1, 1e3, 1, 1e3, 1])  # pairs (6, 5), (4, 3), (2, 1), and 0 left over
    A = S * np.outer(d, d)
    A[0, 1:] = A[1:, 0] = 1e9
    assert H._pair_balance(H._sub(A, tw.matched_reps([1] * 7)[0])) is not None
    assert nat.hafnian_direct(A, True, 1e-5, 1e-8) is None
    raw = np.zeros(8 * 36 + 1, dtype=np.uint8)
    U = raw[1:].view(np.float64).reshape(6, 6)
    U[:] = S[:6, :6]
    assert not U.flags.aligned and U.flags.c_contiguous
    called = []
    monkeypatch.setattr(nat, "hafnian_direct", lambda *a: called.append(a))
    tw.hafnian(U)
    assert not called and len(seen) == 1
    tw.hafnian(U.copy())
    assert len(called) == 1


def test_plans_take_one_precision():
    """Several primes at once are wg_run's; a plan refuses them as it does any other unknown precision."""
    lib = nat.load()
    opt = nat.WgPlanOptions()
    for code in [nat.WG_PREC_PRIMES + k for k in range(1, 6)] + [nat.WG_PREC_PRIMES + 3 | nat.WG_PREC_TERMS, 8, 99, -1]:
        h = ctypes.c_void_p()
        arr = (nat.WgInstance * 1)()
        assert lib.wg_plan_create_ex(arr, 0, code, ctypes.byref(opt), ctypes.byref(h)) == -1  # WG_EINVAL
        assert lib.wg_plan_create(arr, 0, code, 1.0, ctypes.byref(h)) == -1 and not h.value
        assert b"unknown precision" in lib.wg_last_error()
