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
