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
