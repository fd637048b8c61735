"""A served request is evaluated as the same loop hafnian alone: the choice of evaluation looks at the
request's own modes and not at the state they are taken from."""
import numpy as np
import pytest

import thewalrus_gb300 as tw
from thewalrus_gb300 import _native as nat
from thewalrus_gb300 import workloads as wl

pytestmark = pytest.mark.gpu

M = 36


def states():
    B = wl.complex_symmetric(M, seed=1) * 0.05
    gamma = B[0] * 2
    yield "coupled", B, gamma
    vacuum = B.copy()
    vacuum[M - 1, :] = vacuum[:, M - 1] = 0
    yield "one mode apart", vacuum, gamma
    halves = B.copy()
    halves[:14, 14:28] = halves[14:28, :14] = 0
    yield "two halves coupled by the other modes", halves, gamma
    rounded = B.copy()
    rounded[:28, :28] *= 1e-2
    rounded[0, 1] *= 1 + 1e-13  # not symmetric by 2^-48 of the modes' own entries, but of the whole matrix's
    yield "symmetric against other modes' entries", rounded, gamma
    infinite = B.copy()
    infinite[M - 1, 0] = infinite[0, M - 1] = np.inf
    infinite[M - 1, M - 1] = np.nan
    yield "another mode not finite", infinite, gamma


@pytest.mark.parametrize("name,B,gamma", list(states()), ids=lambda x: x if isinstance(x, str) else "")
@pytest.mark.parametrize("modes,rep", [(28, 1), (29, 1), (14, 2), (28, 2), (10, 1)])
def test_route_of_a_request(name, B, gamma, modes, rep):
    pattern = [rep] * modes + [0] * (M - modes)
    plan = nat.Plan.from_requests(nat.DeviceState(B, gamma), [tw.matched_reps(pattern)])
    with np.errstate(invalid="ignore"):
        alone = nat.Plan([tw.prepare_loop_hafnian(B[:modes, :modes].copy(), gamma[:modes].copy(), [rep] * modes)])
    assert plan.kernel_launches == alone.kernel_launches  # a tree reduces in its own launch, terms take two
    plan.execute()
    alone.execute()
    got, want = plan.read()[0], alone.read()[0]
    assert abs(got - want) <= 1e-13 * abs(want)
