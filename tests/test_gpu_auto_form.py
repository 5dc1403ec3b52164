"""Which gravity kernel AUTO picks in the smallest contexts, on both sides of the rule, and that the symmetric one, asked for,
is right there too. Reference and bounds: test_gpu_gravity_shapes.py."""

import numpy as np
import pytest

from grasph2_b200 import ics
from grasph2_b200.params import make_params
from helpers import f32_exact
from test_gpu_gravity_shapes import accel, check, masses

pytestmark = pytest.mark.gpu
TOL = {"plain": 4e-6, "compensated": 2e-6}


def state(n, kind):
    st = ics.plummer_sphere(n, seed=n)
    st["mass"] = masses(kind, n, np.random.default_rng(n))
    return f32_exact(st), make_params(switches=("SELF_GRAVITY",), H=0.05, grav_eps=0.01, fixed_dt=1e-3)


@pytest.mark.parametrize("accum,n,symmetric", [("plain", 1, False), ("plain", 3072, False), ("plain", 3073, True),
                                               ("compensated", 2048, False), ("compensated", 2049, True)])
def test_auto(n, accum, symmetric):
    st, p = state(n, "different")
    got, groups = accel(p, st, accum=accum)
    assert (groups > 0) == symmetric
    check(got, st, 0.01, TOL[accum])


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("kind", ["equal", "two", "different", "massless"])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1025, 2048, 3072])
def test_symmetric_asked_for(n, kind, accum):
    st, p = state(n, kind)
    got, groups = accel(p, st, accum=accum, gravity="symmetric")
    assert groups > 0
    check(got, st, 0.01, TOL[accum])
