"""The FP64 pair potential of the diagnostics at the edges of its row blocks (128, 256 and 512 particles, from 12,288 and
24,576 particles up) and for odd and even block counts, against the FP64 oracle. Both sum the same positive terms in
FP64; a plain sum of n (n - 1) / 2 <= 3e8 of them drifts by up to sqrt(3e8) 2^-53 = 2e-12: 1e-11 of the sum."""

import numpy as np
import pytest

from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import f32_exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 256, 257, 384, 1000, 12287, 12289, 24577])
def test_potential_vs_oracle(oracle, n, precision):
    p = make_params(switches=("SELF_GRAVITY",), H=0.05, grav_eps=0.02, fixed_dt=1e-3)
    st = f32_exact(ics.plummer_sphere(n, seed=n))
    st["mass"] = (st["mass"] * np.random.default_rng(n).uniform(0.5, 2.0, n)).astype(np.float32).astype(np.float64)
    want = oracle.diagnostics(p, st)
    with DeviceParticleBuffer(p, n, make_options(precision=precision)) as pb:
        (pb.upload_f64 if precision == "double" else pb.upload)(st)
        got = pb.diagnostics()
    if n == 1:
        assert got["e_grav"] == 0.0
    else:
        assert abs(got["e_grav"] - want["e_grav"]) <= 1e-11 * abs(want["e_grav"])
    assert abs(got["mass"] - want["mass"]) <= 1e-13 * want["mass"]


def test_unsoftened_potential_of_coincident_particles(oracle):
    """eps = 0: the self pair is left out by its index, and two particles in one place give -infinity, across blocks
    and within one."""
    p = make_params(switches=("SELF_GRAVITY",), H=0.05, grav_eps=0.0, fixed_dt=1e-3)
    st = f32_exact(ics.plummer_sphere(700, seed=1))
    with DeviceParticleBuffer(p, 700) as pb:
        pb.upload(st)
        e = pb.diagnostics()["e_grav"]
        want = oracle.diagnostics(p, st)["e_grav"]
        assert abs(e - want) <= 1e-11 * abs(want)
        for a, b in ((3, 650), (3, 9)):
            two = {k: v.copy() for k, v in st.items()}
            two["pos"][b] = two["pos"][a]
            pb.upload(two)
            assert pb.diagnostics()["e_grav"] == -np.inf
