"""The ensemble's box search and group-pair gravity at the edges of their groups (512 particles) and boxes (32), against
the one-sided sweep: the same neighbours, the same FP32 terms in another order. Bounds: 1e-6 of a density's largest
value, 1e-5 of an acceleration's (the parity bounds), 1e-5 of the rates."""

import numpy as np
import pytest

import ref_variants
from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import Ensemble, pack_states
from helpers import f32_exact, rel_max

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 33, 511, 512, 513, 1023, 1300, 2, 1600]


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("name,masses,h", [("fluid", "equal", 0.3), ("solid", "equal", 0.42), ("solid", "different", 0.42),
                                           ("fluid", "different", 3.0)])
def test_near_form_equals_the_sweep(name, masses, h, accum):
    """h = 3: more neighbours than list slots in the larger simulations."""
    p = make_params(**dict(ref_variants.params_dict(ref_variants.VARIANTS[name]), H=h, grav_eps=0.02))
    rng = np.random.default_rng(1)
    states = []
    for k, n in enumerate(SIZES):
        st = ics.uniform_sphere(n, radius=1.0, rho0=1.0, omega=(0.1, 0.0, 0.2), seed=k)
        if masses == "different":
            st["mass"] *= rng.uniform(0.2, 5.0, n)
        states.append(f32_exact(st))
    st = pack_states(states)
    out = []
    for form in ("auto", "one-sided"):
        with Ensemble(p, SIZES, make_options(accum=accum, gravity=form)) as ens:
            ens.upload(st)
            ens.compute_derivatives()
            out.append(ens.split(ens.download()))
    for n, got, want in zip(SIZES, *out):
        for k, tol in (("density", 1e-6), ("acc", 1e-5), ("dstress_dt", 1e-5)):
            if want[k].any():
                assert np.isfinite(got[k]).all() and rel_max(got[k], want[k]) <= tol, (n, k, rel_max(got[k], want[k]))
