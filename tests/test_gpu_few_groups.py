"""The culled SPH passes on both sides of the size from which a neighbour list is one warp's (28,672 particles), and the
all-pairs passes, against the double-precision context of the same state. The two sum the same terms in different orders,
so the error of one is bounded by that of the other: at most four times it (two maxima over 28,672 values of the same
distribution), or the parity bounds, 1e-6 of the density and 1e-5 of rates and accelerations (per field maximum)."""

import numpy as np
import pytest

import ref_variants
from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import f32_exact, rel_max

pytestmark = pytest.mark.gpu
TOL = {"density": 1e-6, "acc": 1e-5, "dstress_dt": 1e-5, "density_dt": 1e-5, "balsara": 1e-5}


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("name", ["solid", "solid_mc", "fluid_full"])
@pytest.mark.parametrize("n", [33, 28672, 28673])
def test_both_sides_of_the_split(name, n, accum):
    h = 2.5 * n ** (-1.0 / 3.0)
    p = make_params(**dict(ref_variants.params_dict(ref_variants.VARIANTS[name]), H=h, normalsep=0.3 * h))
    st = ics.uniform_sphere(n, radius=1.0, rho0=1.0, omega=(0.1, 0.2, 0.3), seed=n)
    rng = np.random.default_rng(n)
    st["vel"] += rng.normal(0.0, 0.05, (n, 3))
    s = rng.normal(0.0, 0.01, (n, 3, 3))
    st["dstress"][:] = s + s.transpose(0, 2, 1)
    st = f32_exact(st)
    out = []
    for opt in ({"cull": True, "accum": accum}, {"cull": False, "accum": accum}, {"precision": "double"}):
        with DeviceParticleBuffer(p, n, make_options(**opt)) as pb:
            pb.upload(st)
            pb.compute_derivatives()
            out.append(pb.download())
    culled, pairs, exact = out
    for k, tol in TOL.items():
        assert np.isfinite(exact[k]).all()
        err, ref = rel_max(culled[k], exact[k]), rel_max(pairs[k], exact[k])
        assert err <= max(tol, 4.0 * ref), (k, err, ref)
