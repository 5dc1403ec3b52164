"""The culled SPH passes beyond the sizes of test_gpu_parity.py: incomplete neighbour lists, with and without a density
pass, and the fixed-order derivatives of network proposals against the plain ones (same terms, another order of
summation: the parity bounds 1e-6 for the density and 1e-5 for rates and accelerations, per field maximum)."""

import numpy as np
import pytest

import ref_variants
from grasph2_b200 import ics
from grasph2_b200 import surrogate as S
from grasph2_b200.mlp import init_params
from grasph2_b200.params import impact_params, make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import f32_exact, rel_max

pytestmark = pytest.mark.gpu
TOL = {"density": 1e-6, "acc": 1e-5, "dstress_dt": 1e-5, "density_dt": 1e-5, "balsara": 1e-5}


def check(got, want):
    for k, tol in TOL.items():
        assert np.isfinite(want[k]).all() and rel_max(got[k], want[k]) <= tol, (k, rel_max(got[k], want[k]))


def state(n, seed):
    st = ics.uniform_sphere(n, radius=1.0, rho0=1.0, omega=(0.1, 0.2, 0.3), seed=seed)
    rng = np.random.default_rng(seed)
    st["vel"] += rng.normal(0.0, 0.05, (n, 3))
    s = rng.normal(0.0, 0.01, (n, 3, 3))
    st["dstress"][:] = s + s.transpose(0, 2, 1)
    return f32_exact(st)


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("name,h", [("solid", 3.0), ("solid", 1.2), ("solid_mc", 1.2), ("fluid_full", 1.2)])
def test_incomplete_neighbour_lists(name, h, accum):
    """h = 3: everybody neighbours everybody; h = 1.2: lists of some shares are complete and others are not."""
    p = make_params(**dict(ref_variants.params_dict(ref_variants.VARIANTS[name]), H=h, normalsep=0.3 * h))
    st = state(1500, 5)
    out = []
    for cull in (True, False):
        with DeviceParticleBuffer(p, 1500, make_options(cull=cull, accum=accum)) as pb:
            pb.upload(st)
            pb.compute_derivatives()
            out.append(pb.download())
    check(*out)


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("n", [1000, 29250])
def test_proposal_derivatives_equal_the_plain_ones(n, accum):
    """A proposal's derivatives (one-sided and symmetric gravity) against gsph_compute_derivatives of the same state, and
    twice the same bits; an extrapolation without the network takes the plain ones."""
    nb = round(n * 8 / 9)
    p = impact_params(nb, n - nb)
    st = f32_exact(ics.two_sphere_impact(nb, n - nb, v_rel=0.5, y_offset=0.3, seed=n))
    sur = S.Surrogate(8, init_params(1), None, None, np.zeros(13), np.full(13, 1e-9))
    with DeviceParticleBuffer(p, n, make_options(accum=accum)) as pb:
        pb.upload(st)
        pb.compute_derivatives()
        want = pb.download()
        got = []
        for use_net in (True, True, False):
            pb.upload(st)
            sur.propose(pb, use_net=use_net)
            got.append(pb.download())
        for k in ("acc", "dstress_dt"):
            np.testing.assert_array_equal(got[0][k], got[1][k], err_msg=k)
            np.testing.assert_array_equal(got[2][k], want[k], err_msg=k)
    for k in ("acc", "dstress_dt"):
        assert rel_max(got[0][k], want[k]) <= TOL[k], (k, rel_max(got[0][k], want[k]))
