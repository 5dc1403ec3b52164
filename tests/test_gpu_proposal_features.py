"""A proposal takes its features from the neighbour lists of its derivatives, the public entry point from the near
chunks: the same terms in the same order, so the proposal equals its stages to the bit. Without gravity, which proposals
sum in an order of their own. h = 0.9 of the sphere's radius: most lists are longer than is kept."""

import numpy as np
import pytest

from grasph2_b200 import ics
from grasph2_b200 import surrogate as S
from grasph2_b200.mlp import init_params
from grasph2_b200.params import impact_params, make_options
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import f32_exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("n,h", [(1000, None), (1500, 0.9), (29250, None)])
def test_proposal_equals_its_stages(n, h, accum):
    import torch
    nb = round(n * 8 / 9)
    p = impact_params(nb, n - nb)
    p.flags &= ~1  # self gravity
    if h:
        p.H = h
    st = f32_exact(ics.two_sphere_impact(nb, n - nb, v_rel=0.5, y_offset=0.3, seed=n))
    sur = S.Surrogate(8, init_params(1), np.full(32, 0.1), np.full(32, 0.5), np.zeros(13), np.full(13, 1e-4))
    out = []
    with DeviceParticleBuffer(p, n, make_options(accum=accum)) as pb:
        pb.upload(st)
        sur.propose(pb)
        out.append(pb.download())
        pb.upload(st)
        pb.compute_derivatives()
        f = S.features(pb, sur.dev["in_mu"], sur.dev["in_sig"])
        y = torch.empty(n, 13, device="cuda")
        sur.net.forward(f, y, n)
        S.apply(pb, 8, y, sur.dev["out_mu"], sur.dev["out_sig"])
        out.append(pb.download())
    for k in ("pos", "vel", "density", "dstress"):
        assert np.isfinite(out[0][k]).all()
        np.testing.assert_array_equal(out[0][k], out[1][k], err_msg=k)
