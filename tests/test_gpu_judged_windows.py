"""A judged window evaluates the derivatives of its start once where the proposal and the plain steps sum gravity the same
way (gsph_surrogate_judge), and twice only where they do not; its plain path equals K steps to the bit in both."""

import numpy as np
import pytest

from grasph2_b200 import ics
from grasph2_b200 import surrogate as S
from grasph2_b200.mlp import init_params
from grasph2_b200.params import impact_params
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import f32_exact

pytestmark = pytest.mark.gpu
INTEGRATE_DENSITY = 1 << 2
FEATURES = 1  # launches of the context that only a network proposal needs


def setup(n, density):
    nb = round(n * 8 / 9)
    p = impact_params(nb, n - nb)
    if density == "integrated":
        p.flags |= INTEGRATE_DENSITY
    st = f32_exact(ics.two_sphere_impact(nb, n - nb, v_rel=0.5, y_offset=0.3, seed=n))
    rng = np.random.default_rng(n)
    return p, st, S.Surrogate(8, init_params(1), rng.normal(size=32) * 0.1, rng.uniform(0.5, 2.0, 32), np.zeros(13),
                              np.full(13, 1e-7))


def judge_launches(pb, st, sur, use_net):
    pb.upload(st)
    pb.step(1)  # the captured step exists
    before = pb.launch_count()
    S.window_errors(pb, sur, use_net, e_ref=1.0)
    return pb.launch_count() - before


# one-sided steps and proposals; integrated density: proposals and steps in the fixed order of summation
@pytest.mark.parametrize("n,density", [(2025, "summed"), (9000, "integrated"), (30000, "integrated")])
def test_shared_derivatives(n, density):
    p, st, sur = setup(n, density)
    with DeviceParticleBuffer(p, n) as pb:
        assert judge_launches(pb, st, sur, True) - judge_launches(pb, st, sur, False) == FEATURES


@pytest.mark.parametrize("tuned", [False, True])
@pytest.mark.parametrize("n,density", [(2025, "summed"), (9000, "summed"), (9000, "integrated"), (30000, "summed")])
def test_plain_path_is_k_steps(n, density, tuned):
    p, st, sur = setup(n, density)
    with DeviceParticleBuffer(p, n) as pb:
        pb.upload(st)
        if tuned:
            pb.autotune(1)
        S.snapshot(pb, 0, False)
        S.window_errors(pb, sur, True, e_ref=1.0)
        got, x = pb.download(), pb.download_pos64()
        S.snapshot(pb, 0, True)
        pb.step(sur.K)
        want, y = pb.download(), pb.download_pos64()
    np.testing.assert_array_equal(x, y)
    for k in want:
        assert np.isfinite(want[k]).all()
        np.testing.assert_array_equal(got[k], want[k], err_msg=k)
