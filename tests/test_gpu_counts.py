"""gsph_launch_count and gsph_ensemble_launch_count count kernels, those of a captured step and of the energies included."""

import pytest

import ref_variants
from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer, Ensemble, pack_states
from helpers import f32_exact

pytestmark = pytest.mark.gpu
P = make_params(**ref_variants.params_dict(ref_variants.VARIANTS["fluid"]))


def counted(buf, f):
    before = buf.launch_count()
    f()
    return buf.launch_count() - before


@pytest.mark.parametrize("gravity,per_step", [("auto", 3), ("one-sided", 1)])  # boxes, gravity, queue; the queue alone
def test_ensemble_steps(gravity, per_step):
    sizes = [700, 300]
    with Ensemble(P, sizes, make_options(gravity=gravity)) as ens:
        ens.upload(pack_states([f32_exact(ics.uniform_sphere(n, seed=n)) for n in sizes]))
        ens.step(1)
        assert counted(ens, lambda: ens.step(4)) == 4 * per_step


@pytest.mark.parametrize("precision,fast,kernels", [("single", False, 3), ("single", True, 2), ("double", False, 3)])
def test_energies(precision, fast, kernels):
    st = f32_exact(ics.uniform_sphere(500, seed=1))
    with DeviceParticleBuffer(P, 500, make_options(precision=precision)) as pb:
        pb.upload(st)
        pb.compute_derivatives()
        assert counted(pb, lambda: pb.diagnostics(fast=fast)) == kernels
