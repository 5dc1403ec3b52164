"""Gravity in units whose 1/r^3 one FP32 number does not hold (metres between stars, metres between atoms): the symmetric
kernels, which AUTO picks, against an FP64 sum over all pairs. Bound per target, relative to the sum of the pair forces'
magnitudes, as for ordinary separations (test_gpu_gravity_shapes.py): 4e-6 plain, 2e-6 compensated; the two products more
per pair add 2^-23 = 1.2e-7, inside it."""

import numpy as np
import pytest

from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer, Ensemble, pack_states
from helpers import f32_exact
from test_gpu_gravity_shapes import check, masses

pytestmark = pytest.mark.gpu
TOL = {"plain": 4e-6, "compensated": 2e-6}
G = float(np.float32(6.67e-11))


def cluster(n, length, mass, kind, seed=0):
    st = ics.uniform_sphere(n, radius=1.0, rho0=1.0, seed=seed)
    st["pos"] *= length
    if kind == "wide":  # most of them within one unit of length, a few far out
        st["pos"][: n - n // 50] /= length
        mass = min(mass, 1e20)  # m / r^3 of the close pairs stays in range
    st["mass"] = masses("different" if kind == "wide" else kind, n, np.random.default_rng(seed)) * mass * n
    st["density"][:] = 1.0
    return f32_exact(st)


def unit_g(acc, g):
    return acc.astype(np.float64) / g


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("kind", ["equal", "different", "wide"])
@pytest.mark.parametrize("length,mass,eps,g", [(1e13, 1e30, 1e11, G), (1e16, 1e30, 1e14, G), (3e12, 30.0, 0.0, 1.0),
                                               (1e-13, 1e-27, 1e-15, 1.0)])
@pytest.mark.parametrize("n", [4096, 9000, 26000, 60000])
def test_context(n, length, mass, eps, g, kind, accum):
    """Without softening the self pair takes 1/r = 1e12 in every form, so masses stay below 340 (m 1e36 in range)."""
    if kind == "wide":
        if length < 1.0:
            pytest.skip("the same separations as another case")
        eps = min(eps, 1e-3)
    p = make_params(switches=("SELF_GRAVITY",), H=0.05, grav_eps=eps, grav_G=g, fixed_dt=1e-3)
    st = cluster(n, length, mass, kind, seed=n)
    with DeviceParticleBuffer(p, n, make_options(accum=accum)) as pb:
        assert pb.launch_shape()["grav_sym_groups"] > 0
        pb.upload(st)
        pb.compute_derivatives()
        acc = pb.download()["acc"]
    check(unit_g(acc, g), st, p.grav_eps, TOL[accum])


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("kind", ["equal", "different"])
@pytest.mark.parametrize("length", [1e13, 1e16])
def test_ensemble(length, kind, accum):
    """Spheres whose particles have no neighbours within h: gravity alone, in an SPH ensemble."""
    g, sizes = G, [2, 513, 1500, 4097]
    p = make_params(switches=("SELF_GRAVITY", "SPH", "DEAL_WITH_NO_PARTNERS"), H=length * 1e-6, grav_eps=length * 1e-2,
                    grav_G=g, rho0=1.0, soundspeed=1.0, fixed_dt=1e-3)
    states = [cluster(n, length, 1e30, kind, seed=n) for n in sizes]
    with Ensemble(p, sizes, make_options(accum=accum)) as ens:
        ens.upload(pack_states(states))
        ens.compute_derivatives()
        got = ens.split(ens.download())
    for st, out in zip(states, got):
        check(unit_g(out["acc"], g), st, p.grav_eps, TOL[accum])
