"""The double-precision symmetric gravity kernel and culled SPH passes against the sweep over all pairs (no_cull; one-sided
gravity): the same terms in FP64, summed in another order, with x^(-3/2) from a series instead of the library's square root
and division. Bound: 1e-11 of a field's largest value, as against GraSPH2's FP64 build (n <= 2.6e4 terms of 2^-53 each,
a factor 4 for cancellation)."""

import numpy as np
import pytest

import ref_variants
from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import rel_max

pytestmark = pytest.mark.gpu
TOL = 1e-11
FIELDS = ["acc", "density", "dstress_dt", "density_dt", "balsara", "maxvsig", "xvel"]


def run(params, st, steps=0, **opt):
    with DeviceParticleBuffer(params, st["mass"].shape[0], make_options(precision="double", **opt)) as pb:
        pb.upload_f64(st)
        pb.compute_derivatives()
        if steps:
            pb.integrate(True)
            pb.step(steps - 1)
        return pb.download_f64(FIELDS + ["pos", "vel", "dstress"])


def check(got, want, names):
    for k in names:
        assert np.isfinite(want[k]).all(), k
        assert rel_max(got[k], want[k]) <= TOL, (k, rel_max(got[k], want[k]))


def sphere(n, seed=0, radius=1.0):
    st = ics.uniform_sphere(n, radius=radius, rho0=1.0, omega=(0.1, 0.2, 0.3), seed=seed)
    rng = np.random.default_rng(seed + 1)
    st["vel"] += rng.normal(0.0, 0.1, (n, 3))
    s = rng.normal(0.0, 0.01, (n, 3, 3))
    st["dstress"][:] = s + s.transpose(0, 2, 1)
    st["mass"] *= rng.uniform(0.5, 2.0, n)
    return st


@pytest.mark.parametrize("name", ["fluid", "solid", "solid_mc", "fluid_full"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 1000, 1025, 3000])
def test_culled_passes_equal_the_sweep(name, n):
    over = dict(ref_variants.params_dict(ref_variants.VARIANTS[name]), grav_eps=0.02)
    p = make_params(**over)
    st = sphere(n, seed=n)
    st["density"][:] = 0.3 if name.startswith("fluid") else 1.05
    steps = 0 if n == 1 else 2  # a single particle: no acceleration, an unbounded variable step
    check(run(p, st, steps, resort_interval=1), run(p, st, steps, cull=False), FIELDS + ["pos", "vel", "dstress"])


def test_overflowing_neighbour_lists():
    """Every particle neighbours every other: more than the list slots of each warp's share."""
    p = make_params(**dict(ref_variants.params_dict(ref_variants.VARIANTS["solid"]), H=3.0))
    st = sphere(700)
    check(run(p, st), run(p, st, cull=False), FIELDS)


@pytest.mark.parametrize("eps", [0.0, 0.01])
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 1023, 1024, 1025, 13000, 26000])
def test_symmetric_gravity_equals_the_sweep(n, eps):
    """Row blocks of 128, 256 and 512 particles, unequal masses, two coincident particles (skipped: r^2 > 0)."""
    p = make_params(switches=("SELF_GRAVITY", "CONSTANT_ACCELERATION"), H=0.1, grav_eps=eps, fixed_dt=1e-3)
    st = sphere(n, seed=n)
    if n > 2:
        st["pos"][n - 1] = st["pos"][0]
    check(run(p, st), run(p, st, gravity="one-sided"), ["acc"])


def test_extreme_separations_and_nan():
    """Squared separations outside the series' range take the library's functions; a NaN position stays out of the
    other particles' sums, as in the sweep."""
    p = make_params(switches=("SELF_GRAVITY",), H=0.1, grav_eps=0.0, fixed_dt=1e-3)
    st = sphere(300)
    st["pos"][:20] *= 1e-95
    st["pos"][20:40] *= 1e92
    st["mass"][:20] *= 1e-150
    st["pos"][40, 1] = np.nan
    got, want = run(p, st)["acc"], run(p, st, gravity="one-sided")["acc"]
    assert (np.isfinite(got) == np.isfinite(want)).all() and np.isfinite(np.delete(got, 40, axis=0)).all()
    ok = np.isfinite(want)
    assert np.abs(got[ok] - want[ok]).max() <= TOL * np.abs(want[ok]).max()
    for rows in (slice(20, 40), slice(41, 300)):
        assert rel_max(got[rows], want[rows]) <= TOL
