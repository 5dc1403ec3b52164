"""The symmetric gravity kernel's block shapes (n picks blocks of 128, 256, 512 or 1,024) and its equal-mass tiles against
an FP64 sum over all pairs: equal masses, two masses that meet inside a block, masses all different, massless particles.

Bound per target, relative to the sum of the pair forces' magnitudes (what rounding scales with): a pair's force carries
at most 8 roundings of 2^-24 (separation, r^2, 2 ulp of rsqrt cubed, masses, product): 4.8e-7; a tile's FP32 sum of up
to 256 terms adds sqrt(256) 2^-24 = 1e-6 typically, the plain form's sum over up to 240 tiles as much again. 2e-6
compensated, 4e-6 plain."""

import numpy as np
import pytest

from grasph2_b200 import ics
from grasph2_b200.params import make_options, make_params
from grasph2_b200.sim import DeviceParticleBuffer
from helpers import f32_exact

pytestmark = pytest.mark.gpu


def accel(p, st, **opt):
    with DeviceParticleBuffer(p, st["mass"].shape[0], make_options(**opt)) as pb:
        pb.upload(st)
        pb.compute_derivatives()
        return pb.download()["acc"].astype(np.float64), pb.launch_shape()["grav_sym_groups"]


def exact(st, eps):
    """FP64 accelerations and the sums of the pair forces' magnitudes."""
    import torch
    x, m = (torch.from_numpy(st[k]).double().cuda() for k in ("pos", "mass"))
    acc, mag = torch.empty_like(x), torch.empty(len(x), dtype=torch.float64, device="cuda")
    step = max(1, 2 ** 24 // len(x))
    for a in range(0, len(x), step):
        d = x[None, :, :] - x[a:a + step, None, :]
        r2 = (d * d).sum(2)
        f = torch.where(r2 > 0, m[None, :] * (r2 + eps * eps) ** -1.5, 0.0)
        acc[a:a + step] = (f[:, :, None] * d).sum(1)
        mag[a:a + step] = (f * r2.sqrt()).sum(1)
    return acc.cpu().numpy(), mag.cpu().numpy()


def check(got, st, eps, tol):
    want, mag = exact(st, eps)
    assert np.isfinite(got).all()
    assert (np.linalg.norm(got - want, axis=1) <= tol * mag).all()


def masses(kind, n, rng):
    m = np.full(n, 1.0 / n)
    if kind == "two":
        m[n // 3:] *= 3.0
    elif kind == "different":
        m *= rng.uniform(0.1, 10.0, n)
    elif kind == "massless":
        m[rng.random(n) < 0.3] = 0.0
        m[: n // 2] = 0.0
    return m


@pytest.mark.parametrize("accum,tol", [("plain", 4e-6), ("compensated", 2e-6)])
@pytest.mark.parametrize("kind", ["equal", "two", "different", "massless"])
@pytest.mark.parametrize("n", [2, 127, 129, 1025, 4097, 9000, 17000, 26000, 60000])
def test_shapes_and_masses(n, kind, accum, tol):
    p = make_params(switches=("SELF_GRAVITY",), H=0.05, grav_eps=0.01, fixed_dt=1e-3)
    st = ics.plummer_sphere(n, seed=n)
    st["mass"] = masses(kind, n, np.random.default_rng(n))
    st = f32_exact(st)
    got, groups = accel(p, st, accum=accum)
    assert groups > 0
    check(got, st, 0.01, tol)


@pytest.mark.parametrize("kind", ["equal", "different"])
def test_unsoftened_with_coincident_particles(kind):
    """eps = 0: coincident particles and the self pair add nothing (1/r is limited to 1e12 and the separation is 0)."""
    n = 5000
    p = make_params(switches=("SELF_GRAVITY",), H=0.05, grav_eps=0.0, fixed_dt=1e-3)
    st = ics.uniform_sphere(n, seed=2)
    st["mass"] = masses(kind, n, np.random.default_rng(1))
    st["pos"][n - 1] = st["pos"][0]
    st["pos"][1] = st["pos"][0]
    st = f32_exact(st)
    got, _ = accel(p, st)
    check(got, st, 0.0, 4e-6)
