"""The forms of the ensemble that AUTO does not take: the one-sided sweep (asked for, or where the slots of the pair form do
not fit) against the oracle, as test_gpu_ensemble.py does for the pair form; and what autotuning may choose in each."""

import pytest

from grasph2_b200.params import make_options
from grasph2_b200.sim import Ensemble, pack_states
from helpers import check_within, fp32_sensitivity
from test_gpu_ensemble import SIZES, VARIANTS, fields, oracle_derivs, sim_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accum", ["plain", "compensated"])
@pytest.mark.parametrize("name", list(VARIANTS))
def test_one_sided_derivatives_vs_oracle(oracle, name, accum):
    p = VARIANTS[name]()
    states = [sim_state(n, seed=100 + k, rho0=p.rho0, omega=0.1 * k) for k, n in enumerate(SIZES)]
    with Ensemble(p, SIZES, make_options(accum=accum, gravity="one-sided")) as ens:
        ens.upload(pack_states(states))
        ens.compute_derivatives()
        got = ens.split(ens.download())
    for k, st in enumerate(states):
        ref, sens = fp32_sensitivity(oracle_derivs(oracle, p), st, trials=1)
        for f, tol in fields(p).items():
            check_within(got[k][f], ref[f], sens[f], tol, "%s/%s/one-sided sim %d (n=%d) %s" % (name, accum, k, SIZES[k], f))


def test_only_the_sweep_has_a_tile_to_tune():
    """Launches of one autotuning call: the sweep tries three tiles with four CTA counts, the box search the counts alone."""
    p = VARIANTS["solid"]()
    sizes, reps = [3000, 700], 1
    timed = {}
    for form in ("auto", "one-sided"):
        with Ensemble(p, sizes, make_options(gravity=form)) as ens:
            ens.upload(pack_states([sim_state(n, seed=n) for n in sizes]))
            before = ens.launch_count()
            ens.compute_derivatives()
            each = ens.launch_count() - before
            shape = ens.autotune(reps)
            assert shape["ctas_per_sm"] in (0, 2, 3, 4)
            timed[form] = (ens.launch_count() - before - each) // (each * (reps + 1))
            if form == "auto":
                assert shape["tile"] == 512  # the default, untouched
    assert timed == {"auto": 4, "one-sided": 12}
