"""Rosenbluth steps whose energies are not finite (a force field with an infinite or undefined shift for
some type pairs): FP64 Widom insertions into a thinned framework, where some trials meet such a pair
and others do not, against the FP64 oracle, which sums the weights one by one: the same selections,
success and non-finite weights; finite weights to 1e-10 (energies to 1e-12, as the selection tests)."""
import numpy as np
import pytest

from graspa_gb300 import synth
from tests.test_gpu_parity import oracle_widom

pytestmark = pytest.mark.gpu


def _system(guest_type, value):
    s = synth.silica_co2()
    keep = np.sort(np.random.default_rng(2).choice(s["comp_start"][1], 12, replace=False))
    s["molsize"] = [12, 3]
    synth._set_atoms(s, s["pos"][keep], s["type"][keep], np.zeros(12), [np.zeros((0, 3))])
    s["no_charges"] = 1
    shift = np.asarray(s["shift"]).reshape(s["ntypes"], s["ntypes"]).copy()
    shift[:2, guest_type] = shift[guest_type, :2] = value
    s["shift"] = shift.reshape(-1)
    return s


@pytest.mark.parametrize("ntrials", [4, 31, 32, 40])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("guest_type", [2, 3])  # the first bead, the chain beads
def test_weights_that_are_not_finite(grx_lib, guest_type, value, ntrials):
    s = _system(guest_type, value)
    n = 60
    box = grx_lib.Box(s, capacity=[12, 3 * 32])
    box.ewald_total()
    got = box.widom(grx_lib.widom_desc(s, 1, ntrials, 10), 0, n, prec=grx_lib.GRX_FP64)
    if np.isnan(value) and guest_type == 2:  # a first bead without a defined weight is no insertion
        assert not got["success"].any() and not got["rosenbluth"].any()
        return
    ref, _ = oracle_widom(s, 1, n, ntrials=ntrials, norient=10)
    for k in ("n_ok_first", "success", "sel_first", "n_ok_orient", "sel_orient"):
        assert np.array_equal(got[k], [getattr(r, k) for r in ref]), k
    w = np.array([r.rosenbluth for r in ref])
    odd = ~np.isfinite(w)
    assert np.array_equal(got["rosenbluth"][odd], w[odd], equal_nan=True)
    assert np.all(np.abs(got["rosenbluth"] - w)[~odd] <= 1e-10 * np.abs(w[~odd]))
    assert odd.any() == (value != -np.inf)


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_recorded_weights_that_are_not_finite(grx_lib, value):
    """GCMC: a chain's undefined or infinite weight is recorded in the insertions' weights."""
    s = _system(3, value)
    box = grx_lib.Box(s, capacity=[12, 3 * 32])
    box.ewald_total()
    d = grx_lib.gcmc_desc(1, p_translation=0.0, p_rotation=0.0, p_reinsertion=0.0, p_swap=1.0, pressure_pa=1e-30)
    st = grx_lib.gcmc_run([box], [d], 0, 40, grx_lib.GRX_FP64)[0]
    assert st.attempts[2] > 0
    assert (np.isnan if np.isnan(value) else np.isinf)(st.rosen[0])
