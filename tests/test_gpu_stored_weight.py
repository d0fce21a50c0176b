"""Reinsertions where one first-bead trial outweighs the others by 1e15 and more (CO2 beside 34 charged
atoms of either sign, not neutral): the weight that the retrace takes over, the sum without the chosen
trial, is then roundings of the sum, and the decisions follow the order in which it was added up.
FP64 GCMC against the oracle, 60 systems of 40 reinsertions: the same accepted moves and positions.

A decision can hang on the last bit of the two exp functions (device and host); two systems of the 60
may differ for that."""
import numpy as np
import pytest

from graspa_gb300 import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _system(k):
    s = synth.silica_co2(n_co2=3)
    h = s["comp_start"][1]
    keep = np.sort(np.random.default_rng(k).choice(h, 34, replace=False))
    idx = np.concatenate([keep, np.arange(h, len(s["pos"]))])
    for f in ("pos", "charge", "scale", "scale_coul", "type", "molid"):
        s[f] = np.asarray(s[f])[idx]
    s["comp_start"] = [0] + [x - (h - 34) for x in s["comp_start"][1:]]
    s["molsize"] = [34, 3]
    return s


def test_retrace_takes_over_the_same_weight(grx_lib):
    same = accepted = 0
    for k in range(60):
        s = _system(k)
        box = grx_lib.Box(s, capacity=[34, 96])
        box.ewald_total()
        d = grx_lib.gcmc_desc(1, 35, 26, p_translation=0.0, p_rotation=0.0, p_reinsertion=1.0, p_swap=1.0,
                              pressure_pa=1e5, seed=k)
        st = grx_lib.gcmc_run([box], [d], 0, 40, grx_lib.GRX_FP64)[0]
        g = O.OraGcmc()
        g.component, g.ntrials, g.norient = 1, 35, 26
        g.p_translation, g.p_rotation, g.p_reinsertion, g.p_swap = 0.0, 0.0, 1.0, 1.0
        for i in range(3):
            g.max_translation[i], g.max_rotation[i] = d.max_translation[i], d.max_rotation[i]
        g.beta, g.pressure, g.fugacity_coeff, g.mol_fraction, g.ideal_rosenbluth = d.beta, d.pressure, 1.0, 1.0, 1.0
        g.seed, g.stream = d.seed, d.stream
        ost, after, _ = O.OracleSystem(s).gcmc(g, [34, 96], 0, 40)
        accepted += sum(ost.accepted)
        same += (list(st.accepted) == list(ost.accepted) and
                 np.max(np.abs(box.positions(1) - after["pos"][34:])) <= 1e-6)
        box.close()
    assert accepted >= 60
    assert same >= 58
