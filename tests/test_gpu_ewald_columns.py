"""The column form of a move's Fourier delta (grx_ewcol.cuh) at the edges of its k ranges: flat and
missing axes, one or many |kz| per (kx, ky) row (the row-product form), on one block and on a
cluster. The adsorbate structure factor committed by 40 GCMC steps must equal the one recomputed in
FP64 from the final positions, and the drift of the Fourier energy must vanish: |dS| <= 1e-10 (the
reference's CPU/GPU check), energies to 1e-9 of the Fourier total of the recomputation (FP64) and to
the mixed bar per accepted move.
"""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", [1, 2])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("kmax", [(0, 2, 1), (3, 0, 2), (2, 0, 20), (1, 1, 0), (9, 9, 6)])
def test_committed_structure_factor(grx_lib, kmax, prec, cluster):
    s = synth.silica_co2(kmax=kmax, n_co2=6)
    box = grx_lib.Box(s, capacity=[s["comp_start"][1], 3 * 64])
    e0 = box.total_energy()
    d = grx_lib.gcmc_desc(1, p_translation=0.4, p_rotation=0.6, p_reinsertion=0.7, p_swap=1.0, pressure_pa=1e6, seed=9)
    batch = grx_lib.GcmcBatch([box], [d], prec=grx_lib.PRECISIONS[prec])
    batch.set_cluster(cluster)
    batch.launch(40)
    st, _ = batch.stats()
    batch.close()
    got = box.structure_factors()[1]
    e1 = box.total_energy()
    want = box.structure_factors()[1]
    assert np.max(np.abs(got - want)) <= 1e-10
    accepted = sum(st[0].accepted)
    assert accepted > 0
    fourier = (e1["hg_ewald"] + e1["gg_ewald"]) - (e0["hg_ewald"] + e0["gg_ewald"])
    scale = abs(e1["gg_ewald"]) * 1e-13 + 1e-9
    bar = scale if prec == "fp64" else scale + accepted * 1e-6 / d.beta
    assert abs(fourier - st[0].energy[2]) <= bar
