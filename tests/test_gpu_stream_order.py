"""Uploads and the kernels that read them on a non-blocking stream, which nothing orders behind the
default stream: a box whose stream is set before its components, its voxel lists and its structure
factors gives what a box on the default stream gives, to the last bit."""
import numpy as np
import pytest

from graspa_gb300 import synth

pytestmark = pytest.mark.gpu


def _calls(grx_lib, box, s):
    rng = np.random.default_rng(12)
    n = 24
    pos = rng.uniform(0, 1, (n, 3)) @ np.array(s["cell"]).reshape(3, 3)
    out = [box.trial_energies(pos, np.full(n, -0.35), np.full(n, 3), 10 ** 6, n, 1, 1, prec=p)[0]
           for p in (grx_lib.GRX_FP64, grx_lib.GRX_MIXED)]
    out.append(np.array(list(box.total_energy().values())))
    mol = s["templates"][1]["pos"] + [3.0, 4.0, 5.0]
    q = s["templates"][1]["charge"]
    box.write_molecule(1, 0, mol, q, s["templates"][1]["type"])
    fw, ads, _ = box.structure_factors()
    box.set_structure_factors(fw, 0.5 * ads)
    out.append(np.array(box.ewald_delta(1, grx_lib.MOVE_TRANSLATION, mol, q, mol + 0.4, q)))
    out.append(box.positions(1))
    return out


@pytest.mark.parametrize("which", ["silica", "water"])  # images in the entries, and by rounded fractions
def test_set_up_on_a_non_blocking_stream(grx_lib, which):
    torch = pytest.importorskip("torch")
    s = synth.silica_co2(n_co2=3) if which == "silica" else synth.tip4p_hex_system(n_water=3)
    cap = [s["comp_start"][1], 64]
    want = _calls(grx_lib, grx_lib.Box(s, capacity=cap), s)
    stream = torch.cuda.Stream()
    for _ in range(3):
        box = grx_lib.Box(s, capacity=cap)
        box.set_stream(stream.cuda_stream)
        box.set_voxel_lists(0)
        box.set_voxel_lists(1)
        assert box.voxel_lists()[0]
        for c in (0, 1):
            box.set_component(c)
        for got, ref in zip(_calls(grx_lib, box, s), want):
            assert np.array_equal(got, ref)
        box.close()
