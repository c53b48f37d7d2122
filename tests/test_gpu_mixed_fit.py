"""The mixed form's fitting kernel (k_mix_fit) at its edges against the float64
oracle: every padded hidden width, one to four layers with and without dt
residuals, descriptor lengths with a remainder of a stage, an absent type, and
enough frames of the same configuration that the launch takes the shape with two
CTAs per SM (the first and last frame are compared).

Bars: the mixed form's relative ones (force rms <= 3e-2 of the rms force, energy
per atom <= 2e-2 of the mean |E_atom|)."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu

# name: embedding widths, axis, fitting widths, molecules, frames
CASES = {
    "one_layer_64": ((32, 32, 64), 12, (64,), 20, 1),
    "rem_one": ((25, 50, 100), 4, (100, 100), 43, 1),            # K = 400: 25 steps
    "rem_three": ((25, 50, 100), 12, (208, 208, 208), 20, 1),    # K = 1200: 75 steps
    "no_residual": ((32, 32, 64), 12, (128, 64, 128), 64, 1),
    "four_layers_256": ((25, 50, 100), 16, (256, 256, 256, 256), 20, 1),
    "one_type": ((32, 32, 64), 12, (240, 240, 240), 20, 1),
    "frames_64": ((32, 32, 64), 12, (50, 50), 20, 350),
    "frames_rem_one": ((25, 50, 100), 4, (100, 100), 20, 350),
    "frames_240": ((25, 50, 100), 16, (240, 240, 240), 20, 350),
    "frames_256": ((25, 50, 100), 12, (250, 250), 20, 350),
}


@pytest.mark.parametrize("name", list(CASES))
def test_mixed_fit_edges(name):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    from oracle import model as om
    embed, axis, fit, waters, frames = CASES[name]
    rng = np.random.default_rng(8)
    params, variables = init_dp_params(embed_widths=embed, axis=axis, fit_widths=fit, nnbrs=50.0, seed=5)
    for t in range(2):
        for d in variables["params"]["fitting_net_%d" % t].values():
            if isinstance(d, dict):
                d["bias"] = (0.1 * rng.normal(size=d["bias"].shape)).astype(np.float32)
    w = water_box(6, 16.0, seed=4, n_water=waters)
    pos, typ = w["position"].astype(np.float32), w["type_idx"]
    if name == "one_type":
        typ = np.ones_like(typ)
    out = run_gpu(params, variables, np.repeat(pos[None], frames, 0), w["box"], typ, sel=(100, 200), precision="mixed")
    assert out["status"] == 0
    ref = om.energy_force(om.OracleModel(params, variables, torch.float64), pos, w["box"], typ)
    rms_f = np.sqrt((ref["force"] ** 2).mean())
    for f in {0, frames - 1}:
        rms = np.sqrt(((out["force"][f] - ref["force"]) ** 2).mean())
        dE = abs(float(out["energy"][f]) - ref["energy"]) / len(typ)
        print("%s: force rms %.2e of rms, energy %.2e of mean |E|" % (name, rms / rms_f,
                                                                    dE / np.abs(ref["atom_energy"]).mean()))
        assert rms <= 3e-2 * rms_f
        assert dE <= 2e-2 * np.abs(ref["atom_energy"]).mean()
