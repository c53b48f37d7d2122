"""The FP32 form's fitting GEMMs whose operand the previous kernel leaves as split
tiles, where a CTA runs through several output tiles (two groups of warps take
turns at them) with one, two, three and more chunks of K each: 26 frames of one
configuration, every frame against the float64 oracle.

Bars: the FP32 form's (energy <= 2e-6 sum|E_atom| + 1e-6 eV, forces <= 2e-4 of
the largest component)."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fit", [(16,), (30, 30), (50, 50, 50), (96, 64), (13, 13, 100), (240, 240, 240)])
def test_split_gemm_operand_tiles(fit):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    from oracle import model as om
    rng = np.random.default_rng(8)
    params, variables = init_dp_params(embed_widths=(25, 50, 100), axis=16, fit_widths=fit, nnbrs=50.0, seed=5)
    for t in range(2):
        for d in variables["params"]["fitting_net_%d" % t].values():
            if isinstance(d, dict):
                d["bias"] = (0.1 * rng.normal(size=d["bias"].shape)).astype(np.float32)
    w = water_box(6, 16.0, seed=4, n_water=20)
    pos = w["position"].astype(np.float32)
    out = run_gpu(params, variables, np.repeat(pos[None], 26, 0), w["box"], w["type_idx"], sel=(100, 200))
    assert out["status"] == 0
    ref = om.energy_force(om.OracleModel(params, variables, torch.float64), pos, w["box"], w["type_idx"])
    dE = np.abs(out["energy"] - ref["energy"]).max()
    dF = np.abs(out["force"] - ref["force"]).max() / np.abs(ref["force"]).max()
    print("%s: |dE| %.2e (sum|E| %.2e)  dF %.2e" % (fit, dE, np.abs(ref["atom_energy"]).sum(), dF))
    assert dE <= 2e-6 * np.abs(ref["atom_energy"]).sum() + 1e-6
    assert dF <= 2e-4
