"""The FP32 form's fitting GEMMs on the tensor cores (gemm_split.cu) at their
edges against the float64 oracle: hidden widths below, at and above a column
tile, widths that are no multiple of 4, 16 or 32 (remainders of K and of a row's
quads), one to four layers with and without dt residuals, descriptors of very
small magnitude (the per-atom operand scale), and row counts
around the 128-row tile.

Bars: the FP32 form's (energy <= 2e-6 sum|E_atom| + 1e-6 eV, forces <= 2e-4 of
the largest component)."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu

# name: embedding widths, axis, fitting widths, molecules, Nnbrs (scales T, so G as its square)
CASES = {
    "narrow": ((25, 50, 100), 16, (16,), 20, 50.0),
    "odd_widths": ((25, 50, 100), 16, (13, 13, 30), 20, 50.0),
    "odd_k0": ((5, 10, 20), 7, (50, 50), 20, 50.0),             # K = 140
    "tile_edge": ((32, 32, 64), 12, (128, 128), 43, 50.0),      # 43 + 86 rows
    "past_tile": ((32, 32, 64), 12, (130, 130, 130), 64, 50.0),
    "wide": ((25, 50, 100), 16, (300, 300), 65, 50.0),
    "four_layers": ((25, 50, 100), 16, (48, 48, 48, 48), 64, 50.0),
    "small_g": ((25, 50, 100), 16, (64, 64), 20, 5e4),
    "rows_129": ((25, 50, 100), 16, (240, 240, 240), 129, 50.0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_split_gemm_edges(name):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    from oracle import model as om
    embed, axis, fit, waters, nnbrs = CASES[name]
    rng = np.random.default_rng(8)
    params, variables = init_dp_params(embed_widths=embed, axis=axis, fit_widths=fit, nnbrs=nnbrs, seed=5)
    for t in range(2):
        for d in variables["params"]["fitting_net_%d" % t].values():
            if isinstance(d, dict):
                d["bias"] = (0.1 * rng.normal(size=d["bias"].shape)).astype(np.float32)
    w = water_box(6, 16.0, seed=4, n_water=waters)
    out = run_gpu(params, variables, w["position"], w["box"], w["type_idx"], sel=(100, 200))
    assert out["status"] == 0
    ref = om.energy_force(om.OracleModel(params, variables, torch.float64), w["position"].astype(np.float32), w["box"],
                          w["type_idx"])
    dE = abs(float(out["energy"][0]) - ref["energy"])
    dF = np.abs(out["force"][0] - ref["force"]).max() / np.abs(ref["force"]).max()
    print("%s: |dE| %.2e (sum|E| %.2e)  dF %.2e" % (name, dE, np.abs(ref["atom_energy"]).sum(), dF))
    assert dE <= 2e-6 * np.abs(ref["atom_energy"]).sum() + 1e-6
    assert dF <= 2e-4
