"""The compressed nets' adjoint (k_embed_bwd) at the edges of its rounds against
the float64 oracle with the same tables: 0 to 2 neighbours, below and above 16
and 32 rows of a type, both table widths, an odd axis.

Bars: the FP32 form's (energy <= 2e-6 sum|E_atom| + 1e-6 eV, forces <= 2e-4 of
the largest component)."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("embed,axis", [((32, 32, 64), 12), ((25, 50, 100), 16), ((32, 32, 64), 7)])
@pytest.mark.parametrize("waters", [1, 9, 17, 34])
def test_compressed_adjoint_rounds(embed, axis, waters):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    from make_golden import hermite_compressed
    from oracle import model as om
    params, variables = hermite_compressed(*init_dp_params(embed_widths=embed, axis=axis, fit_widths=(32, 32),
                                                           nnbrs=50.0, seed=5))
    w = water_box(6, 16.0, seed=4, n_water=waters)
    pos = w["position"].astype(np.float32)
    out = run_gpu(params, variables, pos, w["box"], w["type_idx"], sel=(48, 96))
    assert out["status"] == 0
    ref = om.energy_force(om.OracleModel(params, variables, torch.float64), pos, w["box"], w["type_idx"])
    dE = abs(float(out["energy"][0]) - ref["energy"])
    dF = np.abs(out["force"][0] - ref["force"]).max() / np.abs(ref["force"]).max()
    print("%d %s: |dE| %.2e (sum|E| %.2e)  dF %.2e" % (waters, embed, dE, np.abs(ref["atom_energy"]).sum(), dF))
    assert dE <= 2e-6 * np.abs(ref["atom_energy"]).sum() + 1e-6
    assert dF <= 2e-4
