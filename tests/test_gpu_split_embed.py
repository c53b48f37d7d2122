"""The FP32 form's tensor-core embedding (embed_split.cu) at its edges against
the float64 oracle: blocks of 1 to 4 centre atoms with remainders, tiles of few
and of many rows, a list wider than the row store (the kernels compact it
themselves), several periodic images per pair, a workspace without room for the
row store, both tuned shapes, and one and three atom types.

Bars: the FP32 form's (energy <= 2e-6 sum|E_atom| + 1e-6 eV, forces and virial
<= 2e-4 of the largest component)."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu

WATER = dict(embed_widths=(25, 50, 100), fit_widths=(240, 240, 240), axis=16)
SMALL = dict(embed_widths=(32, 32, 64), fit_widths=(128, 128, 128), axis=12)
CASES = {
    "one_molecule": (dict(WATER), 1, 16.0, (4, 4)),                # 1 to 2 rows per tile
    "pair": (dict(WATER), 2, 14.0, (8, 8)),
    "odd_43": (dict(WATER), 43, 14.0, (46, 92)),                   # blocks of 1
    "blocks_of_4": (dict(WATER), 511, 24.83, (46, 92)),            # remainder of 3 atoms per type block
    "wide_list": (dict(WATER), 64, 12.7, (100, 130)),              # 230 list columns: no row store
    "images": (dict(WATER), 32, 9.86, (46, 92)),                   # several images per pair
    "no_room": (dict(WATER, fit_widths=(512, 512)), 43, 14.0, (46, 92)),  # wider than the mixed form's fitting
    "shape_64": (dict(SMALL), 100, 14.4, (56, 104)),
}


def _perturbed(params, variables, rng):
    """Every bias, dt and the descriptor statistics away from their zeros and ones."""
    params["sr_mean"] = np.linspace(0.05, 0.11, params["ntypes"])
    params["sr_std"] = np.linspace(0.8, 1.1, params["ntypes"])
    v = variables["params"]
    v["Tbias"] = (0.05 * rng.normal(size=v["Tbias"].shape)).astype(np.float32)
    for net in v.values():
        if isinstance(net, dict):
            for d in net.values():
                if isinstance(d, dict):
                    d["bias"] = (0.1 * rng.normal(size=d["bias"].shape)).astype(np.float32)


def _check(params, variables, pos, box, types, sel):
    from oracle import model as om
    out = run_gpu(params, variables, pos, box, types, sel=sel)
    assert out["status"] == 0
    ref = om.energy_force(om.OracleModel(params, variables, torch.float64), pos.astype(np.float32), box, types)
    dE = abs(float(out["energy"][0]) - ref["energy"])
    dF = np.abs(out["force"][0] - ref["force"]).max() / np.abs(ref["force"]).max()
    dW = np.abs(out["virial"][0] - ref["virial"]).max() / np.abs(ref["virial"]).max()
    print("|dE| %.2e  dF %.2e  dW %.2e" % (dE, dF, dW))
    assert dE <= 2e-6 * np.abs(ref["atom_energy"]).sum() + 1e-6
    assert dF <= 2e-4 and dW <= 2e-4


@pytest.mark.parametrize("name", list(CASES))
def test_split_embedding_edges(name):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    spec, waters, side, sel = CASES[name]
    rng = np.random.default_rng(3)
    params, variables = init_dp_params(nnbrs=50.0, seed=2, **spec)
    _perturbed(params, variables, rng)
    w = water_box(int(np.ceil(waters ** (1 / 3) - 1e-9)), side, seed=4, n_water=waters)
    _check(params, variables, w["position"], w["box"], w["type_idx"], sel)


@pytest.mark.parametrize("ntypes", [1, 3])
def test_split_embedding_types(ntypes):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    rng = np.random.default_rng(5)
    params, variables = init_dp_params(ntypes=ntypes, nnbrs=50.0, seed=2, **WATER)
    _perturbed(params, variables, rng)
    w = water_box(5, 14.5, seed=6, n_water=90)
    types = rng.permutation(np.arange(len(w["type_idx"])) % ntypes)
    _check(params, variables, w["position"], w["box"], types, tuple(np.bincount(types, minlength=ntypes)))
