"""The FP32 form on wide and deep fitting nets with small dt, where a bound on the
adjoint gates through every layer is thousands of times the gates themselves: forces
as close to the float64 oracle as with a narrow net.

Bar: 2^-20 (9.5e-7) of the rms force, 16 times the FP32 unit 2^-24: the embedding,
the same in every case, leaves about half of it, and a fitting net of FP32 accuracy
adds a few units in quadrature.  Gates with 11 to 13 bits miss it by a factor of two
and more."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu

# name: fitting widths, factor on the weights, dt
CASES = {
    "240x3": ((240, 240, 240), 1.0, 0.1),
    "512x4": ((512, 512, 512, 512), 3.0, 0.1),
    "1024x4": ((1024, 1024, 1024, 1024), 3.0, 0.1),
    "1024x4_small_dt": ((1024, 1024, 1024, 1024), 3.0, 0.01),
    "unequal": ((1024, 512, 256, 128), 3.0, 0.1),
    "no_quads": ((510, 510, 201, 201), 3.0, 0.01),
}


@pytest.mark.parametrize("name", list(CASES))
def test_wide_fitting_nets(name):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    from oracle import model as om
    fit, factor, dt = CASES[name]
    w = water_box(6, 16.0, seed=4, n_water=43)
    rng = np.random.default_rng(5)
    params, variables = init_dp_params(embed_widths=(25, 50, 100), axis=16, fit_widths=fit, nnbrs=50.0, seed=5)
    for t in range(2):
        net = variables["params"]["fitting_net_%d" % t]
        for k, d in net.items():
            if isinstance(d, dict):
                d["kernel"] = (factor * d["kernel"]).astype(np.float32)
                d["bias"] = (0.1 * rng.normal(size=d["bias"].shape)).astype(np.float32)
            else:
                net[k] = (dt * rng.uniform(0.5, 1.5, size=d.shape)).astype(np.float32)
    out = run_gpu(params, variables, w["position"], w["box"], w["type_idx"], sel=(100, 200))
    assert out["status"] == 0
    ref = om.energy_force(om.OracleModel(params, variables, torch.float64), w["position"].astype(np.float32), w["box"],
                          w["type_idx"])
    rms = np.sqrt(((out["force"][0] - ref["force"]) ** 2).mean() / (ref["force"] ** 2).mean())
    print("%s: force rms %.2e of rms" % (name, rms))
    assert rms <= 2.0 ** -20
    assert abs(float(out["energy"][0]) - ref["energy"]) <= 2e-6 * np.abs(ref["atom_energy"]).sum() + 1e-6
