"""The same call gives the same bits: forces are sums over pairs in FP64, so the order
in which the GPU adds them does not show in FP32.  (An FP64 rounding that flips an FP32
one has a chance of about 1e-8 per component.)  Tuned, general and tabulated
embedding nets, both forms, single frames, frames and several images."""
import numpy as np
import pytest

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("net", ["tuned", "tuned64", "general", "table"])
@pytest.mark.parametrize("case", ["list", "frames", "images"])
def test_same_call_same_bits(net, case, precision):
    from make_golden import golden_models
    from deepmd_jax_b200.engine import DeviceModel
    from deepmd_jax_b200.systems import init_dp_params, water_box
    shape = {"tuned": ((25, 50, 100), 16), "tuned64": ((32, 32, 64), 12), "general": ((8, 16), 8)}
    if net == "table":
        params, variables = golden_models()["C"]
    else:
        params, variables = init_dp_params(embed_widths=shape[net][0], axis=shape[net][1], fit_widths=(64, 64, 64),
                                           nnbrs=50.0, seed=5)
    n, side, frames = {"list": (8, 24.84, 1), "frames": (4, 12.9, 16), "images": (4, 10.0, 1)}[case]
    w = water_box(n, side, seed=1, n_water=32 if case == "images" else None)
    pos = np.repeat(w["position"][None], frames, 0)
    model = DeviceModel(params, variables)
    runs = [run_gpu(params, variables, pos, w["box"], w["type_idx"], sel=(100, 200), precision=precision,
                    device_model=model) for _ in range(4)]
    assert all(r["status"] == 0 for r in runs)
    for r in runs[1:]:
        assert np.array_equal(r["force"], runs[0]["force"])
        assert np.array_equal(r["atom_energy"], runs[0]["atom_energy"])
