"""The mixed fitting kernel's shape for many tiles is made for two CTAs per SM: their
shared memory (228 KB per SM, 1 KB of it the system's per CTA) has to hold two at
every depth and width."""
import json

import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [1, 3, 4])
@pytest.mark.parametrize("width", [50, 240, 256])
def test_two_fitting_ctas_fit_an_sm(width, layers, tmp_path):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    params, variables = init_dp_params(embed_widths=(25, 50, 100), axis=16, fit_widths=(width,) * layers, nnbrs=50.0,
                                       seed=5)
    w = water_box(6, 16.0, seed=4, n_water=20)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        run_gpu(params, variables, np.repeat(w["position"][None], 350, 0), w["box"], w["type_idx"], sel=(100, 200),
                precision="mixed")
    prof.export_chrome_trace(str(tmp_path / "trace.json"))
    with open(tmp_path / "trace.json") as f:
        events = [e for e in json.load(f)["traceEvents"] if "grid" in e.get("args", {})]
    if not events:
        pytest.skip("kernels cannot be traced here (another CUPTI client)")
    fits = [e for e in events if "k_mix_fit" in e["name"]]
    assert len(fits) == 1 and "false>" in fits[0]["name"]      # the shape for many tiles
    args = fits[0]["args"]
    print(fits[0]["name"][:40], args["shared memory"], args["registers per thread"])
    assert 2 * (args["shared memory"] + 1024) <= 228 * 1024
    assert 2 * args["block"][0] * args["registers per thread"] <= 65536
