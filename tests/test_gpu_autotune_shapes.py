"""dpb_md_autotune times the shapes that it names: with fewer fitting tiles than SMs
(12,288 atoms, 96 tiles) both weight rings run, and the one that it reports is the one
that later steps launch; the dE/dT candidates fill the SMs."""
import json

import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernels(fn, path):
    """(name, args) of every kernel launched by fn, in order of time."""
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    with open(path) as f:
        events = [e for e in json.load(f)["traceEvents"] if "grid" in e.get("args", {})]
    if not events:
        pytest.skip("kernels cannot be traced here (another CUPTI client)")
    return [(e["name"], e["args"]) for e in sorted(events, key=lambda e: e["ts"])]


@pytest.fixture(scope="module")
def tuned(tmp_path_factory):
    from deepmd_jax_b200.md import Simulation
    from deepmd_jax_b200.systems import init_dp_params, water_box
    params, variables = init_dp_params(embed_widths=(25, 50, 100), axis=16, fit_widths=(240, 240, 240), nnbrs=100.0)
    w = water_box(16, 49.66, seed=0)
    sims = []

    def create():
        sims.append(Simulation((params, variables), w["box"], w["type_idx"], w["mass_per_type"], "NVE", 0.5, w["position"],
                               initial_velocity=w["velocity"], precision="mixed", verbose=False, autotune=True))

    path = tmp_path_factory.mktemp("trace") / "trace.json"
    create()  # kernels are loaded before the traced one
    during = _kernels(create, path)
    after = _kernels(lambda: sims[1].run(1, trajectory=False), path)
    return sims[1].launch_shapes, during, after


def test_both_rings_are_timed_and_the_choice_runs(tuned):
    shapes, during, after = tuned
    ring = {n: "true>" in n for n, _ in during if "k_mix_fit" in n}
    assert sorted(ring.values()) == [False, True]
    ran = [("true>" in n) for n, _ in after if "k_mix_fit" in n]
    assert ran and all(deep == (shapes["fit_ring_stages"] == 12) for deep in ran)


def test_dT_candidates_fill_the_sms(tuned):
    """Every dE/dT candidate launches as many blocks as its registers and shared memory let an SM hold."""
    shapes, during, _ = tuned
    grids = {}
    for name, a in during:
        if "k_mix_dT<" in name:
            warps = a["block"][0] // 32
            by_regs = 4 * (16384 // (-(-a["registers per thread"] // 8) * 256)) // warps
            grids[warps] = (a["grid"][0], min(by_regs, 64 // warps, 228 * 1024 // (a["shared memory"] + 1024)))
    print(grids)
    assert sorted(grids) == [2, 4, 8]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for warps, (grid, per_sm) in grids.items():
        assert grid == min(-(-12288 // warps), sms * per_sm)
