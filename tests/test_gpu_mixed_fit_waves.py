"""Every tile of the mixed fitting kernel's shape for many tiles (two CTAs per SM, two
and more waves, tiles across frame boundaries, both centre types): 350 frames of one
configuration against each other.

The embedding sums the two neighbour types in an order that changes from one wave of
2 x SMs blocks of 8 atoms to the next, so frames are compared with those whose blocks
have the same orders.  Then nothing but the tile, wave and CTA of an atom differs:
its energy is a sum in one fixed order, bit for bit; a frame's energy agrees up to
the order of FP64 additions (1e-12), forces up to the order of float atomics (2e-6 of
the largest component: about 170 terms of 2^-24 each, at random 8e-7)."""
import numpy as np
import pytest
import torch

from gpu_helpers import run_gpu
from test_gpu_mixed_fit import CASES

pytestmark = pytest.mark.gpu

FRAMES = 350


def _orders(counts):
    """Per frame, the neighbour types' order in each of its blocks."""
    wave = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    keys = [()] * FRAMES
    for n in counts:
        blocks = -(-n // 8)
        turn = min(blocks * FRAMES, wave)
        for f in range(FRAMES):
            keys[f] += tuple((f * blocks + b) // turn % 2 for b in range(blocks))
    return keys


@pytest.mark.parametrize("name", [n for n in CASES if n.startswith("frames_")] + ["four_layers_256"])
def test_frames_of_one_configuration_agree(name):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    embed, axis, fit, waters, _ = CASES[name]
    rng = np.random.default_rng(8)
    params, variables = init_dp_params(embed_widths=embed, axis=axis, fit_widths=fit, nnbrs=50.0, seed=5)
    for t in range(2):
        for d in variables["params"]["fitting_net_%d" % t].values():
            if isinstance(d, dict):
                d["bias"] = (0.1 * rng.normal(size=d["bias"].shape)).astype(np.float32)
    w = water_box(6, 16.0, seed=4, n_water=waters)
    pos = w["position"].astype(np.float32)
    out = run_gpu(params, variables, np.repeat(pos[None], FRAMES, 0), w["box"], w["type_idx"], sel=(100, 200),
                  precision="mixed")
    assert out["status"] == 0
    groups = {}
    for f, key in enumerate(_orders((waters, 2 * waters))):
        groups.setdefault(key, []).append(f)
    print("%s: %d groups, the largest of %d frames" % (name, len(groups), max(map(len, groups.values()))))
    assert max(map(len, groups.values())) >= 50
    for frames in groups.values():
        e, a, x = out["energy"][frames], out["atom_energy"][frames], out["force"][frames]
        assert np.array_equal(a, np.repeat(a[:1], len(frames), 0))
        assert np.abs(e - e[0]).max() <= 1e-12 * np.abs(e[0])
        assert np.abs(x - x[0]).max() <= 2e-6 * np.abs(x[0]).max()
