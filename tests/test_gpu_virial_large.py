"""The FP32 form's virial does not lose bits as the system grows: a periodic cell
repeated 6 x 6 x 6 (81,000 atoms) has 216 times the virial of the cell.

Coordinates are multiples of 2^-17 A and the boxes 16 and 96 A, so every
displacement is the same FP32 number in both and only the summation differs.

Bar: 2^-26 of the largest component.  Rows are summed in FP32 within a block of
four atoms (a dozen additions) and in FP64 from block to block, so the cell's own
virial carries 2^-24 sqrt(12) / sqrt(376) of it (94 blocks of four warps, rounding
errors at random), 1.1e-8, and the repeated one less; one FP32 sum over a whole
launch's blocks does not reach it."""
import numpy as np
import pytest

from gpu_helpers import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [4, 5])
def test_virial_of_a_repeated_cell(seed):
    from deepmd_jax_b200.systems import init_dp_params, water_box
    params, variables = init_dp_params(embed_widths=(25, 50, 100), axis=16, fit_widths=(240, 240, 240), nnbrs=100.0,
                                       seed=5)
    w = water_box(6, 16.0, seed=seed, n_water=125)
    cell = np.round(w["position"] * 2 ** 17) / 2 ** 17
    virial = []
    for k in (1, 6):
        shift = 16.0 * np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
        out = run_gpu(params, variables, (cell[None] + shift).reshape(-1, 3), np.full(3, 16.0 * k),
                      np.tile(w["type_idx"], k ** 3), sel=(64, 128))
        assert out["status"] == 0
        virial.append(out["virial"][0] / k ** 3)
    err = np.abs(virial[1] - virial[0]).max() / np.abs(virial[0]).max()
    print("seed %d: %.2e" % (seed, err))
    assert err <= 2.0 ** -26
