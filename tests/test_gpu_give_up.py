"""An evaluation in which a tensor-core wait gave up: the word that the kernels set
reaches the results (every one NaN) and the status, whatever the sums hold.  The
word is preset here; no wait runs out."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gave_up", [False, True])
@pytest.mark.parametrize("natoms,nframes", [(1, 1), (300, 3), (1, 700)])
def test_give_up_reaches_every_result(gave_up, natoms, nframes):
    from deepmd_jax_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(0)

    def dev(shape, dtype=torch.float32):
        return torch.tensor(rng.normal(size=shape), dtype=dtype, device="cuda")

    acc = dev((nframes, natoms, 4), torch.float64)
    pos, atom_energy = dev((nframes, natoms, 3)), dev((nframes, natoms))
    energy, force = dev((nframes,), torch.float64), torch.zeros((nframes, natoms, 3), device="cuda")
    err = torch.full((1,), int(gave_up), dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    before = [t.clone() for t in (acc[..., :3].float(), energy, atom_energy)]
    p = [ctypes.c_void_p(t.data_ptr()) for t in (acc, pos, err, energy, atom_energy, force, status)]
    assert lib.dpb_selftest_finalize(natoms, nframes, *p, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    for was, now in zip(before, (force, energy, atom_energy)):
        assert bool(torch.isnan(now).all()) if gave_up else torch.equal(was, now)
    assert int(status.item()) == (16 if gave_up else 0)
