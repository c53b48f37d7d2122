"""Neighbour lists in a box so long (123,456 A, 512 cells of 241 A) that one float32
step of a coordinate, 7.8e-3 A, is far above the rounding that short boxes see: one
atom on a cell face or a step behind it, the other just within the cutoff in the next
cell, bit for bit against the brute-force oracle."""
import numpy as np
import pytest

from oracle import nlist as onl
from test_gpu_nlist import gpu_nlist

pytestmark = pytest.mark.gpu

RC, LONG, CELLS = 6.297, 123456.0, 512
f32 = np.float32


def _raw(target):
    """float32 coordinates whose canonical ones (times 1 - 5e-7) are target, as nearly as float32 has them."""
    p = (target / (1 - 5e-7)).astype(f32)
    for step in (-1, 1):
        q = np.nextafter(p, f32(step * 1e9))
        better = np.abs(q * f32(1 - 5e-7) - target) < np.abs(p * f32(1 - 5e-7) - target)
        p = np.where(better, q, p)
    return p


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("side", [-1, 1])
def test_nlist_in_a_long_box(axis, side):
    rng = np.random.default_rng(3)
    box = np.full(3, 20.0)
    box[axis] = LONG
    face = (np.arange(2, CELLS - 2) * (LONG / CELLS)).astype(f32)
    n = len(face)
    near = (face + side * rng.integers(0, 2, size=n) * np.spacing(face)).astype(f32)
    far = (near - f32(side * RC)).astype(f32)
    far = (far + side * rng.integers(0, 4, size=n) * np.spacing(far)).astype(f32)
    pos = np.repeat(rng.uniform(2.0, 18.0, size=(n, 1, 3)), 2, axis=1).astype(f32)
    pos[:, 0, axis], pos[:, 1, axis] = _raw(near), _raw(far)
    pos = pos.reshape(-1, 3)
    types = (np.arange(2 * n) % 3 == 0).astype(int)
    got, counts, status, ref_pos, cnt = gpu_nlist(dict(position=pos, type_idx=types, box=box), [20, 20], RC,
                                                  perm_input=True)
    c = onl.canonicalize(pos, box, types)
    assert np.array_equal(ref_pos[0], c)
    want, wcounts, ovf = onl.typed_nlist(c, box.astype(f32), onl.cutoff_sq(RC), cnt, [20, 20])
    assert not ovf and status == 0
    assert n < wcounts.sum()                  # most of the pairs are neighbours
    assert np.array_equal(counts[0], wcounts)
    assert np.array_equal(got[0], want)
