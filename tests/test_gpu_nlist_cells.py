"""The neighbour search's cell walk at its edges, bit for bit against the
brute-force oracle: 4 to 7 half-cutoff cells per axis (every cell once, or five
with wrap-around), unequal axes, a sparse box (cells of a whole cutoff), clusters
with empty rows, atoms on cell faces and outside the box, and one atom alone."""
import numpy as np
import pytest

from oracle import nlist as onl
from test_gpu_nlist import gpu_nlist

pytestmark = pytest.mark.gpu

RC = 6.3
CASES = {
    "cells_4": ((12.7, 12.7, 12.7), 200, "uniform"),
    "cells_5": ((15.9, 15.9, 15.9), 400, "uniform"),
    "cells_4_6_13": ((12.61, 19.1, 41.0), 900, "uniform"),
    "cells_5_4_7": ((15.76, 12.7, 23.0), 420, "faces"),
    "sparse": ((100.0, 60.0, 80.0), 60, "uniform"),
    "cluster": ((40.0, 40.0, 40.0), 700, "cluster"),
    "outside": ((20.0, 16.0, 25.3), 500, "outside"),
    "alone": ((30.0, 30.0, 30.0), 1, "uniform"),
}


@pytest.mark.parametrize("name", list(CASES))
def test_nlist_cell_walk(name):
    box, n, how = CASES[name]
    rng = np.random.default_rng(11)
    box = np.array(box)
    pos = rng.uniform(size=(n, 3)) * box
    if how == "faces":    # on multiples of half the cutoff's cells, and a float above and below
        nc = np.floor(2 * box / RC)
        pos = np.round(pos / box * nc) * (box / nc)
        pos += rng.choice([-1e-5, 0.0, 1e-5], size=pos.shape) + rng.normal(scale=1e-4, size=pos.shape) * (rng.uniform(size=(n, 1)) < 0.5)
    elif how == "cluster":
        pos = (rng.choice([3.0, 37.0, 20.0], size=(n, 3)) + rng.normal(scale=2.0, size=(n, 3)))
    elif how == "outside":
        pos += rng.integers(-2, 3, size=pos.shape) * box
    types = rng.permutation(np.arange(n) % 3 == 0).astype(int)
    sel = [300, 200]
    w = dict(position=pos, type_idx=types, box=box)
    got, counts, status, ref_pos, cnt = gpu_nlist(w, sel, RC, perm_input=True)
    c = onl.canonicalize(pos, box, types)
    assert np.array_equal(ref_pos[0], c)
    want, wcounts, ovf = onl.typed_nlist(c, box.astype(np.float32), onl.cutoff_sq(RC), cnt, sel)
    assert not ovf and status == 0
    assert np.array_equal(counts[0], wcounts)
    assert np.array_equal(got[0], want)
