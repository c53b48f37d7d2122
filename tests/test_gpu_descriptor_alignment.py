"""dpb_eval_descriptors takes T, G and a workspace at any float: the FP32 form's
tuned nets (16- and 8-byte stores) at addresses 4, 8 and 12 bytes off give the bits of
the aligned call."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("embed,axis", [((25, 50, 100), 16), ((32, 32, 64), 12)])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_descriptors_at_any_float(embed, axis, off):
    from deepmd_jax_b200 import _lib
    from deepmd_jax_b200.engine import DeviceModel, NeighborBuilder, _ptr, _stream, sort_by_type
    from deepmd_jax_b200.systems import init_dp_params, water_box
    params, variables = init_dp_params(embed_widths=embed, axis=axis, fit_widths=(32, 32), nnbrs=50.0, seed=5)
    w = water_box(4, 12.9, seed=4)
    perm, cnt = sort_by_type(w["type_idx"], 2)
    n, sel = len(perm), [64, 128]
    pos = torch.tensor(w["position"][None], dtype=torch.float32, device="cuda")
    pm = torch.tensor(perm, dtype=torch.int32, device="cuda")
    box = torch.tensor(np.asarray(w["box"])[None], dtype=torch.float32, device="cuda")
    nbrs, status = NeighborBuilder(n, 1, cnt, sel, w["box"], 6.3).build(pos, perm=pm)
    assert int(status.item()) == 0
    dm = DeviceModel(params, variables)
    T, G = dm.descriptors(pos, box, nbrs, cnt, sel, perm=pm)
    t_buf = torch.zeros(T.numel() + 8, device="cuda")
    g_buf = torch.zeros(G.numel() + 8, device="cuda")
    ws = dm.eval_workspace(n, 1)
    ws_buf = torch.empty(ws.numel() + 64, dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = dm.lib.dpb_eval_descriptors(dm.handle, 0, _ptr(pos), _ptr(pm), n, 1, _lib.int_array(cnt), _ptr(box), _ptr(nbrs),
                                     _lib.int_array(sel), ctypes.c_void_p(t_buf.data_ptr() + 4 * off),
                                     ctypes.c_void_p(g_buf.data_ptr() + 4 * off), _ptr(err),
                                     ctypes.c_void_p(ws_buf.data_ptr() + 4 * off), ws.numel(), _stream())
    torch.cuda.synchronize()
    assert rc == 0 and int(err.item()) == 0
    assert torch.equal(t_buf[off:off + T.numel()].view_as(T), T)
    assert torch.equal(g_buf[off:off + G.numel()].view_as(G), G)
    for buf, k in ((t_buf, T.numel()), (g_buf, G.numel())):   # nothing outside
        assert bool((buf[:off] == 0).all()) and bool((buf[off + k:] == 0).all())
