"""GPU: dk/dv of launches with few key tiles, whose query steps are divided over a cluster of 2 or 4 CTAs:
tiles with fewer steps than CTAs, odd step counts, a last tile of one key, every mode that reaches it.
Reference: the fp32 oracle on the same rounded inputs, tolerances of ``tests/helpers.py``."""
import pytest
import torch

from oracle import moda_oracle as mo
from tests.helpers import check_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode,B,T,H,G,L", [
    ("causal", 1, 300, 2, 2, 3),      # 10 steps: four CTAs; the last tile has two steps
    ("causal", 1, 257, 1, 1, 0),      # 5 steps: two CTAs; the last tile has one key and one step
    ("all", 2, 193, 3, 2, 5),         # 7 steps for every tile
    ("chunk", 1, 320, 2, 4, 2),       # 20 steps
    ("all", 1, 1024, 16, 1, 0),       # 128 tiles of 16 steps: two CTAs
])
def test_split_dkv(built_library, mode, B, T, H, G, L, D, dt):
    import moda_b200 as M
    q, k, v, kd, vd, dout = mo.make_inputs(T + G + L, B, T, H, D, max(L, 1), G, dtype=dt)
    if L == 0:
        kd = vd = None
    om = {"causal": mo.MODE_CAUSAL, "all": mo.MODE_NONCAUSAL, "chunk": mo.MODE_CHUNK_VISIBLE}[mode]
    ref = mo.moda_attention_ref_grads(q, k, v, kd, vd, dout, None, G, om, 64 // G)
    leaves = [x.cuda().requires_grad_(True) for x in (q, k, v, kd, vd) if x is not None]
    deps = dict(cached_k=leaves[3], cached_v=leaves[4]) if L else {}

    def grads():
        if mode == "chunk":
            o = M.parallel_moda_chunk_visible(*leaves[:3], **deps, moda_group_num=G, warn_shape=False)
        else:
            o = M.parallel_moda(*leaves[:3], **deps, moda_group_num=G, is_causal=mode == "causal")
        o = o[0] if isinstance(o, tuple) else o
        return torch.autograd.grad(o, leaves, dout.cuda())

    first, again = grads(), grads()
    for name, a, b, g in zip(("dq", "dk", "dv", "d_depth_k", "d_depth_v"), first, again, [x for x in ref[2:] if x is not None]):
        assert torch.equal(a, b), name
        check_grad(name, a.float().cpu(), g)
        rows, err = g.norm(dim=-1), (a.float().cpu() - g).norm(dim=-1)     # no row missing: the same bound row by row
        assert (err <= 5e-2 * (rows + rows.mean())).all(), name
    assert M.device_status() == 0
