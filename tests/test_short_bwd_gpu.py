"""GPU: the backward of short sequences (D = 64, at most 256 keys, one CTA per head) at the edges of its
tiles: 16 keys a warp, 32 query rows a block, 13 and 16 warps; with and without a depth part to add to.
Reference: the fp32 oracle on the same rounded inputs, tolerances of ``tests/helpers.py``."""
import pytest
import torch

from oracle import moda_oracle as mo
from tests.helpers import check_grad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("T,G,L", [(1, 1, 2), (15, 1, 0), (33, 1, 3), (64, 2, 0), (197, 1, 11), (208, 1, 1), (209, 2, 0), (256, 1, 5), (256, 2, 0)])
def test_short_backward(built_library, T, G, L, causal, dt):
    import moda_b200 as M
    B, H, D = 2, 3, 64
    q, k, v, kd, vd, dout = mo.make_inputs(7 * T + L, B, T, H, D, L, G, dtype=dt)
    ref = mo.moda_attention_ref_grads(q, k, v, kd, vd, dout, None, G, mo.MODE_CAUSAL if causal else mo.MODE_NONCAUSAL, 64)
    # channel-last views with a wider row: strides other than the packed ones
    wide = [torch.zeros(*x.shape[:3], 2 * D, dtype=dt, device="cuda") for x in (q, k, v)]
    leaves = [w[..., :D].copy_(x).requires_grad_(True) for w, x in zip(wide, (q, k, v))]
    leaves += [x.cuda().requires_grad_(True) for x in (kd, vd) if x is not None]
    deps = dict(cached_k=leaves[3], cached_v=leaves[4]) if L else {}

    def grads():
        o = M.parallel_moda(*leaves[:3], **deps, moda_group_num=G, is_causal=causal)
        o = o[0] if isinstance(o, tuple) else o
        return torch.autograd.grad(o, leaves, dout.cuda())

    first, again = grads(), grads()
    for name, a, b, g in zip(("dq", "dk", "dv", "d_depth_k", "d_depth_v"), first, again, [x for x in ref[2:] if x is not None]):
        assert torch.equal(a, b), name
        check_grad(name, a.float().cpu(), g)
        rows, err = g.norm(dim=-1), (a.float().cpu() - g).norm(dim=-1)     # no row missing: the same bound row by row
        assert (err <= 5e-2 * (rows + rows.mean()) + 1e-2).all(), name
    assert M.device_status() == 0


def _kernels(call):
    """What `call` returns, and the names of the library's kernels that it ran."""
    from moda_b200 import _cabi
    _cabi.profile_begin()
    try:
        r = call()
        torch.cuda.synchronize()
    finally:
        names = set(_cabi.profile_end())
    return r, names


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mode,T,G,L", [("causal", 197, 1, 11), ("all", 197, 1, 2), ("causal", 209, 2, 0), ("all", 256, 1, 0),
                                        ("causal", 170, 3, 0), ("chunk", 128, 4, 0), ("chunk", 64, 8, 0), ("chunk", 33, 2, 0),
                                        ("all", 13, 3, 0)])
def test_short_backward_of_many_heads(built_library, mode, T, G, L, dt):
    """Heads enough for the one-CTA-per-head kernel whatever the length, in every mode and with query groups that do
    and do not divide a block of 32 rows."""
    import moda_b200 as M
    from moda_b200 import ops
    B, H, D = (70, 2, 64) if T >= 170 else (64, 4, 64)
    om = {"causal": mo.MODE_CAUSAL, "all": mo.MODE_NONCAUSAL, "chunk": mo.MODE_CHUNK_VISIBLE}[mode]
    q, k, v, kd, vd, dout = mo.make_inputs(3 * T + L, B, T, H, D, L, G, dtype=dt)
    ref = mo.moda_attention_ref_grads(q, k, v, kd, vd, dout, None, G, om, max(64 // G, 1))
    dev = [x if x is None else x.cuda() for x in (q, k, v, kd, vd)]
    o, lse = ops._forward(*dev, D ** -0.5, G, om)
    grads, names = _kernels(lambda: ops._backward(*dev, o, lse, dout.cuda(), D ** -0.5, G, om))
    assert "short_bwd" in names, names
    for name, a, g in zip(("dq", "dk", "dv", "d_depth_k", "d_depth_v"), grads, ref[2:]):
        if g is None:
            continue
        check_grad(name, a.float().cpu(), g)
        rows, err = g.norm(dim=-1), (a.float().cpu() - g).norm(dim=-1)     # no row missing: the same bound row by row
        assert (err <= 5e-2 * (rows + rows.mean()) + 1e-2).all(), name
    assert M.device_status() == 0


@pytest.mark.parametrize("T,G,heads,short", [(64, 1, 4, True), (197, 1, 8, True), (197, 1, 128, True), (256, 2, 1, False),
                                             (256, 2, 192, False), (197, 1, 384, True), (128, 4, 16, False)])
def test_few_heads_take_the_tile_kernels(built_library, T, G, heads, short):
    from moda_b200 import ops
    q, k, dout = [torch.randn(heads, n, 1, 64, device="cuda", dtype=torch.bfloat16) for n in (T * G, T, T * G)]
    o, lse = ops._forward(q, k, k, None, None, 0.125, G, mo.MODE_CAUSAL)
    _, names = _kernels(lambda: ops._backward(q, k, k, None, None, o, lse, dout, 0.125, G, mo.MODE_CAUSAL))
    assert ("short_bwd" in names) == short, names
