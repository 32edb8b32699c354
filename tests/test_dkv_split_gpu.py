"""GPU: dk/dv of launches with few key tiles, whose query steps may be divided over a cluster of 2 or 4 CTAs:
tiles with fewer steps than CTAs, odd step counts, a last tile of one key, every mode that reaches it.
Reference: the fp32 oracle on the same rounded inputs, tolerances of ``tests/helpers.py``."""
import pytest
import torch

from oracle import moda_oracle as mo
from tests.helpers import check_grad, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode,B,T,H,G,L", [
    ("causal", 1, 300, 2, 2, 3),      # 10 steps; the last tile has two
    ("causal", 1, 257, 1, 1, 0),      # 5 steps; the last tile has one key and one step
    ("all", 2, 193, 3, 2, 5),         # 7 steps for every tile
    ("chunk", 1, 320, 2, 4, 2),       # 20 steps: four CTAs
    ("all", 1, 1024, 16, 1, 0),       # 128 tiles of 16 steps
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


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode,B,T,H,G,L,split", [
    ("causal", 1, 2048, 2, 2, 0, True),     # 32 tiles of up to 64 steps: two CTAs
    ("all", 1, 1100, 3, 2, 0, True),        # 27 tiles of 35 steps: two
    ("causal", 1, 700, 1, 2, 0, True),      # 6 tiles of up to 22 steps, the last of two: four
    ("all", 1, 1281, 1, 1, 0, True),        # 11 tiles of 21 steps, the last one of one key: four
    ("chunk", 1, 1000, 2, 4, 1, True),      # beside the depth gradients
    ("causal", 1, 1024, 12, 1, 0, False),   # shares would wait for dq's CTAs: 36 us unsplit, 42 with two
    ("all", 1, 1024, 16, 1, 0, False),      # as many tiles as SMs, all alike
    ("causal", 2, 512, 8, 1, 0, False),     # short chains
])
def test_which_launches_are_split(built_library, mode, B, T, H, G, L, split, D, dt):
    """The rule's two sides; against the mma.sync kernels, which the oracle tests cover: roundings of P and dS and
    of the results, some 2^-8 (bf16) or 2^-11 (fp16) each."""
    import moda_b200 as M
    from moda_b200 import _cabi, ops
    m = {"causal": mo.MODE_CAUSAL, "all": mo.MODE_NONCAUSAL, "chunk": mo.MODE_CHUNK_VISIBLE}[mode]
    gen = torch.Generator(device="cuda").manual_seed(T + G)
    mk = lambda n: torch.randn(B, n, H, D, generator=gen, device="cuda").to(dt) if n else None  # noqa: E731
    xs, dout = [mk(T * G), mk(T), mk(T), mk(T * L), mk(T * L)], mk(T * G)
    o, lse = ops._forward(*xs, D ** -0.5, G, m)
    call = lambda: ops._backward(*xs, o, lse, dout, D ** -0.5, G, m)  # noqa: E731
    _cabi.profile_begin()
    grads = call()
    torch.cuda.synchronize()
    names = set(_cabi.profile_end())
    assert ("tc_dkv_split" in names, "tc_dkv" in names) == (split, not split), names
    again = call()
    old = M.set_kernel_path(M.PATH_SIMT_MMA)
    try:
        want = call()
    finally:
        M.set_kernel_path(old)
    for name, a, b, c in zip(("dq", "dk", "dv", "d_depth_k", "d_depth_v"), grads, again, want):
        if a is not None:
            assert torch.equal(a, b), name
            assert rel_l2(a, c) <= (2e-2 if dt == torch.bfloat16 else 2.5e-3), name
    assert M.device_status() == 0
