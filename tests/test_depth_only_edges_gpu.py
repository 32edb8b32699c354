"""GPU: the depth-only bandwidth kernels (``parallel_fda``, and the depth half of own-position MoDA at
G = 1) at the edges of their blocks: 16 depth rows a step (L = 1, 15, 16, 17, 33, 40), 8 query rows
a group (G = 1, 3, 8, 9), one-step and many-step units, packed depth K/V and an in-place layer cache.
Reference: the fp32 oracle on the same rounded inputs, tolerances of ``tests/helpers.py``."""
import pytest
import torch

from oracle import moda_oracle as mo
from tests.helpers import TOL_LSE_MAX_ABS, TOL_O_MAX_ABS, check_grad, max_abs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("L,G", [(1, 1), (15, 3), (16, 8), (17, 1), (33, 9), (40, 8), (2, 5)])
def test_depth_only_block_edges(built_library, L, G, D, dt):
    import moda_b200 as M
    B, T, H = 2, 37, 3
    q, _, _, kd, vd, dout = mo.make_inputs(100 + L + G, B, T, H, D, L, G, dtype=dt)
    ref = mo.moda_attention_ref_grads(q, None, None, kd, vd, dout, None, G, mo.MODE_DEPTH_ONLY, 1)
    leaves = [x.cuda().requires_grad_(True) for x in (q, kd, vd)]
    o, lse = M.parallel_fda(leaves[0], cached_k=leaves[1], cached_v=leaves[2], moda_group_num=G, need_lse=True)
    o.backward(dout.cuda())
    assert max_abs(o.float().cpu(), ref[0]) <= TOL_O_MAX_ABS and max_abs(lse.cpu(), ref[1]) <= TOL_LSE_MAX_ABS
    for name, leaf, g in zip(("dq", "d_depth_k", "d_depth_v"), leaves, [x for x in ref[2:] if x is not None]):
        check_grad(name, leaf.grad.float().cpu(), g)
    assert M.device_status() == 0


@pytest.mark.parametrize("L", [11, 16, 27])
def test_a_position_with_nan_leaves_the_others_alone(built_library, L):
    """The rows of a block past L are not read: neither the next position's, nor a layer cache's
    unwritten slots, nor what an earlier unit left in shared memory."""
    import moda_b200 as M
    B, T, H, D, G, cap = 1, 500, 4, 64, 2, 32
    gen = torch.Generator(device="cuda").manual_seed(L)
    mk = lambda n: torch.randn(B, n, H, D, generator=gen, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    q, kd, vd, dout = mk(T * G), mk(T * L), mk(T * L), mk(T * G)
    clean = M.parallel_fda_fwd(q, cached_k=kd, cached_v=vd, moda_group_num=G)
    grads = M.parallel_fda_bwd(q, *clean[:1], None, clean[1], dout, cached_k=kd, cached_v=vd, moda_group_num=G)
    bad = torch.arange(7, T, 13, device="cuda")
    kn, vn = kd.clone().view(B, T, L, H, D), vd.clone().view(B, T, L, H, D)
    kn[:, bad] = float("nan")
    vn[:, bad] = float("nan")
    kn, vn = kn.view_as(kd), vn.view_as(vd)
    o, lse = M.parallel_fda_fwd(q, cached_k=kn, cached_v=vn, moda_group_num=G)
    dirty = M.parallel_fda_bwd(q, o, None, lse, dout, cached_k=kn, cached_v=vn, moda_group_num=G)
    keep = torch.ones(T, dtype=torch.bool, device="cuda")
    keep[bad] = False
    for a, b, rows in ((o, clean[0], G), (dirty[0], grads[0], G), (dirty[2], grads[2], L), (dirty[3], grads[3], L)):
        a, b = a.view(B, T, rows, H, D)[:, keep], b.view(B, T, rows, H, D)[:, keep]
        assert torch.equal(a, b)

    # an in-place cache of which the first L layers are written: the rest holds NaN
    cache = M.DepthKVCache(B, T, cap, H, D, torch.bfloat16, "cuda")
    cache.k.fill_(float("nan"))
    cache.v.fill_(float("nan"))
    for j in range(L):
        cache.append(kd.view(B, T, L, H, D)[:, :, j], vd.view(B, T, L, H, D)[:, :, j])
    q1, k1, v1 = [mk(T).requires_grad_(True) for _ in range(3)]
    o1 = cache.attend(q1, k1, v1)
    o2 = M.parallel_moda(q1, k1, v1, cached_k=kd, cached_v=vd)
    assert torch.equal(o1, o2)
    g1, g2 = torch.autograd.grad(o1, q1, mk(T).fill_(1.0)), torch.autograd.grad(o2, q1, mk(T).fill_(1.0))
    assert torch.equal(g1[0], g2[0])
    assert M.device_status() == 0
