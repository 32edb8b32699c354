"""GPU: an in-place layer cache of any layer count on the tcgen05 kernels (depth tiles of whole positions):
tiles that a box does not fill, positions past the end, a depth tile in a ring slot that nothing has been
loaded into, unwritten layers that hold NaN, query groups that do (G = 2, 4, 8) and do not (G = 3) divide 64.
Reference: the packed layout of the same rows, which the oracle tests cover, within the rounding of P and dS."""
import pytest
import torch

from tests.helpers import max_abs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode", ["causal", "all", "chunk"])
@pytest.mark.parametrize("T,G,L,cap", [(70, 4, 3, 5), (33, 2, 11, 12), (3, 8, 7, 16), (200, 8, 5, 6), (150, 3, 9, 11), (129, 2, 33, 40),
                                       (40, 2, 64, 65), (300, 4, 10, 12)])
def test_layer_count(built_library, T, G, L, cap, mode, D):
    import moda_b200 as M
    if mode == "chunk" and 64 % G:
        pytest.skip("a chunk holds whole positions")
    B, H, dt = 2, 3, torch.bfloat16
    gen = torch.Generator(device="cuda").manual_seed(T + L)
    mk = lambda n: torch.randn(B, n, H, D, generator=gen, device="cuda", dtype=dt)  # noqa: E731
    q, k, v, dout = mk(T * G), mk(T), mk(T), mk(T * G)
    layers = [(mk(T), mk(T)) for _ in range(L)]
    # what the shared memory holds before the kernels under test run: NaN
    nan = torch.full((1, 4096, 8, D), float("nan"), device="cuda", dtype=dt)
    M.parallel_moda_fwd(nan, nan, nan)

    leaves = [x.requires_grad_(True) for x in (q, k, v)]
    rows = [x.requires_grad_(True) for lay in layers for x in lay]
    cache = M.DepthKVCache(B, T, cap, H, D, dt, "cuda")
    cache.k.fill_(float("nan"))
    cache.v.fill_(float("nan"))
    for lk, lv in layers:
        cache.append(lk, lv)
    o, lse = cache.attend(q, k, v, moda_group_num=G, is_causal=mode == "causal", chunk_visible=mode == "chunk", need_lse=True)
    grads = torch.autograd.grad(o, leaves + rows, dout)

    kd, vd = [torch.stack([lay[i].detach() for lay in layers], dim=2).view(B, T * L, H, D).requires_grad_(True) for i in (0, 1)]
    if mode == "chunk":
        o2, lse2 = M.parallel_moda_chunk_visible(q, k, v, cached_k=kd, cached_v=vd, moda_group_num=G, need_lse=True)
    else:
        o2, lse2 = M.parallel_moda(q, k, v, cached_k=kd, cached_v=vd, moda_group_num=G, is_causal=mode == "causal", need_lse=True)
    ref = torch.autograd.grad(o2, leaves + [kd, vd], dout)
    assert max_abs(o, o2) <= 2 ** -6 * o2.abs().max().item() and max_abs(lse, lse2) <= 1e-4     # two roundings to bf16
    got = list(grads[:3]) + [torch.stack(grads[3 + i::2], dim=2).view_as(kd) for i in (0, 1)]
    for name, a, b in zip(("dq", "dk", "dv", "d_depth_k", "d_depth_v"), got, ref):
        a, b = a.float(), b.float()
        err, size = (a - b).norm(dim=-1), b.norm(dim=-1)          # row by row: none missing, none foreign
        assert (err <= 2e-2 * (size + size.mean()) + 1e-3).all(), name
    assert M.device_status() == 0


@pytest.mark.parametrize("D", [64, 128])
def test_a_later_sequence_row_that_is_not_finite(built_library, D):
    """Two query tiles share the forward's V slots: what the second one's sequence tile leaves behind a depth
    tile that does not fill its slot is not multiplied into the first one's rows.  L = 33: depth tiles of 99
    rows, 43 of them for the first query tile (rows 256..383) and 37 for the second (384..493), so that the
    first meets both slots after the key tile of positions 384..493."""
    import moda_b200 as M
    B, T, H, L, dt = 10, 494, 8, 33, torch.bfloat16
    gen = torch.Generator(device="cuda").manual_seed(D)
    mk = lambda: torch.randn(B, T, H, D, generator=gen, device="cuda", dtype=dt)  # noqa: E731
    q, k, v = mk(), mk(), mk()
    cache = M.DepthKVCache(B, T, L + 1, H, D, dt, "cuda")
    for _ in range(L):
        cache.append(mk(), mk())
    clean = cache.attend(q, k, v, chunk_visible=True)
    v[:, 384 + 105] = float("inf")
    dirty = cache.attend(q, k, v, chunk_visible=True)
    assert torch.equal(clean[:, :384], dirty[:, :384])
