"""GPU: gradients of a stack of layers over ``DepthKVCache`` when the pass is not the plain one (every layer
recorded, on one stream, one backward).  Reference: the packed cache rebuilt before every layer
(``torch.stack`` of the earlier layers' K/V) through the ordinary operator."""
import pytest
import torch

from tests.helpers import check_grad

pytestmark = pytest.mark.gpu

T, H, D, G = 150, 3, 64, 2


def _leaves(seed, n_layers):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mk = lambda n: torch.randn(2, n, H, D, generator=gen, device="cuda", dtype=torch.bfloat16).requires_grad_(True)  # noqa: E731
    return [(mk(T * G), mk(T), mk(T)) for _ in range(n_layers)], [mk(T * G).detach() for _ in range(n_layers)]


def _rebuilt(layers, frozen=()):
    """Outputs of all layers; those in `frozen` are not recorded, neither the attention nor the append."""
    import moda_b200 as M
    outs, kv = [], []
    for i, (q, k, v) in enumerate(layers):
        ck, cv = [torch.stack([x[j] for x in kv], dim=2).view(2, T * i, H, D) if kv else None for j in (0, 1)]
        with torch.set_grad_enabled(i not in frozen):
            outs.append(M.parallel_moda(q, k, v, cached_k=ck, cached_v=cv, moda_group_num=G))
        kv.append((k.detach(), v.detach()) if i in frozen else (k, v))
    return outs


def _cached(layers, frozen=()):
    """The same through the in-place cache."""
    import moda_b200 as M
    cache = M.DepthKVCache(2, T, len(layers) - 1, H, D, torch.bfloat16, "cuda")
    outs = []
    for i, (q, k, v) in enumerate(layers):
        with torch.set_grad_enabled(i not in frozen):
            outs.append(cache.attend(q, k, v, moda_group_num=G))
        if i + 1 < len(layers):
            with torch.set_grad_enabled(i not in frozen):
                cache.append(k, v)
    return outs


def _check(got, want):
    for i, (a, b) in enumerate(zip(got, want)):
        check_grad(f"leaf {i}", a.float().cpu(), b.float().cpu())


@pytest.mark.parametrize("frozen", [(1,), (2,), (0, 1), (1, 2)])
def test_layers_that_are_not_recorded(built_library, frozen):
    """They hand no gradient on themselves and take none from the layers before them."""
    layers, dout = _leaves(1, 4)
    live = [i for i in range(4) if i not in frozen]
    leaves = [x for i in live for x in layers[i]]
    got, want = [torch.autograd.grad([outs[i] for i in live], leaves, [dout[i] for i in live])
                 for outs in (_cached(layers, frozen), _rebuilt(layers, frozen))]
    _check(got, want)
