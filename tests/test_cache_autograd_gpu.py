"""GPU: gradients of a stack of layers over ``DepthKVCache`` when the pass is not the plain one (every layer
recorded, on one stream, one backward).  Reference: the packed cache rebuilt before every layer
(``torch.stack`` of the earlier layers' K/V) through the ordinary operator."""
import copy
import pickle
import time

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


def _cached(layers, frozen=(), streams=lambda i: (None, None)):
    """The same through the in-place cache, layer i's attention and append on `streams(i)`."""
    import moda_b200 as M
    cache = M.DepthKVCache(2, T, len(layers) - 1, H, D, torch.bfloat16, "cuda")
    outs = []
    for i, (q, k, v) in enumerate(layers):
        attend_on, append_on = streams(i)
        with torch.cuda.stream(attend_on), torch.set_grad_enabled(i not in frozen):
            outs.append(cache.attend(q, k, v, moda_group_num=G))
        if i + 1 < len(layers):
            with torch.cuda.stream(append_on), torch.set_grad_enabled(i not in frozen):
                cache.append(k, v)
        if attend_on is not None:
            torch.cuda.synchronize()             # the forward's own order is the caller's to keep
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


@pytest.mark.parametrize("which", ["append", "layers"])
def test_streams(built_library, which):
    """The gradient cache is ordered between the streams that the backward runs on: here every attention's
    share of it comes late."""
    layers, dout = _leaves(2, 5)
    leaves = [x for lay in layers for x in lay]
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    streams = (lambda i: (main, side)) if which == "append" else (lambda i: (main, side) if i % 2 else (side, side))
    outs = _cached(layers, streams=streams)

    def late(grad):
        torch.cuda._sleep(4_000_000)
        return grad

    for o in outs:
        o.register_hook(late)
    got = torch.autograd.grad(outs, leaves, dout)
    torch.cuda.synchronize()
    _check(got, torch.autograd.grad(_rebuilt(layers), leaves, dout))


@pytest.mark.parametrize("how", ["twice", "one leaf first", "a loss a layer"])
def test_several_backwards_of_one_forward(built_library, how):
    """Each delivers its own gradients once."""
    layers, dout = _leaves(3, 4)
    leaves = [x for lay in layers for x in lay]

    def backwards(outs):
        if how == "twice":
            torch.autograd.grad(outs, leaves, dout, retain_graph=True)
        elif how == "one leaf first":
            torch.autograd.grad(outs[-1], layers[-1][0], dout[-1], retain_graph=True)
        else:
            for x in leaves:
                x.grad = None
            for o, d in zip(outs, dout):
                o.backward(d)
            return [x.grad for x in leaves]
        return torch.autograd.grad(outs, leaves, dout)

    _check(backwards(_cached(layers)), backwards(_rebuilt(layers)))


@pytest.mark.parametrize("how", ["deepcopy", "pickle"])
@pytest.mark.parametrize("train", [False, True])
def test_copies_of_a_used_cache(built_library, how, train):
    """A module that keeps one stays copyable; what was recorded stays with the original."""
    import moda_b200 as M
    layers, dout = _leaves(4, 3)
    cache = M.DepthKVCache(2, T, 3, H, D, torch.bfloat16, "cuda")
    with torch.set_grad_enabled(train):
        for q, k, v in layers[:2]:
            o = cache.attend(q, k, v, moda_group_num=G)
            cache.append(k, v)
    if train:
        o.backward(dout[0])
        if how == "deepcopy":                    # a tensor with a history, as ever
            with pytest.raises(RuntimeError):
                copy.deepcopy(cache)
            return
    other = copy.deepcopy(cache) if how == "deepcopy" else pickle.loads(pickle.dumps(cache))
    assert other.L == 2 and other.k.data_ptr() != cache.k.data_ptr()
    assert (other.grad_k is None) == (not train)
    if train:                                    # the first backward filled one layer of three
        at = lambda x: x.view(2, T, 3, H, D)[:, :, 0]  # noqa: E731
        assert torch.equal(at(other.grad_k), at(cache.grad_k)) and torch.equal(at(other.grad_v), at(cache.grad_v))
    with torch.no_grad():
        assert torch.equal(other.attend(*layers[2], moda_group_num=G), cache.attend(*layers[2], moda_group_num=G))


def test_a_deeper_layer_after_an_earlier_one(built_library):
    """The first attention whose backward runs stores its share of the gradient cache; one that read more layers
    and comes later (its gradient comes by way of the CPU) finds the slots beyond it cleared."""
    layers, dout = _leaves(5, 4)
    leaves = [x for lay in layers for x in lay]

    def grads(outs):
        last = outs[3].cpu()
        last.register_hook(lambda g: time.sleep(0.3))
        for x in leaves:
            x.grad = None
        torch.autograd.backward([outs[0], outs[1], outs[2], last], dout[:3] + [dout[3].cpu()])
        return [x.grad for x in leaves]

    _check(grads(_cached(layers)), grads(_rebuilt(layers)))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_deep_stack(built_library, causal, D):
    """G = 1, up to 21 cached layers: the bandwidth kernels add gradients in more than one step of a unit."""
    import moda_b200 as M
    gen = torch.Generator(device="cuda").manual_seed(D)
    B, T, H, N = 2, 45, 2, 22
    mk = lambda: torch.randn(B, T, H, D, generator=gen, device="cuda", dtype=torch.bfloat16).requires_grad_(True)  # noqa: E731
    layers, dout = [(mk(), mk(), mk()) for _ in range(N)], [mk().detach() for _ in range(N)]
    leaves = [x for lay in layers for x in lay]
    cache = M.DepthKVCache(B, T, N + 1, H, D, torch.bfloat16, "cuda")
    cache.k.fill_(float("nan"))
    cache.v.fill_(float("nan"))
    outs, want, kv = [], [], []
    for i, (q, k, v) in enumerate(layers):
        outs.append(cache.attend(q, k, v, is_causal=causal))
        ck, cv = [torch.stack([x[j] for x in kv], dim=2).view(B, T * i, H, D) if kv else None for j in (0, 1)]
        want.append(M.parallel_moda(q, k, v, cached_k=ck, cached_v=cv, is_causal=causal))
        cache.append(k, v)
        kv.append((k, v))
    assert all(torch.equal(a, b) for a, b in zip(outs, want))
    _check(torch.autograd.grad(outs, leaves, dout), torch.autograd.grad(want, leaves, dout))
    assert M.device_status() == 0
