"""GPU: what the depth-only kernels keep of fp32 probabilities and score gradients.  Reference: the same in 64
bits from the same rounded inputs (the backward's o and lse among them)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

U = {torch.bfloat16: 2. ** -8, torch.float16: 2. ** -11}      # unit roundoff of a result
STEP = {torch.bfloat16: 0., torch.float16: 2. ** -24}         # spacing of the smallest results


def _case(dt, G, L, D, sizes, seed=0):
    """The operator's outputs, their 64-bit values, and for each the sum of the magnitudes of its terms."""
    import moda_b200 as M
    B, T, H = 1, 200, 4
    gen = torch.Generator(device="cuda").manual_seed(seed + L * G + D)
    mk = lambda n, size: (torch.randn(B, n, H, D, generator=gen, device="cuda") * size).to(dt)  # noqa: E731
    q, kd, vd, do = [mk(n, size) for n, size in zip((T * G, T * L, T * L, T * G), sizes)]
    Q, K, V, DO = [x.double().view(B, T, -1, H, D) for x in (q, kd, vd, do)]
    scores = torch.einsum("btghd,btlhd->btghl", Q, K) * D ** -0.5
    lse = torch.logsumexp(scores, -1)
    P = torch.exp(scores - lse[..., None])
    O = torch.einsum("btghl,btlhd->btghd", P, V)
    o, _ = M.parallel_fda_fwd(q, cached_k=kd, cached_v=vd, moda_group_num=G)
    o_in, lse_in = O.to(dt).reshape(q.shape), (lse / torch.log(torch.tensor(2., device="cuda"))).float().reshape(B, T * G, H)
    dq, _, dk, dv = M.parallel_fda_bwd(q, o_in, None, lse_in, do, cached_k=kd, cached_v=vd, moda_group_num=G)
    P2 = torch.exp2(scores / torch.log(torch.tensor(2., dtype=torch.double, device="cuda")) - lse_in.double().view(B, T, G, H)[..., None])
    dP, delta = torch.einsum("btghd,btlhd->btghl", DO, V), (o_in.double().view(B, T, G, H, D) * DO).sum(-1)[..., None]
    dS = P2 * (dP - delta) * D ** -0.5
    sizeS = P2 * (torch.einsum("btghd,btlhd->btghl", DO.abs(), V.abs()) + delta.abs()) * D ** -0.5
    out = {"o": (o, O, torch.einsum("btghl,btlhd->btghd", P, V.abs())),
           "dq": (dq, torch.einsum("btghl,btlhd->btghd", dS, K), torch.einsum("btghl,btlhd->btghd", sizeS, K.abs())),
           "dk": (dk, torch.einsum("btghl,btghd->btlhd", dS, Q), torch.einsum("btghl,btghd->btlhd", sizeS, Q.abs())),
           "dv": (dv, torch.einsum("btghl,btghd->btlhd", P2, DO), torch.einsum("btghl,btghd->btlhd", P2, DO.abs()))}
    return {n: (a.double().flatten(), e.flatten(), m.flatten()) for n, (a, e, m) in out.items()}


@pytest.mark.parametrize("sizes", [(1., 1., 1., 1e-5),                     # gradients near the smallest fp16 numbers
                                   (2. ** -6, 2. ** -6, 64., 8000.)],      # scale dS beyond the largest, no result is
                         ids=["small", "large"])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("G,L,D", [(1, 4, 64), (1, 24, 64), (2, 11, 128), (4, 24, 128), (3, 17, 64), (8, 24, 64), (8, 11, 128)])
def test_range(built_library, G, L, D, dt, sizes):
    """Element by element: half a step of the result, and fp32 sums (2^-24 for each of up to 128 + 64 terms, of the
    sum of their magnitudes; two parts, G > 4 in bf16: 2^-16 of it)."""
    for name, (a, e, m) in _case(dt, G, L, D, sizes).items():
        assert ((a - e).abs() <= U[dt] * e.abs() + STEP[dt] / 2 + 2. ** -16 * m).all(), name


@pytest.mark.parametrize("D", [64, 128])
def test_bits(built_library, D):
    """How many bf16 results are not the rounded exact one: o 1e-4 and dv 4e-5 with fp32 P, 1.4e-3 and 5e-4 with P
    of 17 bits."""
    total = {"o": [], "dv": []}
    for G, L in ((1, 11), (2, 32), (4, 24), (3, 5)):
        case = _case(torch.bfloat16, G, L, D, (1., 1., 1., 1.))
        for name in total:
            a, e, _ = case[name]
            total[name].append((a != e.to(torch.bfloat16).double()).double().mean().item())
    assert sum(total["o"]) / 4 < 4e-4 and sum(total["dv"]) / 4 < 2e-4, total


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("G,L", [(1, 4), (2, 24), (8, 4), (8, 24)])
def test_an_infinite_row_of_v(built_library, G, L, dt):
    """Its channel of o is infinite, as P V is, and the others are what they are without it."""
    import moda_b200 as M
    T, D = 64, 64
    gen = torch.Generator(device="cuda").manual_seed(L)
    q, kd, vd = [torch.randn(1, n, 2, D, generator=gen, device="cuda").to(dt) for n in (T * G, T * L, T * L)]
    clean, _ = M.parallel_fda_fwd(q, cached_k=kd, cached_v=vd, moda_group_num=G)
    vd.view(1, T, L, 2, D)[:, :, 1, :, 3] = float("inf")
    o, _ = M.parallel_fda_fwd(q, cached_k=kd, cached_v=vd, moda_group_num=G)
    assert (o[..., 3] == float("inf")).all()
    keep = [i for i in range(D) if i != 3]
    assert torch.equal(o[..., keep], clean[..., keep])
