"""GPU: key gradients written over the keys themselves (a caller that has no other buffer): the kernels that
read the keys have ended, or own the rows, when a gradient row is stored.  Reference: the same call into
separate buffers, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,T,G,D,L", [
    ("causal", 1500, 4, 128, 3),      # dq, dk/dv and depth gradients would overlap; dk/dv in clusters
    ("causal", 700, 3, 64, 5),        # the key-parallel kernel takes the depth rows
    ("chunk", 1024, 2, 128, 8),
    ("all", 900, 1, 128, 4),          # depth rows in the bandwidth kernels
    ("all", 197, 1, 64, 11),          # one CTA a head
])
def test_key_gradients_over_the_keys(built_library, mode, T, G, D, L):
    import moda_b200 as M
    from moda_b200 import _cabi, ops
    m = {"causal": _cabi.MODE_CAUSAL, "all": _cabi.MODE_NONCAUSAL, "chunk": _cabi.MODE_CHUNK_VISIBLE}[mode]
    mk = lambda n: torch.randn(1, n, 2, D, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    q, k, v, kd, vd, dout = mk(T * G), mk(T), mk(T), mk(T * L), mk(T * L), mk(T * G)
    o, lse = ops._forward(q, k, v, kd, vd, D ** -0.5, G, m)
    want = [torch.empty_like(x) for x in (q, k, v, kd, vd)]
    ops.backward_into_static_scratch(q, k, v, kd, vd, o, lse, dout, *want, D ** -0.5, G, m)
    for _ in range(5):
        ks = [x.clone() for x in (k, v, kd, vd)]
        dq = torch.empty_like(q)
        ops.backward_into_static_scratch(q, *ks, o, lse, dout, dq, *ks, D ** -0.5, G, m)
        for name, a, b in zip(("dq", "dk", "dv", "d_depth_k", "d_depth_v"), [dq] + ks, want):
            assert torch.equal(a, b), name
    assert M.device_status() == 0
