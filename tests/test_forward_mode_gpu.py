"""GPU: the operators have no forward-mode derivative and say so, instead of dropping the tangent."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [0, 2, 3])
@pytest.mark.parametrize("warn_shape", [True, False])    # T < H: with the warning the call takes the Python wrapper
def test_a_dual_number_is_refused(built_library, which, warn_shape):
    import moda_b200 as M
    xs = [torch.randn(1, n, 4, 64, device="cuda", dtype=torch.bfloat16) for n in (3, 3, 3, 6, 6)]
    cache = M.DepthKVCache(1, 3, 2, 4, 64, torch.bfloat16, "cuda")
    with fwAD.dual_level(), torch.no_grad(), pytest.warns(UserWarning) if warn_shape else torch.no_grad():
        xs[which] = fwAD.make_dual(xs[which], torch.ones_like(xs[which]))
        with pytest.raises(NotImplementedError):
            M.parallel_moda(*xs[:3], cached_k=xs[3], cached_v=xs[4], warn_shape=warn_shape)
        if which < 3:
            with pytest.raises(NotImplementedError):
                cache.attend(*xs[:3])
        if which == 2:
            with pytest.raises(NotImplementedError):
                cache.append(*xs[1:3])
