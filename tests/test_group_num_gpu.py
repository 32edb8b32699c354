"""GPU: ``moda_group_num`` as the integers that a configuration may hold it in, on the call that goes straight
to the kernels and on the one that takes the Python wrapper (head_first)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("g", [np.int64(2), np.int32(2), np.uint8(2), torch.tensor(2)], ids=lambda g: str(g.dtype))
@pytest.mark.parametrize("head_first", [False, True])
def test_any_integer(built_library, g, head_first):
    import moda_b200 as M
    q, k, v, kd, vd = [torch.randn(1, n, 4, 64, device="cuda", dtype=torch.bfloat16) for n in (128, 64, 64, 192, 192)]
    xs = [x.transpose(1, 2).contiguous() if head_first else x for x in (q, k, v, kd, vd)]
    for call in (lambda n: M.parallel_moda(*xs[:3], cached_k=xs[3], cached_v=xs[4], moda_group_num=n, head_first=head_first),
                 lambda n: M.parallel_moda_chunk_visible(*xs[:3], cached_k=xs[3], cached_v=xs[4], moda_group_num=n, head_first=head_first),
                 lambda n: M.parallel_fda(xs[0], cached_k=xs[3], cached_v=xs[4], moda_group_num=n, head_first=head_first)):
        assert torch.equal(call(g), call(2))


def test_a_number_that_is_no_integer_is_refused(built_library):
    import moda_b200 as M
    q, k = [torch.randn(1, n, 4, 64, device="cuda", dtype=torch.bfloat16) for n in (128, 64)]
    with pytest.raises(TypeError):
        M.parallel_moda(q, k, k, moda_group_num=2.0)
