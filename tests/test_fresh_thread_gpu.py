"""GPU: the library's calls from a thread that has done nothing on the GPU before (an autograd thread whose
allocations the caching allocator serves without a CUDA call)."""
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

_PROGRAM = """
import threading
import torch
import moda_b200 as M
mk = lambda n: torch.randn(1, n, 2, 64, device="cuda", dtype=torch.bfloat16).requires_grad_(True)
q, k, v, kd, vd = mk(300), mk(300), mk(300), mk(900), mk(900)
want = M.parallel_moda(q, k, v, cached_k=kd, cached_v=vd)
want = torch.autograd.grad(want, [q, k, v, kd, vd], torch.ones_like(want))       # the first backward: the engine's thread
got = []
t = threading.Thread(target=lambda: got.append(M.parallel_fda_fwd(q.detach(), cached_k=kd.detach(), cached_v=vd.detach())))
t.start()
t.join()
assert got and torch.equal(got[0][0], M.parallel_fda_fwd(q.detach(), cached_k=kd.detach(), cached_v=vd.detach())[0])
assert all(torch.isfinite(g.float()).all() for g in want) and M.device_status() == 0
"""


def test_first_call_of_a_thread(built_library):
    r = subprocess.run([sys.executable, "-c", _PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
