"""Device memory that the library keeps between calls (no counterpart in the
reference) goes back to the device on request."""
import pytest

import libigl_gb300 as G
from libigl_gb300 import synth

pytestmark = pytest.mark.gpu


def _make_and_close_a_cloud(torch, n):
    P = torch.randn(n, 3, device="cuda", dtype=torch.float64)
    P /= P.norm(dim=1, keepdim=True)
    A = torch.full((n,), 12.566 / n, device="cuda", dtype=torch.float64)
    G.CloudExpansion(P, P, A).close()


def test_release_memory(cuda):
    """What closed handles and workspaces have left mapped (a few GB here, at
    most a sixteenth of the device of the handles') goes back to the device."""
    V, F = synth.icosphere(2)
    bvh = G.FastWindingNumberBVH(V, F)
    bvh.eval(V)
    _make_and_close_a_cloud(cuda, 1000)  # the kernels are loaded
    G.release_memory()
    cuda.cuda.empty_cache()
    before, _ = cuda.cuda.mem_get_info()
    _make_and_close_a_cloud(cuda, 3_000_000)
    cuda.cuda.empty_cache()
    kept = before - cuda.cuda.mem_get_info()[0]
    G.release_memory()
    left = before - cuda.cuda.mem_get_info()[0]
    assert left <= 64 << 20 < kept
    # kept handles are not touched
    assert abs(bvh.eval(V * 0.1)[0] - 1) <= 1e-2
    bvh.close()
