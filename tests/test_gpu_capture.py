"""A stand-alone projection in a CUDA graph: after a first call (which makes the
plan and its lists) it is launches only, so a capture on the same stream replays
it; the bits are the eager call's."""
import pytest

import hilbert_b200 as hb

pytestmark = pytest.mark.gpu


def test_projection_captured_after_its_first_call(cuda_device):
    import torch
    p = hb.V2RDMProblem(8, 4, 4)
    U = torch.randn(p.n_primal, dtype=torch.float64, device=cuda_device)
    V = torch.randn(p.n_primal, dtype=torch.float64, device=cuda_device)
    want = [p.project(W, 0.6) for W in (U, V)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        p.project(U, 0.6)
    torch.cuda.synchronize()
    W = U.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        x, z = p.project(W, 0.6)
    for src, (xr, zr) in zip((U, V), want):
        W.copy_(src)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, xr) and torch.equal(z, zr)
    with torch.cuda.stream(s):   # the stream's next eager call
        x2, _ = p.project(U, 0.6)
    torch.cuda.synchronize()
    assert torch.equal(x2, want[0][0])
    p.close()
