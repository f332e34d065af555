"""Stand-alone projections (matrix sign function) against LAPACK at the edges:
block sizes around one MMA tile, one CTA and one GEMM tile, spectra that the
iteration has to resolve over many decades, magnitudes near the type's range."""
import numpy as np
import pytest

import hilbert_b200 as hb
from oracle.bpsdp import project_blocks

pytestmark = pytest.mark.gpu

# 43 steps of two products, each rounding by a few n eps of a matrix of norm
# one, over blocks of up to 162 rows
TOL = 1e-12


def spectrum(d, kind, rng):
    if kind == "zero":
        return np.zeros(d)
    if kind == "decades":   # both signs over 16 decades
        return np.where(rng.random(d) < 0.5, 1.0, -1.0) * 10.0 ** rng.uniform(-16.0, 0.0, d)
    if kind == "lowrank":
        return np.where(np.arange(d) < max(1, d // 10), 1.0, 0.0)
    if kind == "definite":
        return rng.uniform(0.1, 1.0, d) * (1.0 if d % 2 else -1.0)
    return rng.standard_normal(d)


@pytest.mark.parametrize("kind,n,na,nb", [("doci", 10, 5, 5), ("v2rdm", 3, 2, 1), ("v2rdm", 8, 4, 4),
                                          ("v2rdm", 9, 5, 4)])
@pytest.mark.parametrize("spec", ["normal", "zero", "decades", "lowrank", "definite"])
@pytest.mark.parametrize("scale", [1.0, 1e-200, 1e150])
def test_projection_from_scratch(cuda_device, kind, n, na, nb, spec, scale):
    import torch
    p = (hb.DOCIProblem if kind == "doci" else hb.V2RDMProblem)(n, na, nb, "DQG")
    rng = np.random.default_rng(n)
    U = []
    for d in (int(v) for v in p.dims):
        q = np.linalg.qr(rng.standard_normal((d, d)))[0]
        U.append(((q * spectrum(d, spec, rng)) @ q.T).ravel())
    U = np.concatenate(U)
    xr, zr = project_blocks(U, p.dims, 0.5)   # the reference at magnitude one
    x, z = p.project(torch.from_numpy(U * scale).to(cuda_device), 0.5)
    tol = TOL * max(np.linalg.norm(U), 1e-300)
    assert np.max(np.abs(x.cpu().numpy() / scale - xr)) <= tol
    assert np.max(np.abs(z.cpu().numpy() / scale - zr)) <= tol
    p.close()


def test_projection_then_other_stream(cuda_device):
    """A projection on one stream, then a warm one and a second one on another
    without a synchronisation between: the work arrays are shared."""
    import torch
    p = hb.V2RDMProblem(9, 5, 4)
    rng = np.random.default_rng(1)
    U = [torch.from_numpy(rng.standard_normal(p.n_primal)).to(cuda_device) for _ in range(3)]
    ref = [project_blocks(u.cpu().numpy(), p.dims, 0.5) for u in U]
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    out = [p.project(U[0], 0.5)]
    with torch.cuda.stream(other):
        out.append(p.project(U[1], 0.5))
        out.append(p.project(U[2], 0.5, warm=True))
    torch.cuda.synchronize()
    for (x, z), (xr, zr), u in zip(out, ref, U):
        tol = 1e-11 * float(torch.linalg.vector_norm(u))
        assert np.max(np.abs(x.cpu().numpy() - xr)) <= tol
        assert np.max(np.abs(z.cpu().numpy() - zr)) <= tol
