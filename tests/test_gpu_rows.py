"""The map kernels' split of rows (a thread for a short one, a warp with chunks
of 128 entries for a long one) and the one-CTA Jacobi kernel around its edges."""
import ctypes

import numpy as np
import pytest

import hilbert_b200 as hb
from hilbert_b200 import _capi
from oracle.bpsdp import project_blocks
from oracle.maps import OracleProblem

pytestmark = pytest.mark.gpu


# rows of up to n^2 entries: 1 to 36, 121 (one chunk), 169 (two)
@pytest.mark.parametrize("n,na,nb,pos", [(1, 1, 1, "DQG"), (5, 3, 2, "DQG"), (6, 3, 3, "DQGT1T2"),
                                         (11, 6, 6, "DQG"), (13, 7, 6, "DG")])
def test_rows_bit_exact(cuda_device, n, na, nb, pos):
    import torch
    rng = np.random.default_rng(n)
    o = OracleProblem(n, na, nb, pos, 1, 1, h=rng.standard_normal((n, n)), g=rng.standard_normal((n,) * 4))
    p = hb.V2RDMProblem(n, na, nb, pos)
    x, y = rng.standard_normal(o.n_primal), rng.standard_normal(o.n_dual)
    assert np.array_equal(p.Au(torch.from_numpy(x).to(cuda_device)).cpu().numpy(), o.Au(x))
    assert np.array_equal(p.ATu(torch.from_numpy(y).to(cuda_device)).cpu().numpy(), o.ATu(y))
    p.close()


# odd sizes, one warp of pairs and more, both sides of the size up to which the
# eigenvectors stay in shared memory
@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 63, 66, 79, 80, 81, 82, 127, 128])
@pytest.mark.parametrize("spec", ["normal", "zero"])
def test_one_cta_jacobi(cuda_device, n, spec):
    import torch
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n))
    U = {"normal": a + a.T, "zero": 0.0 * a}[spec].ravel()
    xr, zr = project_blocks(U, [n], 0.5)
    d = torch.from_numpy(U).to(cuda_device)
    x, z = torch.full_like(d, float("nan")), torch.full_like(d, float("nan"))
    rc = _capi.load().v2b_project_block_noalloc(
        ctypes.c_void_p(d.data_ptr()), n, 0.5, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(z.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _capi.V2B_OK
    # 10 sweeps of n rotations a row, each rounding by a few eps: 10 * 128 * 4 eps
    tol = 1.2e-12 * max(np.linalg.norm(U), 1e-300)
    assert np.max(np.abs(x.cpu().numpy() - xr)) <= 2 * tol   # x = U+ / mu
    assert np.max(np.abs(z.cpu().numpy() - zr)) <= tol


# the acceptance test's 32-row tile pairs: blocks of one partial tile, of whole
# tiles (64, 128), of a last tile of one to four rows (36, 66, 100), of seven
@pytest.mark.parametrize("n,na,nb", [(5, 3, 2), (8, 4, 4), (9, 5, 4), (10, 5, 5)])
@pytest.mark.parametrize("step", [1e-12, 1e-5, 1e-2])
def test_acceptance_on_ragged_tiles(cuda_device, n, na, nb, step):
    import torch
    p = hb.V2RDMProblem(n, na, nb)
    rng = np.random.default_rng(n)
    def symmetric():
        blocks = [rng.standard_normal((int(d), int(d))) for d in p.dims]
        return np.concatenate([(a + a.T).ravel() for a in blocks])
    U = symmetric()
    for k in range(3):   # from scratch, then warm: accepted, rotated, restarted
        V = U + k * step * symmetric()
        xr, zr = project_blocks(V, p.dims, 0.8)
        x, z = p.project(torch.from_numpy(V).to(cuda_device), 0.8, warm=True)
        tol = 1e-11 * np.linalg.norm(V)   # as the other projection tests, which the acceptance rule sets
        assert np.max(np.abs(x.cpu().numpy() - xr)) <= tol
        assert np.max(np.abs(z.cpu().numpy() - zr)) <= tol
    p.close()
