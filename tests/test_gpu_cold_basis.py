"""Projections that start a basis (the first warm call after none: block-Jacobi
sweeps, as a solve's first iteration) and the plain mode (Jacobi kernels on every
block) against LAPACK.  A stand-alone projection in the default mode takes
neither: it goes by the matrix sign function."""
import numpy as np
import pytest

import hilbert_b200 as hb
from oracle.bpsdp import project_blocks

pytestmark = pytest.mark.gpu

TOL = 1e-11   # |x - x_ref|_max <= TOL * max(1, |U|_F), as for every eigenvector route


def cold(p, U, mu):
    """a projection from the identity basis by the route that keeps one"""
    p.project(U, mu)   # forgets the basis
    return p.project(U, mu, warm=True)


def matches(x, z, U, dims, mu):
    xr, zr = project_blocks(U, dims, mu)
    bound = TOL * max(1.0, np.linalg.norm(U))
    ex, ez = np.max(np.abs(x.cpu().numpy() - xr)), np.max(np.abs(z.cpu().numpy() - zr))
    assert ex <= bound and ez <= bound, (ex, ez, bound)


def from_spectra(dims, rng, spectrum):
    U = []
    for k, d in enumerate(int(v) for v in dims):
        q = np.linalg.qr(rng.standard_normal((d, d)))[0]
        U.append(((q * spectrum(k, d)) @ q.T).ravel())
    return np.concatenate(U)


@pytest.mark.parametrize("mode", ["refine", "jacobi"])
@pytest.mark.parametrize("n,na,nb", [(5, 3, 2), (7, 4, 4), (9, 5, 4)])
def test_ragged_blocks_with_clusters(cuda_device, n, na, nb, mode):
    """Blocks of 25, 50, 21, 49, 98, 36, 81 and 162 rows end in groups of 1 to 31
    rows, odd pairs and an odd group count; clusters of equal eigenvalues and
    exact zeros keep pairs that never rotate."""
    import torch
    p = hb.V2RDMProblem(n, na, nb)
    rng = np.random.default_rng(n)

    def spectrum(k, d):
        lam = rng.uniform(-2.0, 2.0, d)
        lam[: d // 3] = 1.0
        lam[d // 3: d // 2] = 0.0
        return lam
    U = from_spectra(p.dims, rng, spectrum)
    Ud = torch.from_numpy(U).to(cuda_device)
    p.set_projection_mode(mode)
    out = []
    for _ in range(2):
        x, z = cold(p, Ud, 0.8) if mode == "refine" else p.project(Ud, 0.8)
        matches(x, z, U, p.dims, 0.8)
        out.append((x, z))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    rc = p.refine_counts()
    assert rc["block_jacobi_sweeps"] > 0 if mode == "refine" else rc["jacobi"] >= 2 * len(p.dims), rc
    p.close()


@pytest.mark.parametrize("mode", ["refine", "jacobi"])
@pytest.mark.parametrize("n", [4, 10])
def test_degenerate_and_definite_blocks(cuda_device, n, mode):
    """Blocks that are positive, negative or split in two clusters at +-1; with
    n = 10 up to 200 rows (two CTA sizes of the Jacobi kernels)."""
    import torch
    p = hb.V2RDMProblem(n, n // 2, n // 2)

    def spectrum(k, d):
        return (np.full(d, 2.0), np.full(d, -1.0), np.repeat([1.0, -1.0], (d + 1) // 2)[:d])[k % 3]
    U = from_spectra(p.dims, np.random.default_rng(5), spectrum)
    Ud = torch.from_numpy(U).to(cuda_device)
    p.set_projection_mode(mode)
    x, z = cold(p, Ud, 1.0) if mode == "refine" else p.project(Ud, 1.0)
    matches(x, z, U, p.dims, 1.0)
    p.close()


@pytest.mark.parametrize("n", [10, 20])
def test_repeated_cold_basis_of_general_blocks(cuda_device, n):
    """General (non-symmetric) blocks of up to 200 and 800 rows, slowly changed:
    the work arrays are reused between calls."""
    import torch
    p = hb.V2RDMProblem(n, n // 2, n // 2)
    rng = np.random.default_rng(3)
    U = rng.standard_normal(p.n_primal)
    for k in range(2):
        U2 = U + 1e-4 * k * rng.standard_normal(p.n_primal)
        before = p.refine_counts()["block_jacobi_sweeps"]
        x, z = cold(p, torch.from_numpy(U2).to(cuda_device), 0.5)
        matches(x, z, U2, p.dims, 0.5)
        assert p.refine_counts()["block_jacobi_sweeps"] > before
    p.close()


def test_split_k_gemm_matches_lapack_and_repeats(cuda_device):
    """Blocks of 324 and 648 rows (n = 18) with their GEMM tiles cut along K and in
    one piece; the parts are summed in a fixed order, so two projections with one
    plan give the same bits."""
    import torch
    p = hb.V2RDMProblem(18, 9, 9)
    rng = np.random.default_rng(18)
    U = rng.standard_normal(p.n_primal)
    Ud = torch.from_numpy(U).to(cuda_device)
    out = {}
    for on in (True, False, True):
        p.set_gemm_split(on)
        x, z = cold(p, Ud, 0.61)
        matches(x, z, U, p.dims, 0.61)
        if on in out:
            assert torch.equal(out[on][0], x) and torch.equal(out[on][1], z)
        out[on] = (x, z)
    # the autotuner's choice here is 2 parts (full list) and 4 (upper list); at
    # n = 12 .. 16 it leaves the tiles whole
    assert max(p.gemm_split_choice()) > 1
    p.close()
