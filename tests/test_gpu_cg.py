"""The conjugate-gradient kernel in each of its forms (one CTA, one CTA per SM
with one, two or three virtual CTAs, tables in shared memory side by side, in
one region, or streamed): the y of one outer iteration solves
(A A^T) y = A c + mu (b - A x0) to the CG tolerance, checked with the bit-exact
maps."""
import numpy as np
import pytest

import hilbert_b200 as hb

pytestmark = pytest.mark.gpu

CASES = [("doci", 10, 5, 5, "DQG"),        # one CTA, two virtual CTAs
         ("v2rdm", 2, 1, 1, "DQG"),        # one virtual CTA
         ("v2rdm", 4, 2, 2, "DQG"),        # one per SM; a few CTAs
         ("v2rdm", 7, 4, 3, "DQG+D3"),     # long rows, group flags, odd size
         ("v2rdm", 9, 5, 4, "DQG"),        # two per SM
         ("v2rdm", 6, 3, 3, "DQGT2"),      # three per SM, both passes' tables in shared memory
         ("v2rdm", 18, 9, 9, "DQG"),       # three per SM, one region
         ("v2rdm", 10, 5, 5, "DQGT2")]     # three per SM, streamed tables


@pytest.mark.parametrize("kind,n,na,nb,pos", CASES)
def test_cg_solves_its_system(cuda_device, kind, n, na, nb, pos):
    import torch
    p = (hb.DOCIProblem if kind == "doci" else hb.V2RDMProblem)(n, na, nb, pos)
    rng = np.random.default_rng(n)
    c = torch.from_numpy(rng.standard_normal(p.n_primal)).to(cuda_device)
    b = torch.from_numpy(p.b()).to(cuda_device)
    x0 = torch.from_numpy(p.guess("RANDOM")).to(cuda_device)
    rhs = p.Au(c) + 0.1 * (b - p.Au(x0))   # the first iteration: mu = 0.1, z = 0
    out = []
    for _ in range(2):
        x = x0.clone()
        its = []
        p.solve_device(x, b, c, hb.Options({"MAXITER": 1, "CG_CONVERGENCE": 1e-9, "R_CONVERGENCE": 1e-12,
                                            "E_CONVERGENCE": 1e-12}),
                       monitor=lambda pl, oi, ii, *a: its.append(ii))
        y = torch.from_numpy(p.get_y()).to(cuda_device)
        res = float(torch.linalg.vector_norm(rhs - p.Au(p.ATu(y))))
        # the recurrence stops below 1e-9; each of its (at most a few hundred)
        # updates rounds r by at most a few eps |rhs|
        assert 0 < its[0] < 1000
        assert res <= 1e-9 + 1e-12 * float(torch.linalg.vector_norm(rhs)), (res, its)
        out.append(y)
    assert torch.equal(out[0], out[1])   # the sums' order is fixed
    p.close()
