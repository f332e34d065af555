"""The forms of the conjugate-gradient kernel that large problems take
(test_cg_tables.py holds which): tables in turn in one region of shared memory,
at its smallest problem and at the (20e,20o) one, and streamed tables of two-body
conditions alone."""
import pytest

import test_gpu_cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,na,nb", [(19, 10, 9), (20, 10, 10), (22, 11, 11)])
def test_cg_solves_its_system(cuda_device, n, na, nb):
    test_gpu_cg.test_cg_solves_its_system(cuda_device, "v2rdm", n, na, nb, "DQG")
