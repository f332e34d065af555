"""v2RDM-DOCI with orbital optimisation on the device against the recorded energy
of the CPU chain under hilbert's schedule, for machines without hilbert's
compiled code."""
import pytest

import hilbert_b200 as hb
import hilbert_b200.orbital as ho
from test_gpu_doci import ORBITAL_OPTS

pytestmark = pytest.mark.gpu


def test_doci_helper_reaches_the_recorded_schedule_energy(cuda_device):
    n, npair = 4, 2
    h_mo, B_mo, *_ = ho.casscf_df_problem(nbf=n, naux=10, ncore=0, nact=n)
    helper = hb.v2RDM_DOCIHelper(npair, npair, n, h_mo, None, ORBITAL_OPTS, B=B_mo)
    e = helper.compute_energy(macro_iterations=400)
    assert helper.stats["converged"] and helper.stats["orbitals_converged"]
    # test_doci.py's value, and the bound that the comparison with a fresh run has
    assert abs(e - (-33.57490517)) <= 5e-5
    assert helper.variables["v2RDM-DOCI TOTAL ENERGY"] == e
