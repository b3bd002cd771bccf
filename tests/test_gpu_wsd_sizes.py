"""The joint diagonalisation over the numbers of matrices at which its tree of
sums changes form: one matrix per lane (up to 8), two and four per lane (up to
16 and 32), and 32 lanes with two and four matrices each (beyond); bit for bit
against the restatement on the device's own inputs."""
import pytest

import test_gpu_cdvr as cdvr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_modes,p,bond", [(3, 5, 3), (9, 4, 3), (18, 4, 2), (34, 4, 2), (66, 4, 2)])
def test_wsd_bit_exact_for_any_number_of_matrices(n_modes, p, bond):
    cdvr.test_wsd_kernel_is_bit_exact(n_modes, p, bond)
