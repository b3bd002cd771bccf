"""The tensor-core kernels at reductions shorter than the three warps that
search the rows' exponents (one, two, four and seven elements; tiles of few
rows; node tensors with the reduction contiguous and strided), against the
oracle, at the tolerance of the other tensor-core tests (1e-10 per contraction
and projected derivative)."""
import numpy as np
import pytest

import oracle as O
from helpers import deriv_errors
from qutree_gb300 import qtgpu
from qutree_gb300.model import balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,low,high", [(4, 2, 1), (4, 2, 2), (7, 4, 7), (34, 5, 2)])
def test_short_reductions_on_the_tensor_cores(leaf, low, high):
    tree = balanced_tree(8, leaf, low, bonds=lambda h, p: low if h == 0 else high)
    sop = coupled_oscillators(tree, n_pairs=5, coupling=0.2, quartic=0.1, rng=np.random.default_rng(8), omega=1.0)
    flat = random_wavefunction(tree, 8).flat()
    O.attach_openblas(fast=True)
    ref = O.derivative(tree, sop, flat, backend=O.BLAS, fast=True, want_mats=True)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED | qtgpu.QT_PREC_DF64_TC,
                                        tc_thresholds=(1, 1, 1))
    try:
        d = qtgpu.Derivative(h, flat)
        e = h.energy()
    finally:
        h.close()
    assert abs(e - ref.energy) <= 1e-10 * max(1.0, abs(ref.energy))
    err, noise = deriv_errors(tree, d, ref.dpsi, ref.rho)
    assert err <= 1e-10 and noise <= 1e-10
