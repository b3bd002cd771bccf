"""Sweeps of the tensor-core double-float plan on trees whose bonds exceed 64
(column blocks: one column short of a block, 65, 72, 112; leaves below 32),
against the oracle, at the tolerance of the other tensor-core tests (1e-10 per
contraction and projected derivative)."""
import numpy as np
import pytest

import oracle as O
from helpers import deriv_errors
from qutree_gb300 import qtgpu
from qutree_gb300.model import balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf,low,high", [(70, 65, 65), (24, 24, 72), (66, 66, 96), (112, 33, 112)])
def test_wide_bonds_sweep(leaf, low, high):
    tree = balanced_tree(4, leaf, low, bonds=lambda h, p: low if h == 0 else high)
    sop = coupled_oscillators(tree, n_pairs=3, coupling=0.2, quartic=0.1, rng=np.random.default_rng(6), omega=1.0)
    flat = random_wavefunction(tree, 6).flat()
    O.attach_openblas(fast=True)
    ref = O.derivative(tree, sop, flat, backend=O.BLAS, fast=True, want_mats=True)
    for grad in (0, qtgpu.QT_PLAN_GRADIENT):
        h = qtgpu.HamiltonianRepresentation(sop, tree,
                                            flavour=qtgpu.QT_PLAN_COMPRESSED | qtgpu.QT_PREC_DF64_TC | grad)
        try:
            d = qtgpu.Derivative(h, flat)
            e = h.energy()
            d2 = qtgpu.Derivative(h, flat)
            h.build()
            h.layer_derivatives()
            d3 = h.dpsi()
        finally:
            h.close()
        assert np.array_equal(d, d2)
        assert abs(e - ref.energy) <= 1e-10 * max(1.0, abs(ref.energy))
        for x in (d, d3):
            err, noise = deriv_errors(tree, x, ref.dpsi, ref.rho)
            assert err <= 1e-10 and noise <= 1e-10
