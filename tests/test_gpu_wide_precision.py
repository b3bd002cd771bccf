"""Precision of the tensor-core contractions beyond 64 columns: against the
complex128 plan they may be no further off than the double-float multiply-adds
of the same plan with every kind on the FP32 pipe (bounds 65).  Density
matrices (hole products alone) are compared directly, energies and gradients
with a quarter on top, since further roundings act on both.  Bonds of two
blocks of 40 columns, of two of 48 (five level accumulators) and of three; root
mean square over three wavefunctions."""
import numpy as np
import pytest

from qutree_gb300 import qtgpu
from qutree_gb300.model import balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu


def outputs(tree, sop, states, flavour, bounds=None):
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=flavour | qtgpu.QT_PLAN_GRADIENT, tc_thresholds=bounds)
    try:
        out = []
        for flat in states:
            qtgpu.Derivative(h, flat)
            out.append((h.matrices(qtgpu.QT_MAT_RHO), np.array([h.energy()]), h.gradient()))
        return out
    finally:
        h.close()


def errors(got, ref):
    e = [[np.linalg.norm(a - b) / np.linalg.norm(b) for a, b in zip(x, y)] for x, y in zip(got, ref)]
    return np.sqrt(np.mean(np.square(e), axis=0))


@pytest.mark.parametrize("bond", [72, 96, 112])
@pytest.mark.parametrize("plan", [qtgpu.QT_PLAN_GROUPED, qtgpu.QT_PLAN_COMPRESSED])
def test_wide_tensor_products_are_no_less_precise(bond, plan):
    tree = balanced_tree(8, bond, bond)
    sop = coupled_oscillators(tree, n_pairs=10, coupling=0.2, quartic=0.1, rng=np.random.default_rng(6), omega=1.0)
    states = [random_wavefunction(tree, 100 + s).flat() for s in range(3)]
    ref = outputs(tree, sop, states, qtgpu.QT_PLAN_COMPRESSED | qtgpu.QT_PREC_F64)
    tc = errors(outputs(tree, sop, states, plan | qtgpu.QT_PREC_DF64_TC), ref)
    fp32 = errors(outputs(tree, sop, states, plan | qtgpu.QT_PREC_DF64_TC, (65, 65, 65)), ref)
    assert tc[0] <= fp32[0]
    assert tc[1] <= 1.25 * fp32[1]
    assert tc[2] <= 1.25 * fp32[2]
