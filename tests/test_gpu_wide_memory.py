"""Wide tensor-core plans when device memory is short: a scratch budget that
cuts their stages gives the same derivative (tolerance of the other tensor-core
tests, 1e-10 per contraction and projected derivative; the budget regroups the
chains, whose sums are then added in another order), and an allocation that
fails once makes qt_prepare plan them on the FP32 pipe, bit for bit the plan
of bounds 65."""
import os
import uuid

import numpy as np
import pytest

from helpers import deriv_errors
from qutree_gb300 import qtgpu
from qutree_gb300.model import balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu
TC = qtgpu.QT_PLAN_COMPRESSED | qtgpu.QT_PREC_DF64_TC


@pytest.fixture
def problem():
    tree = balanced_tree(4, 72, 72)
    sop = coupled_oscillators(tree, n_pairs=3, coupling=0.2, quartic=0.1, rng=np.random.default_rng(6), omega=1.0)
    yield tree, sop, random_wavefunction(tree, 6).flat()
    os.environ.pop("QT_FAULT_INJECT", None)
    os.environ.pop("QT_SCRATCH_MIB", None)


def derivative(problem, **kw):
    tree, sop, flat = problem
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=TC, **kw)
    try:
        return qtgpu.Derivative(h, flat), h.matrices(qtgpu.QT_MAT_RHO), len(h.stages())
    finally:
        h.close()


def test_cut_stages(problem):
    want, rho, whole = derivative(problem)
    os.environ["QT_SCRATCH_MIB"] = "32"
    got, _, cut = derivative(problem)
    assert cut > whole
    err, noise = deriv_errors(problem[0], got, want, rho)
    assert err <= 1e-10 and noise <= 1e-10


@pytest.mark.parametrize("nth", [1, 8])
def test_failed_allocation_falls_back(problem, nth):
    want, _, _ = derivative(problem, tc_thresholds=(65, 65, 65))
    assert not np.array_equal(derivative(problem)[0], want)
    os.environ["QT_FAULT_INJECT"] = f"alloc:{nth}#{uuid.uuid4().hex}"
    got, _, _ = derivative(problem)
    assert np.array_equal(got, want)
