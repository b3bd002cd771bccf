"""The tensor-core contractions where their epilogue leaves its common path, at
bonds whose products, hole products and accumulations all take them: rows of
zeros, rows whose scale falls below the normal numbers beside rows of order
one, and operands that are not finite.  Derivatives against the oracle at the
tolerance of the other tensor-core tests (1e-10); a NaN or an infinity in any
node tensor reaches the energy."""
import numpy as np
import pytest

import oracle as O
from helpers import deriv_errors
from qutree_gb300 import qtgpu
from qutree_gb300.model import TensorTree, balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu
TC = qtgpu.QT_PLAN_COMPRESSED | qtgpu.QT_PREC_DF64_TC


def problem(bond):
    tree = balanced_tree(4, bond + 4, bond)
    sop = coupled_oscillators(tree, n_pairs=3, coupling=0.2, quartic=0.1, rng=np.random.default_rng(9), omega=1.0)
    return tree, sop, random_wavefunction(tree, 9)


@pytest.mark.parametrize("bond", [36, 72, 96])
@pytest.mark.parametrize("shift", [-60, -122])
@pytest.mark.parametrize("axis", [0, 1])
def test_rows_of_zeros_and_of_tiny_scale(bond, shift, axis):
    tree, sop, psi = problem(bond)
    tensors = []
    for n, t in zip(tree.nodes, psi.tensors):
        t = np.array(t, order="F")
        if not n.is_bottom and not n.is_top:
            rows = np.moveaxis(t, axis, 0)  # a view
            rows[3] = 0.0
            rows[5:9] *= 2.0 ** shift
            rows[20, 2:6] = 0.0
        tensors.append(t)
    flat = TensorTree(tree, tensors).flat()
    O.attach_openblas(fast=True)
    ref = O.derivative(tree, sop, flat, backend=O.BLAS, fast=True, want_mats=True)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=TC)
    try:
        d = qtgpu.Derivative(h, flat)
        e = h.energy()
    finally:
        h.close()
    assert abs(e - ref.energy) <= 1e-10 * abs(ref.energy)
    err, noise = deriv_errors(tree, d, ref.dpsi, ref.rho)
    assert err <= 1e-10 and noise <= 1e-10


@pytest.mark.parametrize("bond", [36, 72])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("node", ["leaf", "inner", "top"])
def test_non_finite_operands_reach_the_energy(bond, value, node):
    import torch
    tree, sop, psi = problem(bond)
    flat = psi.flat().copy()
    pick = {"leaf": lambda n: n.is_bottom, "inner": lambda n: not n.is_bottom and not n.is_top,
            "top": lambda n: n.is_top}[node]
    a = next(n.address for n in tree.nodes if pick(n))
    flat[int(tree.offsets()[a]) + 7] = value
    dev = torch.from_numpy(flat.view(np.float64)).cuda()
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=TC)
    try:
        h.upload_device(dev.data_ptr())
        h.derivative()
        with pytest.raises(qtgpu.QtError, match="QT_ERR_NUMERIC"):
            h.energy()
        h.upload(psi.flat())  # and leaves nothing behind
        h.derivative()
        assert np.isfinite(h.energy())
    finally:
        h.close()
