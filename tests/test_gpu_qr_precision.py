"""Rounding of the cluster Householder QR: the thin Q of leaves against one in
extended precision, compared with a binary64 QR that applies one reflector
after the other (as the device did on one block per node).  The compact form
may be no further off, up to a tenth for the scatter of a mean over 32
leaves."""
import numpy as np
import pytest

from qutree_gb300 import qtgpu
from qutree_gb300.model import MLO, OP_DIAG, SOP, OperatorTable, TensorTree, balanced_tree

pytestmark = pytest.mark.gpu


def house_q(a, dtype):
    """Thin Q; reflectors map a column to -e^{i arg x0} |x| e_1."""
    m, n = a.shape
    w, vs = a.astype(dtype), []
    for j in range(n):
        v = w[j:, j].copy()
        below = (v[1:].real ** 2 + v[1:].imag ** 2).sum()
        a0 = v[0].real ** 2 + v[0].imag ** 2
        v[0] += v[0] / np.sqrt(a0) * np.sqrt(below + a0)
        tau = 2 / (below + v[0].real ** 2 + v[0].imag ** 2)
        w[j:, j + 1:] -= np.outer(v, tau * (v.conj() @ w[j:, j + 1:]))
        vs.append((v, tau))
    q = np.eye(m, n).astype(dtype)
    for j in reversed(range(n)):
        v, tau = vs[j]
        q[j:, j:] -= np.outer(v, tau * (v.conj() @ q[j:, j:]))
    return q


@pytest.mark.parametrize("p,bond", [(64, 16), (200, 12), (300, 17)])
def test_leaf_q_is_as_precise_as_reflectors_in_turn(p, bond):
    tree = balanced_tree(32, p, bond, bonds=lambda h, q: bond if h == 0 else 4)
    rng = np.random.default_rng(p)
    tensors = []
    for n in tree.nodes:
        t = rng.standard_normal(n.shape) + 1j * rng.standard_normal(n.shape)
        if n.is_bottom:  # near an isometry, as a propagated wavefunction is
            t = np.linalg.qr(t)[0] + 1e-3 / np.sqrt(n.size) * t
        tensors.append(np.asfortranarray(t / np.sqrt(n.size) if not n.is_bottom else t))
    ops = OperatorTable()
    sop = SOP(ops)
    sop.push_back(MLO([(0, ops.add("u", OP_DIAG, np.ones(p)))]), 1.0)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED)
    try:
        h.upload(TensorTree(tree, tensors).flat())
        h.qr_orthogonal()
        got = TensorTree.from_flat(tree, h.psi()).tensors
    finally:
        h.close()
    device, reflectors = [], []
    for n in tree.nodes:
        if n.is_bottom:
            want = house_q(tensors[n.address], np.clongdouble)
            device.append(np.sqrt(float((abs(got[n.address] - want) ** 2).sum())))
            reflectors.append(np.sqrt(float((abs(house_q(tensors[n.address], complex) - want) ** 2).sum())))
    assert np.mean(device) <= 1.1 * np.mean(reflectors)
