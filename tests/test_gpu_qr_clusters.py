"""qt_qr_orthogonal at the edges of its cluster split: leaves and nodes of one
row block per CTA up to many CTAs, blocks in shared memory and (wide bonds)
in place, more columns than rows, bond 1, siblings at different heights.
Every non-top node is compared with a Householder QR in numpy with the
device's own reflector convention, its children's R multiplied in; bound:
Householder QR of an m x n matrix is backward stable to about
8 (m + n) 2^-53 per column, and the comparison of Q multiplies by the
condition number of the (random, well-conditioned or square) node."""
import numpy as np
import pytest

from qutree_gb300 import qtgpu
from qutree_gb300.model import (MLO, OP_DIAG, SOP, OperatorTable, TensorTree, Tree, _Build, balanced_tree,
                                mode_product)

pytestmark = pytest.mark.gpu


def house_qr(a):
    """Thin Q and R; reflectors map a column to -e^{i arg x0} |x| e_1."""
    m, n = a.shape
    w, vs = a.copy(), []
    for j in range(min(m, n)):
        v = w[j:, j].copy()
        v[0] += v[0] / abs(v[0]) * np.linalg.norm(v)
        v /= np.linalg.norm(v)
        w[j:] -= 2 * np.outer(v, v.conj() @ w[j:])
        vs.append(v)
    q = np.eye(m, n, dtype=complex)
    for j in reversed(range(len(vs))):
        q[j:] -= 2 * np.outer(vs[j], vs[j].conj() @ q[j:])
    return q, np.triu(w[:n]) if m >= n else np.vstack([np.triu(w), np.zeros((n - m, n))])


def reference(tree, tensors):
    out, cond = list(tensors), 1.0
    for n in tree.nodes:
        if n.is_top:
            continue
        a = out[n.address].reshape((-1, n.d_up), order="F")
        q, r = house_qr(a)
        cond = max(cond, np.linalg.cond(a))
        out[n.address] = q.reshape(n.shape, order="F")
        out[n.parent] = mode_product(r, out[n.parent], n.child_idx)
    return out, cond


def ragged():
    leaf = lambda p, b: _Build([p, b], leaf=True)
    mid = _Build([5, 7, 9], [leaf(11, 5), leaf(9, 7)])
    return Tree(_Build([9, 4, 1, 1], [mid, leaf(6, 4), leaf(4, 1)]))


TREES = {
    "leaf_32": lambda: balanced_tree(4, 32, 32),
    "odd": lambda: balanced_tree(6, 13, 7),
    "ragged_heights": ragged,
    "one_column": lambda: balanced_tree(4, 5, 1),
    "clusters": lambda: balanced_tree(8, 20, 17),
    "wide_in_place": lambda: balanced_tree(4, 70, 70, bonds=lambda h, p: 70 if h == 0 else 96),
}


@pytest.mark.parametrize("name", sorted(TREES))
def test_qr_against_householder(name):
    tree = TREES[name]()
    rng = np.random.default_rng(5)
    ts = [np.asfortranarray((rng.standard_normal(n.shape) + 1j * rng.standard_normal(n.shape)) / np.sqrt(2 * n.size))
          for n in tree.nodes]
    want, cond = reference(tree, ts)
    ops = OperatorTable()
    sop = SOP(ops)
    sop.push_back(MLO([(0, ops.add("u", OP_DIAG, np.ones(tree.leaf_dim(0))))]), 1.0)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED)
    try:
        h.upload(TensorTree(tree, ts).flat())
        h.qr_orthogonal()
        got = TensorTree.from_flat(tree, h.psi()).tensors
    finally:
        h.close()
    rows = max(n.size // n.d_up + n.d_up for n in tree.nodes)
    for n in tree.nodes:
        scale = np.abs(want[n.address]).max()
        assert np.abs(got[n.address] - want[n.address]).max() <= 8 * rows * 2.0 ** -53 * cond * scale
        if not n.is_top:
            q = got[n.address].reshape((-1, n.d_up), order="F")
            if q.shape[0] >= q.shape[1]:
                assert np.abs(q.conj().T @ q - np.eye(n.d_up)).max() <= 8 * rows * 2.0 ** -53


def guarded_qr(a):
    """house_qr where a column may be zero below (no reflection)."""
    m, n = a.shape
    w, vs = a.copy(), []
    for j in range(min(m, n)):
        v = w[j:, j].copy()
        norm = np.linalg.norm(v)
        if norm > 0.0:
            v[0] += (v[0] / abs(v[0]) if abs(v[0]) > 0 else 1.0) * norm
            v /= np.linalg.norm(v)
        w[j:] -= 2 * np.outer(v, v.conj() @ w[j:])
        vs.append(v)
    q = np.eye(m, n, dtype=complex)
    for j in reversed(range(len(vs))):
        q[j:] -= 2 * np.outer(vs[j], vs[j].conj() @ q[j:])
    return q, np.triu(w[:n]) if m >= n else np.vstack([np.triu(w), np.zeros((n - m, n))])


def _leaf(p, b):
    return _Build([p, b], leaf=True)


RANK_TREES = {  # rows below columns, alone and beside a node that sets a cluster of 16 CTAs
    "wide_leaf": lambda: Tree(_Build([9, 5, 1], [_leaf(4, 9), _leaf(12, 5)])),
    "wide_leaf_in_a_cluster": lambda: Tree(_Build([9, 9, 1], [_leaf(4, 9), _leaf(1500, 9)])),
    "one_row": lambda: Tree(_Build([3, 9, 1], [_leaf(1, 3), _leaf(40, 9)])),
    "square": lambda: balanced_tree(4, 13, 13),
}


@pytest.mark.parametrize("zero", [None, 0, 2])
@pytest.mark.parametrize("name", sorted(RANK_TREES))
def test_qr_with_few_rows_and_with_a_zero_column(name, zero):
    """More columns than rows (steps = rows, zero rows of R below), and a column
    of zeros in the leaves (the first: no reflection at all; a later one: the
    rest of it below the rows already reduced, zero too)."""
    tree = RANK_TREES[name]()
    rng = np.random.default_rng(7)
    ts = [np.asfortranarray((rng.standard_normal(n.shape) + 1j * rng.standard_normal(n.shape)) / np.sqrt(2 * n.size))
          for n in tree.nodes]
    if zero is not None:
        for n in tree.nodes:
            if n.is_bottom and zero < n.d_up:
                ts[n.address][:, zero] = 0.0
    out, cond = list(ts), 1.0
    for n in tree.nodes:
        if n.is_top:
            continue
        a = out[n.address].reshape((-1, n.d_up), order="F")
        q, r = guarded_qr(a)
        s = np.linalg.svd(a, compute_uv=False)
        cond = max(cond, s[0] / s[s > 1e-12 * s[0]][-1])
        out[n.address] = q.reshape(n.shape, order="F")
        out[n.parent] = mode_product(r, out[n.parent], n.child_idx)
    ops = OperatorTable()
    sop = SOP(ops)  # enough chains for the scratch that the factorisation borrows
    for q in range(24):
        sop.push_back(MLO([(m, ops.add(("u", q, m), OP_DIAG, rng.standard_normal(tree.leaf_dim(m))))
                           for m in range(tree.n_leaves)]), 1.0)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED)
    try:
        h.upload(TensorTree(tree, ts).flat())
        h.qr_orthogonal()
        got = TensorTree.from_flat(tree, h.psi()).tensors
    finally:
        h.close()
    rows = max(n.size // n.d_up + n.d_up for n in tree.nodes)
    for n in tree.nodes:
        scale = np.abs(out[n.address]).max()
        assert np.abs(got[n.address] - out[n.address]).max() <= 8 * rows * 2.0 ** -53 * cond * scale
