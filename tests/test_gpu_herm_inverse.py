"""The sweep-operator inverse of Hermitian positive definite matrices at the
edges of its 16 x 16 thread grid and around the eigenvalue (40 eps) below
which the regularisation acts: density inverses against numpy's eigh, and the
projector's inverse of Phi^dagger Phi (non-orthonormal node tensors, odd
bonds) through a sweep against the oracle.  Bounds: an unpivoted symmetric
inversion of a positive definite matrix of order d and condition number c is
exact to 8 d c 2^-53 of the inverse's largest entry (d eliminations, forward
and backward); the sweep's tolerances are those of the other parity tests."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_err
from qutree_gb300 import qtgpu
from qutree_gb300.model import TensorTree, balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu


def hermitian(rng, w):
    d = len(w)
    q, _ = np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
    m = (q * w) @ q.conj().T
    return 0.5 * (m + m.conj().T)


@pytest.mark.parametrize("d", [1, 2, 15, 16, 17, 31, 33, 65, 112])
@pytest.mark.parametrize("low", [1e-3, 200.0, 41.0, 30.0, 3.0, 0.0, -1e-3])
def test_density_inverse(d, low):
    """Smallest eigenvalue 1e-3, or a multiple of eps on either side of the
    shortcut's bound, or zero, or slightly negative (rounding of a
    rank-deficient density)."""
    eps = 1e-8
    rng = np.random.default_rng(d)
    w = 10.0 ** rng.uniform(-3, 0, d)
    w[0] = low if low == 1e-3 else low * eps
    m = hermitian(rng, w)
    lam, u = np.linalg.eigh(m)
    want = (u / (lam + eps * np.exp(-lam / eps))) @ u.conj().T
    ctx = qtgpu.Context(0)
    try:
        a, b = ctx.to_device(m.ravel(order="F")), ctx.to_device(np.zeros(d * d, complex))
        ctx.rho_inverse_noalloc(b, a, 1, d, eps)
        got = ctx.from_device(b, (d * d,)).reshape((d, d), order="F")
        ctx.free(a)
        ctx.free(b)
    finally:
        ctx.close()
    # the regularised function changes by at most 1 / eps^2 per unit of the
    # eigenvalue, its largest value is about 1 / max(lam_min, eps)
    cond = max(1.0, lam[-1] / max(lam[0], eps))  # a condition number is at least one
    assert rel_err(got, want) <= 8 * d * cond * 2.0 ** -53 + 64 * 2.0 ** -53 * cond


@pytest.mark.parametrize("bond", [3, 15, 17, 33])
@pytest.mark.parametrize("prec,tol", [(qtgpu.QT_PREC_F64, 1e-12), (qtgpu.QT_PREC_DF64, 1e-11)])
def test_projector_of_non_orthonormal_nodes(bond, prec, tol):
    """The top node of dPsi does not see the projector; the others do."""
    tree = balanced_tree(4, 40, bond)
    sop = coupled_oscillators(tree, n_pairs=None, coupling=0.2, quartic=0.1, rng=np.random.default_rng(1), omega=1.0)
    psi = random_wavefunction(tree, 3)
    rng = np.random.default_rng(4)
    tensors = []
    for n, t in zip(tree.nodes, psi.tensors):
        d = n.d_up
        g = np.eye(d) + 0.2 / np.sqrt(d) * (rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))
        tensors.append(t if n.is_top else np.asfortranarray(np.tensordot(t, g, axes=([-1], [0]))))
    flat = TensorTree(tree, tensors).flat()
    ref = O.derivative(tree, sop, flat)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED | prec)
    try:
        got = qtgpu.Derivative(h, flat)
    finally:
        h.close()
    off, ro = tree.offsets(), 0
    num = den = 0.0
    for n in tree.nodes:  # weighted back by rho, as in the other sweep tests
        d = n.d_up
        r = ref.rho[ro:ro + d * d].reshape((d, d), order="F")
        ro += d * d
        a, b = (x[off[n.address]:off[n.address + 1]].reshape((-1, d), order="F") for x in (got, ref.dpsi))
        if not n.is_top:
            a, b = a @ r.T, b @ r.T
        num, den = max(num, np.abs(a - b).max()), max(den, np.abs(b).max())
    assert num <= 10 * tol * den


@pytest.mark.parametrize("d", [17, 64, 112])
@pytest.mark.parametrize("low,rest", [(110.0, 250.0), (60.0, 90.0), (90.0, 260.0)])
def test_density_inverse_between_the_certificates(d, low, rest):
    """All eigenvalues within a few hundred eps: the Frobenius norm of the
    inverse alone does not decide.  The spectrum lies above 100 eps (the
    factorisation certifies it), below (no factorisation is tried at d = 112),
    or has one eigenvalue below (it is tried and fails)."""
    eps = 1e-8
    rng = np.random.default_rng(d)
    w = eps * rng.uniform(0.5 * (low + rest), rest, d)
    w[0] = eps * low
    m = hermitian(rng, w)
    lam, u = np.linalg.eigh(m)
    want = (u / (lam + eps * np.exp(-lam / eps))) @ u.conj().T
    ctx = qtgpu.Context(0)
    try:
        a, b = ctx.to_device(m.ravel(order="F")), ctx.to_device(np.zeros(d * d, complex))
        ctx.rho_inverse_noalloc(b, a, 1, d, eps)
        got = ctx.from_device(b, (d * d,)).reshape((d, d), order="F")
        ctx.free(a)
        ctx.free(b)
    finally:
        ctx.close()
    cond = lam[-1] / lam[0]
    assert rel_err(got, want) <= 8 * d * cond * 2.0 ** -53 + 64 * 2.0 ** -53 * cond


@pytest.mark.parametrize("decades", [2, 3, 4])
@pytest.mark.parametrize("prec,unit", [(qtgpu.QT_PREC_F64, 2.0 ** -53), (qtgpu.QT_PREC_DF64, 2.0 ** -47)])
def test_projector_of_nearly_dependent_columns(decades, prec, unit):
    """Node tensors whose columns span `decades` orders of magnitude in all
    directions: cond(S) is the square.  The bound is that of the inverse
    alone, 8 d cond(S) units."""
    tree = balanced_tree(4, 40, 17)
    sop = coupled_oscillators(tree, n_pairs=None, coupling=0.2, quartic=0.1, rng=np.random.default_rng(1), omega=1.0)
    psi = random_wavefunction(tree, 3)
    rng = np.random.default_rng(4)
    tensors = []
    for n, t in zip(tree.nodes, psi.tensors):
        d = n.d_up
        a, b = (np.linalg.qr(rng.standard_normal((d, d)) + 1j * rng.standard_normal((d, d)))[0] for _ in range(2))
        g = (a * 10.0 ** (-decades * np.arange(d) / max(1, d - 1))) @ b
        tensors.append(t if n.is_top else np.asfortranarray(np.tensordot(t, g, axes=([-1], [0]))))
    flat = TensorTree(tree, tensors).flat()
    ref = O.derivative(tree, sop, flat)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED | prec)
    try:
        got = qtgpu.Derivative(h, flat)
    finally:
        h.close()
    off, ro = tree.offsets(), 0
    num = den = 0.0
    for n in tree.nodes:  # weighted back by rho, as in the other sweep tests
        d = n.d_up
        r = ref.rho[ro:ro + d * d].reshape((d, d), order="F")
        ro += d * d
        a, b = (x[off[n.address]:off[n.address + 1]].reshape((-1, d), order="F") for x in (got, ref.dpsi))
        if not n.is_top:
            a, b = a @ r.T, b @ r.T
        num, den = max(num, np.abs(a - b).max()), max(den, np.abs(b).max())
    assert num <= 8 * 17 * 10.0 ** (2 * decades) * unit * den
