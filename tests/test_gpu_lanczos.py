"""The Lanczos recursion of the SCF driver on the device at the edges of its
slices and clusters: node tensors smaller than the Krylov space (invariant
spaces that end early), of 8000 and 9261 elements (either side of one slice),
of several slices, one and many Krylov vectors; Ritz values and the final
energy against the oracle's scf(), at the tolerances of the other SCF tests
(1e-11 in complex128, 1e-10 in double-float)."""
import numpy as np
import pytest

from qutree_gb300 import qtgpu
from qutree_gb300.model import balanced_tree, coupled_oscillators, random_wavefunction
from test_gpu_scf import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(qtgpu.QT_PREC_F64, 1e-11), (qtgpu.QT_PREC_DF64, 1e-10)])
@pytest.mark.parametrize("leaf,bond,n_krylov", [(3, 2, 8), (5, 4, 1), (21, 20, 2), (22, 21, 3), (30, 29, 2)])
def test_lanczos_edges(leaf, bond, n_krylov, prec, tol):
    tree = balanced_tree(4, leaf, bond)
    sop = coupled_oscillators(tree, n_pairs=None, coupling=0.2, quartic=0.1, rng=np.random.default_rng(2), omega=1.0)
    _check(tree, sop, random_wavefunction(tree, 2), tol=tol, prec=prec, n_iter=1, n_krylov=n_krylov)


@pytest.mark.parametrize("prec,tol", [(qtgpu.QT_PREC_F64, 1e-11), (qtgpu.QT_PREC_DF64, 1e-10)])
def test_lanczos_more_slices_than_ctas(prec, tol):
    """Inner nodes of 74088 elements: ten slices on a cluster of eight CTAs, two
    of which own two."""
    tree = balanced_tree(4, 43, 42)
    sop = coupled_oscillators(tree, n_pairs=None, coupling=0.2, quartic=0.1, rng=np.random.default_rng(2), omega=1.0)
    _check(tree, sop, random_wavefunction(tree, 2), tol=tol, prec=prec, n_iter=1, n_krylov=2)
