"""SCF on a converged state: every Lanczos space ends after its first vector,
and the driver must not run the products of H that a larger space would need.
Bound: with one product per solve as the unit (n_krylov = 1), a solve that
looks one product ahead needs at most twice the launches, whatever n_krylov."""
import numpy as np
import pytest

from qutree_gb300 import qtgpu
from qutree_gb300.model import balanced_tree, coupled_oscillators, random_wavefunction

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [qtgpu.QT_PREC_F64, qtgpu.QT_PREC_DF64])
@pytest.mark.parametrize("leaf,bond", [(6, 3), (44, 42)])  # one product ahead of the end, and none
def test_converged_state_runs_few_products(prec, leaf, bond):
    tree = balanced_tree(4, leaf, bond)
    sop = coupled_oscillators(tree, n_pairs=None, coupling=0.0, rng=np.random.default_rng(1), omega=1.0)
    h = qtgpu.HamiltonianRepresentation(sop, tree, flavour=qtgpu.QT_PLAN_COMPRESSED | qtgpu.QT_PLAN_SCF | prec)
    try:
        h.upload(random_wavefunction(tree, 1).flat())
        h.scf(12, 20)
        counts = []
        for n_krylov in (1, 30):
            c0 = h.ctx.launch_count()
            ritz = h.scf(1, n_krylov)
            counts.append(h.ctx.launch_count() - c0)
        assert abs(ritz - ritz[-1]).max() <= 1e-9 * abs(ritz[-1])
        assert counts[1] <= 2 * counts[0]
    finally:
        h.close()
