"""Device memory of tensor-core contractions beyond 64 columns, on the CPU: the
operand images and partial tiles of a stage stay within an eighth of the
scratch budget (or one task's, where that is more); stages that would need
more are cut, every task staying in exactly one stage, in order."""
import numpy as np
import pytest

from plan_emulator import ST_ACC, ST_HP, ST_MP, PlanView
from qutree_gb300.model import balanced_tree, coupled_oscillators

TENSOR = 0x8000


def tasks_of(T):
    out = {k: [] for k in (ST_MP, ST_HP, ST_ACC)}
    for kind, t0, nt, _, _ in T[0]:
        if kind in out:
            out[int(kind)] += range(int(t0), int(t0) + int(nt))
    return out


@pytest.mark.parametrize("bond", [72, 96, 112])
@pytest.mark.parametrize("log2_budget", [28, 24])
def test_wide_stages_stay_within_their_share(bond, log2_budget):
    tree = balanced_tree(32, bond, bond)
    sop = coupled_oscillators(tree, n_pairs=128, coupling=0.05, quartic=0.05, rng=np.random.default_rng(11))
    pv = PlanView(tree, sop, flavour=2 | TENSOR, prec=1, budget=1 << log2_budget)
    whole = PlanView(tree, sop, flavour=2 | TENSOR, prec=1, budget=1 << 34)  # a share that nothing exceeds
    T = pv.tables
    share = 16 * (1 << log2_budget) // 8
    chunks = -(-bond * bond // 64)  # of an inner hole product, the largest task: at most this many,
    one = chunks * (16 * bond * bond + 3 * (8 * 7 * 3 * 48 * 32 + 256 + 128))  # three column blocks of 48
    for si, (kind, t0, nt, _, _) in enumerate(T[0]):
        if kind != ST_HP:
            continue
        hti0, nhti, _, nhtu = (int(x) for x in T[55][si])
        groups = [T[52][int(i[0])] for i in T[53][hti0:hti0 + nhti]]
        tc = {int(m) for g in groups for m in g[8:8 + int(g[5])]}
        partial = sum(16 * int(T[44][t][0]) * int(T[2][t][7]) ** 2 for t in tc if int(T[44][t][0]) > 1)
        images = max((int(g[7]) for g in groups), default=0)  # the last image's offset
        assert partial + images <= max(share, one)
    assert int(T[56][0]) <= max(share, one)
    a, b = tasks_of(T), tasks_of(whole.tables)
    for k in a:
        assert a[k] == sorted(set(a[k]))
    if log2_budget == 28:  # the chains' own scratch groups are those of the large budget
        assert a == b
    else:
        assert len(T[0]) > len(whole.tables[0])
