"""Order of a stage's blocks, on the CPU: small matrix products, accumulations
and mode products with the longest sums come first in their stage's tiles (a
block starts when an SM is free, in table order)."""
import numpy as np
import pytest

from plan_emulator import ST_ACC, ST_MM, ST_MP, PlanView
from qutree_gb300.model import balanced_tree, coupled_oscillators


@pytest.mark.parametrize("flavour", [0, 1, 2])
def test_longest_sums_first(flavour):
    tree = balanced_tree(7, 9, 4, bonds=lambda h, p: 4 + h)
    sop = coupled_oscillators(tree, n_pairs=None, coupling=0.2, rng=np.random.default_rng(2), omega=1.0)
    T = PlanView(tree, sop, flavour=flavour, prec=1).tables
    cost = {ST_MM: lambda t: int(T[22][t][4]) * int(T[22][t][2]), ST_ACC: lambda t: int(T[3][t][7]) * int(T[3][t][5]),
            ST_MP: lambda t: 1 if T[1][t][10] else int(T[1][t][7])}
    tiles = {ST_MM: T[50], ST_ACC: T[49], ST_MP: T[43]}
    seen = set()
    for kind, _, _, tile0, ntile in T[0]:
        if kind in cost:
            c = [cost[kind](int(r[0])) for r in tiles[kind][tile0:tile0 + ntile]]
            assert c == sorted(c, reverse=True)
            seen.add(int(kind))
    assert {ST_ACC, ST_MP} <= seen
