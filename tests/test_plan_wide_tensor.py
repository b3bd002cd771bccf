"""Planner side of the tensor-core contractions beyond 64 output columns, on
the CPU (double-float plan, tree with bonds 65..112): every wide mode
product, hole product and accumulation is cut into column blocks of at most 64
columns (multiples of 8, the last one shorter), each covering its rows or
chunks exactly once; operand images are disjoint inside B_OZ; workspace
slots are given once per task; wide leaf products with fewer than 128 rows,
and wide accumulations outside the compressed plan's sweep (they cancel), keep
classic tiles."""
import numpy as np
import pytest

from plan_emulator import ST_ACC, ST_HP, ST_MP, PlanView
from qutree_gb300.model import balanced_tree, coupled_oscillators

TENSOR = 0x8000
BLOCK_SHIFT, TASK_SHIFT = 26, 28


def n_blocks(n):
    return 1 if n <= 64 else -(-n // 48)


def width(n):
    return (-(-n // n_blocks(n)) + 7) // 8 * 8


def blocks(n):
    out = [(c, min(width(n), n - c)) for c in range(0, n_blocks(n) * width(n), width(n))]
    assert all(w > 0 for _, w in out) and sum(w for _, w in out) == n
    return out


def image_bytes(w, steps):
    return steps * 7 * 3 * w * 32 + 256


def steps(k):
    return 4 if k <= 64 else -(-k // 16)


def problem(bond):
    tree = balanced_tree(4, 70, bond, bonds=lambda h, p: min(70, bond) if h == 0 else bond)
    return tree, coupled_oscillators(tree, n_pairs=None, coupling=0.2, rng=np.random.default_rng(8), omega=1.0)


@pytest.mark.parametrize("bond", [65, 72, 96, 112])
@pytest.mark.parametrize("plan", [1, 2])
def test_wide_contractions_cover_their_outputs(bond, plan):
    tree, sop = problem(bond)
    pv = PlanView(tree, sop, flavour=plan | TENSOR, prec=1)
    T, main_end = pv.tables, pv.main_end
    mp, hp, acc, hpx = T[1], T[2], T[3], T[44]
    oz_bytes = int(T[56][0])
    wide = {ST_MP: 0, ST_HP: 0, ST_ACC: 0}
    for si, (kind, t0, nt, _, _) in enumerate(T[0]):
        spans = []
        if kind == ST_MP:
            oz0, noz, ozt0, nozt = (int(x) for x in T[41][si])
            rows = {}
            for t, y in T[40][oz0:oz0 + noz]:
                rows.setdefault(int(t), []).append((int(y) >> BLOCK_SHIFT, int(y) & ((1 << BLOCK_SHIFT) - 1)))
            imgs = {}
            for v, off in T[42][ozt0:ozt0 + nozt]:
                t, cb = int(v) & ((1 << TASK_SHIFT) - 1), int(v) >> TASK_SHIFT
                imgs.setdefault(t, []).append(cb)
                size = image_bytes(width(int(mp[t][8])), steps(int(mp[t][7])))
                spans.append((int(off) + cb * size, int(off) + (cb + 1) * size))
            assert set(rows) == set(imgs)
            for t, r in rows.items():
                nr, ncb = -(-int(mp[t][6]) * int(mp[t][9]) // 128), len(blocks(int(mp[t][8])))
                assert sorted(r) == [(c, i) for c in range(ncb) for i in range(nr)]
                assert sorted(imgs[t]) == list(range(ncb))
                wide[kind] += int(mp[t][7]) > 64
            for t in range(t0, t0 + nt):
                a, b, n = int(mp[t][7]), int(mp[t][8]), int(mp[t][6]) * int(mp[t][9])
                want = not mp[t][10] and min(a, b) >= 32 and (max(a, b) <= 64 or (max(a, b) <= 112 and n >= 128))
                assert (t in rows) == want
        elif kind == ST_HP:
            hti0, nhti, htu0, nhtu = (int(x) for x in T[55][si])
            groups = sorted({int(i[0]) for i in T[53][hti0:hti0 + nhti]})
            per_task = {}
            for g in groups:
                row = [int(x) for x in T[52][g]]
                chunks = sorted(int(i[2]) for i in T[53][hti0:hti0 + nhti] if int(i[0]) == g)
                assert chunks == list(range(row[6]))
                for m in row[8:8 + row[5]]:
                    per_task.setdefault(m, []).append(row)
            for t in range(t0, t0 + nt):
                a, k = int(hp[t][7]), int(hp[t][6]) * int(hp[t][8])
                assert len(per_task.get(t, [])) == (len(blocks(a)) if 32 <= a <= 112 and k >= 128 else 0)
                wide[kind] += a > 64 and t in per_task
            for g, c in T[54][htu0:htu0 + nhtu]:
                row = [int(x) for x in T[52][int(g)]]
                w = width(row[3])
                size = image_bytes(w, 8 if w > 32 else 4)
                spans.append((row[7] + int(c) * size, row[7] + (int(c) + 1) * size))
            ws = sorted((int(hpx[t][2]), int(hpx[t][2]) + int(hpx[t][0]) * int(hp[t][7]) ** 2)
                        for t in range(t0, t0 + nt) if int(hpx[t][0]) > 1)
            assert all(e <= s for (_, e), (s, _) in zip(ws, ws[1:])) and all(e <= int(T[48][0]) for _, e in ws)
        elif kind == ST_ACC:
            ati0, nati, atu0, natu, nunits = (int(x) for x in T[59][si])
            got, units = {}, 0
            for t, b, before, cb in T[57][ati0:ati0 + nati]:
                assert int(before) == units
                units += int(acc[t][7])
                got.setdefault(int(t), []).append((int(b), int(cb)))
            assert units == nunits
            seen = {}
            for t, s in T[58][atu0:atu0 + natu]:
                seen.setdefault(int(t), []).append(int(s))
                d = int(acc[t][5])
                size = image_bytes(width(d), steps(d))
                spans.append((int(T[60][t]) + int(s) * size, int(T[60][t]) + (int(s) + 1) * size))
            assert set(got) == set(seen)
            for t, g in got.items():
                ncb = len(blocks(int(acc[t][5])))
                assert sorted(g) == [(b, c) for b in range(-(-int(acc[t][4]) // 128)) for c in range(ncb)]
                assert sorted(seen[t]) == list(range(int(acc[t][7]) * ncb))
                wide[kind] += int(acc[t][5]) > 64
                assert int(acc[t][5]) <= 64 or (plan == 2 and si < main_end)
            for t in range(t0, t0 + nt):
                if 64 < int(acc[t][5]) <= 112 and int(acc[t][4]) >= 64 and int(acc[t][7]) and plan == 2 and si < main_end:
                    assert t in got
        spans.sort()
        assert all(e <= s for (_, e), (s, _) in zip(spans, spans[1:]))
        assert all(0 <= s and e <= oz_bytes for s, e in spans)
    assert wide[ST_MP] and wide[ST_HP] and bool(wide[ST_ACC]) == (plan == 2)
