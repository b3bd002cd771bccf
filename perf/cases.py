"""The work users have this framework do, as cases that can be timed and
checked: one pass each through the public entry points of
``qutree_gb300.qtgpu``.

  listed()            the cases, by what they stand for
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call (on the GPU)
  run(state)          one pass, its outputs whole
  work(case)          the bytes and flops a pass cannot do without
  exact(case, seed)   run's outputs in 64 bits, by plain torch

Wavefunctions are the seeded random states of ``qutree_gb300.model`` with the
top tensor replaced by one whose natural weights decay geometrically from 1 to
1e-3, the spread of a moderately correlated state (a Gaussian top tensor has
an accidental, much wider one).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from qutree_gb300 import model as M
from qutree_gb300 import qtgpu as Q

PRECISION = {"complex128": Q.QT_PREC_F64, "double-float": Q.QT_PREC_DF64,
             "double-float-tensor": Q.QT_PREC_DF64_TC}
REGULARISATION = 1e-10
CMF_DT = 0.01


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------
def listed():
    return [
        # one node's products through the device-pointer primitives, as the
        # matvec_ / rhomat_ binding issues them: a node of an 8-mode tree
        # (latency), and a node under the top of a 64-mode tree
        {"name": "products_small", "kind": "products", "d0": 7, "d1": 9, "up": 6},
        {"name": "products_large", "kind": "products", "d0": 64, "d1": 58, "up": 64},
        # the first call of a program moving from QuTree: all defaults
        # (reference call sequence, complex128), host arrays in and out
        {"name": "derivative_host_8_modes", "kind": "derivative_host", "modes": 8, "p": 16, "lo": 4, "hi": 4,
         "pairs": 28, "quartic": False},
        # sweeps with the wavefunction on the device, the integrator's inner call:
        # the 16-mode and 64-mode configurations, and the wide-bond one, whose
        # shapes leave the tensor cores' range
        {"name": "sweep_16_modes", "kind": "sweep", "modes": 16, "p": 32, "lo": 32, "hi": 32, "pairs": 120,
         "quartic": False, "precision": "double-float-tensor"},
        {"name": "sweep_64_modes", "kind": "sweep", "modes": 64, "p": 32, "lo": 32, "hi": 64, "pairs": 256,
         "quartic": True, "precision": "double-float-tensor"},
        {"name": "sweep_64_modes_wide", "kind": "sweep", "modes": 64, "p": 32, "lo": 48, "hi": 96, "pairs": 256,
         "quartic": True, "precision": "double-float-tensor"},
        # many small uneven trees advanced together
        {"name": "forest_64_trees", "kind": "forest", "trees": 64, "structure": 2,
         "precision": "double-float"},
        # sweep and energy gradient of every node, read back to the host
        {"name": "gradient_16_modes", "kind": "gradient", "modes": 16, "p": 32, "lo": 32, "hi": 32, "pairs": 120,
         "quartic": False, "precision": "double-float-tensor"},
        # one constant-mean-field step of a propagation, odd sizes
        {"name": "cmf_step_12_modes", "kind": "cmf", "modes": 12, "p": 21, "lo": 13, "hi": 19, "pairs": 40,
         "quartic": True, "precision": "double-float"},
        # one SCF iteration (ground-state search)
        {"name": "scf_8_modes", "kind": "scf", "modes": 8, "p": 16, "lo": 6, "hi": 8, "pairs": 28,
         "quartic": False, "precision": "double-float"},
        # a sweep with a potential that is no sum of products
        {"name": "cdvr_8_modes", "kind": "cdvr", "modes": 8, "p": 12, "lo": 7, "hi": 7},
        # re-orthonormalisation of a propagated wavefunction
        {"name": "qr_16_modes", "kind": "qr", "modes": 16, "p": 32, "lo": 32, "hi": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_tree(rng, modes, p, bonds):
    lo = _log_int(rng, *bonds)
    return {"modes": _log_int(rng, *modes), "p": _log_int(rng, *p), "lo": lo,
            "hi": min(bonds[1], int(round(lo * rng.uniform(1.0, 2.0)))),
            "quartic": rng.random() < 0.5}


def draw(rng):
    kind = rng.choice(["products", "products", "derivative_host", "sweep", "sweep", "sweep", "forest",
                       "gradient", "cmf", "scf", "cdvr", "qr"])
    if kind == "products":
        return {"kind": kind, "d0": _log_int(rng, 4, 72), "d1": _log_int(rng, 4, 72), "up": _log_int(rng, 4, 72)}
    if kind == "forest":
        return {"kind": kind, "trees": _log_int(rng, 4, 96), "structure": rng.randrange(1 << 20),
                "precision": rng.choice(["double-float", "double-float-tensor"])}
    if kind in ("scf", "cdvr"):
        c = {"kind": kind, **_draw_tree(rng, (4, 10), (8, 16), (4, 8))}
    elif kind == "derivative_host":
        c = {"kind": kind, **_draw_tree(rng, (4, 12), (6, 20), (3, 10))}
    elif kind == "cmf":
        c = {"kind": kind, **_draw_tree(rng, (6, 20), (8, 36), (6, 28))}
    elif kind in ("gradient", "qr"):
        c = {"kind": kind, **_draw_tree(rng, (6, 24), (10, 40), (8, 40))}
    else:
        c = {"kind": kind, **_draw_tree(rng, (6, 64), (10, 40), (8, 64))}
    f = c["modes"]
    if kind in ("cdvr", "qr"):
        c.pop("quartic")
    else:
        c["pairs"] = min(f * (f - 1) // 2, _log_int(rng, f, 4 * f))
    if kind in ("sweep", "gradient", "cmf"):
        c["precision"] = rng.choice(["double-float", "double-float-tensor", "double-float-tensor"])
    elif kind == "scf":
        c["precision"] = rng.choice(["complex128", "double-float"])
    if kind == "sweep" and f <= 16 and rng.random() < 0.3:
        c["precision"] = "complex128"
    return c


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _tree(case):
    heights = max(2, math.ceil(math.log2(max(2, case["modes"]))))
    return M.balance_bonds(M.balanced_tree(case["modes"], case["p"], case["hi"],
                                           bonds=M.linear_bonds(case["lo"], case["hi"], heights)))


def _sop(case, tree):
    return M.coupled_oscillators(tree, n_pairs=case["pairs"], coupling=0.05,
                                 quartic=0.05 if case["quartic"] else 0.0, rng=np.random.default_rng(11))


def _top_tensor(shape, rng):
    """Unit-norm top tensor with natural weights from 1 down to 1e-3 along its
    first index (the weights of a binary top; more children mix them)."""
    a, b = shape[0], int(np.prod(shape[1:]))
    r = min(a, b)

    def iso(n):
        return np.linalg.qr(rng.standard_normal((n, r)) + 1j * rng.standard_normal((n, r)))[0]

    t = (iso(a) * 10.0 ** (-1.5 * np.arange(r) / max(1, r - 1))) @ iso(b).T
    return (t / np.linalg.norm(t)).reshape(shape, order="F")


def _psi(tree, seed):
    psi = M.random_wavefunction(tree, seed)
    rng = np.random.default_rng(seed + 1)
    for n in tree.nodes:
        if n.is_top:
            psi.tensors[n.address] = np.asfortranarray(_top_tensor(n.shape, rng))
    return psi


def _forest_parts(case):
    """(trees, sops) of a forest: its structure does not depend on the seed."""
    trees, sops = [], []
    for t in range(case["trees"]):
        rng = np.random.default_rng([case["structure"], t])
        f, p = int(rng.choice((8, 16, 32, 48))), int(rng.choice((8, 16, 32)))
        edge = np.random.default_rng([case["structure"], t, 1])
        trees.append(M.balance_bonds(M.balanced_tree(f, p, 24, bonds=lambda h, q: int(edge.integers(6, 25)))))
        sops.append(M.coupled_oscillators(trees[-1], coupling=0.1, rng=rng, pairs_per_mode=(2, 6)))
    return trees, sops


def _problem(case, seed):
    """(tree, sop, flat wavefunction) of a case that has all three."""
    if case["kind"] == "forest":
        trees, sops = _forest_parts(case)
        tree, _, mode_off = M.forest(trees)
        psi = M.forest_psi(tree, [_psi(t, seed + 31 * k) for k, t in enumerate(trees)])
        return tree, M.forest_sop(sops, mode_off), psi.flat()
    tree = _tree(case)
    return tree, _sop(case, tree), _psi(tree, seed).flat()


def _qr_input(case, seed):
    """A wavefunction that has drifted from orthonormality by about 1e-3."""
    tree = _tree(case)
    psi = _psi(tree, seed)
    rng = np.random.default_rng(seed + 2)
    for n, t in zip(tree.nodes, psi.tensors):
        t += 1e-3 / math.sqrt(n.size) * (rng.standard_normal(t.shape) + 1j * rng.standard_normal(t.shape))
    return tree, psi.flat()


def _products_input(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(seed)
    d0, d1, up = case["d0"], case["d1"], case["up"]

    def normal(*shape):  # reversed shapes: the first index runs fastest
        return torch.randn(*shape, dtype=torch.complex128, device=dev, generator=g)

    return {"phi": normal(up, d1, d0), "h0": normal(d0, d0) / d0 ** 0.5, "h1": normal(d1, d1) / d1 ** 0.5,
            "rho": normal(up, up) / up ** 0.5}


class _DeviceArray:
    """A raw device pointer as torch reads it (complex128).  torch keeps this
    object for as long as a tensor looks at the memory, and it keeps the
    memory's owner."""

    def __init__(self, ptr, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<c16", "data": (ptr, False), "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "products":
        s = _products_input(case, seed)
        phi = s["phi"]
        s.update(case=case, ctx=Q.Context(0), t0=torch.empty_like(phi), t1=torch.empty_like(phi),
                 hmat=torch.empty(case["up"], case["up"], dtype=phi.dtype, device=phi.device),
                 out=torch.empty_like(phi))
        s["stream"] = torch.cuda.ExternalStream(_stream_of(s["ctx"]))
        return s
    if kind == "qr":
        tree, flat = _qr_input(case, seed)
        sop = M.SOP(M.OperatorTable())
        unit = sop.ops.add("unit", M.OP_DIAG, np.ones(tree.leaf_dim(0)))
        sop.push_back(M.MLO([(0, unit)]), 1.0)
        return {"case": case, "hrep": Q.HamiltonianRepresentation(sop, tree, flavour=Q.QT_PLAN_COMPRESSED),
                "psi": torch.from_numpy(flat).cuda()}
    if kind == "cdvr":
        tree, sop, leaf_x, potential = _cdvr_problem(case)
        hrep = Q.HamiltonianRepresentation(sop, tree, flavour=Q.QT_PLAN_GROUPED, potential=potential, leaf_x=leaf_x)
        return _sweep_state(case, hrep, _psi(tree, seed).flat())
    tree, sop, flat = _problem(case, seed)
    if kind == "derivative_host":
        return {"case": case, "hrep": Q.HamiltonianRepresentation(sop, tree), "psi": flat}
    flavour = Q.QT_PLAN_COMPRESSED | PRECISION[case["precision"]]
    flavour |= {"gradient": Q.QT_PLAN_GRADIENT, "scf": Q.QT_PLAN_SCF}.get(kind, 0)
    hrep = Q.HamiltonianRepresentation(sop, tree, flavour=flavour, eps=REGULARISATION)
    return _sweep_state(case, hrep, flat)


def _stream_of(ctx):
    p = Q.ctypes.c_void_p()
    ctx.check(ctx.L.qt_get_stream(ctx.h, Q.ctypes.byref(p)))
    return p.value or 0


def _sweep_state(case, hrep, flat):
    return {"case": case, "hrep": hrep, "psi": torch.from_numpy(flat).cuda(),
            "stream": torch.cuda.ExternalStream(hrep.stream()),
            "dpsi": torch.as_tensor(_DeviceArray(hrep.dpsi_device(), flat.size, hrep), device="cuda")}


def _cdvr_problem(case):
    """The Hamiltonian of model.cdvr_problem on the case's tree: kinetic terms
    and contrib's coupled-oscillator potential."""
    tree = _tree(case)
    basis = M.HOBasis(case["p"], omega=M.OMEGA_AU)
    sop = M.SOP(M.OperatorTable())
    kin = sop.ops.add("kin", M.OP_DENSE, basis.kin.astype(np.complex128))
    for m in range(case["modes"]):
        sop.push_back(M.MLO([(m, kin)]), 1.0)
    return tree, sop, {m: basis.x.copy() for m in range(case["modes"])}, M.PolyPotential.cdvr_model(case["modes"])


# --------------------------------------------------------------------------
# One pass
# --------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "products":
        c, d0, d1, up = s["ctx"], case["d0"], case["d1"], case["up"]
        c.mode_product(s["t0"].data_ptr(), s["h0"].data_ptr(), s["phi"].data_ptr(), 1, d0, d0, d1 * up)
        c.mode_product(s["t1"].data_ptr(), s["h1"].data_ptr(), s["t0"].data_ptr(), d0, d1, d1, up)
        c.hole_product(s["hmat"].data_ptr(), s["phi"].data_ptr(), s["t1"].data_ptr(), d0 * d1, up, up, 1)
        c.last_mode_product(s["out"].data_ptr(), s["rho"].data_ptr(), s["t1"].data_ptr(), d0 * d1, up)
        torch.cuda.current_stream().wait_stream(s["stream"])
        return {"chain": s["t1"], "matrix": s["hmat"], "applied": s["out"]}
    h = s["hrep"]
    if kind == "derivative_host":
        dpsi = Q.Derivative(h, s["psi"])
        return {"dpsi": dpsi, "expectation": np.complex128(Q.Expectation(h))}
    h.upload_device(s["psi"].data_ptr())
    if kind == "gradient":
        h.derivative()
        return {"dpsi": s["dpsi"], "gradient": h.gradient()}
    if kind == "cmf":
        h.cmf(CMF_DT, 1)
        return h.psi()
    if kind == "scf":
        ritz = h.scf(1, 5)
        return {"ritz": ritz, "psi": h.psi()}
    if kind == "qr":
        h.qr_orthogonal()
        return h.psi()
    h.derivative()
    torch.cuda.current_stream().wait_stream(s["stream"])
    return s["dpsi"]


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
def _restrictions(tree, sop):
    """(sub, inside): the modes under every node, and per node the distinct
    restrictions to it of the terms that reach outside it."""
    sub = {}
    for n in tree.nodes:
        sub[n.address] = {n.leaf_mode} if n.is_bottom else set().union(*(sub[c] for c in n.children))
    bound = {n.address: set() for n in tree.nodes}
    for t in sop.terms:
        modes = {m for m, _ in t.factors}
        for a in {a for m in modes for a in tree.path_to_root(m)}:
            if not modes <= sub[a]:
                bound[a].add(tuple(f for f in t.factors if f[0] in sub[a]))
    return sub, bound


def _sweep_flops(tree, sop, gradient=False, layer_only=False):
    """Complex multiply-adds (8 flops) of the sums a sweep consumes: per node
    and child one product with the child's block matrix, per distinct boundary
    restriction its chain, represent matrix and mean field, and the projected
    sum of products."""
    sub, bound = _restrictions(tree, sop)
    total = 0.0
    for n in tree.nodes:
        up = n.d_up
        chain = 0.0
        for u in bound[n.address]:
            kids = [n] if n.is_bottom else [tree.nodes[c] for c in n.children
                                            if any(f[0] in sub[c] for f in u)]
            chain += sum(1 if n.is_bottom else k.d_up for k in kids)
        block = n.shape[0] if n.is_bottom else sum(n.shape[:-1])
        per_node = chain + block + up * (len(bound[n.address]) + 2)          # X, Y and their sum
        if not layer_only:
            per_node += up * (len(bound[n.address]) + 2)                     # represent, block, density
            if not n.is_top:
                p = tree.nodes[n.parent]
                per_node += 2.0 * up * (1 + len(bound[n.address])) * p.size / n.size  # mean fields
        if gradient and not n.is_top:
            per_node += 2.0 * up
        total += 8.0 * n.size * per_node
    return total


def work(case):
    kind = case["kind"]
    if kind == "products":
        d0, d1, up = case["d0"], case["d1"], case["up"]
        n = d0 * d1 * up
        return {"bytes": 16.0 * (n + d0 * d0 + d1 * d1 + 2 * up * up + 2 * n), "flops": 8.0 * n * (d0 + d1 + 2 * up)}
    if kind == "forest":
        trees, sops = _forest_parts(case)
        return {"bytes": 32.0 * sum(n.size for t in trees for n in t.nodes),
                "flops": sum(_sweep_flops(t, s) for t, s in zip(trees, sops))}
    tree = _tree(case)
    size = float(sum(n.size for n in tree.nodes))
    if kind == "qr":
        # Householder QR, thin Q, and R multiplied into the parent
        flops = sum(0.0 if n.is_top else 8.0 * n.size * 3 * n.d_up + 8.0 * tree.nodes[n.parent].size * n.d_up
                    for n in tree.nodes)
        return {"bytes": 32.0 * size, "flops": flops}
    sop = _cdvr_problem(case)[1] if kind == "cdvr" else _sop(case, tree)
    flops = _sweep_flops(tree, sop, gradient=kind == "gradient")
    passes = 2.0
    if kind == "gradient":
        passes = 3.0
    elif kind == "cmf":  # two builds, twelve derivatives with frozen matrices
        layer = _sweep_flops(tree, sop, layer_only=True)
        flops = 2.0 * (flops - layer) + 12.0 * layer
    elif kind == "scf":  # per visit of a node: five effective-Hamiltonian products, one rebuild
        layer = _sweep_flops(tree, sop, layer_only=True)
        flops = 2.0 * (5.0 * layer + (flops - layer))
    elif kind == "cdvr":  # one joint-diagonalisation sweep per node, the correction tensors
        flops += sum(8.0 * case["modes"] * n.d_up ** 4 + 8.0 * n.d_up ** 5 for n in tree.nodes)
    return {"bytes": 16.0 * passes * size, "flops": flops}


# --------------------------------------------------------------------------
# The same outputs in 64 bits, by plain torch
# --------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("scf", "cdvr"):
        # iterates of a truncated Krylov sweep, grids of a joint
        # diagonalisation: defined by the steps taken, not by their inputs
        return None
    if kind == "products":
        s = _products_input(case, seed)
        t1 = _mode(s["h1"].T, _mode(s["h0"].T, s["phi"], 0), 1)
        up = case["up"]
        hole = s["phi"].reshape(up, -1).conj() @ t1.reshape(up, -1).T
        return {"chain": t1, "matrix": hole.T.contiguous(), "applied": _mode(s["rho"].T, t1, 2)}
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "qr":
        tree, flat = _qr_input(case, seed)
        return _exact_qr(tree, _split(tree, flat, dev))
    tree, sop, flat = _problem(case, seed)
    sweep = _ExactSweep(tree, sop, dev)
    phi = _split(tree, flat, dev)
    if kind == "cmf":
        return _exact_cmf(sweep, phi)
    mats = sweep.build(phi)
    dpsi = _join(sweep.layer(phi, mats))
    if kind == "derivative_host":
        top = tree.top.address
        hphi = sweep.internal(phi, mats, top)
        return {"dpsi": dpsi, "expectation": torch.vdot(phi[top].reshape(-1), hphi.reshape(-1)).cpu().numpy()[()]}
    if kind == "gradient":
        return {"dpsi": dpsi, "gradient": _exact_gradient(sweep, phi)}
    return dpsi


def _split(tree, flat, dev):
    """Node tensors with reversed indices (the bond up first)."""
    off = tree.offsets()
    x = torch.from_numpy(flat).to(dev)
    return [x[off[n.address]:off[n.address + 1]].reshape(tuple(reversed(n.shape))) for n in tree.nodes]


def _join(tensors):
    return torch.cat([t.reshape(-1) for t in tensors])


def _mode(m, t, k):
    """sum_a m(j, a) t[.., a, ..] along QuTree index k of a reversed tensor."""
    ax = t.dim() - 1 - k
    return torch.movedim(torch.tensordot(m, t, dims=([1], [ax])), 0, ax)


def _hole(a, b, k):
    """S(i, j) = sum conj(a[.., i, ..]) b[.., j, ..] over all indices but k."""
    ax = a.dim() - 1 - k
    x = torch.movedim(a, ax, 0).reshape(a.shape[ax], -1)
    return x.conj() @ torch.movedim(b, ax, 0).reshape(b.shape[ax], -1).T


class _ExactSweep:
    """The derivative of a tree-network wavefunction under a sum of products,
    from its definition: represent matrices and summed mean fields per
    restriction, projector, regularised inverse density."""

    def __init__(self, tree, sop, dev):
        self.tree = tree
        self.op = [torch.from_numpy(np.ascontiguousarray(sop.ops.dense(o))).to(dev) for o in range(len(sop.ops.kind))]
        sub = {}
        for n in tree.nodes:
            sub[n.address] = {n.leaf_mode} if n.is_bottom else set().union(*(sub[c] for c in n.children))
        self.sub = sub
        self.lca = {n.address: {} for n in tree.nodes}    # restriction -> coefficient
        self.bound = {n.address: set() for n in tree.nodes}
        for c, t in zip(sop.coeffs, sop.terms):
            u = tuple(t.factors)
            modes = {m for m, _ in u}
            found = False
            for a in sorted({a for m in modes for a in tree.path_to_root(m)}):
                if modes <= sub[a]:
                    if not found:
                        self.lca[a][u] = self.lca[a].get(u, 0) + c
                    found = True
                else:
                    self.bound[a].add(self.restrict(u, a))

    def restrict(self, u, a):
        return tuple(f for f in u if f[0] in self.sub[a])

    def chain(self, phi, mats, a, u, skip=None):
        """phi_a with the factors of u inside a applied (child `skip` left out)."""
        n = self.tree.nodes[a]
        x = phi[a]
        if n.is_bottom:
            for _, o in u:
                x = _mode(self.op[o], x, 0)
            return x
        for k, c in enumerate(n.children):
            r = self.restrict(u, c)
            if r and c != skip:
                x = _mode(mats["H"][c][r], x, k)
            elif not r and c != skip and "S" in mats:
                x = _mode(mats["S"][c], x, k)
        return x

    def internal(self, phi, mats, a):
        """Y = the terms wholly inside a applied to phi_a."""
        n = self.tree.nodes[a]
        y = torch.zeros_like(phi[a])
        for k, c in enumerate(n.children):
            x = phi[a]
            if "S" in mats:
                for j, d in enumerate(n.children):
                    if j != k:
                        x = _mode(mats["S"][d], x, j)
            y = y + _mode(mats["block"][c], x, k)
        for u, c in self.lca[a].items():
            y = y + c * self.chain(phi, mats, a, u)
        return y

    def represent(self, phi, mats):
        for n in self.tree.nodes:
            a, last = n.address, n.order - 1
            mats["H"][a] = {u: _hole(phi[a], self.chain(phi, mats, a, u), last) for u in self.bound[a]}
            mats["block"][a] = _hole(phi[a], self.internal(phi, mats, a), last)
            if "S" in mats:
                x = phi[a]
                for k, c in enumerate(n.children):
                    x = _mode(mats["S"][c], x, k)
                mats["S"][a] = _hole(phi[a], x, last)

    def build(self, phi):
        mats = {"H": {}, "block": {}, "rho": {}, "inv": {}, "C": {}}
        self.represent(phi, mats)
        for n in reversed(self.tree.nodes):
            a = n.address
            if n.is_top:
                mats["rho"][a], mats["C"][a] = torch.ones(1, 1, dtype=phi[a].dtype, device=phi[a].device), {}
                continue
            p, k = n.parent, n.child_idx
            last = self.tree.nodes[p].order - 1
            weighted = _mode(mats["rho"][p], phi[p], last)
            rho = _hole(phi[p], weighted, k)
            w, v = torch.linalg.eigh(rho)
            w = w + REGULARISATION * torch.exp(-w / REGULARISATION)
            mats["rho"][a], mats["inv"][a] = rho, (v / w) @ v.conj().T
            field = {u: 0 for u in self.bound[a]}
            for u, c in self.lca[p].items():
                r = self.restrict(u, a)
                if r in field:
                    x = _mode(mats["rho"][p], self.chain(phi, mats, p, u, skip=a), last)
                    field[r] = field[r] + c * _hole(phi[p], x, k)
            for w_ in self.bound[p]:
                r = self.restrict(w_, a)
                if r:
                    x = _mode(mats["C"][p][w_], self.chain(phi, mats, p, w_, skip=a), last)
                    field[r] = field[r] + _hole(phi[p], x, k)
            mats["C"][a] = field
        return mats

    def layer(self, phi, mats):
        """-i (1 - P) rho^-1 H phi of every node, the matrices held."""
        out = []
        for n in self.tree.nodes:
            a, last = n.address, n.order - 1
            y = self.internal(phi, mats, a)
            if n.is_top:
                out.append(-1j * y)
                continue
            y = _mode(mats["rho"][a], y, last)
            for u in self.bound[a]:
                y = y + _mode(mats["C"][a][u], self.chain(phi, mats, a, u), last)
            overlap = _hole(phi[a], phi[a], last)
            part = torch.linalg.solve(overlap, _hole(phi[a], y, last))
            y = y - _mode(part.T, phi[a], last)
            out.append(-1j * _mode(mats["inv"][a], y, last))
        return out


def _exact_cmf(sweep, phi):
    """One second-order constant-mean-field step with RK4 substeps."""
    def rk4(y, mats, h, steps):
        for _ in range(steps):
            k1 = sweep.layer(y, mats)
            k2 = sweep.layer([a + 0.5 * h * b for a, b in zip(y, k1)], mats)
            k3 = sweep.layer([a + 0.5 * h * b for a, b in zip(y, k2)], mats)
            k4 = sweep.layer([a + h * b for a, b in zip(y, k3)], mats)
            y = [a + h / 6 * (p + 2 * q + 2 * r + s) for a, p, q, r, s in zip(y, k1, k2, k3, k4)]
        return y

    half = rk4(phi, sweep.build(phi), 0.5 * CMF_DT, 1)
    return _join(rk4(phi, sweep.build(half), 0.5 * CMF_DT, 2))


def _exact_gradient(sweep, phi):
    """dE/dPhi^* by differentiating E = <Psi|H|Psi> / <Psi|Psi>."""
    phi = [t.clone().requires_grad_(True) for t in phi]
    mats = {"H": {}, "block": {}, "S": {}}
    sweep.represent(phi, mats)
    top = sweep.tree.top.address
    (mats["block"][top][0, 0].real / mats["S"][top][0, 0].real).backward()
    return _join([t.grad for t in phi]) / 2


def _exact_qr(tree, phi):
    """Householder QR of every node (columns mapped to -e^{i arg x0} |x| e_1),
    R multiplied into the parent."""
    phi = list(phi)
    for n in tree.nodes:
        if n.is_top:
            continue
        a = phi[n.address].reshape(n.d_up, -1).T.clone()
        m, d = a.shape
        work_, vs = a.clone(), []
        for j in range(min(m, d)):
            x = work_[j:, j].clone()
            v = x.clone()
            v[0] += x[0] / x[0].abs() * torch.linalg.vector_norm(x)
            v = v / torch.linalg.vector_norm(v)
            work_[j:] -= 2 * torch.outer(v, v.conj() @ work_[j:])
            vs.append(v)
        q = torch.eye(m, d, dtype=a.dtype, device=a.device)
        for j, v in reversed(list(enumerate(vs))):
            q[j:] -= 2 * torch.outer(v, v.conj() @ q[j:])
        phi[n.address] = q.T.reshape(phi[n.address].shape)
        phi[n.parent] = _mode(q.conj().T @ a, phi[n.parent], n.child_idx)
    return _join(phi)
