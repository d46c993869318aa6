"""The performance cases of the J/K framework: what is timed, on which inputs, and how exact the results have to be.

Every case is one pass through a public entry point, as an SCF, response, force or packed-integral program
calls it, on seeded water clusters (gradscf_b200.workloads) and densities with the structure that an SCF meets:
occupied orbitals that sit on a molecule and decay with distance, and their change between two iterations.

  jk        DirectJKPlan.jk: J and K of one symmetric density, FP64 or split precision
  graph     JKGraph.run: the captured build that an SCF replays each iteration, on one or many molecules
  response  direct_jk: J and K of a batch of nonsymmetric trial densities
  autograd  direct_jk_ad forward and backward: J, K, the density and the coordinate gradients
  force     rhf_gradient: the nuclear gradient of an RHF result, split precision
  eri       packed_eri: every two-electron integral in s8 storage
  packed    packed_jk: J and K from stored s8 integrals
  hvp       direct_jk_geometry_hvp: one product with the second coordinate derivatives

`exact` evaluates the integrals anew in 64 bits, by the McMurchie-Davidson scheme in torch, unscreened.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gradscf_b200 import autograd as AD
from gradscf_b200 import basis as B
from gradscf_b200 import flop_model
from gradscf_b200 import jk as JK
from gradscf_b200 import scf as S
from gradscf_b200 import workloads as W

CUT = 1e-12          # Schwarz cutoff of the SCF workloads
STEP = 1e-2          # relative change of the orbitals between two SCF iterations
BATCH_SEED = 3


def listed():
    return [
        # the smallest call: J/K of one water, where latency and launches count
        {"name": "jk_water_dz_fp64", "kind": "jk", "waters": 1, "basis": "cc-pvdz", "precision": "fp64", "cart": False},
        # the first FP64 build of an SCF on a small cluster (whole density)
        {"name": "jk_w8_dz_fp64", "kind": "jk", "waters": 8, "basis": "cc-pvdz", "precision": "fp64", "cart": False},
        # one split-precision SCF iteration of the benchmark cluster, replayed from a graph
        {"name": "graph_w32_dz_split", "kind": "graph", "waters": 32, "molecules": 1, "basis": "cc-pvdz",
         "precision": "split"},
        # a triple-zeta build with f shells in FP64
        {"name": "jk_w6_tz_fp64", "kind": "jk", "waters": 6, "basis": "cc-pvtz", "precision": "fp64", "cart": False},
        # a triple-zeta SCF increment in split precision, larger cluster
        {"name": "graph_w11_tz_split", "kind": "graph", "waters": 11, "molecules": 1, "basis": "cc-pvtz",
         "precision": "split"},
        # many small uneven molecules in one plan: one packed split build per SCF iteration of all of them
        {"name": "graph_batch32_dz_split", "kind": "graph", "waters": 16, "molecules": 32, "basis": "cc-pvdz",
         "precision": "split"},
        # response equations: several nonsymmetric trial densities in one call, Cartesian d shells
        {"name": "response4_w5_631gs", "kind": "response", "waters": 5, "basis": "6-31g*", "batch": 4, "cart": True},
        # a differentiable J/K: forward, density gradient and coordinate gradient
        {"name": "autograd_w6_631gs", "kind": "autograd", "waters": 6, "basis": "6-31g*"},
        # RHF forces with the split-precision coordinate gradient, f shells
        {"name": "force_w4_tz_split", "kind": "force", "waters": 4, "basis": "cc-pvtz"},
        # the stored integrals of a small cluster
        {"name": "eri_w4_dz", "kind": "eri", "waters": 4, "basis": "cc-pvdz"},
        # J/K of alpha and beta densities from stored integrals
        {"name": "packed2_w7_dz", "kind": "packed", "waters": 7, "basis": "cc-pvdz", "batch": 2},
        # a Hessian-vector product of a small molecule
        {"name": "hvp_w2_631gs", "kind": "hvp", "waters": 2, "basis": "6-31g*"},
    ]


def _spread(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["jk", "jk", "graph", "graph", "response", "autograd", "force", "eri", "packed", "hvp"])
    if kind == "jk":
        basis = rng.choice(["cc-pvdz", "6-31g*", "cc-pvtz"])
        top = {"cc-pvdz": 24, "6-31g*": 32, "cc-pvtz": 6}[basis]
        return {"kind": kind, "waters": _spread(rng, 1, top), "basis": basis, "precision": rng.choice(["fp64", "split"]),
                "cart": basis == "6-31g*" and rng.random() < 0.5}
    if kind == "graph":
        if rng.random() < 0.5:
            return {"kind": kind, "waters": rng.randint(2, 20), "molecules": _spread(rng, 2, 40), "basis": "cc-pvdz",
                    "precision": rng.choice(["fp64", "split"])}
        basis = rng.choice(["cc-pvdz", "6-31g*", "cc-pvtz"])
        top = {"cc-pvdz": 32, "6-31g*": 40, "cc-pvtz": 10}[basis]
        return {"kind": kind, "waters": _spread(rng, 2, top), "molecules": 1, "basis": basis,
                "precision": rng.choice(["fp64", "split"])}
    if kind == "response":
        basis = rng.choice(["cc-pvdz", "6-31g*"])
        return {"kind": kind, "waters": _spread(rng, 1, 8), "basis": basis, "batch": rng.randint(1, 7),
                "cart": basis == "6-31g*" and rng.random() < 0.5}
    if kind == "autograd":
        return {"kind": kind, "waters": _spread(rng, 1, 12), "basis": rng.choice(["cc-pvdz", "6-31g*"])}
    if kind == "force":
        basis = rng.choice(["cc-pvdz", "cc-pvtz"])
        return {"kind": kind, "waters": _spread(rng, 1, 16 if basis == "cc-pvdz" else 5), "basis": basis}
    if kind == "eri":
        return {"kind": kind, "waters": _spread(rng, 1, 6), "basis": rng.choice(["cc-pvdz", "6-31g*"])}
    if kind == "packed":
        return {"kind": kind, "waters": rng.randint(1, 9), "basis": rng.choice(["cc-pvdz", "6-31g*"]),
                "batch": rng.randint(1, 6)}
    return {"kind": "hvp", "waters": _spread(rng, 1, 3), "basis": rng.choice(["6-31g*", "3-21g"])}


# ---------------------------------------------------------------- inputs
def _sizes(case):
    """Waters of every molecule of the case."""
    if case.get("molecules", 1) == 1:
        return [case["waters"]]
    return [int(n) for n in W.batch_sizes(case["molecules"], BATCH_SEED, 1, case["waters"])]


def _molecule(case, seed, waters):
    """(specification, libcint tables, AO centres, water of every AO) of one seeded cluster."""
    spec = W.water_cluster(waters, seed)
    top, par, owner = B.prepare_basis(spec, case["basis"], cart=case.get("cart", False))
    atm, bas, env = B.pack(top, par)
    dim = np.diff(B.ao_offsets(bas, top.cart))
    return {"spec": spec, "top": top, "par": par, "owner": owner, "tables": (atm, bas, env),
            "centres": np.repeat(par.centers, dim, axis=0), "water": np.repeat(owner // 3, dim), "nao": int(dim.sum())}


def _orbitals(mol, rng):
    """Five occupied orbitals per water: normal coefficients that decay with the distance from the water."""
    water = mol["water"]
    count = int(water.max()) + 1
    middle = np.stack([mol["centres"][water == w].mean(0) for w in range(count)])
    dist = np.linalg.norm(mol["centres"][:, None, :] - middle[None], axis=-1)
    scale = np.exp(-0.6 * dist) / math.sqrt(mol["nao"] / count)
    return rng.normal(size=(mol["nao"], 5 * count)) * np.repeat(scale, 5, axis=1)


def _density(mol, rng):
    c = _orbitals(mol, rng)
    return 2.0 * c @ c.T


def _increment(mol, rng):
    """D' - D of orbitals changed by STEP, as an SCF iteration hands it to the build."""
    c, x = _orbitals(mol, rng), _orbitals(mol, rng)
    d = STEP * (c @ x.T + x @ c.T) + STEP * STEP * (x @ x.T)
    return d + d.T


def _trial(mol, rng):
    """A nonsymmetric trial density (occupied times virtual orbitals)."""
    return _orbitals(mol, rng) @ _orbitals(mol, rng).T


def _inputs(case, seed):
    """The molecules and every array of the case, as numpy (the same for `prepare` and `exact`)."""
    rng = np.random.default_rng(seed)
    sizes = _sizes(case)
    mols = [_molecule(case, 1000 * seed + m, n) for m, n in enumerate(sizes)]
    mol, kind = mols[0], case["kind"]
    out = {"mols": mols, "mol": mol}
    if kind == "jk":
        out["d"] = _density(mol, rng) if case["precision"] == "fp64" else _increment(mol, rng)
    elif kind == "graph":
        make = _density if case["precision"] == "fp64" else _increment
        out["ds"] = [make(m, rng) for m in mols]
    elif kind == "response":
        out["d"] = np.stack([_trial(mol, rng) for _ in range(case["batch"])])
    elif kind == "packed":
        out["d"] = np.stack([_density(mol, rng) for _ in range(case["batch"])])
    elif kind in ("autograd", "hvp"):
        out["d"] = _density(mol, rng)
        a, b = _density(mol, rng), _density(mol, rng)
        out["cj"], out["ck"] = a, -0.5 * b
        if kind == "hvp":
            env = np.zeros(len(mol["tables"][2]))
            u = rng.normal(size=mol["par"].nuclear_coords.shape)
            nnuc = len(u)
            for row, xyz in enumerate(np.concatenate([u, u[mol["owner"]]])):
                p = mol["tables"][0][row, 1]
                env[p:p + 3] = xyz
            out["u"], out["u_nuc"] = env, u
            assert nnuc + len(mol["owner"]) == len(mol["tables"][0])
    elif kind == "force":
        c = _orbitals(mol, rng)
        out["c"], out["e"] = c, np.linspace(-20.0, -0.3, c.shape[1])
    return out


def prepare(case, seed):
    x = _inputs(case, seed)
    mol, kind = x["mol"], case["kind"]

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a), device="cuda")

    state = {"case": case, "kind": kind}
    if kind == "jk":
        state["plan"] = JK.DirectJKPlan([mol["tables"]], cart=case["cart"], cutoff=CUT)
        state["d"] = dev(x["d"])
    elif kind == "graph":
        plan = JK.DirectJKPlan([m["tables"] for m in x["mols"]], cart=False, cutoff=CUT)
        state["graph"] = JK.JKGraph(plan, 1, hermi=1, precision=case["precision"])
        state["d"] = dev(np.concatenate([d.ravel() for d in x["ds"]])).reshape(1, -1)
    elif kind == "response":
        state["action"] = JK.NativeDirectBasis(JK.make_plan(mol["top"]), mol["par"]).prepare_jk(screening_threshold=CUT)
        state["d"] = dev(x["d"])
    elif kind == "autograd":
        state["basis"] = AD.BasisContext(mol["top"], mol["par"], mol["owner"], cutoff=CUT)
        state["d"], state["coords"] = dev(x["d"]).requires_grad_(), dev(mol["par"].nuclear_coords).requires_grad_()
        state["cj"], state["ck"] = dev(x["cj"]), dev(x["ck"])
    elif kind == "force":
        state["mol"] = S.Molecule(mol["spec"], case["basis"], schwarz_cut=CUT)
        c = dev(x["c"])
        nocc = c.shape[1]
        state["res"] = S.SCFResult(energy=0.0, converged=True, cycles=1, density=2.0 * c @ c.T, mo_energy=dev(x["e"]),
                                   mo_coeff=c, nocc=nocc)
    elif kind == "eri":
        state["tables"] = mol["tables"]
    elif kind == "packed":
        state["eri"] = JK.packed_eri(*mol["tables"], cart=False, aosym="s8")
        state["d"] = dev(x["d"])
    elif kind == "hvp":
        state["tables"], state["u"] = mol["tables"], x["u"]
        state["d"], state["cot"] = dev(x["d"]), (dev(x["cj"]), dev(x["ck"]))
    return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "jk":
        return state["plan"].jk(state["d"], hermi=True, precision=case["precision"])
    if kind == "graph":
        return state["graph"].run(state["d"])
    if kind == "response":
        return state["action"](state["d"])
    if kind == "autograd":
        j, k = AD.direct_jk_ad(state["basis"], state["d"], state["coords"])
        gd, gc = torch.autograd.grad((j, k), (state["d"], state["coords"]), (state["cj"], state["ck"]))
        return j.detach(), k.detach(), gd, gc
    if kind == "force":
        return S.rhf_gradient(state["mol"], state["res"], precision="split")
    if kind == "eri":
        return JK.packed_eri(*state["tables"], cart=False, aosym="s8")
    if kind == "packed":
        return JK.packed_jk(state["eri"], state["d"])
    return JK.direct_jk_geometry_hvp(*state["tables"], state["d"], state["u"], state["cot"], cart=False, cutoff=CUT)


# ---------------------------------------------------------------- work and tolerance
def _pair_counts(tables, cart, cut):
    """Shell pairs of one molecule: per pair of angular momenta the sorted estimated bounds with the running sum of the
    primitive pairs.  A pair's bound is estimated from its s-type overlap charges, sum |c c'| K sqrt(2 pi^2.5 / (p^2 sqrt(2p)))."""
    atm, bas, env = tables
    shells = []
    for at, l, np_, nc, _, pe, pc, *_ in bas.tolist():
        p = atm[at, 1]
        a = env[pe:pe + np_]
        c = np.abs(env[pc:pc + np_ * nc].reshape(nc, np_)).max(0)
        # an s function of the same self-overlap stands in for the shell
        c = c * np.sqrt((math.gamma(l + 1.5) / math.gamma(1.5)) / (2.0 * a) ** l) * (0.282 * math.sqrt(2 * l + 1))
        shells.append((l, env[p:p + 3], a, c, nc))
    found = {}
    for i, (li, ri, ai, ci, ni) in enumerate(shells):
        for lj, rj, aj, cj, nj in shells[:i + 1]:
            p = ai[:, None] + aj[None]
            ex = ai[:, None] * aj[None] / p * ((ri - rj) ** 2).sum()
            q = (ci[:, None] * cj[None] * np.exp(-ex) * np.sqrt(2 * math.pi ** 2.5 / (p * p * np.sqrt(2 * p)))).sum()
            found.setdefault((max(li, lj), min(li, lj)), []).append((q, int((ex < 40).sum()), ni * nj))
    return {k: np.array(sorted(v, reverse=True)) for k, v in found.items()}


def _quartet_flops(tables, cart, densities, cut=CUT, derivative=1.0):
    """Operations of the significant quartets (gradscf_b200.flop_model) under the estimated bounds."""
    pairs, total = _pair_counts(tables, cart, cut), 0.0
    for x, px in pairs.items():
        for y, py in pairs.items():
            if x < y:
                continue
            # the partners of each bra pair: its prefix of the sorted ket bounds
            upto = np.searchsorted(-py[:, 0], -cut / np.maximum(px[:, 0], 1e-300)) if cut > 0 else np.full(len(px), len(py))
            prims = np.concatenate([[0.0], np.cumsum(py[:, 1])])[upto]
            count = np.concatenate([[0.0], np.cumsum(py[:, 2])])[upto]
            share = 0.5 if x == y else 1.0
            cls = (*x, *y)
            total += share * derivative * float((px[:, 1] * prims).sum()) * flop_model.per_primitive_quartet(*cls)
            total += share * float((px[:, 2] * count).sum()) * flop_model.per_quartet_digestion(*cls, densities)
    return total


def work(case):
    """One read of the inputs and one write of the results, and the Rys-quadrature operations of the quartets."""
    kind = case["kind"]
    mols = [_molecule(case, 1000 + m, n) for m, n in enumerate(_sizes(case))]
    n2 = sum(8.0 * m["nao"] ** 2 for m in mols)
    tables = sum(8.0 * len(m["tables"][2]) for m in mols)
    cart = case.get("cart", False)

    def flops(densities, **kw):
        return sum(_quartet_flops(m["tables"], cart, densities, **kw) for m in mols)

    if kind in ("jk", "graph"):
        return {"bytes": 3 * n2 + tables, "flops": flops(1)}
    if kind == "response":
        return {"bytes": 3 * n2 * case["batch"] + tables, "flops": flops(2 * case["batch"])}
    if kind == "autograd":  # J/K, the density gradient from the same integrals, and a first derivative
        return {"bytes": 6 * n2 + tables, "flops": flops(3) + flops(1, derivative=3.0)}
    if kind == "force":
        return {"bytes": 2 * n2 + tables, "flops": flops(1, derivative=3.0)}
    if kind == "hvp":
        return {"bytes": 3 * n2 + tables, "flops": flops(1, derivative=9.0)}
    n = mols[0]["nao"]
    pairs = n * (n + 1) // 2
    packed = 8.0 * (pairs * (pairs + 1) // 2)
    if kind == "eri":
        return {"bytes": packed + tables, "flops": flops(0, cut=0.0)}
    return {"bytes": packed + 3 * n2 * case["batch"], "flops": 12.0 * case["batch"] * packed / 8.0}


def tolerance(case):
    """Split precision: quartets below the bound 1e-6 run in FP32; against the FP64 build 2e-10 (2-norm) and 1.2e-8
    (largest element) were measured up to 32 waters.  FP64: builds repeat to 6e-15 and differ from the unscreened 64-bit
    results by 2e-12, what the Schwarz cutoff leaves out; nearly empty densities and small molecules reach 3e-11."""
    if case["kind"] == "force" or case.get("precision") == "split":
        return {"rel": 1e-9, "max": 1e-7}
    return {"rel": 1e-11, "max": 1e-9}


# ---------------------------------------------------------------- exact results
class _Boys(torch.autograd.Function):
    """F_0..F_m(t): the ascending series and downward recursion below t = 40, erf and upward recursion above."""

    @staticmethod
    def forward(ctx, t, m):
        ctx.save_for_backward(t)
        ctx.m = m
        small = t.clamp(max=40.0)
        term = torch.full_like(t, 1.0 / (2 * m + 1))
        total = term.clone()
        for k in range(1, 190):
            term = term * (2.0 * small) / (2 * m + 2 * k + 1)
            total += term
            if k % 16 == 0 and bool((term < 1e-17 * total).all()):
                break
        low = [None] * (m + 1)
        ex = torch.exp(-small)
        low[m] = ex * total
        for i in range(m - 1, -1, -1):
            low[i] = (2.0 * small * low[i + 1] + ex) / (2 * i + 1)
        big = t.clamp(min=40.0)
        ex = torch.exp(-big)
        up = 0.5 * torch.sqrt(math.pi / big) * torch.erf(torch.sqrt(big))
        out = torch.empty((m + 1,) + t.shape, dtype=t.dtype, device=t.device)
        for i in range(m + 1):
            out[i] = torch.where(t < 40.0, low[i], up)
            up = ((2 * i + 1) * up - ex) / (2.0 * big)
        return out

    @staticmethod
    def backward(ctx, g):
        (t,) = ctx.saved_tensors
        return -(g * _Boys.apply(t, ctx.m + 1)[1:]).sum(0), None


def _components(l):
    return [(x, y, l - x - y) for x in range(l, -1, -1) for y in range(l - x, -1, -1)]


def _output_matrix(l, cart):
    """Raw Cartesian components -> output functions: real solid harmonics, or libcint's Cartesian factors."""
    n = len(_components(l))
    if cart:
        return np.eye(n) * {0: 0.5 / math.sqrt(math.pi), 1: math.sqrt(0.75 / math.pi)}.get(l, 1.0)
    c = math.sqrt(1.0 / math.pi)
    rows = {
        0: [{(0, 0, 0): 0.5 * c}],
        1: [{(1, 0, 0): math.sqrt(0.75) * c}, {(0, 1, 0): math.sqrt(0.75) * c}, {(0, 0, 1): math.sqrt(0.75) * c}],
        2: [{(1, 1, 0): math.sqrt(15.0) / 2 * c}, {(0, 1, 1): math.sqrt(15.0) / 2 * c},
            {(2, 0, 0): -math.sqrt(5.0) / 4 * c, (0, 2, 0): -math.sqrt(5.0) / 4 * c, (0, 0, 2): math.sqrt(5.0) / 2 * c},
            {(1, 0, 1): math.sqrt(15.0) / 2 * c},
            {(2, 0, 0): math.sqrt(15.0) / 4 * c, (0, 2, 0): -math.sqrt(15.0) / 4 * c}],
        3: [{(2, 1, 0): 3 * math.sqrt(35.0 / 32) * c, (0, 3, 0): -math.sqrt(35.0 / 32) * c},
            {(1, 1, 1): math.sqrt(105.0) / 2 * c},
            {(0, 1, 2): 4 * math.sqrt(21.0 / 32) * c, (2, 1, 0): -math.sqrt(21.0 / 32) * c,
             (0, 3, 0): -math.sqrt(21.0 / 32) * c},
            {(0, 0, 3): math.sqrt(7.0) / 2 * c, (2, 0, 1): -1.5 * math.sqrt(7.0) / 2 * c,
             (0, 2, 1): -1.5 * math.sqrt(7.0) / 2 * c},
            {(1, 0, 2): 4 * math.sqrt(21.0 / 32) * c, (3, 0, 0): -math.sqrt(21.0 / 32) * c,
             (1, 2, 0): -math.sqrt(21.0 / 32) * c},
            {(2, 0, 1): math.sqrt(105.0) / 4 * c, (0, 2, 1): -math.sqrt(105.0) / 4 * c},
            {(3, 0, 0): math.sqrt(35.0 / 32) * c, (1, 2, 0): -3 * math.sqrt(35.0 / 32) * c}]}[l]
    out = np.zeros((n, 2 * l + 1))
    for f, row in enumerate(rows):
        for comp, v in row.items():
            out[_components(l).index(comp), f] = v
    return out


def _hermite_1d(la, lb, a, b, xa, xb):
    """Hermite coefficients E[i][j][t] of x_A^i x_B^j exp(-a x_A^2 - b x_B^2)."""
    p, ab = a + b, xa - xb
    pa, pb, half = -b / p * ab, a / p * ab, 0.5 / p
    zero = torch.zeros_like(p)
    e = {(0, 0): [torch.exp(-a * b / p * ab * ab)]}

    def step(row, shift):
        get = lambda t: row[t] if 0 <= t < len(row) else zero  # noqa: E731
        return [half * get(t - 1) + shift * get(t) + (t + 1) * get(t + 1) for t in range(len(row) + 1)]

    for i in range(la):
        e[i + 1, 0] = step(e[i, 0], pa)
    for i in range(la + 1):
        for j in range(lb):
            e[i, j + 1] = step(e[i, j], pb)
    return e


def _hermites(n):
    return [(t, u, v) for t in range(n + 1) for u in range(n + 1 - t) for v in range(n + 1 - t - u)]


class _Exact:
    """The contracted two-electron integrals of one molecule, pair class by pair class, in float64."""

    def __init__(self, tables, cart, xyz, device):
        atm, bas, env = tables
        self.device, self.cart, self.xyz = device, cart, xyz     # xyz: (atm rows, 3), may carry a gradient
        shells, ao = [], 0
        for at, l, np_, nc, _, pe, pc, *_ in bas.tolist():
            for k in range(nc):
                shells.append((l, at, env[pe:pe + np_], env[pc + k * np_:pc + (k + 1) * np_], ao))
                ao += len(_components(l)) if cart else 2 * l + 1
        self.n = ao
        where = xyz.detach().cpu().numpy()
        raw = {}
        for i, s in enumerate(shells):
            for r in shells[:i + 1]:
                x, y = (s, r) if s[0] >= r[0] else (r, s)
                cls = raw.setdefault((x[0], y[0]), {k: [] for k in ("a", "b", "c", "at", "bt", "pair", "ao", "deg")})
                ex = x[2][:, None] * y[2][None] / (x[2][:, None] + y[2][None]) * ((where[x[1]] - where[y[1]]) ** 2).sum()
                cc = x[3][:, None] * y[3][None]
                keep = (ex < 60.0) & (cc != 0.0)
                if not keep.any():
                    continue
                cls["a"].append(np.broadcast_to(x[2][:, None], keep.shape)[keep])
                cls["b"].append(np.broadcast_to(y[2][None], keep.shape)[keep])
                cls["c"].append(cc[keep])
                count = int(keep.sum())
                cls["at"] += [x[1]] * count
                cls["bt"] += [y[1]] * count
                cls["pair"] += [len(cls["ao"])] * count
                cls["ao"].append((x[4], y[4]))
                cls["deg"].append(1.0 if x is y else 2.0)
        self.classes = {k: self._tensors(v) for k, v in sorted(raw.items()) if v["ao"]}

    def _tensors(self, v):
        f = lambda x: torch.as_tensor(np.asarray(x), device=self.device)  # noqa: E731
        return {"a": f(np.concatenate(v["a"])), "b": f(np.concatenate(v["b"])), "c": f(np.concatenate(v["c"])),
                "at": f(v["at"]), "bt": f(v["bt"]), "pair": f(v["pair"]), "ao": f(v["ao"]), "deg": f(v["deg"])}

    def charges(self, cls, sel=slice(None)):
        """(exponent sums, centres, E[primitive pair, output pair, Hermite]) of the pairs of a class."""
        la, lb = cls
        v = self.classes[cls]
        a, b, c = v["a"][sel], v["b"][sel], v["c"][sel]
        ra, rb = self.xyz[v["at"][sel]], self.xyz[v["bt"][sel]]
        p = a + b
        e = [_hermite_1d(la, lb, a, b, ra[:, i], rb[:, i]) for i in range(3)]
        zero = torch.zeros_like(p)
        rows = []
        for x in _components(la):
            for y in _components(lb):
                one = [e[i][x[i], y[i]] for i in range(3)]
                rows.append(torch.stack([
                    one[0][t] * one[1][u] * one[2][w] if t < len(one[0]) and u < len(one[1]) and w < len(one[2]) else zero
                    for t, u, w in _hermites(la + lb)], -1))
        raw = torch.stack(rows, 1) * c[:, None, None]
        t = np.kron(_output_matrix(la, self.cart), _output_matrix(lb, self.cart))
        eo = torch.einsum("pch,cf->pfh", raw, torch.as_tensor(t, device=self.device))
        return p, (a[:, None] * ra + b[:, None] * rb) / p[:, None], eo

    def blocks(self, bra, ket, budget=1 << 25):
        """Yields (first contracted bra pair, ERI[bra pair, bra output pair, ket pair, ket output pair])."""
        top, nk = sum(bra) + sum(ket), len(self.classes[ket]["ao"])
        q, rq, ek = self.charges(ket)
        hk = _hermites(sum(ket))
        sign = torch.as_tensor([(-1.0) ** sum(h) for h in hk], device=self.device, dtype=torch.float64)
        ek = ek * sign
        index = {h: i for i, h in enumerate(_hermites(top))}
        owner = self.classes[bra]["pair"].cpu().numpy()
        starts = np.concatenate([np.nonzero(np.diff(owner, prepend=-1))[0], [len(owner)]])
        size = len(q) * (len(index) * 3 + ek.shape[1]) + nk * ek.shape[1] * len(_hermites(sum(bra)))
        room = max(1, budget * 8 // max(1, size))
        first = 0
        while first < len(starts) - 1:
            last = first + 1
            while last < len(starts) - 1 and starts[last + 1] - starts[first] <= room:
                last += 1
            sel = slice(int(starts[first]), int(starts[last]))
            p, rp, eb = self.charges(bra, sel)
            d = rp[:, None, :] - rq[None]
            alpha = p[:, None] * q[None] / (p[:, None] + q[None])
            pre = 2.0 * math.pi ** 2.5 / (p[:, None] * q[None] * torch.sqrt(p[:, None] + q[None]))
            f = _Boys.apply(alpha * (d * d).sum(-1), top)
            level = {}
            for m in range(top, -1, -1):
                now = {(0, 0, 0): pre * (-2.0 * alpha) ** m * f[m]}
                for h in _hermites(top - m):
                    if h == (0, 0, 0):
                        continue
                    ax = max(range(3), key=lambda i: h[i])
                    one = tuple(h[i] - (i == ax) for i in range(3))
                    val = d[..., ax] * level[one]
                    if h[ax] > 1:
                        val = val + (h[ax] - 1) * level[tuple(h[i] - 2 * (i == ax) for i in range(3))]
                    now[h] = val
                level = now
            pair = self.classes[bra]["pair"][sel] - first
            out = 0
            for ib, hb in enumerate(_hermites(sum(bra))):
                r = torch.stack([level[tuple(x + y for x, y in zip(hb, h))] for h in hk], -1)
                w = torch.einsum("pqh,qch->pqc", r, ek)
                part = torch.zeros((len(p), nk, ek.shape[1]), dtype=torch.float64, device=self.device)
                part = part.index_add(1, self.classes[ket]["pair"], w)
                out = out + torch.einsum("pf,pkc->pfkc", eb[:, :, ib], part)
            done = torch.zeros((last - first,) + tuple(out.shape[1:]), dtype=torch.float64, device=self.device)
            yield first, done.index_add(0, pair, out)
            first = last

    def _outputs(self, cls, first=0, count=None):
        """(i, j) AO indices of the contracted pairs' output functions."""
        na, nb = ((len(_components(l)) if self.cart else 2 * l + 1) for l in cls)
        ao = self.classes[cls]["ao"][first:None if count is None else first + count]
        i = ao[:, 0, None, None] + torch.arange(na, device=self.device)[None, :, None] + torch.zeros((1, 1, nb), dtype=torch.int64, device=self.device)
        j = ao[:, 1, None, None] + torch.arange(nb, device=self.device)[None, None, :] + torch.zeros((1, na, 1), dtype=torch.int64, device=self.device)
        return i.reshape(len(ao), -1), j.reshape(len(ao), -1)

    def pair_matrix(self):
        """(ij|kl) over packed pairs i >= j (i (i+1) / 2 + j), the whole symmetric matrix."""
        npair = self.n * (self.n + 1) // 2
        m = torch.zeros((npair, npair), dtype=torch.float64, device=self.device)

        def place(i, j):
            hi, lo = torch.maximum(i, j), torch.minimum(i, j)
            return hi * (hi + 1) // 2 + lo

        for bra in self.classes:
            for ket in self.classes:
                if ket > bra:
                    continue
                cols = place(*self._outputs(ket)).reshape(-1)
                for first, v in self.blocks(bra, ket):
                    rows = place(*self._outputs(bra, first, len(v))).reshape(-1)
                    v = v.reshape(len(rows), len(cols))
                    m[rows[:, None], cols[None]] = v
                    m[cols[:, None], rows[None]] = v.T
        return m

    def jk(self, dens, m=None):
        """J and K of (batch, n, n) densities."""
        m = self.pair_matrix() if m is None else m
        n = self.n
        i, j = torch.meshgrid(torch.arange(n, device=self.device), torch.arange(n, device=self.device), indexing="ij")
        pos = torch.maximum(i, j) * (torch.maximum(i, j) + 1) // 2 + torch.minimum(i, j)
        js, ks = torch.empty_like(dens), torch.empty_like(dens)
        for a in range(n):
            block = m[pos[a]][:, pos.reshape(-1)].reshape(n, n, n)    # (a j | k l)
            js[:, a] = torch.einsum("jkl,ekl->ej", block, dens)
            ks[:, a] = torch.einsum("jkl,ejl->ek", block, dens)
        return js, ks

    def contracted(self, dens, cj, ck, order):
        """d/dxyz of sum(cj J + ck K) (order 1), or the pieces of it that are still differentiable (order 2), block by block."""
        for bra in self.classes:
            for ket in self.classes:
                k, l = self._outputs(ket)
                k, l = k[None, None], l[None, None]
                for first, v in self.blocks(bra, ket, 1 << (22 if order == 1 else 20)):
                    i, j = self._outputs(bra, first, len(v))
                    i, j = i[:, :, None, None], j[:, :, None, None]
                    gamma = 0.0
                    for x, y in ((i, j), (j, i)):
                        for z, w in ((k, l), (l, k)):
                            gamma = gamma + cj[x, y] * dens[z, w] + cj[z, w] * dens[x, y] + ck[x, z] * dens[y, w] + ck[z, x] * dens[w, y]
                    deg = self.classes[bra]["deg"][first:first + len(v)][:, None, None, None] * self.classes[ket]["deg"][None, None, :, None]
                    yield (v * gamma * deg / 8.0).sum()


#: The largest basis whose integrals `exact` evaluates, per kind (its time stays well below 20 s).
_MOST = {"jk": 200, "graph": 200, "response": 200, "packed": 200, "eri": 150, "autograd": 116, "hvp": 40, "force": 0}


def exact(case, seed):
    kind = case["kind"]
    if case["basis"] == "cc-pvtz" and 58 * case["waters"] > 60:
        return None
    x = _inputs(case, seed)
    mol = x["mol"]
    if max(m["nao"] for m in x["mols"]) > _MOST[kind] or len(x["mols"]) > 1:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    atm, bas, env = mol["tables"]
    xyz = torch.as_tensor(np.stack([env[p:p + 3] for p in atm[:, 1]]), device=dev)

    def put(a):
        return torch.as_tensor(a, device=dev)

    if kind == "jk":
        j, k = _Exact(mol["tables"], case["cart"], xyz, dev).jk(put(x["d"])[None])
        return j[0], k[0]
    if kind == "graph":
        j, k = _Exact(mol["tables"], False, xyz, dev).jk(put(x["ds"][0])[None])
        return torch.stack([j, k]).reshape(2, 1, -1)
    if kind in ("response", "packed"):
        return _Exact(mol["tables"], case.get("cart", False), xyz, dev).jk(put(x["d"]))
    if kind == "eri":
        m = _Exact(mol["tables"], False, xyz, dev).pair_matrix()
        i, j = torch.tril_indices(len(m), len(m), device=dev)
        return m[i, j]
    d, cj, ck = put(x["d"]), put(x["cj"]), put(x["ck"])
    if kind == "autograd":
        ints = _Exact(mol["tables"], False, xyz, dev)
        m = ints.pair_matrix()
        j, k = ints.jk(d[None], m)
        gj, _ = ints.jk(cj[None], m)
        _, gk = ints.jk(ck[None], m)
        del m
        ints.xyz = xyz.clone().requires_grad_()
        for part in ints.contracted(d, cj, ck, 1):
            part.backward(retain_graph=True)     # the blocks of a class pair share the ket's coefficients
        g = ints.xyz.grad
        nuc = g[:len(atm) - len(bas)].index_add(0, put(mol["owner"]), g[len(atm) - len(bas):])
        return j[0], k[0], gj[0] + gk[0], nuc
    rows = xyz.clone().requires_grad_()
    u = put(np.stack([x["u"][p:p + 3] for p in atm[:, 1]]))
    ints = _Exact(mol["tables"], False, rows, dev)
    total = torch.zeros_like(rows)
    for part in ints.contracted(d, cj, ck, 2):
        (g,) = torch.autograd.grad(part, rows, create_graph=True)
        total = total + torch.autograd.grad((g * u).sum(), rows, retain_graph=True)[0]
    out = np.zeros(len(env))
    for p, v in zip(atm[:, 1], total.cpu().numpy()):
        out[p:p + 3] = v
    return out
