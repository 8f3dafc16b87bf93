"""The work whose speed is tracked: what users of this package have it do, through its public entry points.

Four calls carry the use of a ReaxFF calculator, and every case is one of them:

- ``evaluate``: one system, its energy, forces, charges and bonds (``Calculator.evaluate``), from a
  single molecule to a periodic box of tens of thousands of atoms, with fixed-charge or
  charge-response forces;
- ``batch``: the requests a serving worker takes together (``Calculator.evaluate_many``), of uneven
  sizes, some periodic, some charged;
- ``relax``: steps of a relaxation (``Calculator.relax``), each one a warm-started evaluation on the
  device's skin list;
- ``gradient``: energies, forces and force-field parameter gradients of many copies of a system, each
  with its own parameter set (``Calculator.parameter_gradient_many``), a step of a fit.

Systems are molecules at the densities and force fields of ``xreac_gb300.workloads``, on jittered
lattice sites with random orientations (quick to make at any size). ``exact`` evaluates the same
model in plain torch float64: dense QEq, every term over explicit lists, derivatives by autograd.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from xreac_gb300 import Calculator, ForceField
from xreac_gb300.differentiation import ParameterVector
from xreac_gb300.workloads import MOLECULES, anatase_slab_water

HO, CHO, TIO = "ffield.reax.HO.2015", "ffield.reax.CHO.2008", "ffield.reax.TiOH.Kim2013"
# Molecules of each force field's systems and the volume of one (A^3): liquid water; the C/H/O
# clusters of the request stream; the C/H/O gas-like mixture at 0.6 g/cm^3 in periodic boxes.
KINDS = {HO: ("H2O",), CHO: ("CH4", "O2", "H2O", "CO2")}
VOLUME = {(HO, False): 29.9, (HO, True): 29.9, (CHO, False): 35.0, (CHO, True): 67.0}
JITTER = 0.05          # A, Gaussian, on every atom
EXACT_ATOMS = 5000     # the dense reference solve stays within seconds up to here


def listed():
    return [
        # the smallest request: launches and host work only
        dict(name="molecule", call="evaluate", force_field=HO, molecules=1, periodic=False, response=False),
        # 64 H2O, the usual small cluster
        dict(name="cluster_192", call="evaluate", force_field=HO, molecules=64, periodic=False, response=False),
        # a C/H/O cluster near the top of the request sizes, with torsions and conjugation
        dict(name="cho_cluster_125", call="evaluate", force_field=CHO, molecules=125, periodic=False, response=False),
        # liquid water at 1 g/cm^3, 35.8 A cube
        dict(name="water_box_4608", call="evaluate", force_field=HO, molecules=1536, periodic=True, response=False),
        # periodic C/H/O mixture
        dict(name="cho_box_1000", call="evaluate", force_field=CHO, molecules=1000, periodic=True, response=False),
        # charge-response forces of an oxide slab under water: exact energy derivatives for a fit or a phonon run
        dict(name="slab_response", call="evaluate", force_field=TIO, molecules=32, periodic=True, response=True),
        # the largest single system
        dict(name="water_box_36864", call="evaluate", force_field=HO, molecules=12288, periodic=True, response=False),
        # a worker's batch of small requests
        dict(name="requests_small", call="batch", force_field=HO, systems=192, largest=64),
        # a worker's batch over the whole range of request sizes
        dict(name="requests_mixed", call="batch", force_field=CHO, systems=128, largest=512),
        # relaxation steps of a periodic system
        dict(name="relax_648", call="relax", force_field=HO, molecules=216, periodic=True, steps=10),
        # a fit's gradient step over perturbed oxide slabs
        dict(name="gradient_slabs", call="gradient", force_field=TIO, molecules=32, systems=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("cluster", "cluster", "box", "box", "response", "batch", "batch", "relax", "gradient"))
    ff = rng.choice((HO, CHO))
    if kind == "cluster":
        return dict(call="evaluate", force_field=ff, molecules=_log(rng, 1, 170), periodic=False, response=False)
    if kind == "box":
        return dict(call="evaluate", force_field=ff, molecules=_log(rng, 60, 12000), periodic=True, response=False)
    if kind == "response":
        if rng.random() < 0.5:
            return dict(call="evaluate", force_field=TIO, molecules=rng.randint(4, 40), periodic=True, response=True)
        return dict(call="evaluate", force_field=ff, molecules=_log(rng, 1, 300), periodic=False, response=True)
    if kind == "batch":
        return dict(call="batch", force_field=ff, systems=_log(rng, 8, 256), largest=_log(rng, 12, 512))
    if kind == "relax":
        return dict(call="relax", force_field=ff, molecules=_log(rng, 1, 1500), periodic=rng.random() < 0.5, steps=rng.randint(4, 12))
    return dict(call="gradient", force_field=TIO, molecules=rng.randint(8, 40), systems=_log(rng, 2, 32))


# ---------------------------------------------------------------------------------------- inputs
def _system(rng, ff, kinds, side=None):
    """(symbols, positions, cell or None) of the molecules ``kinds`` in a cube of their usual density,
    or in a periodic cube of ``side``: distinct random sites of a lattice, random shifts and orientations."""
    count = len(kinds)
    periodic = side is not None
    length = side or (count * VOLUME[ff, False]) ** (1 / 3)
    sites = max(math.ceil(count ** (1 / 3) - 1e-9), int(length / 3.3))
    length = max(length, 2.95 * sites)  # heavy atoms stay 2.4 A apart
    step = length / sites
    pick = np.sort(rng.choice(sites**3, count, replace=False))
    centres = np.stack((pick // sites**2, pick // sites % sites, pick % sites), axis=1) * step
    centres += rng.uniform(-0.08, 0.08, (count, 3)) * step
    quat = rng.normal(size=(count, 4))
    w, x, y, z = (quat / np.linalg.norm(quat, axis=1, keepdims=True)).T
    turn = np.stack((1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)), axis=1).reshape(-1, 3, 3)
    shapes = {k: MOLECULES[k]() for k in set(kinds)}
    symbols, xyz = [], []
    for k, c, t in zip(kinds, centres, turn):
        s, local = shapes[k]
        symbols.extend(s)
        xyz.append(local @ t.T + c)
    xyz = np.concatenate(xyz)
    xyz += rng.normal(0.0, JITTER, xyz.shape)
    return symbols, xyz, np.diag([length] * 3) if periodic else None


def _kinds(rng, ff, count):
    # with water in every system no charges vanish by symmetry (an O2 alone has none)
    return ["H2O"] + [KINDS[ff][k] for k in rng.integers(len(KINDS[ff]), size=count - 1)]


def _slab(case, seed):
    s = anatase_slab_water(n_water=case["molecules"], seed=seed, displacement=JITTER)
    return s.symbols, s.positions, s.cell


def _systems(case, seed):
    """The case's systems as keyword dicts of ``Calculator.evaluate``: compositions and sizes belong to the
    case, positions, shapes of the cells and orientations to the seed."""
    rng = np.random.default_rng(seed)
    ff = case["force_field"]
    of_case = np.random.default_rng([case.get(k, 0) for k in ("molecules", "systems", "largest", "steps")])
    if ff == TIO:
        made = [(*_slab(case, seed * 1000 + k), 0.0) for k in range(case.get("systems", 1))]
    elif case["call"] == "batch":
        made = []
        for _ in range(case["systems"]):
            atoms = math.exp(of_case.uniform(math.log(3), math.log(case["largest"])))
            kinds = _kinds(of_case, ff, max(1, round(atoms / (3.0 if ff == HO else 3.25))))
            # one request in ten is a periodic cell of 20 to 30 A, one in a hundred an ion
            side = rng.uniform(20.0, 30.0) if of_case.random() < 0.1 else None
            charge = float(of_case.choice((-1.0, 1.0))) if of_case.random() < 0.01 else 0.0
            made.append((*_system(rng, ff, kinds, side), charge))
    else:
        count = case["molecules"]
        # a cell is wider than the cutoff (10 A), and in the smaller ones an atom sees several images of another
        side = max(10.5, (count * VOLUME[ff, True]) ** (1 / 3)) if case["periodic"] else None
        made = [(*_system(rng, ff, _kinds(of_case, ff, count), side), 0.0)]
    return [dict(symbols=s, positions=x, cell=c, pbc=c is not None, total_charge=q) for s, x, c, q in made]


def _parameter_sets(case, seed):
    """One variant of the force field for each system: +-2 % on bond, vdW and angle parameters."""
    rng = np.random.default_rng(seed + 77)
    out = []
    for _ in range(case["systems"]):
        ff = ForceField.bundled(case["force_field"])
        for p in {id(p): p for p in ff.pairs.values()}.values():
            for name in ("De_s", "De_p", "p_be1", "p_bo1", "p_bo2", "D", "alpha", "r_vdW"):
                p[name] *= 1 + rng.uniform(-0.02, 0.02)
        for rec in {id(r): r for records in ff.angles.values() for r in records}.values():
            rec *= 1 + rng.uniform(-0.02, 0.02, rec.shape)
        out.append(ff)
    return out


@functools.lru_cache(maxsize=None)
def _calculator(name, use):
    """A program keeps one calculator per force field (a fit, which loads parameter sets, its own)."""
    return Calculator(ForceField.bundled(name))


def prepare(case, seed):
    systems = _systems(case, seed)
    fit = case["call"] == "gradient"
    state = dict(case=case, systems=systems, calc=_calculator(case["force_field"], "fit" if fit else "evaluate"))
    if fit:
        base = state["calc"].force_field
        state["vector"] = ParameterVector(base)
        state["base"] = base.tables()
        state["thetas"] = np.stack([state["vector"].values(ff) for ff in _parameter_sets(case, seed)])
        state["sets"] = np.arange(1, len(systems) + 1, dtype=np.int32)
    return state


# --------------------------------------------------------------------------------------- one pass
def _result(ev):
    return dict(energy=ev.energy, components=np.array(list(ev.components.values())), forces=ev.forces, charges=ev.charges,
                total_bond_orders=ev.total_bond_orders, lone_pairs=ev.lone_pairs, bond_counts=ev.bond_counts, dipole=ev.dipole)


def _batch_result(evs):
    cat = np.concatenate
    return dict(energy=np.array([e.energy for e in evs]), components=np.array([list(e.components.values()) for e in evs]),
                forces=cat([e.forces for e in evs]), charges=cat([e.charges for e in evs]),
                total_bond_orders=cat([e.total_bond_orders for e in evs]), dipole=np.array([e.dipole for e in evs]))


def run(state):
    case, systems, calc = state["case"], state["systems"], state["calc"]
    if case["call"] == "evaluate":
        return _result(calc.evaluate(**systems[0], full_derivative=case["response"]))
    if case["call"] == "batch":
        return _batch_result(calc.evaluate_many(systems))
    if case["call"] == "relax":
        done = calc.relax(**systems[0], max_iterations=case["steps"], force_tolerance=1e-6, backend="native")
        return dict(positions=done.positions, iterations=done.iterations, **_result(done.evaluation))
    # a fit's step: this step's parameters, then energies, forces and gradients of every copy
    vector = state["vector"]
    pair, angle = vector.tables(state["base"], state["thetas"])
    calc.load_parameter_tables(pair=pair, angle=angle, count=len(systems))
    evs, pair, angle = calc.parameter_gradient_many(systems, parameter_sets=state["sets"], raw=True)
    return dict(gradient=vector.gradient_rows(pair, angle), **_batch_result(evs))


# ------------------------------------------------------------------------------------------- work
def work(case):
    """Bytes: every position, type and result once. Operations (FP64): about 120 per pair of atoms within
    10 A (shield, taper, vdW, their derivatives and the force), 30 products of the QEq matrix per solve,
    and 4,000 per atom for the bonded terms and their adjoints."""
    systems = _systems(case, 1)
    flops = atoms = 0.0
    for s in systems:
        n = len(s["symbols"])
        volume = s["cell"][0, 0] * s["cell"][1, 1] * s["cell"][2, 2] if s["cell"] is not None else 10.0 * n
        near = n / volume * 4.19e3
        near = near if s["cell"] is not None else min(n - 1.0, near)
        solves = 2 if case.get("response") else 1
        flops += n * near / 2 * (120 + solves * 30 * 4) + 4000 * n
        atoms += n
    passes = case.get("steps", 0) + 1
    return {"bytes": passes * atoms * (28 + 72), "flops": passes * flops}


# ------------------------------------------------------------------------------------------ exact
_ATOM = ("r_s r_pi r_pi_pi valency valency_e valency_boc valency_val mass chi eta p_lp2 p_ovun2 p_ovun5 p_val3 p_val5 "
         "p_hbond").split()
_PAIR = ("De_s De_p De_pp p_be1 p_be2 p_bo1 p_bo2 p_bo3 p_bo4 p_bo5 p_bo6 p_ovun1 ovc v13cor r_s r_p r_pp p_boc3 p_boc4 "
         "p_boc5 D alpha gamma_w r_vdW gamma").split()


def _images(x, cell, cutoff, dev):
    """Half list of one system: (i, j, integer shift, vector) of every image pair within the cutoff once."""
    n = len(x)
    xt = torch.tensor(x, device=dev)
    m = torch.tensor(cell if cell is not None else np.eye(3), device=dev)
    shifts = torch.zeros((1, 3), dtype=torch.float64, device=dev)
    if cell is not None:
        height = 1.0 / np.linalg.norm(np.linalg.inv(cell), axis=0)
        reach = [0 if h > 2 * cutoff * (1 + 1e-9) else int(cutoff / h) + 1 for h in height]
        axes = [torch.arange(-r, r + 1, dtype=torch.float64, device=dev) for r in reach]
        shifts = torch.cartesian_prod(*axes).reshape(-1, 3)
        inv = torch.linalg.inv(m)
    found = []
    rows = max(1, 20_000_000 // (n * len(shifts)))
    for a in range(0, n, rows):
        d = xt[None] - xt[a:a + rows, None]
        base = -torch.round(d @ inv) if cell is not None else torch.zeros_like(d)
        s = base[:, :, None] + shifts
        v = d[:, :, None] + s @ m
        i, j, k = torch.nonzero((v * v).sum(-1) <= cutoff * cutoff, as_tuple=True)
        sk = s[i, j, k]
        gi = i + a
        first = torch.where(sk[:, 0] != 0, sk[:, 0], torch.where(sk[:, 1] != 0, sk[:, 1], sk[:, 2]))
        half = (gi < j) | ((gi == j) & (first < 0))
        found.append((gi[half], j[half], sk[half]))
    i, j, s = (torch.cat(c) for c in zip(*found))
    return i, j, s, s @ m


def _power(x, p):
    return torch.where(x > 0, torch.where(x > 0, x, 1.0) ** p, 0.0)


class _FixedAngle(torch.autograd.Function):
    """arccos whose derivative is -1 / max(sin, 1e-5): the fixed-charge forces' rule near 180 degrees."""

    @staticmethod
    def forward(ctx, c):
        theta = torch.arccos(torch.clamp(c, -1.0, 1.0))
        ctx.save_for_backward(theta)
        return theta

    @staticmethod
    def backward(ctx, g):
        return -g / torch.clamp(torch.sin(ctx.saved_tensors[0]), min=1e-5)


def _pairs_of(first, count):
    """All (a, b), a < b, of positions in consecutive runs that start at ``first`` with ``count`` entries."""
    a, b = [], []
    for c in np.unique(count[count > 1]):
        p, q = np.triu_indices(c, 1)
        f = first[count == c][:, None]
        a.append((f + p).ravel())
        b.append((f + q).ravel())
    empty = np.zeros(0, dtype=np.int64)
    return (np.concatenate(a), np.concatenate(b)) if a else (empty, empty)


def _product(first_a, count_a, first_b, count_b):
    """All (k, a, b): for every k, a entry of run A and an entry of run B."""
    total = count_a * count_b
    k = np.repeat(np.arange(len(total)), total)
    at = np.arange(total.sum()) - np.repeat(np.cumsum(total) - total, total)
    nb = np.maximum(count_b[k], 1)
    return k, first_a[k] + at // nb, first_b[k] + at % nb


def _model(ff, systems, response, gradient=False):
    """Every output of the given systems with force field ``ff``, as one concatenated set of lists."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t64 = functools.partial(torch.as_tensor, dtype=torch.float64, device=dev)
    g = [float(v) for v in ff.general]
    rc = g[12]
    tab = ff.tables()
    T = tab["ntypes"]
    from_name = {s: k for k, s in enumerate(ff.elements)}
    size = np.array([len(s["symbols"]) for s in systems])
    start = np.concatenate(([0], np.cumsum(size)))
    n, S = int(start[-1]), len(systems)
    sysn = torch.as_tensor(np.repeat(np.arange(S), size), device=dev)
    types = np.array([from_name[a] for s in systems for a in s["symbols"]])
    tt = torch.as_tensor(types, device=dev)
    atoms = {c: t64([float(ff.atoms[s][c]) for s in ff.elements])[tt] for c in _ATOM}
    x = t64(np.concatenate([s["positions"] for s in systems])).requires_grad_(True)
    parts = [_images(np.asarray(s["positions"]), s["cell"], rc, dev) for s in systems]
    I = torch.cat([p[0] + int(o) for p, o in zip(parts, start)])
    J = torch.cat([p[1] + int(o) for p, o in zip(parts, start)])
    shift, offset = torch.cat([p[2] for p in parts]), torch.cat([p[3] for p in parts])
    types_of_pair = tt[I] * T + tt[J]
    table = t64([[float(ff.pairs[s, u][c]) for c in _PAIR] for s in ff.elements for u in ff.elements])
    table.requires_grad_(gradient)
    pair = lambda c, sel=slice(None): table[types_of_pair[sel], _PAIR.index(c)]  # noqa: E731
    vec = x[J] - x[I] + offset
    r = torch.sqrt((vec * vec).sum(1))
    E = {}
    add = lambda value, of: torch.zeros(S, dtype=torch.float64, device=dev).index_add(0, of, value)  # noqa: E731
    ps = sysn[I]

    # nonbonded: taper, shielded Coulomb with QEq charges, shielded vdW (all bundled force fields' kind)
    u = r / rc
    taper = torch.where(r < rc, 1 + u**4 * (-35 + u * (84 + u * (-70 + 20 * u))), 0.0)
    shield = taper / (r**3 + pair("gamma")) ** (1 / 3)
    qs = []
    sh = shield if response else shield.detach()
    for k, s in enumerate(systems):
        mine = ps == k
        a, b, m = I[mine] - int(start[k]), J[mine] - int(start[k]), int(size[k])
        h = torch.zeros(m * m, dtype=torch.float64, device=dev)
        h = h.index_add(0, a * m + b, 14.4 * sh[mine]).index_add(0, b * m + a, 14.4 * sh[mine]).reshape(m, m)
        kkt = torch.ones((m + 1, m + 1), dtype=torch.float64, device=dev)
        kkt[m, m] = 0.0
        own = slice(int(start[k]), int(start[k + 1]))
        kkt[:m, :m] = h + torch.diag(atoms["eta"][own])
        rhs = torch.cat((-atoms["chi"][own], t64([float(s["total_charge"])])))
        qs.append(torch.linalg.solve(kkt, rhs)[:m])
    q = torch.cat(qs)
    E["coulomb"] = add(332.06371 * q[I] * q[J] * shield, ps)
    E["qeq"] = add(23.02 * (atoms["chi"] * q + 0.5 * atoms["eta"] * q * q), sysn)
    f13 = (r ** g[28] + (1 / pair("gamma_w")) ** g[28]) ** (1 / g[28])
    ev = torch.exp(0.5 * pair("alpha") * (1 - f13 / pair("r_vdW")))
    E["vdw"] = add(taper * pair("D") * (ev * ev - 2 * ev), ps)

    # bond orders of the pairs within 5 A, then their corrections
    near = torch.nonzero(r <= min(5.0, rc))[:, 0]
    i, j, rn = I[near], J[near], r[near]
    cut = 0.01 * g[29]

    def order(radius, pr, p1, p2):
        ok = (atoms[radius][i] > 0) & (atoms[radius][j] > 0)
        return torch.where(ok, torch.exp(pair(p1, near) * (rn / torch.where(ok, pair(pr, near), 1.0)) ** pair(p2, near)), 0.0)

    sig = (1 + cut) * order("r_s", "r_s", "p_bo1", "p_bo2")
    pi, pp = order("r_pi", "r_p", "p_bo3", "p_bo4"), order("r_pi_pi", "r_pp", "p_bo5", "p_bo6")
    on = torch.nonzero(sig + pi + pp >= cut)[:, 0]
    sel, i, j, pi, pp = near[on], i[on], j[on], pi[on], pp[on]
    bo = sig[on] + pi + pp - cut
    ends = torch.cat((i, j))
    gather = lambda v: torch.zeros(n, dtype=torch.float64, device=dev).index_add(0, ends, torch.cat((v, v)))  # noqa: E731
    raw = gather(bo)
    d, db = raw - atoms["valency"], raw - atoms["valency_val"]
    strong, angular = pair("ovc", sel) >= 0.001, pair("v13cor", sel) >= 0.001
    f2 = torch.exp(-g[0] * d[i]) + torch.exp(-g[0] * d[j])
    f3 = -torch.log(0.5 * (torch.exp(-g[1] * d[i]) + torch.exp(-g[1] * d[j]))) / g[1]
    vi, vj = atoms["valency"][i], atoms["valency"][j]
    f1 = torch.where(strong, 0.5 * ((vi + f2) / (vi + f2 + f3) + (vj + f2) / (vj + f2 + f3)), 1.0)
    b3, b4, b5 = (torch.where(strong | angular, torch.nan_to_num(pair(c, sel)), 0.0) for c in ("p_boc3", "p_boc4", "p_boc5"))
    f45 = 1.0
    for a in (i, j):
        f45 = f45 / (1 + torch.exp(-(b4 * bo * bo - db[a]) * b3 + b5))
    corr = f1 * torch.where(angular, f45, 1.0)
    bo, pi, pp = bo * corr, pi * corr * f1, pp * corr * f1
    sigma = bo - pi - pp
    bo, sigma, pi, pp = (torch.where(v >= 1e-10, v, 0.0) for v in (bo, sigma, pi, pp))

    # per-atom sums and the terms of one bond or one atom
    total = gather(bo)
    d, db, de = (total - atoms[c] for c in ("valency", "valency_boc", "valency_e"))
    whole = torch.trunc(de.detach() / 2)
    odd = de - 2 * whole
    nlp = torch.exp(-g[15] * (2 + odd) ** 2) - whole
    dlp = 0.5 * (atoms["valency_e"] - atoms["valency"]) - nlp
    light = (atoms["mass"] <= 21).double()
    dlpt = dlp * light
    bs = sysn[i]
    bond = -(pair("De_s", sel) * sigma * torch.exp(pair("p_be1", sel) * (1 - _power(sigma, pair("p_be2", sel))))
             + pair("De_p", sel) * pi + pair("De_pp", sel) * pp)
    mass_i, mass_j = atoms["mass"][i], atoms["mass"][j]
    stab = g[10] * torch.exp(-g[7] * (bo - 2.5) ** 2) / (1 + 25 * torch.exp(g[4] * (d[i] + d[j]))) \
        * (torch.exp(-g[3] * (total[i] - bo)) + torch.exp(-g[3] * (total[j] - bo)))
    triple = (bo >= 1.0) & (((mass_i == 12.0) & (mass_j == 15.999)) | ((mass_j == 12.0) & (mass_i == 15.999)) | (int(g[37]) == 2))
    E["bond"] = add(bond + torch.where(triple, stab, 0.0), bs)
    E["lone_pair"] = add(atoms["p_lp2"] * dlp / (1 + torch.exp(-75 * dlp)), sysn)
    if g[5] > 0.001:
        carbon = t64([s.upper() == "C" for s in ff.elements]).bool()[tt]
        for a in (i, j):
            over = bo - d[a] - 0.040 * d[a] ** 4
            E["lone_pair"] = E["lone_pair"] + add(torch.where(carbon[i] & carbon[j] & (over > 3), g[5] * (over - 3) ** 2, 0.0), bs)
    ov1 = gather(pair("p_ovun1", sel) * pair("De_s", sel) * bo)
    other = torch.cat((j, i))
    ov2 = torch.zeros(n, dtype=torch.float64, device=dev).index_add(
        0, ends, (d[other] - light[ends] * dlpt[other]) * torch.cat((pi + pp, pi + pp)))
    dc = d - light * dlpt / (1 + g[32] * torch.exp(g[31] * ov2))
    E["atom"] = add(ov1 * dc / (dc + atoms["valency"] + 1e-8) / (1 + torch.exp(atoms["p_ovun2"] * dc))
                    - atoms["p_ovun5"] * (1 - torch.exp(g[6] * dc)) / (1 + torch.exp(-atoms["p_ovun2"] * dc))
                    / (1 + g[8] * torch.exp(g[9] * ov2)), sysn)

    # directed entries of the bonds above the three-body cut, row by row
    host = lambda v: v.detach().cpu().numpy()  # noqa: E731
    si = np.rint(host(shift[sel])).astype(np.int64)
    hi, hj, hb = host(i), host(j), host(bo)
    src, dst = np.concatenate((hi, hj)), np.concatenate((hj, hi))
    img, sign = np.concatenate((si, -si)), np.repeat((1, -1), len(hi))
    ident = np.tile(np.arange(len(hi)), 2)
    order_ = np.lexsort((img[:, 2], img[:, 1], img[:, 0], dst, src))
    order_ = order_[hb[ident[order_]] > 0.001]
    src, dst, img, sign, ident = src[order_], dst[order_], img[order_], sign[order_], ident[order_]
    count = np.bincount(src, minlength=n)
    first = np.concatenate(([0], np.cumsum(count)[:-1]))
    dev_i = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=dev)  # noqa: E731
    vb, rb = vec[sel], r[sel]
    entry_vec = vb[dev_i(ident)] * t64(sign)[:, None]

    # valence angles, penalty, three-body conjugation
    left, right = _pairs_of(first, count)
    keep = hb[ident[left]] * hb[ident[right]] > 1e-5
    left, right = left[keep], right[keep]
    rows, many = tab["angle_index"][(types[dst[left]] * T + types[src[left]]) * T + types[dst[right]]].T
    rep = np.repeat(np.arange(len(left)), many)
    rec = rows[rep] + np.arange(len(rep)) - np.repeat(np.cumsum(many) - many, many)
    keep = np.abs(tab["angle"][rec, 1]) > 0.001
    left, right, rec = left[rep][keep], right[rep][keep], rec[keep]
    angle_table = t64(tab["angle"]).requires_grad_(gradient)
    theta00, v1, v2, coa1, v7, pen1, v4 = angle_table[dev_i(rec)].unbind(1)
    lb, rb_, c = dev_i(ident[left]), dev_i(ident[right]), dev_i(src[left])
    la, ra = dev_i(dst[left]), dev_i(dst[right])
    cos = (entry_vec[dev_i(left)] * entry_vec[dev_i(right)]).sum(1) / (rb[lb] * rb[rb_])
    theta = torch.arccos(torch.clamp(cos, -1 + 1e-14, 1 - 1e-14)) if response else _FixedAngle.apply(cos)
    sbo = gather(pi + pp) + (1 - torch.exp(-gather(bo**8))) * (-db - g[33] * torch.where(odd >= 0, 0.0, nlp))
    sbo2 = torch.where(sbo <= 0, 0.0, torch.where(sbo <= 1, _power(sbo, g[16]), torch.where(sbo < 2, 2 - _power(2 - sbo, g[16]), 2.0)))
    theta0 = (180 - theta00 * (1 - torch.exp(-g[17] * (2 - sbo2[c])))) * (3.14159265 / 180)
    bl, br = bo[lb] - 0.001, bo[rb_] - 0.001
    f7 = (1 - torch.exp(-atoms["p_val3"][c] * bl**v4)) * (1 - torch.exp(-atoms["p_val3"][c] * br**v4))
    e6, pv5 = torch.exp(g[14] * db[c]), atoms["p_val5"][c]
    f8 = pv5 - (pv5 - 1) * (2 + e6) / (1 + e6 + torch.exp(-v7 * db[c]))
    bend = torch.exp(-v2 * (theta0 - theta) ** 2)
    E["angle"] = add(f7 * f8 * v1 * torch.where(v1 >= 0, 1 - bend, -bend), sysn[c])
    e3, e4 = torch.exp(-g[20] * d[c]), torch.exp(g[21] * d[c])
    E["penalty"] = add(pen1 * (2 + e3) / (1 + e3 + e4) * torch.exp(-g[19] * ((bl - 2) ** 2 + (br - 2) ** 2)), sysn[c])
    E["angle_conjugation"] = add(
        coa1 / (1 + torch.exp(g[2] * (total[c] - atoms["valency_val"][c])))
        * torch.exp(-g[38] * ((total[la] - bl) ** 2 + (total[ra] - br) ** 2))
        * torch.exp(-g[30] * ((bl - 1.5) ** 2 + (br - 1.5) ** 2)), sysn[c])

    # torsions and four-body conjugation about every bond
    mid = np.nonzero(sign > 0)[0]
    k, left, right = _product(first[src[mid]], count[src[mid]], first[dst[mid]], count[dst[mid]])
    mid = mid[k]
    row = tab["torsion_index"][((types[dst[left]] * T + types[src[mid]]) * T + types[dst[mid]]) * T + types[dst[right]]]
    back = (ident[right] == ident[mid]) & (sign[right] < 0)
    ring = (dst[left] == dst[right]) & np.all(img[left] == img[mid] + img[right], axis=1)
    keep = (left != mid) & ~back & ~ring & (row >= 0) & (hb[ident[left]] * hb[ident[mid]] * hb[ident[right]] > 0.001)
    left, mid, right, row = left[keep], mid[keep], right[keep], row[keep]
    t1, t2, t3, tor1, cot1 = t64(tab["torsion"][row]).unbind(1)
    bl, bm, br = (dev_i(ident[v]) for v in (left, mid, right))
    a, b = dev_i(src[mid]), dev_i(dst[mid])
    va, vm, vc = (entry_vec[dev_i(v)] for v in (left, mid, right))
    n1, n2 = torch.linalg.cross(va, vm, dim=1), torch.linalg.cross(vc, vm, dim=1)
    area1, area2 = (n1 * n1).sum(1), (n2 * n2).sum(1)
    sines = torch.sqrt(area1 / (rb[bl] * rb[bm]) ** 2 * (area2 / (rb[bm] * rb[br]) ** 2))
    cw = (n1 * n2).sum(1) / torch.sqrt(area1 * area2)
    o1, o2, o3 = bo[bl] - 0.001, bo[bm] - 0.001, bo[br] - 0.001
    e3, e4 = torch.exp(-g[24] * (db[a] + db[b])), torch.exp(g[25] * (db[a] + db[b]))
    e1 = torch.exp(tor1 * (2 - pi[bm] - (2 + e3) / (1 + e3 + e4)) ** 2)
    f10 = (1 - torch.exp(-g[23] * o1)) * (1 - torch.exp(-g[23] * o2)) * (1 - torch.exp(-g[23] * o3))
    wave = 0.5 * (t1 * (1 + cw) + t2 * e1 * (2 - 2 * cw * cw) + t3 * (1 + 4 * cw**3 - 3 * cw))
    E["torsion"] = add(f10 * sines * wave, sysn[a])
    f12 = torch.exp(-g[27] * ((o1 - 1.5) ** 2 + (o2 - 1.5) ** 2 + (o3 - 1.5) ** 2))
    E["conjugation"] = add(cot1 * f12 * (1 + (cw * cw - 1) * sines), sysn[a])

    # hydrogen bonds: donors (bond order at least 0.01) and acceptors (within 7.5 A) of every hydrogen
    role = np.array([int(ff.atoms[s]["p_hbond"]) for s in ff.elements])[types]
    wide = torch.nonzero(r <= min(7.5, rc))[:, 0]
    place = torch.full((len(r),), -1, dtype=torch.int64, device=dev)
    place[sel] = torch.arange(len(sel), device=dev)
    wi, wj, wb = host(I[wide]), host(J[wide]), host(place[wide])
    src, dst = np.concatenate((wi, wj)), np.concatenate((wj, wi))
    pid, sign, bid = np.tile(host(wide), 2), np.repeat((1, -1), len(wi)), np.tile(wb, 2)
    keep = np.nonzero((role[src] == 1) & (role[dst] == 2))[0]
    keep = keep[np.argsort(src[keep], kind="stable")]
    src, dst, pid, sign, bid = src[keep], dst[keep], pid[keep], sign[keep], bid[keep]
    donor = np.nonzero((bid >= 0) & (np.append(hb, 0.0)[bid] >= 0.01))[0]
    count = np.bincount(src, minlength=n)
    first = np.concatenate(([0], np.cumsum(count)[:-1]))
    k, _, acc = _product(donor, np.ones(len(donor), dtype=np.int64), first[src[donor]], count[src[donor]])
    donor = donor[k]
    row = tab["hbond_index"][(types[dst[donor]] * T + types[src[donor]]) * T + types[dst[acc]]]
    keep = (donor != acc) & (row >= 0)
    donor, acc, row = donor[keep], acc[keep], row[keep]
    keep = tab["hbond"][row, 0] > 0
    donor, acc, row = donor[keep], acc[keep], row[keep]
    r0, h1, h2, h3 = t64(tab["hbond"][row]).unbind(1)
    pd, pa = dev_i(pid[donor]), dev_i(pid[acc])
    cos = (vec[pd] * vec[pa]).sum(1) * t64(sign[donor] * sign[acc]) / (r[pd] * r[pa])
    E["hydrogen_bond"] = add(h1 * (1 - torch.exp(-h2 * bo[dev_i(bid[donor])])) * torch.exp(-h3 * (r0 / r[pa] + r[pa] / r0 - 2))
                             * 0.25 * (1 - torch.clamp(cos, -1.0, 1.0)) ** 2, sysn[dev_i(src[donor])])

    names = ("bond atom lone_pair molecule angle penalty angle_conjugation hydrogen_bond torsion conjugation vdw coulomb "
             "electric_field qeq").split()
    comps = torch.stack([E.get(k, torch.zeros(S, dtype=torch.float64, device=dev)) for k in names], dim=1)
    wanted = [x] + ([table, angle_table] if gradient else [])
    grads = torch.autograd.grad(comps.sum(), wanted)
    mass, xd, qd = atoms["mass"], x.detach(), q.detach()
    centre = torch.stack([add(mass * xd[:, k], sysn) for k in range(3)], 1) / add(mass, sysn)[:, None]
    dipole = torch.stack([add((xd - centre[sysn])[:, k] * qd, sysn) for k in range(3)], 1)
    return dict(energy=host(comps.sum(1)), components=host(comps), forces=-host(grads[0]), charges=host(q),
                total_bond_orders=host(total), lone_pairs=host(nlp), dipole=host(dipole),
                bond_counts=np.bincount(np.concatenate((hi, hj)), weights=np.tile(hb > 0.3, 2), minlength=n).astype(np.int64),
                gradient=_by_record(ff, tab, host(grads[1]), host(grads[2])) if gradient else None)


# The pair parameters with a gradient, in their order within a record; the last three belong to another kind of vdW.
_GIVEN = ("De_s De_p De_pp p_be1 p_be2 p_ovun1 p_bo1 p_bo2 p_bo3 p_bo4 p_bo5 p_bo6 r_s r_p r_pp D alpha gamma_w r_vdW "
          "rcore ecore acore").split()


def _by_record(ff, tab, pair_rows, angle_rows):
    """Table rows' derivatives summed over the rows of each distinct record, pairs first, in the file's order."""
    names, T = {s: k for k, s in enumerate(ff.elements)}, tab["ntypes"]
    records = {}
    for (s, t), rec in ff.pairs.items():
        row = pair_rows[names[s] * T + names[t]]
        mine = np.array([row[_PAIR.index(c)] if c in _PAIR else 0.0 for c in _GIVEN if c in rec])
        records[id(rec)] = records.get(id(rec), 0.0) + mine
    at = 0
    for recs in ff.angles.values():
        for rec in recs:
            records[id(rec)] = records.get(id(rec), 0.0) + angle_rows[at]
            at += 1
    return np.concatenate(list(records.values()))


_BATCH = ("energy", "components", "forces", "charges", "total_bond_orders", "dipole")


def _one(ff, system, response):
    out = _model(ff, [system], response)
    del out["gradient"]
    return dict(out, energy=float(out["energy"][0]), components=out["components"][0], dipole=out["dipole"][0])


def _relaxed(ff, system, steps):
    """FIRE (Bitzek et al., Phys. Rev. Lett. 97, 170201, 2006) with unit masses, as ``Calculator.relax`` documents it."""
    x = np.array(system["positions"])
    v, dt, alpha, streak = np.zeros_like(x), 0.02, 0.1, 0
    for step in range(steps + 1):
        got = _one(ff, dict(system, positions=x), False)
        if step == steps:
            return dict(positions=x, iterations=steps, **got)
        f = got["forces"]
        if float((v * f).sum()) > 0:
            v = (1 - alpha) * v + alpha * np.linalg.norm(v) / np.linalg.norm(f) * f
            streak += 1
            if streak > 5:
                dt, alpha = min(dt * 1.1, 0.2), alpha * 0.99
        else:
            v, streak, alpha = np.zeros_like(x), 0, 0.1
            dt = dt * 0.5 if step else dt
        v = v + dt * f
        move = dt * v
        far = float(np.linalg.norm(move, axis=1).max())
        x = x + (move * (0.1 / far) if far > 0.1 else move)


def exact(case, seed):
    systems = _systems(case, seed)
    if sum(len(s["symbols"]) for s in systems) * (case.get("steps", 0) + 1) > (5 * EXACT_ATOMS if case["call"] != "evaluate" else EXACT_ATOMS):
        return None
    ff = ForceField.bundled(case["force_field"])  # the parameters as data
    if case["call"] == "evaluate":
        return _one(ff, systems[0], case["response"])
    if case["call"] == "batch":
        out = _model(ff, systems, False)
        return {k: out[k] for k in _BATCH}
    if case["call"] == "relax":
        return _relaxed(ff, systems[0], case["steps"])
    each = [_model(v, [s], False, gradient=True) for v, s in zip(_parameter_sets(case, seed), systems)]
    return dict({k: np.concatenate([e[k] for e in each]) for k in _BATCH}, gradient=np.stack([e["gradient"] for e in each]))
