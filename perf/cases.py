"""What a user of this framework has it do, as cases that can be timed: single energy routines called from a host
move loop (the drop-in use), the plain move loop, batches of isotherm points, and the request server.

Frameworks are seeded random rigid crystals at the density, type mix, charges and Lennard-Jones parameters of
`fastmc_b200.synth` (a unit cell replicated to a supercell, as real frameworks are), 400 to 6,000 atoms; guests are
CO2, N2 and CH4 at 273 to 348 K and 0.01 to 10 bar; the cut-off is 12.5 A and kmax follows a 0.9 1/A reciprocal cut-off
unless a case says otherwise.  All energies are 64-bit.
"""
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fastmc-1.4.0_b200"))
import fastmc_b200 as fm  # noqa: E402
from fastmc_b200 import synth  # noqa: E402

RCUT, ALPHA, RHO = 12.5, 0.26, 0.025
R4PIE0, KCAL = 138935.4835, 418.4
# a production run that no timing ever ends: production starts after EQ moves
EQ, STEPS = 500, 2000000000


def listed():
    return [
        # one trial of a host move loop in the smallest cell: an insertion's reciprocal and real-space energies
        {"name": "trial_insert_424", "kind": "trial", "move": "insert", "unit": 424, "edge": 25.832, "reps": 1,
         "skew": 0.0, "gas": "CO2", "guests": 5, "kmax": 8},
        # a displacement trial (old and new sites) in an odd-sized triclinic cell
        {"name": "trial_displace_triclinic", "kind": "trial", "move": "displace", "unit": 337, "edge": 0.0, "reps": 3,
         "skew": 0.17, "gas": "N2", "guests": 41, "kmax": 0},
        # an insertion and a deletion with their commits, in the 2x2x2 supercell with many guests and k-vectors
        {"name": "trial_exchange_3392", "kind": "trial", "move": "exchange", "unit": 424, "edge": 25.832, "reps": 8,
         "skew": 0.0, "gas": "CO2", "guests": 280, "kmax": 12},
        # S(k) of every atom from scratch: the drift check of a running simulation, ordinary and large
        {"name": "ewald1_1011", "kind": "ewald1", "unit": 337, "edge": 0.0, "reps": 3, "skew": 0.0, "gas": "CO2",
         "guests": 53, "kmax": 0},
        {"name": "ewald1_5928", "kind": "ewald1", "unit": 741, "edge": 0.0, "reps": 8, "skew": 0.0, "gas": "CO2",
         "guests": 410, "kmax": 12},
        # the full energy of a loaded framework: a restart or the first step of a run
        {"name": "single_point_3392", "kind": "single_point", "unit": 424, "edge": 25.832, "reps": 8, "skew": 0.0,
         "gas": "CO2", "guests": 280, "kmax": 12},
        # the plain move loop (one chain, moves on the host, energies on the GPU), small and large
        {"name": "run_424", "kind": "run", "unit": 424, "edge": 25.832, "reps": 1, "skew": 0.0, "gas": "CO2",
         "bar": 0.15, "kmax": 8, "moves": 200},
        {"name": "run_3392", "kind": "run", "unit": 424, "edge": 25.832, "reps": 8, "skew": 0.0, "gas": "CO2",
         "bar": 1.0, "kmax": 12, "moves": 200},
        # one isotherm: a framework at 16 pressures, one chain each
        {"name": "batch_isotherm_16", "kind": "batch", "frameworks": 1, "lo": 24.0, "hi": 34.0, "skew": 0.0,
         "gases": "CO2", "pressures": 16, "voxel_edge": 2.0, "moves": 1000},
        # the screening batch: 16 orthorhombic frameworks (edges 18 to 52 A) at 16 pressures each
        {"name": "batch_256", "kind": "batch", "frameworks": 16, "lo": 18.0, "hi": 52.0, "skew": 0.0,
         "gases": "CO2", "pressures": 16, "voxel_edge": 1.0, "moves": 2000},
        # a binary mixture in triclinic cells, more chains than fit one per SM
        {"name": "batch_mixture_triclinic", "kind": "batch", "frameworks": 6, "lo": 24.0, "hi": 40.0, "skew": 0.15,
         "gases": "CO2,N2", "pressures": 33, "voxel_edge": 2.0, "moves": 1000},
        # a burst of requests to a running server: unequal frameworks, gases, conditions and budgets
        {"name": "serve_60", "kind": "serve", "requests": 60, "frameworks": 10, "slots": 40, "lo": 400, "hi": 6000,
         "moves_lo": 500, "moves_hi": 4000, "step": 500},
    ]


def draw(rng):
    kind = rng.choice(["trial", "trial", "ewald1", "single_point", "run", "batch", "batch", "serve"])
    logu = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    if kind == "batch":
        nf, npress = rng.randint(1, 12), rng.randint(3, 21)
        lo = rng.uniform(18.0, 30.0)
        mix = rng.random() < 0.3
        return {"kind": kind, "frameworks": nf, "lo": lo, "hi": rng.uniform(lo + 2.0, 45.0),
                "skew": rng.choice([0.0, rng.uniform(0.05, 0.2)]), "gases": "CO2,N2" if mix else rng.choice(["CO2", "N2", "CH4"]),
                "pressures": npress, "voxel_edge": rng.choice([1.0, 1.5, 2.0]), "moves": int(logu(300, 2000))}
    if kind == "serve":
        lo = int(logu(400, 2000))
        nf = rng.randint(2, 9)
        return {"kind": kind, "requests": nf * rng.randint(2, 6), "frameworks": nf, "slots": rng.randint(8, 48),
                "lo": lo, "hi": rng.randint(lo, 5500), "moves_lo": 300, "moves_hi": rng.randint(500, 4000),
                "step": rng.choice([250, 500, 1000])}
    atoms = logu(400, 5900)
    reps = 1 if atoms < 600 else rng.choice([2, 3, 4, 8])
    unit = max(50, min(740, int(atoms / reps)))
    c = {"kind": kind, "unit": unit, "edge": 0.0, "reps": reps, "skew": rng.choice([0.0, rng.uniform(0.05, 0.2)]),
         "gas": rng.choice(["CO2", "N2", "CH4"]), "kmax": rng.choice([0, 0, 0, rng.randint(7, 11)])}
    if kind == "run":
        return dict(c, bar=logu(0.01, 10.0), moves=rng.randint(50, 200))
    if kind == "trial":
        c["move"] = rng.choice(["insert", "delete", "displace", "exchange"])
    return dict(c, guests=int(logu(2, 60 if atoms < 1500 else 300)))


# ------------------------------------------------------------------------------------ inputs
def _min_dist(points, others, cell):
    """Smallest periodic distance of each point to `others`."""
    if not len(others):
        return np.full(len(points), np.inf)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    h = torch.tensor(cell, device=dev)
    f = torch.tensor(np.linalg.solve(cell.T, points.T).T, device=dev)
    g = torch.tensor(np.linalg.solve(cell.T, others.T).T, device=dev)
    best = torch.empty(len(points), dtype=torch.float64, device=dev)
    for a in range(0, len(points), 512):
        d = f[a:a + 512, None, :] - g[None, :, :]
        d = (d - torch.round(d)) @ h
        best[a:a + 512] = (d * d).sum(-1).min(1).values
    return best.sqrt().cpu().numpy()


def _place(rng, cell, n, dmin):
    """n random positions with a periodic minimum separation."""
    pts, inv = np.zeros((n, 3)), np.linalg.inv(cell)
    count = 0
    while count < n:
        for p in rng.uniform(0.0, 1.0, (256, 3)) @ cell:
            d = (pts[:count] - p) @ inv
            d = (d - np.round(d)) @ cell
            if not count or np.min(np.einsum("ij,ij->i", d, d)) >= dmin * dmin:
                pts[count] = p
                count += 1
                if count == n:
                    break
    return pts


REPS = {1: (1, 1, 1), 2: (1, 1, 2), 3: (1, 1, 3), 4: (1, 2, 2), 8: (2, 2, 2)}


def _cell(lengths, skew):
    """Cell rows a, b, c: orthorhombic, or sheared by `skew` times the edges."""
    a, b, c = (float(v) for v in lengths)
    return np.array([[a, 0.0, 0.0], [skew * a, b, 0.0], [-skew * a, skew * b, c]]) if skew else np.diag([a, b, c])


def _framework(rng, cell, natoms, reps):
    """A rigid random crystal: `natoms` atoms in the unit cell, replicated; numbers as the decks print them."""
    counts = [int(round(f * natoms)) for _, _, f in synth.FRAMEWORK_TYPES]
    counts[2] += natoms - sum(counts)
    names = [t for (t, _, _), c in zip(synth.FRAMEWORK_TYPES, counts) for _ in range(c)]
    xyz = _place(rng, cell, natoms, 1.8)
    q = rng.normal(0.0, 0.4, natoms)
    q = np.round(q - q.mean(), 10)
    lj = {t: (float(rng.uniform(0.02, 0.3)), float(rng.uniform(2.5, 3.8))) for t, _, _ in synth.FRAMEWORK_TYPES}
    fw = synth.Framework(np.round(cell, 12), names, xyz, q, lj).replicate(*reps)
    fw.xyz = np.round(fw.xyz, 12)
    return fw


def _kmax(fw, kmax):
    return (kmax,) * 3 if kmax else tuple(synth.kmax_for(float(np.linalg.norm(r))) for r in fw.cell)


def _single(case, seed):
    """The framework of a one-chain case: (framework, kmax, rng)."""
    rng = np.random.default_rng([seed, case["unit"], case["reps"]])
    reps = REPS[case["reps"]]
    edge = case["edge"]
    if edge:  # cubic supercell
        L = np.full(3, edge)
    else:  # a supercell near 1 : 1.1 : 1.2 whose edges exceed twice the cut-off
        V = case["unit"] * case["reps"] / RHO
        s = (V / 1.32) ** (1.0 / 3.0)
        L = np.maximum(np.array([s, 1.1 * s, 1.2 * s]), 2.0 * RCUT + 0.8 + 6.0 * case["skew"]) / np.array(reps)
    fw = _framework(rng, _cell(L, case["skew"]), case["unit"], reps)
    return fw, _kmax(fw, case["kmax"]), rng


def _molecules(rng, fw, gas, n):
    """n molecules in the framework's voids, clear of the atoms and of one another."""
    site = np.array([s[3:6] for s in synth.GASES[gas][1]])
    out = np.zeros((0, len(site), 3))
    for clear, apart in ((2.0, 2.6), (1.6, 2.2), (1.2, 1.8)):
        for _ in range(4):
            if len(out) >= n:
                break
            m = 6000 if n > 60 else 1500
            com = rng.uniform(0.0, 1.0, (m, 3)) @ fw.cell
            u = rng.normal(size=(m, 3))
            u /= np.linalg.norm(u, axis=1)[:, None]
            mols = com[:, None, :] + site[None, :, :1] * u[:, None, :]
            ok = (_min_dist(mols.reshape(-1, 3), fw.xyz, fw.cell).reshape(m, -1) > clear).all(1)
            inv = np.linalg.inv(fw.cell)
            for x in mols[ok]:
                d = (out.reshape(-1, 1, 3) - x[None]) @ inv
                d = (d - np.round(d)) @ fw.cell
                if not len(out) or np.min((d * d).sum(-1)) > apart * apart:
                    out = np.concatenate([out, x[None]])
                    if len(out) >= n:
                        break
    if len(out) < n:
        raise RuntimeError("could not place the guests")
    return out[:n]


def _loaded(case, seed):
    """Framework, kmax, the guests present, a molecule beside them and a displaced copy of one."""
    fw, kmax, rng = _single(case, seed)
    mols = _molecules(rng, fw, case["gas"], case["guests"] + 1)
    moved = mols[case["guests"] // 2] + rng.uniform(-0.3, 0.3, 3)
    return fw, kmax, mols[:-1], mols[-1], moved


def _one_chain(case, seed):
    tmp = tempfile.TemporaryDirectory()
    fw, kmax, guests, new, moved = _loaded(case, seed)
    d = synth.write_inputs(os.path.join(tmp.name, "deck"), fw, [case["gas"]], [1.0], 298.0, kmax, eq_cycles=EQ,
                           prod_cycles=STEPS)
    ch = fm.Chain(d, seed=(12, 34, 56, 1 + seed % 168))
    ch.set_guests(0, guests)
    return {"kind": case["kind"], "tmp": tmp, "chain": ch, "guests": guests, "new": new, "moved": moved,
            "move": case.get("move"), "mol": len(guests) // 2}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("trial", "ewald1", "single_point"):
        return _one_chain(case, seed)
    tmp = tempfile.TemporaryDirectory()
    if kind == "run":
        fw, kmax, _ = _single(case, seed)
        d = synth.write_inputs(os.path.join(tmp.name, "deck"), fw, [case["gas"]], [case["bar"]], 298.0, kmax,
                               eq_cycles=EQ, prod_cycles=STEPS)
        ch = fm.Chain(d, seed=(12, 34, 56, 1 + seed % 168))
        ch.run(4000, trace=False)  # into production, with guests present
        return {"kind": kind, "tmp": tmp, "chain": ch, "moves": case["moves"]}
    rng = np.random.default_rng([seed, case["frameworks"]])
    if kind == "batch":
        gases = case["gases"].split(",")
        dirs, seeds = [], []
        for f in range(case["frameworks"]):
            L = rng.uniform(case["lo"], case["hi"], 3)
            L[0] += 6.0 * case["skew"] * (L[0] < 2.0 * RCUT + 6.0)
            cell = _cell(L, case["skew"])
            reps = [max(1, int(math.ceil((2.0 * RCUT + 0.1) / w))) for w in _widths(cell)]
            fw = _framework(rng, cell, max(8, int(round(RHO * L.prod()))), reps)
            for p, bar in enumerate(np.logspace(-2, 1, case["pressures"])):
                part = [0.15 * bar, 0.85 * bar] if len(gases) == 2 else [bar]
                dirs.append(_deck(tmp.name, f, p, fw, gases, part, 298.0))
                seeds.append((12, 34, 56, (1 + seed + 7 * len(seeds)) % 169))
        b = fm.Batch(dirs, seeds, voxel_edge=case["voxel_edge"])
        b.run(10000)  # into production, near the loading of each pressure
        return {"kind": kind, "tmp": tmp, "batch": b, "moves": case["moves"]}
    fws = []
    for f in range(case["frameworks"]):
        atoms = rng.integers(case["lo"], case["hi"] + 1)
        reps = 1 if atoms < 740 else 8
        edge = max((atoms / RHO) ** (1.0 / 3.0), 25.2) / REPS[reps][0]
        fws.append(_framework(rng, _cell((edge,) * 3, 0.0), int(atoms / reps), REPS[reps]))
    jobs = []
    for i in range(case["requests"]):
        f = i % case["frameworks"]
        gas = ("CO2", "N2", "CH4")[int(rng.integers(0, 3))]
        d = _deck(tmp.name, f, i, fws[f], [gas], [float(10 ** rng.uniform(-2, 1))], float(rng.uniform(273.0, 348.0)))
        moves = int(math.exp(rng.uniform(math.log(case["moves_lo"]), math.log(case["moves_hi"]))))
        jobs.append((d, (12, 34, 56, (1 + seed + 7 * i) % 169), moves))
    return {"kind": kind, "tmp": tmp, "server": fm.Server(slots=case["slots"]), "jobs": jobs, "step": case["step"]}


def _widths(cell):
    v = abs(np.linalg.det(cell))
    return [v / np.linalg.norm(np.cross(cell[(i + 1) % 3], cell[(i + 2) % 3])) for i in range(3)]


def _deck(root, f, i, fw, gases, bars, temp):
    """The deck of one point; points of one framework and gas share their FIELD and CONFIG."""
    first = os.path.join(root, "fw%03d_%s" % (f, "-".join(gases)))
    d = os.path.join(root, "point_%03d_%03d" % (f, i))
    kmax = _kmax(fw, 0)
    if not os.path.isdir(first):
        synth.write_inputs(first, fw, gases, [1.0] * len(gases), 298.0, kmax, eq_cycles=EQ, prod_cycles=STEPS)
    empty = synth.Framework(fw.cell, [], np.zeros((0, 3)), [], fw.lj)
    synth.write_inputs(d, empty, gases, bars, temp, kmax, eq_cycles=EQ, prod_cycles=STEPS)
    for name in ("FIELD", "CONFIG"):
        os.remove(os.path.join(d, name))
        os.link(os.path.join(first, name), os.path.join(d, name))
    return d


# ------------------------------------------------------------------------------------ one pass
STATE = ("status", "moves", "gcmccount", "nmol0", "nmol1", "accept_ins", "accept_del", "ins_count", "del_count",
         "prodcount")
VALUE = ("energy0", "energy1", "elrc", "N", "E", "EN", "N2", "E2")
RESULT = ("moves", "status", "nmol0", "prodcount", "accept_ins", "accept_del", "gcmccount", "finished", "budget")
RESULT_VALUE = ("energy0", "N", "E", "EN", "N2", "E2")


def run(s):
    kind = s["kind"]
    if kind == "trial":
        return _trial(s)
    if kind == "ewald1":
        e = s["chain"].ewald1()
        return {"energy": np.array([e]), "sk": s["chain"].sk()}
    if kind == "single_point":
        return {"energy": np.array(s["chain"].single_point())}
    if kind == "run":
        tr = s["chain"].run(s["moves"])
        return {k: np.ascontiguousarray(tr[k]) for k in tr.dtype.names if not k.startswith("pad")}
    if kind == "batch":
        b = s["batch"]
        b.run(s["moves"])
        st = [b.state(c) for c in range(b.n)]
        return {"counts": np.array([[int(x[k]) for k in STATE] for x in st]),
                **{k: np.array([x[k] for x in st]) for k in VALUE}}
    srv, done = s["server"], {}
    ids = [srv.submit(d, seed, moves) for d, seed, moves in s["jobs"]]
    while srv.busy():
        srv.step(s["step"])
        for rid, state, res in srv.poll_done():
            done[rid] = (state, res)
    return {"counts": np.array([[done[i][0]] + [int(done[i][1][k]) for k in RESULT] for i in ids]),
            **{k: np.array([done[i][1][k] for i in ids]) for k in RESULT_VALUE}}


def _trial(s):
    ch, mol, old, new, moved = s["chain"], s["mol"], s["guests"][s["mol"]], s["new"], s["moved"]
    recip, real = [], []
    if s["move"] in ("insert", "exchange"):
        recip.append(ch.ewald1_guest(0, new, fm.INSERT))
        real.append(ch.guest_realspace(0, new))
    if s["move"] == "exchange":  # accepted, then the same molecule deleted: the state is as it was
        ch.commit(fm.INSERT, 0, -1, new)
        mol = len(s["guests"])
        old = new
    if s["move"] in ("delete", "exchange"):
        recip.append(ch.ewald1_guest(0, old, fm.DELETE))
        real.append(ch.guest_realspace(0, old, mol))
    if s["move"] == "exchange":
        ch.commit(fm.DELETE, 0, mol)
    if s["move"] == "displace":
        ch.ewald1_guest(0, old, fm.DISPLACE, 1)
        recip.append(ch.ewald1_guest(0, moved, fm.DISPLACE, 2))
        real.append(ch.guest_realspace(0, old, mol))
        real.append(ch.guest_realspace(0, moved, mol))
    if s["move"] != "exchange":
        ch.reject()
    return {"recip": np.array(recip), "real": np.array(real)}


# ------------------------------------------------------------------------------------ floors
def _k_count(volume, kcut):
    """Half-space k-vectors within kcut (1/A)."""
    return volume * kcut ** 3 / (12.0 * math.pi ** 2)


def _one_chain_sizes(case):
    n = case["unit"] * case["reps"]
    V = case["edge"] ** 3 * case["reps"] if case["edge"] else max(n / RHO, (2.0 * RCUT) ** 3)
    kcut = 2.0 * math.pi * 1.05 * case["kmax"] / V ** (1.0 / 3.0) if case["kmax"] else 0.95
    ns = len(synth.GASES[case["gas"]][1])
    g = case.get("guests", 20) * ns
    near = 4.0 / 3.0 * math.pi * RCUT ** 3 / V
    return n, V, _k_count(V, kcut), ns, g, near * n, near * g


# operations of one pair within the cut-off (image, distance, two interpolations) and of one site's term of a k-vector
PAIR, TERM = 45.0, 18.0


def _move_work(K, ns, near, sites_per_move=1.5):
    """One trial move: S(k) read, S_new written, akk read; every neighbour within the cut-off read once per site."""
    return {"bytes": 40.0 * K + sites_per_move * ns * near * 36.0,
            "flops": sites_per_move * ns * (K * TERM + near * PAIR) + 8.0 * K}


def work(case):
    kind = case["kind"]
    if kind in ("trial", "run"):
        n, V, K, ns, g, nf, ngu = _one_chain_sizes(case)
        sites = {"insert": 1, "delete": 1, "displace": 2, "exchange": 2}.get(case.get("move"), 1.5)
        w = _move_work(K, ns, nf + ngu, sites)
        return {k: v * case.get("moves", 1) for k, v in w.items()}
    if kind == "ewald1":
        n, V, K, ns, g, _, _ = _one_chain_sizes(case)
        return {"bytes": 32.0 * (n + g) + 24.0 * K, "flops": 8.0 * K * (n + g)}
    if kind == "single_point":
        n, V, K, ns, g, nf, ngu = _one_chain_sizes(case)
        return {"bytes": 32.0 * (n + g) + 24.0 * K, "flops": 8.0 * K * (n + g) + PAIR * g * (nf + 0.5 * ngu)}
    if kind == "batch":
        L = 0.5 * (case["lo"] + case["hi"])
        V = L ** 3 * (8.0 if L < 2.0 * RCUT else 1.0)
        w = _move_work(_k_count(V, 0.95), 3, 4.0 / 3.0 * math.pi * RCUT ** 3 * RHO)
        n = case["frameworks"] * case["pressures"] * case["moves"]
        return {k: v * n for k, v in w.items()}
    V = 0.5 * (case["lo"] + case["hi"]) / RHO
    w = _move_work(_k_count(V, 0.95), 2.3, 4.0 / 3.0 * math.pi * RCUT ** 3 * RHO)
    n = case["requests"] * (case["moves_hi"] - case["moves_lo"]) / math.log(case["moves_hi"] / case["moves_lo"])
    return {k: v * n for k, v in w.items()}


# ------------------------------------------------------------------------------------ 64-bit results without the framework
class _Exact:
    """Energies of a one-chain case restated in torch: the reference's tables, cut-offs and k-vectors."""

    def __init__(self, case, seed):
        self.fw, self.kmax, self.guests, self.new, self.moved = _loaded(case, seed)
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device=self.dev)  # noqa: E731
        self.t = t
        h = self.fw.cell
        self.h, self.inv, self.V = t(h), t(np.linalg.inv(h)), abs(np.linalg.det(h))
        sites = synth.GASES[case["gas"]][1]
        self.gname = [s[0] for s in sites]
        self.gq = np.array([s[2] for s in sites])
        self.mxgrid = max(1000, int(RCUT / 0.01 + 0.5) + 4)
        self.dr = RCUT / (self.mxgrid - 4)
        r = np.arange(1, self.mxgrid + 1) * self.dr
        a = (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)
        tt = 1.0 / (1.0 + 0.3275911 * ALPHA * r)
        erc = tt * (a[0] + tt * (a[1] + tt * (a[2] + tt * (a[3] + tt * a[4])))) * np.exp(-(ALPHA * r) ** 2) / r
        lj = {s[0]: (s[6], s[7]) for s in sites}
        lj.update(self.fw.lj)
        self.types = list(dict.fromkeys([s[0] for s in sites] + [x for x, _, _ in synth.FRAMEWORK_TYPES if x in self.fw.names]))
        nt = len(self.types)
        self.prm = {}
        tab = np.zeros((nt * nt, self.mxgrid))
        for i in range(nt):
            for j in range(nt):
                (ea, sa), (eb, sb) = lj[self.types[max(i, j)]], lj[self.types[min(i, j)]]
                e = float("%.6f" % math.sqrt(ea * eb)) * KCAL
                sg = float("%.6f" % (0.5 * (sa + sb))) if e > 0 else 0.0
                self.prm[i, j] = (e, sg)
                tab[i * nt + j] = 4.0 * e * ((sg / r) ** 12 - (sg / r) ** 6)
        first = lambda x: np.concatenate([x[..., :1], x], axis=-1)  # noqa: E731
        self.erc, self.vvv = t(first(erc)), t(first(tab))
        idx = {n: i for i, n in enumerate(self.types)}
        self.fx, self.fq = t(self.fw.xyz), t(self.fw.charges)
        self.ft = torch.tensor([idx[n] for n in self.fw.names], device=self.dev)
        self.gt = torch.tensor([idx[n] for n in self.gname], device=self.dev)
        self.engsic = -R4PIE0 * ALPHA * float((self.gq ** 2).sum()) / math.sqrt(math.pi)
        self._kvectors()

    def _kvectors(self):
        inv, twopi = np.linalg.inv(self.fw.cell), 2.0 * math.pi
        w = _widths(inv)
        cut = (min(k * x for k, x in zip(self.kmax, w)) * 1.05 * twopi) ** 2
        lmn = []
        mmin, nmin = 0, 1
        for ll in range(self.kmax[0] + 1):
            for mm in range(mmin, self.kmax[1] + 1):
                n = np.arange(nmin, self.kmax[2] + 1)
                lmn.append(np.stack([np.full(len(n), ll), np.full(len(n), mm), n], 1))
                nmin = -self.kmax[2]
            mmin = -self.kmax[1]
        lmn = np.concatenate(lmn)
        k = twopi * lmn @ inv.T
        k2 = (k * k).sum(1)
        keep = k2 <= cut
        self.k = self.t(lmn[keep])
        self.akk = self.t(np.exp(-0.25 / ALPHA ** 2 * k2[keep]) / k2[keep])
        self.pref = 2.0 * (twopi / self.V) * R4PIE0

    def sk(self, xyz, q):
        out = torch.zeros(len(self.k), dtype=torch.complex128, device=self.dev)
        f = xyz @ self.inv
        for a in range(0, len(f), 512):
            g = f[a:a + 512]
            ph = self.k @ (g - torch.round(g)).T
            ph = 2.0 * math.pi * (ph - torch.round(ph))
            out += (torch.complex(torch.cos(ph), torch.sin(ph)) * q[a:a + 512]).sum(1)
        return out

    def mol_sk(self, mol):
        return self.sk(self.t(mol), self.t(self.gq))

    def total_sk(self):
        s = self.sk(self.fx, self.fq)
        n = len(self.guests)
        return s + self.sk(self.t(self.guests.reshape(-1, 3)), self.t(np.tile(self.gq, n))) if n else s

    def recip(self, s):
        return float(self.pref * (self.akk * (s.real ** 2 + s.imag ** 2)).sum())

    def d_recip(self, s, d):
        return float(self.pref * (self.akk * (2.0 * (s.real * d.real + s.imag * d.imag) + d.real ** 2 + d.imag ** 2)).sum())

    def _interp(self, tab, base, x):
        l = x.long()  # noqa: E741
        p = x - l
        v0, v1, v2 = tab[base + l], tab[base + l + 1], tab[base + l + 2]
        t1 = v0 + (v1 - v0) * p
        t2 = v1 + (v2 - v1) * (p - 1.0)
        return t1 + (t2 - t1) * p * 0.5

    def real(self, mol, xyz, q, types):
        """Coulomb and vdW of one molecule's sites against atoms at xyz."""
        ec = ev = 0.0
        nt, n = len(self.types), self.mxgrid + 1
        x = self.t(mol)
        for i in range(len(x)):
            d = (x[i] - xyz) @ self.inv
            d = (d - torch.round(d)) @ self.h
            r2 = (d * d).sum(1)
            near = r2 < RCUT * RCUT
            u = r2[near].sqrt() / self.dr
            c = float(self.gq[i]) * R4PIE0 * q[near]
            ec += float((self._interp(self.erc, 0, u) * c).sum())
            row = int(self.gt[i]) * nt + types[near]
            ev += float(self._interp(self.vvv.reshape(-1), row * n, u).sum())
        return ec, ev

    def around(self, mol, skip=-1):
        """Real-space energies of a molecule among the framework and all guests but `skip`."""
        keep = [g for i, g in enumerate(self.guests) if i != skip]
        m = len(keep)
        xyz = torch.cat([self.fx] + ([self.t(np.concatenate(keep))] if m else []))
        q = torch.cat([self.fq, self.t(np.tile(self.gq, m))])
        return self.real(mol, xyz, q, torch.cat([self.ft, self.gt.repeat(m)]))

    def _erf_pair(self, q, r):
        a = (0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)
        tt = 1.0 / (1.0 + 0.3275911 * ALPHA * r)
        e = math.exp(-(ALPHA * r) ** 2)
        return (1.0 - tt * (a[0] + tt * (a[1] + tt * (a[2] + tt * (a[3] + tt * a[4])))) * e) * q / r

    def _tail(self):
        counts = np.array([float((self.ft == i).sum()) for i in range(len(self.types))])
        frozen = counts.copy()
        for i in self.gt.tolist():
            counts[i] += len(self.guests)
        e = 0.0
        for i in range(len(self.types)):
            for j in range(i + 1):
                eps, sg = self.prm[i, j]
                s = 4.0 * eps * (sg ** 12 / (9.0 * RCUT ** 9) - sg ** 6 / (3.0 * RCUT ** 3)) * (2.0 if i != j else 1.0)
                e += 2.0 * math.pi * (counts[i] * counts[j] - frozen[i] * frozen[j]) / self.V * s
        return e

    def single_point(self):
        self_term = lambda q2: -R4PIE0 * ALPHA * q2 / math.sqrt(math.pi)  # noqa: E731
        n = len(self.guests)
        fw = self.recip(self.sk(self.fx, self.fq)) + self_term(float((self.fq ** 2).sum()))
        every = self.recip(self.total_sk()) + self_term(float((self.fq ** 2).sum()) + n * float((self.gq ** 2).sum()))
        coul = vdw = corr = 0.0
        gx = self.t(self.guests.reshape(-1, 3))
        gq, gt = self.t(np.tile(self.gq, n)), self.gt.repeat(n)
        ns = len(self.gq)
        for m, mol in enumerate(self.guests):
            a = self.real(mol, self.fx, self.fq, self.ft)
            keep = torch.ones(n * ns, dtype=torch.bool, device=self.dev)
            keep[m * ns:(m + 1) * ns] = False
            b = self.real(mol, gx[keep], gq[keep], gt[keep])
            coul += a[0] + 0.5 * b[0]
            vdw += a[1] + 0.5 * b[1]
            for i in range(ns):
                for j in range(i + 1, ns):
                    corr -= self._erf_pair(self.gq[i] * R4PIE0 * self.gq[j], float(np.linalg.norm(mol[i] - mol[j])))
        tail = self._tail()
        guest = every - fw + coul + corr + vdw + tail
        return np.array([guest / KCAL, (every + coul + vdw + tail + corr) / KCAL])


def exact(case, seed):
    """What run() returns, in 64 bits without the framework; no value for whole move loops (their results are the
    trajectories of a seeded chain)."""
    kind = case["kind"]
    if kind not in ("trial", "ewald1", "single_point"):
        return None
    x = _Exact(case, seed)
    if kind == "single_point":
        return {"energy": x.single_point()}
    s = x.total_sk()
    if kind == "ewald1":
        q2 = float((x.fq ** 2).sum()) + len(x.guests) * float((x.gq ** 2).sum())
        return {"energy": np.array([x.recip(s) - R4PIE0 * ALPHA * q2 / math.sqrt(math.pi)]), "sk": s.cpu().numpy()}
    recip, real = [], []
    mol = len(x.guests) // 2
    if case["move"] in ("insert", "exchange"):
        d = x.mol_sk(x.new)
        recip.append(x.d_recip(s, d) + x.engsic)
        real.append(x.around(x.new))
    if case["move"] == "exchange":
        recip.append(x.d_recip(s + d, -d) - x.engsic)
        real.append(x.around(x.new))
    if case["move"] == "delete":
        recip.append(x.d_recip(s, -x.mol_sk(x.guests[mol])) - x.engsic)
        real.append(x.around(x.guests[mol], mol))
    if case["move"] == "displace":
        recip.append(x.d_recip(s, x.mol_sk(x.moved) - x.mol_sk(x.guests[mol])))
        real += [x.around(x.guests[mol], mol), x.around(x.moved, mol)]
    return {"recip": np.array(recip), "real": np.array(real)}
