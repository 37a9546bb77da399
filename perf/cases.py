"""Work that programs give this engine: what is timed when its speed is judged.

A case is a dict of plain values.  Its "kind" is the entry point:

  force   Potential.compute: energy, forces and virials of one periodic box
  batch   Potential.compute_batch: many independent structures in one call
  md      MD.run: device-resident dynamics, with thermo rows
  serve   Server.submit / Server.wait: requests from host arrays, some of them
          short NVE segments, results in host arrays

Structures are those of the benchmark (diamond C, FCC Cu with vacancies and
ZBL, liquid water, and a four-type C/H/O/Cu stream), the potentials are
synthetic NEP files of the benchmark's shapes, and of the larger n_max and
basis that published single-element potentials use.  exact() restates the
potential in 64-bit torch with automatic derivatives.
"""
import importlib
import math
import os
import tempfile

import numpy as np
import torch

nepx = importlib.import_module("dmg-md_b200.nepx")

MODELS = {
    # O/H of the 24,000-atom water box
    "water": dict(version=4, symbols=("O", "H"), rc=(6.0, 4.0), mn=(250, 100), n_max=(4, 4),
                  basis=(8, 8), l_max=(4, 2, 0), H=50, seed=2024, scale=0.02),
    # diamond and amorphous carbon
    "carbon": dict(version=4, symbols=("C",), rc=(4.2, 3.7), mn=(100, 60), n_max=(4, 4),
                   basis=(8, 8), l_max=(4, 2, 1), H=30, seed=2025, scale=0.02),
    # FCC copper with the universal ZBL
    "copper": dict(version=4, symbols=("Cu",), zbl=(1.0, 2.0), rc=(5.0, 4.0), mn=(100, 60),
                   n_max=(4, 4), basis=(8, 8), l_max=(4, 2, 1), H=40, seed=2026, scale=0.02),
    # the serving stream's shared four-type NEP5
    "stream": dict(version=5, symbols=("C", "H", "O", "Cu"), rc=(5.0, 4.0), mn=(160, 80),
                   n_max=(4, 4), basis=(8, 8), l_max=(4, 2, 1), H=64, seed=2027, scale=0.02),
    # the shape of the published carbon potential (long cutoff, many radial functions)
    "carbon_wide": dict(version=4, symbols=("C",), rc=(7.0, 4.0), mn=(358, 71), n_max=(12, 8),
                        basis=(16, 12), l_max=(4, 2, 1), H=100, seed=2028, scale=0.02),
}
MASS = {"H": 1.008, "C": 12.011, "O": 15.999, "Cu": 63.546}
K_B = 8.617343e-5          # eV/K
TIME_UNIT = 10.18051       # fs per natural time unit (eV, A, amu)
COULOMB = 14.399645        # eV A
ATOMIC_NUMBER = {"H": 1, "C": 6, "O": 8, "Cu": 29}
DIAMOND = ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0),
           (.25, .25, .25), (.25, .75, .75), (.75, .25, .75), (.75, .75, .25))
FCC = ((0, 0, 0), (0, .5, .5), (.5, 0, .5), (.5, .5, 0))
LATTICE = {"carbon": (DIAMOND, 3.567), "carbon_wide": (DIAMOND, 3.567), "copper": (FCC, 3.615)}


def listed():
    return [
        # one geometry of a fit or a relaxation: a small cell whose images all count
        dict(name="cell_c64", kind="force", model="carbon", nx=2, ny=2, nz=2, precision="fp32"),
        # a small solvent box in a sheared cell, odd size: a test set's structure
        dict(name="force_water1551_tilted", kind="force", model="water", molecules=517, tilt=0.12,
             precision="fp32"),
        # the 24,000-atom water box, one force call of an outer program's integrator
        dict(name="force_water24k", kind="force", model="water", molecules=8000, tilt=0.0,
             precision="fp32"),
        # the same with the ANN on the tensor cores
        dict(name="force_water24k_mixed", kind="force", model="water", molecules=8000, tilt=0.0,
             precision="mixed"),
        # a potential of the published carbon shape on a block of diamond
        dict(name="force_wide14k", kind="force", model="carbon_wide", nx=12, ny=12, nz=12,
             precision="fp32"),
        # one GPU's share of the largest systems: 8,000,000 carbon atoms
        dict(name="force_carbon8m", kind="force", model="carbon", nx=100, ny=100, nz=100,
             precision="fp32"),
        # a ragged mid-size carbon block in the mixed mode
        dict(name="force_carbon200k_mixed", kind="force", model="carbon", nx=29, ny=31, nz=29,
             precision="mixed"),
        # screening many candidate structures, 16 to 8,192 atoms, in one call
        dict(name="batch188", kind="batch", model="stream", count=188, lo=16, hi=8192,
             precision="fp32"),
        # long trajectories of a small system: steps per second at 4,096 atoms
        dict(name="md_carbon4096_nve", kind="md", model="carbon", nx=8, ny=8, nz=8,
             ensemble="nve", steps=100, dt=1.0, every=10, precision="fp32"),
        # thermostatted water
        dict(name="md_water24k_bdp", kind="md", model="water", molecules=8000, tilt=0.0,
             ensemble="nvt_bdp", steps=40, dt=0.5, every=10, precision="fp32"),
        # copper with vacancies under pressure control, 990,148 atoms
        dict(name="md_copper990k_npt", kind="md", model="copper", nx=63, ny=63, nz=63,
             ensemble="npt_ber", steps=10, dt=1.0, every=10, precision="fp32"),
        # a burst of requests at the server, a fifth of them 100-step segments
        dict(name="serve48", kind="serve", model="stream", count=48, lo=16, hi=8192, steps=100,
             precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, model, lo, hi):
    """Near-cubic supercell of lo..hi atoms, its three edges up to a fifth apart,
    and how far its atoms are off their sites (A)."""
    per = len(LATTICE[model][0])
    m = max(2, int(round((_log(rng, lo, hi) / per) ** (1.0 / 3.0))))
    top = max(2, int((hi / per) ** (1.0 / 3.0)))
    c = {k: max(2, min(top, m + rng.randrange(-(m // 10), m // 10 + 2))) for k in ("nx", "ny", "nz")}
    c["jitter"] = round(rng.uniform(0.02, 0.08), 4)
    return c


def draw(rng):
    kind = rng.choice(("force", "force", "force", "force", "md", "md", "batch", "serve"))
    if kind == "batch":
        return dict(kind=kind, model="stream", count=_log(rng, 8, 188), lo=16,
                    hi=_log(rng, 200, 8192), precision=rng.choice(("fp32", "mixed")))
    if kind == "serve":
        return dict(kind=kind, model="stream", count=_log(rng, 8, 48), lo=16,
                    hi=_log(rng, 200, 8192), steps=rng.randrange(10, 101), precision="mixed")
    c = dict(kind=kind, model=rng.choice(("water", "carbon", "copper") +
                                         (("carbon_wide",) if kind == "force" else ())))
    hi = {"carbon_wide": 30000, "water": 400000}.get(c["model"], 4000000)
    lo = 64
    if kind == "md":
        lo, hi = 2000, min(hi, 400000)
    if c["model"] == "water":
        c.update(molecules=max(40, _log(rng, lo, hi) // 3),
                 tilt=0.0 if kind == "md" else rng.choice((0.0, round(rng.uniform(0.02, 0.2), 3))))
    else:
        c.update(_cells(rng, c["model"], lo, hi))
    if kind == "md":
        ens = rng.choice(("nve", "nvt_ber", "nvt_bdp", "npt_ber"))
        steps = rng.randrange(5, 41)
        c.update(ensemble=ens, steps=steps, dt=0.5 if c["model"] == "water" else 1.0,
                 every=rng.choice((1, 5)))
    c["precision"] = rng.choice(("fp32", "fp32", "mixed"))
    return c


# ---- inputs ---------------------------------------------------------------------------------

def _model(name):
    """The potential's parameters as NumPy arrays of 32-bit values, and its file's text."""
    m = MODELS[name]
    T = len(m["symbols"])
    nR, nA = m["n_max"][0] + 1, m["n_max"][1] + 1
    kR, kA = m["basis"][0] + 1, m["basis"][1] + 1
    dim = nR + nA * (m["l_max"][0] + sum(1 for f in m["l_max"][1:] if f))
    H = m["H"]
    rng = np.random.default_rng(m["seed"])

    def weights(*shape):
        return rng.normal(0.0, 0.1, shape).astype(np.float32)

    ann = []
    for _ in range(T):
        ann.append(dict(w0=weights(H, dim), b0=weights(H), w1=weights(H),
                        own=weights(1) if m["version"] == 5 else None))
    bias = weights(1)
    c_r, c_a = weights(nR, kR, T, T), weights(nA, kA, T, T)
    q_scale = np.full(dim, m["scale"], dtype=np.float32)
    flat = []
    for a in ann:
        flat += [a["w0"].ravel(), a["b0"], a["w1"]] + ([a["own"]] if a["own"] is not None else [])
    flat += [bias, c_r.ravel(), c_a.ravel(), q_scale]
    zbl = m.get("zbl")
    lines = ["nep%d%s %d %s" % (m["version"], "_zbl" if zbl else "", T, " ".join(m["symbols"]))]
    if zbl:
        lines.append("zbl %g %g" % zbl)
    lines += ["cutoff %g %g %d %d" % (m["rc"] + m["mn"]), "n_max %d %d" % m["n_max"],
              "basis_size %d %d" % m["basis"], "l_max %d %d %d" % m["l_max"], "ANN %d 0" % H]
    lines += ["%.9e" % v for v in np.concatenate(flat)]
    return dict(m, T=T, nR=nR, nA=nA, kR=kR, kA=kA, dim=dim, ann=ann, bias=bias, c_r=c_r, c_a=c_a,
                q_scale=q_scale), "\n".join(lines) + "\n"


def _potential(case, atoms):
    """The handle a program makes once: potential file, capacity, precision."""
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "nep.txt")
        with open(path, "w") as f:
            f.write(_model(case["model"])[1])
        pot = nepx.Potential(path, max_atoms=atoms)
    if case["precision"] != "fp32":
        pot.set_precision(case["precision"])
    return pot


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)
    return g


def _crystal(base, a, dims, g, jitter):
    b = torch.tensor(base, dtype=torch.float64, device="cuda")
    ix = [torch.arange(d, dtype=torch.float64, device="cuda") for d in dims]
    cell = torch.stack(torch.meshgrid(*ix, indexing="ij"), -1).reshape(-1, 1, 3)
    pos = ((cell + b) * a).reshape(-1, 3)
    pos += jitter * torch.randn(pos.shape, generator=g, dtype=torch.float64, device="cuda")
    return pos, np.diag(np.array(dims, dtype=np.float64) * a)


def _system(case, seed):
    """(types int32 (n,), box rows-major 3x3 with the cell vectors as columns,
    positions (3, n)) on the GPU."""
    g = _generator(seed)
    model = case["model"]
    if model == "water":
        n = case["molecules"]
        L = (n * 18.015 / 0.60221408) ** (1.0 / 3.0)
        m = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
        ix = torch.arange(m, dtype=torch.float64, device="cuda")
        sites = torch.stack(torch.meshgrid(ix, ix, ix, indexing="ij"), -1).reshape(-1, 3)
        sites = sites[torch.randperm(len(sites), generator=g, device="cuda")[:n]]
        O = (sites + 0.5 + 0.3 * (torch.rand(n, 3, generator=g, dtype=torch.float64,
                                             device="cuda") - 0.5)) * (L / m)
        u = torch.randn(n, 3, generator=g, dtype=torch.float64, device="cuda")
        u /= u.norm(dim=1, keepdim=True)
        v = torch.randn(n, 3, generator=g, dtype=torch.float64, device="cuda")
        v -= (v * u).sum(1, keepdim=True) * u
        v /= v.norm(dim=1, keepdim=True)
        th = math.radians(104.5)
        H1 = O + 0.96 * u
        H2 = O + 0.96 * (math.cos(th) * u + math.sin(th) * v)
        pos = torch.stack([O, H1, H2], 1).reshape(-1, 3)
        types = torch.tensor([0, 1, 1], dtype=torch.int32, device="cuda").repeat(n)
        h = np.eye(3) * L
    else:
        base, a = LATTICE[model]
        dims = (case["nx"], case["ny"], case["nz"])
        pos, h = _crystal(base, a, dims, g, case.get("jitter", 0.05))
        n = len(pos)
        if model == "copper":      # one site in a hundred is empty
            keep = torch.randperm(n, generator=g, device="cuda")[:n - n // 100].sort().values
            pos = pos[keep]
        elif n > 1000:             # a tenth of the atoms far off their sites
            pick = torch.rand(n, 1, generator=g, device="cuda", dtype=torch.float64) < 0.1
            pos = pos + pick * 0.3 * torch.randn(pos.shape, generator=g, dtype=torch.float64,
                                                 device="cuda")
        types = torch.zeros(len(pos), dtype=torch.int32, device="cuda")
    tilt = case.get("tilt", 0.0)
    H = torch.tensor(h, device="cuda")
    frac = torch.remainder(torch.linalg.solve(H, pos.T), 1.0)
    if tilt:
        h = h @ np.array([[1.0, tilt, -0.5 * tilt], [0.0, 1.0, tilt], [0.0, 0.0, 1.0]])
    pos = torch.tensor(h, device="cuda") @ frac
    return types, h, pos.contiguous()


def _structures(case, seed):
    """The screening stream: jittered diamond and copper supercells and packed
    four-type boxes of log-uniform size.  The sizes are the case's, the
    coordinates the seed's.  Host arrays (types, h, positions (3, n))."""
    sizes, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed + 1)
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        kind = sizes.integers(0, 3)
        if kind < 2:
            base, a = (DIAMOND, 3.567) if kind == 0 else (FCC, 3.615)
            m = max(1, int(round((n / len(base)) ** (1.0 / 3.0))))
            dims = np.array([m, m, max(1, int(round(n / (len(base) * m * m))))])
            cell = np.stack(np.meshgrid(*[np.arange(d) for d in dims], indexing="ij"), -1)
            pos = (cell.reshape(-1, 1, 3) + np.array(base)).reshape(-1, 3) * a
            pos = pos + rng.normal(0.0, 0.1, pos.shape)
            L = dims * a
            types = np.full(len(pos), 0 if kind == 0 else 3, dtype=np.int32)
        else:
            L = np.full(3, (n / 0.08) ** (1.0 / 3.0))
            m = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
            cell = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
            cell = cell[rng.permutation(len(cell))[:n]]
            sp = L[0] / m
            pos = (cell + 0.5) * sp + rng.uniform(-0.25, 0.25, (n, 3)) * max(sp - 0.9, 0.0)
            types = rng.integers(0, 4, n).astype(np.int32)
        out.append((types, np.diag(L), np.ascontiguousarray((pos % L).T)))
    return out


def _velocities(masses, T, seed):
    """Maxwell-Boltzmann velocities (3, n) in A/fs without drift."""
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(3, len(masses))) * np.sqrt(K_B * T / masses)
    v -= ((v * masses).sum(axis=1) / masses.sum())[:, None]
    return v / TIME_UNIT


class _DeviceArray:
    """A device pointer of the engine as something torch can view; the view
    keeps its owner, which frees the memory when it goes."""

    def __init__(self, owner, ptr, shape, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=dtype, data=(ptr, False),
                                             version=3)


def _md_inputs(case, seed):
    types, h, pos = _system(case, seed)
    symbols = MODELS[case["model"]]["symbols"]
    t = types.cpu().numpy()
    masses = np.array([MASS[s] for s in symbols])[t]
    return t, h, pos.cpu().numpy(), masses, _velocities(masses, 300.0, seed)


def _segments(case, seed):
    """The server's requests: every fifth one an NVE segment."""
    reqs = []
    masses = np.array([MASS[s] for s in MODELS[case["model"]]["symbols"]])
    for k, (t, h, p) in enumerate(_structures(case, seed)):
        r = dict(types=t, pos=p, h=h, md_steps=0)
        if k % 5 == 2:
            m = masses[t]
            r.update(md_steps=case["steps"], dt_fs=1.0, masses=m, want_state=True,
                     vel=_velocities(m, 300.0, 1000 * seed + k))
        reqs.append(r)
    return reqs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "force":
        types, h, pos = _system(case, seed)
        n = len(types)
        out = (torch.empty(n, dtype=torch.float64, device="cuda"),
               torch.empty(3, n, dtype=torch.float64, device="cuda"),
               torch.empty(9, n, dtype=torch.float64, device="cuda"))
        return dict(case=case, pot=_potential(case, n), types=types, h=h.reshape(-1), pos=pos,
                    out=out)
    if kind == "batch":
        s = _structures(case, seed)
        n = sum(len(t) for t, _, _ in s)
        out = (torch.empty(n, dtype=torch.float64, device="cuda"),
               torch.empty(3, n, dtype=torch.float64, device="cuda"),
               torch.empty(9, n, dtype=torch.float64, device="cuda"))
        return dict(case=case, pot=_potential(case, n), out=out,
                    structs=[(len(t), h.reshape(-1), (1, 1, 1)) for t, h, _ in s],
                    types=torch.as_tensor(np.concatenate([t for t, _, _ in s]), device="cuda"),
                    pos=torch.as_tensor(np.concatenate([p for _, _, p in s], axis=1),
                                        device="cuda"))
    if kind == "md":
        t, h, pos, masses, vel = _md_inputs(case, seed)
        pot = _potential(case, len(t))
        md = nepx.MD(pot, t, masses, pos, vel, h.reshape(-1))
        ens = case["ensemble"]
        if ens == "nve":
            md.set_ensemble("nve")
        elif ens == "npt_ber":
            md.set_ensemble(ens, T0=300.0, Tdamp=100.0, p_gpa=0.0, bulk_gpa=140.0, tau_p=1000.0,
                            seed=seed % 100000)
        else:
            md.set_ensemble(ens, T0=300.0, Tdamp=100.0, seed=seed % 100000)
        p = md.device_state()
        view = [torch.as_tensor(_DeviceArray(md, q, (3, len(t)), "<f8"), device="cuda")
                for q in p[:3]]
        return dict(case=case, pot=pot, md=md, view=view)
    if kind == "serve":
        reqs = _segments(case, seed)
        pot = _potential(case, 65536)
        return dict(case=case, pot=pot, reqs=reqs,
                    srv=nepx.Server(pot, max_atoms=65536, max_struct=256))
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "force":
        pe, f, w = state["pot"].compute(state["types"], state["h"], state["pos"],
                                        out=state["out"])
        return dict(pe=pe, force=f, virial=w)
    if kind == "batch":
        pe, f, w = state["pot"].compute_batch(state["structs"], state["types"], state["pos"],
                                              out=state["out"])
        return dict(pe=pe, force=f, virial=w)
    if kind == "md":
        rows = state["md"].run(case["steps"], case["dt"], thermo_every=case["every"])
        pos, vel, force = state["view"]
        return dict(thermo=rows, pos=pos, vel=vel, force=force)
    srv = state["srv"]
    tickets = [srv.submit(**r) for r in state["reqs"]]
    res = [srv.wait(t) for t in tickets]
    out = {k: np.concatenate([r[k] for r in res], axis=-1) for k in ("pe", "force", "virial")}
    moved = [r for r in res if "vel" in r]
    out.update({k: np.concatenate([r[k] for r in moved], axis=-1) for k in ("pos", "vel")})
    return out


# ---- what a pass cannot do without ------------------------------------------------------------

def _atoms(case):
    if "molecules" in case:
        return 3 * case["molecules"]
    if "nx" in case:
        n = len(LATTICE[case["model"]][0]) * case["nx"] * case["ny"] * case["nz"]
        return n - n // 100 if case["model"] == "copper" else n
    return sum(len(t) for t, _, _ in _structures(case, 0))


def _flops(case):
    """Operations of one force evaluation per atom: per radial edge geometry,
    cutoff, basis, the contraction with c, and the two derivative sums of the
    pair force; per angular edge the same for the moments, the harmonics, and
    the gradient; per atom the network forward and backward."""
    m, _ = _model(case["model"])
    rho = {"water": 0.1003, "copper": 0.0838, "stream": 0.1}.get(case["model"], 0.1763)
    nr, na = (rho * 4.18879 * r ** 3 for r in m["rc"])
    nlm = (m["l_max"][0] + 1) ** 2 - 1
    radial = nr * (2 * (32 + 4 * m["kR"]) + 2 * m["kR"] + 4 * m["kR"] + 4 * m["kR"] + 24)
    angular = na * (32 + 12 * m["kA"] + 6 * m["nA"] * m["kA"] + 13 * nlm + 6 * m["nA"] * nlm + 40)
    center = 4 * m["dim"] * m["H"] + 12 * m["H"] + 10 * m["nA"] * nlm + 2 * m["T"] * m["nR"] * m["kR"]
    return radial + angular + center


def work(case):
    n, flops = _atoms(case), _flops(case)
    if case["kind"] in ("force", "batch"):
        return dict(bytes=132.0 * n, flops=flops * n)     # positions, types; energy, force, virial
    if case["kind"] == "md":      # types, masses, positions, velocities; positions, velocities, forces
        return dict(bytes=132.0 * n, flops=flops * n * case["steps"])
    s = _structures(case, 0)
    evals = sum(len(t) * (1 + (case["steps"] if k % 5 == 2 else 0)) for k, (t, _, _) in enumerate(s))
    return dict(bytes=132.0 * n, flops=flops * evals)


def tolerance(case):
    """32-bit forces of these gentle landscapes are small differences of large
    sums, the virial less so; the mixed mode has 11-bit operands in the network."""
    if case["precision"] != "fp32":
        return {"rel": 5e-3, "max": 5e-2}
    return {"rel": 2e-5, "max": 1e-3}


# ---- the same in 64 bits ----------------------------------------------------------------------

def _edges(pos, h, rc, lo, hi):
    """Directed edges (center, neighbour, r_j - r_i) of the centers lo..hi within rc,
    periodic images counted one by one."""
    H = torch.tensor(h, device="cuda")
    inv = torch.linalg.inv(H)
    thick = 1.0 / inv.norm(dim=1)
    d = pos.T[None, :, :] - pos.T[lo:hi, None, :]
    out = [[], [], []]
    if bool((thick > 2.0 * rc).all()):
        s = d @ inv.T
        d = d - torch.round(s) @ H.T
        r2 = (d * d).sum(-1)
        hit = r2 < rc * rc
        hit[torch.arange(hi - lo, device="cuda"), torch.arange(lo, hi, device="cuda")] = False
        i, j = hit.nonzero(as_tuple=True)
        return i + lo, j, d[i, j]
    span = [int(math.ceil(rc / float(t))) + 1 for t in thick]
    for a in range(-span[0], span[0] + 1):
        for b in range(-span[1], span[1] + 1):
            for c in range(-span[2], span[2] + 1):
                shift = H @ torch.tensor([a, b, c], dtype=torch.float64, device="cuda")
                e = d + shift
                hit = (e * e).sum(-1) < rc * rc
                if a == b == c == 0:
                    hit[torch.arange(hi - lo, device="cuda"),
                        torch.arange(lo, hi, device="cuda")] = False
                i, j = hit.nonzero(as_tuple=True)
                out[0].append(i + lo)
                out[1].append(j)
                out[2].append(e[i, j])
    return tuple(torch.cat(x) for x in out)


def _functions(d, rc, c, pair, size):
    """sum_k c[n, k, pair] f_k(d), with f_k the cut-off Chebyshev basis."""
    x = 2.0 * (d / rc - 1.0) ** 2 - 1.0
    fc = 0.5 + 0.5 * torch.cos(math.pi * d / rc)
    f, t0, t1 = [fc], torch.ones_like(x), x
    for _ in range(1, size):
        f.append(0.5 * (t1 + 1.0) * fc)
        t0, t1 = t1, 2.0 * x * t1 - t0
    c = torch.tensor(c.reshape(c.shape[0], c.shape[1], -1), dtype=torch.float64, device="cuda")
    return torch.einsum("ke,nke->en", torch.stack(f), c[:, :, pair])


def _harmonics(u):
    """Z_Lm(z) {1, Re, Im}(x + iy)^m for L = 1..4, and the weights of q_L."""
    x, y, z = u.unbind(-1)
    one = torch.ones_like(z)
    poly = {(1, 0): z, (1, 1): one, (2, 0): 3 * z ** 2 - 1, (2, 1): z, (2, 2): one,
            (3, 0): 5 * z ** 3 - 3 * z, (3, 1): 5 * z ** 2 - 1, (3, 2): z, (3, 3): one,
            (4, 0): 35 * z ** 4 - 30 * z ** 2 + 3, (4, 1): 7 * z ** 3 - 3 * z,
            (4, 2): 7 * z ** 2 - 1, (4, 3): z, (4, 4): one}
    # the m-th derivative of the Legendre polynomial is kappa times Z
    kappa = {(1, 0): 1, (1, 1): 1, (2, 0): .5, (2, 1): 3, (2, 2): 3, (3, 0): .5, (3, 1): 1.5,
             (3, 2): 15, (3, 3): 15, (4, 0): .125, (4, 1): 2.5, (4, 2): 7.5, (4, 3): 105,
             (4, 4): 105}
    Y, weight = [], []
    for L in range(1, 5):
        re, im = one, torch.zeros_like(one)
        for m in range(L + 1):
            w = (2 * L + 1) / (4 * math.pi) * kappa[L, m] ** 2 * math.factorial(L - m) / \
                math.factorial(L + m)
            if m == 0:
                Y.append(poly[L, 0])
                weight.append(w)
            else:
                re, im = x * re - y * im, x * im + y * re
                Y += [poly[L, m] * re, poly[L, m] * im]
                weight += [2 * w, 2 * w]
    return torch.stack(Y, -1), weight


def _zbl(m, ti, tj, d):
    Z = torch.tensor([float(ATOMIC_NUMBER[s]) for s in m["symbols"]], dtype=torch.float64,
                     device="cuda")
    zi, zj = Z[ti], Z[tj]
    x = d * (zi ** 0.23 + zj ** 0.23) * 2.134563
    phi = sum(a * torch.exp(-b * x) for a, b in ((0.18175, 3.1998), (0.50986, 0.94229),
                                                 (0.28022, 0.4029), (0.02817, 0.20162)))
    r1, r2 = m["zbl"]
    s = torch.clamp((d - r1) / (r2 - r1), 0.0, 1.0)
    return 0.5 * COULOMB * zi * zj * phi / d * (0.5 + 0.5 * torch.cos(math.pi * s))


def _site_energies(m, types, i, j, r, lo, hi):
    """Energies of the centers lo..hi from their edges."""
    n, T = hi - lo, m["T"]
    d = r.norm(dim=1)
    t_i, t_j = types[i].long(), types[j].long()
    pair = t_i * T + t_j
    rows = i - lo

    def per_center(v):
        return torch.zeros((n,) + v.shape[1:], dtype=torch.float64,
                           device="cuda").index_add(0, rows[:len(v)], v)

    q = [per_center(_functions(d, m["rc"][0], m["c_r"], pair, m["kR"]))]
    near = (d.detach() < m["rc"][1]).nonzero().squeeze(1)
    d, r, rows, pair = d[near], r[near], rows[near], pair[near]
    g = _functions(d, m["rc"][1], m["c_a"], pair, m["kA"])
    Y, weight = _harmonics(r / d[:, None])
    s = torch.stack([per_center(g * Y[:, k:k + 1]) for k in range(24)], -1)     # [n][nA][24]
    at = 0
    for L in range(1, 5):
        size = 2 * L + 1
        w = torch.tensor(weight[at:at + size], dtype=torch.float64, device="cuda")
        q.append((s[..., at:at + size] ** 2 * w).sum(-1))
        at += size
    s0, s1, s2, s3, s4, s5, s6, s7 = (s[..., k] for k in range(8))
    if m["l_max"][1]:
        c = (-0.007499480826664, -0.134990654879954, 0.067495327439977, 0.404971964639861,
             -0.809943929279723)
        q.append(c[0] * s3 ** 3 + s3 * (c[1] * (s4 ** 2 + s5 ** 2) + c[2] * (s6 ** 2 + s7 ** 2)) +
                 c[3] * s6 * (s5 ** 2 - s4 ** 2) + c[4] * s4 * s5 * s7)
    if m["l_max"][2]:
        c = (0.026596810706114, 0.053193621412227, 0.026596810706114)
        p = s1 ** 2 + s2 ** 2
        q.append(c[0] * s0 ** 4 + c[1] * s0 ** 2 * p + c[2] * p ** 2)
    q = torch.cat(q, -1) * torch.tensor(m["q_scale"], dtype=torch.float64, device="cuda")
    E = torch.zeros(n, dtype=torch.float64, device="cuda")
    own = types[lo:hi]
    for t, a in enumerate(m["ann"]):
        w0, b0, w1 = (torch.tensor(a[k], dtype=torch.float64, device="cuda")
                      for k in ("w0", "b0", "w1"))
        e = torch.tanh(q @ w0.T - b0) @ w1 - float(m["bias"][0])
        if a["own"] is not None:
            e = e - float(a["own"][0])
        E = torch.where(own == t, e, E)
    if m.get("zbl"):
        E = E + per_center(_zbl(m, t_i[near], t_j[near], d)[:, None])[:, 0]
    return E


def _exact_force(m, types, h, pos):
    """Energies, forces and virials W_i = sum_j r_ij (x) dU_j/dr_ji in 64 bits."""
    n = len(types)
    pe = torch.zeros(n, dtype=torch.float64, device="cuda")
    F = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    W = torch.zeros(n, 9, dtype=torch.float64, device="cuda")
    order = [0, 4, 8, 1, 2, 5, 3, 6, 7]      # xx yy zz xy xz yz yx zx zy
    step = max(1, min(4096, 40_000_000 // n))
    for lo in range(0, n, step):
        hi = min(n, lo + step)
        i, j, r = _edges(pos, h, m["rc"][0], lo, hi)
        r = r.requires_grad_(True)
        E = _site_energies(m, types, i, j, r, lo, hi)
        pe[lo:hi] = E.detach()
        if r.numel() == 0:
            continue
        g, = torch.autograd.grad(E.sum(), r)
        r = r.detach()
        F.index_add_(0, i, g)
        F.index_add_(0, j, -g)
        W.index_add_(0, j, (-r[:, :, None] * g[:, None, :]).reshape(-1, 9)[:, order])
    return pe, F.T.contiguous(), W.T.contiguous()


def _exact_nve(m, t, h, pos, masses, vel, steps, dt_fs):
    """Velocity Verlet; velocities in and out in natural units."""
    types = torch.as_tensor(t, device="cuda")
    x, v = torch.as_tensor(pos, device="cuda"), torch.as_tensor(vel, device="cuda")
    mass, dt = torch.as_tensor(masses, device="cuda"), dt_fs / TIME_UNIT
    H = torch.tensor(h, device="cuda")
    e, f, w = _exact_force(m, types, h, x)
    for _ in range(steps):
        v = v + f / mass * (0.5 * dt)
        s = torch.linalg.solve(H, x + v * dt)
        x = H @ (s - torch.floor(s))
        e, f, w = _exact_force(m, types, h, x)
        v = v + f / mass * (0.5 * dt)
    return x, v, e, f, w


def exact(case, seed):
    m, _ = _model(case["model"])
    n, kind = _atoms(case), case["kind"]
    if n > 210_000 and kind != "batch":     # minutes of pair distances
        return None
    if kind == "force":
        types, h, pos = _system(case, seed)
        return dict(zip(("pe", "force", "virial"), _exact_force(m, types, h, pos)))
    if kind == "batch":
        res = [_exact_force(m, torch.as_tensor(t, device="cuda"), h, torch.as_tensor(p, device="cuda"))
               for t, h, p in _structures(case, seed)]
        return {k: torch.cat([r[q] for r in res], -1) for q, k in enumerate(("pe", "force", "virial"))}
    if kind == "md":
        if case["ensemble"] != "nve" or n * case["steps"] > 1_000_000:
            return None
        t, h, pos, masses, vel = _md_inputs(case, seed)
        x, v, _, f, _ = _exact_nve(m, t, h, pos, masses, vel * TIME_UNIT, case["steps"], case["dt"])
        return dict(thermo=None, pos=x, vel=v, force=f)
    reqs = _segments(case, seed)
    if sum(len(r["types"]) * r["md_steps"] for r in reqs) > 600_000:
        return None
    rows = []
    for r in reqs:
        if r["md_steps"]:
            x, v, e, f, w = _exact_nve(m, r["types"], r["h"], r["pos"], r["masses"],
                                       r["vel"] * TIME_UNIT, r["md_steps"], r["dt_fs"])
            rows.append((e, f, w, x, v / TIME_UNIT))
        else:
            rows.append(_exact_force(m, torch.as_tensor(r["types"], device="cuda"), r["h"],
                                     torch.as_tensor(r["pos"], device="cuda")))
    out = {k: torch.cat([r[q] for r in rows], -1) for q, k in enumerate(("pe", "force", "virial"))}
    moved = [r for r in rows if len(r) > 3]
    out.update({k: torch.cat([r[q] for r in moved], -1) for q, k in ((3, "pos"), (4, "vel"))})
    return out
