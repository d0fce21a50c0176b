"""Performance cases of the engine's public entry points.

Every case is one call (or one short sequence of calls) that a Monte Carlo program makes:
the host-driven trial energies and moves, the FP64 totals of a drift check, batched Widom
insertions and persistent GCMC launches. Systems come from graspa_gb300.synth with the sizes of
the benchmark configurations; the seed of a case sets the adsorbate positions, the trial
configurations and the random stream.

exact() restates each computed call in FP64 torch without the engine.
"""
import copy
import functools
import math

import numpy as np
import torch

from graspa_gb300 import grx, synth

BASE_SEED = 42


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one CBMC first-bead step of a host-driven insertion: the smallest call of the C ABI
        dict(name="trial_co2_first_fp64", op="trial", system="silica", guests=24, prec="fp64", ntrials=10, chain=0),
        # one CBMC orientation step of water in a triclinic channel framework (odd trial count)
        dict(name="trial_water_orient_mixed", op="trial", system="water", guests=16, prec="mixed", ntrials=37, chain=1),
        # one accepted host-driven translation: pair delta, Fourier delta, commit, atom write
        dict(name="move_co2_fp64", op="move", system="silica", guests=24, prec="fp64"),
        # FP64 totals of a drift check, benchmark box
        dict(name="total_co2_silica", op="total", system="silica", guests=24),
        # the same on the largest serving framework (20,000 atoms, automatic Ewald set-up)
        dict(name="total_co2_20000", op="total", system="CO2", natoms=20000, fseed=7, guests=12),
        # Henry coefficient run: batched Widom insertions, production precision
        dict(name="widom_co2_mixed", op="widom", system="silica", guests=0, prec="mixed", n=20000, k=10),
        # the same in FP64 (parity runs against the reference's arithmetic), a loaded box
        dict(name="widom_co2_fp64", op="widom", system="silica", guests=8, prec="fp64", n=1500, k=10),
        # flagship: independent GCMC chains, three per SM, production precision
        dict(name="gcmc_co2_456_mixed", op="gcmc", system="silica", guests=8, prec="mixed", chains=456, steps=50, k=10),
        # charge-dominated water GCMC (Ewald-heavy, reinsertions, triclinic cell)
        dict(name="gcmc_water_456_mixed", op="gcmc", system="water", guests=16, prec="mixed", chains=456, steps=25, k=10),
        # LJ-only mixture GCMC on 64 different triclinic frameworks, 32 trials, clusters of 2
        dict(name="gcmc_ch4_xe_64_mixed", op="gcmc", system="ch4_xe", guests=6, prec="mixed", chains=64, steps=100, k=32),
        # the flagship chains in FP64
        dict(name="gcmc_co2_152_fp64", op="gcmc", system="silica", guests=8, prec="fp64", chains=152, steps=10, k=10),
        # one long chain on a large charged framework, on a cluster of 8 CTAs
        dict(name="gcmc_co2_20000_single", op="gcmc", system="CO2", natoms=20000, fseed=7, guests=12, prec="mixed",
             chains=1, steps=50, k=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["trial", "trial", "move", "total", "widom", "gcmc", "gcmc"])
    system = rng.choice(["silica", "water", "ch4_xe", "CO2", "N2"])
    c = dict(op=op, system=system, guests=rng.randint(2, 24))
    if system in ("CO2", "N2", "ch4_xe"):
        c.update(natoms=_log(rng, 400, 8000), fseed=rng.randint(0, 40))
        c["guests"] = rng.randint(2, 8)
    if op == "trial":
        c.update(prec=rng.choice(["fp64", "mixed"]), ntrials=_log(rng, 4, 64), chain=rng.randint(0, 1))
        if system == "ch4_xe":
            c["chain"] = 0
    elif op == "move":
        c.update(prec=rng.choice(["fp64", "mixed"]))
    elif op == "widom":
        c.update(prec=rng.choice(["fp64", "mixed"]), k=rng.randint(5, 20))
        c.update(n=_log(rng, 50, 1000 if c["prec"] == "fp64" else 5000))
    elif op == "gcmc":
        c.update(prec=rng.choice(["fp64", "mixed", "mixed"]), k=rng.randint(5, 20), chains=_log(rng, 1, 400))
        c.update(steps=_log(rng, 5, 10 if c["prec"] == "fp64" else 30))
    return c


# ------------------------------------------------------------------ systems
TEMPERATURE = 300.0
TOP = 1e100  # weights are reported up to here: point charges that meet give weights whose squares overflow


@functools.lru_cache(maxsize=128)
def _framework(system, natoms, fseed):
    """The empty box of a case (framework, force field, templates); the same for every seed."""
    if system == "silica":
        return synth.silica_co2(seed=BASE_SEED)
    if system == "water":
        return synth.tip4p_hex_system(seed=BASE_SEED)
    if system == "ch4_xe":
        return synth.ch4_xe_system(fseed, n_atoms=natoms)
    return synth.adsorbate_system(system, fseed, n_atoms=natoms)


def _empty(case, i=0):
    natoms = case.get("natoms")
    return _framework(case["system"], natoms, int(case.get("fseed", 0)) + i if natoms is None or i else case["fseed"])


def _loaded(base, guests, seed):
    """`base` with `guests` molecules of every adsorbate (fewer when they do not fit)."""
    s = dict(base)
    g = np.random.Generator(np.random.Philox(int(seed) + 77))
    for c in range(s["nhost"], len(s["comp_start"]) - 1):
        if guests:
            synth.place_molecules(s, c, guests, g, min_dist=2.5, max_tries=300)
    return s


def _capacity(s, molecules=160):
    cs, nh = s["comp_start"], s["nhost"]
    return [cs[c + 1] - cs[c] if c < nh else s["molsize"][c] * molecules for c in range(len(cs) - 1)]


def _box(s):
    b = grx.Box(s, capacity=_capacity(s))
    b.ewald_total()
    return b


def _take_last(s, comp):
    """Removes the last molecule of `comp` from the system; returns (system, its atoms)."""
    s = dict(s)
    ms = s["molsize"][comp]
    end = s["comp_start"][comp + 1]
    if end - s["comp_start"][comp] < ms:
        tm = s["templates"][comp]
        centre = np.array(s["cell"]).reshape(3, 3).T @ np.array([0.5, 0.5, 0.5])
        return s, tm["pos"] - tm["pos"][0] + centre
    mol = s["pos"][end - ms:end].copy()
    for k in ("pos", "type", "charge", "molid", "scale", "scale_coul"):
        s[k] = np.delete(s[k], np.s_[end - ms:end], axis=0)
    s["comp_start"] = [x - (ms if c > comp else 0) for c, x in enumerate(s["comp_start"])]
    return s, mol


def _rotations(g, n):
    q = g.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    w, x, y, z = q.T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                     2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                     2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


@functools.lru_cache(maxsize=8)
def _call_inputs_key(key, seed):
    return _call_inputs_of(dict(key), seed)


def _call_inputs(case, seed):
    """System and trial beads / moved molecule of a trial or move case."""
    return copy.deepcopy(_call_inputs_key(tuple(sorted(case.items())), int(seed)))


def _call_inputs_of(case, seed):
    s = _loaded(_empty(case), case["guests"] + 1, seed)
    comp = s["nhost"]
    s, mol = _take_last(s, comp)
    tm = s["templates"][comp]
    ms = s["molsize"][comp]
    g = np.random.Generator(np.random.Philox(int(seed) + 9001))
    d = dict(system=s, comp=comp, newmol=(s["comp_start"][comp + 1] - s["comp_start"][comp]) // ms)
    if case["op"] == "trial":
        n = case["ntrials"]
        if case["chain"] and ms > 1:  # orientations about the molecule's first bead
            ch = ms - 1
            v = np.einsum("nij,aj->nai", _rotations(g, n), tm["pos"][1:] - tm["pos"][0])
            d.update(pos=(mol[0] + v).reshape(-1, 3), charge=np.tile(tm["charge"][1:], n),
                     type=np.tile(tm["type"][1:], n), ntrials=n, chain=ch)
        else:  # first-bead positions over the cell
            diag = np.array([s["cell"][0], s["cell"][4], s["cell"][8]])
            pos = g.uniform(size=(n, 3)) * diag
            pos[0] = mol[0]
            d.update(pos=pos, charge=np.tile(tm["charge"][:1], n), type=np.tile(tm["type"][:1], n), ntrials=n, chain=1)
    else:  # the molecule sits in the box and is translated
        cs = s["comp_start"]
        s = dict(s)
        for k, v in (("pos", mol), ("type", tm["type"]), ("charge", tm["charge"]), ("molid", np.full(ms, d["newmol"])),
                     ("scale", np.ones(ms)), ("scale_coul", np.ones(ms))):
            s[k] = np.insert(s[k], cs[comp + 1], v, axis=0)
        s["comp_start"] = [x + (ms if c > comp else 0) for c, x in enumerate(cs)]
        d.update(system=s, old=mol, new=mol + g.uniform(-0.3, 0.3, 3), charge=np.asarray(tm["charge"], dtype=float),
                 type=np.asarray(tm["type"]))
    return d


# ------------------------------------------------------------------ prepare / run
def _prec(case):
    return grx.PRECISIONS[case["prec"]]


def prepare(case, seed):
    op = case["op"]
    if op in ("trial", "move"):
        d = _call_inputs(case, seed)
        d.update(op=op, prec=_prec(case), box=_box(d["system"]), beta=grx.beta_from_temperature(TEMPERATURE))
        return d
    if op == "total":
        s = _loaded(_empty(case), case["guests"], seed)
        return dict(op=op, box=grx.Box(s, capacity=_capacity(s)))
    if op == "widom":
        s = _loaded(_empty(case), case["guests"], seed)
        k = case["k"]
        return dict(op=op, box=_box(s), n=case["n"], prec=_prec(case),
                    desc=grx.widom_desc(s, s["nhost"], ntrials=k, norient=k, temperature=TEMPERATURE, seed=int(seed)))
    chains = case["chains"]
    if case["system"] == "ch4_xe":
        bases = [_framework("ch4_xe", case.get("natoms"), int(case.get("fseed", 0)) + i) for i in range(min(chains, 64))]
        # one box per framework; more chains than frameworks are replicas
        parents = [_box(_loaded(b, case["guests"], int(seed) + i)) for i, b in enumerate(bases)]
    else:
        parents = [_box(_loaded(_empty(case), case["guests"], seed))]
    boxes = [parents[i] if i < len(parents) else parents[i % len(parents)].replica() for i in range(chains)]
    k = case["k"]
    pressure = {"water": 3.5e3, "ch4_xe": 1e6}.get(case["system"], 1e5)
    descs = []
    for i, b in enumerate(boxes):
        kw = dict(ntrials=k, norient=k, p_translation=0.25, p_rotation=0.5, p_swap=1.0, temperature=TEMPERATURE,
                  pressure_pa=pressure, seed=int(seed), stream=i)
        if case["system"] == "water":
            kw.update(p_reinsertion=0.75, max_translation=0.5, max_rotation=0.4)
        if case["system"] == "ch4_xe":  # a different trial count per box, as a screening batch has
            kw.update(p_translation=0.3, p_rotation=0.3, p_reinsertion=0.5, norient=1, max_translation=0.7,
                      ntrials=k - (5 * i) % (1 + 3 * k // 4))
        comps = range(b.nhost, b.ncomp)
        descs.append([grx.gcmc_desc(c, **kw) for c in comps])
    batch = grx.GcmcBatch(boxes, descs, prec=_prec(case))
    # the launch shape the autotuner keeps for few boxes: thread-block clusters
    if chains == 1:
        batch.set_cluster(8)
    elif chains <= 64:
        batch.set_cluster(2)
    return dict(op=op, batch=batch, steps=case["steps"], boxes=boxes, parents=parents)


_STATS = np.dtype([("attempts", "i8", 5), ("accepted", "i8", 5), ("n_molecules", "i8"), ("capacity_hits", "i8"),
                   ("energy", "f8", 4), ("sum_n", "f8"), ("identity_out", "i8", 2), ("identity_in", "i8", 2),
                   ("rosen", "f8", 3), ("trial_configs", "i8"), ("trial_beads", "i8")])  # grx.GcmcStats


def _stats(st):
    a = np.frombuffer(b"".join(map(bytes, st)), dtype=_STATS)
    out = {k: a[k].copy() for k in ("attempts", "accepted", "n_molecules", "capacity_hits", "trial_configs", "trial_beads",
                                    "energy", "sum_n", "rosen")}
    out["rosen"] = np.minimum(out["rosen"], TOP)
    return out


def run(state):
    op = state["op"]
    if op == "trial":
        e, flag = state["box"].trial_energies(state["pos"], state["charge"], state["type"], state["newmol"], state["ntrials"],
                                              state["chain"], state["comp"], prec=state["prec"])
        weight = np.where(flag == 0, np.exp(np.minimum(-state["beta"] * e.sum(1), 200.0)), 0.0)
        return {"energy": e, "overlap": flag, "weight": weight}
    if op == "move":
        b, q, ty, comp, mol = state["box"], state["charge"], state["type"], state["comp"], state["newmol"]
        old, new = state["old"], state["new"]
        de, flag = b.single_body(dict(pos=old, charge=q, type=ty, molid=mol), dict(pos=new, charge=q, type=ty, molid=mol), comp,
                                 prec=state["prec"])
        ew = b.ewald_delta(comp, grx.MOVE_TRANSLATION, old, q, new, q)
        b.ewald_commit(comp)
        b.write_molecule(comp, mol, new, q, ty)
        state["old"], state["new"] = new, old  # the next pass moves it back
        return {"pair": de, "overlap": flag, "ewald": ew}
    if op == "total":
        return {k: np.array([v]) for k, v in state["box"].total_energy().items()}
    if op == "widom":
        r = state["box"].widom(state["desc"], 0, state["n"], prec=state["prec"])
        out = {k: r[k] for k in ("e_first", "e_chain", "ewald", "sel_first", "sel_orient", "n_ok_first", "n_ok_orient", "success")}
        out.update((k, np.minimum(r[k], TOP)) for k in ("rosenbluth", "w_first", "w_chain"))
        return out
    state["batch"].launch(state["steps"])
    st, nxt = state["batch"].stats()
    out = _stats(st)
    out["next_step"] = nxt
    if len(state["boxes"]) == 1:  # a single simulation reads its structure factor back
        out["s_ads"] = state["boxes"][0].structure_factors()[1]
    return out


# ------------------------------------------------------------------ work
def _pairs_per_bead(s):
    """Atoms inside the cutoff of a bead at the box's mean density (at most all of them)."""
    cell = np.array(s["cell"]).reshape(3, 3).T
    n = len(s["pos"])
    return min(n, n / abs(np.linalg.det(cell)) * 4.18879 * s["cutoff_vdw"] ** 3)


def _nact(s):
    return len(_kvectors(s)[0]) if not s["no_charges"] else 0


def work(case):
    base = _empty(case)
    s = base if case["op"] != "gcmc" or case["system"] != "ch4_xe" else _framework("ch4_xe", case.get("natoms"),
                                                                                   int(case.get("fseed", 0)))
    ms, natom = s["molsize"][s["nhost"]], len(s["pos"])
    per, nk = _pairs_per_bead(s), _nact(s)
    fl = 40.0 if s["no_charges"] else 70.0  # flops of one pair inside the cutoff (LJ, real Coulomb)
    atom_bytes, k_bytes, kf = 34.0 * natom, 56.0 * nk, 24.0  # flops per (k, atom) of a structure factor
    op = case["op"]
    if op == "trial":
        beads = case["ntrials"] * (ms - 1 if case["chain"] and ms > 1 else 1)
        return {"bytes": atom_bytes + beads * 64, "flops": beads * per * fl}
    if op == "move":
        return {"bytes": atom_bytes + k_bytes + 32.0 * nk, "flops": 2 * ms * per * fl + nk * 2 * ms * kf}
    if op == "total":
        n = natom + case["guests"] * ms
        excl = 0.0 if s["no_charges"] else natom * natom / 2 * 30.0  # erf of every framework pair
        return {"bytes": atom_bytes + k_bytes, "flops": excl + nk * n * kf + case["guests"] * ms * per * fl}
    k = case["k"]
    if op == "widom":
        beads = k + (k * (ms - 1) if ms > 1 else 0)
        return {"bytes": atom_bytes + k_bytes + 136.0 * case["n"], "flops": case["n"] * (beads * per * fl + nk * ms * kf)}
    grow = k + k * (ms - 1)
    beads = 0.5 * 2 * ms + 0.5 * grow
    return {"bytes": (atom_bytes + k_bytes) if case["system"] != "ch4_xe" else atom_bytes * case["chains"],
            "flops": case["chains"] * case["steps"] * (beads * per * fl + nk * 1.5 * ms * kf)}


# ------------------------------------------------------------------ exact
# FP64 torch restatements: minimum image by rounded fractional coordinates, shifted 12-6 LJ,
# erfc Coulomb inside their cutoffs, LAMMPS- or index-cutoff k vectors, rigid exclusions.
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device=DEV)


class _Exact:
    def __init__(self, s):
        self.s = s
        self.h = _t(np.array(s["cell"]).reshape(3, 3).T)
        self.hi = torch.linalg.inv(self.h)
        self.pos, self.q = _t(s["pos"]), _t(np.asarray(s["charge"]) * np.asarray(s["scale_coul"]))
        self.type = torch.as_tensor(np.asarray(s["type"], dtype=np.int64), device=DEV)
        nt = s["ntypes"]
        self.eps, self.sig, self.shift = (_t(np.asarray(s[k]).reshape(nt, nt)) for k in ("epsilon", "sigma", "shift"))
        self.nh = s["comp_start"][s["nhost"]]

    def r2(self, a, b):
        d = b[None, :, :] - a[:, None, :]
        f = d @ self.hi.T
        f -= torch.round(f)
        d = f @ self.h.T
        return (d * d).sum(-1)

    def beads(self, pos, q, ty, skip=None):
        """Per bead {host vdw, host real, guest vdw, guest real} and the overlap flag; `skip`: atoms left out."""
        s = self.s
        out, flags = [], []
        step = max(1, 6_000_000 // max(1, len(self.pos)))
        for a in range(0, len(pos), step):
            p, qb, tb = pos[a:a + step], q[a:a + step], ty[a:a + step]
            rr = self.r2(p, self.pos)
            if skip is not None:
                rr = torch.where(skip[None, :], torch.full_like(rr, 1e30), rr)
            inv = rr < s["cutoff_vdw"] ** 2
            row = (self.type[None, :], tb[:, None])
            t = rr / self.sig[row] ** 2
            i3 = 1.0 / (t * t * t)
            lj = torch.where(inv, 4 * self.eps[row] * (i3 * (i3 - 1.0)) - self.shift[row], torch.zeros_like(rr))
            flags.append((inv & ((lj > s["overlap_criteria"]) | (rr < 0.01))).any(1))
            if s["no_charges"]:
                co = torch.zeros_like(lj)
            else:
                r = torch.sqrt(rr)
                co = torch.where(rr < s["cutoff_coul"] ** 2,
                                 s["prefactor"] * self.q[None, :] * qb[:, None] * torch.erfc(s["alpha"] * r) / r,
                                 torch.zeros_like(rr))
            n = self.nh
            out.append(torch.stack([lj[:, :n].sum(1), co[:, :n].sum(1), lj[:, n:].sum(1), co[:, n:].sum(1)], 1))
        return torch.cat(out), torch.cat(flags)

    def kvec(self):
        k, temp = _kvectors(self.s)
        return torch.as_tensor(k, device=DEV, dtype=torch.float64), _t(temp)

    def sk(self, pos, q, k):
        """S(k) of weighted atoms (real, imaginary)."""
        f = pos @ self.hi.T
        re, im = torch.zeros(len(k), device=DEV, dtype=torch.float64), torch.zeros(len(k), device=DEV, dtype=torch.float64)
        step = max(1, 20_000_000 // max(1, len(k)))
        for a in range(0, len(pos), step):
            ph = 2 * math.pi * torch.remainder(f[a:a + step] @ k.T, 1.0)
            re += q[a:a + step] @ torch.cos(ph)
            im += q[a:a + step] @ torch.sin(ph)
        return re, im

    def molecule_exclusion(self, pos, q):
        """Intramolecular erf sum and self energy of one molecule."""
        s = self.s
        e = 0.0
        n = len(pos)
        step = max(1, 8_000_000 // max(1, n))
        ar = torch.arange(n, device=DEV)
        for a in range(0, n, step):
            r = torch.sqrt(self.r2(pos[a:a + step], pos))
            m = ar[None, :] > ar[a:a + step, None]
            v = s["prefactor"] * q[a:a + step, None] * q[None, :] * torch.erf(s["alpha"] * r) / torch.where(m, r, torch.ones_like(r))
            e += float(torch.where(m, v, torch.zeros_like(v)).sum())
        return e, float((s["prefactor"] * s["alpha"] / math.sqrt(math.pi) * q * q).sum())


def _kvectors(s):
    """Active (kx >= 0) integer k vectors and their Fourier prefactors."""
    h = np.array(s["cell"]).reshape(3, 3).T
    rec = 2 * math.pi * np.linalg.inv(h)  # rows: reciprocal vectors
    km = s["kmax"]
    k = np.stack(np.meshgrid(np.arange(0, km[0] + 1), np.arange(-km[1], km[1] + 1), np.arange(-km[2], km[2] + 1),
                             indexing="ij"), -1).reshape(-1, 3)
    kv = k @ rec
    k2 = (kv * kv).sum(1)
    cut = s.get("reciprocal_cutoff")
    if cut is None:
        cut = max((km[d] * 2 * math.pi / s["cell"][4 * d]) ** 2 for d in range(3)) * 1.00001
    if s.get("use_lammps_ewald", 1):
        act = (k2 > 1e-10) & (k2 < cut)
    else:
        n2 = (k * k).sum(1)
        act = (n2 > 0) & (n2 < cut)
    vol = abs(np.linalg.det(h))
    fac = np.where(k[:, 0] == 0, 1.0, 2.0) * s["prefactor"] * 2 * math.pi / vol
    k2a = np.where(act, k2, 1.0)
    return k[act], (fac * np.exp(-k2a / (4 * s["alpha"] ** 2)) / k2a)[act]


def exact(case, seed):
    op = case["op"]
    beta = grx.beta_from_temperature(TEMPERATURE)
    if op == "trial":
        d = _call_inputs(case, seed)
        X = _Exact(d["system"])
        e, f = X.beads(_t(d["pos"]), _t(d["charge"]), torch.as_tensor(np.asarray(d["type"], dtype=np.int64), device=DEV))
        e = e.reshape(d["ntrials"], d["chain"], 4).sum(1)
        f = f.reshape(d["ntrials"], d["chain"]).any(1)
        w = torch.where(f, torch.zeros_like(e[:, 0]), torch.exp(torch.clamp(-beta * e.sum(1), max=200.0)))
        return {"energy": e.cpu().numpy(), "overlap": None, "weight": w.cpu().numpy()}
    if op == "move":
        d = _call_inputs(case, seed)
        s = d["system"]
        X = _Exact(s)
        skip = torch.zeros(len(X.pos), dtype=torch.bool, device=DEV)
        ms = s["molsize"][d["comp"]]
        end = s["comp_start"][d["comp"] + 1]
        skip[end - ms:end] = True
        q, ty = _t(d["charge"]), torch.as_tensor(np.asarray(d["type"], dtype=np.int64), device=DEV)
        dv = (X.beads(_t(d["new"]), q, ty, skip)[0] - X.beads(_t(d["old"]), q, ty, skip)[0]).sum(0).cpu().numpy()
        ew = np.zeros(2)
        if not s["no_charges"]:
            k, temp = X.kvec()
            hr, hm = X.sk(X.pos[:X.nh], X.q[:X.nh], k)
            ar, am = X.sk(X.pos[X.nh:], X.q[X.nh:], k)
            nr, nm = X.sk(_t(d["new"]), q, k)
            orr, om = X.sk(_t(d["old"]), q, k)
            dr, dm = nr - orr, nm - om
            ew = np.array([float((temp * (2 * (ar * dr + am * dm) + dr * dr + dm * dm)).sum()),
                           2 * float((temp * (hr * dr + hm * dm)).sum())])
        return {"pair": np.concatenate([np.zeros(2), dv]), "overlap": None, "ewald": ew}
    if op == "total":
        s = _loaded(_empty(case), case["guests"], seed)
        return _exact_total(s)
    if op == "widom":
        s = _loaded(_empty(case), case["guests"], seed)
        return _exact_widom(s, case, seed, beta)
    return None


def _exact_total(s):
    X = _Exact(s)
    o = {n: 0.0 for n in ("hh_vdw", "hh_real", "hg_vdw", "hg_real", "gg_vdw", "gg_real", "hh_ewald", "hg_ewald", "gg_ewald")}
    cs, nh = s["comp_start"], s["nhost"]
    for c in range(nh, len(cs) - 1):
        for m in range((cs[c + 1] - cs[c]) // s["molsize"][c]):
            a, b = cs[c] + m * s["molsize"][c], cs[c] + (m + 1) * s["molsize"][c]
            skip = torch.zeros(len(X.pos), dtype=torch.bool, device=DEV)
            skip[a:b] = True
            e = X.beads(X.pos[a:b], X.q[a:b], X.type[a:b], skip)[0].sum(0).cpu().numpy()
            o["hg_vdw"] += e[0]
            o["hg_real"] += e[1]
            o["gg_vdw"] += 0.5 * e[2]
            o["gg_real"] += 0.5 * e[3]
    k, temp = X.kvec() if len(_kvectors(s)[0]) else (None, None)
    f = np.zeros(3)
    if k is not None:
        hr, hm = X.sk(X.pos[:X.nh], X.q[:X.nh], k)
        ar, am = X.sk(X.pos[X.nh:], X.q[X.nh:], k)
        f = np.array([float((temp * (ar * ar + am * am)).sum()), float((temp * (hr * hr + hm * hm)).sum()),
                      2 * float((temp * (hr * ar + hm * am)).sum())])
    excl, self_ = np.zeros(2), np.zeros(2)  # all, host
    for c in range(len(cs) - 1):
        ms = s["molsize"][c]
        for m in range((cs[c + 1] - cs[c]) // ms):
            a, b = cs[c] + m * ms, cs[c] + (m + 1) * ms
            e, v = X.molecule_exclusion(X.pos[a:b], X.q[a:b])
            excl += np.array([e, e if c < nh else 0.0])
            self_ += np.array([v, v if c < nh else 0.0])
    o["hh_ewald"] = f[1] - self_[1] - excl[1]
    o["hg_ewald"] = f[2]
    o["gg_ewald"] = f[0] + f[1] - self_[0] - excl[0]
    out = {n: np.array([float(v)]) for n, v in o.items()}
    if not s["no_charges"] and np.abs(np.array(s["cell"])[[3, 6, 7]]).sum() > 0:
        # framework pairs of a replicated triclinic cell lie exactly half a cell apart: rounding
        # picks the image of their exclusion, so 64 bits alone do not define these two sums
        out["hh_ewald"] = out["gg_ewald"] = None
    return out


def _philox(seed, stream, move, slot):
    """Philox4x32-10 (Salmon et al., SC'11), counter {slot, move, move >> 32, stream}, key = seed: uniforms (..., 4)."""
    move, slot = np.broadcast_arrays(np.asarray(move, dtype=np.uint64), np.asarray(slot, dtype=np.uint64))
    m32 = np.uint64(0xFFFFFFFF)
    c = [slot & m32, move & m32, move >> np.uint64(32), np.full_like(move, stream)]
    k0, k1 = int(seed) & 0xFFFFFFFF, (int(seed) >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return np.stack(c, -1).astype(np.float64) * 2.0 ** -32


def _select(e, f, beta, u):
    """Rosenbluth selection over trials (n, t): (selected, mean weight, trials without overlap)."""
    lw = torch.where(f, torch.full_like(e, -math.inf), -beta * e)
    ok = ~f
    mx = torch.clamp(lw.max(1, keepdim=True).values, min=-1e300)
    ws = torch.where(ok, torch.exp(lw - mx), torch.zeros_like(lw))
    cum = torch.cumsum(ws, 1)
    hit = ok & ~(cum < (u * ws.sum(1))[:, None])
    idx = torch.arange(e.shape[1], device=e.device)
    first = torch.where(hit, idx[None, :], torch.full_like(idx, 10 ** 6)[None, :]).min(1).values
    last = torch.where(ok, idx[None, :], torch.full_like(idx, -1)[None, :]).max(1).values
    sel = torch.clamp(torch.where(first < 10 ** 6, first, last), min=0)
    w = torch.where(ok, torch.exp(lw), torch.zeros_like(lw)).sum(1)
    return sel, w / e.shape[1], (w >= 1e-150) & ok.any(1)


def _exact_widom(s, case, seed, beta):
    X = _Exact(s)
    comp = s["nhost"]
    tm = s["templates"][comp]
    n, k, ms = case["n"], case["k"], s["molsize"][comp]
    per = _pairs_per_bead(s)
    if n * (k * ms) * len(s["pos"]) > 5e9 or per <= 0:
        return None
    ntot = s["comp_start"][comp + 1] - s["comp_start"][comp]
    tpos = s["pos"][s["comp_start"][comp]:s["comp_start"][comp] + ms] if ntot else tm["pos"]
    mv = np.arange(n)
    diag = np.array([s["cell"][0], s["cell"][4], s["cell"][8]])
    u = _philox(seed, 0, mv[:, None], np.arange(k)[None, :])[..., :3]
    usel = _philox(seed, 0, mv, np.full(n, 2048))
    q, ty = _t(tm["charge"]), torch.as_tensor(np.asarray(tm["type"], dtype=np.int64), device=DEV)
    first = _t(u * diag)
    e, f = X.beads(first.reshape(-1, 3), q[:1].expand(n * k), ty[:1].expand(n * k))
    e, f = e.reshape(n, k, 4), f.reshape(n, k)
    sel, w1, ok = _select(e.sum(2), f, beta, _t(usel[:, 0]))
    ok &= w1 > 1e-150
    rows = torch.arange(n, device=DEV)
    zero = torch.zeros(n, device=DEV, dtype=torch.float64)
    e1 = torch.where(ok[:, None], e[rows, sel], torch.zeros_like(e[:, 0]))
    ros = torch.where(ok, w1, zero)
    w_first = ros.clone()
    mol = first[rows, sel][:, None, :].expand(n, ms, 3).clone()
    e2, w_chain = torch.zeros_like(e1), zero.clone()
    if ms > 1:
        uo = _philox(seed, 0, mv[:, None], (1024 + np.arange(k))[None, :])
        uu, vv, ww = (_t(uo[..., j]) for j in range(3))
        q0, q1 = torch.sqrt(1 - uu) * torch.sin(2 * math.pi * vv), torch.sqrt(1 - uu) * torch.cos(2 * math.pi * vv)
        q2, q3 = torch.sqrt(uu) * torch.sin(2 * math.pi * ww), torch.sqrt(uu) * torch.cos(2 * math.pi * ww)
        R = torch.stack([1 - 2 * (q2 * q2 + q3 * q3), 2 * (q1 * q2 - q0 * q3), 2 * (q1 * q3 + q0 * q2),
                         2 * (q1 * q2 + q0 * q3), 1 - 2 * (q1 * q1 + q3 * q3), 2 * (q2 * q3 - q0 * q1),
                         2 * (q1 * q3 - q0 * q2), 2 * (q2 * q3 + q0 * q1), 1 - 2 * (q1 * q1 + q2 * q2)], -1).reshape(n, k, 3, 3)
        v = torch.einsum("nkij,aj->nkai", R, _t(tpos[1:] - tpos[0]))
        beads = mol[:, None, :1, :] + v
        m = n * k
        e, f = X.beads(beads.reshape(-1, 3), q[1:].repeat(m), ty[1:].repeat(m))
        e, f = e.reshape(n, k, ms - 1, 4).sum(2), f.reshape(n, k, ms - 1).any(2)
        sel2, w2, ok2 = _select(e.sum(2), f, beta, _t(usel[:, 1]))
        ok2 &= ok
        e2 = torch.where(ok2[:, None], e[rows, sel2], e2)
        w_chain = torch.where(ok2, w2, zero)
        ok = ok2 & (ros * w_chain > 1e-150)
        ros = torch.where(ok, ros * w_chain, zero)
        mol[:, 1:] = beads[rows, sel2]
    ew = torch.zeros(n, 2, device=DEV, dtype=torch.float64)
    if not s["no_charges"]:
        kv, temp = X.kvec()
        hr, hm = X.sk(X.pos[:X.nh], X.q[:X.nh], kv)
        ar, am = X.sk(X.pos[X.nh:], X.q[X.nh:], kv)
        ex, se = X.molecule_exclusion(_t(tpos), q)
        for a in range(0, n, 2000):
            f = mol[a:a + 2000] @ X.hi.T
            ph = 2 * math.pi * torch.remainder(f @ kv.T, 1.0)
            dr, dm = (q[None, :, None] * torch.cos(ph)).sum(1), (q[None, :, None] * torch.sin(ph)).sum(1)
            ew[a:a + 2000, 0] = (2 * (dr * (temp * ar) + dm * (temp * am)) + temp * (dr * dr + dm * dm)).sum(1) - (ex + se)
            ew[a:a + 2000, 1] = 2 * (dr * (temp * hr) + dm * (temp * hm)).sum(1)
        ew = torch.where(ok[:, None], ew, torch.zeros_like(ew))
        ros = torch.where(ok, ros * torch.exp(-beta * ew.sum(1)), zero)
    c = lambda x: torch.clamp(x, max=TOP).cpu().numpy()  # noqa: E731
    return {"rosenbluth": c(ros), "w_first": c(w_first), "w_chain": c(w_chain), "e_first": c(e1), "e_chain": c(e2),
            "ewald": c(ew), "sel_first": None, "sel_orient": None, "n_ok_first": None, "n_ok_orient": None, "success": None}
