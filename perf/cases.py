"""Performance cases of the nonbonded library: the calls a simulation program makes.

Each case goes through the public interface (``gromos_nb`` and, for the
allocation-free pair loop, the C ABI), over the sizes of the benchmark and the
tests: from a 343-water box, where launches and latency count, over solvated
solutes of a few thousand waters, to 30,000 waters and to batches of 21
systems.  ``exact`` restates the same physics in plain FP64 torch.
"""
import ctypes as C
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gromos-rs_b200"))

from gromos_nb import _lib, generators  # noqa: E402
from gromos_nb.energy import EnergyParams, trajectory_energies  # noqa: E402
from gromos_nb.nonbonded import Batch, CRFParameters, Forcefield, lj_crf_innerloop  # noqa: E402
from gromos_nb.remd import ReplicaExchange  # noqa: E402
from gromos_nb.serving import Job, NativeServer  # noqa: E402
from gromos_nb.system import NonbondedParams, System  # noqa: E402

NSNB = 5            # pairlist period of every workload of the benchmark
DT = 0.002          # ps
TAU = 0.1           # Berendsen coupling time, ps
EPSRF = 61.0
OPS_PER_PAIR = 37   # FP32 operations of one atom pair (the benchmark's convention)


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # a host integrator calling the force field every step (one pairlist period of steps, host
        # positions in, host forces out): the smallest periodic box of the tests
        {"name": "apply_water_343", "kind": "apply", "waters": 343, "solute": 0, "rcutp": 0.8, "rcutl": 1.0,
         "pinned": False},
        # ... a solvated molecule: multi-atom solute charge groups, twin range
        {"name": "apply_solute_5000", "kind": "apply", "waters": 5000, "solute": 200, "rcutp": 0.8, "rcutl": 1.4,
         "pinned": False},
        # ... the benchmark's large box, host buffers in pinned memory
        {"name": "apply_water_30000", "kind": "apply", "waters": 30000, "solute": 0, "rcutp": 0.8, "rcutl": 1.4,
         "pinned": True},
        # device-resident MD between two analysis points: a small single-range box,
        {"name": "md_water_1000", "kind": "md", "waters": 1000, "solute": 0, "rcutp": 1.4, "rcutl": 1.4, "steps": 20},
        # an ordinary solvated system,
        {"name": "md_ions_3000", "kind": "md", "waters": 3000, "solute": 200, "rcutp": 1.4, "rcutl": 1.4, "steps": 20},
        # and the benchmark's large twin-range box
        {"name": "md_water_30000", "kind": "md", "waters": 30000, "solute": 0, "rcutp": 0.8, "rcutl": 1.4,
         "steps": 20},
        # free-energy windows in one batch (the benchmark's 21 lambdas), dH/dlambda of every window
        {"name": "fep_21x5000", "kind": "fep", "members": 21, "waters": 5000, "solute": 30, "steps": 10},
        # temperature replica exchange: one exchange interval
        {"name": "remd_8x1500", "kind": "remd", "members": 8, "waters": 1500, "solute": 200, "steps": 20},
        # jobs of uneven size through the job server, submit to result
        {"name": "serve_6", "kind": "serve", "members": 6, "waters": 2500, "solute": 100, "steps": 40},
        # energies of a trajectory's frames (analysis)
        {"name": "energies_16x3000", "kind": "energies", "frames": 16, "waters": 3000, "solute": 60, "periodic": True},
        # the explicit pair-list inner loop: on host arrays (the C stub's call),
        {"name": "pairs_host_1000", "kind": "pairs", "waters": 1000, "types": 3, "cutoff": 1.0, "device": False},
        # and on device buffers without allocation
        {"name": "pairs_device_10000", "kind": "pairs", "waters": 10000, "types": 20, "cutoff": 1.0, "device": True},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["apply", "apply", "md", "md", "fep", "remd", "serve", "energies", "pairs"])
    if kind in ("apply", "md"):
        waters = size(300, 25000)
        solute = 0 if rng.random() < 0.5 else size(6, 400)
        rcutl = round(rng.uniform(1.0, 1.4), 2)
        rcutp = 0.8 if waters > 8000 or rng.random() < 0.5 else rcutl
        c = {"kind": kind, "waters": waters, "solute": solute, "rcutp": rcutp, "rcutl": rcutl}
        c.update({"pinned": rng.random() < 0.5} if kind == "apply" else {"steps": 5 * rng.randint(2, 4)})
        return c
    if kind == "fep":
        members = rng.randint(3, 21)
        return {"kind": kind, "members": members, "waters": size(500, min(5000, 60000 // members)),
                "solute": rng.randint(5, 40), "steps": 10}
    if kind == "remd":
        members = rng.randint(3, 12)
        return {"kind": kind, "members": members, "waters": size(400, min(4000, 24000 // members)),
                "solute": size(20, 250), "steps": 5 * rng.randint(2, 4)}
    if kind == "serve":
        return {"kind": kind, "members": rng.randint(2, 6), "waters": size(400, 2500), "solute": size(10, 150),
                "steps": rng.randint(15, 40)}
    if kind == "energies":
        frames = rng.randint(1, 24)
        return {"kind": kind, "frames": frames, "waters": size(300, min(6000, 60000 // frames)),
                "solute": 0 if rng.random() < 0.4 else size(5, 100), "periodic": rng.random() < 0.8}
    return {"kind": "pairs", "waters": size(100, 6000), "types": rng.randint(2, 60),
            "cutoff": round(rng.uniform(0.8, 1.2), 2), "device": rng.random() < 0.6}


# ---- inputs ------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _base(waters, solute, multi_cg, perturbed):
    """A seeded structure of this size; every case's inputs are seeded variations of one."""
    if solute == 0:
        return generators.spc_water_system(waters, generators.box_for_waters(waters), seed=17)
    return generators.solvated_solute_system(waters, solute, seed=17, perturbed=perturbed,
                                             single_atom_cgs=not multi_cg)


def _molecules(topo):
    return np.repeat(np.arange(topo.n_cg), np.diff(topo.cg_offsets))


def _vary(base, seed):
    """Positions of another snapshot of ``base``: the box's axes permuted and reflected, everything
    shifted, every charge group displaced rigidly, the solvent molecules renumbered."""
    rng = np.random.default_rng(seed)
    t, box = base.topo, float(base.box[0])
    x = base.pos[:, rng.permutation(3)]
    flip = rng.random(3) < 0.5
    x = np.where(flip, box - x, x) + rng.uniform(-0.5, 0.5, 3) * box
    x = x + rng.normal(0.0, 0.002, (t.n_cg, 3))[_molecules(t)]
    nsa = t.n_solute_atoms
    w = x[nsa:].reshape(-1, 3, 3)
    return np.concatenate([x[:nsa], w[rng.permutation(len(w))].reshape(-1, 3)])


def _system(case, seed, multi_cg=False, perturbed=False, waters=None, lam=0.0):
    base = _base(waters or case["waters"], case["solute"], multi_cg, perturbed)
    p = NonbondedParams(rcutp=case.get("rcutp", 1.4), rcutl=case.get("rcutl", 1.4), epsrf=EPSRF, nsnb=NSNB, lam=lam)
    return System(topo=base.topo, pos=_vary(base, seed), box=base.box.copy(), params=p)


def _apply_frames(case, seed):
    """One pairlist period of positions: every charge group drifts with a thermal velocity."""
    s = _system(case, seed, multi_cg=True)
    rng = np.random.default_rng([seed, 1])
    v = rng.normal(0.0, 0.37, (s.topo.n_cg, 3))[_molecules(s.topo)]   # sqrt(kT / 18 amu) at 300 K, nm/ps
    return s, [s.pos + k * DT * v for k in range(NSNB)]


def _md_start(case, seed, k=0, T=300.0, **kw):
    s = _system(case, [seed, k], **kw)
    m = generators.masses(s)
    return s, m, generators.maxwell_velocities(m, T, (seed * 1009 + k) % (1 << 31))


def _member(s, mass, vel, T):
    ff = Forcefield(s)
    ff.upload_positions(s.pos)
    ff.md_init(mass, vel, dt=DT, settle=True, dist_oh=generators.OH, dist_hh=generators.SPC_DHH, temperature=T,
               tau=TAU)
    return ff


def _lambdas(case):
    return [round(k / (case["members"] - 1), 3) for k in range(case["members"])]


def _ladder(case):
    return [300.0 * (450.0 / 300.0) ** (k / (case["members"] - 1)) for k in range(case["members"])]


def _jobs(case, seed):
    jobs = []
    for k in range(case["members"]):
        n = max(300, case["waters"] * (k + 1) // case["members"])
        sub = dict(case, solute=case["solute"] if k % 2 else 0)
        s, m, v = _md_start(sub, seed, k, waters=n)
        steps = max(10, case["steps"] * (case["members"] - k) // case["members"])
        jobs.append(Job(job_id=k, system=s, n_steps=steps, mass=m, vel=v, temperature=300.0, tau=TAU))
    return jobs


def _trajectory(case, seed):
    base = _base(case["waters"], case["solute"], True, False)
    fr = np.stack([_vary(base, [seed, f]) for f in range(case["frames"])])
    if not case["periodic"]:
        return base.topo, fr, None
    rng = np.random.default_rng([seed, 2])
    return base.topo, fr, base.box * (1.0 + rng.uniform(0.0, 0.004, (case["frames"], 1)))


def _pair_inputs(case, seed):
    """A typed fluid and its pair list: i-major, j ascending, as a pairlist loop writes it."""
    s = _system(dict(case, solute=0), seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng([seed, 3])
    n, box, T = s.topo.n_atoms, float(s.box[0]), case["types"]
    x = torch.tensor(s.pos, dtype=torch.float32, device=dev)
    mol = torch.arange(n, device=dev) // 3
    rows = []
    for a in range(0, n, 1024):
        d = x[a:a + 1024, None, :] - x[None, :, :]
        d -= box * torch.round(d / box)
        ok = (d * d).sum(-1) <= case["cutoff"] ** 2
        ok &= (torch.arange(n, device=dev)[None, :] > torch.arange(a, min(n, a + 1024), device=dev)[:, None])
        ok &= mol[None, :] != mol[a:a + 1024, None]
        ij = ok.nonzero()
        ij[:, 0] += a
        rows.append(ij.to(torch.int32))
    pairs = torch.cat(rows)
    iac = np.zeros(n, dtype=np.uint32)                      # type 0: hydrogens, no Lennard-Jones
    iac[::3] = 1 + rng.integers(0, T - 1, (n + 2) // 3)
    c6 = np.concatenate([[0.0], generators.SPC_C6 * rng.uniform(0.5, 2.0, T - 1)])
    c12 = np.concatenate([[0.0], generators.SPC_C12 * rng.uniform(0.5, 2.0, T - 1)])
    lj = np.stack([np.sqrt(np.outer(c6, c6)), np.sqrt(np.outer(c12, c12))], axis=-1)
    q = s.topo.charge.astype(np.float32)
    return x, torch.from_numpy(q).to(dev), torch.from_numpy(iac.view(np.int32)).to(dev), pairs, lj, s.box


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind == "apply":
        s, frames = _apply_frames(case, seed)
        st["ff"] = Forcefield(s)
        st["out"] = [None] * NSNB
        if case["pinned"]:
            frames = [torch.from_numpy(f).pin_memory().numpy() for f in frames]
            st["out"] = [torch.empty((s.topo.n_atoms, 3), dtype=torch.float64, pin_memory=True).numpy()
                         for _ in range(NSNB)]
        st["frames"] = frames
    elif kind == "md":
        st["ff"] = _member(*_md_start(case, seed), 300.0)
        st["steps"] = case["steps"]
    elif kind == "fep":
        st["batch"], st["steps"] = Batch(), case["steps"]
        s, m, v = _md_start(case, seed, perturbed=True)
        st["members"] = []
        for lam in _lambdas(case):
            w = s.copy()
            w.params.lam = lam
            st["members"].append(_member(w, m, v, 300.0))
            st["batch"].add(st["members"][-1])
    elif kind == "remd":
        T = _ladder(case)
        st["members"] = [_member(*_md_start(case, seed, k, T=T[k]), T[k]) for k in range(case["members"])]
        st["remd"] = ReplicaExchange(st["members"], T, exchange_interval=case["steps"], seed=seed % (1 << 31))
        st["steps"] = case["steps"]
    elif kind == "serve":
        st["server"], st["jobs"] = NativeServer(hbm_budget=20 << 30, chunk_steps=5), _jobs(case, seed)
    elif kind == "energies":
        st["topo"], st["frames"], st["boxes"] = _trajectory(case, seed)
    else:
        x, q, iac, pairs, lj, box = _pair_inputs(case, seed)
        crf = CRFParameters.new(case["cutoff"], 1.0, EPSRF, 0.0)
        if case["device"]:
            f64 = dict(dtype=torch.float64, device=x.device)
            st["args"] = (x, q, iac, pairs, torch.tensor(lj, **f64), crf, np.ascontiguousarray(box))
            st["forces"] = torch.empty_like(x)
            st["e"], st["v"] = torch.empty(2, **f64), torch.empty(9, **f64)
            st["kind"] = "pairs_device"
        else:
            st["args"] = (x.cpu().numpy(), q.cpu().numpy(), iac.cpu().numpy().view(np.uint32),
                          pairs.cpu().numpy().view(np.uint32), lj, crf, np.ascontiguousarray(box))
    return st


# ---- one pass ----------------------------------------------------------------
def _stats(m, *first):
    st = m.md_stats()
    return [*first, st["e_lj"], st["e_crf"], st["e_kin"]]


def run(st):
    kind = st["kind"]
    if kind == "apply":
        r = [st["ff"].apply(x, count_pairs=False, out=o) for x, o in zip(st["frames"], st["out"])]
        return {"forces": [k["forces"] for k in r], "virial": np.stack([k["virial"] for k in r]),
                "groups": np.array([[k["egroup_lj"], k["egroup_crf"]] for k in r]),
                "total": np.array([[k["e_lj"], k["e_crf"]] for k in r])}
    if kind == "md":
        r = st["ff"].md_run(st["steps"])
        x, v = st["ff"].md_state()
        return {"pos": x, "vel": v, "energies": np.array([r["e_lj"], r["e_crf"], r["e_kin"]])}
    if kind == "fep":
        st["batch"].md_run(st["steps"])
        state = [m.md_state() for m in st["members"]]
        e = [_stats(m, m.result()["dhdl"]) for m in st["members"]]
        return {"pos": [s[0] for s in state], "vel": [s[1] for s in state],
                "dhdl": np.array([k[0] for k in e]), "energies": np.array([k[1:] for k in e])}
    if kind == "remd":
        st["remd"].run(st["steps"])
        state = [m.md_state() for m in st["members"]]
        return {"pos": [s[0] for s in state], "vel": [s[1] for s in state], "at": np.array(st["remd"].at),
                "energies": np.array([_stats(m) for m in st["members"]])}
    if kind == "serve":
        srv, jobs = st["server"], st["jobs"]
        srv.run(jobs)
        for j in jobs:  # results are read: the server may forget the job
            _lib.check(srv._L.gr_server_release(srv._h, srv.ids[j.job_id]))
        return {"pos": [j.result_pos for j in jobs], "vel": [j.result_vel for j in jobs],
                "steps": np.array([j.steps_done for j in jobs])}
    if kind == "energies":
        r = trajectory_energies(st["topo"], st["frames"], st["boxes"], EnergyParams())
        return {"energies": np.array([[e.lj, e.crf] for e in r])}
    if kind == "pairs":
        x, q, iac, pairs, lj, crf, box = st["args"]
        f, e_lj, e_crf, vir = lj_crf_innerloop(x, q, iac, pairs, lj, crf, box)
        return {"forces": f, "energies": np.array([e_lj, e_crf]), "virial": vir}
    x, q, iac, pairs, lj, crf, box = st["args"]
    _lib.check(_lib.lib().gr_lj_crf_innerloop_noalloc(
        x.data_ptr(), q.data_ptr(), iac.data_ptr(), x.shape[0], pairs.data_ptr(), pairs.shape[0], lj.data_ptr(),
        lj.shape[0], box.ctypes.data_as(C.c_void_p), 1, crf.crf_cut, crf.crf_2cut3i, crf.crf_cut3i,
        st["forces"].data_ptr(), st["e"].data_ptr(), st["v"].data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    return {"forces": st["forces"], "energies": st["e"], "virial": st["v"].view(3, 3)}


# ---- what a pass cannot do without ------------------------------------------
def _cg_pairs(n, volume, r):
    return 0.5 * n * min(n - 1.0, n / volume * 4.18879 * r ** 3)


def _step_work(case, waters, solute, steps, rebuilds, rcutp, rcutl):
    """Atom pairs of `steps` evaluations with `rebuilds` long-range refreshes, from the density."""
    vol = (waters + solute / 3.0) / 33.4
    short = 9.0 * _cg_pairs(waters, vol, rcutp) + 3.0 * solute * min(waters, waters / vol * 4.18879 * rcutp ** 3)
    total = 9.0 * _cg_pairs(waters, vol, rcutl) + 3.0 * solute * min(waters, waters / vol * 4.18879 * rcutl ** 3)
    return steps * short + rebuilds * (total - short if rcutp < rcutl else 0.0)


def work(case):
    kind = case["kind"]
    n = 3 * case["waters"] + case.get("solute", 0)
    rp, rl = case.get("rcutp", 1.4), case.get("rcutl", 1.4)
    if kind == "pairs":
        pairs = 4.5 * _cg_pairs(case["waters"], case["waters"] / 33.4, case["cutoff"]) * 2.0
        return {"bytes": 8.0 * pairs + 32.0 * n, "flops": OPS_PER_PAIR * pairs}
    if kind == "apply":
        p = _step_work(case, case["waters"], case["solute"], NSNB, 1, rp, rl)
        return {"bytes": 48.0 * n * NSNB, "flops": OPS_PER_PAIR * p}
    if kind == "energies":
        p = _step_work(case, case["waters"], case["solute"], 1, 0, 1.4, 1.4)
        return {"bytes": 24.0 * n * case["frames"], "flops": OPS_PER_PAIR * p * case["frames"]}
    if kind == "serve":
        b = f = 0.0
        for k in range(case["members"]):
            w = max(300, case["waters"] * (k + 1) // case["members"])
            sol = case["solute"] if k % 2 else 0
            steps = max(10, case["steps"] * (case["members"] - k) // case["members"])
            b += 96.0 * (3 * w + sol)
            f += OPS_PER_PAIR * _step_work(case, w, sol, steps, 0, 1.4, 1.4)
        return {"bytes": b, "flops": f}
    m = case.get("members", 1)
    p = m * _step_work(case, case["waters"], case["solute"], case["steps"], case["steps"] / NSNB, rp, rl)
    return {"bytes": 96.0 * n * m, "flops": OPS_PER_PAIR * p}


def tolerance(case):
    """FP32 pair arithmetic summed in fixed point (the pair loop: FP32 sums), where forces measure up to
    3.6e-6 against exact(); in MD the rounding of the forces grows over the steps (velocities up to 1e-5
    after a job's 40).  About four times that."""
    return {"rel": 5e-5 if case["kind"] == "serve" else 2e-5}


# ---- the same in FP64 --------------------------------------------------------
KB = 0.00831446261815324


class _Reference:
    """Charge-group twin-range nonbonded evaluation, plain torch FP64."""

    def __init__(self, topo, box, rcutp, rcutl, epsrf, lam=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = self.t = topo
        self.box = None if box is None else self.f(box)
        self.c2s, self.c2l, self.twin = rcutp * rcutp, rcutl * rcutl, rcutp < rcutl - 1e-10
        crf = 2.0 * (1.0 - epsrf) / (1.0 + 2.0 * epsrf)
        self.cut = (1.0 - crf / 2.0) / rcutl
        self.k3 = crf / rcutl ** 3
        self.k2 = self.k3 / 2.0
        self.cutoff2 = rcutl * rcutl
        self.off = torch.tensor(t.cg_offsets, device=self.dev, dtype=torch.int64)
        self.q, self.iac = self.f(t.charge), torch.tensor(t.iac, device=self.dev, dtype=torch.int64)
        self.lj, self.fpe = self.f(t.lj[:, :, :2]), t.four_pi_eps_i
        self.G = max(1, int(t.n_egroups))
        eg = np.zeros(t.n_atoms, dtype=np.int64) if t.egroup is None else t.egroup
        self.eg = torch.tensor(eg, device=self.dev, dtype=torch.int64)
        self.grouped = box is None or float(min(box)) * 0.5 > rcutl + 0.3
        self.lam = lam
        a = np.repeat(np.arange(t.n_atoms), np.diff(t.excl_off))
        keep = t.excl > a
        self.ex = torch.tensor(np.stack([a[keep], t.excl[keep]]), device=self.dev, dtype=torch.int64)

    def f(self, x):
        return torch.tensor(np.asarray(x), dtype=torch.float64, device=self.dev)

    def image(self, d):
        return d if self.box is None else d - self.box * torch.round(d / self.box)

    def build(self, x):
        """Charge-group pairs (i < j) of the short and the long range."""
        nsc, n = self.t.n_solute_cg, self.t.n_cg
        ref = x[self.off[:-1]].clone()
        if nsc:
            cg = torch.repeat_interleave(torch.arange(n, device=self.dev), self.off[1:] - self.off[:-1])
            s = torch.zeros_like(ref).index_add_(0, cg, x) / (self.off[1:] - self.off[:-1])[:, None]
            ref[:nsc] = s[:nsc]
        short, far = [], []
        step = max(1, 30_000_000 // n)
        for a in range(0, n, step):
            d2 = torch.zeros((len(ref[a:a + step]), n), dtype=torch.float64, device=self.dev)
            for k in range(3):
                d = ref[a:a + step, None, k] - ref[None, :, k]
                if self.box is not None:
                    d -= self.box[k] * torch.round(d / self.box[k])
                d2 += d * d
            d2.masked_fill_(torch.arange(n, device=self.dev)[None, :] <=
                            torch.arange(a, a + len(d2), device=self.dev)[:, None], 1e30)
            p = (d2 <= self.c2l).nonzero()
            lr = d2[p[:, 0], p[:, 1]] > self.c2s
            p[:, 0] += a
            short.append(p[~lr])
            far.append(p[lr])
        self.lists = [torch.cat(short), torch.cat(far)]

    def atoms(self, p):
        """Atom pairs of charge-group pairs, and the pair's first atoms."""
        ni, nj = self.off[p[:, 0] + 1] - self.off[p[:, 0]], self.off[p[:, 1] + 1] - self.off[p[:, 1]]
        m = ni * nj
        w = torch.repeat_interleave(torch.arange(len(p), device=self.dev), m)
        k = torch.arange(len(w), device=self.dev) - (torch.cumsum(m, 0) - m)[w]
        i0, j0 = self.off[p[:, 0]][w], self.off[p[:, 1]][w]
        return i0 + k // nj[w], j0 + k % nj[w], i0, j0

    def empty(self, x):
        return [torch.zeros_like(x), torch.zeros((2, self.G, self.G), dtype=torch.float64, device=self.dev),
                torch.zeros((3, 3), dtype=torch.float64, device=self.dev)]

    def groups(self, e, k, i, j, v):
        gi, gj = self.eg[i], self.eg[j]
        e[k].view(-1).index_add_(0, torch.minimum(gi, gj) * self.G + torch.maximum(gi, gj), v)

    def add(self, acc, i, j, r, fs, e_lj, e_crf):
        f = r * fs[:, None]
        acc[0].index_add_(0, i, f)
        acc[0].index_add_(0, j, -f)
        if e_lj is not None:
            self.groups(acc[1], 0, i, j, e_lj)
        if e_crf is not None:
            self.groups(acc[1], 1, i, j, e_crf)
        acc[2] += r.T @ f

    def listed_pairs(self, x, far):
        acc = self.empty(x)
        for p in torch.split(self.lists[1 if far else 0], 1_000_000):
            i, j, i0, j0 = self.atoms(p)
            r = x[i] - x[j]
            per_atom = self.image(r)
            if not far:  # one image per charge-group pair where the short-range rules say so
                d0 = x[i0] - x[j0]
                shifted = r + (self.image(d0) - d0)
                solvent = (i >= self.t.n_solute_atoms)[:, None]
                per_atom = torch.where(solvent | self.grouped, shifted, per_atom)
            r = per_atom
            r2 = (r * r).sum(1)
            c = self.lj[self.iac[i], self.iac[j]]
            i6 = 1.0 / r2 ** 3
            ir = 1.0 / torch.sqrt(r2)
            q = self.q[i] * self.q[j] * self.fpe
            fs = (12.0 * c[:, 1] * i6 - 6.0 * c[:, 0]) * i6 / r2 + q * (ir / r2 + self.k3)
            self.add(acc, i, j, r, fs, (c[:, 1] * i6 - c[:, 0]) * i6, q * (ir - self.k2 * r2 - self.cut))
        return acc

    def excluded(self, x, acc):
        nsa = self.t.n_solute_atoms
        s = torch.arange(nsa, device=self.dev)
        self.groups(acc[1], 1, s, s, -0.5 * self.q[:nsa] ** 2 * self.fpe * self.cut)
        i, j = self.ex
        r = self.image(x[i] - x[j])
        r2, q = (r * r).sum(1), self.q[i] * self.q[j] * self.fpe
        sol = (i < nsa).double()
        self.add(acc, i, j, r, sol * q * self.k3, None, -q * self.k2 * r2 - sol * q * self.cut)

    def perturbed(self, x, acc):
        """Soft-core corrections of pairs whose first atom is perturbed, and the self terms (NLAM 1,
        one atom per solute charge group).  Returns dH/dlambda."""
        t, lam = self.t, self.lam
        qa, qb = self.f(t.pert_a_q), self.f(t.pert_b_q)
        ia, ib = (torch.tensor(v, device=self.dev, dtype=torch.int64) for v in (t.pert_a_iac, t.pert_b_iac))
        alj, acrf = float(t.pert_alpha_lj[0]), float(t.pert_alpha_crf[0])
        npert = len(qa)
        Qa, Qb, Ia, Ib = self.q.clone(), self.q.clone(), self.iac.clone(), self.iac.clone()
        Qa[:npert], Qb[:npert], Ia[:npert], Ib[:npert] = qa, qb, ia, ib
        p = torch.cat(self.lists)
        p = p[p[:, 0] < t.n_solute_cg]
        i, j, _, _ = self.atoms(p)
        r = self.image(x[i] - x[j])
        r2 = (r * r).sum(1)
        la, lb = self.lj[Ia[i], Ia[j]], self.lj[Ib[i], Ib[j]]
        q_a, q_b = Qa[i] * Qa[j], Qb[i] * Qb[j]
        A, B = 1.0 - lam, lam

        def state(c, q, soft):
            c126 = torch.where(c[:, 0].abs() > 1e-10, c[:, 1] / c[:, 0].clamp_min(1e-300), torch.zeros_like(r2))
            d2 = r2 + acrf * soft ** 2
            di = 1.0 / torch.sqrt(d2)
            d6 = 1.0 / (r2 ** 3 + alj * soft ** 2 * c126)
            cs2 = self.cutoff2 + acrf * soft ** 2
            k2 = self.k2 / math.sqrt(cs2 ** 3)
            e_lj = (c[:, 1] * d6 - c[:, 0]) * d6
            e_crf = q * (di - k2 * r2 - self.cut)
            force = q * (di / d2 + 2.0 * k2) * self.fpe + (12.0 * c[:, 1] * d6 - 6.0 * c[:, 0]) * d6 * d6 * r2 ** 2
            s_lj = soft * c126 * d6 * d6 * (2.0 * c[:, 1] * d6 - c[:, 0])
            s_crf = q * soft * (di / d2 - 3.0 * k2 / cs2 * r2)
            return e_lj, e_crf, force, s_lj, s_crf

        ea, eb = state(la, q_a, B), state(lb, q_b, A)
        dhdl = (-2.0 * alj * (A * ea[3] - B * eb[3]) + eb[0] - ea[0]
                - (A * ea[4] - B * eb[4]) * self.fpe * acrf + (eb[1] - ea[1]) * self.fpe).sum()
        i6, ir = 1.0 / r2 ** 3, 1.0 / torch.sqrt(r2)
        qf = q_a * self.fpe
        f0 = (12.0 * la[:, 1] * i6 - 6.0 * la[:, 0]) * i6 / r2 + qf * (ir / r2 + self.k3)
        lj0, crf0 = (la[:, 1] * i6 - la[:, 0]) * i6, qf * (ir - self.k2 * r2 - self.cut)
        self.add(acc, i, j, r, A * ea[2] + B * eb[2] - f0, A * ea[0] + B * eb[0] - lj0,
                 (A * ea[1] + B * eb[1]) * self.fpe - crf0)
        s = torch.arange(npert, device=self.dev)
        self.groups(acc[1], 1, s, s, 0.5 * (qa ** 2 - A * qa ** 2 - B * qb ** 2) * self.cut * self.fpe)
        return float(dhdl + 0.5 * ((qa ** 2 - qb ** 2) * self.cut * self.fpe).sum())

    def apply(self, x, rebuild):
        """Forces, group energies and virial of one step of the twin-range scheme."""
        if rebuild:
            self.build(x)
            self.cache = self.listed_pairs(x, True) if self.twin else None
        acc = self.listed_pairs(x, False)
        self.excluded(x, acc)
        self.dhdl = self.perturbed(x, acc) if self.lam is not None else 0.0
        if self.cache is not None:
            acc = [a + b for a, b in zip(acc, self.cache)]
        return acc


class _Dynamics:
    """Leap-frog with a Berendsen bath; rigid solvent by Newton iteration on the three distances."""

    def __init__(self, s, mass, vel, T, lam=None):
        self.ff = _Reference(s.topo, s.box, s.params.rcutp, s.params.rcutl, s.params.epsrf, lam)
        self.x, self.v, self.m = self.ff.f(s.pos), self.ff.f(vel), self.ff.f(mass)[:, None]
        self.T, self.nsa, self.n, self.k = T, s.topo.n_solute_atoms, len(mass), 0
        self.ke = float(0.5 * (self.m * self.v ** 2).sum())
        self.dof = 3.0 * self.n - (self.n - self.nsa)

    def constrain(self, old, new):
        d2 = self.ff.f([generators.OH ** 2, generators.OH ** 2, generators.SPC_DHH ** 2])
        I, J = [0, 0, 1], [1, 2, 2]
        im = 1.0 / self.m[self.nsa:self.nsa + 3, 0]
        o = old[:, I] - old[:, J]
        # displacement of bond c per unit multiplier of bond k
        W = torch.zeros((3, 3), dtype=torch.float64, device=o.device)
        for c in range(3):
            for k in range(3):
                for a, s in ((I[c], 1.0), (J[c], -1.0)):
                    W[c, k] += s * im[a] * ((a == I[k]) * 1.0 - (a == J[k]) * 1.0)
        for _ in range(8):
            b = new[:, I] - new[:, J]
            res = (b * b).sum(-1) - d2
            M = 2.0 * torch.einsum("ncd,nkd->nck", b, o) * W
            g = torch.linalg.solve(M, -res.unsqueeze(-1)).squeeze(-1)
            step = torch.zeros_like(new)
            for k in range(3):
                step[:, I[k]] += im[I[k]] * g[:, k, None] * o[:, k]
                step[:, J[k]] -= im[J[k]] * g[:, k, None] * o[:, k]
            new = new + step
        return new

    def run(self, steps):
        for _ in range(steps):
            f, self.e, _ = self.ff.apply(self.x, self.k % NSNB == 0)
            t = 2.0 * self.ke / (self.dof * KB)
            scale = math.sqrt(1.0 + DT / TAU * (self.T / t - 1.0))
            v = (self.v + f / self.m * DT) * scale
            new = self.x + v * DT
            if self.nsa < self.n:
                fixed = self.constrain(self.x[self.nsa:].view(-1, 3, 3), new[self.nsa:].view(-1, 3, 3)).view(-1, 3)
                v[self.nsa:] += (fixed - new[self.nsa:]) / DT
                new[self.nsa:] = fixed
            self.x, self.v, self.k = new, v, self.k + 1
            self.ke = float(0.5 * (self.m * v ** 2).sum())

    def energies(self):
        e = self.e.sum((1, 2)).tolist()
        return [e[0], e[1], self.ke]


def _np(x):
    return x.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "apply":
        s, frames = _apply_frames(case, seed)
        ff = _Reference(s.topo, s.box, s.params.rcutp, s.params.rcutl, EPSRF)
        r = [ff.apply(ff.f(x), k == 0) for k, x in enumerate(frames)]
        return {"forces": [_np(k[0]) for k in r], "virial": np.stack([_np(k[2]) for k in r]),
                "groups": np.stack([_np(k[1]) for k in r]), "total": np.stack([_np(k[1].sum((1, 2))) for k in r])}
    if kind == "md":
        d = _Dynamics(*_md_start(case, seed), 300.0)
        d.run(case["steps"])
        return {"pos": _np(d.x), "vel": _np(d.v), "energies": np.array(d.energies())}
    if kind == "fep":
        s, m, v = _md_start(case, seed, perturbed=True)
        ds = [_Dynamics(s, m, v, 300.0, lam) for lam in _lambdas(case)]
        for d in ds:
            d.run(case["steps"])
        return {"pos": [_np(d.x) for d in ds], "vel": [_np(d.v) for d in ds],
                "dhdl": np.array([d.ff.dhdl for d in ds]), "energies": np.array([d.energies() for d in ds])}
    if kind == "remd":
        T = _ladder(case)
        ds = [_Dynamics(*_md_start(case, seed, k, T=T[k]), T[k]) for k in range(case["members"])]
        for d in ds:
            d.run(case["steps"])
        rng, at = np.random.default_rng(seed % (1 << 31)), list(range(len(ds)))
        pot = [sum(d.energies()[:2]) for d in ds]
        for p in range(1, len(ds) - 1, 2):  # the first attempt takes the odd neighbour pairs
            delta = (1.0 / (KB * T[p]) - 1.0 / (KB * T[p + 1])) * (pot[p + 1] - pot[p])
            if rng.random() < (1.0 if delta < 0.0 else math.exp(-delta)):
                at[p], at[p + 1] = p + 1, p
                for k, q in ((p, p + 1), (p + 1, p)):
                    f = math.sqrt(T[q] / (2.0 * ds[k].ke / (3.0 * ds[k].n * KB)))
                    ds[k].v, ds[k].ke = ds[k].v * f, ds[k].ke * f * f
        return {"pos": [_np(d.x) for d in ds], "vel": [_np(d.v) for d in ds], "at": np.array(at),
                "energies": np.array([d.energies() for d in ds])}
    if kind == "serve":
        ds = []
        for j in _jobs(case, seed):
            ds.append(_Dynamics(j.system, j.mass, j.vel, 300.0))
            ds[-1].run(j.n_steps)
        return {"pos": [_np(d.x) for d in ds], "vel": [_np(d.v) for d in ds], "steps": np.array([d.k for d in ds])}
    if kind == "energies":
        topo, frames, boxes = _trajectory(case, seed)
        p, out = EnergyParams(), []
        for f, x in enumerate(frames):
            ff = _Reference(topo, None if boxes is None else boxes[f], p.cutoff, p.cutoff, p.rf_epsilon)
            out.append(_np(ff.apply(ff.f(x), True)[1].sum((1, 2))))
        return {"energies": np.stack(out)}
    x, q, iac, pairs, lj, box = _pair_inputs(case, seed)
    crf = CRFParameters.new(case["cutoff"], 1.0, EPSRF, 0.0)
    i, j = pairs[:, 0].long(), pairs[:, 1].long()
    x, q, b = x.double(), q.double(), torch.tensor(box, device=x.device)
    r = x[i] - x[j]
    r -= b * torch.round(r / b)
    r2 = (r * r).sum(1)
    c = torch.tensor(lj, device=x.device)[iac.long()[i], iac.long()[j]]
    i6, ir, qq = 1.0 / r2 ** 3, 1.0 / torch.sqrt(r2), q[i] * q[j] * 138.9354
    fs = (12.0 * c[:, 1] * i6 - 6.0 * c[:, 0]) * i6 / r2 + qq * (ir / r2 + crf.crf_cut3i)
    f = r * fs[:, None]
    forces = torch.zeros_like(x).index_add_(0, i, f).index_add_(0, j, -f)
    e = torch.stack([((c[:, 1] * i6 - c[:, 0]) * i6).sum(), (qq * (ir - crf.crf_2cut3i * r2 - crf.crf_cut)).sum()])
    return {"forces": _np(forces), "energies": _np(e), "virial": _np(r.T @ f)}
