"""Timed cases: the calls that programs using this library make, over the sizes they make them at.

Kinds of case (one pass each, through the package's public entry points):
  run    a simulation job: state in from host memory, `steps` velocity-Verlet steps with a thermo
         record every `thermo` of them, positions and velocities back to host memory
  force  a single point: state in, list build, accelerations and energies out
  batch  many small replicas: states in, `steps` steps in one launch, states and energies out
  grad   the trajectory loss and its gradient: state in, loss and gradients out
  vjp    the vector-Jacobian product of the forces: state and cotangent in, product and parameter gradients out
  sk     the structure factor on the caller's device buffers (the allocation-free entry point)

The state of a simulation is host data by the library's interface (the reference's Atom_data lives on
the host), so `prepare` makes host arrays and a configured handle and a pass takes them through the
whole call; pinned buffers, as a program that cares for the transfer keeps them.  Outputs of the mixed
form, whose forces are FP32, are handed on in FP32; those of the FP64 form in FP64.
"""
import ctypes
import math

import numpy as np
import torch

from caviar_b200 import _abi as abi
from caviar_b200 import workloads as W

TH = slice(1, 9)  # thermo record without the step number and the build counter


def listed():
    return [
        # Energy and forces of a small electrolyte, as a Monte Carlo or minimiser loop asks for: latency.
        dict(name="force_ions_500", kind="force", system="ions", n=500, density=0.122, rc=5.0, alpha=0.6, kmax=4,
             precision="mixed"),
        # A test-sized fluid sampled often: launches and readbacks, not arithmetic.
        dict(name="run_lj_500", kind="run", system="lj", n=500, density=0.8442, precision="mixed", steps=100, thermo=10),
        # The plain LJ fluid benchmark (4000 atoms) in the FP64 form.
        dict(name="run_lj_4000_fp64", kind="run", system="lj", n=4000, density=0.8442, precision="fp64", steps=200,
             thermo=100),
        # A two-species mixture under a thermostat in an elongated box, an odd number of atoms (equilibration run).
        dict(name="run_mix_32001", kind="run", system="mix", n=32001, density=0.8442, stretch=1.5, precision="mixed",
             steps=100, thermo=50, thermostat=True),
        # A mid-sized fluid in the FP64 form, an odd number of atoms.
        dict(name="run_lj_200001_fp64", kind="run", system="lj", n=200001, density=0.8442, precision="fp64", steps=60,
             thermo=30),
        # The large LJ throughput benchmark: 1,048,576 atoms.
        dict(name="run_lj_1m", kind="run", system="lj", n=1048576, density=0.8442, precision="mixed", steps=100,
             thermo=50),
        # The charged electrolyte benchmark: 8000 ions, real and reciprocal space, both forms.
        dict(name="run_ions_8000", kind="run", system="ions", n=8000, density=0.125, rc=10.0, alpha=0.3, kmax=8,
             precision="mixed", steps=100, thermo=50),
        dict(name="run_ions_8000_fp64", kind="run", system="ions", n=8000, density=0.125, rc=10.0, alpha=0.3, kmax=8,
             precision="fp64", steps=40, thermo=20),
        # The ensemble: 1024 replicas of 64 to 2048 atoms, each with its own box and temperature.
        dict(name="batch_1024", kind="batch", n_rep=1024, n_min=64, n_max=2048, kmax=6, steps=20),
        # Gradient through a trajectory of the 4000-atom charged mixture, checkpoints every 10 steps.
        dict(name="grad_4000", kind="grad", cells=10, alpha=0.4, rc=8.0, kmax=7, precision="mixed", steps=20, every=10),
        # One force VJP of a smaller mixture in FP64, as an outer optimiser or a gradient check calls it.
        dict(name="vjp_1372_fp64", kind="vjp", cells=7, alpha=0.6, rc=5.5, kmax=5, precision="fp64"),
        # Structure factor on device buffers for a host program that owns the GPU's memory; an odd number of atoms.
        dict(name="sk_20001", kind="sk", n=20001, box=54.3, kmax=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "force", "force", "batch", "grad", "vjp", "sk"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind in ("run", "force"):
        system = rng.choice(["lj", "mix", "ions"])
        c = dict(kind=kind, system=system, precision=precision)
        if system == "ions":
            c["n"] = 2 * _log(rng, 150, 8000)
            c["density"] = round(rng.uniform(0.11, 0.14), 4)
            box = (c["n"] / c["density"]) ** (1 / 3)
            c["rc"] = round(min(rng.uniform(5.0, 10.0), 0.45 * box / 1.03), 3)
            c["alpha"] = round(3.0 / c["rc"], 4)
            c["kmax"] = rng.randint(4, 10)
            most = 8e5  # atom-steps in a run
        else:
            c["n"] = _log(rng, 400, 1048576)
            c["density"] = round(rng.uniform(0.7, 0.86), 4)
            most = 4e7 if precision == "fp64" else 8e7
            if system == "mix":
                c["stretch"] = round(rng.uniform(1.0, 2.0), 2) if c["n"] > 2000 else 1.0
                c["thermostat"] = kind == "run" and rng.random() < 0.5
        if kind == "run":
            c["steps"] = max(10, min(rng.randint(50, 200), int(most / c["n"])))
            c["thermo"] = rng.choice([c["steps"], max(1, c["steps"] // 2), max(1, c["steps"] // 10)])
        return c
    if kind == "batch":
        return dict(kind=kind, n_rep=_log(rng, 16, 1024), n_min=64, n_max=_log(rng, 128, 2048), kmax=rng.randint(4, 6),
                    steps=rng.randint(8, 20))
    if kind in ("grad", "vjp"):
        cells = rng.randint(4, 10)
        box = cells * (4 / 0.8442) ** (1 / 3)
        rc = round(min(rng.uniform(4.0, 8.0), 0.49 * box), 3)
        c = dict(kind=kind, cells=cells, alpha=round(3.2 / rc, 4), rc=rc, kmax=rng.randint(4, 8), precision=precision)
        if kind == "grad":
            c["steps"] = rng.randint(10, 20)
            c["every"] = rng.randint(5, 10)
        return c
    return dict(kind=kind, n=_log(rng, 1000, 100000), box=round(rng.uniform(20.0, 60.0), 2), kmax=rng.randint(4, 10))


# ------------------------------------------------------------------- inputs


def _fluid(case, rng):
    """n atoms on random sites of an FCC lattice, jittered, as a configuration file of a dense fluid holds them."""
    n, stretch = case["n"], case.get("stretch", 1.0)
    edge = (n / case["density"] / stretch) ** (1 / 3)
    a = (4.0 / case["density"]) ** (1 / 3)
    cells = [max(1, int(math.floor(e / a + 1e-9))) for e in (edge, edge, edge * stretch)]
    while 4 * cells[0] * cells[1] * cells[2] < n:
        cells[min(range(3), key=lambda d: cells[d] / (stretch if d == 2 else 1.0))] += 1
    box = np.array([edge, edge, edge * stretch])
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.stack(np.meshgrid(*[np.arange(c, dtype=np.float64) for c in cells], indexing="ij"), axis=-1).reshape(-1, 3)
    sites = (g[:, None, :] + basis[None] + 0.25).reshape(-1, 3)
    if len(sites) > n:
        sites = sites[np.sort(rng.permutation(len(sites))[:n])]
    pos = sites * (box / np.array(cells)) + rng.uniform(-0.07, 0.07, size=(n, 3))
    return box, pos


def _ions(case, rng):
    """n ions on random sites of a simple cubic grid, jittered (no pair closer than about 0.95)."""
    n = case["n"]
    edge = (n / case["density"]) ** (1 / 3)
    m = int(math.floor(edge / 1.2))
    sites = rng.permutation(m ** 3)[:n]
    pos = (np.stack([sites // (m * m), sites // m % m, sites % m], axis=-1) + 0.5) * (edge / m)
    return np.full(3, edge), pos + rng.uniform(-0.12, 0.12, size=(n, 3))


def _system(case, seed):
    """The simulation's box, force fields and atoms."""
    rng = np.random.default_rng(seed)
    ions = case["system"] == "ions"
    box, pos = _ions(case, rng) if ions else _fluid(case, rng)
    n = case["n"]
    s = W.MDSystem(lo=np.zeros(3), hi=box, mass=np.ones(1), charge=np.zeros(1), pos=pos,
                   vel=W.maxwell_boltzmann(n, 1.0, rng), type=np.zeros(n, np.int32), cutoff=2.5, coef=2.8 / 2.5,
                   ghost_cutoff=2.8, dt=0.005)
    if ions:
        s.mass, s.charge = np.ones(2), np.array([1.0, -1.0])
        s.type = (np.arange(n) % 2).astype(np.int32)
        s.cutoff, s.coef, s.ghost_cutoff = case["rc"], 1.03, case["rc"] * 1.03
        s.ewald_r = W.EwaldRParams(alpha=case["alpha"])
        s.ewald_k = W.EwaldKParams(alpha=case["alpha"], kmax=(case["kmax"],) * 3)
        s.lj = W.LJParams(2.5, np.ones((2, 2)), np.ones((2, 2)))
    elif case["system"] == "mix":
        s.mass, s.charge = np.array([1.0, 2.0]), np.zeros(2)
        s.type = rng.integers(0, 2, n).astype(np.int32)
        s.lj = W.LJParams(2.5, np.array([[1.0, 0.75], [0.75, 0.5]]), np.array([[1.0, 0.94], [0.94, 0.88]]))
    else:
        s.lj = W.LJParams(2.5, np.ones((1, 1)), np.ones((1, 1)))
    return s


BERENDSEN = dict(temperature=1.0, coupling=0.5, dt=0.005)


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.pin_memory() if torch.cuda.is_available() else t


def _prec(case):
    return abi.PREC_FP64 if case.get("precision") == "fp64" else abi.PREC_MIXED


def _adjoint(case, seed):
    return W.adjoint_mixture(ncell=case["cells"], seed=seed, alpha=case["alpha"], rc_r=case["rc"], kmax=case["kmax"])


def _replicas(case, seed):
    sizes = np.random.default_rng(4).integers(case["n_min"], case["n_max"] + 1, size=case["n_rep"])
    b = W.replica_batch(sizes=sizes, seed=seed)
    b.kmax = case["kmax"]
    return b


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("run", "force"):
        s = _system(case, seed)
        sim = abi.Simulation(precision=_prec(case), lo=s.lo, hi=s.hi, bc=s.bc, mass=s.mass, charge=s.charge)
        sim.configure(s)
        if case.get("thermostat"):
            sim.set_berendsen(**BERENDSEN)
        st.update(sim=sim, n=s.n, pos=_pinned(s.pos), vel=_pinned(s.vel), type=_pinned(s.type),
                  out=[_pinned(np.zeros((s.n, 3))) for _ in range(2)])
    elif kind == "batch":
        b = _replicas(case, seed)
        h = abi.Batch(b.n, b.box, b.mass, b.charge)
        h.set_forces(b.epsilon, b.sigma, b.rc_lj, b.rc_r, b.alpha, b.kmax, b.k_e, b.dt)
        st.update(batch=h, pos=b.pos, vel=b.vel, type=b.type)
    elif kind in ("grad", "vjp"):
        s = _adjoint(case, seed)
        h = abi.Adjoint(len(s.pos), s.box, s.mass, _prec(case))
        h.set_params(s.charge, s.epsilon, s.sigma, s.rc_lj, s.alpha, s.rc_r, s.kmax, s.k_e, s.dt)
        st.update(adj=h, pos=s.pos, vel=s.vel, type=s.type, u=_cotangent(case, seed))
    else:
        pos, q = _sk_inputs(case, seed)
        f = abi.load().cvr_structure_factor_noalloc
        f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.POINTER(ctypes.c_double), ctypes.c_int,
                      ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_char_p, ctypes.c_size_t]
        f.restype = ctypes.c_int
        k = case["kmax"]
        st.update(f=f, pos=torch.from_numpy(pos).cuda(), q=torch.from_numpy(q).cuda(),
                  box=(ctypes.c_double * 3)(*[case["box"]] * 3),
                  out=torch.zeros((8 * k ** 3, 2), dtype=torch.float64, device="cuda"))
    return st


def _cotangent(case, seed):
    return np.random.default_rng(seed + 77).normal(size=(4 * case["cells"] ** 3, 3))


def _sk_inputs(case, seed):
    rng = np.random.default_rng(seed)
    q = np.where(np.arange(case["n"]) % 2 == 0, 1.0, -1.0)
    return rng.uniform(0.0, case["box"], size=(case["n"], 3)), q


# --------------------------------------------------------------------- pass


def _kept(case, *arrays):
    """Outputs in the precision the form computes in."""
    out = []
    for a in arrays:
        t = a if isinstance(a, torch.Tensor) else torch.from_numpy(a)
        out.append(t if case.get("precision") == "fp64" else t.float())
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("run", "force"):
        sim = state["sim"]
        sim.set_state_ptr(state["n"], state["pos"].data_ptr(), state["vel"].data_ptr(), state["type"].data_ptr())
        if kind == "force":
            acc, th = sim.compute_forces()
            return _kept(case, acc, np.array([th[k] for k in abi.TH_KEYS[TH]]))
        th = sim.run(case["steps"], case["thermo"])
        pos, vel = state["out"]
        sim.get_state_ptr(pos.data_ptr(), vel.data_ptr(), None)
        return _kept(case, pos, vel, np.ascontiguousarray(th[:, TH]))
    if kind == "batch":
        b = state["batch"]
        b.set_state(state["pos"], state["vel"], state["type"])
        out = b.run(case["steps"])
        return _kept(case, *b.state(), np.ascontiguousarray(out[:, :7]))
    if kind == "grad":
        a = state["adj"]
        a.set_state(state["pos"], state["vel"], state["type"])
        loss, g = a.loss_grad(case["steps"], case["every"])
        return _kept(case, np.array([loss]), *[np.ascontiguousarray(g[k]) for k in ("pos", "vel", "eps", "sigma", "charge")])
    if kind == "vjp":
        a = state["adj"]
        a.set_state(state["pos"], state["vel"], state["type"])
        w, g = a.force_vjp(state["u"])
        return _kept(case, w, *[np.ascontiguousarray(g[k]) for k in ("eps", "sigma", "charge")])
    k = case["kmax"]
    out = state["out"]
    rc = state["f"](state["pos"].data_ptr(), state["q"].data_ptr(), case["n"], state["box"], k, k, k, out.data_ptr(),
                    torch.cuda.current_stream().cuda_stream, None, 0)
    if rc != 0:
        raise RuntimeError(f"cvr_structure_factor_noalloc: {rc}")
    return out


def work(case):
    """Bytes and operations a pass cannot do without: the state in and out once over the host link and, per
    step, positions and velocities read and written once; per step each pair inside its cutoff once (23
    operations for LJ, 40 for the Ewald real-space term) and each k-vector's phase (one of k and -k), charge
    sum and force per atom (16 operations)."""
    kind = case["kind"]
    if kind in ("run", "force"):
        n, steps = case["n"], case.get("steps", 1)
        pairs = n * case["density"] * 2 / 3 * math.pi
        flops = 23 * pairs * 2.5 ** 3
        if case["system"] == "ions":
            flops += 40 * pairs * case["rc"] ** 3 + 16 * n * 4 * case["kmax"] ** 3
        return {"bytes": n * (52 + 48) + 96 * n * (steps if kind == "run" else 0), "flops": flops * steps}
    if kind == "batch":
        ns = (np.linspace(case["n_min"], case["n_max"], case["n_rep"])).astype(np.int64)
        n = float(ns.sum())
        pairs = float((ns.astype(np.float64) ** 2).sum()) / 2 * math.pi / 6
        flops = (case["steps"] + 1) * (63 * pairs + 16 * n * 4 * case["kmax"] ** 3)
        return {"bytes": n * (52 + 72) + 96 * n * case["steps"], "flops": flops}
    if kind in ("grad", "vjp"):
        n = 4 * case["cells"] ** 3
        pairs = n * 0.8442 * 2 / 3 * math.pi * case["rc"] ** 3
        one = 40 * pairs + 16 * n * 4 * case["kmax"] ** 3
        evals = 2 * one if kind == "vjp" else 4 * one * case["steps"]
        return {"bytes": n * (52 + 48) + (192 * n * case["steps"] if kind == "grad" else 24 * n), "flops": evals}
    return {"bytes": case["n"] * 32 + 128 * case["kmax"] ** 3, "flops": 8.0 * case["n"] * 4 * case["kmax"] ** 3}


# ------------------------------------------------- the same in 64 bits, plain


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _kset(k):
    """Integer triples of the k-set: the first (2k)^3 of [-k, k]^3 without the origin, in nested order."""
    r = torch.arange(-k, k + 1, device=_dev())
    t = torch.cartesian_prod(r, r, r)
    return t[(t != 0).any(dim=1)][: 8 * k ** 3].double()


def _kspace(pos, q, box, alpha, kmax, ke=1.0):
    """S(k), force and energy of the Ewald k-space sum."""
    kv = _kset(kmax) * (2 * math.pi / box)
    k2 = (kv * kv).sum(1)
    fk = torch.exp(-k2 / (4 * alpha * alpha)) / k2
    vol = float(box[0] * box[1] * box[2])
    re, im = [], []
    step = max(1, 1 << 24 >> max(0, (len(pos) - 1).bit_length()))
    force = torch.zeros_like(pos)
    for a in range(0, len(kv), step):
        ph = pos @ kv[a:a + step].T
        c, s = ph.cos(), ph.sin()
        sr, si = q @ c, q @ s
        re.append(sr)
        im.append(si)
        force += ((s * sr - c * si) * fk[a:a + step]) @ kv[a:a + step]
    re, im = torch.cat(re), torch.cat(im)
    force = force * (q * (4 * math.pi * ke / vol))[:, None]
    return torch.stack([re, im], 1), force, 2 * math.pi * ke / vol * (fk * (re * re + im * im)).sum()


def _neighbours(pos, box, radius):
    """Indices of the atoms within radius of each atom, one row per atom, padded with len(pos)."""
    n, dev = len(pos), pos.device
    nc = torch.clamp((box / radius).floor().long(), min=1).tolist()
    cells = min(nc) >= 3
    if cells:
        nct = torch.tensor(nc, device=dev)
        ci = torch.minimum((pos / box * nct).floor().long(), nct - 1)
        key = (ci[:, 0] * nc[1] + ci[:, 1]) * nc[2] + ci[:, 2]
        count = torch.bincount(key, minlength=nc[0] * nc[1] * nc[2])
        order = torch.argsort(key)
        slot = torch.arange(n, device=dev) - (torch.cumsum(count, 0) - count)[key[order]]
        occ = int(count.max())
        table = torch.full((len(count), occ), n, device=dev)
        table[key[order], slot] = order
        off = torch.cartesian_prod(*[torch.tensor([-1, 0, 1], device=dev)] * 3)
        width = 27 * occ
    else:
        every = torch.arange(n, device=dev)[None]
        width = n
    rows = max(1, (1 << 24) // width)
    padded = torch.cat([pos, torch.full((1, 3), 1e9, dtype=pos.dtype, device=dev)])
    kept = []
    for a in range(0, n, rows):
        p = pos[a:a + rows]
        if cells:
            c = (ci[a:a + rows, None, :] + off) % nct
            cand = table[(c[..., 0] * nc[1] + c[..., 1]) * nc[2] + c[..., 2]].reshape(len(p), -1)
        else:
            cand = every.expand(len(p), -1)
        r2 = torch.zeros(cand.shape, dtype=pos.dtype, device=dev)
        for d in range(3):
            x = padded[:, d][cand] - p[:, d, None]
            r2 += (x - box[d] * torch.round(x / box[d])) ** 2
        ok = (r2 < radius * radius) & (cand < n) & (cand != torch.arange(a, a + len(p), device=dev)[:, None])
        most = int(ok.sum(1).max())
        row = torch.full((len(p), most + 1), n, device=dev)
        kept.append(row.scatter_(1, torch.where(ok, ok.cumsum(1) - 1, most), torch.where(ok, cand, n))[:, :most])
    most = max(k.shape[1] for k in kept)
    return torch.cat([torch.nn.functional.pad(k, (0, most - k.shape[1]), value=n) for k in kept])


class _Exact:
    """A simulation in 64 bits: pair sums over padded neighbour rows, velocity Verlet."""

    def __init__(self, case, seed):
        s = _system(case, seed)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=_dev())  # noqa: E731
        self.case, self.n = case, s.n
        self.box, self.pos, self.vel = t(s.hi), t(s.pos), t(s.vel)
        self.type = t(s.type).long()
        self.mass, self.q = t(s.mass)[self.type], t(s.charge)[self.type]
        self.eps, self.sig = t(s.lj.epsilon), t(s.lj.sigma)
        self.ions = case["system"] == "ions"
        # the Ewald real-space sum runs over every listed pair, so the list is the run's own; LJ has its
        # cutoff, and any list that covers it does
        self.radius = s.cutoff * s.coef if self.ions else 3.1
        self.half_skin = 0.5 * (self.radius - s.cutoff)
        self.dt = s.dt
        self.build()

    def build(self):
        self.pos = self.pos - self.box * torch.floor(self.pos / self.box)
        self.near = _neighbours(self.pos, self.box, self.radius)
        self.built = self.pos.clone()

    def forces(self):
        n, near = self.n, self.near
        far = torch.full((1, 3), 1e9, dtype=torch.float64, device=_dev())
        p = torch.cat([self.pos, far])
        ty = torch.cat([self.type, self.type[:1]])
        q = torch.cat([self.q, self.q[:1] * 0])
        rc2 = 2.5 ** 2
        acc = torch.zeros_like(self.pos)
        e_lj = e_r = virial = 0.0
        rows = max(1, (1 << 24) // near.shape[1])
        for a in range(0, n, rows):
            j = near[a:a + rows]
            d = [p[:, k][j] - self.pos[a:a + rows, k, None] for k in range(3)]
            d = [x - self.box[k] * torch.round(x / self.box[k]) for k, x in enumerate(d)]
            there = j < n
            r2 = torch.where(there, d[0] ** 2 + d[1] ** 2 + d[2] ** 2, 1e18)
            ti, tj = self.type[a:a + rows, None], ty[j]
            eps = self.eps[ti, tj]
            s2 = self.sig[ti, tj] ** 2
            inside = r2 <= rc2
            rho6, c6 = (s2 / r2) ** 3, (s2 / rc2) ** 3
            shift = 12 * c6 * c6 - 6 * c6
            coef = torch.where(inside, 4 * eps * ((12 * rho6 * rho6 - 6 * rho6) / r2 - shift / rc2), 0.0)
            pot = 4 * eps * (rho6 * rho6 - rho6 - (c6 * c6 - c6) + shift * (r2 - rc2) / (2 * rc2))
            e_lj += 0.5 * torch.where(inside, pot, 0.0).sum()
            if self.ions:
                al = self.case["alpha"]
                r = r2.sqrt()
                qq = torch.where(there, self.q[a:a + rows, None] * q[j], 0.0)
                erfc = torch.erfc(al * r)
                coef = coef + qq * (2 * al / math.sqrt(math.pi) * torch.exp(-al * al * r2) + erfc / r) / r2
                e_r += 0.5 * (qq * erfc / r).sum()
            virial += 0.5 * torch.where(there, coef * r2, 0.0).sum()
            acc[a:a + rows] = -torch.stack([(coef * torch.where(there, x, 0.0)).sum(1) for x in d], 1)
        e_k = e_self = 0.0
        if self.ions:
            _, fk, e_k = _kspace(self.pos, self.q, self.box, self.case["alpha"], self.case["kmax"])
            acc = acc + fk
            e_self = -self.case["alpha"] / math.sqrt(math.pi) * (self.q ** 2).sum()
        return acc / self.mass[:, None], [e_lj, e_r, e_k, e_self, virial]

    def kinetic(self):
        m = self.mass[:, None]
        v = self.vel - (m * self.vel).sum(0) / self.mass.sum()
        ke = 0.5 * (m * v * v).sum()
        return ke, 2 * ke / (3 * self.n - 3)

    def record(self, e):
        ke, temp = self.kinetic()
        vol = self.box.prod()
        return torch.stack([torch.as_tensor(x, dtype=torch.float64, device=_dev()) for x in
                            (ke, temp, *e, self.n * temp / vol + e[4] / (3 * vol))])

    def steps(self, count, every):
        acc, e = self.forces()
        out = []
        for k in range(1, count + 1):
            self.pos = self.pos + self.vel * self.dt + acc * (0.5 * self.dt ** 2)
            if float(((self.pos - self.built) ** 2).sum(1).max()) > self.half_skin ** 2:
                self.build()
            new, e = self.forces()
            self.vel = self.vel + 0.5 * self.dt * (acc + new)
            acc = new
            if self.case.get("thermostat"):
                b = BERENDSEN
                lam = torch.sqrt(1 + b["dt"] / b["coupling"] * (b["temperature"] / self.kinetic()[1] - 1))
                self.vel = self.vel * torch.clamp(lam, 0.8, 1.25)
            if k % every == 0:
                out.append(self.record(e))
        return torch.stack(out)


def _exact_batch(case, seed):
    b = _replicas(case, seed)
    dev, o = _dev(), b.offsets
    res = [[], [], [], []]
    for r in range(len(b.n)):
        sl = slice(int(o[r]), int(o[r + 1]))
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        pos, vel, q = t(b.pos[sl]), t(b.vel[sl]), t(b.charge[b.type[sl]])
        L, rl2, rr2, al, n = float(b.box[r]), float(b.rc_lj[r]) ** 2, float(b.rc_r[r]) ** 2, b.alpha, int(b.n[r])
        box = torch.full((3,), L, dtype=torch.float64, device=dev)
        qq, c6 = q[:, None] * q[None], rl2 ** -3
        shift = 12 * c6 * c6 - 6 * c6

        def forces(energies):
            d = pos[None] - pos[:, None]
            d = d - L * torch.round(d / L)
            r2 = (d * d).sum(2)
            r2.fill_diagonal_(1e18)
            i6, rr = r2 ** -3, r2.sqrt()
            lj, er = r2 <= rl2, r2 <= rr2
            erfc = torch.erfc(al * rr)
            coef = torch.where(lj, 4 * ((12 * i6 * i6 - 6 * i6) / r2 - shift / rl2), 0.0)
            coef = coef + torch.where(er, qq * (2 * al / math.sqrt(math.pi) * torch.exp(-al * al * r2) + erfc / rr) / r2, 0.0)
            _, fk, e_k = _kspace(pos, q, box, al, b.kmax)
            f = pos * 0 + fk - torch.einsum("ij,ijd->id", coef, d)
            if not energies:
                return f, None
            e_lj = 0.5 * torch.where(lj, 4 * (i6 * i6 - i6 - (c6 * c6 - c6) + shift * (r2 - rl2) / (2 * rl2)), 0.0).sum()
            e_r = 0.5 * torch.where(er, qq * erfc / rr, 0.0).sum()
            return f, [e_lj, e_r, e_k, -al / math.sqrt(math.pi) * (q * q).sum(), 0.5 * (coef * r2).sum()]

        f, e = forces(case["steps"] == 0)
        for k in range(case["steps"]):
            pos = pos + vel * b.dt + f * (0.5 * b.dt ** 2)
            new, e = forces(k == case["steps"] - 1)
            vel, f = vel + 0.5 * b.dt * (f + new), new
        v = vel - vel.mean(0)
        ke = 0.5 * (v * v).sum()
        for at, x in zip(res, (pos - L * torch.floor(pos / L), vel, f, torch.stack([ke, *e, 2 * ke / (3 * n - 3)])[None])):
            at.append(x.cpu())
    return [torch.cat(x) for x in res]


class _Potential:
    """The mixture's potential energy over the pairs of one configuration, differentiable in everything."""

    def __init__(self, s):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float64), device=_dev())  # noqa: E731
        self.s, self.type = s, torch.as_tensor(s.type, device=_dev()).long()
        self.theta = [t(s.epsilon), t(s.sigma), t(s.charge)]
        self.mass = t(s.mass)[self.type][:, None]
        self.box = torch.full((3,), s.box, dtype=torch.float64, device=_dev())

    def energy(self, pos, eps, sig, charge):
        s, L, ty = self.s, self.s.box, self.type
        with torch.no_grad():
            near = _neighbours(pos - L * torch.floor(pos / L), self.box, max(s.rc_r, s.rc_lj))
            i = torch.arange(len(pos), device=pos.device)[:, None].expand_as(near)
            once = (near < len(pos)) & (i < near)
            i, j = i[once], near[once]
        # both off-diagonal entries of a symmetric table are the same parameter
        a, b = torch.minimum(ty[i], ty[j]), torch.maximum(ty[i], ty[j])
        d = pos[j] - pos[i]
        d = d - L * torch.round(d.detach() / L)
        r2 = (d * d).sum(1)
        q = charge[ty]
        r = r2.sqrt()
        u = torch.where(r2 <= s.rc_r ** 2, s.k_e * q[i] * q[j] * torch.erfc(s.alpha * r) / r, 0.0).sum()
        m = r2 <= s.rc_lj ** 2
        r2, e, rc2 = r2[m], eps[a[m], b[m]], s.rc_lj ** 2
        s2 = sig[a[m], b[m]] ** 2
        i6, c6 = (s2 / r2) ** 3, (s2 / rc2) ** 3
        u = u + (4 * e * (i6 * i6 - i6 - (c6 * c6 - c6) + (12 * c6 * c6 - 6 * c6) * (r2 - rc2) / (2 * rc2))).sum()
        kv = _kset(s.kmax) * (2 * math.pi / L)
        k2 = (kv * kv).sum(1)
        ph = pos @ kv.T
        re, im = q @ ph.cos(), q @ ph.sin()
        fk = torch.exp(-k2 / (4 * s.alpha ** 2)) / k2
        u = u + 2 * math.pi * s.k_e / L ** 3 * (fk * (re * re + im * im)).sum()
        return u - s.alpha / math.sqrt(math.pi) * s.k_e * (q * q).sum()

    def force(self, pos):
        """U, dU/dtheta and F."""
        x = pos.detach().requires_grad_()
        th = [p.detach().requires_grad_() for p in self.theta]
        u = self.energy(x, *th)
        g = torch.autograd.grad(u, [x, *th])
        return float(u.detach()), list(g[1:]), -g[0]

    def vjp(self, pos, u):
        """(dF/dr)^T u and (dF/dtheta)^T u."""
        x = pos.detach().requires_grad_()
        th = [p.detach().requires_grad_() for p in self.theta]
        f = -torch.autograd.grad(self.energy(x, *th), x, create_graph=True)[0]
        g = torch.autograd.grad((f * u).sum(), [x, *th])
        return g[0], list(g[1:])

    @staticmethod
    def both(g):
        """The gradient of a shared off-diagonal value, written to both entries."""
        out = [x + x.T - torch.diag(torch.diag(x)) for x in g[:2]]
        return [*out, g[2]]


def _exact_grad(case, seed):
    s = _adjoint(case, seed)
    p = _Potential(s)
    dt, M, m = s.dt, case["steps"], p.mass
    pos = torch.as_tensor(s.pos, device=_dev())
    vel = torch.as_tensor(s.vel, device=_dev())
    _, _, f = p.force(pos)
    path, loss = [pos], 0.0
    gth = [torch.zeros_like(t) for t in p.theta]
    kept = [f]
    for _ in range(M):
        pos = pos + vel * dt + f / m * (0.5 * dt * dt)
        u, du, new = p.force(pos)
        vel = vel + 0.5 * dt * (f + new) / m
        f = new
        loss += u / M
        gth = [a + b / M for a, b in zip(gth, du)]
        path.append(pos)
        kept.append(f)
    gr, gv, ga = (torch.zeros_like(pos) for _ in range(3))
    for k in range(M, 0, -1):
        gr = gr - kept[k] / M
        ga = ga + 0.5 * dt * gv
        w, th = p.vjp(path[k], ga / m)
        gr, gth = gr + w, [a + b for a, b in zip(gth, th)]
        gv, ga = gv + dt * gr, 0.5 * dt * gv + 0.5 * dt * dt * gr
    w, th = p.vjp(path[0], ga / m)
    gr, gth = gr + w, [a + b for a, b in zip(gth, th)]
    return [torch.tensor([loss], dtype=torch.float64), gr, gv, *p.both(gth)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "force"):
        x = _Exact(case, seed)
        if kind == "force":
            acc, e = x.forces()
            return [acc, x.record(e)]
        th = x.steps(case["steps"], case["thermo"])
        return [x.pos - x.box * torch.floor(x.pos / x.box), x.vel, th]
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind == "vjp":
        s = _adjoint(case, seed)
        p = _Potential(s)
        w, g = p.vjp(torch.as_tensor(s.pos, device=_dev()), torch.as_tensor(_cotangent(case, seed), device=_dev()))
        return [w, *p.both(g)]
    pos, q = _sk_inputs(case, seed)
    dev = _dev()
    box = torch.full((3,), case["box"], dtype=torch.float64, device=dev)
    return _kspace(torch.from_numpy(pos).to(dev), torch.from_numpy(q).to(dev), box, 1.0, case["kmax"])[0]
