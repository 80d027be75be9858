"""What a user of this framework has it do, as cases that can be timed and checked.

Every case goes through the package's public classes: a pass is what a program does between having
coordinates in hand and having the results of its call in hand. The ranges are those of the
repository's own workloads and tests: single-site Lennard-Jones boxes of a few hundred to a million
molecules, the liquid slab in its vapour, ensembles of small boxes, rigid multi-centre molecules with
and without point polarities, gradients through trajectories, and the molecule side of the coupled
step; the double-precision form (the default) and the mixed form; the reference's per-step binning and
the Verlet-skin lists.

The mixed form evaluates pairs in FP32; what it returns is kept in FP32, as a program that chose it
stores its trajectories. ``exact`` gives the same results in 64 bits from plain torch over windows of
the z-sorted molecules, with no cells, lists or other code of the package.
"""
import math

import numpy as np
import torch

from madpac_b200 import mdgpu as M
from madpac_b200 import workloads as W
from madpac_b200.trajectory import TrajectoryAdjoint

DT = 0.002


def listed():
    return [
        # forces of a small box between a host code's own steps: device buffers in, device buffers out
        dict(name="noalloc_2k", kind="noalloc", n=2048, species=2, rc=2.5, rho=0.8, fp64=True),
        # one thermostatted step of the reference's own loop on a test-sized box: all latency
        dict(name="nvt_step_864", kind="nvt_step", n=864, species=1, rc=2.5, rho=0.8, fp64=True),
        # forces, energy and virial of given coordinates through the container: 32,000 molecules
        dict(name="traverse_32k", kind="traverse", n=32000, species=1, rc=2.5, rho=0.8, fp64=True),
        # the molecule side of the coupled step: walls, wall force, cell-wise thermostat
        dict(name="coupled_32k", kind="coupled", n=32000, species=1, rc=2.5, rho=0.8, fp64=True, steps=5),
        # the drop-in run, binning in every step as the reference does, on an ordinary odd-sized box
        dict(name="run_binned_250k", kind="run", system="box", n=250047, species=1, rc=2.5, rho=0.8, fp64=True,
             skin=0.0, prune=0.0, steps=20),
        # the same on the inhomogeneous two-species slab: most cells nearly empty
        dict(name="slab_binned_786k", kind="run", system="slab", n=786432, species=2, rc=2.5, rho=0.7, fp64=True,
             skin=0.0, prune=0.0, steps=8),
        # the large production run: mixed form, skin lists pruned on the device
        dict(name="run_skin_1m", kind="run", system="box", n=1048576, species=1, rc=3.0, rho=0.75, fp64=False,
             skin=0.4, prune=0.15, steps=200),
        # two species in double precision with skin lists, an odd size
        dict(name="run_skin_fp64_400k", kind="run", system="box", n=400009, species=2, rc=2.5, rho=0.8, fp64=True,
             skin=0.3, prune=0.0, steps=50),
        # an ensemble of independent boxes of 256 to 8192 molecules
        dict(name="batch_512", kind="batch", boxes=512, fp64=False, skin=0.3, steps=30),
        # a two-centre fluid with the skin lists
        dict(name="rigid_2clj_256k", kind="rigid", model="2clj", n=256000, fp64=False, skin=0.3, steps=20),
        # quadrupolar, dipolar and charged molecules in a reaction field: forces and torques
        dict(name="rigid_polar_32k", kind="rigid", model="polar", n=32000, fp64=True, skin=0.0, steps=1),
        # gradient of a loss on the final forces and energy with respect to the start and the parameters
        dict(name="gradient_16k", kind="gradient", n=16384, species=2, rc=2.5, rho=0.8, fp64=True, steps=20, every=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["noalloc", "nvt_step", "traverse", "coupled", "run", "run", "run", "slab", "batch", "rigid",
                       "rigid", "gradient"])
    fp64 = rng.random() < 0.6
    box = dict(species=rng.choice([1, 2]), rc=rng.choice([2.5, 3.0]), rho=round(rng.uniform(0.6, 0.85), 3), fp64=fp64)
    if kind == "noalloc":
        return dict(kind=kind, n=_log(rng, 600, 30000), **box)
    if kind == "nvt_step":
        return dict(kind=kind, n=_log(rng, 500, 20000), **dict(box, fp64=True))
    if kind == "traverse":
        return dict(kind=kind, n=_log(rng, 1000, 400000), **box)
    if kind == "coupled":
        return dict(kind=kind, n=_log(rng, 1000, 60000), steps=5, **dict(box, fp64=True))
    if kind == "gradient":
        return dict(kind=kind, n=_log(rng, 600, 16000), steps=rng.choice([5, 10, 20]), every=rng.choice([3, 5, 10]), **box)
    if kind == "batch":
        return dict(kind=kind, boxes=_log(rng, 8, 400), fp64=fp64, skin=rng.choice([0.0, 0.3]), steps=rng.choice([5, 10]))
    if kind == "rigid":
        model = rng.choice(["2clj", "charged", "mix", "polar"])
        return dict(kind=kind, model=model, n=_log(rng, 1500, 30000 if model == "polar" else 200000), fp64=fp64,
                    skin=rng.choice([0.0, 0.3]), steps=rng.choice([1, 5, 10]))
    skin, prune = rng.choice([(0.0, 0.0), (0.3, 0.0), (0.4, 0.15)])
    system = "slab" if kind == "slab" else "box"
    n = _log(rng, 20000, 700000) if system == "slab" else _log(rng, 1000, 700000)
    case = dict(kind="run", system=system, n=n, skin=skin, prune=prune, **box)
    if system == "slab":
        case.update(species=2, rc=2.5, rho=0.7)
    case["steps"] = rng.choice([10, 40]) if skin else rng.choice([2, 5, 10])
    return case


# ----------------------------------------------------------------------------- inputs

def _components(species):
    return W.two_species() if species == 2 else [W.Component(1.0, 1.0, 1.0, True)]


def _system(case, seed):
    """The case's molecules: a lattice start, every molecule moved a little (a lattice has no net forces)."""
    seed = int(seed) % (1 << 31)
    if case.get("system") == "slab":
        s = W.config_c3(seed, case["n"])
    else:
        n = case["n"]
        s = W.lj_fcc_box(int(math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9)), case["rho"], 1.0, seed, case["rc"],
                         _components(case["species"]), n_atoms=n, dt=DT, nve=case["kind"] != "nvt_step")
    rng = np.random.default_rng(seed + 1)
    s.r = (s.r + rng.uniform(-0.08, 0.08, s.r.shape)) % s.length
    s.r[s.r >= s.length] = 0.0
    return s


def _ensemble(case, seed):
    """Boxes of 256 to 8192 molecules, sizes, densities and temperatures given by the number of boxes."""
    sizes = np.random.default_rng(case["boxes"])
    out = []
    for k in range(case["boxes"]):
        n = int(round(math.exp(sizes.uniform(math.log(256), math.log(8192)))))
        rho, temperature = float(sizes.uniform(0.6, 0.9)), float(sizes.uniform(0.7, 1.5))
        out.append(W.lj_fcc_box(int(math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9)), rho, temperature,
                                (int(seed) * 1009 + k) % (1 << 31), 2.5, _components(1), n_atoms=n, dt=DT))
    return out


def _rigid_system(case, seed):
    n = case["n"]
    seed = int(seed) % (1 << 31)
    if case["model"] == "2clj":
        comps, rho, fr = [W.two_centre()], 0.3, None
    elif case["model"] == "charged":
        comps, rho, fr = [W.charged_two_centre()], 0.3, None
    elif case["model"] == "mix":
        comps, rho, fr = [W.two_centre(), W.three_centre_linear()], 0.25, [0.6, 0.4]
    else:
        comps = [W.quadrupolar_two_centre(0.8), W.dipolar_two_centre(0.9), W.charged_two_centre(0.4)]
        rho, fr = 0.25, [0.4, 0.3, 0.3]
    s = W.rigid_fcc_box(int(math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9)), rho, 2.0, seed, 3.0, comps, fractions=fr,
                        n_atoms=n, dt=DT)
    if case["model"] == "polar":
        s.epsilon_rf = 5.0
    return s


def _precision(case):
    return M.FP64 if case["fp64"] else M.MIXED


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "noalloc":
        s = _system(case, seed)
        state.update(s=s, r=torch.tensor(s.r, device="cuda"), cid=torch.tensor(s.cid, device="cuda"),
                     F=torch.empty((s.n, 3), dtype=torch.float64, device="cuda"))
    elif kind == "nvt_step":
        state["sim"] = M.Simulation(_system(case, seed), _precision(case))
        state["sim"].prepare_start()
    elif kind in ("traverse", "run", "coupled"):
        s = _system(case, seed)
        lc = M.LinkedCells.from_system(s, _precision(case))
        if case.get("skin"):
            lc.setSkin(case["skin"])
            lc.setListPrune(case["prune"])
        state.update(r=s.r, v=s.v, lc=lc)
        if kind == "coupled":
            size = [int(x // 2.5) for x in s.length]
            upper = [2.5 * k for k in size]
            state["thermostat"] = M.CellWiseThermostat(lc, [0.0] * 3, upper, 2.5, size, 3, 1.0, 0.8, case["steps"],
                                                       (1, 0, 0))
    elif kind == "batch":
        systems = _ensemble(case, seed)
        b = M.Batch.from_systems(systems, _precision(case))
        if case["skin"]:
            b.setSkin(case["skin"])
        arrays = [np.concatenate([getattr(s, k) for s in systems]) for k in ("ids", "cid", "r", "v")]
        state.update(batch=b, arrays=arrays)
    elif kind == "rigid":
        s = _rigid_system(case, seed)
        lc = M.RigidLinkedCells.from_system(s, _precision(case))
        if case["skin"]:
            lc.setSkin(case["skin"])
        lc.update()
        lc.traversePairs()
        state["lc"] = lc
    else:
        s = _system(case, seed)
        rng = np.random.default_rng(int(seed) % (1 << 31) + 2)
        state.update(r=s.r, v=s.v, gF=rng.standard_normal((s.n, 3)), gU=float(rng.uniform(0.5, 1.5)),
                     adj=TrajectoryAdjoint(s, case["steps"], case["every"], precision=_precision(case)))
    return state


# ----------------------------------------------------------------------------- one pass

def _kept(case, out):
    """Results as the program keeps them: FP32 from the mixed form."""
    if case["fp64"]:
        return out
    return {k: np.asarray(v, dtype=np.float32) for k, v in out.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "noalloc":
        s = state["s"]
        u, w = M.forces_noalloc(state["r"].data_ptr(), state["cid"].data_ptr(), state["F"].data_ptr(), s.n, s.length,
                                s.cutoff, s.components, s.mix, s.lj_cutoff, _precision(case))
        if case["fp64"]:
            return dict(F=state["F"], U=u, W=w)
        return dict(F=state["F"].float(), **_kept(case, dict(U=u, W=w)))
    if kind == "nvt_step":
        sim = state["sim"]
        sim.simulateStep()
        st = sim.container.getParticles()
        sc = sim.scalars()
        return dict(r=st["r"], v=st["v"], F=st["F"], U=sc["upot"], W=sc["virial"], T=sc["T"])
    if kind == "traverse":
        lc = state["lc"]
        lc.setState(r=state["r"])
        lc.update()
        u, w, p = lc.traversePairs()
        return _kept(case, dict(F=lc.getParticles()["F"], U=u, W=w, pairs=p))
    if kind == "run":
        lc = state["lc"]
        lc.setState(state["r"], state["v"])
        lc.update()
        lc.traversePairs()
        records = lc.run(case["steps"], DT)
        st = lc.getParticles()
        return _kept(case, dict(r=st["r"], v=st["v"], F=st["F"], records=records))
    if kind == "coupled":
        lc = state["lc"]
        lc.setState(state["r"], state["v"])
        lc.update()
        lc.traversePairs()
        energies = []
        for it in range(1, case["steps"] + 1):
            lc.leapfrogPre(DT, 1.0)
            lc.reflectBoundary(3, 0)
            lc.update()
            u, w, p = lc.traversePairs()
            lc.forceBoundary(3, case["rc"], 0, 0.7)
            energies.append((u, w, p, lc.leapfrogPost(0.5 * DT)))
            state["thermostat"].applyThermostat(it)
        st = lc.getParticles()
        return dict(r=st["r"], v=st["v"], F=st["F"], records=np.array(energies))
    if kind == "batch":
        b = state["batch"]
        b.setParticles(*state["arrays"])
        start = b.prepare()
        records = b.run(case["steps"], DT)
        st = b.getParticles()
        return _kept(case, dict(r=st["r"], v=st["v"], F=st["F"], start=start, records=records))
    if kind == "rigid":
        lc = state["lc"]
        records = lc.run(case["steps"], DT)
        st = lc.getParticles()
        return _kept(case, dict(records=records, **{k: st[k] for k in ("r", "v", "F", "q", "D", "M")}))
    adj = state["adj"]
    r, v, F, u = adj.forward(state["r"], state["v"])
    gr, gv, ge, gs = adj.backward(state["gF"], state["gU"])
    return _kept(case, dict(r=r, v=v, F=F, U=u, gr=gr, gv=gv, ge=ge, gs=gs))


# ----------------------------------------------------------------------------- what a pass cannot do without

def _pairs(n, rho, rc):
    return n * 4.18879 * rc ** 3 * rho / 2.0


def work(case):
    """Bytes of a step: positions and velocities read and written, forces written and read again (double),
    each once; flops: 31 per molecule pair within the cutoff, more per site pair and for the derivatives."""
    kind = case["kind"]
    if kind == "batch":
        n = case["boxes"] * 7936.0 / math.log(32.0)          # mean of the log-uniform sizes
        return dict(bytes=n * 144.0 * case["steps"], flops=31.0 * _pairs(n, 0.75, 2.5) * (case["steps"] + 1))
    n = float(case["n"])
    if kind == "rigid":
        sites = {"2clj": 4, "charged": 8, "mix": 6, "polar": 8}[case["model"]]
        flops = 40.0 * sites * _pairs(n, 0.3 if case["model"] in ("2clj", "charged") else 0.25, 3.0)
        return dict(bytes=n * 368.0 * case["steps"], flops=flops * case["steps"])
    rho = 0.67 if case.get("system") == "slab" else case["rho"]
    pair_flops = 31.0 * _pairs(n, rho, case["rc"])
    if kind in ("noalloc", "traverse"):
        return dict(bytes=n * 52.0, flops=pair_flops)
    steps = case.get("steps", 1)
    if kind == "gradient":
        # forward, recomputed and backward steps; a backward pair takes about twice a forward one
        return dict(bytes=n * 144.0 * 3 * steps, flops=pair_flops * 4 * steps)
    return dict(bytes=n * 144.0 * steps, flops=pair_flops * (steps + (0 if kind == "nvt_step" else 1)))


# ----------------------------------------------------------------------------- 64-bit values

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _tables(species, shift, rc):
    """eps24, sigma^2 and shift6 of each ordered component pair; pairs of unlike components always shift."""
    eps, sig = ([1.0], [1.0]) if species == 1 else ([1.0, 0.8], [1.0, 0.9])
    k = len(eps)
    t = torch.zeros((3, k, k), dtype=torch.float64)
    for a in range(k):
        for b in range(k):
            e, s2 = 24.0 * math.sqrt(eps[a] * eps[b]), (0.5 * (sig[a] + sig[b])) ** 2
            q = (s2 / rc ** 2) ** 3
            t[:, a, b] = torch.tensor([e, s2, e * (q - q * q) if shift or a != b else 0.0], dtype=torch.float64)
    return t.to(_device())


def _windows(r, L, rc, budget):
    """Yields (i, j) index tensors: molecules i of a z layer, consecutive in y, and every molecule that can be
    within rc of one of them (the layer and its two neighbours, within rc in y)."""
    z, y, Ly = r[:, 2].cpu().numpy(), r[:, 1].cpu().numpy(), float(L[1])
    layers = int(float(L[2]) / rc)
    layer = np.minimum((z * (layers / float(L[2]))).astype(np.int64), layers - 1)
    order = np.lexsort((y, layer))
    first = np.searchsorted(layer[order], np.arange(layers + 1))
    own = [order[first[k]:first[k + 1]] for k in range(layers)]
    ext = [np.concatenate([y[o] - Ly, y[o], y[o] + Ly]) for o in own]
    for k in range(layers):
        a = 0
        while a < len(own[k]):
            m = 64
            while True:
                b = min(len(own[k]), a + m)
                lo, hi = y[own[k][a]] - rc, y[own[k][b - 1]] + rc
                js = []
                for near in sorted({(k - 1) % layers, k, (k + 1) % layers}):
                    u, w = np.searchsorted(ext[near], [lo, hi + 1e-9])
                    js.append(own[near] if w - u >= len(own[near]) else np.tile(own[near], 3)[u:w])
                j = np.concatenate(js)
                if b == len(own[k]) or 4 * m * len(j) > budget:
                    break
                m *= 2
            yield torch.from_numpy(own[k][a:b]).to(r.device), torch.from_numpy(j).to(r.device)
            a = b


def _near(r, i, j, L, rc):
    """The pairs (rows of i, rows of j) within rc and their minimum-image differences."""
    d = [r[i, k][:, None] - r[j, k][None, :] for k in range(3)]
    d = [x - L[k] * torch.round(x * (1.0 / L[k])) for k, x in enumerate(d)]
    dd = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    a, b = ((dd < rc * rc) & (i[:, None] != j[None, :])).nonzero(as_tuple=True)
    return a, b, torch.stack([x[a, b] for x in d], 1)


def _lj(r, cid, L, rc, tab):
    """(F, Upot, virial, pairs) of the truncated potential, minimum image."""
    F = torch.zeros_like(r)
    sums = torch.zeros(3, dtype=torch.float64, device=r.device)
    for i, j in _windows(r, L, rc, 3e7):
        a, b, d = _near(r, i, j, L, rc)
        e24, s2, sh = (t[cid[i[a]], cid[j[b]]] for t in tab)
        dd = (d * d).sum(1)
        s6 = (s2 / dd) ** 3
        fac = e24 * (2.0 * s6 * s6 - s6) / dd
        F.index_add_(0, i[a], fac[:, None] * d)
        sums[0] += (e24 * (s6 * s6 - s6) + sh).sum() / 12.0
        sums[1] += (fac * dd).sum() / 2.0
        sums[2] += 0.5 * dd.numel()
    return (F, *(float(x) for x in sums))


def _wrap(r, L):
    r = torch.where(r < 0.0, r + L, r)
    return torch.where(r >= L, r - L, r)


def _nve(r, v, cid, L, rc, tab, steps):
    """Leapfrog steps of unit-mass molecules: (r, v, F, records, record of the start)."""
    F, U, W_, P = _lj(r, cid, L, rc, tab)
    start = [U, W_, float((v * v).sum()), P]
    rec = []
    for _ in range(steps):
        v = v + 0.5 * DT * F
        r = _wrap(r + DT * v, L)
        F, U, W_, P = _lj(r, cid, L, rc, tab)
        v = v + 0.5 * DT * F
        rec.append([U, W_, float((v * v).sum()), P])
    return r, v, F, np.array(rec), start


def _rotate(q, d, inverse):
    w, u = q[:, :1], -q[:, 1:] if not inverse else q[:, 1:]
    t = 2.0 * torch.linalg.cross(u, d)
    # unit quaternions: d + w t + u x t
    return d + w * t + torch.linalg.cross(u, t)


def _qdot(q, w):
    a, x, y, z = q.unbind(1)
    p, s, t = w.unbind(1)
    return 0.5 * torch.stack([-x * p - y * s - z * t, a * p - z * s + y * t, z * p + a * s - x * t,
                              -y * p + x * s + a * t], 1)


def _rigid_forces(r, q, L, sites, charges, rc):
    """Two equal centres (and charges) per molecule, truncated-shifted at rc on the molecule centres."""
    body = torch.tensor([[0.0, 0.0, z] for z, _ in sites + charges], dtype=torch.float64, device=r.device)
    n, ns, nl = r.shape[0], len(sites) + len(charges), len(sites)
    off = torch.stack([_rotate(q, body[s].expand(n, 3), True) for s in range(ns)])
    p6 = (1.0 / rc ** 2) ** 3
    shift = 24.0 * (p6 - p6 * p6)
    Fs = torch.zeros((ns, n, 3), dtype=torch.float64, device=r.device)
    U = W_ = P = 0.0
    for i, j in _windows(r, L, rc, 3e7):
        a, b, m = _near(r, i, j, L, rc)
        P += 0.5 * len(a)
        for s in range(ns):
            total = torch.zeros_like(m)
            for t in range(ns):
                if (s < nl) != (t < nl):
                    continue
                d = m + off[s][i][a] - off[t][j][b]
                inv = 1.0 / (d * d).sum(1)
                if s < nl:
                    s6 = inv ** 3
                    fac = 24.0 * (2.0 * s6 * s6 - s6) * inv
                    U += float((24.0 * (s6 * s6 - s6) + shift).sum()) / 12.0
                else:
                    u = charges[s - nl][1] * charges[t - nl][1] * torch.sqrt(inv)
                    fac = u * inv
                    U += float(u.sum()) / 2.0
                total += fac[:, None] * d
            W_ += float((m * total).sum()) / 2.0
            Fs[s].index_add_(0, i[a], total)
    F = Fs.sum(0)
    Mt = sum(torch.linalg.cross(off[s], Fs[s]) for s in range(ns))
    return F, Mt, U, W_, P


def _rigid(case, seed):
    """The rigid Leapfrog of the two-centre models, orientations by the normalised half-step quaternion."""
    s = _rigid_system(case, seed)
    dev = _device()
    r, v, q, D, L = (torch.tensor(x, dtype=torch.float64, device=dev) for x in (s.r, s.v, s.q, s.D, s.length))
    sites = [(-0.25, 0.5), (0.25, 0.5)]
    charges = [(0.35, 0.5), (-0.35, -0.5)] if case["model"] == "charged" else []
    inertia = sum(m * z * z for z, m in sites)
    inv = torch.tensor([1.0 / inertia, 1.0 / inertia, 0.0], dtype=torch.float64, device=dev)
    mom = torch.tensor([inertia, inertia, 0.0], dtype=torch.float64, device=dev)
    F, Mt, _, _, _ = _rigid_forces(r, q, L, sites, charges, 3.0)
    rec = []
    h = 0.5 * DT
    for _ in range(case["steps"]):
        v = v + h * F
        r = r + DT * v
        w = _rotate(q, D, False) * inv
        qh = q + h * _qdot(q, w)
        qh = qh / qh.norm(dim=1, keepdim=True)
        D = D + h * Mt
        w = _rotate(qh, D, False) * inv
        q = q + DT * _qdot(qh, w)
        q = q / q.norm(dim=1, keepdim=True)
        r = _wrap(r, L)
        F, Mt, U, W_, P = _rigid_forces(r, q, L, sites, charges, 3.0)
        v = v + h * F
        D = D + h * Mt
        w = _rotate(q, D, False) * inv
        rec.append([U, W_, float((v * v).sum()), float((mom * w * w).sum()), P])
    out = dict(records=np.array(rec), r=r, v=v, F=F, q=q, D=D, M=Mt)
    return {k: x.cpu().numpy() if torch.is_tensor(x) else x for k, x in out.items()}


def exact(case, seed):
    kind = case["kind"]
    dev = _device()
    if kind in ("coupled", "gradient"):
        return None
    if kind == "rigid":
        if case["model"] not in ("2clj", "charged") or case["n"] * case["steps"] > 5.2e6:
            return None
        return _rigid(case, seed)
    if kind == "batch":
        if case["boxes"] * case["steps"] > 3000:
            return None
        outs = []
        tab = _tables(1, True, 2.5)
        for s in _ensemble(case, seed):
            r, v, L = (torch.tensor(x, device=dev) for x in (s.r, s.v, s.length))
            r, v, F, rec, start = _nve(r, v, torch.zeros(s.n, dtype=torch.long, device=dev), L, 2.5, tab, case["steps"])
            outs.append((r.cpu().numpy(), v.cpu().numpy(), F.cpu().numpy(), rec, start))
        return dict(r=np.concatenate([o[0] for o in outs]), v=np.concatenate([o[1] for o in outs]),
                    F=np.concatenate([o[2] for o in outs]), start=np.array([o[4] for o in outs]),
                    records=np.stack([o[3] for o in outs], 1))
    if case["n"] * case.get("steps", 1) > 6.5e6:
        return None
    s = _system(case, seed)
    rc = case["rc"]
    r, v, L = (torch.tensor(x, device=dev) for x in (s.r, s.v, s.length))
    cid = torch.tensor(s.cid, dtype=torch.long, device=dev)
    tab = _tables(case["species"], True, rc)
    if kind in ("noalloc", "traverse"):
        F, U, W_, P = _lj(r, cid, L, rc, tab)
        out = dict(F=F.cpu().numpy(), U=U, W=W_)
        if kind == "traverse":
            out["pairs"] = P
        return out
    if kind == "nvt_step":
        n = s.n
        target = s.temperature
        beta = (3.0 * n * target / float((v * v).sum())) ** 0.4
        F, _, _, _ = _lj(r, cid, L, rc, tab)
        v = (2.0 - 1.0 / beta) * v + 0.5 * DT * F
        r = _wrap(r + DT * v, L)
        F, U, W_, _ = _lj(r, cid, L, rc, tab)
        v = v + 0.5 * DT * F
        mv2 = float((v * v).sum())
        v = v * (3.0 * n * target / mv2) ** 0.4
        return dict(r=r.cpu().numpy(), v=v.cpu().numpy(), F=F.cpu().numpy(), U=U, W=W_, T=mv2 / (3.0 * n))
    r, v, F, rec, _ = _nve(r, v, cid, L, rc, tab, case["steps"])
    return dict(r=r.cpu().numpy(), v=v.cpu().numpy(), F=F.cpu().numpy(), records=rec)
