"""Measured cases of the framework: the calls its users make, over their sizes.

Four kinds of work, each through the public Python surface:

* ``direct``  NbDirect: a list rebuild and the force evaluations that follow it
  (an MD program rebuilds every 10 steps and asks for the energy once in them),
  or one evaluation on a standing list.
* ``pme``     NbDirect.getforce_ewald: the reciprocal-space term of one step.
* ``batch``   MsldBatch: ten captured steps of a batch of alchemical replicas.
* ``mlp``     BF16MLP: a training step or a forward pass of the flattening network.

Systems come from blade_b200.systems at the sizes of its generators.
"""
import functools
import math

import numpy as np
import torch

from blade_b200 import _lib, alf, msld, systems
from blade_b200.batch import MsldBatch
from blade_b200.mlp import BF16MLP
from blade_b200.nbdirect import NbDirect

WATER_SPACING = 18.856 / 6  # lattice spacing of the 216-water box
DRIFT = 0.01                # A per step and coordinate, as an MD step moves atoms
METHODS = {"pme": (1, 0), "fswitch": (0, 0)}  # (electrostatics, van der Waals): PME+VFSWITCH, FSWITCH+VFSWITCH


def _direct(system, n, rcut, methods="pme", steps=10, rebuild=True):
    return {"kind": "direct", "system": system, "n": n, "rcut": rcut, "methods": methods, "steps": steps,
            "rebuild": rebuild}


def listed():
    return [
        # the smallest call: force and energy of 216 waters on a standing list (minimisers, tests, small boxes)
        {"name": "water-648-eval", **_direct("water", 6, 9.0, steps=1, rebuild=False)},
        # the same of an alchemical box: soft core and dU/dlambda of 12 substituents
        {"name": "msld-water-eval", **_direct("msld", 3, 9.0, steps=1, rebuild=False)},
        # a small solvent box without Ewald sums: force-switched electrostatics, ten MD steps
        {"name": "water-3000-fswitch", **_direct("water", 10, 12.0, "fswitch")},
        # a fixture-sized box at a 9 A cutoff, few atom types (LJ table in shared memory)
        {"name": "water-20577-rc9", **_direct("water", 19, 9.0)},
        # the headline system: chain in water, 2,491 atom types, 12 A cutoff
        {"name": "chain-23558", **_direct("chain", 2489, 12.0)},
        # a large solvated box
        {"name": "water-192000", **_direct("water", 40, 12.0)},
        # reciprocal space of the three box sizes above (1 A grid)
        {"name": "pme-648", "kind": "pme", "n": 6, "order": 6, "energy": True},
        {"name": "pme-20577", "kind": "pme", "n": 19, "order": 6, "energy": False},
        {"name": "pme-192000", "kind": "pme", "n": 40, "order": 6, "energy": False},
        # free-energy production: uneven solvated replicas, every electrostatic term, rigid water
        {"name": "batch-8-complete", "kind": "batch", "system": "chain", "replicas": 8, "n_min": 3000, "n_max": 16000,
         "pme": True},
        # landscape flattening: many small boxes with lambda biases and histograms
        {"name": "batch-32-flatten", "kind": "batch", "system": "flatten", "replicas": 32, "n_min": 0, "n_max": 0,
         "pme": False},
        # training of the flattening network at its own batch size
        {"name": "mlp-train-256", "kind": "mlp", "batch": 256, "train": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng):
    kind = rng.choice(["direct", "direct", "direct", "pme", "batch", "mlp"])
    if kind == "direct":
        system = rng.choice(["water", "water", "chain", "msld"])
        if system == "water":
            n = _log_int(rng, 6, 38)
            rcut = rng.choice([8.0, 8.5, 8.75, 9.25] if n < 8 else [9.0, 9.5, 10.0, 10.5, 11.0, 12.0])
        elif system == "chain":
            n, rcut = _log_int(rng, 300, 4000), 12.0
        else:
            n, rcut = rng.randint(4, 1000), 9.0
        methods = rng.choice(["pme", "pme", "fswitch"])
        if rng.random() < 0.3:
            return _direct(system, n, rcut, methods, 1, False)
        return _direct(system, n, rcut, methods, rng.choice([5, 10]), True)
    if kind == "pme":
        return {"kind": "pme", "n": _log_int(rng, 6, 38), "order": rng.choice([4, 6, 6, 8]),
                "energy": rng.random() < 0.5}
    if kind == "batch":
        if rng.random() < 0.5:
            return {"kind": "batch", "system": "flatten", "replicas": _log_int(rng, 4, 48), "n_min": 0, "n_max": 0,
                    "pme": False}
        return {"kind": "batch", "system": "chain", "replicas": rng.randint(1, 6), "n_min": rng.randint(3000, 5000),
                "n_max": rng.randint(5000, 14000), "pme": rng.random() < 0.7}
    return {"kind": "mlp", "batch": _log_int(rng, 1, 256), "train": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _chain_base(n_chain):
    # solute and water in the proportion and density of the 23,558-atom system
    n_wat = int(round(n_chain * 7023 / 2489))
    return systems.chain_in_water(2, 62.23 * ((n_chain + 3 * n_wat) / 23558) ** (1 / 3), n_chain, n_wat)


@functools.lru_cache(maxsize=64)
def _replica_base(seed, n, sites, subs):
    return systems.msld_chain(seed, n, sites, list(subs))


@functools.lru_cache(maxsize=64)
def _flatten_base(seed):
    return alf.flattening_system(seed)


def _water(rng, n, rc):
    """n^3 waters on the lattice of systems.water_box with dipoles that follow their neighbours' field, as in a
    liquid: its electrostatic energy is a sum of one sign, while that of random orientations cancels to nothing."""
    seed = int(rng.integers(1 << 30))
    s = systems.water_box(seed, n, WATER_SPACING * n, rCut=rc, rSwitch=rc - (1.0 if rc < 10 else 2.0),
                          beta=0.34 if rc < 10 else 0.32)
    mu = rng.normal(size=(n, n, n, 3))
    noise = 0.5 * rng.normal(size=mu.shape)
    parity = (np.indices((n, n, n)).sum(0) % 2)[..., None]
    for sweep in range(12):
        f = 0
        for axis in range(3):
            for step in (1, -1):
                m = np.roll(mu, step, axis)
                f = f - m
                f[..., axis] += 3 * m[..., axis]
        new = f + noise
        new /= np.linalg.norm(new, axis=-1, keepdims=True)
        mu = np.where(parity == sweep % 2, new, mu)
    z = mu.reshape(-1, 3)
    z = z / np.linalg.norm(z, axis=1, keepdims=True)
    x = np.cross(z, rng.normal(size=z.shape))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    rot = np.stack([x, np.cross(z, x), z], -1)  # columns: the molecule's axes, z along its dipole
    o = s.xyz[::3].astype(np.float64)
    s.xyz = (o[:, None] + np.einsum("nij,aj->nai", rot, systems.tip3p_local())).reshape(-1, 3).astype(np.float32)
    return s


def _copy(s):
    out = systems.dataclasses.replace(s, xyz=s.xyz.copy(), nbonds=s.nbonds.copy())
    if s.msld is not None:
        out.msld = systems.dataclasses.replace(s.msld, theta=s.msld.theta.copy())
    return out


def _moved(s, rng, theta_range=1.2):
    """Another input of the same system: moved as a whole across the box faces, other thetas."""
    s = _copy(s)
    s.xyz = (s.xyz + rng.uniform(0, 1, 3) * s.box).astype(np.float32)
    if s.msld is not None:
        s.msld.theta[1:] = rng.uniform(-theta_range, theta_range, s.msld.blockCount - 1)
    return s


def _system(case, seed):
    """The system of a ``direct`` or ``pme`` case and its frames [steps, N, 3]."""
    rng = np.random.default_rng(seed)
    kind = case.get("system", "water")
    if kind == "water":
        s = _water(rng, case["n"], case.get("rcut", 9.0))
    elif kind == "chain":
        s = _moved(_chain_base(case["n"]), rng)
        nc = case["n"]
        q = rng.normal(0, 0.35, nc)
        s.nbonds["q"][:nc] = (q - q.mean()).astype(np.float32)
    else:
        s = systems.msld_water(case["n"])
        s = _moved(s, rng)
    s.elecMethod, s.vdwMethod = METHODS[case.get("methods", "pme")]
    steps = case.get("steps", 1)
    frames = np.empty((steps,) + s.xyz.shape, np.float32)
    x = s.xyz.astype(np.float64)
    for k in range(steps):
        x = x + rng.normal(0, DRIFT, x.shape)
        frames[k] = x
    return s, frames


def _grid(case):
    """Points per edge at 1 A: the smallest of j*{32,27,24,20,18} above the edge, j a power of two."""
    edge, j = float(np.float32(WATER_SPACING * case["n"])), 1
    while edge >= 32 * j:
        j *= 2
    return min(j * k for k in (32, 27, 24, 20, 18) if j * k > edge)


def _replicas(case, seed):
    rng = np.random.default_rng(seed)
    R = case["replicas"]
    if case["system"] == "flatten":
        return [_moved(_flatten_base(100 + r), rng) for r in range(R)]
    out = []
    for r in range(R):
        n = int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** (r / max(1, R - 1))))
        out.append(_moved(_replica_base(4000 + r, n, 1 + r % 3, (2 + r % 4, 5 - r % 3, 3)[:1 + r % 3]), rng))
    return out


def _mlp_data(case, seed):
    """Histogram-like features (non-negative, many zeros) and targets, as the flattening loop makes them."""
    rng = np.random.default_rng(seed)
    M = case["batch"]
    x = np.maximum(rng.normal(-0.3, 1.0, (M, alf.FEAT_PAD)), 0.0) * 0.2
    y = rng.normal(0, 0.5, (M, alf.OUT_PAD))
    return x.astype(np.float32), y.astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "direct":
        s, frames = _system(case, seed)
        nb = NbDirect(s)
        pos = [torch.from_numpy(f.reshape(-1)).cuda() for f in frames]
        nb.update_domdec(pos[0], True)  # the first build sizes the list
        return {"case": case, "nb": nb, "pos": pos, "lam": nb.lambdas_tensor(),
                "force": [torch.zeros(3 * nb.N, device="cuda") for _ in pos],
                "lforce": [torch.zeros(nb.L, device="cuda") for _ in pos],
                "energy": torch.zeros(nb.R, dtype=torch.float64, device="cuda")}
    if case["kind"] == "pme":
        s, frames = _system(case, seed)
        nb = NbDirect(s)
        pos = torch.from_numpy(frames[0].reshape(-1)).cuda()
        nb.update_domdec(pos, True)
        nb.set_pme(case["order"])
        return {"case": case, "nb": nb, "pos": pos, "lam": nb.lambdas_tensor(),
                "force": torch.zeros(3 * nb.N, device="cuda"),
                "energy": torch.zeros(nb.R, dtype=torch.float64, device="cuda")}
    if case["kind"] == "batch":
        reps = _replicas(case, seed)
        flat = case["system"] == "flatten"
        B = MsldBatch(reps, seed=1 + seed % 1000003, constraints=not flat, pme=case["pme"],
                      gamma_ps=5.0 if flat else 1.0, gamma_theta_ps=1.0 if flat else None)
        if flat:  # fixed and pairwise quadratic biases, as the flattening loop sets them
            rng = np.random.default_rng(seed)
            pairs = []
            for r, s in enumerate(reps):
                b = s.msld.siteBound
                for t in range(1, s.msld.siteCount):
                    blocks = int(B.nb.lam_starts[r]) + np.arange(b[t], b[t + 1])
                    pairs += [(i, j) for k, i in enumerate(blocks) for j in blocks[k + 1:]]
            var = np.zeros(len(pairs), msld.VARBIAS_DTYPE)
            var["i"], var["j"] = np.array(pairs).T
            var["type"], var["k"] = 6, rng.uniform(-20, 20, len(pairs))
            B.set_bias(rng.uniform(-5, 5, B.theta.numel()), var)
            B.enable_histograms(np.array(pairs))
        B.capture()
        return {"case": case, "batch": B}
    x, y = _mlp_data(case, seed)
    net = BF16MLP([alf.FEAT_PAD, *alf.HIDDEN, alf.OUT_PAD], max_batch=256, seed=seed % 1000003)
    return {"case": case, "net": net, "x": torch.from_numpy(x).cuda(), "y": torch.from_numpy(y).cuda()}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "direct":
        nb, pos, e = state["nb"], state["pos"], state["energy"]
        if case["rebuild"]:
            nb.update_domdec(pos[0], True, asynchronous=True)
        for k, x in enumerate(pos):
            nb.getforce_nbdirect(x, state["lam"], k == 0, force=state["force"][k], lambda_force=state["lforce"][k],
                                 energy=e if k == 0 else None, mode=_lib.BNB_OUT_SET)
        return {"force": state["force"], "lforce": state["lforce"], "energy": e}
    if case["kind"] == "pme":
        state["nb"].getforce_ewald(state["pos"], state["lam"], case["energy"], force=state["force"],
                                   energy=state["energy"] if case["energy"] else None, mode=_lib.BNB_OUT_SET)
        return {"force": state["force"], **({"energy": state["energy"]} if case["energy"] else {})}
    if case["kind"] == "batch":
        B = state["batch"]
        B.run_graph(10)
        return {"x": B.x, "v": B.v, "theta": B.theta, "lambda": B.lam, "force": B.force, "lforce": B.lforce,
                "energy": B.energy}
    net = state["net"]
    if not case["train"]:
        return net.forward(state["x"])
    loss = net.train_step(state["x"], state["y"])
    return {"loss": loss, "gW": net.gW, "gb": net.gb, "W": net.W, "b": net.b}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _atoms(case):
    if case.get("system", "water") == "water":
        return 3 * case["n"] ** 3
    if case["system"] == "chain" and "n" in case:
        return case["n"] + 3 * int(round(case["n"] * 7023 / 2489))
    return 520


def work(case):
    if case["kind"] == "direct":
        # positions in, forces out; 60 operations for each pair within the cutoff
        n = _atoms(case)
        pairs = n * 0.5 * 0.0965 * 4 / 3 * math.pi * case["rcut"] ** 3
        return {"bytes": 24.0 * n * case["steps"], "flops": 60.0 * pairs * case["steps"]}
    if case["kind"] == "pme":
        # per atom p^3 grid points spread (2) and gathered (8); two real 3-D transforms (2.5 K^3 log2 K^3 each)
        n, g = _atoms(case), _grid(case) ** 3
        return {"bytes": 28.0 * n, "flops": 10.0 * n * case["order"] ** 3 + 5.0 * g * math.log2(g)}
    if case["kind"] == "batch":
        R = case["replicas"]
        if case["system"] == "flatten":
            n, rcut = [520] * R, 9.0
        else:
            n = [case["n_min"] * (case["n_max"] / case["n_min"]) ** (r / max(1, R - 1)) for r in range(R)]
            rcut = 12.0
        n = sum(n)
        # FP64 x and v read and written each step; 60 operations a pair, grid work as above
        flops = 60.0 * n * 0.5 * 0.0965 * 4 / 3 * math.pi * rcut ** 3
        if case["pme"]:
            flops += 10.0 * n * 216 + 5.0 * (n / 0.0965) * math.log2(n / 0.0965)
        return {"bytes": 96.0 * n * 10, "flops": 10 * flops}
    sizes = [alf.FEAT_PAD, *alf.HIDDEN, alf.OUT_PAD]
    params = sum(a * b for a, b in zip(sizes[:-1], sizes[1:]))
    M = case["batch"]
    if not case["train"]:
        return {"bytes": 2.0 * params + 4.0 * M * (sizes[0] + sizes[-1]), "flops": 2.0 * M * params}
    # master weights, both Adam moments and gradients: read and written
    return {"bytes": 28.0 * params + 4.0 * M * (sizes[0] + sizes[-1]),
            "flops": 2.0 * M * (3 * params - sizes[0] * sizes[1])}


def tolerance(case):
    # about four times the error against 64 bits (direct, pme, mlp), or the difference that another split of the
    # pair sums makes after ten steps (batch)
    if case["kind"] == "direct":
        return {"rel": 2e-5 if case["system"] == "msld" else 1e-5, "max": 4e-4}
    if case["kind"] == "pme":
        return {"rel": 3e-5, "max": 4e-4}
    if case["kind"] == "batch":
        return {"rel": 1.5e-5, "max": 1e-3}
    return {"rel": 3.2e-3, "max": 0.25}


# ---------------------------------------------------------------------------
# the same in 64 bits, with torch and numpy alone
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "direct":
        s, frames = _system(case, seed)
        none = [None] * len(frames)
        force, lforce = list(none), list(none)
        energy = None
        for k in sorted({0, len(frames) - 1}):
            f, l, e = _exact_direct(s, frames[k])
            force[k], lforce[k] = f, l
            energy = e if k == 0 else energy
        return {"force": force, "lforce": lforce, "energy": energy}
    if case["kind"] == "pme":
        s, frames = _system(case, seed)
        f, e = _exact_pme(s, frames[0], case["order"], _grid(case))
        return {"force": f, **({"energy": e} if case["energy"] else {})}
    if case["kind"] == "batch":
        return None  # ten steps of every term for all replicas: more than 20 seconds
    return _exact_mlp(case, seed)


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pairs_within(x, box, rc):
    """All i < j with minimum-image distance below rc: (i, j), by slabs of x."""
    N = len(x)
    xw = x[:, 0] - torch.floor(x[:, 0] / box[0]) * box[0]
    order = torch.argsort(xw)
    xs, xo = xw[order], x[order]
    step = max(32, min(1024, 20_000_000 // N))
    out = []
    xs_h = xs.cpu().numpy()
    L = float(box[0])
    for a in range(0, N, step):
        b = min(N, a + step)
        # sorted atoms from a on whose x lies within rc of the slab, directly or through the face
        e = int(np.searchsorted(xs_h, xs_h[b - 1] + rc, side="right"))
        w = max(e, int(np.searchsorted(xs_h, xs_h[a] + L - rc, side="left")))
        cand = torch.cat([torch.arange(a, e, device=x.device), torch.arange(w, N, device=x.device)])
        r2 = torch.zeros((b - a, len(cand)), dtype=torch.float64, device=x.device)
        for d in range(3):
            t = xo[a:b, None, d] - xo[None, cand, d]
            t -= box[d] * torch.round(t / box[d])
            r2 += t * t
        i, j = torch.nonzero((r2 < rc * rc) & (cand[None, :] > torch.arange(a, b, device=x.device)[:, None]),
                             as_tuple=True)
        i, j = order[a + i], order[cand[j]]
        out.append(torch.stack([torch.minimum(i, j), torch.maximum(i, j)]))
    return torch.cat(out, 1)


def _pair_energy(s, r, qq, c12, c6):
    rc, rs, beta = float(np.float32(s.rCut)), float(np.float32(s.rSwitch)), float(np.float32(s.betaEwald))
    if s.elecMethod == 1:
        ee = qq * torch.erfc(beta * r) / r
    else:  # force switching (CHARMM FSWITCH)
        c2, o2 = rc * rc, rs * rs
        g = 1 / (c2 - o2) ** 3
        A, B, C, D = c2 * c2 * (c2 - 3 * o2) * g, 6 * c2 * o2 * g, -(o2 + c2) * g, 2 * g / 5
        dv = 8 * (o2 * c2 * (rc - rs) - (c2 * c2 * rc - o2 * o2 * rs) / 5) * g
        ee = qq * torch.where(r <= rs, 1 / r + dv,
                              A * (1 / r - 1 / rc) + B * (rc - r) + C * (rc ** 3 - r ** 3) + D * (rc ** 5 - r ** 5))
    r3, r6 = r ** -3, r ** -6
    if s.vdwMethod == 0:
        dv6 = 1 / (rc * rs) ** 3
        k6, k12 = rc ** 3 / (rc ** 3 - rs ** 3), rc ** 6 / (rc ** 6 - rs ** 6)
        el = torch.where(r < rs, c12 * (r6 * r6 - dv6 * dv6) - c6 * (r6 - dv6),
                         c12 * k12 * (r6 - rc ** -6) ** 2 - c6 * k6 * (r3 - rc ** -3) ** 2)
    else:
        d, u = rs * rs - r * r, rc * rc - r * r
        fsw = torch.where(r < rs, torch.ones_like(r), u * u * (u - 3 * d) / (rc * rc - rs * rs) ** 3)
        el = fsw * (c12 * r6 - c6) * r6
    return ee + el


def _exact_direct(s, xyz):
    dev = _dev()
    x = torch.from_numpy(xyz).to(dev).double()
    box = torch.from_numpy(np.asarray(s.box, np.float32)).to(dev).double()
    N = len(x)
    rc = float(np.float32(s.rCut))
    ij = _pairs_within(x, box, rc)
    key = ij[0] * N + ij[1]
    ex = torch.from_numpy(np.unique(np.min(s.excl, 1).astype(np.int64) * N + np.max(s.excl, 1))).to(dev)
    at = torch.searchsorted(ex, key).clamp(max=len(ex) - 1)
    ij = ij[:, ex[at] != key]
    q = torch.from_numpy(np.asarray(s.nbonds["q"])).to(dev).double()
    t = torch.from_numpy(np.asarray(s.nbonds["typeIdx"]).astype(np.int64)).to(dev)
    vdw = torch.from_numpy(np.ascontiguousarray(s.vdw)).to(dev)
    sb = torch.from_numpy(np.asarray(s.nbonds["siteBlock"]).astype(np.int64)).to(dev)
    lam = torch.from_numpy(s.lambdas().astype(np.float32)).to(dev).double().requires_grad_(True)
    force = torch.zeros_like(x)
    lforce = torch.zeros_like(lam)
    energy = 0.0
    for c in torch.split(ij, 8_000_000, dim=1):
        i, j = c
        d = x[i] - x[j]
        d = d - box * torch.round(d / box)
        r = d.square().sum(1).sqrt().requires_grad_(True)
        c12, c6 = vdw[t[i], t[j]].double().unbind(1)
        qq = float(np.float32(systems.KELEC_AKMA)) * q[i] * q[j]
        if s.msld is None:
            E = _pair_energy(s, r, qq, c12, c6)
        else:
            bi, bj = sb[i], sb[j]
            li = torch.where(bi > 0, lam[bi & 0xFFFF], 1.0)
            lj = torch.where(bj > 0, lam[bj & 0xFFFF], 1.0)
            scale = torch.where((bi >> 16) == (bj >> 16), torch.where(bi == bj, li, 0.0), li * lj)
            reff = r
            if s.msld.useSoftCore:
                rs = systems.SOFTCORE_RADIUS_AKMA * (1 - scale)
                u = r / rs.clamp(min=1e-30)
                reff = torch.where(((bi | bj) > 0) & (r < rs), rs * (u ** 3 * (1 - 0.5 * u) + 0.5), r)
            E = scale * _pair_energy(s, reff, qq, c12, c6)
        wanted = [r] + ([lam] if s.msld is not None else [])
        g = torch.autograd.grad(E.sum(), wanted)
        f = (g[0] / r.detach())[:, None] * d
        force.index_add_(0, i, f)
        force.index_add_(0, j, -f)
        if s.msld is not None:
            lforce += g[1]
        energy += float(E.detach().sum())
    lforce[0] = 0.0  # the environment's lambda is no variable
    return force.reshape(-1), lforce.detach(), torch.tensor([energy], dtype=torch.float64)


def _spline(u, order):
    """Weights M_n and derivatives at the n grid points from floor(u) on (cardinal B-splines)."""
    f = u - torch.floor(u)
    m = [torch.ones_like(f)]  # M_1(f + j)
    prev = m
    zero = torch.zeros_like(f)
    for k in range(2, order + 1):
        prev = m
        get = lambda j, v: v[j] if 0 <= j < len(v) else zero  # noqa: E731
        m = [((f + j) * get(j, prev) + (k - f - j) * get(j - 1, prev)) / (k - 1) for j in range(k)]
    get = lambda j: prev[j] if 0 <= j < len(prev) else zero  # noqa: E731
    der = [get(j) - get(j - 1) for j in range(order)]
    return torch.stack(m[::-1], 1), torch.stack(der[::-1], 1)


def _moduli(K, order, dev):
    m = {1: 1.0}  # M_2 at the integers
    for k in range(3, order + 1):
        m = {l: (l * m.get(l, 0.0) + (k - l) * m.get(l - 1, 0.0)) / (k - 1) for l in range(k + 1)}
    ph = 2 * math.pi * torch.arange(K, dtype=torch.float64, device=dev) / K
    re = sum(m.get(l, 0.0) * torch.cos(ph * l) for l in range(1, order))
    im = sum(m.get(l, 0.0) * torch.sin(ph * l) for l in range(1, order))
    return 1 / (re * re + im * im)


def _exact_pme(s, xyz, order, K):
    dev = _dev()
    x = torch.from_numpy(xyz).to(dev).double()
    box = torch.from_numpy(np.asarray(s.box, np.float32)).to(dev).double()
    q = torch.from_numpy(np.asarray(s.nbonds["q"])).to(dev).double()
    beta = float(np.float32(s.betaEwald))
    ke = float(np.float32(systems.KELEC_AKMA))
    u = x * K / box
    w, dw = zip(*[_spline(u[:, d], order) for d in range(3)])
    g0 = torch.floor(u).long()
    at = [(g0[:, d, None] + torch.arange(order, device=dev)) % K for d in range(3)]
    idx = ((at[0][:, :, None, None] * K + at[1][:, None, :, None]) * K + at[2][:, None, None, :]).reshape(-1)
    grid = torch.zeros(K ** 3, dtype=torch.float64, device=dev)
    grid.index_add_(0, idx, torch.einsum("n,na,nb,nc->nabc", q, w[0], w[1], w[2]).reshape(-1))
    spec = torch.fft.rfftn(grid.view(K, K, K))
    m = torch.fft.fftfreq(K, 1.0 / K, dtype=torch.float64, device=dev)
    mz = torch.arange(K // 2 + 1, dtype=torch.float64, device=dev)
    k2 = (m / box[0])[:, None, None] ** 2 + (m / box[1])[None, :, None] ** 2 + (mz / box[2])[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    b = _moduli(K, order, dev)
    infl = b[:, None, None] * b[None, :, None] * b[None, None, :K // 2 + 1] * torch.exp(-math.pi ** 2 / beta ** 2 * k2) / k2
    infl *= ke / (2 * math.pi * float(box.prod()))
    infl[0, 0, 0] = 0.0
    phi = torch.fft.irfftn(spec * infl, s=(K, K, K), norm="forward").reshape(-1)
    P = phi[idx].view(len(q), order, order, order)
    f = torch.stack([torch.einsum("nabc,na,nb,nc->n", P, *(dw[d] if d == e else w[d] for d in range(3)))
                     for e in range(3)], 1)
    e = (q * torch.einsum("nabc,na,nb,nc->n", P, *w)).sum()
    return (2 * q[:, None] * f * K / box).reshape(-1), e.reshape(1)


def _exact_mlp(case, seed):
    dev = _dev()
    bf = lambda t: t.float().bfloat16().double()  # noqa: E731  (the network's stored precision)
    x, y = (torch.from_numpy(a).to(dev).double() for a in _mlp_data(case, seed))
    net = BF16MLP([alf.FEAT_PAD, *alf.HIDDEN, alf.OUT_PAD], max_batch=1, seed=seed % 1000003, device=dev)
    W = [w.double() for w in net.W]
    L = len(W)
    h, hs, zs = bf(x), [], []
    for l in range(L):
        hs.append(h)
        z = h @ bf(W[l]).T
        zs.append(z)
        h = bf(z * torch.sigmoid(z)) if l < L - 1 else z
    if not case["train"]:
        return h
    M = len(x)
    loss = ((h - y) ** 2).sum() / M
    g = 2 * (h - y) / M
    gW, gb = [None] * L, [None] * L
    for l in range(L - 1, -1, -1):
        if l < L - 1:
            sg = torch.sigmoid(zs[l])
            g = g * sg * (1 + zs[l] * (1 - sg))
        gW[l], gb[l] = (bf(g).T @ hs[l]).reshape(-1), g.sum(0)
        g = bf(g) @ bf(W[l])
    # first Adam step from zero moments
    step = lambda w, d: w - 1e-3 * d / (d.abs() + 1e-8)  # noqa: E731
    return {"loss": loss.reshape(1), "gW": gW, "gb": gb,
            "W": [step(w.reshape(-1), d).reshape(w.shape) for w, d in zip(W, gW)],
            "b": [step(torch.zeros_like(d), d) for d in gb]}
