"""Timed cases of the MDDF engine: what users of this package run, through its public entry points.

A case is one system (or one batch of systems), its frames and its options; one pass
is what a user's program does with them:

  engine  frames given to an Engine that the program keeps, and the counts read back
  dcd     the same with the bytes of a DCD trajectory file
  batch   several engines' frames as one Batch.submit, and every engine's counts
  mddf    the whole mddf(...) call on a trajectory, from engine to Result

Systems are seeded and made on the GPU.  Three kinds of solute:

  self    the solvent itself (an autocorrelation MDDF)
  mols    many small molecules in another solvent
  chain   one large molecule (a random-walk chain that fills a sphere)
"""
import importlib
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

BINSTEP = 0.02
COUNTS = ("md_count", "md_count_random", "rdf_count", "rdf_count_random", "solute_group_count",
          "solute_group_count_random", "solvent_group_count", "solvent_group_count_random")
RAW = ("md", "md_random", "rdf", "rdf_random", "solute_group", "solute_group_random", "solvent_group",
       "solvent_group_random")
RESULT = ("md_count", "md_count_random", "rdf_count", "rdf_count_random", "mddf", "rdf", "kb", "kb_rdf",
          "coordination_number", "solute_group_count", "solvent_group_count")

_package = None


def package():
    global _package
    if _package is None:
        _package = importlib.import_module("__graft_entry__").load_package()
    return _package


def case(name, **kw):
    c = dict(entry="engine", solute="self", solute_mols=1, solute_atoms=1, solvent_mols=1, solvent_atoms=3, edge=60.0,
             gamma=90.0, chain_radius=0.0, clearance=0.0, group=0, cutoff=10.0, dbulk=0.0, samples=10, frames=10,
             sigma=0.5, dtype="f32", memory="device", systems=1, coordination=False)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: a few molecules, one frame at a time (a script that looks at frames as they come)
        case("one small frame", solute_mols=40, solvent_mols=40, solvent_atoms=3, solute_atoms=3, edge=18.0, cutoff=6.0,
             samples=4, frames=1, sigma=0.1, dtype="f64", memory="host"),
        # co-solvent around itself in a solvated-protein box (the NAMD example), bulk between 8 and 10 A
        case("tmao-tmao", solute_mols=181, solute_atoms=14, solvent_mols=181, solvent_atoms=14, edge=84.5, dbulk=8.0,
             frames=20, dtype="f64", memory="host"),
        # co-solvent around the protein of the same box, read from the DCD file
        case("protein-tmao dcd", entry="dcd", solute="chain", solute_atoms=1463, solvent_mols=181, solvent_atoms=14,
             edge=84.5, chain_radius=18.0, clearance=2.0, dbulk=8.0, frames=20, memory="host"),
        # water around each co-solvent molecule of the same box
        case("water-tmao", solute="mols", solute_mols=181, solute_atoms=14, solvent_mols=19338, edge=84.5, dbulk=8.0,
             frames=20),
        # water around water, the same box
        case("water-water", solute_mols=19338, solute_atoms=3, solvent_mols=19338, edge=84.5, dbulk=8.0, frames=16),
        # a 1,200-atom chain in 5,000 waters, FP64 coordinates from host memory
        case("chain in water", solute="chain", solute_atoms=1200, solvent_mols=5000, edge=60.0, chain_radius=25.0,
             clearance=2.0, group=10, frames=10, dtype="f64", memory="host"),
        # a compact 20,000-atom chain: 50,000 waters, then 2,000 14-atom co-solvent molecules
        case("large chain, water", solute="chain", solute_atoms=20000, solvent_mols=50000, edge=120.0, chain_radius=35.0,
             group=10, cutoff=12.0, frames=8),
        case("large chain, cosolvent", solute="chain", solute_atoms=20000, solvent_mols=2000, solvent_atoms=14, edge=120.0,
             chain_radius=35.0, group=10, cutoff=12.0, frames=16),
        # the headline: 10,000 14-atom molecules around themselves in a triclinic cell
        case("self triclinic", solute_mols=10000, solute_atoms=14, solvent_mols=10000, solvent_atoms=14, edge=110.0,
             gamma=60.0, samples=5, frames=64, sigma=0.4),
        # the largest request of a serving load: 35,000 molecules, the widest cutoff
        case("self large", solute_mols=35000, solute_atoms=14, solvent_mols=35000, solvent_atoms=14, edge=167.0,
             gamma=60.0, cutoff=14.0, samples=5, frames=8, sigma=0.4),
        # many systems of uneven size (2,000 to 200,000 atoms) in one resident batch
        case("batch of systems", entry="batch", solute="chain", solute_atoms=10000, solvent_mols=63333, edge=0.0, group=10,
             frames=8, systems=24),
        # a whole mddf() call on a 43,000-atom system
        case("mddf call", entry="mddf", solute="chain", solute_atoms=2150, solvent_mols=13616, edge=75.5,
             chain_radius=22.6, group=10, frames=50, memory="host"),
    ]


def log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def pairs(c):
    """Expected atom pairs within the cutoff in one pass: (real frames, random insertions)."""
    if c["entry"] == "batch":
        parts = [pairs(s) for s in batch_systems(c)]
        return sum(p[0] for p in parts), sum(p[1] for p in parts)
    volume = c["edge"] ** 3 * math.sin(math.radians(c["gamma"]))
    near = 4.0 / 3.0 * math.pi * c["cutoff"] ** 3 * c["solvent_mols"] * c["solvent_atoms"] / volume
    near = min(near, c["solvent_mols"] * c["solvent_atoms"])
    real = c["frames"] * c["solute_mols"] * c["solute_atoms"] * near * (0.5 if c["solute"] == "self" else 1.0)
    rand = 0 if c["coordination"] else c["frames"] * c["samples"] * c["solute_atoms"] * near
    return real, rand


MOST_PAIRS = 1.3e9  # about half of what the largest listed case has


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["self", "self", "self", "mols", "mols", "chain", "chain", "chain", "chain", "batch", "mddf", "dcd"])
    opts = dict(cutoff=rng.choice([8.0, 8.5, 9.0, 9.5, 10.0, 10.0, 10.5, 11.0, 12.0, 12.5, 13.0, 14.0]), samples=rng.choice([1, 3, 5, 10, 10, 20]),
                dtype=rng.choice(["f32", "f32", "f64"]), memory=rng.choice(["device", "device", "host"]),
                coordination=rng.random() < 0.1, frames=int(log_uniform(rng, 1, 64)))
    if rng.random() < 0.4:
        opts["dbulk"] = opts["cutoff"] - 2.0
    density = rng.uniform(0.08, 0.125)  # atoms per cubic Angstrom
    if kind == "self":
        apm = rng.choice([1, 3, 3, 5, 9, 14, 14, 20, 31])
        n = int(log_uniform(rng, 1500, 500000) / apm)
        gamma = rng.choice([90.0, 90.0, 60.0, 75.0])
        edge = (n * apm / density / math.sin(math.radians(gamma))) ** (1 / 3)
        c = case(None, solute_mols=n, solute_atoms=apm, solvent_mols=n, solvent_atoms=apm, edge=edge, gamma=gamma, **opts)
    elif kind == "mols":
        aps, apv = rng.choice([3, 5, 14, 20, 27]), rng.choice([1, 3, 3, 5, 12])
        n, m = int(log_uniform(rng, 20, 2000)), int(log_uniform(rng, 500, 40000))
        gamma = rng.choice([90.0, 90.0, 60.0])
        edge = ((n * aps + m * apv) / density / math.sin(math.radians(gamma))) ** (1 / 3)
        c = case(None, solute="mols", solute_mols=n, solute_atoms=aps, solvent_mols=m, solvent_atoms=apv, edge=edge,
                 gamma=gamma, **opts)
    else:
        apv = 3 if kind == "batch" else rng.choice([1, 3, 3, 3, 5, 14])
        atoms = log_uniform(rng, 8000, 200000)
        aps = max(60, int(atoms * log_uniform(rng, 0.02, 0.15)))
        m = max(20, int((atoms - aps) / apv))
        edge = (atoms / density) ** (1 / 3)
        if kind in ("mddf", "dcd"):
            opts["memory"] = "host"
        if kind == "dcd":
            opts["dtype"] = "f32"
        if kind == "batch":
            opts.update(dtype="f32", memory="device", coordination=False, cutoff=10.0, dbulk=0.0, samples=10)
        c = case(None, entry=kind if kind in ("batch", "mddf", "dcd") else "engine", solute="chain", solute_atoms=aps,
                 solvent_mols=m, solvent_atoms=apv, edge=0.0 if kind == "batch" else edge, chain_radius=0.3 * edge,
                 clearance=rng.choice([0.0, 2.0]), group=rng.choice([0, 10]) if aps < 3000 else 10, **opts)
        if kind == "batch":
            c["systems"] = rng.randrange(4, 25)
            c["chain_radius"] = 0.0
    if c["edge"]:  # a box of at least two cutoffs between faces
        least = (2.0 * c["cutoff"] + 1.0) / math.sin(math.radians(c["gamma"]))
        c["edge"] = float("%.3f" % max(c["edge"], least))
    if c["entry"] == "mddf":
        c["frames"] = max(2, c["frames"])
    work = sum(pairs(c))
    if work > MOST_PAIRS:
        c["frames"] = max(1, int(c["frames"] * MOST_PAIRS / work))
    return c


def batch_systems(c):
    """The systems of a batch: total atoms spread over a factor of 100 up to the case's own, a chain of 5 % of the
    atoms and water at 0.1 atoms per cubic Angstrom."""
    out = []
    top = c["solute_atoms"] + c["solvent_mols"] * c["solvent_atoms"]
    for k in range(c["systems"]):
        n = top * 100.0 ** (-((k * 0.6180339887) % 1.0) if k else 0.0)
        aps = max(33, int(0.05 * n))
        m = max(1, int((n - aps) / 3))
        s = dict(c, entry="engine", solute_atoms=aps, solvent_mols=m, solvent_atoms=3, edge=((aps + 3 * m) / 0.1) ** (1 / 3))
        s["chain_radius"] = 0.3 * s["edge"]
        s["edge"] = max(s["edge"], 2.0 * c["cutoff"] + 1.0)
        out.append(s)
    return out


# ------------------------------------------------------------------- inputs
def lattice(c):
    g = math.radians(c["gamma"])
    H = np.diag([c["edge"]] * 3)
    if c["gamma"] != 90.0:
        H[0, 1], H[1, 1] = c["edge"] * math.cos(g), c["edge"] * math.sin(g)
    return H


def template(atoms, gen):
    """A rigid molecule about its centre: water for 3 atoms, else atoms uniform in a ball (4 A for 14 atoms)."""
    if atoms == 3:
        r, t = 0.9572, math.radians(104.52)
        x = torch.tensor([[0.0, 0.0, 0.0], [r, 0.0, 0.0], [r * math.cos(t), r * math.sin(t), 0.0]], dtype=torch.float64)
    else:
        x = torch.randn((atoms, 3), generator=gen, dtype=torch.float64)
        x = x / x.norm(dim=1, keepdim=True) * torch.rand((atoms, 1), generator=gen, dtype=torch.float64) ** (1 / 3)
        x = x * 4.0 * (atoms / 14.0) ** (1 / 3)
    return x - x.mean(0)


def rotations(q):
    w, x, y, z = (q / q.norm(dim=-1, keepdim=True)).unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).reshape(q.shape[:-1] + (3, 3))


def chain(atoms, radius, rng):
    """Random walk of 1.53 A bonds that stays inside a sphere."""
    steps = rng.standard_normal((4 * atoms + 64, 3))
    steps *= 1.53 / np.linalg.norm(steps, axis=1, keepdims=True)
    r2, p, out, k, tries = max(radius, 3.0) ** 2, (0.0, 0.0, 0.0), [(0.0, 0.0, 0.0)], 0, steps.tolist()
    while len(out) < atoms:
        dx, dy, dz = tries[k % len(tries)]
        k += 1
        q = (p[0] + dx, p[1] + dy, p[2] + dz)
        if q[0] * q[0] + q[1] * q[1] + q[2] * q[2] <= r2:
            p = q
            out.append(q)
    return np.array(out)


def molecules(n, tpl, H, gen, avoid=None, clearance=0.0):
    """Centres and orientations of n molecules at uniform places, none with its centre closer than `clearance` to a
    point of `avoid`."""
    dev = gen.device
    h = torch.as_tensor(H, device=dev)
    centres = []
    have = 0
    while have < n:
        f = torch.rand((int((n - have) * 1.5) + 64, 3), generator=gen, device=dev, dtype=torch.float64) @ h.T
        if avoid is not None and clearance > 0:
            keep = torch.ones(len(f), dtype=torch.bool, device=dev)
            for b in range(0, len(f), 4096):
                keep[b:b + 4096] = torch.cdist(f[b:b + 4096].float(), avoid.float()).min(1).values > clearance + 0.6
            f = f[keep]
        centres.append(f[: n - have])
        have += len(centres[-1])
    q = torch.randn((n, 4), generator=gen, device=dev, dtype=torch.float64)
    body = torch.einsum("nij,aj->nai", rotations(q), tpl.to(dev))
    return torch.cat(centres), body


def jittered(centres, body, frames, sigma, gen, dtype):
    """[frames, atoms, 3]: the molecules moved and turned rigidly from frame to frame."""
    n, atoms = body.shape[:2]
    rg = max(1e-3, float((body[0] ** 2).sum(1).mean().sqrt()))
    out = torch.empty((frames, n * atoms, 3), dtype=dtype, device=body.device)
    for f in range(frames):
        move = torch.randn((n, 1, 3), generator=gen, device=body.device, dtype=torch.float64) * sigma
        turn = torch.randn((n, 3), generator=gen, device=body.device, dtype=torch.float64) * (sigma / rg / math.sqrt(3.0) / 2)
        R = rotations(torch.cat([torch.ones_like(turn[:, :1]), turn], 1))
        out[f] = (torch.einsum("nij,naj->nai", R, body) + centres[:, None] + move).reshape(-1, 3).to(dtype)
    return out


def system(c, seed):
    """(solute frames, solvent frames or None, cells) of one system, on the GPU."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(1000003 * seed + 17)
    host = torch.Generator().manual_seed(1000003 * seed + 18)
    dtype = torch.float32 if c["dtype"] == "f32" else torch.float64
    H = lattice(c)
    cells = np.repeat(H[None], c["frames"], axis=0)
    solvent = template(c["solvent_atoms"], host)
    if c["solute"] == "self":
        centres, body = molecules(c["solvent_mols"], solvent, H, gen)
        return jittered(centres, body, c["frames"], c["sigma"], gen, dtype), None, cells
    if c["solute"] == "mols":
        centres, body = molecules(c["solute_mols"], template(c["solute_atoms"], host), H, gen)
        xs = jittered(centres, body, c["frames"], c["sigma"], gen, dtype)
        avoid = None
    else:
        walk = chain(c["solute_atoms"], c["chain_radius"], np.random.default_rng(seed)) + 0.5 * c["edge"]
        avoid = torch.as_tensor(walk, device=dev)
        noise = torch.randn((c["frames"],) + walk.shape, generator=gen, device=dev, dtype=torch.float64)
        xs = (avoid + c["sigma"] * noise).to(dtype)
    centres, body = molecules(c["solvent_mols"], solvent, H, gen, avoid, c["clearance"])
    return xs, jittered(centres, body, c["frames"], c["sigma"], gen, dtype), cells


def options(c, seed):
    """Engine(...) keywords of one system."""
    cm = package()
    dbulk = c["dbulk"] or c["cutoff"]
    kw = dict(solute_nmols=c["solute_mols"], solute_natomspermol=c["solute_atoms"], solvent_nmols=c["solvent_mols"],
              solvent_natomspermol=c["solvent_atoms"], autocorrelation=c["solute"] == "self", irefatom=1,
              cutoff=c["cutoff"], binstep=BINSTEP, dbulk=dbulk, usecutoff=bool(c["dbulk"]),
              nbins=cm.setbin(c["cutoff"], BINSTEP), n_random_samples=c["samples"], seed=321 + seed % 1000,
              coordination_number_only=c["coordination"])
    if c["group"]:
        g = c["group"]
        kw.update(solute_groups=[[i // g] for i in range(c["solute_atoms"])], solute_ngroups=-(-c["solute_atoms"] // g))
    return kw


def dcd_bytes(xs, xv):
    """Frames as a DCD file holds them after its header (unit-cell record, then the x, y and z records), the solute's
    atoms first, and the layout of one frame."""
    frames, ns, nv = xs.shape[0], xs.shape[1], xv.shape[1]
    n = ns + nv
    record = 8 + 4 * n
    size = 56 + 3 * record
    raw = np.zeros((frames, size), np.uint8)
    xyz = np.concatenate([xs, xv], 1).astype(np.float32)
    for k in range(3):
        at = 56 + k * record + 4
        raw[:, at:at + 4 * n] = np.ascontiguousarray(xyz[:, :, k]).view(np.uint8).reshape(frames, -1)
    lay = dict(natoms=n, frame_bytes=size, x_offset=60, y_offset=60 + record, z_offset=60 + 2 * record, big_endian=False,
               solute_atoms=np.arange(ns), solvent_atoms=np.arange(ns, n))
    return raw, lay


def prepare(c, seed):
    cm = package()
    if c["entry"] == "batch":
        engines, items = [], []
        for k, s in enumerate(batch_systems(c)):
            engines.append(cm.Engine(**options(s, seed + k)))
            items.append(system(s, seed + 100 * k + 1))
        return dict(entry="batch", engines=engines, batch=cm.Batch(engines), items=items)
    xs, xv, cells = system(c, seed)
    if c["memory"] == "host":
        xs, xv = xs.cpu().numpy(), None if xv is None else xv.cpu().numpy()
    if c["entry"] == "mddf":
        ns, nv = c["solute_atoms"], c["solvent_mols"] * c["solvent_atoms"]
        groups = {}
        if c["group"]:
            g = c["group"]
            atoms = [list(range(i + 1, min(i + g, ns) + 1)) for i in range(0, ns, g)]
            groups = dict(group_atom_indices=atoms, group_names=["G%d" % i for i in range(len(atoms))])
        solute = cm.AtomSelection.from_indices(list(range(1, ns + 1)), nmols=1, **groups)
        solvent = cm.AtomSelection.from_indices(list(range(ns + 1, ns + nv + 1)), natomspermol=c["solvent_atoms"])
        bulk = dict(bulk_range=(c["dbulk"], c["cutoff"])) if c["dbulk"] else dict(dbulk=c["cutoff"], usecutoff=False)
        opts = cm.make_options(n_random_samples=c["samples"], binstep=BINSTEP, irefatom=1, seed=321 + seed % 1000,
                               silent=True, **bulk)
        traj = cm.ArrayTrajectory(solute, solvent, solute_frames=xs, solvent_frames=xv, cells=cells)
        return dict(entry="mddf", traj=traj, opts=opts, coordination=c["coordination"])
    eng = cm.Engine(**options(c, seed))
    if c["entry"] == "dcd":
        raw, lay = dcd_bytes(xs, xv)
        eng.set_dcd_layout(**lay)
        return dict(entry="dcd", eng=eng, raw=raw, cells=cells)
    return dict(entry="engine", eng=eng, xs=xs, xv=xv, cells=cells)


def run(s):
    cm = package()
    if s["entry"] == "mddf":
        R = cm.mddf(s["traj"], s["opts"], coordination_number_only=s["coordination"])
        return {k: getattr(R, k) for k in RESULT}
    if s["entry"] == "batch":
        for e in s["engines"]:
            e.reset()
        s["batch"].submit(s["items"])
        got = [e.raw_counts() for e in s["engines"]]
        return {k: np.concatenate([g[k] for g in got]) for k in RAW}
    eng = s["eng"]
    eng.reset()
    if s["entry"] == "dcd":
        eng.submit_dcd(s["raw"], s["cells"])
    else:
        eng.submit(s["xs"], s["xv"], s["cells"])
    out = eng.counts()
    return {k: out[k] for k in COUNTS + ("volume_total",)}


def work(c):
    """Coordinates read once, histograms written once; 8 FP32 operations (three differences, a product and two
    multiply-adds) for each atom pair within the cutoff, real and inserted."""
    parts = batch_systems(c) if c["entry"] == "batch" else [c]
    nbytes = 0
    for p in parts:
        atoms = p["solvent_mols"] * p["solvent_atoms"]
        if p["solute"] != "self":
            atoms += p["solute_mols"] * p["solute_atoms"]
        groups = (-(-p["solute_atoms"] // p["group"]) if p["group"] else p["solute_atoms"]) + p["solvent_atoms"]
        nbytes += p["frames"] * atoms * 3 * (4 if p["dtype"] == "f32" else 8)
        nbytes += 2 * (2 + groups) * int(round(p["cutoff"] / BINSTEP)) * 8
    return {"bytes": nbytes, "flops": 8.0 * sum(pairs(c))}


# -------------------------------------------------------------------- exact
MOST_EXACT = 1.5e10  # atom-pair distances


def exact(c, seed):
    """The counts of the real frames by brute force over all pairs and images in 64 bits.  The random insertions
    follow the package's own stream of placements and have no value here."""
    if c["entry"] == "batch":
        return None
    self_mode = c["solute"] == "self"
    images = 27 if c["gamma"] != 90.0 else 1
    ms, aps, mv, apv = c["solute_mols"], c["solute_atoms"], c["solvent_mols"], c["solvent_atoms"]
    if float(ms) * aps * mv * apv * c["frames"] * images > MOST_EXACT:
        return None
    xs, xv, cells = system(c, seed)
    xs = xs.double()
    xv = xs if self_mode else xv.double()
    H = torch.as_tensor(lattice(c), device=xs.device)
    Hi = torch.linalg.inv(H)
    nb = int(round(c["cutoff"] / BINSTEP))
    g = c["group"] or 1
    ngroups = -(-aps // g)
    z = lambda *n: torch.zeros(n, dtype=torch.float64, device=xs.device)  # noqa: E731
    md, rdf, gs, gv = z(nb), z(nb), z(ngroups * nb), z(apv * nb)

    def bins(d):
        return (torch.ceil(d / BINSTEP).long().clamp_min(1) - 1)

    shifts = [(0, 0, 0)] if images == 1 else [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)]
    per = max(1, int(3e7 // (ms * aps * apv)))  # solvent molecules at a time
    rows = max(1, int(3e7 // (aps * apv * min(per, mv))))
    for f in range(c["frames"]):
        for s0 in range(0, ms, rows):
            x = xs[f, s0 * aps:min(ms, s0 + rows) * aps]
            sn = len(x) // aps
            for v0 in range(0, mv, per):
                y = xv[f, v0 * apv:min(mv, v0 + per) * apv]
                vn = len(y) // apv
                d = [y[None, :, k] - x[:, k, None] for k in range(3)]
                n = [torch.round(Hi[k, 0] * d[0] + Hi[k, 1] * d[1] + Hi[k, 2] * d[2]) for k in range(3)]
                d2 = None
                for sh in shifts:
                    m = [n[k] + sh[k] for k in range(3)]
                    e2 = sum((d[k] - (H[k, 0] * m[0] + H[k, 1] * m[1] + H[k, 2] * m[2])) ** 2 for k in range(3))
                    d2 = e2 if d2 is None else torch.minimum(d2, e2)
                d2 = d2.view(sn, aps, vn, apv)
                ref = d2[:, :, :, 0].amin(1).sqrt()
                best, at = d2.permute(0, 2, 1, 3).reshape(sn, vn, aps * apv).min(-1)
                best = best.sqrt()
                keep = best <= c["cutoff"]
                rkeep = ref <= c["cutoff"]
                if self_mode:
                    other = (s0 + torch.arange(sn, device=x.device))[:, None] != (v0 + torch.arange(vn, device=x.device))[None]
                    keep, rkeep = keep & other, rkeep & other
                b, a = bins(best[keep]), at[keep]
                md += torch.bincount(b, minlength=nb).double()
                rdf += torch.bincount(bins(ref[rkeep]), minlength=nb).double()
                w = 0.5 if self_mode else 1.0
                gs += w * torch.bincount((a // apv // g) * nb + b, minlength=ngroups * nb).double()
                if self_mode:
                    gs += w * torch.bincount((a % apv) * nb + b, minlength=ngroups * nb).double()
                else:
                    gv += torch.bincount((a % apv) * nb + b, minlength=apv * nb).double()
    found = {"md_count": md, "rdf_count": rdf, "solute_group_count": gs.view(-1, nb), "solvent_group_count": gv.view(-1, nb)}
    found = {k: v.cpu().numpy() for k, v in found.items()}
    if c["entry"] == "mddf":
        found = {k: v / c["frames"] for k, v in found.items()}
        found["coordination_number"] = np.cumsum(found["md_count"])
        return {k: found.get(k) for k in RESULT}
    found["volume_total"] = float(c["frames"] * abs(np.linalg.det(lattice(c))))
    return {k: found.get(k) for k in COUNTS + ("volume_total",)}
