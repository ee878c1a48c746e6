"""Workloads of the gravity step as its users run it, for timing and comparing.

A case is one of four ways into the library:

  loop     a simulation resident on the GPU: `steps` frames per call
           (Simulation.step), then the state read back into page-locked
           arrays (ge_download), as a viewer does every frame and a recording
           run every few frames
  host     the drop-in frame on page-locked host arrays (Simulation.frame_host)
  records  the drop-in frame on the application's own particle records
           (Simulation.frame_aos), page-locked
  batch    many independent simulations in one context: `steps` frames, then
           the whole state read back

on a 2D disk galaxy, two disks that meet, or a 3D Plummer sphere, in the
reference arithmetic ("fast") or the mixed mode, at opening angles 0.5 to 1.0,
with the options an application turns on: heat exchange, periodic wrap, the
direct sum below 5,000 particles.  `flung` throws a few particles far out, as
close passes do after some thousand frames: the root box is then some 20 times
the disks, and the disks' particles share long runs of equal Morton keys.
"""
import importlib
import math

import numpy as np
import torch

ge = importlib.import_module("galaxy-engine_b200")

DT = 1e-3
DOMAIN = 100.0          # side of the periodic domain, larger than the systems
EXACT_PAIRS = 4e11      # pair terms that the FP64 direct sum of exact() may take


def _case(**kw):
    c = dict(entry="loop", dims=2, n=1, sims=1, mode="fast", theta=0.7, steps=1, heat=False,
             periodic=False, direct=False, flung=False)
    c.update(kw)
    return c


def listed():
    return [
        # a small scene on screen: below 5,000 particles the application takes
        # the direct sum, and the viewer reads every frame
        _case(name="viewer 2k direct", n=2000, direct=True),
        # the single-galaxy workload, recorded every 16 frames: latency of a step
        _case(name="disk 16k", n=16384, steps=16),
        # temperatures switched on, the application's default opening angle
        _case(name="disk 60k heat", n=60013, heat=True, theta=0.8, steps=4),
        # the two-galaxy workload, recorded every 12 frames: the headline
        _case(name="two disks 1M", n=1048576, steps=12),
        # the same system late in its run, at the coarse end of the angles
        _case(name="two disks 700k flung", n=700001, theta=1.0, steps=8, flung=True),
        # a 3D cluster in the application's periodic domain, every frame read
        _case(name="plummer 250k periodic", dims=3, n=250007, periodic=True),
        # the accurate mode on the two-galaxy workload
        _case(name="two disks 1M mixed", n=1048576, mode="mixed", steps=4),
        # the largest cluster in the accurate mode, at the fine end of the angles
        _case(name="plummer 4M mixed", dims=3, n=4194304, mode="mixed", theta=0.5, steps=2),
        # a parameter study: 64 disks of 1k to 64k particles side by side, every
        # frame read
        _case(name="batch of 64 mixed", entry="batch", n=65536, sims=64, mode="mixed"),
        # the same in the reference arithmetic, more and smaller ones
        _case(name="batch of 96 fast", entry="batch", n=16384, sims=96, steps=4),
        # the application's frame with its arrays on the host
        _case(name="host frame 262k", entry="host", n=262144),
        # ... and with its own records
        _case(name="records 100k", entry="records", n=100003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes from 1,000 particles up (log-uniform), any of the
    entries, modes, angles and options."""
    entry = rng.choice(("loop", "loop", "loop", "batch", "host", "records"))
    dims = rng.choice((2, 2, 3))
    c = _case(entry=entry, dims=dims, theta=round(rng.uniform(0.5, 1.0), 2),
              mode=rng.choice(("fast", "fast", "mixed")))
    if entry == "batch":
        c["sims"] = rng.randint(2, 100)
        c["n"] = _log(rng, 1100, 40000 if dims == 2 else 15000)
        c["steps"] = rng.randint(1, 6)
        return c
    if entry in ("host", "records"):
        c["n"] = _log(rng, 1000, 1000000 if entry == "host" and dims == 2 else 300000)
        c["mode"] = "fast"
    else:
        c["n"] = _log(rng, 1000, 1500000 if dims == 2 else 1000000)
        most = (16 if dims == 2 else 8) if c["n"] < 300000 else (8 if dims == 2 else 2)
        c["steps"] = rng.randint(1, most)
        c["flung"] = dims == 2 and rng.random() < 0.25
    if c["mode"] == "fast":
        c["direct"] = c["n"] < 5000 and rng.random() < 0.5
        if entry == "loop" and not c["direct"]:
            c["heat"] = rng.random() < 0.2
        c["periodic"] = not c["flung"] and rng.random() < 0.2
    return c


# --- inputs ----------------------------------------------------------------

def _disk(g, n, total, center=(0.0, 0.0), bulk=(0.0, 0.0)):
    """Exponential disk of n particles (scale length 1, cut at 5): masses
    1 / total around a central mass of 0.1, on circular orbits with a
    dispersion of 0.02."""
    cut = 1.0 - math.exp(-5.0)
    r = np.concatenate([[0.0], -np.log(1.0 - g.random(n - 1) * cut)])
    phi = g.random(n) * (2.0 * math.pi)
    inside = (1.0 - np.exp(-r) * (1.0 + r)) / (1.0 - 6.0 * math.exp(-5.0)) * (n / total) + 0.1
    v = np.sqrt(inside / np.maximum(r, 1e-12))
    v[0] = 0.0
    s = g.normal(0.0, 0.02, (2, n))
    s[:, 0] = 0.0
    m = np.full(n, 1.0 / total)
    m[0] = 0.1
    return dict(x=r * np.cos(phi) + center[0], y=r * np.sin(phi) + center[1],
                vx=s[0] - v * np.sin(phi) + bulk[0], vy=s[1] + v * np.cos(phi) + bulk[1], m=m)


def _two_disks(g, n):
    """Two disks 10 apart that approach each other at 0.5."""
    half = n // 2
    bx, by = 0.25 * math.cos(math.radians(30.0)), 0.25 * math.sin(math.radians(30.0))
    a = _disk(g, half, n, (-5.0, 0.0), (bx, -by))
    b = _disk(g, n - half, n, (5.0, 0.0), (-bx, by))
    return {k: np.concatenate([a[k], b[k]]) for k in a}


def _ball(g, n):
    """n directions, uniform on the sphere."""
    c = 2.0 * g.random(n) - 1.0
    s, p = np.sqrt(1.0 - c * c), 2.0 * math.pi * g.random(n)
    return s * np.cos(p), s * np.sin(p), c


def _plummer(g, n):
    """Plummer sphere of scale radius 1 and mass 1 (outermost 0.1 % left out),
    isotropic velocities by rejection from q^2 (1 - q^2)^3.5."""
    r = 1.0 / np.sqrt((g.random(n) * 0.999 + 1e-12) ** (-2.0 / 3.0) - 1.0)
    q = np.zeros(0)
    while len(q) < n:
        t, u = g.random((2, 4 * (n - len(q)) + 64))
        q = np.concatenate([q, t[0.1 * u < t * t * (1.0 - t * t) ** 3.5]])
    v = q[:n] * math.sqrt(2.0) * (1.0 + r * r) ** -0.25
    (x, y, z), (vx, vy, vz) = _ball(g, n), _ball(g, n)
    return dict(x=r * x, y=r * y, z=r * z, vx=v * vx, vy=v * vy, vz=v * vz,
                m=np.full(n, 1.0 / n))


def _system(g, c, n):
    if c["dims"] == 3:
        st = _plummer(g, n)
    elif c["entry"] == "loop" and n >= 500000:
        st = _two_disks(g, n)
    else:
        st = _disk(g, n, n)
    if c["flung"]:
        # one particle in 50,000 (at least two) thrown out, up to 300 away
        far = g.choice(np.arange(1, n), max(2, n // 50000), replace=False)
        d, p = 300.0 ** g.uniform(0.6, 1.0, len(far)), g.uniform(0.0, 2.0 * math.pi, len(far))
        st["x"][far], st["y"][far] = d * np.cos(p), d * np.sin(p)
        st["vx"][far], st["vy"][far] = 5.0 * np.cos(p), 5.0 * np.sin(p)
    if c["periodic"] and c["dims"] == 2:   # the 2D domain starts at 0
        st["x"], st["y"] = st["x"] + 0.5 * DOMAIN, st["y"] + 0.5 * DOMAIN
    out = {k: np.ascontiguousarray(v, np.float32) for k, v in st.items()}
    out["id"] = np.arange(n, dtype=np.uint32)
    if c["heat"]:
        out["temp"] = g.uniform(100.0, 5000.0, n).astype(np.float32)
    return out


def _inputs(c, seed):
    """The particle systems of a case, one dict of float32 arrays each."""
    g = np.random.Generator(np.random.PCG64([int(seed), c["n"]]))
    if c["entry"] != "batch":
        return [_system(g, c, c["n"])]
    u = np.random.Generator(np.random.PCG64([c["n"], c["sims"]])).random(c["sims"])
    sizes = 1024.0 * (c["n"] / 1024.0) ** u   # the case's own, whatever the seed
    return [_system(g, c, int(k)) for k in sizes]


def _softening(c):
    """(added to r^2 by the walk, added by the direct sum)"""
    if c["dims"] == 3:
        return 0.01, 0.01
    s = 0.01 if c["entry"] == "batch" else 0.005
    return s * s, s


def _params(c):
    eps2, direct_eps2 = _softening(c)
    kw = dict(G=1.0, theta=c["theta"], eps2=eps2, direct_eps2=direct_eps2, dt=DT)
    if c["mode"] == "mixed":   # what the autotuner picks for these systems
        kw.update(precision=ge.PREC_MIXED, leaf_cap=16, group_size=128 if c["dims"] == 3 else 64)
    if c["direct"]:
        kw["direct_below"] = 5000
    if c["periodic"]:
        kw.update(periodic=1, domain=(DOMAIN, DOMAIN, DOMAIN))
    if c["heat"]:
        kw["temp_enabled"] = 1
    return ge.default_params(c["dims"], **kw)


def _locked(shape, dtype):
    """A zeroed page-locked array (the tensor keeps the memory alive)."""
    t = torch.zeros(shape, dtype=dtype, pin_memory=True)
    return t.numpy(), t


ORDER = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az", "m", "id")


def _keys(c):
    return [k for k in ORDER if c["dims"] == 3 or k[-1] != "z"]


def _records(c, st):
    """The application's records of a system: 32-bit views of both arrays."""
    lay, n, d = ge.aos_layout(c["dims"]), len(st["x"]), c["dims"]
    phys, keep1 = _locked((n, lay.stride), torch.uint8)
    rend, keep2 = _locked((n, lay.r_stride), torch.uint8)
    f, u = phys.view(np.float32), phys.view(np.uint32)
    for k, name in enumerate("xyz"[:d]):
        f[:, lay.off_pos // 4 + k] = st[name]
        f[:, lay.off_vel // 4 + k] = st["v" + name]
    f[:, lay.off_mass // 4] = st["m"]
    u[:, lay.off_id // 4] = st["id"]
    part = {k: f[:, o // 4:o // 4 + d] for k, o in
            (("pos", lay.off_pos), ("vel", lay.off_vel), ("acc", lay.off_acc))}
    return phys, rend, part, (keep1, keep2)


def prepare(case, seed):
    c, systems = case, _inputs(case, seed)
    sim = ge.Simulation(_params(c))
    state = dict(case=c, sim=sim, keep=[])
    if c["entry"] == "records":
        state["phys"], state["rend"], state["part"], state["keep"] = _records(c, systems[0])
        return state
    n = sum(len(s["x"]) for s in systems)
    out = {}
    for k in _keys(c) + (["temp"] if c["heat"] else []):
        out[k], t = _locked(n, torch.int32 if k == "id" else torch.float32)
        state["keep"].append(t)
    out["id"] = out["id"].view(np.uint32)
    state["out"] = out
    if c["entry"] == "host":   # the frame works in place on these
        for k, v in systems[0].items():
            out[k][:] = v
    elif c["entry"] == "batch":
        for s in systems:
            sim.add_sim(s)
    else:
        sim.upload(systems[0])
        if c["heat"]:
            sim.upload_temp(systems[0]["temp"])
    return state


def _ptr(a):
    return None if a is None else a.ctypes.data


def run(state):
    c, sim = state["case"], state["sim"]
    if c["entry"] == "records":
        order = sim.frame_aos(state["phys"], state["rend"])
        return dict(state["part"], order=order)
    out = state["out"]
    if c["entry"] == "host":
        sim.frame_host(out)
        return out
    sim.step(c["steps"])
    lib = ge.lib()
    sim._check(lib.ge_download(sim._h, *[_ptr(out.get(k)) for k in ORDER]))
    if c["heat"]:
        sim._check(lib.ge_download_temp(sim._h, _ptr(out["temp"])))
    return out


# --- what a pass cannot do without ------------------------------------------

def work(case):
    """Bytes: each frame reads and writes a particle's position, velocity and
    acceleration once and reads its mass; the call moves the state across
    where it does.  Operations: the accepted sources of a walk, about a
    constant number per tree level that falls with the opening angle (10 / theta^2
    in 2D, 40 / theta^3 in 3D, measured on these systems), 18 or 24 operations
    each; every pair with the direct sum."""
    c, d = case, case["dims"]
    if c["entry"] == "batch":   # mean of log-uniform sizes
        lo, hi = 1024.0, float(c["n"])
        size = (hi - lo) / math.log(hi / lo)
        n = size * c["sims"]
    else:
        size = n = float(c["n"])
    if c["direct"]:
        inter = size
    elif d == 2:
        inter = min(size, 10.0 / c["theta"] ** 2 * math.log(size, 4.0))
    else:
        inter = min(size, 40.0 / c["theta"] ** 3 * math.log(size, 8.0))
    frame = n * (2 * 3 * d + 1) * 4
    io = n * (3 * d + 2) * 4
    if c["entry"] in ("host", "records"):
        io *= 2
    return {"bytes": c["steps"] * frame + io,
            "flops": c["steps"] * n * inter * (18.0 if d == 2 else 24.0)}


# --- the same in 64 bits ------------------------------------------------------

def _forces(pos, m, eps2, periodic):
    """Direct sum over all pairs (what the tree walk approximates)."""
    d, n = pos.shape
    acc = torch.empty_like(pos)
    rows = max(1, (1 << 26) // n)
    for a in range(0, n, rows):
        diff = [pos[k][None, :] - pos[k][a:a + rows, None] for k in range(d)]
        if periodic:
            diff = [t - DOMAIN * ((t > 0.5 * DOMAIN).double() - (t < -0.5 * DOMAIN).double())
                    for t in diff]
        r2 = diff[0] * diff[0] + eps2
        for t in diff[1:]:
            r2 += t * t
        f = r2.pow_(-1.5).mul_(m)
        for k in range(d):
            acc[k, a:a + rows] = (diff[k] * f).sum(1)
    return acc


def _morton_order(pos, order):
    """The order of a frame: stable by the Morton keys, which are taken in 32
    bits from the square (cubic) box of the positions."""
    d = len(pos)
    p = pos.float()[:, order]
    lo, hi = p.min(1).values, p.max(1).values
    size = (hi - lo).max()
    corner = (lo + hi) * 0.5 - size * 0.5
    end = corner + (size.clamp(min=1e-6) if d == 2 else size)
    bits = 18 if d == 2 else 21
    scale, top = (262144.0, 262143) if d == 2 else (2097151.0, 2097151)
    key = torch.zeros(p.shape[1], dtype=torch.int64, device=p.device)
    for k in range(d):
        q = (((p[k].clamp(corner[k], end[k]) - corner[k]) / (end[k] - corner[k])) * scale)
        q = q.to(torch.int64).clamp(max=top)
        for b in range(bits):
            key |= ((q >> b) & 1) << (d * b + k)
    return order[torch.sort(key, stable=True).indices]


def exact(case, seed):
    """The frame with every pair summed, in 64 bits: what the walk's tree
    approximates.  None where that takes too many pairs, and after several
    frames: results come in the last frame's Morton order, in which the tree's
    error swaps neighbours.  No value for ids, orders and temperatures."""
    c = case
    if c["steps"] > 1:
        return None
    systems = _inputs(c, seed)
    if sum(len(s["x"]) ** 2 for s in systems) > EXACT_PAIRS:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    names = "xyz"[:c["dims"]]
    dt = float(np.float32(DT))
    soft = _softening(c)[1 if c["direct"] else 0]
    low = 0.0 if c["dims"] == 2 else -0.5 * DOMAIN
    parts = []
    for s in systems:
        get = lambda k: torch.as_tensor(s[k], device=dev).double()  # noqa: E731
        pos, vel = (torch.stack([get(p + k) for k in names]) for p in ("", "v"))
        m = get("m")
        pos += vel * dt   # a fresh system's accelerations are zero: no first kick
        if c["periodic"]:
            pos += DOMAIN * ((pos < low).double() - (pos >= low + DOMAIN).double())
        order = torch.arange(pos.shape[1], device=dev)
        if c["entry"] != "records":
            order = _morton_order(pos, order)
        acc = _forces(pos, m, float(np.float32(soft)), c["periodic"])
        vel += acc * (0.5 * dt)
        parts.append([t[..., order].cpu().numpy() for t in (pos, vel, acc, m)])
    pos, vel, acc, m = (np.concatenate([p[k] for p in parts], axis=-1) for k in range(4))
    if c["entry"] == "records":
        return dict(pos=pos.T.copy(), vel=vel.T.copy(), acc=acc.T.copy(), order=None)
    out = dict(m=m, id=None)
    for k, a in enumerate(names):
        out[a], out["v" + a], out["a" + a] = pos[k], vel[k], acc[k]
    if c["heat"]:
        out["temp"] = None
    return out
