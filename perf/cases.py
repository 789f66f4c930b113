"""The workloads that this framework is timed on, with a plain FP64 statement of what each returns.

One pass is what a user's program does between two looks at the particles: an input/output step of an external
loop (positions in, one step, positions out through one pinned buffer), or a sample interval of a simulation
(a number of steps, then the positions, the forces and where asked the fluid velocity, as the driver of
`fluam data.main` takes them at a sample), a step of a batch of replicas, or a set of requests through the
server.  `exact` restates the schemes in 64 bits with torch; it uses nothing of this repository.
"""
import math

import numpy as np
import torch

import fluam_b200 as fsl

EDGES = (16, 24, 32, 48, 64)  # of the replicas of a batch
SMOOTH = [n for n in range(16, 161) if not [p for p in (13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61, 67, 71, 73, 79, 83, 89, 97,
                                                       101, 103, 107, 109, 113, 127, 131, 137, 139, 149, 151, 157) if n % p == 0]]


def _step(name, m, n, **more):
    """A single 3-D instance: m cells a side (spacing 1), n particles."""
    c = dict(kind="step", mx=m[0], my=m[1], mz=m[2], n=n, kernel=3, pair="soft", beads=0, scheme="midpoint", precision=0,
             rfd=0, extra=0.0, dt=0.01, steps=1, io=False, field=False)
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: a handful of particles moved one step by an external loop; launches and latency
        _step("io_16", (16,) * 3, 16, io=True),
        # the small single instance of the benchmark set, sampled with its fluid field every 10 steps
        _step("plain_32", (32,) * 3, 256, steps=10, field=True),
        # the reference's default pair force (the Lennard-Jones table) on a medium suspension
        _step("lj_64", (64,) * 3, 8000, pair="lj", steps=10),
        # the headline workload: bead-spring chains in 128^3, positions in and out every step
        _step("chains_128", (128,) * 3, 65536, kernel=4, beads=16, dt=0.005, io=True),
        # the precision-study size: a million particles in 256^3
        _step("large_256", (256,) * 3, 1000000, dt=0.002, io=True),
        # a box of unequal, non-power-of-two edges
        _step("ragged_60_72_100", (60, 72, 100), 6000, kernel=4, steps=10),
        # the first-order integrator with extra mobility, bonded chains and the fluid field at the samples
        _step("first_48", (48,) * 3, 2048, kernel=4, beads=16, pair="none", scheme="first", extra=0.3, steps=20, field=True),
        # the reference's own arithmetic: everything in FP64
        _step("fp64_64", (64,) * 3, 4096, kernel=4, precision=2, steps=5, field=True),
        # a colloidal monolayer: quasi-2D Gaussian blobs, FP64 as the reference
        dict(name="quasi2d_256", kind="q2d", mx=256, my=256, n=4096, scheme="quasi2D", pc=0, steps=10),
        # the incompressible fluctuating fluid alone, FP64 as the reference
        dict(name="fluid_64", kind="inc", mx=64, my=64, mz=64, steps=5),
        # replicas of mixed sizes stepped together, positions in and out every step
        dict(name="batch_256", kind="batch", n=256, mix=7, np_max=2048),
        # requests of mixed sizes and lengths through the server
        dict(name="served_12", kind="served", n=12, mix=3, np_max=4096, steps_max=60),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(rng, hi):
    n = _log(rng, 16, hi)
    return min(SMOOTH, key=lambda s: abs(s - n))


def draw(rng):
    k = rng.random()
    if k < 0.6:
        f64 = rng.random() < 0.15
        hi = 72 if f64 else 160
        e = _smooth(rng, hi)
        m = (e, e, e) if rng.random() < 0.6 else (e, _smooth(rng, hi), _smooth(rng, hi))
        nc = m[0] * m[1] * m[2]
        n = _log(rng, 16, min(65536, max(32, nc // 24)))
        pair = rng.choice(["soft", "soft", "lj", "none"])
        beads = rng.choice([0, 0, 16, 10]) if pair != "lj" else 0
        n = max(1, n // beads) * beads if beads else n
        io = rng.random() < 0.5
        return _step("", m, n, kernel=rng.choice([3, 4]), pair=pair, beads=beads, scheme=rng.choice(["midpoint"] * 3 + ["first"]),
                     precision=2 if f64 else rng.choice([0, 0, 0, 1]), rfd=rng.choice([0, 0, 1]), extra=rng.choice([0.0, 0.0, 0.3]),
                     dt=rng.choice([0.005, 0.01]), steps=1 if io else 5, io=io, field=not io and nc <= 2 ** 17)
    if k < 0.72:
        return dict(kind="q2d", mx=_smooth(rng, 160) * rng.choice([1, 2]), my=_smooth(rng, 160) * rng.choice([1, 2]), n=_log(rng, 64, 6000),
                    scheme=rng.choice(["quasi2D", "stokes2D"]), pc=rng.choice([0, 1]), steps=5)
    if k < 0.82:
        return dict(kind="inc", mx=_smooth(rng, 72), my=_smooth(rng, 72), mz=_smooth(rng, 72), steps=3)
    if k < 0.94:
        return dict(kind="batch", n=_log(rng, 16, 256), mix=rng.randrange(1000), np_max=_log(rng, 64, 2048))
    return dict(kind="served", n=_log(rng, 2, 12), mix=rng.randrange(1000), np_max=_log(rng, 64, 4096), steps_max=40)


# ---------------------------------------------------------------- inputs ---
def _sizes(case):
    """Of every replica of a batch or request of a server: edge, particles, viscosity, kernel, steps."""
    r = np.random.default_rng(case["mix"])
    served = case["kind"] == "served"
    out = []
    for _ in range(case["n"]):
        m = int(r.choice([16, 24, 32, 40, 48, 56, 64] if served else EDGES))
        n = int(round(math.exp(r.uniform(math.log(16 if served else 8), math.log(case["np_max"])))))
        eta = float(r.uniform(0.5, 2.0))
        kernel = int(r.choice((3, 4))) if served else 3
        steps = int(round(math.exp(r.uniform(math.log(10), math.log(case["steps_max"]))))) if served else 1
        out.append((m, n, eta, kernel, steps))
    return out


def _positions(m, n, pair, beads, seed):
    """Seeded positions (3, n) in a box of edges m and bonds (i, j, k, r0) or None."""
    r = np.random.default_rng(seed)
    L = np.asarray(m, dtype=float)[:, None]
    if pair == "lj":  # no overlaps: a jittered lattice (the pair force has a core of two cells)
        per = [max(1, int(e // 3)) for e in m]
        sites = r.permutation(per[0] * per[1] * per[2])[:n]
        s = np.stack([sites % per[0], sites // per[0] % per[1], sites // (per[0] * per[1])])
        q = (s + 0.5) * (L / np.asarray(per, dtype=float)[:, None]) - 0.5 * L
        return q + r.uniform(-0.2, 0.2, q.shape), None
    if not beads:
        return r.uniform(-0.5, 0.5, (3, n)) * L, None
    nch = n // beads
    start = r.uniform(-0.5, 0.5, (nch, 3)) * L[:, 0]
    d = r.standard_normal((nch, beads - 1, 3))
    d /= np.linalg.norm(d, axis=2, keepdims=True)
    q = np.concatenate([start[:, None], start[:, None] + np.cumsum(d, axis=1)], axis=1).reshape(-1, 3).T.copy()
    idx = np.arange(n).reshape(nch, beads)
    bi, bj = idx[:, :-1].ravel().astype(np.int32), idx[:, 1:].ravel().astype(np.int32)
    return q, (bi, bj, np.full(len(bi), 10.0), np.ones(len(bi)))


def _limit_lj(case):
    """The particles that the lattice of an LJ case has room for."""
    if case["pair"] != "lj":
        return case["n"]
    return min(case["n"], max(1, case["mx"] // 3) * max(1, case["my"] // 3) * max(1, case["mz"] // 3))


_PAIRS = {"none": 0, "lj": 1, "soft": 2}


def _setup(case, seed):
    """The plain description of a single 3-D instance: what both prepare and exact start from."""
    m = (case["mx"], case["my"], case["mz"])
    q, bonds = _positions(m, _limit_lj(case), case["pair"], case["beads"], seed)
    return dict(m=m, L=tuple(float(e) for e in m), q=q, bonds=bonds, eta=1.0, kT=0.01, dt=case["dt"],
                cutoff=5.0 if case["pair"] == "lj" else 1.5, kernel=case["kernel"], pair=case["pair"], rfd=case["rfd"],
                extra=case["extra"], first=case["scheme"] == "first", seed=1000003 * (seed + 1))


def _config(p, precision=0):
    pairs = {"none": fsl.PAIR_NONE, "lj": fsl.PAIR_TABLE_LJ, "soft": fsl.PAIR_SOFT}
    return fsl.make_config(p["m"], p["L"], eta=p["eta"], kT=p["kT"], dt=p["dt"], cutoff=p["cutoff"], kernel=p["kernel"],
                           pair=pairs[p["pair"]], soft_epsilon=1.0, rfd=fsl.RFD_PAPER if p["rfd"] else fsl.RFD_REFERENCE,
                           extra_mobility=p["extra"], seed=p["seed"], precision=precision,
                           scheme=fsl.SCHEME_FIRST_ORDER if p["first"] else fsl.SCHEME_MIDPOINT)


def _replicas(case, seed):
    out = []
    for i, (m, n, eta, kernel, steps) in enumerate(_sizes(case)):
        q, _ = _positions((m,) * 3, n, "soft", 0, 7919 * (seed + 1) + i)
        out.append((dict(m=(m,) * 3, L=(float(m),) * 3, q=q, bonds=None, eta=eta, kT=0.01, dt=0.01, cutoff=1.5, kernel=kernel,
                         pair="soft", rfd=0, extra=0.0, first=False, seed=100003 * (seed + 1) + i), steps))
    return out


def _setup_q2d(case, seed):
    r = np.random.default_rng(seed)
    L = (float(case["mx"]), float(case["my"]), 4.0)
    n = case["n"]
    q = r.uniform(-0.5, 0.5, (3, n)) * np.asarray(L)[:, None]
    q[2] = 0.0
    return dict(m=(case["mx"], case["my"], 1), L=L, q=q, eta=1.0, kT=0.01, dt=0.01, cutoff=1.5, radius=1.0, rpy=case["scheme"] == "quasi2D",
                pc=case["pc"], seed=1000003 * (seed + 1))


def _setup_inc(case, seed):
    r = np.random.default_rng(seed)
    m = (case["mx"], case["my"], case["mz"])
    return dict(m=m, L=tuple(float(e) for e in m), v=0.1 * r.standard_normal((3, m[2], m[1], m[0])), eta=1.0, kT=0.01, dt=0.05, rho=1.0,
                seed=1000003 * (seed + 1))


def _pinned(q):
    """One page-locked buffer that a step reads its positions from and writes them to."""
    buf = torch.empty(q.shape, dtype=torch.float64, pin_memory=True)
    buf.copy_(torch.from_numpy(np.ascontiguousarray(q)))
    return buf


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        p = _setup(case, seed)
        sim = fsl.StokesLimit(_config(p, case["precision"]), p["q"])
        if p["bonds"]:
            sim.load_bonds(*p["bonds"])
        return dict(case=case, sim=sim, buf=_pinned(p["q"]) if case["io"] else None)
    if kind == "q2d":
        p = _setup_q2d(case, seed)
        cfg = fsl.make_config(p["m"], p["L"], eta=p["eta"], kT=p["kT"], dt=p["dt"], cutoff=p["cutoff"], pair=fsl.PAIR_SOFT, seed=p["seed"],
                              scheme=fsl.SCHEME_QUASI2D if p["rpy"] else fsl.SCHEME_STOKES2D, radius=p["radius"],
                              predictor_corrector=p["pc"])
        return dict(case=case, sim=fsl.StokesLimit(cfg, p["q"]))
    if kind == "inc":
        p = _setup_inc(case, seed)
        cfg = fsl.make_config(p["m"], p["L"], eta=p["eta"], kT=p["kT"], dt=p["dt"], seed=p["seed"], density=p["rho"],
                              scheme=fsl.SCHEME_INCOMPRESSIBLE)
        sim = fsl.StokesLimit(cfg, np.zeros((3, 0)))
        sim.set_velocity64(p["v"])
        return dict(case=case, sim=sim)
    reps = _replicas(case, seed)
    if kind == "batch":
        b = fsl.Batch([_config(p) for p, _ in reps], [p["q"] for p, _ in reps])
        return dict(case=case, batch=b, buf=_pinned(np.concatenate([p["q"].ravel() for p, _ in reps])))
    return dict(case=case, server=fsl.Server(), requests=[(_config(p), p["q"], steps) for p, steps in reps])


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        a = state["buf"].data_ptr()
        state["batch"].step_io(a, a)
        return state["buf"]
    if case["kind"] == "served":
        srv = state["server"]
        ids = [srv.submit(c, q, n) for c, q, n in state["requests"]]
        for i in ids:
            srv.wait(i)
        got = [srv.result(i) for i in ids]
        return dict(q=np.concatenate([q.ravel() for q, _ in got]), F=np.concatenate([f.ravel() for _, f in got]))
    sim = state["sim"]
    if case["kind"] == "step" and case["io"]:
        a = state["buf"].data_ptr()
        sim.step_io(a, a)
        return state["buf"]
    sim.step(case["steps"])
    if case["kind"] == "inc":
        return sim.velocity64()
    out = dict(q=sim.positions(), F=sim.forces())
    if case["kind"] == "step" and case["field"]:
        out["v"] = sim.velocity64()
    return out


# ------------------------------------------------- what a pass needs ---
def _step_work(nc, n, first, wide):
    """Bytes and flops of one 3-D step: per solve three real fields through a transform, its solve and its inverse
    (72 bytes a cell in 32 bits), the particles' positions, forces and increments; transforms, normals and stencils."""
    solves = 1 if first else 2
    return (72 * wide * solves * nc + 384 * n,
            solves * nc * (6 * 2.5 * math.log2(max(nc, 2)) + 60) + 6 * solves * nc * 40 + 64 * 3 * 4 * 2 * n)


def work(case):
    kind = case["kind"]
    if kind == "step":
        b, f = _step_work(case["mx"] * case["my"] * case["mz"], _limit_lj(case), case["scheme"] == "first", 2 if case["precision"] == 2 else 1)
        return {"bytes": b * case["steps"], "flops": f * case["steps"]}
    if kind == "q2d":
        nc = case["mx"] * case["my"]
        return {"bytes": case["steps"] * (160 * nc + 96 * case["n"]), "flops": case["steps"] * (nc * (20 * math.log2(nc) + 200) + 81 * 40 * 2 * case["n"])}
    if kind == "inc":
        nc = case["mx"] * case["my"] * case["mz"]
        return {"bytes": case["steps"] * 336 * nc, "flops": case["steps"] * nc * (2 * (15 * math.log2(nc) + 300) + 400)}
    got = [(_step_work(m ** 3, n, False, 1), steps) for m, n, _, _, steps in _sizes(case)]
    return {"bytes": sum(b * s for (b, _), s in got), "flops": sum(f * s for (_, f), s in got)}


def tolerance(case):
    """About four times what `run` differs by from `exact` over the declared ranges.  The FP64 forms differ by rounding
    (1e-15 seen).  Of the 32-bit forms the fluid field shows the fields' own precision (6e-7); forces follow from
    positions that differ by it (up to 2e-7), and through the table of the Lennard-Jones force, whose filter has 8-bit
    weights, some of them by a step of the table (6e-7); positions alone differ in the rounding of an increment of a
    thousandth of a cell (3e-10 of a box of 16, 5e-11 of one of 256)."""
    if case["kind"] in ("inc", "q2d") or case["kind"] == "step" and case["precision"] == 2:
        return {"rel": 1e-13, "max": 1e-11}
    if case["kind"] == "batch":
        return {"rel": 5e-8 / 48, "max": 5e-6 / 48}
    if case["kind"] == "served":
        return {"rel": 1e-6}
    if case["io"]:
        e = min(case["mx"], case["my"], case["mz"])
        return {"rel": 5e-8 / e, "max": 5e-6 / e}
    if case["field"] or case["pair"] == "lj":
        return {"rel": 2.5e-6, "max": 1e-3 if case["pair"] == "lj" else 1e-4}
    return {"rel": 1e-6}


# ------------------------------------------------------- the 64-bit side ---
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())


def _normals(seed, t, count):
    """Normals 0 .. count-1 of draw t: Philox4x32-10 keyed by the seed on the counter (index / 4, t), Box-Muller."""
    mask = 0xFFFFFFFF
    b = torch.arange((count + 3) // 4, dtype=torch.int64, device=_dev())
    c = [b & mask, b >> 32, torch.full_like(b, t & mask), torch.full_like(b, t >> 32)]
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [(p1 >> 32) & mask ^ c[1] ^ k0, p1 & mask, (p0 >> 32) & mask ^ c[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    u = [(2 * (w >> 9) + 1).to(torch.float64) * 2.0 ** -24 for w in c]
    ra, rb = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    out = [ra * torch.cos(2 * math.pi * u[1]), ra * torch.sin(2 * math.pi * u[1]), rb * torch.cos(2 * math.pi * u[3]), rb * torch.sin(2 * math.pi * u[3])]
    return torch.stack(out, dim=1).reshape(-1)[:count]


def _wrap(r, L):
    """r minus the periods that bring it into the box, as the schemes take them: r - int(r/L + sign(r)/2) L."""
    return r - torch.trunc(r * (1.0 / L) + 0.5 * torch.sign(r)) * L


def _index(r, m, L):
    return torch.trunc(r * (m / L) + 0.5 * m).to(torch.int64) % m


def _sqrtf(x):
    return x.clamp(min=0).float().double().sqrt().float().double()


def _delta(kernel, x):
    """Peskin's 3-point kernel (its square root in single precision, as the reference's) or 4-point kernel."""
    x = x.abs()
    zero = torch.zeros_like(x)
    if kernel == 3:
        near = (1 + _sqrtf(1 - 3 * x * x)) / 3
        far = (5 - 3 * x - _sqrtf(1 - 3 * (1 - x) * (1 - x))) / 6
        return torch.where(x < 0.5, near, torch.where(x > 1.5, zero, far))
    near = (3 - 2 * x + (1 + 4 * x - 4 * x * x).clamp(min=0).sqrt()) / 8
    far = (5 - 2 * x - (-7 + 12 * x - 4 * x * x).clamp(min=0).sqrt()) / 8
    return torch.where(x <= 1, near, torch.where(x >= 2, zero, far))


def _stencil(p, posc, posw):
    """Nodes and weights [component][dimension] -> (K, n): nodes from posc, weights from posw."""
    K, made, out = p["kernel"], {}, []
    k = torch.arange(K, device=posc.device)[:, None] - 1
    for comp in range(3):
        row = []
        for d in range(3):
            if (d, d == comp) not in made:
                m, L = p["m"][d], p["L"][d]
                h = L / m
                off = 0.5 * h if d == comp else 0.0
                at = posc[d] - off if K == 3 else (posc[d] - off) - 0.5 * h
                j = (_index(_wrap(at, L), m, L)[None] + k) % m
                node = (j.double() + 0.5) * h - 0.5 * L
                made[d, d == comp] = j, _delta(K, _wrap(posw[d][None] - node - off, L) * (m / L))
            row.append(made[d, d == comp])
        out.append(row)
    return out


def _nodes(p, row):
    """Flat node indices and weights of one component, one (y, z) offset pair at a time."""
    (jx, wx), (jy, wy), (jz, wz) = row
    for b in range(p["kernel"]):
        for c in range(p["kernel"]):
            yield jx + p["m"][0] * (jy[b] + p["m"][1] * jz[c])[None], wx * (wy[b] * wz[c])[None]


def _spread(p, f, st, val):
    for comp in range(3):
        for at, w in _nodes(p, st[comp]):
            f[comp].index_add_(0, at.reshape(-1), (w * val[comp][None]).reshape(-1))


def _interp(p, v, st):
    out = []
    for comp in range(3):
        u = 0
        for at, w in _nodes(p, st[comp]):
            u = u + (w * v[comp][at]).sum(0)
        out.append(u)
    return torch.stack(out)


def _lj_table(p):
    """The float table of the pair force over r^2 / rc^2: sigma of two cells, epsilon of kT, float accumulation."""
    f32 = np.float32
    sigma, eps, c2 = f32(2 * p["L"][0] / p["m"][0]), f32(p["kT"]), f32(p["cutoff"] ** 2)
    dr = f32(c2 / f32(4096))
    r, t = f32(f32(0.5) * dr), np.zeros(4096, f32)
    for i in range(4096):
        rr = float(np.sqrt(r))
        fr = f32(48.0 * float(eps) * ((float(sigma) / rr) ** 12 - 0.5 * (float(sigma) / rr) ** 6) / rr)
        t[i] = fr / np.sqrt(r)
        r = f32(r + dr)
    t[0] = t[-1] = 0
    return torch.as_tensor(t, device=_dev())


def _pair_factor(p, r2, tab):
    if p["pair"] == "soft":
        rc = p["cutoff"]
        return torch.where((r2 < rc * rc) & (r2 > 0), 2 / rc * (1 / r2.clamp(min=1e-300).sqrt() - 1 / rc), torch.zeros_like(r2))
    xb = (r2 * (1 / p["cutoff"] ** 2)).float().double() * 4096 - 0.5
    fl = torch.floor(xb)
    a = (torch.round((xb - fl) * 256) / 256).float()
    i = fl.clamp(-1, 4096).long()
    return ((1 - a) * tab[i.clamp(0, 4095)] + a * tab[(i + 1).clamp(0, 4095)]).double()


def _forces(p, q, tab, dims=3):
    """Pair forces within the cutoff through a cell list, and bonds."""
    n = q.shape[1]
    F = torch.zeros_like(q)
    if p["pair"] != "none" and n:
        L, rc = p["L"], p["cutoff"]
        m = [max(3, int(L[d] / rc)) if d < dims else 1 for d in range(3)]
        w = [_wrap(q[d], L[d]) for d in range(3)]
        c = [_index(w[d], m[d], L[d]) if d < dims else torch.zeros(n, dtype=torch.int64, device=q.device) for d in range(3)]
        cell = c[0] + m[0] * (c[1] + m[1] * c[2])
        order = torch.argsort(cell)
        count = torch.bincount(cell, minlength=m[0] * m[1] * m[2])
        start = torch.cumsum(count, 0) - count
        most = int(count.max())
        for o in range(3 ** dims):
            s = [o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1 if dims == 3 else 0]
            other = (c[0] + s[0]) % m[0] + m[0] * ((c[1] + s[1]) % m[1] + m[1] * ((c[2] + s[2]) % m[2]))
            first, have = start[other], count[other]
            for k in range(most):
                on = torch.nonzero(have > k).reshape(-1)
                j = order[first[on] + k]
                on, j = on[on != j], j[on != j]
                d = torch.stack([_wrap(q[e][on] - q[e][j], L[e]) for e in range(dims)])
                r2 = d[0] * d[0] + d[1] * d[1]
                r2 = r2 + d[2] * d[2] if dims == 3 else r2
                F[:dims].index_add_(1, on, _pair_factor(p, r2, tab) * d)
    if p.get("bonds"):
        bi, bj, bk, br = (torch.as_tensor(x, device=q.device) for x in p["bonds"])
        bi, bj = bi.long(), bj.long()
        d = q[:, bi] - q[:, bj]
        r = d.square().sum(0).sqrt()
        f = -(bk * (1 - br / r)) * d
        F.index_add_(1, bi, f)
        F.index_add_(1, bj, -f)
    return F


def _divergence(p, s, f1, f4):
    """div of a stress sample (6, mz, my, mx): diagonals at the centres, the others on edges."""
    def g(a, axis, shift):  # a[+1] - a (shift -1) or a - a[-1] (shift +1) along x, y, z
        moved = torch.roll(s[a], shift, 2 - axis)
        return (moved - s[a] if shift < 0 else s[a] - moved) * (p["m"][axis] / p["L"][axis])
    return torch.stack([f1 * g(0, 0, -1) + f4 * (g(1, 1, 1) + g(2, 2, 1)), f1 * g(3, 1, -1) + f4 * (g(1, 0, 1) + g(4, 2, 1)),
                        f1 * g(5, 2, -1) + f4 * (g(2, 0, 1) + g(4, 1, 1))])


def _modes(p):
    """Per component: the gradient 2/h sin(pi j/m) and the half-cell shift exp(i pi j/m), shaped to broadcast."""
    g, e = [], []
    for d in range(3):
        m = p["m"][d]
        a = math.pi * torch.arange(m, dtype=torch.float64, device=_dev()) / m
        shape = [1, 1, 1]
        shape[2 - d] = m
        g.append((2 * m / p["L"][d] * torch.sin(a)).reshape(shape))
        e.append(torch.polar(torch.ones_like(a), a).reshape(shape))
    return g, e


def _project(p, W, den):
    """Inverse transform of (W - g (g.W) / |g|^2) / den(|g|^2) with the staggered shifts; the zero mode is kept as W / den."""
    g, e = _modes(p)
    W = torch.fft.fftn(W.to(torch.complex128), dim=(1, 2, 3))
    for d in range(3):
        W[d] *= e[d].conj()
    G2 = g[0] ** 2 + g[1] ** 2 + g[2] ** 2
    G2[0, 0, 0] = 1.0
    s = (g[0] * W[0] + g[1] * W[1] + g[2] * W[2]) / G2
    G2[0, 0, 0] = 0.0
    f = den(G2)
    for d in range(3):
        W[d] = (W[d] - g[d] * s) * f * e[d]
    return torch.fft.ifftn(W, dim=(1, 2, 3)).real


def _stokes(p, W):
    def den(G2):
        G2 = G2.clone()
        G2[0, 0, 0] = math.inf
        return 1 / (p["eta"] * G2)
    return _project(p, W, den)


def _simulate(p, steps):
    """The Stokes-limit step in 64 bits: positions, the forces the last step used and its last velocity field."""
    m, n = p["m"], p["q"].shape[1]
    nc = m[0] * m[1] * m[2]
    dV = p["L"][0] * p["L"][1] * p["L"][2] / nc
    f1, f4 = (math.sqrt(c * p["kT"] * p["eta"] / (dV * p["dt"])) for c in (4.0, 2.0))
    f2 = math.sqrt(p["kT"] * p["extra"] * p["dt"])
    shape = (m[2], m[1], m[0])
    q, tab = _t(p["q"]), _lj_table(p) if p["pair"] == "lj" else None
    F = v = None

    def drift(f, W):
        delta = 0.001
        for s in (1, -1):
            at = q + s * 0.5 * delta * W
            _spread(p, f, _stencil(p, at, at if p["rfd"] else q), s * p["kT"] / delta * W)

    for t in range(steps):
        z = _normals(p["seed"], t, 12 * nc + 9 * n)
        D1 = _divergence(p, z[: 6 * nc].reshape(6, *shape), f1, f4)
        W, xi1, xi2 = z[6 * nc:6 * nc + 9 * n].reshape(3, 3, n)
        F = _forces(p, q, tab)
        st = _stencil(p, q, q)
        f = torch.zeros(3, nc, dtype=torch.float64, device=q.device)
        _spread(p, f, st, F)
        if p["first"]:
            drift(f, W)
        v = _stokes(p, f.reshape(3, *shape) / dV + (1.0 if p["first"] else math.sqrt(2.0)) * D1)
        half = q + 0.5 * p["dt"] * _interp(p, v.reshape(3, -1), st)
        if p["extra"]:
            half = half + 0.5 * p["dt"] * p["extra"] * F + f2 * xi1
        if not p["first"] or p["extra"]:
            F = _forces(p, half, tab)
        st = _stencil(p, half, half)
        if not p["first"]:
            f.zero_()
            _spread(p, f, st, F)
            drift(f, W)
            D1 = D1 + _divergence(p, z[6 * nc + 9 * n:].reshape(6, *shape), f1, f4)
            v = _stokes(p, f.reshape(3, *shape) / dV + math.sqrt(0.5) * D1)
        q = q + p["dt"] * _interp(p, v.reshape(3, -1), st)
        if p["extra"]:
            q = q + p["dt"] * p["extra"] * F + f2 * (xi1 + xi2)
    return q, F, v


def _simulate_q2d(p, steps):
    """The quasi-2D (RPY) or 2-D Stokes scheme of Gaussian blobs: positions and the last step's forces."""
    (mx, my, _), (lx, ly, _) = p["m"], p["L"]
    nc, modes = mx * my, mx * my + mx + my
    a = p["radius"]
    var = (a / math.sqrt(math.pi)) ** 2 if p["rpy"] else (a * 0.66556976637237890625) ** 2
    kw = min(int(3 * a * mx / lx) + 1, mx // 2)
    q = _t(p["q"])
    n, dev = q.shape[1], q.device
    p = dict(p, pair="soft", bonds=None)
    i = torch.arange(nc, device=dev)
    ix, iy = i % mx, i // mx
    # signed wave numbers, the Nyquist rows and columns folded onto one sign
    sx, sy = torch.where(ix > mx // 2, ix - mx, ix), torch.where(iy > my // 2, iy - my, iy)
    xh, yh = (sx == mx // 2) & (mx % 2 == 0), (sy == my // 2) & (my % 2 == 0)
    gx = torch.where(xh & (sy < 0), -sx, sx)
    gy = torch.where(~(xh & (sy < 0)) & yh & (sx < 0), -sy, sy)
    kx, ky = gx.double() * (2 * math.pi / lx), gy.double() * (2 * math.pi / ly)
    k2 = kx * kx + ky * ky
    k2[0] = 1.0
    k = k2.sqrt()
    # the canonical mode that holds the noise of a conjugate pair
    cx, cy = torch.where(ix > mx // 2, mx - ix, ix), torch.where(iy > my // 2, my - iy, iy)
    xH, yH = (cx == mx // 2) & (mx % 2 == 0), (cy == my // 2) & (my % 2 == 0)
    fx = torch.where(xH & (sy < 0), -sx, sx)
    fy = torch.where(~(xH & (sy < 0)) & yH & (sx < 0), -sy, sy)
    far = fx * fy < 0
    at = cy * mx + cx + torch.where(far, modes // 2, 0)
    nx, ny = cx.double() * (2 * math.pi / lx) * torch.where(far, -1.0, 1.0), cy.double() * (2 * math.pi / ly)
    edge = (xH & (cy == 0)) | (yH & (cx == 0)) | (xH & yH)
    flip = torch.where((fx < 0) | ((fx == 0) & (fy < 0)), -1.0, 1.0)
    pref = math.sqrt(p["kT"] / (p["eta"] * p["dt"] * lx * ly)) * nc
    if p["rpy"]:
        def fg(k):
            s = math.sqrt(var) * k
            E = torch.special.erfcx(s)
            return 0.5 * (E * (0.5 + s * s) - s / math.sqrt(math.pi)), 0.5 * E
        f, g = fg(k)
        nk = (nx * nx + ny * ny).sqrt()
        nk[0] = 1.0
        hf, hg = (c.clamp(min=0).sqrt() for c in fg(nk))
        amp = pref / (nk ** 3).sqrt()
        coef = [amp * hg * ny, amp * hf * nx, -amp * hg * nx, amp * hf * ny]
        dead = i == 0
    else:
        amp = pref / torch.where(i == 0, torch.ones_like(k2), nx * nx + ny * ny)
        coef = [amp * ny, 0 * amp, -amp * nx, 0 * amp]
        dead = ((cx == mx // 2) & (mx % 2 == 0)) | ((cy == my // 2) & (my % 2 == 0)) | (i == 0)
    coef = [torch.where(dead, torch.zeros_like(c), c) for c in coef]
    o = torch.arange(-kw, kw + 1, device=dev)
    F = None

    def blob(pos):
        jx = (_index(_wrap(pos[0], lx), mx, lx)[None] + o[:, None]) % mx
        jy = (_index(_wrap(pos[1], ly), my, ly)[None] + o[:, None]) % my
        dx = _wrap(pos[0][None] - jx.double() * lx / mx + 0.5 * lx, lx)
        dy = _wrap(pos[1][None] - jy.double() * ly / my + 0.5 * ly, ly)
        at = jx[:, None] + mx * jy[None]
        w = torch.exp(-(dx * dx)[:, None] / (2 * var) - (dy * dy)[None] / (2 * var)) / (2 * math.pi * var)
        return at, w, dx[:, None], dy[None]

    def move(pos, v, h):
        at, w, _, _ = blob(pos)
        u = torch.stack([(w * c[at]).sum((0, 1)) for c in v])
        return (lx * ly / nc) * h * u

    for t in range(steps):
        R = _normals(p["seed"], t, 4 * modes).reshape(4, modes)[:, at]
        F = _forces(p, q, None, dims=2)
        F[2] = 0.0
        at2, w, dx, dy = blob(q)
        s = torch.zeros(2, nc, dtype=torch.float64, device=dev)
        for c, d in ((0, dx), (1, dy)):
            s[c].index_add_(0, at2.reshape(-1), (w * F[c] - w * (p["kT"] / var) * d).reshape(-1))
        z = torch.fft.fftn(s.reshape(2, my, mx).to(torch.complex128), dim=(1, 2)).reshape(2, nc)
        if p["rpy"]:
            c, l = ky * z[0] - kx * z[1], kx * z[0] + ky * z[1]
            ux, uy = (g * ky * c + f * kx * l) / (p["eta"] * k ** 3), (-g * kx * c + f * ky * l) / (p["eta"] * k ** 3)
        else:
            l = (kx * z[0] + ky * z[1]) / k2
            ux, uy = (z[0] - kx * l) / (p["eta"] * k2), (z[1] - ky * l) / (p["eta"] * k2)
        ux[0] = uy[0] = 0
        out = []
        for u, (ca, cb) in ((ux, coef[:2]), (uy, coef[2:])):
            re, im = ca * R[0] + cb * R[1], ca * R[2] + cb * R[3]
            out.append(u + torch.complex(torch.where(edge, math.sqrt(2.0) * re, re), torch.where(edge, torch.zeros_like(im), im) * flip))
        v = torch.fft.ifftn(torch.stack(out).reshape(2, my, mx), dim=(1, 2)).real.reshape(2, nc)
        new = q.clone()
        at_pos = q
        if p["pc"]:
            at_pos = q.clone()
            at_pos[:2] += move(q, v, 0.5 * p["dt"])
        new[:2] += move(at_pos, v, p["dt"])
        q = new
    return q, F


def _simulate_inc(p, steps):
    """The incompressible fluctuating fluid: the velocity field after the steps."""
    m, shape = p["m"], (p["m"][2], p["m"][1], p["m"][0])
    nc = m[0] * m[1] * m[2]
    inv = [m[d] / p["L"][d] for d in range(3)]
    dV, dt, rho, eta = p["L"][0] * p["L"][1] * p["L"][2] / nc, p["dt"], p["rho"], p["eta"]
    f1, f4 = (math.sqrt(c * p["kT"] * eta * dt / (dV * rho * rho)) for c in (4.0, 2.0))
    u = _project(p, _t(p["v"]), lambda G2: torch.ones_like(G2))

    def up(a, d):  # the value one cell further along d
        return torch.roll(a, -1, 2 - d)

    def dn(a, d):
        return torch.roll(a, 1, 2 - d)

    def flux(a):
        """4 x the divergence of the momentum flux a a on the staggered grid."""
        out = []
        for c in range(3):
            r = 0
            for d in range(3):
                s = up(a[c], d) + a[c]
                if d == c:
                    r = r + inv[d] * (s * s - dn(s * s, d))
                else:
                    r = r + inv[d] * (s * (up(a[d], c) + a[d]) - dn(s * (up(a[d], c) + a[d]), d))
            out.append(r)
        return torch.stack(out)

    for t in range(steps):
        s = _normals(p["seed"], t, 6 * nc).reshape(6, *shape).clone()
        tr = (s[0] + s[3] + s[5]) / 3
        for k in (0, 3, 5):
            s[k] -= tr
        D = _divergence(p, s, f1, f4)
        lap = torch.stack([sum(inv[d] ** 2 * (up(u[c], d) - 2 * u[c] + dn(u[c], d)) for d in range(3)) for c in range(3)])
        base = u + 0.5 * dt * eta / rho * lap + D

        def den(G2):
            return 1 / (1 + 0.5 * dt * eta * G2 / rho)
        first = _project(p, base - 0.25 * dt * flux(u), den)
        u = _project(p, base - 0.25 * dt * flux(0.5 * (first + u)), den)
    return u


def exact(case, seed):
    kind = case["kind"]
    host = lambda x: x.cpu().numpy()  # noqa: E731
    if kind == "inc":
        return host(_simulate_inc(_setup_inc(case, seed), case["steps"]))
    if kind == "q2d":
        q, F = _simulate_q2d(_setup_q2d(case, seed), case["steps"])
        return dict(q=host(q), F=host(F))
    if kind == "step":
        q, F, v = _simulate(_setup(case, seed), case["steps"])
        if case["io"]:
            return host(q)
        out = dict(q=host(q), F=host(F))
        if case["field"]:
            out["v"] = host(v)
        return out
    got = [_simulate(p, steps) for p, steps in _replicas(case, seed)]
    q = np.concatenate([host(q).ravel() for q, _, _ in got])
    return q if kind == "batch" else dict(q=q, F=np.concatenate([host(F).ravel() for _, F, _ in got]))
