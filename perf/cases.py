"""The work that users of the soup have it do, as cases that can be timed and checked.

Every case goes through the package's public entry points.  Its `kind` says which:

  steps    SoupSystem.step(n), then the state read back in one checkpoint payload (soup/cli's campaign loop)
  batch    SoupBatch.step(n) over uneven replicas, then every replica's particles, velocities and charges
  forces   SoupSystem.forces(): list rebuild, force pass, readback
  sweep    SoupSystem.protonation_sweep(): one constant-pH sweep, then the charges
  window   adjoint.SoupWindow forward + backward of the thickness proxy (the force-field gradient)
  sample   the campaign's progress sample: amphiphiles, aggregates, their shapes and their closures

A pass of a larger system is five steps: over more of them two FP32 trajectories that round differently part by
more than their velocities' rounding (an ulp of a position in a 76 sigma box is 7.6e-6 sigma).

Starts are seeded and made here, without stepping the library: a small periodic cell of beads (free ones,
or five-bead amphiphiles in water) is pushed apart to liquid-like contacts in torch FP64, tiled over the
box, and given random kinds, Maxwell velocities and random charges on the heads.
"""
import functools
import importlib
import math

import numpy as np
import torch

pg = importlib.import_module("protocell-genesis_b200")
config = importlib.import_module("protocell-genesis_b200.config")
adjoint = importlib.import_module("protocell-genesis_b200.adjoint")
observables = importlib.import_module("protocell-genesis_b200.observables")

NONE = 0xFFFFFFFF
# the reference's largest campaign (76 sigma box, 483,268 beads) by kind
CAMPAIGN = {"C": 55988, "O": 18659, "H": 55988, "M": 1452, "W": 351181}
PLAIN = {"C": 600, "O": 100, "H": 500, "M": 20, "W": 0}          # the reference's small test box
KIND = {"C": 0, "O": 1, "H": 2, "M": 3, "W": 4}


def _case(name, kind, mix, n, density, steps=0, **kw):
    c = {"kind": kind, "mix": mix, "n": n, "density": density, "steps": steps, "pH": 7.0, "ionic": 0.01,
         "skin": 1.0, "drift": True, "sweep_every": 10, "first_step": 0, "confined": False, "replicas": 1}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a force evaluation of the reference's small charged test box: the smallest call
        _case("forces 1.2k", "forces", "plain", 1220, 0.298, ionic=0.1, skin=1.5, drift=False, sweep_every=1000),
        # the small preassembled soup (200 amphiphiles), the reference's fixed rebuild cadence, charges held
        _case("steps 3.3k", "steps", "amphiphile", 3277, 0.80, 10, ionic=0.0034, skin=1.5, drift=False,
              sweep_every=10 ** 9, first_step=1),
        # a medium preassembled soup with the charge Monte Carlo on, rebuilt on drift
        _case("steps 24k", "steps", "amphiphile", 23833, 0.80, 10, pH=6.0),
        # a finite parcel behind its wall
        _case("steps 60k parcel", "steps", "amphiphile", 60000, 1.10, 5, confined=True),
        # a quarter campaign on the reference's own schedule (skin 1.5, rebuild every 10, sweep every 1000)
        _case("steps 121k", "steps", "campaign", 120817, 1.1009, 5, skin=1.5, drift=False, sweep_every=1000),
        # the full campaign at the benchmark's schedule
        _case("steps 483k", "steps", "campaign", 483268, 1.1009, 5),
        # uneven replicas in one batch
        _case("batch 16", "batch", "amphiphile", 900000, 0.80, 5, replicas=16),
        # one constant-pH sweep: a medium box and the campaign's
        _case("sweep 121k", "sweep", "campaign", 120817, 1.1009),
        _case("sweep 483k", "sweep", "campaign", 483268, 1.1009),
        # forces of the full campaign: rebuild, force pass and readback
        _case("forces 483k", "forces", "campaign", 483268, 1.1009),
        # the gradient of an observable over a short window of the preassembled soup
        _case("window 33k", "window", "amphiphile", 32768, 0.80, 8, pH=9.0),
        # the progress sample of a preassembled soup
        _case("sample 110k", "sample", "amphiphile", 110000, 0.80),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choices(["steps", "batch", "forces", "sweep", "window", "sample"], [6, 1, 2, 2, 1, 1])[0]
    mix = "amphiphile" if kind in ("batch", "window", "sample") else rng.choice(["amphiphile", "campaign"])
    confined = kind == "steps" and mix == "amphiphile" and rng.random() < 0.25
    lo, hi = {"steps": (3000, 480000), "batch": (60000, 900000), "forces": (3000, 480000), "sweep": (20000, 480000),
              "window": (3000, 60000), "sample": (10000, 200000)}[kind]
    if confined:
        lo, hi = 10000, 120000
    dens = 1.10 if confined else (0.80 if mix == "amphiphile" else 1.1009)
    lo = max(lo, int(15.0 ** 3 * dens) + 1)
    drift = rng.random() < 0.7
    c = _case(None, kind, mix, int(_log(rng, lo, hi)), dens, pH=round(rng.uniform(5.0, 9.0), 2),
              ionic=float("%.4g" % _log(rng, 0.003, 0.1)), skin=round(rng.uniform(0.8, 1.2), 2) if drift else 1.5,
              drift=drift, sweep_every=rng.choice([10, 20, 1000]), confined=confined)
    if kind in ("steps", "batch"):
        c["steps"] = 5 if c["n"] > 30000 or confined else rng.choice([7, 10])
    if kind == "batch":
        c["replicas"] = max(2, min(32, int(c["n"] / _log(rng, 25000, 90000))))
    if kind == "window":
        c["steps"] = rng.randint(4, 8)
    return c


# ---- starts ----------------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _cell(side, beads, chains, seed):
    """(beads, 3) positions in a periodic cube of `side`: `chains` five-bead amphiphiles first (head, then
    four carbons), then free beads, pushed apart until contacts are about one bead diameter.  Positions of a
    chain stay unwrapped."""
    g = np.random.default_rng(seed)
    x = g.uniform(0.0, side, (beads, 3))
    if chains:
        u = g.normal(size=(chains, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        c = g.uniform(0.0, side, (chains, 3))
        x[:5 * chains] = (c[:, None, :] + ((np.arange(5) - 2.0) * 0.95)[None, :, None] * u[:, None, :]).reshape(-1, 3)
    x = torch.tensor(x, dtype=torch.float64, device="cuda")
    eye = torch.eye(beads, dtype=torch.bool, device="cuda")
    for it in range(240):
        d = x[:, None, :] - x[None, :, :]
        d = d - side * torch.round(d / side)
        r = d.norm(dim=-1).clamp_min(1e-3).masked_fill(eye, 9.0)
        w = torch.where(r < 1.0, (1.0 - r) / r, torch.zeros_like(r))
        move = 0.3 * (w[:, :, None] * d).sum(dim=1)
        if chains:                       # bonds towards 0.95, second neighbours towards 1.9
            p = x[:5 * chains].view(chains, 5, 3)
            m = torch.zeros_like(p)
            for k, rest, f in ((1, 0.95, 0.3), (2, 1.9, 0.1)):
                v = p[:, k:] - p[:, :-k]
                s = f * (1.0 - rest / v.norm(dim=-1, keepdim=True))
                m[:, :-k] += s * v
                m[:, k:] -= s * v
            move = torch.cat([move[:5 * chains] + m.reshape(-1, 3), move[5 * chains:]])
        x = x + move.clamp(-0.15, 0.15)
    return x.cpu().numpy()


def _beads(mix, n, side, confined_r, seed):
    """Positions (n, 3) in a cube of `side` (or in a parcel of radius confined_r about its centre), kinds (n,)
    and bond slots (n, 3)."""
    g = np.random.default_rng(seed + 1)
    k = max(1, int(side / 8.0))
    a = side / k
    per = -(-n // k ** 3) if not confined_r else int(round(n / (4.0 / 3.0 * math.pi * confined_r ** 3) * a ** 3))
    chains = {"amphiphile": int(0.15 * per) // 5}.get(mix, 0)
    cell = _cell(a, per, chains, seed % 1000003)
    t = np.stack(np.meshgrid(*[np.arange(k) * a] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    pos = np.mod(t + cell[None] + g.uniform(0.0, side, 3), side)      # (tiles, per, 3)
    cb = 5 * chains
    head, free = pos[:, :cb].reshape(-1, 5, 3), pos[:, cb:].reshape(-1, 3)
    if confined_r:                                                    # the innermost chains and beads
        na = int(n * cb / per) // 5
        head = head[np.argsort(np.linalg.norm(head - side / 2, axis=-1).max(axis=1), kind="stable")[:na]]
        free = free[np.argsort(np.linalg.norm(free - side / 2, axis=-1), kind="stable")[: n - 5 * na]]
    else:                                                             # drop the few beads over n
        free = free[np.sort(g.permutation(len(free))[: n - head.shape[0] * 5])]
    na = len(head)
    xyz = np.concatenate([head.reshape(-1, 3), free])
    if mix == "amphiphile":
        kinds = np.concatenate([np.tile([1, 0, 0, 0, 0], na), np.full(len(free), 4)])
    else:
        census = CAMPAIGN if mix == "campaign" else PLAIN
        total = sum(census.values())
        counts = {q: int(round(n * v / total)) for q, v in census.items()}
        counts["W" if mix == "campaign" else "C"] += n - sum(counts.values())
        kinds = np.concatenate([np.full(counts[q], KIND[q]) for q in KIND])
        xyz = xyz[g.permutation(n)]
    slots = np.full((len(xyz), 3), NONE, np.uint32)
    b = 5 * np.arange(na, dtype=np.uint32)
    slots[b, 0] = b + 1
    slots[b + 1, 2], slots[b + 1, 0] = b, b + 2
    slots[b + 2, 0], slots[b + 2, 1] = b + 1, b + 3
    slots[b + 3, 0], slots[b + 3, 1] = b + 2, b + 4
    slots[b + 4, 0] = b + 3
    return xyz, kinds, slots


def _system(case, n, seed):
    """(SoupConfig, start state) of one system."""
    radius = (n / case["density"] / (4.0 / 3.0 * math.pi)) ** (1.0 / 3.0) if case["confined"] else 0.0
    # a parcel's face clearance has to exceed the head-list range
    debye = 0.304 / math.sqrt(case["ionic"]) / 0.8
    side = 2.0 * radius + 2.0 * (4.0 * debye + case["skin"]) + 2.0 if radius else (n / case["density"]) ** (1.0 / 3.0)
    xyz, kinds, slots = _beads(case["mix"], n, side, radius, seed)
    m = len(xyz)
    heads = kinds == KIND["O"]
    # room for the heads' clumping: in a parcel all of them are near one another
    cap = int(heads.sum())
    if not radius and case["mix"] == "amphiphile":
        reach = min(4.0 * debye, 0.45 * side) + case["skin"]
        cap = min(cap, int(3.0 * cap / side ** 3 * 4.0 / 3.0 * math.pi * reach ** 3) + 128)
    opts = pg.SoupOptions(
        box=[side] * 3, seed=seed % (1 << 31), kT=1.1, start={q: int((kinds == KIND[q]).sum()) for q in KIND},
        electrostatics={"enabled": True, "pH": case["pH"], "ionicStrengthMolar": case["ionic"]},
        skin=case["skin"], rebuild_on_drift=case["drift"], sweep_every=case["sweep_every"],
        chunk_steps=min(1000, case["sweep_every"]), global_step=case["first_step"],
        confine={"radiusSigma": radius, "stiffness": 100.0} if radius else None,
        es_list_capacity=max(64, cap) if case["mix"] == "amphiphile" else None)
    g = np.random.default_rng(seed + 2)
    pos = np.zeros((m, 4), np.float32)
    pos[:, :3], pos[:, 3] = xyz, kinds
    pos[:, :3][pos[:, :3] >= np.float32(side)] = 0.0                  # rounded onto the far face
    vel = np.zeros((m, 4), np.float32)
    vel[:, :3] = g.normal(scale=math.sqrt(1.1), size=(m, 3))
    state = dict(positions=pos.reshape(-1), velocities=vel.reshape(-1), bond_slots=slots.reshape(-1),
                 charges=np.where(heads & (g.random(m) < 0.5), -1.0, 0.0).astype(np.float32),
                 frozen=np.zeros(m, np.uint32), bond_rng=g.integers(1 << 32, size=m, dtype=np.uint32),
                 thermo_rng=g.integers(1 << 32, size=m, dtype=np.uint32))
    return config.resolve(opts), state


def _replica_sizes(case):
    """Uneven replicas, box sides within +-30%, `n` beads in all; none below the smallest box."""
    w = np.random.default_rng(case["n"]).uniform(0.7, 1.3, case["replicas"]) ** 3
    return [max(4000, int(v)) for v in case["n"] * w / w.sum()]


def _start(case, seed):
    if case["kind"] == "batch":
        return [_system(case, m, seed + 17 * r) for r, m in enumerate(_replica_sizes(case))]
    return [_system(case, case["n"], seed)]


def prepare(case, seed):
    starts = _start(case, seed)
    s = {"case": case}
    if case["kind"] == "batch":
        s["soup"] = pg.SoupBatch([c for c, _ in starts], [st for _, st in starts])
        return s
    cfg, st = starts[0]
    s["soup"] = pg.SoupSystem(cfg, st)
    kinds = st["positions"][3::4].astype(np.int64)
    if case["kind"] == "window":
        s["heads"] = torch.tensor(np.nonzero(kinds == KIND["O"])[0], device="cuda")
        s["tails"] = torch.tensor(np.nonzero(kinds == KIND["C"])[0], device="cuda")
        s["theta"] = torch.tensor(s["soup"].get_diff_params(), dtype=torch.float32)
    if case["kind"] == "sample":
        s["water"] = np.nonzero(kinds == KIND["W"])[0].astype(np.uint32)
        s["cutoff"] = float(cfg.rc_attr + cfg.wc)
        s["params"] = config.load_params()
    return s


def run(state):
    case, soup = state["case"], state["soup"]
    kind = case["kind"]
    if kind == "steps":
        soup.step(case["steps"])
        a, _ = soup.checkpoint_payload()
        return {q: a[q] for q in ("positions", "velocities", "charges", "bondSlots", "thermoRng")}
    if kind == "batch":
        soup.step(case["steps"])
        return [(r.particles(), r.velocities()) if case["replicas"] > 21 else
                (r.particles(), r.velocities(), r.charges()) for r in soup.replicas]
    if kind == "forces":
        return soup.forces()
    if kind == "sweep":
        r = soup.protonation_sweep()
        return soup.charges(), r["accepted"], r["deprotonated"]
    if kind == "window":
        theta = state["theta"].clone().requires_grad_(True)
        traj = adjoint.SoupWindow.apply(theta, soup, case["steps"], case["steps"])
        loss = adjoint.thickness_proxy(traj, state["heads"], state["tails"], float(soup.cfg.box[2]))
        loss.backward()
        return traj.detach(), theta.grad
    # sample
    P = state["params"]["stageThresholds"]
    amphiphiles, head_of = soup.amphiphile_labels()
    members = np.nonzero(head_of != NONE)[0].astype(np.uint32)
    comps, labels = soup.aggregate_labels(members, state["cutoff"])
    _, shapes = soup.aggregate_shapes(members, labels, int(P["detailAggregateCount"]))
    pos = soup.particles()
    inside = []
    for sh in shapes:
        m = members[labels == sh["label"]]
        c = observables.periodic_centre(pos, m, list(soup.cfg.box), state["params"]["circularAlpha"])
        if c is None:      # the aggregate spans the box: about its own centre instead
            c = [v % b for v, b in zip(sh["centre"], soup.cfg.box)]
        r = soup.closure(m, state["water"], c, P["closureCell"], P["closureRadius"], P["enclosedVolume"])
        inside.append([r["encapsulatedCount"], r["totalEmptyCells"], r["unreachedCells"], r["seedCell"]])
    return head_of, labels, [amphiphiles, comps], inside, [sh["gyration"] for sh in shapes]


# ---- work ------------------------------------------------------------------------------------
def work(case):
    """One pass: state in and out once a step, each pair of beads in reach once (about 40 operations), each
    pair of heads in reach once a sweep; host results once."""
    n, dens, steps = case["n"], case["density"], case["steps"]
    share = {"amphiphile": 0.03, "campaign": 0.0386, "plain": 0.082}[case["mix"]]
    heads = share * n
    pairs = n * 0.5 * dens * 4.0 / 3.0 * math.pi * 2.947 ** 3
    rc = min(4.0 * 0.304 / math.sqrt(case["ionic"]) / 0.8, 0.45 * (n / case["replicas"] / dens) ** (1.0 / 3.0))
    hpairs = heads * 0.5 * dens * share * 4.0 / 3.0 * math.pi * rc ** 3
    force = {"bytes": 56.0 * n, "flops": 40.0 * pairs + 25.0 * hpairs}
    sweep = {"bytes": 28.0 * heads, "flops": 60.0 * hpairs}
    kind = case["kind"]
    if kind in ("steps", "batch"):
        k = steps // case["sweep_every"]
        return {"bytes": steps * 144.0 * n + k * sweep["bytes"] + 52.0 * n, "flops": steps * force["flops"] + k * sweep["flops"]}
    if kind == "forces":
        return {"bytes": force["bytes"] + 16.0 * n, "flops": force["flops"]}
    if kind == "sweep":
        return {"bytes": sweep["bytes"] + 4.0 * n, "flops": sweep["flops"] + force["flops"]}
    if kind == "window":
        return {"bytes": steps * 400.0 * n, "flops": 4.0 * steps * force["flops"]}
    return {"bytes": 40.0 * n + 5 * 2.0 * n / dens / 0.125, "flops": 10.0 * share * 5.0 * n * 40.0}


# ---- 64-bit results ----------------------------------------------------------------------------
def _pairs(x, box, reach):
    """(i, j), i < j, of the beads within reach of one another, by minimum image (cubic box)."""
    nc = max(1, min(64, int(box / reach)))
    if nc < 3:
        out = []
        for r0 in range(0, len(x), 2048):
            d = x[r0:r0 + 2048, None, :] - x[None, :, :]
            d = d - box * torch.round(d / box)
            i, j = ((d * d).sum(-1) < reach * reach).nonzero(as_tuple=True)
            i = i + r0
            out.append(torch.stack([i, j])[:, i < j])
        return torch.cat(out, dim=1)
    c = (x / box * nc).long().clamp(0, nc - 1)
    key = (c[:, 0] * nc + c[:, 1]) * nc + c[:, 2]
    order = torch.argsort(key, stable=True)
    count = torch.bincount(key, minlength=nc ** 3)
    start = torch.cumsum(count, 0) - count
    m = int(count.max())
    at = start[:, None] + torch.arange(m, device=x.device)
    table = torch.where(torch.arange(m, device=x.device) < count[:, None], order[at.clamp(max=len(x) - 1)], -1)
    cells = torch.arange(nc ** 3, device=x.device)
    cc = torch.stack([cells // (nc * nc), cells // nc % nc, cells % nc], 1)
    rows = max(1, (1 << 25) // (m * m))
    out = []
    for o in range(27):
        off = torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device=x.device)
        nb = (cc + off) % nc
        nb = (nb[:, 0] * nc + nb[:, 1]) * nc + nb[:, 2]
        for r0 in range(0, nc ** 3, rows):
            a, b = table[r0:r0 + rows, :, None], table[nb[r0:r0 + rows], None, :]
            ok = (a >= 0) & (b > a)
            i, j = a.expand(ok.shape)[ok], b.expand(ok.shape)[ok]
            d = x[i] - x[j]
            d = d - box * torch.round(d / box)
            near = (d * d).sum(-1) < reach * reach
            out.append(torch.stack([i[near], j[near]]))
    return torch.cat(out, dim=1)


class _Exact:
    """The force and the Langevin step of one system in FP64 torch (bonded and bend terms of static bonds,
    screened Coulomb, wall)."""

    def __init__(self, cfg, st):
        t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.c, self.box = cfg, float(cfg.box[0])
        p = np.asarray(st["positions"], np.float64).reshape(-1, 4)
        self.x, self.v = t(p[:, :3]), t(np.asarray(st["velocities"], np.float64).reshape(-1, 4)[:, :3])
        self.q, self.kind = t(st["charges"]), torch.tensor(p[:, 3].astype(np.int64), device="cuda")
        self.radius = t([cfg.radius[k] for k in range(8)])
        self.cls = torch.tensor([cfg.kind_class[k] & 3 for k in range(8)], device="cuda")
        self.c6 = 2.0 ** float(np.float32(1.0 / 6.0))
        self.reach = max(self.c6 * cfg.b_tt + cfg.wc, self.c6 * float(cfg.sigma) * 1.2, float(cfg.es_split_radius))
        self.heads = (self.q != 0).nonzero()[:, 0]
        s = st["bond_slots"].reshape(-1, 3).astype(np.int64)
        b, mid = set(), {}
        for i, k in zip(*np.nonzero(s != NONE)):
            b.add((min(i, s[i, k]), max(i, s[i, k])))
            mid.setdefault(i, set()).add(int(s[i, k]))
        bend = {(a, c) for v in mid.values() for a in v for c in v if a < c}
        pt = lambda z: torch.tensor(np.array(sorted(z), np.int64).reshape(-1, 2).T.copy(), device="cuda")  # noqa: E731
        self.bond, self.bend = pt(b), pt(bend)
        self.rng = np.asarray(st["thermo_rng"], np.uint64).copy()

    def theta(self):
        c = self.c
        d = [c.attr_scale[a][b] for a, b in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))]
        th = np.array(d + [c.k_fene, c.k_bend, c.es_kappa]).astype(np.float32).astype(np.float64)
        return torch.tensor(th, dtype=torch.float64, device="cuda")

    def _add(self, f, ij, x, scalar):
        d = x[ij[0]] - x[ij[1]]
        d = d - self.box * torch.round(d / self.box).detach()
        s = scalar(d.norm(dim=-1), ij[0], ij[1])[:, None] * d
        return f.index_add(0, ij[0], s).index_add(0, ij[1], -s)

    def force(self, x, theta=None):
        c, pi = self.c, math.pi
        eps, wc, rc = float(c.epsilon), float(c.wc), self.c6 * float(c.b_tt)
        depth = torch.tensor([[c.attr_scale[a][b] for b in range(4)] for a in range(4)], dtype=torch.float64, device="cuda")
        kf, kb, kap = float(c.k_fene), float(c.k_bend), float(c.es_kappa)
        if theta is not None:
            kf, kb, kap = theta[6], theta[7], theta[8]
            for k, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
                m = torch.zeros_like(depth)
                m[a, b] = m[b, a] = 1.0
                depth = depth * (1 - m) + theta[k] * m
        kap = torch.as_tensor(kap, dtype=torch.float64, device="cuda")

        def near(r, i, j):
            ki, kj = self.kind[i], self.kind[j]
            b = float(c.sigma) * (self.radius[ki] + self.radius[kj]) / 2
            ci, cj = self.cls[ki], self.cls[kj]
            s6 = (b / r) ** 6
            s = torch.where(r < self.c6 * b, 24 * eps * (2 * s6 * s6 - s6) / r ** 2, torch.zeros_like(r))
            acid = float(c.acid_soap_scale) * ((ci == 1) & (cj == 1) & ((self.q[i] != 0) != (self.q[j] != 0)))
            on = (r >= rc) & (r <= rc + wc)
            return s - torch.where(on, (depth[ci, cj] + acid) * eps * pi / (2 * wc) * torch.sin(pi * (r - rc) / wc) / r,
                                   torch.zeros_like(r))

        def coulomb(r, i, j):
            re, A = float(c.es_cutoff), float(c.es_coeff_a)
            shift = A * torch.exp(-kap * re) * (1 / re ** 2 + kap / re)
            return torch.where(r < re, self.q[i] * self.q[j] * (A * torch.exp(-kap * r) * (1 / r ** 2 + kap / r) - shift) / r,
                               torch.zeros_like(r))

        with torch.no_grad():
            ij = _pairs(x.detach(), self.box, self.reach)
            hh = self.heads[_pairs(x.detach()[self.heads], self.box, float(c.es_cutoff))]
        f = self._add(torch.zeros_like(x), ij, x, near)
        f = self._add(f, hh, x, coulomb)
        f = self._add(f, self.bond, x, lambda r, i, j: -kf / (1 - (r / float(c.r_inf)) ** 2))
        f = self._add(f, self.bend, x, lambda r, i, j: -kb * (r - float(c.r_bend)) / r)
        if c.wall_radius > 0:
            d = x - self.box / 2
            r = d.norm(dim=-1, keepdim=True)
            f = f - torch.where(r > c.wall_radius, float(c.wall_k) * (r - float(c.wall_radius)) / r, torch.zeros_like(r)) * d
        return f

    def _noise(self):
        """The thermostat's three normals per bead from its 32-bit stream (PCG hash, Box-Muller)."""
        out, m = np.empty((len(self.rng), 3)), np.uint64(0xFFFFFFFF)

        def nxt(v):
            s = (v * np.uint64(747796405) + np.uint64(2891336453)) & m
            w = (((s >> ((s >> np.uint64(28)) + np.uint64(4))) ^ s) * np.uint64(277803737)) & m
            return (w >> np.uint64(22)) ^ w
        for a in range(3):
            self.rng = nxt(self.rng)
            u = np.maximum(self.rng.astype(np.float32) / np.float32(2.0 ** 32), np.float32(1e-7)).astype(np.float64)
            self.rng = nxt(self.rng)
            w = (self.rng.astype(np.float32) / np.float32(2.0 ** 32)).astype(np.float64)
            out[:, a] = np.sqrt(-2.0 * np.log(u)) * np.cos(float(np.float32(6.28318531)) * w)
        return torch.tensor(out, device="cuda")

    def steps(self, k, theta=None):
        """Positions after 0..k steps and the last velocities."""
        c = self.c
        dt, g = float(np.float32(c.dt)), float(np.float32(c.gamma))
        sv = math.sqrt(2.0 * g * float(c.kT) * dt)
        x, v, out = self.x, self.v, [self.x]
        f = self.force(x, theta)
        for _ in range(k):
            v = v + 0.5 * dt * f
            x = x + dt * v
            x = x - self.box * torch.floor(x.detach() / self.box)
            f = self.force(x, theta)
            v = (1.0 - g * dt) * (v + 0.5 * dt * f) + sv * self._noise()
            out.append(x)
        return out, v

    def rows(self, x, w=None):
        """(n * 4) as the library lays beads out."""
        w = self.kind.double() if w is None else torch.zeros_like(self.q)
        return torch.cat([x, w[:, None]], 1)


def exact(case, seed):
    kind, k = case["kind"], case["steps"]
    if kind == "forces":
        e = _Exact(*_system(case, case["n"], seed))
        return e.rows(e.force(e.x), 0).reshape(-1)
    if kind == "steps" and k < case["sweep_every"] and 0 < case["first_step"] <= 20 - k and case["n"] <= 60000:
        e = _Exact(*_system(case, case["n"], seed))           # no Monte Carlo pass falls into these steps
        xs, v = e.steps(k)
        return {"positions": e.rows(xs[-1]).reshape(-1), "velocities": e.rows(v, 0).reshape(-1),
                "charges": e.q, "bondSlots": None, "thermoRng": None}
    if kind == "window":
        e = _Exact(*_system(case, case["n"], seed))
        theta = e.theta().requires_grad_(True)
        xs, _ = e.steps(k, theta)
        traj = torch.stack([e.rows(x) for x in xs])
        heads, tails = (torch.nonzero(e.kind == KIND[q])[:, 0] for q in ("O", "C"))
        z = traj[:, :, 2]                                     # the thickness proxy, in FP64
        both = torch.cat([heads, tails])
        ref = z[0, both].mean()
        z = z - torch.round((z - ref) / e.box).detach() * e.box
        loss = 2.0 * (z[:, heads] - z[:, both].mean(dim=1, keepdim=True)).abs().mean()
        loss.backward()
        return traj.detach(), theta.grad
    return None
