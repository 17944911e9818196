"""The performance cases of softmold_gb300: what a user of the framework has it do.

Six kinds of call, each through the public Python mirror of the C ABI:

  run       a stretch of a production run: advance some loop iterations, then read the state and the box
            (one checkpoint or trajectory-frame interval)
  measure   a measurement interval as the `MD` executable runs it: advance to a measure step, reduce the
            measurements and the energies on the device, read the frame
  frame     forces and energies of a given configuration (re-analysis of stored frames, a driver that
            owns the integration)
  static    non-bonded forces of device-resident coordinates owned by another framework
            (smd_pair_forces_static)
  adjoint   gradient of a time-averaged potential through a window of loop steps

Systems are the generators' (flat bilayer, vesicle, vesicle with a continuum sphere, a batch of bilayers)
at the reference's constants, melted from their lattice start before they are handed over, so that every
pass meets the running membrane's density and energies.
"""
import dataclasses
import math
import os
import tempfile

import numpy as np
import torch

import softmold_gb300 as smd

MELT = 400    # loop steps from the generator's lattice to the running membrane
LEAD_IN = 17  # loop steps of a fresh handle before the first pass: one, then two barostat periods
DENSITY = 3.45
Z_BILAYER = 15.0
TAIL = 3


def listed():
    return [
        # a patch small enough for statistics over many short runs: launch latency decides
        dict(name="run bilayer 400", kind="run", shape="bilayer", lipids=400, replicas=1, fp64=False, steps=48),
        # the reference's customary vesicle, mostly empty box, no barostat
        dict(name="run vesicle 5k", kind="run", shape="vesicle", lipids=5000, replicas=1, fp64=False, steps=48),
        # the headline workload: tensionless bilayer with the Monte-Carlo barostat
        dict(name="run bilayer 20k", kind="run", shape="bilayer", lipids=20000, replicas=1, fp64=False, steps=48),
        # nanoparticle on a large vesicle: the sphere terms and a large sparse cell grid
        dict(name="run sphere 40k", kind="run", shape="sphere", lipids=40000, replicas=1, fp64=False, steps=24),
        # parameter sweep of independent bilayers in one handle, own box, seed and tension each
        dict(name="run batch 16", kind="run", shape="bilayer", lipids=2500, replicas=16, fp64=False, steps=24),
        # the all-FP64 form, for validation and for steep potentials: a bilayer and a vesicle, odd sizes
        dict(name="run bilayer 1537 fp64", kind="run", shape="bilayer", lipids=1537, replicas=1, fp64=True, steps=24),
        dict(name="run vesicle 6k fp64", kind="run", shape="vesicle", lipids=6001, replicas=1, fp64=True, steps=16),
        # measurement and frame every 40 steps of a mid-size vesicle
        dict(name="measure vesicle 2.5k", kind="measure", shape="vesicle", lipids=2501, replicas=1, fp64=False,
             steps=40),
        # forces and energies of stored frames, both forms
        dict(name="frame bilayer 10k", kind="frame", shape="bilayer", lipids=10000, replicas=1, fp64=False, steps=0),
        dict(name="frame vesicle 3k fp64", kind="frame", shape="vesicle", lipids=3001, replicas=1, fp64=True,
             steps=0),
        # pair forces for a caller that owns the device memory, near the entry point's bead limit
        dict(name="static bilayer 10k", kind="static", shape="bilayer", lipids=10000, replicas=1, fp64=True, steps=0),
        # gradient of a 40-step average, checkpoints every 20
        dict(name="adjoint bilayer 5k", kind="adjoint", shape="bilayer", lipids=5000, replicas=1, fp64=False,
             steps=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "run", "measure", "frame", "static", "adjoint"])
    fp64 = rng.random() < 0.35
    shape = rng.choice(["bilayer", "vesicle"])
    replicas = 1
    if kind == "run":
        if not fp64 and rng.random() < 0.2:
            shape = "sphere"
        lipids = _log_int(rng, 3000, 30000) if shape == "sphere" else _log_int(rng, 300, 6000 if fp64 else 30000)
        if shape == "bilayer" and not fp64 and rng.random() < 0.3:
            replicas = rng.randint(2, 24)
            lipids = _log_int(rng, 500, 30000 // replicas + 500)
        steps = 8 * rng.randint(1, 3 if fp64 else 6)
    elif kind == "measure":
        lipids, steps = _log_int(rng, 700, 3000 if fp64 else 15000), rng.randint(8, 24 if fp64 else 60)
    elif kind == "frame":
        lipids, steps = _log_int(rng, 2000, 6000 if fp64 else 25000), 0
    elif kind == "static":
        shape, fp64, lipids, steps = "bilayer", True, _log_int(rng, 300, 10900), 0
    else:
        shape, lipids, steps = "bilayer", _log_int(rng, 400, 1500 if fp64 else 8000), rng.randint(10, 20 if fp64 else 50)
    return dict(kind=kind, shape=shape, lipids=lipids, replicas=replicas, fp64=fp64, steps=steps)


# ------------------------------------------------------------------ inputs
def _lattice(case, seed, k, folder):
    """Replica k of the case from the generators (the adjoint holds the box fixed)."""
    p = os.path.join(folder, "s%d.mpd" % k)
    n, s = case["lipids"], 1 + (1000003 * seed + 7919 * k) % 2147480000
    if case["shape"] == "bilayer":
        lipids = n if case["replicas"] == 1 else max(300, n * (6 + k % 9) // 10)  # ragged replicas
        tension = 0.0 if case["replicas"] == 1 else (k % 5) * 0.25
        smd.synth_bilayer(p, s, lipids, DENSITY, Z_BILAYER, 0.0 if case["kind"] == "adjoint" else 0.01, tension)
    elif case["shape"] == "vesicle":
        smd.synth_vesicle(p, s, n, DENSITY, max(30.0, 60.0 * math.sqrt(n / 5000.0)))
    else:
        # heads keep a barrier inside the surface (Umax 300) and a well on it (Umin -10)
        box = max(190.0 * math.sqrt(n / 80000.0), 2.0 * (math.sqrt(n / (4.0 * math.pi * DENSITY)) + 22.0))
        smd.synth_vesicle_sphere(p, s, n, DENSITY, box, 5.0, -10.0, 300.0, 2.0, 100.0)
    m = smd.read_mpd(p)
    os.remove(p)
    return m


def _membranes(case, seed):
    """The case's systems at a melted state: what a checkpoint of a running simulation holds."""
    with tempfile.TemporaryDirectory() as folder:
        ms = [_lattice(case, seed, k, folder) for k in range(case["replicas"])]
    h = smd.System(ms, precision=smd.MIXED)
    h.prepare()
    h.advance(MELT)
    pos, vel = h.state()
    out, at = [], 0
    for k, m in enumerate(ms):
        n = len(m.type)
        out.append(dataclasses.replace(m, pos=pos[at:at + n].copy(), vel=vel[at:at + n].copy(), box=h.box(k),
                                       initial_time=0.0))
        at += n
    h.close()
    return out


def _pinned(n):
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    ms = _membranes(case, seed)
    n = sum(len(m.type) for m in ms)
    st = {"case": case, "n": n}
    if case["kind"] == "static":
        m = ms[0]
        st.update(pos=torch.from_numpy(m.pos).cuda(), type=torch.from_numpy(m.type.astype(np.int32)).cuda(),
                  fconst=torch.from_numpy(m.fconst).cuda(), n_types=m.n_types, cutoff=float(m.cutoff),
                  box=np.ascontiguousarray(m.box, np.float64),
                  out=torch.empty((n, 3), dtype=torch.float64, device="cuda"))
        return st
    s = smd.System(ms, precision=smd.PLAIN_FP64 if case["fp64"] else smd.MIXED)
    s.autotune()  # what a run does by itself after 256 steps
    st.update(s=s, pos=_pinned(n), vel=_pinned(n))
    if case["kind"] == "frame":
        st.update(frame_pos=_pinned(n), frame_vel=_pinned(n))
        st["frame_pos"][:] = np.concatenate([m.pos for m in ms])
        st["frame_vel"][:] = np.concatenate([m.vel for m in ms])
        return st
    s.prepare()
    if case["kind"] != "adjoint":
        s.advance(1)
        s.advance(LEAD_IN - 1)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "static":
        rc = smd.lib().smd_pair_forces_static(st["pos"].data_ptr(), st["type"].data_ptr(), st["n"],
                                              st["box"].ctypes.data, st["cutoff"], st["n_types"],
                                              st["fconst"].data_ptr(), st["out"].data_ptr(), None)
        if rc:
            raise smd.SmdError(smd.last_error())
        return {"force": st["out"]}
    s = st["s"]
    if kind == "run":
        s.advance(case["steps"])
        pos, vel = s.state(st["pos"], st["vel"])
        return {"pos": pos, "vel": vel, "box": np.stack([s.box(r) for r in range(case["replicas"])])}
    if kind == "measure":
        s.advance(case["steps"], stop_at_measure=True)
        box = s.box()
        e = s.energy()[0]
        q = s.measure()
        pos, vel = s.state(st["pos"], st["vel"])
        return {"pos": pos, "vel": vel, "box": box, "energy": e, "kinetic": q["kinetic"], "lo": q["lo"], "hi": q["hi"]}
    if kind == "frame":
        s.set_state(st["frame_pos"], st["frame_vel"])
        return {"force": s.forces(), "energy": s.energy()}
    r = s.adjoint(case["steps"], checkpoint_every=20, umin_types=(TAIL, TAIL), segment_local=True)
    pos, vel = s.state(st["pos"], st["vel"])
    return {"pos": pos, "vel": vel, "mean_potential": r["mean_potential"], "grad": r["grad"]}


def work(case):
    """State in and out once; about 25 pairs within the cutoff per bead (each pair once) at 36 operations for
    the force and 20 for the energy, 300 per bead and step for the bonded terms, the noise and the update."""
    n = 3 * case["lipids"] * case["replicas"]
    steps = case["steps"]
    pairs = 25.0 * n
    if case["kind"] == "static":
        return {"bytes": n * (24 + 4 + 24), "flops": pairs * 36}
    if case["kind"] == "frame":
        return {"bytes": n * (48 + 24), "flops": pairs * (36 + 20) + n * 300.0}
    if case["kind"] == "adjoint":  # forward, then the Hessian-vector product of each step
        return {"bytes": n * 96, "flops": steps * (pairs * (36 + 20 + 70) + n * 1200.0)}
    return {"bytes": n * 96, "flops": steps * (pairs * 36 + n * 300.0)}


# ------------------------------------------------------------------ 64-bit values
def _philox(seed, n, it, phase):
    """The Langevin draws of one loop step: Philox4x32-10 (Salmon et al., SC'11), uniform in (-1, 1)."""
    low = np.uint64(0xFFFFFFFF)
    c = [np.arange(n, dtype=np.uint64), np.full(n, it & 0xFFFFFFFF, np.uint64),
         np.full(n, (it >> 32) ^ (phase << 31), np.uint64), np.full(n, 0x6D2B, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, 0x5A17
    for _ in range(10):
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & low, (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return (np.stack(c[:3], 1).astype(np.float64) - 2147483648.0 + 0.5) / 2147483648.0


class _Exact:
    """One membrane's potential, forces and loop in FP64 torch operations."""

    def __init__(self, m):
        self.m, self.dev = m, torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.box = torch.as_tensor(np.asarray(m.box, np.float64), device=self.dev).clone()
        self.type = torch.as_tensor(m.type.astype(np.int64), device=self.dev)
        self.u = torch.as_tensor(m.uconst, device=self.dev).reshape(-1, 6)
        self.x = torch.as_tensor(m.pos, device=self.dev).clone()
        self.v = torch.as_tensor(m.vel, device=self.dev).clone()
        self.move = (self.type != 0)[:, None]
        self.sigma = math.sqrt(6.0 * m.temperature * m.gamma / m.dt)
        self.draws = np.random.RandomState(m.seed & 0xFFFFFFFF)
        bonds, bends = [], []
        for start, count, length in np.asarray(m.chain_blocks).reshape(-1, 3):
            first = start + length * np.arange(count)
            bonds += [first + q for q in range(length - 1)]
            bends += [first + q for q in range(length - 2)]
        self.bond = torch.as_tensor(np.concatenate(bonds), device=self.dev)
        self.bend = torch.as_tensor(np.concatenate(bends), device=self.dev)
        self.k = torch.as_tensor(np.asarray(m.chain_consts, np.float64).reshape(-1, 4)[0], device=self.dev)

    def image(self, d, box):
        return d - box * torch.round(d / box)

    def pairs(self, x, box, cut):
        """Every pair within cut once, from a table of the cells' beads."""
        nc = [max(3, int(b / cut)) for b in box.tolist()]
        if min(float(b) / c for b, c in zip(box, nc)) < cut:
            raise ValueError("box below three cells")
        size = torch.as_tensor(nc, device=self.dev)
        c3 = torch.minimum((x / box * size).floor().long().clamp_min(0), size - 1)
        key = c3[:, 0] + nc[0] * (c3[:, 1] + nc[1] * c3[:, 2])
        count = torch.bincount(key, minlength=nc[0] * nc[1] * nc[2])
        order = torch.argsort(key, stable=True)
        start = torch.cumsum(count, 0) - count
        slot = torch.arange(len(x), device=self.dev) - start[key[order]]
        table = torch.full((len(count), int(count.max())), -1, dtype=torch.long, device=self.dev)
        table[key[order], slot] = order
        me = torch.arange(len(x), device=self.dev)[:, None]
        found = []
        for o in range(14):  # the cell itself and half of its 26 neighbours
            step = torch.as_tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device=self.dev)
            c = (c3 + step) % size
            j = table[c[:, 0] + nc[0] * (c[:, 1] + nc[1] * c[:, 2])]
            ok = j >= 0 if o != 13 else j > me
            d = self.image(x[:, None, :] - x[j.clamp_min(0)], box)
            ok &= (d * d).sum(-1) < cut * cut
            at = ok.nonzero()
            found.append(torch.stack([at[:, 0], j[at[:, 0], at[:, 1]]]))
        return torch.cat(found, 1)

    def pair_energy(self, x, box, ij, u=None):
        u = self.u if u is None else u
        c = u[self.type[ij[0]] * self.m.n_types + self.type[ij[1]]]
        r = self.image(x[ij[0]] - x[ij[1]], box).square().sum(-1).sqrt()
        inner, m = c[:, 0] - r, c[:, 3] - r
        e = torch.where(r <= c[:, 0], c[:, 1] * inner * inner + c[:, 2], m * m * (c[:, 4] - m * c[:, 5]))
        return torch.where(r < self.m.cutoff, e, torch.zeros_like(e)).sum()

    def bonded_energy(self, x, box, k=None):
        k = self.k if k is None else k
        d = self.image(x[self.bond] - x[self.bond + 1], box)
        e = 0.5 * k[1] * (d.square().sum(-1).sqrt() - k[0]).square().sum()
        a, b = self.image(x[self.bend] - x[self.bend + 1], box), self.image(x[self.bend + 1] - x[self.bend + 2], box)
        cos = (a * b).sum(-1) / (a.square().sum(-1) * b.square().sum(-1)).sqrt()
        return e + 0.5 * k[3] * (k[2] - cos).square().sum()

    def potential(self, x, box):
        return self.pair_energy(x, box, self.pairs(x.detach(), box, self.m.cutoff)) + self.bonded_energy(x, box)

    def force(self, pair_only=False):
        x = self.x.detach().requires_grad_(True)
        e = self.pair_energy(x, self.box, self.pairs(self.x, self.box, self.m.cutoff))
        if not pair_only:
            e = e + self.bonded_energy(x, self.box)
        return -torch.autograd.grad(e, x)[0]

    def noise(self, it, phase=0):
        return self.sigma * torch.as_tensor(_philox(self.m.seed, len(self.x), it, phase), device=self.dev)

    def kick(self, a):
        self.v = torch.where(self.move, self.v + 0.5 * self.m.dt * a, self.v)

    def drift(self):
        self.x = torch.where(self.move, self.x + self.m.dt * self.v, self.x)
        self.x = torch.where(self.x > self.box, self.x - self.box, self.x)
        self.x = torch.where(self.x < 0, self.x + self.box, self.x)

    def start(self):
        a = self.force() - self.m.gamma * self.v + self.noise(0, 1)
        self.kick(a)
        self.drift()
        self.it = 0

    def step(self, stop=False):
        a = self.force() - self.m.gamma * self.v + self.noise(self.it)
        self.kick(a)
        if stop:
            self.held = a
            return
        self.finish(a)

    def finish(self, a):
        if self.m.delta_lxy != 0 and self.it % 8 == 0 and self.it != 0:
            u1, u2 = self.draws.random_sample(), self.draws.random_sample()
            b = self.box.tolist()
            f = self.m.delta_lxy * (2.0 * u1 - 1.0)
            new = torch.as_tensor([b[0] + f, b[1] + f, b[2] * (b[0] * b[1]) / ((b[0] + f) * (b[1] + f))],
                                  dtype=torch.float64, device=self.dev)
            s = new / self.box
            d = float(self.potential(self.x, self.box) - self.potential(self.x * s, new))
            d += self.m.tension * float(new[0] * new[1] - self.box[0] * self.box[1])
            if d >= 0 or math.exp(d / self.m.temperature) >= u2:
                self.x, self.box = self.x * s, new
        self.kick(a)
        self.drift()
        self.it += 1

    def energy(self):
        ij = self.pairs(self.x, self.box, self.m.cutoff)
        return {"pair": float(self.pair_energy(self.x, self.box, ij)), "bonded": float(self.bonded_energy(self.x, self.box)),
                "sphere": 0.0, "kinetic": float(0.5 * self.v.square().sum())}

    def adjoint(self, steps, every):
        """dJ/d(Umin, kbond, kbend) by automatic differentiation, segment by segment."""
        m = self.m
        rows = torch.zeros(len(self.u), 1, dtype=torch.float64, device=self.dev)
        rows[TAIL * m.n_types + TAIL] = 1.0
        r0, rc = self.u[TAIL * m.n_types + TAIL, 0], self.u[TAIL * m.n_types + TAIL, 3]
        w = rc - r0
        slope = torch.stack([0 * w, -1 / (r0 * r0), 1 + 0 * w, 0 * w, 3 / (w * w), 2 / (w * w * w)])
        th = torch.zeros(3, dtype=torch.float64, device=self.dev, requires_grad=True)
        u = self.u + rows * slope * th[0]
        k = self.k + th[1] * torch.tensor([0., 1, 0, 0], dtype=torch.float64, device=self.dev) + \
            th[2] * torch.tensor([0., 0, 0, 1], dtype=torch.float64, device=self.dev)
        total, grad = 0.0, torch.zeros(3, dtype=torch.float64, device=self.dev)
        for base in range(0, steps, every):
            x, h, seg = self.x.detach().requires_grad_(True), self.v.detach(), 0.0
            for _ in range(min(every, steps - base)):
                ij = self.pairs(x.detach(), self.box, m.cutoff)
                e = self.pair_energy(x, self.box, ij, u) + self.bonded_energy(x, self.box, k)
                f = -torch.autograd.grad(e, x, create_graph=True)[0]
                seg = seg + e / steps
                h = (1.0 - m.gamma * m.dt) * h + m.dt * f + m.dt * self.noise(self.it)
                x = x + m.dt * h
                x = x - self.box * torch.floor(x.detach() / self.box)
                self.it += 1
            grad += torch.autograd.grad(seg, th, retain_graph=True)[0]
            total += float(seg)
            self.x, self.v = x.detach(), h.detach()
        return total, grad


def exact(case, seed):
    """The pass in FP64 torch operations: the pair and chain potentials and their gradients, the Langevin
    loop with its Philox draws and the barostat with its MT19937 draws.  None for the sphere systems."""
    if case["shape"] == "sphere":
        return None
    sys_ = [_Exact(m) for m in _membranes(case, seed)]
    e, kind = sys_[0], case["kind"]

    def host(a):
        return torch.cat(a).cpu().numpy()

    if kind == "static":
        return {"force": e.force(pair_only=True).cpu().numpy()}
    if kind == "frame":
        return {"force": e.force().cpu().numpy(), "energy": [e.energy()]}
    for q in sys_:
        q.start()
    if kind == "adjoint":
        j, g = e.adjoint(case["steps"], 20)
        return {"pos": host([e.x]), "vel": host([e.v]), "mean_potential": j, "grad": g.cpu().numpy()}
    for q in sys_:
        for _ in range(LEAD_IN + case["steps"] - (1 if kind == "measure" else 0)):
            q.step()
    if kind == "run":
        return {"pos": host([q.x for q in sys_]), "vel": host([q.v for q in sys_]),
                "box": np.stack([q.box.cpu().numpy() for q in sys_])}
    e.step(stop=True)
    en = e.energy()
    return {"pos": host([e.x]), "vel": host([e.v]), "box": e.box.cpu().numpy(), "energy": en, "kinetic": en["kinetic"],
            "lo": e.x.min(0).values.cpu().numpy(), "hi": e.x.max(0).values.cpu().numpy()}
