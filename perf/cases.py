"""Performance cases: what a user of this framework has it do, at the sizes it is used at.

Kinds of case (each through the entry points a program calls: the Python front ends over the C ABI of include/mdg.h, with
device buffers where the caller's data live on the device):

  md       steps of one periodic Lennard-Jones box: MDManager.calculate, the observers, the state read into device arrays.  A pass
           goes on from where the last one stopped, as a simulation does: list rebuilds and re-selections come as they come.
  batch    steps of many independent replica boxes of uneven size, density and temperature, then observers and state.
  adjoint  gradient of a trajectory-averaged potential energy or pressure: forward and backward pass.
  forces   forces of positions that a program outside hands over (its own integrator, a relaxation): state in, list, forces out.
  observe  energy and virial of a caller's own device arrays, without a handle (mdg_observe_noalloc).

`exact` integrates the same inputs in plain torch in 64 bits, with its own neighbour search.
"""
import ctypes
import math

import numpy as np
import torch

from mdacp_gb300 import native
from mdacp_gb300.adjoint import Adjoint
from mdacp_gb300.batch import Batch
from mdacp_gb300.manager import MDManager


def _md(name, cells, density, precision, steps, **kw):
    c = dict(name=name, kind="md", n=4 * cells ** 3, cells=cells, density=density, aspect=1.0, precision=precision, steps=steps,
             single_calls=False, thermostat="nve", dt=0.001, cutoff=2.5, margin=0.5, temperature=1.0, policy="halfmargin")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest boxes: teaching runs and unit tests of a program's own, stepped one call at a time as the reference's projects do
        _md("fp64 864 atoms, single steps", 6, 0.8, "fp64", 50, single_calls=True),
        # the ordinary drop-in run: 32,000 atoms in the reference's precision, observed every 100 steps
        _md("fp64 32k atoms", 20, 0.5, "fp64", 100),
        # a thermostatted run of ordinary size, mixed form, larger time step
        _md("mixed langevin 108k atoms", 30, 0.5, "mixed", 100, thermostat="langevin", dt=0.005, temperature=0.9),
        # parity runs against the reference: its own rebuild policy and thermostat, 256k atoms, dense
        _md("fp64 nose-hoover 256k atoms", 40, 0.8, "fp64", 20, thermostat="nosehoover", policy="reference"),
        # a ragged system: odd particle count with vacancies in an oblong box, plain mixed form, the default cut-off and margin
        _md("mixed_plain ragged 1M atoms", 64, 0.7, "mixed_plain", 20, n=1000003, aspect=1.37, cutoff=3.0, margin=0.3),
        # the large runs: 4,000,000 atoms in both forms, and the largest, 16.4M atoms with the Langevin heat bath
        _md("mixed 4M atoms", 100, 0.5, "mixed", 20),
        _md("fp64 4M atoms", 100, 0.5, "fp64", 10),
        _md("mixed langevin 16.4M atoms", 160, 0.5, "mixed", 10, thermostat="langevin", dt=0.005, temperature=0.9),
        # replica ensembles in the fast form and in double precision
        dict(name="batch mixed 256 boxes", kind="batch", boxes=256, n_min=500, n_max=8000, precision="mixed", steps=100, dt=0.002,
             cutoff=2.5, margin=0.4),
        dict(name="batch fp64 48 boxes", kind="batch", boxes=48, n_min=500, n_max=8000, precision="fp64", steps=100, dt=0.002,
             cutoff=2.5, margin=0.4),
        # parameter fitting: gradient of a 200-step average, checkpoint every 20
        dict(name="adjoint 4000 atoms", kind="adjoint", n=4000, cells=10, density=0.8, steps=200, every=20, objective="pe", dt=0.002,
             margin=0.5, temperature=1.0),
        # an outside integrator's force call
        dict(name="forces fp64 131k atoms", kind="forces", n=131072, cells=32, density=0.7, aspect=1.0, precision="fp64", cutoff=2.5,
             margin=0.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["md", "batch", "adjoint", "forces", "observe"], [8, 2, 1, 1, 1])[0]
    density = round(rng.uniform(0.3, 0.9), 3)
    if kind == "md":
        precision = rng.choice(["fp64", "mixed", "mixed_plain"])
        n = _log_int(rng, 600, 2500000 if precision == "fp64" else 6000000)
        c = _md("", _cells(n), density, precision, max(10, min(100, 15000000 // n)), n=n,
                aspect=rng.choice([1.0, 1.0, 1.2]), single_calls=n < 20000 and rng.random() < 0.5, thermostat=rng.choice(["nve", "nve", "langevin", "nosehoover"]), dt=rng.choice([0.001, 0.002, 0.005]),
                temperature=round(rng.uniform(0.7, 1.5), 3), policy=rng.choice(["halfmargin"] * 4 + ["reference"]))
        c["cutoff"], c["margin"] = rng.choice([(2.5, 0.5), (2.5, 0.3), (3.0, 0.3)])
        del c["name"]
        return c
    if kind == "batch":
        precision = rng.choice(["fp64", "mixed"])
        n_min = rng.randint(500, 2000)
        return dict(kind=kind, boxes=_log_int(rng, 4, 48 if precision == "fp64" else 300), n_min=n_min,
                    n_max=rng.randint(n_min, 8000), precision=precision, steps=rng.randint(20, 100), dt=rng.choice([0.001, 0.002]),
                    cutoff=2.5, margin=rng.choice([0.3, 0.4, 0.5]))
    if kind == "adjoint":
        n, every = _log_int(rng, 700, 8000), rng.choice([10, 20])
        return dict(kind=kind, n=n, cells=_cells(n), density=round(rng.uniform(0.5, 0.85), 3), steps=rng.randint(20, 100), every=every,
                    objective=rng.choice(["pe", "pressure"]), dt=rng.choice([0.001, 0.002]), margin=0.5,
                    temperature=round(rng.uniform(0.7, 1.2), 3))
    n = _log_int(rng, 1000, 600000)
    c = dict(kind=kind, n=n, cells=_cells(n), density=density, aspect=rng.choice([1.0, 1.2]))
    if kind == "forces":
        c.update(precision=rng.choice(["fp64", "mixed"]), cutoff=2.5, margin=rng.choice([0.3, 0.5]))
    else:
        c.update(cutoff=rng.choice([2.5, 3.0]), temperature=round(rng.uniform(0.7, 1.5), 3))
    return c


def _cells(n):
    """FCC cells per side that hold n atoms."""
    c = max(1, round((n / 4.0) ** (1.0 / 3.0)) - 1)
    while 4 * c ** 3 < n:
        c += 1
    return c


# ---------------------------------------------------------------- inputs


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _lattice(c, g):
    """(positions [n, 4], box [3]) on the device: n sites of an FCC lattice, chosen at random where there are more, each displaced
    as a thermal crystal's or fresh liquid's atoms are, wrapped into the box.  The box has the case's density."""
    n, cells, aspect = c["n"], c["cells"], c.get("aspect", 1.0)
    volume = n / c["density"]
    side = (volume / aspect) ** (1.0 / 3.0)
    box = torch.tensor([side, side, side * aspect], dtype=torch.float64)
    k = torch.arange(cells, device="cuda", dtype=torch.float64)
    z, y, x = torch.meshgrid(k, k, k, indexing="ij")
    base = torch.stack([x, y, z], -1).reshape(-1, 1, 3)
    basis = torch.tensor([[0, 0, 0], [0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]], dtype=torch.float64, device="cuda")
    q = (base + basis).reshape(-1, 3)
    if len(q) > n:
        q = q[torch.randperm(len(q), generator=g, device="cuda")[:n].sort().values]
    a = box.cuda() / cells
    nearest = float(a.min()) / math.sqrt(2.0)
    q = (q + 0.25) * a + (torch.rand(q.shape, generator=g, device="cuda", dtype=torch.float64) - 0.5) * (0.14 * nearest)
    out = torch.zeros((n, 4), device="cuda", dtype=torch.float64)
    out[:, :3] = torch.remainder(q, box.cuda())
    return out, box.numpy()


def _velocities(n, temperature, g):
    p = torch.zeros((n, 4), device="cuda", dtype=torch.float64)
    v = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64) * math.sqrt(temperature)
    p[:, :3] = v - v.mean(0)
    return p


def _replicas(c, seed):
    """[(q, p, box)] on the host: sizes spread evenly over their range (in a mixed order), densities and temperatures uniform."""
    g = _generator(seed)
    u = torch.rand((c["boxes"], 2), generator=g, device="cuda", dtype=torch.float64).cpu().numpy()
    out = []
    for k, (b, t) in enumerate(u):
        n = int(c["n_min"] + (0.5 + 0.6180339887498949 * k) % 1.0 * (c["n_max"] - c["n_min"]))
        q, box = _lattice(dict(n=n, cells=_cells(n), density=0.3 + 0.6 * b), g)
        p = _velocities(n, 0.7 + 0.8 * t, g)
        out.append((q[:, :3].cpu().numpy(), p[:, :3].cpu().numpy(), box))
    return out


def _pointer(t):
    return ctypes.c_void_p(t.data_ptr())


def _doubles(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _host(n):
    """A pinned host array, as a program that reads its state often keeps one."""
    return torch.zeros((n, 4), dtype=torch.float64, pin_memory=True).numpy()


def _md_inputs(c, seed):
    g = _generator(seed)
    q, box = _lattice(c, g)
    return q, _velocities(c["n"], c["temperature"], g), box


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        boxes = _replicas(case, seed)
        b = Batch(boxes, cutoff=case["cutoff"], margin=case["margin"], dt=case["dt"], precision=case["precision"])
        # the shape that the autotuner picks for such ensembles, fixed so that every run has the same one
        b.set_shape(256, 1, 4)
        b.set_flat(True)
        total = int(b.offsets[-1])
        return dict(kind=kind, steps=case["steps"], batch=b, q=_host(total), p=_host(total))
    if kind == "adjoint":
        q, p, box = _md_inputs(case, seed)
        a = Adjoint(box, case["n"], steps=case["steps"], checkpoint_every=case["every"], dt=case["dt"], cutoff=2.5,
                    margin=case["margin"], objective=case["objective"])
        return dict(kind=kind, adjoint=a, q=q[:, :3].cpu().numpy(), p=p[:, :3].cpu().numpy())
    if kind == "observe":
        q, p, box = _md_inputs(case, seed)
        return dict(kind=kind, lib=native.load(), q=q, p=p, box=np.ascontiguousarray(box), cutoff=case["cutoff"],
                    out=torch.zeros(3, device="cuda", dtype=torch.float64))
    if kind == "forces":
        q, box = _lattice(case, _generator(seed))
        m = MDManager(box, capacity=case["n"], cutoff=case["cutoff"], margin=case["margin"], precision=case["precision"])
        torch.cuda.synchronize()
        m.n = case["n"]
        return dict(kind=kind, manager=m, q=q, p=torch.zeros_like(q))
    q, p, box = _md_inputs(case, seed)
    m = MDManager(box, capacity=case["n"], cutoff=case["cutoff"], margin=case["margin"], dt=case["dt"], precision=case["precision"],
                  thermostat=case["thermostat"], temperature=case["temperature"], gamma=1.0, tau=0.1, seed=_noise_seed(seed),
                  rebuild_policy=case["policy"])
    torch.cuda.synchronize()
    native.check(m.lib.mdg_set_state_device(m._h, _pointer(q), _pointer(p), case["n"]), m._h)
    m.n = case["n"]
    m.make_pairlist()
    return dict(kind=kind, manager=m, steps=case["steps"], single_calls=case["single_calls"], q=q, p=p)


def _noise_seed(seed):
    return 1 + int(seed) % 1000003


def run(state):
    kind = state["kind"]
    if kind == "md":
        m = state["manager"]
        if state["single_calls"]:
            for _ in range(state["steps"]):
                m.calculate(1)
        else:
            m.calculate(state["steps"])
        native.check(m.lib.mdg_get_state_device(m._h, _pointer(state["q"]), _pointer(state["p"])), m._h)
        return {"q": state["q"], "p": state["p"], "sums": m.observe_raw()}
    if kind == "batch":
        b = state["batch"]
        b.calculate(state["steps"])
        sums = b.observe_raw()
        b._ck(b.lib.mdg_batch_get_state(b._h, _doubles(state["q"]), _doubles(state["p"])))
        return {"q": state["q"], "p": state["p"], "sums": sums}
    if kind == "adjoint":
        value = state["adjoint"].forward(state["q"], state["p"])
        dq, dp, de, ds = state["adjoint"].backward()
        return {"value": value, "dq": dq, "dp": dp, "depsilon": de, "dsigma": ds}
    if kind == "forces":
        m = state["manager"]
        native.check(m.lib.mdg_set_state_device(m._h, _pointer(state["q"]), _pointer(state["p"]), m.n), m._h)
        return {"f": m.forces()}
    native.check(state["lib"].mdg_observe_noalloc(_pointer(state["q"]), _pointer(state["p"]), len(state["q"]), _doubles(state["box"]),
                                                  state["cutoff"], _pointer(state["out"]),
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"sums": state["out"]}


def work(case):
    """Bytes: positions and momenta, three doubles each, read and written once a step (a force call: positions in, forces out).
    Operations: each pair within the cut-off once, 23 for separation, distance, force factor and the two sums."""
    kind = case["kind"]
    cutoff = case.get("cutoff", 2.5)
    if kind == "batch":
        n, density = case["boxes"] * (case["n_min"] + case["n_max"]) / 2, 0.6
    else:
        n, density = case["n"], case["density"]
    pairs = n * density * 4.0 / 3.0 * math.pi * cutoff ** 3 / 2
    if kind == "observe":
        return {"bytes": 48.0 * n, "flops": 20.0 * pairs}
    if kind == "forces":
        return {"bytes": 48.0 * n, "flops": 23.0 * pairs}
    if kind == "adjoint":  # forward step with its objective, recomputed step, Hessian-vector product with the objective's gradient
        return {"bytes": 3 * 96.0 * n * case["steps"], "flops": 120.0 * pairs * case["steps"]}
    return {"bytes": 96.0 * n * case["steps"], "flops": 23.0 * pairs * case["steps"]}


# ---------------------------------------------------------------- the same in plain torch, 64 bits


def _pairs(q, box_of, L, reach):
    """Half list (i, j, shift [k, 3]) of every image pair within `reach`: boxes side by side, cells at least `reach` wide."""
    nc = torch.floor(L / reach).long().clamp(min=2)
    first = torch.cat([torch.zeros(1, dtype=torch.long, device=q.device), nc.prod(1).cumsum(0)])
    Lq, ncq = L[box_of], nc[box_of]
    cell = torch.minimum(torch.clamp(torch.floor(q / Lq * ncq).long(), min=0), ncq - 1)
    flat = first[box_of] + (cell[:, 2] * ncq[:, 1] + cell[:, 1]) * ncq[:, 0] + cell[:, 0]
    order = torch.argsort(flat)
    count = torch.bincount(flat, minlength=int(first[-1]))
    start = torch.cat([torch.zeros(1, dtype=torch.long, device=q.device), count.cumsum(0)])
    got = []
    for code in range(14):
        off = torch.tensor([code % 3 - 1, code // 3 % 3 - 1, code // 9 - 1], device=q.device)
        other = cell + off
        wrap = torch.where(other < 0, -1, 0) + torch.where(other >= ncq, 1, 0)
        other = other - wrap * ncq
        target = first[box_of] + (other[:, 2] * ncq[:, 1] + other[:, 1]) * ncq[:, 0] + other[:, 0]
        many = count[target]
        i = torch.repeat_interleave(torch.arange(len(q), device=q.device), many)
        k = torch.arange(len(i), device=q.device) - torch.repeat_interleave(many.cumsum(0) - many, many)
        j = order[start[target][i] + k]
        shift = (wrap.double() * Lq)[i]
        near = ((q[j] + shift - q[i]) ** 2).sum(1) <= reach * reach
        if code == 13:  # the cell itself: each pair once
            near &= i < j
        got.append((i[near], j[near], shift[near]))
    return tuple(torch.cat(x) for x in zip(*got))


class _Exact:
    """Drift-kick-drift of the smoothly truncated Lennard-Jones potential in 64 bits; boxes side by side."""

    def __init__(self, q, p, box_of, L, cutoff, dt):
        self.q, self.p, self.box_of, self.L, self.rc, self.dt = q, p, box_of, L, cutoff, dt
        s2 = 1.0 / cutoff ** 2
        self.c2 = 6 * s2 ** 7 - 3 * s2 ** 4
        self.c0 = -s2 ** 6 + s2 ** 3 - self.c2 / s2
        self.listed, self.at = None, None

    def _list(self, q):
        skin = 0.4
        if self.listed is None or float(((q - self.at) ** 2).sum(1).max()) > (0.5 * skin) ** 2:
            # the pairs of the wrapped positions, their shifts taken back to the positions at hand
            Lq = self.L[self.box_of]
            turns = torch.floor(q / Lq)
            i, j, shift = _pairs(q - turns * Lq, self.box_of, self.L, self.rc + skin)
            self.listed, self.at = (i, j, shift - ((turns * Lq)[j] - (turns * Lq)[i])), q.clone()
        return self.listed

    def _near(self, q):
        i, j, shift = self._list(q)
        d = q[j] + shift - q[i]
        r2 = (d * d).sum(1)
        near = r2 <= self.rc ** 2
        return i[near], j[near], d[near], r2[near]

    def forces(self, q):
        i, j, d, r2 = self._near(q)
        r6 = r2 * r2 * r2
        f = (((24 * r6 - 48) / (r6 * r6 * r2)) + 8 * self.c2)[:, None] * d
        return torch.zeros_like(q).index_add_(0, i, f).index_add_(0, j, -f)

    def step(self, noise=None, gamma=1.0):
        q = self.q + self.p * (0.5 * self.dt)
        p = self.p + self.forces(q) * self.dt
        if noise is not None:  # the heat bath, without the second half-drift
            self.p, self.q = p + (-gamma * p + noise) * self.dt, q
            return
        self.q, self.p = q + p * (0.5 * self.dt), p

    def step_nose_hoover(self, zeta, temperature, tau):
        h = 0.5 * self.dt
        instant = lambda: float((self.p * self.p).sum()) / (3.0 * len(self.p))  # noqa: E731
        zeta = zeta + (instant() - temperature) / tau ** 2 * h
        q = self.q + self.p * h
        e = math.exp(-h * zeta)
        self.p = (self.p * e + self.forces(q) * self.dt) * e
        self.q = q + self.p * h
        return zeta + (instant() - temperature) / tau ** 2 * h

    def sums(self):
        i, j, d, r2 = self._near(self.q)
        r6 = r2 * r2 * r2
        energy = 4 * (1 / (r6 * r6) - 1 / r6 + self.c2 * r2 + self.c0)
        virial = ((24 * r6 - 48) / (r6 * r6 * r2) + 8 * self.c2) * r2
        of = self.box_of[i]
        out = torch.zeros((len(self.L), 3), dtype=torch.float64, device=self.q.device)
        out[:, 0].index_add_(0, self.box_of, 0.5 * (self.p * self.p).sum(1))
        out[:, 1].index_add_(0, of, energy)
        out[:, 2].index_add_(0, of, virial / 3)
        return out


def _noise(n, seed, step, scale):
    """The Langevin stream: Philox4x32-10 of (particle, step) under the seed, Box-Muller."""
    mask = 0xFFFFFFFF
    c = [torch.arange(n, device="cuda", dtype=torch.int64), torch.full((n,), step & mask, device="cuda"),
         torch.full((n,), step >> 32, device="cuda"), torch.full((n,), 0x4C4A4D44, device="cuda")]
    k0, k1 = seed & mask, seed >> 32

    def product(a, b):  # 32 x 32 bits in two halves, inside 63 bits
        lo = a * (b & 0xFFFF)
        hi = a * (b >> 16) + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        h0, l0 = product(c[0], 0xD2511F53)
        h1, l1 = product(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    u = [((c[k] >> 8) + (1 - k % 2)).double() / 2 ** 24 for k in range(4)]
    a, b = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    w = 2 * math.pi
    return torch.stack([a * torch.cos(w * u[1]), a * torch.sin(w * u[1]), b * torch.cos(w * u[3])], 1) * scale


def _four(x):
    return torch.cat([x, torch.zeros_like(x[:, :1])], 1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind == "batch":
        boxes = _replicas(case, seed)
        q, p = (torch.cat([torch.from_numpy(b[k]) for b in boxes]).cuda() for k in (0, 1))
        of = torch.repeat_interleave(torch.arange(len(boxes)), torch.tensor([len(b[0]) for b in boxes])).cuda()
        e = _Exact(q, p, of, torch.from_numpy(np.array([b[2] for b in boxes])).cuda(), case["cutoff"], case["dt"])
        for _ in range(case["steps"]):
            e.step()
        # positions come back wrapped where the engine's last rebuild left them: no value of their own here
        return {"q": None, "p": _four(e.p).cpu().numpy(), "sums": e.sums().cpu().numpy()}
    if case["n"] > 5000000:
        return None
    if kind == "forces":
        q, box = _lattice(case, _generator(seed))
        p = torch.zeros_like(q)
    else:
        q, p, box = _md_inputs(case, seed)
    q, p = q[:, :3].clone(), p[:, :3].clone()
    of = torch.zeros(len(q), dtype=torch.long, device="cuda")
    e = _Exact(q, p, of, torch.from_numpy(box).cuda()[None], case["cutoff"], case.get("dt", 0.001))
    if kind == "forces":
        return {"f": e.forces(q).cpu().numpy()}
    if kind == "observe":
        return {"sums": e.sums()[0]}
    zeta, moved = 0.0, 0.0
    for k in range(case["steps"]):
        if case["thermostat"] == "nosehoover":
            zeta = e.step_nose_hoover(zeta, case["temperature"], 0.1)
        elif case["thermostat"] == "langevin":
            e.step(_noise(len(q), _noise_seed(seed), k, math.sqrt(2 * case["temperature"] / case["dt"])))
        else:
            e.step()
        moved = max(moved, float(((e.q + e.p * (0.5 * case["dt"]) - q) ** 2).sum(1).max()))
    # no rebuild yet: the positions are still in the images they were given in
    still = moved < (0.49 * case["margin"]) ** 2 and case["policy"] == "halfmargin"
    return {"q": _four(e.q) if still else None, "p": _four(e.p), "sums": e.sums()[0].cpu().numpy()}


def _exact_adjoint(case, seed):
    """The gradient by torch's own differentiation through every step."""
    q, p, box = _md_inputs(case, seed)
    of = torch.zeros(len(q), dtype=torch.long, device="cuda")
    L = torch.from_numpy(box).cuda()[None]
    q0 = q[:, :3].clone().requires_grad_()
    p0 = p[:, :3].clone().requires_grad_()
    eps = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
    sig = torch.ones((), dtype=torch.float64, device="cuda", requires_grad=True)
    finder = _Exact(q0.detach(), p0.detach(), of, L, 2.5, case["dt"])
    dt, n, volume = case["dt"], case["n"], float(L.prod())

    def reduced(x):
        i, j, shift = finder._list(x.detach())
        d = x[j] + shift - x[i]
        x2 = (d * d).sum(1) / sig ** 2
        near = x2.detach() <= 2.5 ** 2
        return i[near], j[near], d[near], x2[near]

    def psi(x2):
        x6 = x2 * x2 * x2
        return (24 * x6 - 48) / (x6 * x6 * x2) + 8 * finder.c2

    total, x, v = 0.0, q0, p0
    for _ in range(case["steps"]):
        h = x + v * (0.5 * dt)
        i, j, d, x2 = reduced(h)
        f = (eps / sig ** 2 * psi(x2))[:, None] * d
        v = v + torch.zeros_like(v).index_add(0, i, f).index_add(0, j, -f) * dt
        x = h + v * (0.5 * dt)
        i, j, d, x2 = reduced(x)
        if case["objective"] == "pe":
            x6 = x2 * x2 * x2
            total = total + (4 * eps * (1 / (x6 * x6) - 1 / x6 + finder.c2 * x2 + finder.c0)).sum() / n
        else:
            total = total + ((v * v).sum() - (eps * psi(x2) * x2).sum()) / (3 * volume)
    total = total / case["steps"]
    dq, dp, de, ds = torch.autograd.grad(total, (q0, p0, eps, sig))
    return {"value": float(total), "dq": dq.cpu().numpy(), "dp": dp.cpu().numpy(), "depsilon": float(de), "dsigma": float(ds)}
