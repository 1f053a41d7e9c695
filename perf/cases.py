"""The work a program has the library do, as a list of timed cases.

A case names a set-up (grid, grains, options) and one pass of a user's loop over it:

  steps     restore the saved start state, run a number of time steps, read the state on the device
  loop      the same with one call per step and the grain volumes read after each (the reference's
            own time loop: step, then per-step output)
  host      a whole job from host memory: upload the lists, finalize, per step a driving-force
            upload, a step and the grain volumes, then the lists back to the host
  adjoint   one iteration of a calibration: set the parameters, roll forward, sweep backward
  tangent   a directional derivative of the grain volumes (tangent-linear model)

Initial states are seeded Voronoi grains with spread boundaries, or spherical nuclei in a matrix,
relaxed by a few steps where a pass starts from a saved state.  `exact` restates the step in plain
torch in 64 bits, with the discrete decisions of the model and the arithmetic in an order of its own.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from openphase_b200.adjoint import Rollout
from openphase_b200.context import Context

PI = 3.14159265358979323846
EPS = float(np.finfo(np.float64).eps)
ROOM = 3   # entries per voxel the host job has room for

BASE = {
    "kind": "steps", "nx": 64, "ny": 64, "nz": 64, "grains": 32, "steps": 10, "relax": 10, "precision": "fp64",
    "k": 16, "stencil": "LB", "iwidth": 5.0, "dt": 0.08, "pairs": "phase", "dg": 0.0, "average": False,
    "nuclei": 0.0, "interval": 4,
}


def _case(name, **kw):
    return {"name": name, **BASE, **kw}


def listed():
    dg = {"pairs": "table", "dg": 0.05, "iwidth": 6.0}
    return [
        # the smallest runs: a test problem stepped one call at a time, latency and launches count
        _case("loop_small", kind="loop", nx=40, ny=36, nz=44, grains=10, k=8, stencil="ISOTROPIC", dt=0.1),
        # normal grain growth as the reference's example runs it
        _case("growth_64", nx=64, ny=64, nz=64, grains=32, steps=25, dt=0.1),
        # the grain-growth benchmark with driving force, scaled to 128^3 at the same grain size
        _case("growth_dg_128", nx=128, ny=128, nz=128, grains=250, steps=10, **dg),
        # the benchmark itself in both forms: the largest runs
        _case("growth_dg_256", nx=256, ny=256, nz=256, grains=2000, steps=10, **dg),
        _case("growth_dg_256_fp32", nx=256, ny=256, nz=256, grains=2000, steps=10, precision="fp32", **dg),
        # a ragged box, the 7-point Laplacian, pair energies generated on the device
        _case("ragged_simple", nx=150, ny=97, nz=203, grains=180, steps=8, k=12, stencil="SIMPLE", pairs="hash",
              dg=0.03, iwidth=5.5, precision="fp32"),
        # a whole job from and to host memory
        _case("host_job_128", kind="host", nx=128, ny=128, nz=128, grains=250, steps=10, relax=0, **dg),
        # two-phase solidification with cubic anisotropy
        _case("solidification_128", nx=128, ny=128, nz=128, grains=65, steps=10, nuclei=6.0, dt=0.05),
        # the reference's default: driving forces averaged across the interface
        _case("averaged_96", nx=96, ny=96, nz=96, grains=105, steps=4, average=True, **dg),
        # the calibration rollout with its adjoint in both forms, shortened
        _case("adjoint_128_fp32", kind="adjoint", nx=128, ny=128, nz=128, grains=256, steps=12, relax=5,
              precision="fp32", pairs="table", dg=0.03),
        _case("adjoint_56", kind="adjoint", nx=56, ny=60, nz=50, grains=24, steps=8, relax=5, pairs="table", dg=0.03),
        # a directional derivative of the final grain volumes
        _case("tangent_64", kind="tangent", nx=64, ny=64, nz=64, grains=32, steps=8, relax=5, pairs="table", dg=0.03),
    ]


def draw(rng):
    kind = rng.choice(("steps", "steps", "steps", "loop", "host", "solid", "average", "adjoint", "tangent"))
    top = {"steps": 256, "loop": 80, "host": 128, "solid": 128, "average": 96, "adjoint": 112, "tangent": 72}[kind]
    side = math.exp(rng.uniform(math.log(30), math.log(top)))
    ax, ay = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    dims = [max(24, round(side * f)) for f in (ax, ay, 1.0 / (ax * ay))]
    while dims[0] * dims[1] * dims[2] > top ** 3:
        dims[dims.index(max(dims))] -= 1
    n = dims[0] * dims[1] * dims[2]
    c = {**BASE, "nx": dims[0], "ny": dims[1], "nz": dims[2], "kind": kind if kind in ("loop", "host", "adjoint", "tangent") else "steps"}
    c["grains"] = max(6, min(4000, round(n / math.exp(rng.uniform(math.log(4000), math.log(20000))))))
    c["iwidth"] = rng.choice((4.5, 5.0, 5.5, 6.0))
    c["precision"] = "fp64" if kind in ("host", "tangent") else rng.choice(("fp64", "fp32"))
    c["stencil"] = rng.choice(("LB", "LB", "ISOTROPIC", "SIMPLE"))
    c["k"] = rng.choice((12, 16))
    c["pairs"] = rng.choice(("phase", "table", "hash"))
    c["dg"] = rng.choice((0.0, 0.03, 0.05))
    c["steps"] = rng.randint(4, 10)
    if kind in ("host", "average", "adjoint", "tangent"):
        c["dg"] = c["dg"] or 0.04
    if kind == "solid":
        c.update(nuclei=round(rng.uniform(4.0, 8.0), 2), grains=1 + max(4, min(100, n // 30000)), dt=0.05, pairs="phase", dg=0.0,
                 iwidth=5.0, stencil=rng.choice(("LB", "ISOTROPIC")))
    if kind == "average":
        c.update(average=True, steps=rng.randint(1, 4))
    if kind in ("adjoint", "tangent"):
        c.update(pairs="table", relax=5)
    if kind == "host":
        c.update(relax=0)
    return c


# ---- inputs ---------------------------------------------------------------------------------------

def _spread(owner):
    """Ragged lists of an owner map: every voxel lists its own grain first, then each other grain
    among its 26 neighbours, all with value 1 (finalize normalises)."""
    n, cap = owner.numel(), 16
    flat = owner.reshape(-1)
    lists = torch.full((cap, n), -1, dtype=torch.int32, device=owner.device)
    lists[0] = flat
    count = torch.ones(n, dtype=torch.int64, device=owner.device)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                g = torch.roll(owner, (-dx, -dy, -dz), (0, 1, 2)).reshape(-1)
                at = torch.nonzero(g != flat).reshape(-1)   # only next to another grain
                g = g[at]
                at = at[~(lists[:, at] == g).any(0)]
                g = torch.roll(owner, (-dx, -dy, -dz), (0, 1, 2)).reshape(-1)[at]
                lists[count[at], at] = g
                count[at] += 1
    keep = lists.t() >= 0
    idx = lists.t()[keep]
    return count.int().cpu().numpy(), idx.cpu().numpy(), np.ones(idx.numel())


def _voronoi(c, rng):
    """Owner map: the nearest of uniformly drawn seeds under the periodic distance, ties to the lower index."""
    dims, G = (c["nx"], c["ny"], c["nz"]), c["grains"]
    d2 = []
    for n in dims:
        d = torch.remainder(torch.arange(n).reshape(-1, 1) - torch.from_numpy(rng.integers(0, n, G)).reshape(1, -1), n)
        d = torch.minimum(d, n - d)
        d2.append((d * d).to(torch.int64).cuda())
    key = torch.arange(G, device="cuda", dtype=torch.int64)
    owner = torch.empty(dims, dtype=torch.int32, device="cuda")
    bits = 1 << max(1, (G - 1).bit_length())
    small = bits * sum(n * n // 4 for n in dims) < 2 ** 31
    kind = torch.int32 if small else torch.int64
    a, b, z = ((d * bits).to(kind) for d in d2)
    z = z + key.to(kind)
    rows = max(1, 400_000_000 // (dims[2] * G * (4 if small else 8)))
    for x in range(dims[0]):
        for y in range(0, dims[1], rows):
            best = (a[x] + b[y:y + rows]).unsqueeze(1) + z.unsqueeze(0)
            owner[x, y:y + rows] = (best.amin(-1) % bits).int()
    return owner


def _nuclei(c, rng):
    """Grain 0 with spheres of grains 1.. in it, each with the sine profile of the interface."""
    dims, G, R, w = (c["nx"], c["ny"], c["nz"]), c["grains"], c["nuclei"], c["iwidth"]
    n = dims[0] * dims[1] * dims[2]
    gs, vs = np.full((n, 8), -1, np.int32), np.zeros((n, 8))
    gs[:, 0], vs[:, 0] = 0, 1.0
    reach = int(math.ceil(R + 0.5 * w)) + 1
    for g in range(1, G):
        centre = rng.random(3) * dims
        axes, dist = [], []
        for m, x in zip(dims, centre):
            i = np.unique(np.arange(int(x) - reach, int(x) + reach + 2) % m)
            d = np.abs(i - x)
            axes.append(i)
            dist.append(np.minimum(d, m - d) ** 2)
        v = ((axes[0][:, None, None] * dims[1] + axes[1][None, :, None]) * dims[2] + axes[2][None, None, :]).ravel()
        r = np.sqrt(dist[0][:, None, None] + dist[1][None, :, None] + dist[2][None, None, :]).ravel()
        core, shell = v[r < R - 0.5 * w], (r >= R - 0.5 * w) & (r <= R + 0.5 * w)
        gs[core], vs[core] = -1, 0.0
        gs[core, 0], vs[core, 0] = g, 1.0
        p = 0.5 - 0.5 * np.sin(PI * (r[shell] - R) / w)
        v = v[shell]
        at = (gs[v] >= 0).sum(1)
        v, p, at = v[at < 8], p[at < 8], at[at < 8]
        vs[v] *= (1.0 - p)[:, None]
        gs[v, at], vs[v, at] = g, p
    keep = gs >= 0
    return keep.sum(1).astype(np.int32), gs[keep], vs[keep]


def _problem(c, seed):
    """Everything both `prepare` and `exact` need, in host memory, from the case and the seed alone."""
    rng = np.random.default_rng([seed, 11])
    G = c["grains"]
    P = {"phase": np.zeros(G, np.int32), "quat": None, "sigma_p": np.array([[1.2]]), "mu_p": np.array([[1.0]]),
         "solid": np.array([1], np.int32), "eps": None, "maxe": np.array([[1.2]]), "sigma": None, "dg": None}
    if c["nuclei"]:
        P["lists"] = _nuclei(c, rng)
        P["phase"][1:] = 1
        q = rng.standard_normal((G, 4))
        P["quat"] = q / np.linalg.norm(q, axis=1, keepdims=True)
        P["sigma_p"], P["mu_p"] = np.array([[1.0, 1.0], [1.0, 1.2]]), np.array([[2.0, 2.0], [2.0, 0.5]])
        P["solid"], P["eps"] = np.array([0, 1], np.int32), np.array([[0.0, 0.02], [0.02, 0.0]])
        P["maxe"] = P["sigma_p"] * (1.0 + 1.41 * P["eps"])
        P["dg"] = np.where(P["phase"] == 0, 0.1, 0.0)
    else:
        P["lists"] = _spread(_voronoi(c, rng))
    if c["pairs"] == "table":
        s = np.triu(rng.uniform(0.8, 1.2, (G, G)), 1)
        P["sigma"] = s + s.T + 0.8 * np.eye(G)
    if c["dg"]:
        P["dg"] = rng.uniform(0.0, c["dg"], G)
    if c["kind"] in ("adjoint", "tangent"):
        P["mu"] = np.ones((G, G))
        P["weight"] = rng.standard_normal(G)
        d = np.triu(rng.standard_normal((G, G)), 1)
        m = np.triu(rng.standard_normal((G, G)), 1)
        P["dsigma"], P["dmu"], P["ddg"] = 0.01 * (d + d.T), 0.01 * (m + m.T), 0.01 * rng.standard_normal(G)
    return P


def prepare(case, seed):
    P = _problem(case, seed)
    c = case
    ctx = Context(c["nx"], c["ny"], c["nz"], iwidth=c["iwidth"], stencil=c["stencil"], precision=c["precision"], k_slots=c["k"])
    aniso = P["eps"] is not None
    ctx.set_model(P["sigma_p"], P["mu_p"], limit=np.full(P["mu_p"].shape, 0.95), phase_solid=P["solid"],
                  energy_model=(P["eps"] != 0).astype(np.int32) if aniso else None, cubic_eps=P["eps"])
    ctx.set_grains(c["grains"], phase=P["phase"])
    if aniso:
        ctx.set_orientations(P["quat"])
    if c["pairs"] == "table":
        ctx.set_pair_table(P["sigma"], None)
    elif c["pairs"] == "hash":
        ctx.set_pair_hash(seed, 0.8, 0.4)
    ctx.set_driving_force(P["dg"])
    if c["average"]:
        ctx.set_averaging(True)
    s = {"case": c, "ctx": ctx, "P": P}
    if c["kind"] == "host":
        # pinned host memory for the lists, in and out
        pin = lambda a: torch.from_numpy(a).pin_memory().numpy()  # noqa: E731
        s["lists"] = [pin(a) for a in P["lists"]]
        room = ROOM * ctx.n
        s["out"] = [torch.zeros(k, dtype=t).pin_memory().numpy() for k, t in
                    ((ctx.n, torch.int32), (room, torch.int32), (room, torch.float64))]
        s["used"] = 0
        return s
    ctx.upload(*P["lists"])
    ctx.finalize_initialization()
    ctx.step(c["dt"], c["relax"])
    if c["kind"] in ("adjoint", "tangent"):
        s["rollout"] = Rollout(ctx, c["dt"], c["steps"], interval=c["interval"])
        return s
    ctx.checkpoint_reserve(1)
    ctx.checkpoint_save(0)
    ctx.set_stream_ordered(True)
    s["stream"] = torch.cuda.ExternalStream(ctx.stream)
    s["planes"] = torch.empty((c["nx"], ctx.plane_bytes()), dtype=torch.uint8, device="cuda")
    ctx.sync()
    return s


# ---- one pass -------------------------------------------------------------------------------------

def _read_state(s):
    """The state on the device, through the plane calls: per x-plane the counts, grains and values
    of the K slots, with the slots that hold nothing set to zero."""
    c, ctx, buf, stream = s["case"], s["ctx"], s["planes"], s["stream"]
    nx, k, m = c["nx"], c["k"], c["ny"] * c["nz"]
    stream.wait_stream(torch.cuda.current_stream())
    for x in range(nx):
        ctx.pack_plane(x, buf.data_ptr() + x * buf.stride(0))
    torch.cuda.current_stream().wait_stream(stream)
    count = buf[:, :m].clone()
    real = torch.float32 if c["precision"] == "fp32" else torch.float64
    grain = buf[:, m:m + 2 * k * m].clone().view(torch.int16).reshape(nx, k, m)
    value = buf[:, m + 2 * k * m:].clone().view(real).reshape(nx, k, m)
    empty = torch.arange(k, device="cuda", dtype=torch.uint8).reshape(1, k, 1) >= count.unsqueeze(1)
    return {"count": count, "grain": grain.masked_fill_(empty, 0), "value": value.masked_fill_(empty, 0)}


def run(state):
    s, c, ctx = state, state["case"], state["ctx"]
    if c["kind"] == "adjoint":
        R, P = s["rollout"], s["P"]
        R.set_parameters(P["sigma"], P["mu"], P["dg"])
        volume = R.forward()
        dsigma, dmu, ddg = R.backward(P["weight"])
        return {"volume": volume, "dsigma": dsigma, "dmu": dmu, "ddg": ddg}
    if c["kind"] == "tangent":
        R, P = s["rollout"], s["P"]
        R.set_parameters(P["sigma"], P["mu"], P["dg"])
        return {"dvolume": R.tangent(P["dsigma"], P["dmu"], P["ddg"])}
    if c["kind"] == "host":
        ctx.upload(*s["lists"])
        ctx.finalize_initialization()
        volumes = []
        for _ in range(c["steps"]):
            ctx.set_driving_force(s["P"]["dg"])
            ctx.step(c["dt"], 1)
            volumes.append(ctx.grains()["volume"])
        count, grain, value = s["out"]
        total = ctx.download(out=s["out"])[1].size
        grain[total:s["used"]], value[total:s["used"]] = 0, 0.0   # what a longer list left behind
        s["used"] = total
        return {"count": count, "grain": grain, "value": value, "volume": np.stack(volumes)}
    ctx.checkpoint_load(0)
    if c["kind"] == "loop":
        volumes = []
        for _ in range(c["steps"]):
            ctx.step(c["dt"], 1)
            volumes.append(ctx.grains()["volume"])
        volume = np.stack(volumes)
    else:
        ctx.step(c["dt"], c["steps"])
        volume = ctx.grains()["volume"]
    return {**_read_state(s), "volume": volume}


# ---- what a pass cannot do without ----------------------------------------------------------------

def work(case):
    """Per step every voxel's count and every stored field (index, value) is read and written once; a
    field costs its 27-point (7-point) Laplacian, a pair of a voxel's list its kinetics and
    projection.  Voronoi grains have 2.91 rho^(1/3) interface per volume, iwidth thick."""
    c = case
    n = c["nx"] * c["ny"] * c["nz"]
    size = 4 if c["precision"] == "fp32" else 8
    if c["nuclei"]:
        shell = 4.0 * PI * c["nuclei"] ** 2 * c["iwidth"] * (c["grains"] - 1) / n
    else:
        shell = 2.91 * (c["grains"] / n) ** (1.0 / 3.0) * c["iwidth"]
    wide = min(1.0, shell * (1.0 + 2.0 / c["iwidth"]))
    fields = 1.0 + 1.1 * min(1.0, shell)
    step_bytes = 2.0 * n * (1.0 + fields * (2 + size))
    step_flops = n * wide * (3.0 * 2 * (7 if c["stencil"] == "SIMPLE" else 27) + 3.0 * 40)
    passes = float(c["steps"])
    if c["kind"] == "adjoint":
        passes *= 2.0   # forward and reverse
    if c["kind"] == "tangent":
        passes *= 2.0   # the state and its tangent
    extra = 2.0 * n * fields * 12 if c["kind"] == "host" else 0.0   # the lists in and out
    return {"bytes": passes * step_bytes + extra, "flops": passes * step_flops}


def tolerance(case):
    """The model decides by thresholds (a field erased below DBL_EPSILON, list lengths that count
    candidates), so a sum in another order tips single voxels, by some 1e-3 a step each: against
    `exact` the states of ten steps are off by up to 4e-6 in 64 bits and 3e-5 in 32."""
    if case["precision"] == "fp32":
        return {"rel": 1e-4, "max": 0.1, "differ": 1e-3}
    return {"rel": 1e-5, "max": 0.05, "differ": 1e-4}


# ---- the same pass in plain torch, 64 bits --------------------------------------------------------

def _stencils(kind):
    """Laplacian offsets with their weights, then the offsets that only bring candidates (the
    isotropic gradient's), and the gradient weights, all in x, y, z order."""
    off = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]
    far = [sum(map(abs, o)) for o in off]
    w = {"SIMPLE": (-6.0, 1.0, 0.0, 0.0), "ISOTROPIC": (-64 / 15, 7 / 15, 0.1, 1 / 30), "LB": (-38 / 9, 4 / 9, 1 / 9, 1 / 36)}[kind]
    lap = [(o, w[f]) for o, f in zip(off, far) if w[f]]
    more = [o for o, f in zip(off, far) if f] if kind == "SIMPLE" else []
    gw = (0.0, 1 / 4.64, 0.245 / 4.64, 0.085 / 4.64)
    grad = [(o, [x * gw[f] for x in o]) for o, f in zip(off, far) if f]
    return lap, more, grad


class _Exact:
    """The model's step on padded lists (g [N, K] with -1 for empty, v [N, K]) in double precision."""

    def __init__(self, c, P, seed):
        self.c, self.dims = c, (c["nx"], c["ny"], c["nz"])
        self.n = c["nx"] * c["ny"] * c["nz"]
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        self.lap, self.more, self.grad = _stencils(c["stencil"])
        self.pref, self.pref_df = PI * PI / c["iwidth"] ** 2, PI / c["iwidth"]
        self.phase = torch.as_tensor(P["phase"], dtype=torch.int64, device="cuda")
        self.sigma_p, self.mu_p, self.maxe = t(P["sigma_p"]), t(P["mu_p"]), t(P["maxe"])
        self.solid, self.eps = t(P["solid"]) > 0, None if P["eps"] is None else t(P["eps"])
        self.sigma = None if P["sigma"] is None else t(P["sigma"])
        self.mu = t(P["mu"]) if "mu" in P else None
        self.dg = None if P["dg"] is None else t(P["dg"])
        self.refvol = 4.0 / 3.0 * PI * c["iwidth"] ** 3
        if c["pairs"] == "hash":
            self.sigma = t(_pair_hash(c["grains"], seed))
        if P["quat"] is not None:
            s, x, y, z = t(P["quat"]).unbind(1)
            self.rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * s), 2 * (x * z + y * s),
                                    2 * (x * y + z * s), 1 - 2 * (x * x + z * z), 2 * (y * z - x * s),
                                    2 * (x * z - y * s), 2 * (y * z + x * s), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
        counts, idx, val = (torch.as_tensor(a, device="cuda") for a in P["lists"])
        K = max(c["k"], int(counts.max()))
        take = torch.arange(K, device="cuda") < counts.unsqueeze(1)
        self.g = torch.full((self.n, K), -1, dtype=torch.int64, device="cuda")
        self.v = torch.zeros((self.n, K), dtype=torch.float64, device="cuda")
        self.g[take], self.v[take] = idx.long(), val.double()
        several = counts > 1   # a list read with several fields is finalized
        w, keep = self._finalize(self.v[several], take[several])
        self.g[several], self.v[several] = self._pack(self.g[several], w, keep)
        self.round()
        self.maxvol = torch.zeros(c["grains"], dtype=torch.float64, device="cuda")
        self.alive = torch.ones(c["grains"], dtype=torch.bool, device="cuda")
        self.volumes()

    def round(self):
        """The values as the single-precision form stores its input."""
        if self.c["precision"] == "fp32":
            self.v = self.v.float().double()

    @staticmethod
    def _finalize(v, member):
        """Snap to 0 and 1, erase, normalise to sum 1; returns the values and which are kept."""
        w = torch.where(v >= 1.0 - EPS, torch.ones_like(v), v)
        keep = member & (w > EPS)
        w = torch.where(keep, w, torch.zeros_like(w))
        w = torch.where((keep.sum(1) > 1).unsqueeze(1), w / w.sum(1, keepdim=True), keep.to(w.dtype))
        return w, keep

    @staticmethod
    def _pack(g, v, keep):
        """The kept entries moved to the front in their order."""
        at = torch.argsort((~keep).to(torch.uint8), dim=1, stable=True)
        k = keep.gather(1, at)
        return torch.where(k, g.gather(1, at), torch.full_like(g, -1)), torch.where(k, v.gather(1, at), torch.zeros_like(v))

    def volumes(self):
        G = self.c["grains"]
        self.volume = torch.zeros(G, dtype=torch.float64, device="cuda").index_add(
            0, self.g.clamp(min=0).reshape(-1), self.v.reshape(-1))
        V = self.volume.detach()
        big = torch.maximum(V, self.maxvol)
        gone = self.alive & (V <= 0)
        self.alive = (self.alive & ~gone) | (V > 0)
        self.vr = torch.where(gone, torch.ones_like(V), torch.where(V > 0, (big / self.refvol).clamp(max=1.0), big / self.refvol))
        self.maxvol = torch.where(gone, torch.zeros_like(V), big)

    def neighbour(self, at, o):
        nx, ny, nz = self.dims
        x, y, z = at // (ny * nz), at // nz % ny, at % nz
        return ((x + o[0]) % nx * ny + (y + o[1]) % ny) * nz + (z + o[2]) % nz

    def lists(self, at):
        """Fields of the voxels: their own, then the candidates in the order of the stencil and the
        neighbours' lists; values, Laplacians and (for anisotropic energies) gradients."""
        K, cap = self.g.shape[1], 28
        g = torch.full((len(at), cap), -1, dtype=torch.int64, device="cuda")
        g[:, :K] = self.g[at]
        n = (g >= 0).sum(1)
        deep = int(n.max())
        offsets = [o for o, _ in self.lap] + self.more
        for o in offsets:
            u = self.neighbour(at, o)
            gu = self.g[u]
            for s in range(min(deep, K)):
                new = torch.nonzero((gu[:, s] >= 0) & ~(g == gu[:, s:s + 1]).any(1)).reshape(-1)
                g[new, n[new]] = gu[new, s]
                n[new] += 1
        g = g[:, :int(n.max())]
        v = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
        v[:, :min(K, g.shape[1])] = self.v[at][:, :g.shape[1]]
        lap = torch.zeros_like(v)
        grad = [torch.zeros_like(v) for _ in range(3)] if self.eps is not None else None
        gw = dict(self.grad)
        for o, w in self.lap:
            u = self.neighbour(at, o)
            gu, vu = self.g[u], self.v[u]
            for s in range(min(deep, K)):
                term = (g == gu[:, s:s + 1]) & (g >= 0)
                lap = lap + w * vu[:, s:s + 1] * term
                if grad is not None and o in gw:
                    for a in range(3):
                        grad[a] = grad[a] + gw[o][a] * vu[:, s:s + 1] * term
        return g, n, v, lap, None if grad is None else torch.stack(grad, 2)

    def strong(self):
        """Per voxel the pairs of stored fields whose weight sqrt(v_a v_b) passes the averaging
        threshold, as keys min*G + max (padded with -1)."""
        t = 1.0 / 3.0 if self.c["iwidth"] >= 5.0 else self.c["iwidth"] / 15.0
        thr, G, K = math.sqrt(t * (1.0 - t)), self.c["grains"], self.g.shape[1]
        found = []
        deep = int((self.g >= 0).sum(1).max())
        for a in range(deep):
            for b in range(a + 1, deep):
                ga, gb = self.g[:, a], self.g[:, b]
                ok = (gb >= 0) & (torch.sqrt(self.v[:, a] * self.v[:, b]) > thr * self.vr[ga] * self.vr[gb.clamp(min=0)])
                if bool(ok.any()):
                    found.append(torch.where(ok, torch.minimum(ga, gb) * G + torch.maximum(ga, gb), torch.full_like(ga, -1)))
        return torch.stack(found, 1) if found else torch.full((self.n, 1), -1, device="cuda")

    def averaged(self, at, g, stored, F):
        """A pair's force averaged over the sphere: every voxel holding the pair has the same raw force,
        so the average is that force where some voxel of the sphere is above the threshold, else none."""
        reach, G = int(self.c["iwidth"]), self.c["grains"]
        lo, hi = torch.minimum(g.unsqueeze(2), g.unsqueeze(1)), torch.maximum(g.unsqueeze(2), g.unsqueeze(1))
        key, hit = lo * G + hi, torch.zeros(F.shape, dtype=torch.bool, device="cuda")
        for x in range(-reach, reach + 1):
            for y in range(-reach, reach + 1):
                for z in range(-reach, reach + 1):
                    if reach - math.sqrt(x * x + y * y + z * z) > 0.0:
                        near = self.keys[self.neighbour(at, (x, y, z))]
                        for s in range(near.shape[1]):
                            hit |= near[:, s].reshape(-1, 1, 1) == key
        both = stored.unsqueeze(2) & stored.unsqueeze(1)
        return torch.where(both & ~hit, torch.zeros_like(F), F)

    def energy(self, g, v, grad):
        """Interface energy of every pair of a list."""
        pa = self.phase[g]
        base = self.sigma_p[pa.unsqueeze(2), pa.unsqueeze(1)]
        if self.sigma is not None:
            return self.sigma[g.unsqueeze(2), g.unsqueeze(1)]
        if self.eps is None:
            return base
        norm = grad.norm(dim=2, keepdim=True)
        normal = torch.where(norm > EPS, -grad / norm.clamp(min=EPS), torch.zeros_like(grad))
        normal = torch.einsum("mkij,mki->mkj", self.rot[g], normal)
        weight = (v * (1.0 - v)).abs() * self.solid[pa]
        weight = torch.where(weight > EPS, weight, torch.zeros_like(weight))
        eps = self.eps[pa.unsqueeze(2), pa.unsqueeze(1)]
        shape = (1.5 - 2.5 * (normal ** 4).sum(2))
        total = weight.unsqueeze(2) + weight.unsqueeze(1)
        mean = (weight * shape).unsqueeze(2) + (weight * shape).unsqueeze(1)
        model = torch.where(total > EPS, base * (1.0 + eps * mean / total.clamp(min=EPS)), self.maxe[pa.unsqueeze(2), pa.unsqueeze(1)])
        return torch.where(eps != 0, model, base)

    def update(self, at, g, v, lap, grad, two, stored):
        """New values of lists that all hold n fields; what is kept.  Increments x[i, j] = -x[j, i]."""
        n, dt = g.shape[1], self.c["dt"]
        off = ~torch.eye(n, dtype=torch.bool, device="cuda")
        vr, pa = self.vr[g], self.phase[g]
        scale = torch.sqrt(vr.unsqueeze(2) * vr.unsqueeze(1))
        h = 0.5 * (1.0 + scale) * self.pref
        sg = self.energy(g, v, grad) * off
        L, Q = (sg @ lap.unsqueeze(2)), (sg @ v.unsqueeze(2))
        x = (L.transpose(1, 2) - L) + h * (Q.transpose(1, 2) - Q)
        sp = self.sigma_p[pa.unsqueeze(2), pa.unsqueeze(1)]
        R = (sp @ v.unsqueeze(2)) - (torch.diagonal(sp, dim1=1, dim2=2) * v).unsqueeze(2)
        vi, vj = v.unsqueeze(2), v.unsqueeze(1)
        third = sp * (v.sum(1).reshape(-1, 1, 1) - vi - vj) + (R - sp * vj) + (R.transpose(1, 2) - sp * vi)
        x = x + torch.where(scale < 1.0, 1.0 - scale, torch.zeros_like(scale)) * self.pref * third * (vi - vj)
        mu = self.mu_p[pa.unsqueeze(2), pa.unsqueeze(1)] if self.mu is None else self.mu[g.unsqueeze(2), g.unsqueeze(1)]
        x = x * mu * scale / vr.sum(1).reshape(-1, 1, 1)
        if self.dg is not None:
            allowed = 0.95 * self.pref_df * self.maxe[pa.unsqueeze(2), pa.unsqueeze(1)]
            F = allowed * torch.tanh((self.dg[g].unsqueeze(1) - self.dg[g].unsqueeze(2)) / allowed)
            if self.c["average"]:
                F = self.averaged(at, g, stored, F)
            both = vi * vj
            root = torch.where(both > 0, torch.sqrt(torch.where(both > 0, both, torch.ones_like(both))), torch.zeros_like(both))
            x = x + torch.where(two.reshape(-1, 1, 1), F * mu * root * self.pref_df, torch.zeros_like(F))
        x = torch.where(off, x, torch.zeros_like(x))
        x = self._pair(x, v, dt) if n == 2 else self._limited(x, v, dt)
        value = x * dt
        new = v + torch.where(value.abs() >= EPS, value, torch.zeros_like(value)).sum(2)
        return self._finalize(new, torch.ones_like(new, dtype=torch.bool))

    @staticmethod
    def _pair(x, v, dt):
        a, old = x[:, 0, 1] * dt, v[:, 0]
        stay = ((old == 0) & (a < 0)) | ((old == 1) & (a > 0)) | (a == 0)
        safe = torch.where(stay, torch.ones_like(a), a)
        norm = torch.where(old + a < 0, -old / safe, torch.where(old + a > 1, (1.0 - old) / safe, torch.ones_like(a)))
        a = torch.where(stay | ~(norm > EPS), torch.zeros_like(a), x[:, 0, 1] * norm)
        zero = torch.zeros_like(a)
        return torch.stack([torch.stack([zero, a], 1), torch.stack([-a, zero], 1)], 1)

    @staticmethod
    def _limited(x, v, dt):
        n, zero = v.shape[1], torch.zeros((), dtype=torch.float64, device="cuda")
        for i in range(n):   # a field at its bound takes no increment beyond it
            s = x[:, i].sum(1)
            stop = ((v[:, i] == 0) & (s < 0)) | ((v[:, i] == 1) & (s > 0))
            line = torch.zeros((n, n), dtype=torch.bool, device="cuda")
            line[i], line[:, i] = True, True
            x = torch.where(stop.reshape(-1, 1, 1) & line, zero, x)
        going = torch.ones(len(v), dtype=torch.bool, device="cuda")
        for _ in range(25):
            pos, neg = torch.where(x > 0, x, zero).sum(2), torch.where(x < 0, x, zero).sum(2)
            new = v + (pos + neg) * dt
            under, over = new < 0, new > 1
            one = torch.ones_like(v)
            low = torch.where(under, -(v + pos * dt) / torch.where(under, neg * dt, -one), one).clamp(max=1.0)
            high = torch.where(over, (1.0 - (v + neg * dt)) / torch.where(over, pos * dt, one), one).clamp(max=1.0)
            down = torch.minimum(low.unsqueeze(2), high.unsqueeze(1))
            up = torch.minimum(high.unsqueeze(2), low.unsqueeze(1))
            limit = torch.where(x < 0, down, torch.where(x > 0, up, torch.ones_like(x)))
            x = torch.where(going.reshape(-1, 1, 1), x * limit, x)
            going = going & (limit < 1.0).any(2).any(1)
            if not bool(going.any()):
                break
        return torch.where((x * dt).abs() < EPS, zero, x)

    def step(self):
        count = (self.g >= 0).sum(1)
        grid = (count > 1).reshape(1, 1, *self.dims).float()
        wide = torch.nn.functional.max_pool3d(torch.nn.functional.pad(grid, (1,) * 6, mode="circular"), 3, 1)
        if self.c["average"]:
            self.keys = self.strong()
        out_g, out_v = self.g.clone(), self.v.clone()
        K = self.g.shape[1]
        for at in torch.split(torch.nonzero(wide.reshape(-1) > 0).reshape(-1), 400_000):
            g, n, v, lap, grad = self.lists(at)
            for k in range(2, g.shape[1] + 1):
                rows = torch.nonzero(n == k).reshape(-1)
                if not len(rows):
                    continue
                vk = v[rows, :k]
                w, keep = self.update(at[rows], g[rows, :k], vk, lap[rows, :k], None if grad is None else grad[rows, :k],
                                      count[at[rows]] > 1, torch.arange(k, device="cuda") < count[at[rows]].unsqueeze(1))
                pg, pv = self._pack(g[rows, :k], w, keep)
                m = min(k, K)
                fresh_g = torch.full((len(rows), K), -1, dtype=torch.int64, device="cuda")
                fresh_g[:, :m] = pg[:, :m]
                out_g[at[rows]] = fresh_g
                out_v = out_v.index_put((at[rows],), torch.nn.functional.pad(pv[:, :m], (0, K - m)))
        self.g, self.v = out_g, out_v
        self.volumes()


def _splitmix(x):
    z = x + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _pair_hash(G, seed):
    """The generated pair energies 0.8 + 0.4 u(seed, stream 2, min, max): SplitMix64 over the key."""
    with np.errstate(over="ignore"):
        k = np.arange(G, dtype=np.uint64)
        lo, hi = np.minimum(k[:, None], k[None, :]), np.maximum(k[:, None], k[None, :])
        h = _splitmix(np.full((G, G), seed, np.uint64) ^ (np.uint64(2) * np.array(0xD1B54A32D192ED03, np.uint64)))
        h = _splitmix(_splitmix(h ^ lo) ^ (hi * np.uint64(0x8CB92BA72F3D8DD7)))
    return 0.8 + 0.4 * ((h >> np.uint64(11)).astype(np.float64) * 2.0 ** -53)


def exact(case, seed):
    c = case
    n = c["nx"] * c["ny"] * c["nz"]
    steps = c["steps"] + c["relax"]
    cost = n * steps * (6 if c["average"] or c["nuclei"] else 1) * (8 if c["kind"] in ("adjoint", "tangent") else 1)
    if cost > 60_000_000:   # some twenty seconds
        return None
    P = _problem(c, seed)
    E = _Exact(c, P, seed)
    for _ in range(c["relax"]):
        E.step()
        E.round()
    if c["kind"] == "adjoint":
        leaves = [t.requires_grad_() for t in (E.sigma, E.mu, E.dg)]

        for _ in range(c["steps"]):
            E.step()
        grads = torch.autograd.grad((E.volume * torch.as_tensor(P["weight"], device="cuda")).sum(), leaves)
        off = 1.0 - torch.eye(c["grains"], dtype=torch.float64, device="cuda")
        both = [((t + t.t()) * off).cpu().numpy() for t in grads[:2]]
        return {"volume": E.volume.detach().cpu().numpy(), "dsigma": both[0], "dmu": both[1], "ddg": grads[2].cpu().numpy()}
    if c["kind"] == "tangent":
        import torch.autograd.forward_ad as fwd
        with fwd.dual_level():
            t = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
            E.sigma, E.mu, E.dg = (fwd.make_dual(a, t(b)) for a, b in ((E.sigma, P["dsigma"]), (E.mu, P["dmu"]), (E.dg, P["ddg"])))
            for _ in range(c["steps"]):
                E.step()
            return {"dvolume": fwd.unpack_dual(E.volume).tangent.cpu().numpy()}
    volumes = []
    for _ in range(c["steps"]):
        E.step()
        volumes.append(E.volume.cpu().numpy())
    count = (E.g >= 0).sum(1)
    if c["kind"] == "host":
        value = np.zeros(ROOM * n)
        kept = E.v[E.g >= 0].cpu().numpy()
        value[:kept.size] = kept
        return {"count": None, "grain": None, "value": value, "volume": np.stack(volumes)}
    k, nx = c["k"], c["nx"]
    value = E.v[:, :k].reshape(nx, -1, k).transpose(1, 2).contiguous()
    return {"count": None, "grain": None, "value": value, "volume": np.stack(volumes) if c["kind"] == "loop" else volumes[-1]}
