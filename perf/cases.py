"""Performance cases: the work that a user of the DPD engine has it do, through its public
Python API (the mirror of the reference's DPDEngine interface) and its C entry points.

``listed()`` names the cases, ``draw(rng)`` makes more of the same ranges, ``prepare`` builds
what a program holds before the call (worlds from the seeded generators, an engine with the
world attached), ``run`` is one pass as a program calls it, ``work`` the bytes and operations
a pass cannot do without, and ``exact`` the same results from plain torch in 64 bits.

Sizes are those of the repository's benchmark configurations (the 8^3 FP64 water box, the
32^3 and 128^3 polymer boxes, the grid of uneven polymer boxes, the served job mix) and odd
ones between them.  Box sides are cells of edge r_c = 1 at density 3.
"""

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(ROOT, "poets-dpd_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import pdpd_engine as E  # noqa: E402
import pdpd_world as W  # noqa: E402


def _case(kind, precision, box, chains, dt, steps, name=None, **more):
    c = {"kind": kind, "precision": precision, "sx": box[0], "sy": box[1], "sz": box[2], "chains": chains,
         "dt": dt, "steps": steps, **more}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the plain engine's own configuration: 1,536 water beads stepped in FP64
        _case("run", "fp64", (8, 8, 8), 0.0, 0.02, 100, "fp64_water8"),
        # an ordinary FP64 polymer box of uneven odd sides
        _case("run", "fp64", (23, 31, 27), 0.1, 0.01, 20, "fp64_polymer_23x31x27"),
        # a large FP64 box (786,432 beads), a few steps between looks at the state
        _case("run", "fp64", (64, 64, 64), 0.05, 0.01, 5, "fp64_polymer64"),
        # the smallest FP32 boxes: a parameter scan's water box
        _case("run", "fp32", (9, 9, 9), 0.0, 0.02, 40, "fp32_water9"),
        # the 98,304-bead polymer box of the FP32-against-FP64 configuration
        _case("run", "fp32", (32, 32, 32), 0.1, 0.01, 100, "fp32_polymer32"),
        # an uneven odd box followed interval by interval, the state read at each callback
        _case("intervals", "fp32", (37, 50, 61), 0.05, 0.01, 10, "fp32_intervals_37x50x61", intervals=5),
        # the 6.3M-bead box, the largest single state
        _case("run", "fp32", (128, 128, 128), 0.05, 0.01, 20, "fp32_polymer128"),
        # a batch of independent uneven states with their own parameters, stepped together
        _case("batch", "fp32", (8, 32, 0), 0.05, 0.01, 20, "fp32_grid96", states=96),
        # one whole job from host arrays: attach a fresh state, run it, read it back
        _case("job", "fp32", (56, 56, 56), 0.05, 0.01, 20, "fp32_job56"),
        # the job server: water boxes of sides log-uniform on the range, uneven step counts
        _case("serve", "fp32", (8, 32, 0), 0.0, 0.01, 100, "fp32_serve20", states=20, intervals=25),
        # a compact snapshot of the current state
        _case("snapshot", "fp32", (64, 64, 64), 0.05, 0.01, 1, "fp32_snapshot64"),
        # stepping on the caller's own device arrays without allocating (bond-free, FP64)
        _case("arrays", "fp64", (16, 16, 16), 0.0, 0.02, 25, "fp64_arrays16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """Three sides around a common log-uniform one, odd and uneven among them."""
    c = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return tuple(max(lo, min(hi, int(round(c * rng.uniform(0.8, 1.25))))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["run32", "run32", "run32", "run64", "run64", "intervals", "batch", "job", "serve", "snapshot",
                       "arrays"])
    chains = round(rng.choice([0.0, rng.uniform(0.03, 0.12)]), 3)
    dt = 0.01 if chains else 0.02
    if kind == "run32":
        s = _sides(rng, 8, 120)
        n = 3 * s[0] * s[1] * s[2]
        return _case("run", "fp32", s, chains, dt, max(5, min(100 if chains else 40, int(6e7 / n))))
    if kind == "run64":
        s = _sides(rng, 6, 64)
        n = 3 * s[0] * s[1] * s[2]
        return _case("run", "fp64", s, chains, dt, max(3, min(100, int(3e6 / n))))
    if kind == "intervals":
        return _case("intervals", rng.choice(["fp32", "fp32", "fp64"]), _sides(rng, 8, 52), chains, dt,
                     rng.randint(3, 12), intervals=rng.randint(2, 6))
    if kind == "batch":
        lo = rng.randint(6, 12)
        return _case("batch", "fp32", (lo, rng.randint(lo + 4, 32), 0), round(rng.uniform(0.03, 0.12), 3), 0.01,
                     rng.randint(5, 25), states=_log_int(rng, 4, 96))
    if kind == "job":
        return _case("job", rng.choice(["fp32", "fp32", "fp64"]), _sides(rng, 8, 56), chains, dt, rng.randint(3, 20))
    if kind == "serve":
        return _case("serve", "fp32", (8, rng.randint(16, 32), 0), 0.0, 0.01, rng.randint(50, 100),
                     states=rng.randint(4, 20), intervals=rng.choice([10, 25]))
    if kind == "snapshot":
        return _case("snapshot", rng.choice(["fp32", "fp64"]), _sides(rng, 8, 64), chains, dt, 1)
    return _case("arrays", "fp64", _sides(rng, 4, 20), 0.0, 0.02, rng.randint(5, 25))


# ------------------------------------------------------------------------------------------
# inputs

def _settle(w, rng):
    """Positions as a run has them after its first steps, not the overlaps of independent
    uniform ones: the monomers near the sites of a slightly sparse lattice, the chains nearly
    straight."""
    L = np.asarray(w.box, float)
    n, n_chain = w.n_beads, 6 * (len(w.flat_bonds()[0]) // 5)
    if n_chain:
        d = rng.standard_normal((n_chain // 6, 1, 3))
        d /= np.linalg.norm(d, axis=2, keepdims=True)
        head = w.x[:n_chain].reshape(-1, 6, 3)[:, :1]
        w.x[:n_chain] = np.mod(head + 0.5 * np.arange(6)[None, :, None] * d, L).reshape(-1, 3)
    m = np.ceil(1.45 * L).astype(np.int64)
    site = rng.choice(int(np.prod(m)), n - n_chain, replace=False, shuffle=False)
    at = np.stack(np.unravel_index(site, m), 1)
    w.x[n_chain:] = (at + 0.5 + 0.6 * (rng.random((n - n_chain, 3)) - 0.5)) * (L / m)
    w.x[w.x >= L] = 0.0
    return w


def _worlds(case, seed):
    """The case's worlds (for the server also each job's step count): their sizes from the
    case, their states from the seed."""
    rng = np.random.default_rng([7, int(seed)])
    shape = np.random.default_rng([11, case.get("states", 1), case["steps"]])
    kind, chains, dt = case["kind"], case["chains"], case["dt"]

    def one(box, **par):
        state_seed, gen = int(rng.integers(1, 1 << 40)), int(rng.integers(1 << 40))
        if chains == 0.0:
            w = W.make_water(box, seed=state_seed, dt=dt, gen_seed=gen)
        else:
            w = W.make_polymer_box(box, chain_fraction=chains, seed=state_seed, dt=dt, gen_seed=gen, **par)
        return _settle(w, rng)

    if kind == "batch":
        return [one(int(shape.integers(case["sx"], case["sy"] + 1)), a_wt=float(rng.uniform(25.0, 100.0)),
                    gamma=float(rng.uniform(3.0, 6.0))) for _ in range(case["states"])], None
    if kind == "serve":
        lo, hi = math.log(case["sx"]), math.log(case["sy"])
        sides = [int(round(math.exp(shape.uniform(lo, hi)))) for _ in range(case["states"])]
        steps = [int(shape.integers(case["steps"] // 4, case["steps"] + 1)) for _ in sides]
        return [one(side) for side in sides], steps
    return [one((case["sx"], case["sy"], case["sz"]))], None


def prepare(case, seed):
    worlds, steps = _worlds(case, seed)
    kind = case["kind"]
    s = {"case": case, "worlds": worlds, "steps": steps}
    if kind == "serve":
        s["server"] = E.GB300DPDServer(case["precision"], memory_budget_bytes=1 << 30,
                                       interval_steps=case["intervals"])
        return s
    if kind == "arrays":
        w = worlds[0]
        dev = torch.device("cuda")
        s["x"], s["v"], s["f"] = (torch.from_numpy(a.copy()).to(dev) for a in (w.x, w.v, w.f))
        s["hash"] = torch.from_numpy(w.hashes().view(np.int32).copy()).to(dev)
        s["t"] = 0
        return s
    if kind == "batch":
        # the states' vectors are rows of three common arrays, each World a view of its own
        n = sum(w.n_beads for w in worlds)
        s["x"], s["v"], s["f"] = (np.empty((n, 3)) for _ in range(3))
        at = 0
        for w in worlds:
            for k in ("x", "v", "f"):
                view = s[k][at:at + w.n_beads]
                view[:] = getattr(w, k)
                setattr(w, k, view)
            at += w.n_beads
    eng = s["engine"] = E.GB300DPDEngine(case["precision"])
    if kind == "batch":
        eng.AttachBatch(worlds)
    elif kind != "job":
        eng.Attach(worlds[0])
    if kind == "snapshot":
        eng.Run(case["steps"])
        eng.v2binary_prepare()
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = state["server"]
        jobs = [srv.submit(w, n) for w, n in zip(state["worlds"], state["steps"])]
        srv.drain()
        return [srv.results.pop(j)[:3] for j in jobs]
    w = state["worlds"][0]
    if kind == "arrays":
        E.step_noalloc(w, state["x"].data_ptr(), state["v"].data_ptr(), state["f"].data_ptr(),
                       state["hash"].data_ptr(), case["steps"], t=state["t"],
                       stream=torch.cuda.current_stream().cuda_stream)
        state["t"] += case["steps"]
        return [state["x"], state["v"], state["f"]]
    eng = state["engine"]
    if kind == "snapshot":
        return eng.v2binary_encode()
    if kind == "batch":
        eng.Run(case["steps"])
        return [state["x"], state["v"], state["f"]]
    if kind == "intervals":
        eng.Run(case["intervals"], case["steps"], lambda: True)
        return [w.x, w.v, w.f]
    if kind == "job":
        eng.Attach(w)
    eng.Run(case["steps"])
    return [w.x, w.v, w.f]


# ------------------------------------------------------------------------------------------
# what a pass cannot do without

# Each bead has 4/3 pi 3 / 2 = 6.28 neighbours in range of its own half; a pair force is about
# 60 operations, an update of position and momentum about 20.
_FLOPS_PER_BEAD_STEP = 6.28 * 60 + 20


def work(case):
    kind = case["kind"]
    state_bytes = 36 + 4 if case["precision"] == "fp32" else 72 + 4  # x, v, f, hash in the engine's precision
    if kind == "batch":
        mean = sum(3.0 * k ** 3 for k in range(case["sx"], case["sy"] + 1)) / (case["sy"] + 1 - case["sx"])
        n, steps = mean * case["states"], case["steps"]
    elif kind == "serve":
        lo, hi = math.log(case["sx"]), math.log(case["sy"])
        n = case["states"] * (math.exp(3 * hi) - math.exp(3 * lo)) / (hi - lo)  # mean of 3 side^3, times the jobs
        steps = case["steps"] * 0.625
    else:
        n, steps = 3.0 * case["sx"] * case["sy"] * case["sz"], case["steps"]
    if kind == "snapshot":
        return {"bytes": n * (state_bytes + 22), "flops": n * 9}
    if kind == "intervals":
        steps = steps * case["intervals"]
    # each step reads the state once and writes it once; x, v, f go to the host in FP64
    # after a run, and come from there for a job
    total = n * steps * (2 * state_bytes)
    if kind != "arrays":
        total += n * 72 * (case["intervals"] if kind == "intervals" else 1)
    if kind in ("job", "serve"):
        total += n * 76
    return {"bytes": total, "flops": n * steps * _FLOPS_PER_BEAD_STEP}


# ------------------------------------------------------------------------------------------
# the same results in 64 bits

_M32 = 0xFFFFFFFF
_MIX = 0xD392D2A7


def _t_hash(t, seed):
    def mix(x):
        x ^= x >> 32
        x = (x * _MIX) & 0xFFFFFFFFFFFFFFFF
        x ^= x >> 32
        x = (x * _MIX) & 0xFFFFFFFFFFFFFFFF
        return x ^ (x >> 32)
    return mix(((seed & 0xFFFFFFFFFFFFFFFF) + mix(t & _M32)) & 0xFFFFFFFFFFFFFFFF)


def _pair_uniform(lo, hi, a, b):
    """The symmetric pair random number: 32-bit words of a 64-bit mix, in int64 tensors."""
    x = torch.minimum(a, b) ^ lo
    y = torch.maximum(a, b) ^ hi
    for _ in range(2):
        x = x ^ y
        p = x * _MIX                       # (wraps: its low 64 bits are what is wanted)
        x, y = p & _M32, ((p >> 32) + y * _MIX) & _M32
    h = (x ^ y)
    h = torch.where(h >= 1 << 31, h - (1 << 32), h)
    return h.to(torch.float32).to(torch.float64) * 2.0 ** -32


class _Exact:
    """Plain torch DPD in FP64 over some worlds together: half-step velocity Verlet."""

    def __init__(self, worlds, dev):
        self.dev, f64 = dev, torch.float64
        up = lambda a, t: torch.as_tensor(np.ascontiguousarray(a)).to(dev, t)  # noqa: E731
        n = [w.n_beads for w in worlds]
        self.n = n
        self.world = torch.repeat_interleave(torch.arange(len(worlds), device=dev), torch.tensor(n, device=dev))
        self.x, self.v, self.f = (torch.cat([up(getattr(w, k), f64) for w in worlds]) for k in ("x", "v", "f"))
        self.hash = torch.cat([up(w.hashes().astype(np.int64), torch.int64) for w in worlds])
        self.type = self.hash >> 28
        self.box = up(np.array([w.box for w in worlds]), torch.int64)
        self.L = self.box.to(f64)
        cells = np.array([int(np.prod(w.box.astype(np.int64))) for w in worlds])
        self.cell0 = up(np.concatenate([[0], np.cumsum(cells)[:-1]]), torch.int64)
        self.n_cells = int(cells.sum())
        self.nt = worlds[0].n_types
        self.a = torch.cat([up(w.conservative.reshape(-1), f64) for w in worlds])
        self.sg = torch.cat([up(w.dissipative.reshape(-1), f64) for w in worlds]).sqrt()
        self.dt = up(np.array([w.dt for w in worlds]), f64)
        self.seed, self.t = [int(w.seed) for w in worlds], [int(w.t) for w in worlds]
        base = np.concatenate([[0], np.cumsum(n)[:-1]]).astype(np.int64)
        bonds = [w.flat_bonds() for w in worlds]
        cat = lambda k, o: up(np.concatenate([np.asarray(b[k], np.int64 if o else np.float64) + (s if o else 0)  # noqa: E731
                                              for b, s in zip(bonds, base)]), torch.int64 if o else f64)
        self.bb, self.bk, self.br, self.ab, self.ak, self.at = (cat(0, 1), cat(1, 0), cat(2, 0), cat(3, 1), cat(4, 0),
                                                                cat(5, 0))

    def _cell(self, c, w):
        b = self.box[w]
        return self.cell0[w] + (c[:, 0] * b[:, 1] + c[:, 1]) * b[:, 2] + c[:, 2]

    def _image(self, d, w):
        L = self.L[w]
        return d - torch.where(d > L / 2, L, torch.zeros_like(L)) + torch.where(d < -L / 2, L, torch.zeros_like(L))

    def _pairs(self):
        """(i, j, x_i - x_j) of the pairs closer than 1, each once."""
        w = self.world
        c = self.x.floor().to(torch.int64)
        key = self._cell(c, w)
        order = torch.argsort(key)
        start = torch.zeros(self.n_cells + 1, dtype=torch.int64, device=self.dev)
        start[1:] = torch.cumsum(torch.bincount(key, minlength=self.n_cells), 0)
        most = int((start[1:] - start[:-1]).max())
        out = []
        step = max(1, (1 << 26) // max(1, most))
        for lo in range(0, len(w), step):
            i = torch.arange(lo, min(len(w), lo + step), device=self.dev)
            wi, ci, xi = w[i], c[i], self.x[i]
            for dx in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    for dz in (-1, 0, 1):
                        if (dx, dy, dz) < (0, 0, 0):
                            continue
                        raw = ci + torch.tensor([dx, dy, dz], device=self.dev)
                        b = self.box[wi]
                        wrap = torch.div(raw, b, rounding_mode="floor")
                        nc = self._cell(raw - wrap * b, wi)
                        s, e = start[nc], start[nc + 1]
                        at = s[:, None] + torch.arange(most, device=self.dev)[None, :]
                        r, k = torch.nonzero(at < e[:, None], as_tuple=True)
                        j = order[s[r] + k]
                        ii = i[r]
                        if (dx, dy, dz) == (0, 0, 0):
                            keep = ii < j
                            r, j, ii = r[keep], j[keep], ii[keep]
                        d = xi[r] - (self.x[j] + (wrap[r] * b[r]).to(torch.float64))
                        r2 = (d * d).sum(1)
                        keep = (r2 < 1.0) & (r2 >= 1e-18)
                        out.append((ii[keep], j[keep], d[keep]))
        return [torch.cat(q) for q in zip(*out)]

    def step(self):
        w, dt = self.world, self.dt[self.world][:, None]
        L = self.L[w]
        x = self.x + self.v * dt + self.f * (dt * dt / 2)
        x = torch.where(x < 0, x + L, torch.where(x >= L, x - L, x))
        self.x = torch.where(x == L, torch.zeros_like(x), x)
        self.v = self.v + self.f * (dt / 2)
        f = torch.zeros_like(self.f)
        th = [_t_hash(t, s) for t, s in zip(self.t, self.seed)]
        lo = torch.tensor([h & _M32 for h in th], device=self.dev)
        hi = torch.tensor([h >> 32 for h in th], device=self.dev)
        i, j, d = self._pairs()
        wi = w[i]
        r = (d * d).sum(1).sqrt()
        e = d / r[:, None]
        k = wi * self.nt * self.nt + self.type[i] * self.nt + self.type[j]
        s = self.sg[k] * (1 - r)
        u = _pair_uniform(lo[wi], hi[wi], self.hash[i], self.hash[j])
        m = self.a[k] * (1 - r) - s * s * (e * (self.v[i] - self.v[j])).sum(1) + s * (24 / self.dt[wi]).sqrt() * u
        p = e * m[:, None]
        f.index_add_(0, i, p)
        f.index_add_(0, j, -p)
        if len(self.bk):
            h, t = self.bb[:, 0], self.bb[:, 1]
            d = self._image(self.x[t] - self.x[h], w[h])
            r = (d * d).sum(1).sqrt()
            p = d * (self.bk * (self.br - r) / r)[:, None]
            f.index_add_(0, h, -p)
            f.index_add_(0, t, p)
        if len(self.ak):
            h, m, t = self.ab.unbind(1)
            b1, b2 = self._image(self.x[m] - self.x[h], w[h]), self._image(self.x[t] - self.x[m], w[h])
            n1, n2, dot = (b1 * b1).sum(1), (b2 * b2).sum(1), (b1 * b2).sum(1)
            mag = (n1 * n2).sqrt()
            bend = (1 / (1 / (dot * dot / (n1 * n2)) - 1).sqrt()).nan_to_num(0.0, 0.0, 0.0)
            sin = torch.sin(self.at)
            fm = self.ak / mag * torch.where((dot.abs() > 1e-6) & (sin > 0), torch.cos(self.at) - sin * bend,
                                             torch.ones_like(dot))
            fm = torch.where(mag > 1e-4, fm, torch.zeros_like(fm))[:, None]
            ph, pt = (b1 * (dot / n1)[:, None] - b2) * fm, (b1 - b2 * (dot / n2)[:, None]) * fm
            f.index_add_(0, h, ph)
            f.index_add_(0, t, pt)
            f.index_add_(0, m, -(ph + pt))
        self.f = f
        self.v = self.v + f * (dt / 2)
        self.t = [t + 1 for t in self.t]


def exact(case, seed):
    if case["kind"] == "snapshot":
        return None  # bytes
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    worlds, steps = _worlds(case, seed)
    if case["kind"] == "serve":
        out = []
        for w, n in zip(worlds, steps):
            q = _Exact([w], dev)
            for _ in range(n):
                q.step()
            out.append([q.x, q.v, q.f])
        return out
    q = _Exact(worlds, dev)
    for _ in range(case["steps"] * (case["intervals"] if case["kind"] == "intervals" else 1)):
        q.step()
    return [q.x, q.v, q.f]
