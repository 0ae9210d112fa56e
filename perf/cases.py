"""Workloads of the solver through its public entry points.

A case is one of three kinds of call:

  solve    one resident problem: back to the initial state, the calc_flow loop
           for `iters` iterations, the permeability, and (where `fields` is
           set) the exported velocity and pressure fields;
  tensor   solve_tensor from host geometry: set-up, the three axis-rotated
           solves and the tensor, as one call;
  server   a stream of uneven requests through the batched server, from the
           first submit to the last completion.

`sweep` names the form of a solve: "mixed" (FP32 correction sweeps with FP64
refinement), "redblack" (FP64, the package's default), "jacobi" (FP64) and
"reference" (FP64 in the reference program's in-place order).

The media are seeded: straight pores of jittered radius and position, periodic
packs of overlapping spheres (radii 4 to 10 voxels) and thresholded Gaussian
fields.  `exact` is the same iteration in plain 64-bit torch on dense arrays.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import poremaps_gb300 as pm

VOXEL = 1e-5
RE, DT, C2, OMEGA = 0.01, 1.0e-4, 1.5e6, 1.2
FLOPS_PER_VOXEL = 62  # 31 multiply-adds per fluid voxel and sweep


def _case(name, kind, medium, size, porosity, sweep, solver, bc, iters, fields=False, **more):
    c = {"name": name, "kind": kind, "medium": medium, "nx": size[0], "ny": size[1],
         "nz": size[2], "porosity": porosity, "sweep": sweep, "solver": solver, "bc": bc,
         "iters": iters, "fields": fields}
    c.update(more)
    if not name:
        del c["name"]
    return c


def listed():
    return [
        # the smallest sample of the configurations: a short solve is bound by
        # launches and latency; a user reads k and looks at the flow field
        _case("pore 48x48x64 mixed", "solve", "pore", (48, 48, 64), 0.55, "mixed", 2, 0, 1101,
              True),
        # one rotation of the tensor benchmark's sphere pack
        _case("pack 128 mixed", "solve", "pack", (128, 128, 128), 0.35, "mixed", 3, 0, 1101),
        # an odd, elongated sample between slip walls
        _case("gauss 157x93x211 mixed", "solve", "gauss", (157, 93, 211), 0.30, "mixed", 2, 1,
              1101),
        # a medium sample between no-slip walls, larger than the caches
        _case("gauss 256 mixed", "solve", "gauss", (256, 256, 256), 0.20, "mixed", 2, 2, 501),
        # the large single sample: the sweeps stream device memory
        _case("gauss 512 mixed", "solve", "gauss", (512, 512, 512), 0.20, "mixed", 2, 2, 201),
        # the package's default order and precision on an odd sample, fields out
        _case("pack 97x61x118 redblack", "solve", "pack", (97, 61, 118), 0.40, "redblack", 2, 1,
              501, True),
        # the default form at the tensor benchmark's size
        _case("pack 128 redblack", "solve", "pack", (128, 128, 128), 0.35, "redblack", 3, 0, 301),
        # plain FP64 Jacobi: the form the others are checked against
        _case("pack 128 jacobi", "solve", "pack", (128, 128, 128), 0.35, "jacobi", 3, 0, 301),
        # drop-in runs: the reference program's in-place order, bit for bit
        _case("pore 48x48x64 reference", "solve", "pore", (48, 48, 64), 0.55, "reference", 2, 0,
              31, True),
        # the whole tensor call from host geometry, as a user with one scan makes it
        _case("tensor pack 128 mixed", "tensor", "pack", (128, 128, 128), 0.35, "mixed", 3, 0,
              1201),
        # serving: uneven samples, more requests than slots, so finished ones
        # make room for queued ones while the rest run on
        _case("server 24 of 32..128", "server", "mix", (32, 128, 24), 0.35, "mixed", 2, 0, 1601,
              eps=1e-3, mix=11, slots=16),
        # serving with few, larger requests
        _case("server 6 of 96..192", "server", "mix", (96, 192, 6), 0.30, "mixed", 3, 0, 1301,
              eps=1e-3, mix=5, slots=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "mixed", "redblack", "jacobi", "reference", "tensor",
                       "server"])
    medium = rng.choice(["pack", "gauss"])
    phi = round(rng.uniform(0.2, 0.5), 3)
    if kind == "server":
        lo = rng.choice([32, 48, 64])
        n = rng.randint(4, 13)
        return _case("", "server", "mix", (lo, _log_int(rng, 2 * lo, 128), n), phi, "mixed",
                     rng.choice([2, 3]), 0, rng.randint(1101, 1301), eps=1e-3,
                     mix=rng.randrange(1000), slots=rng.randint(2, n))
    if kind == "tensor":
        return _case("", "tensor", medium, [_log_int(rng, 40, 128) for _ in range(3)], phi,
                     "mixed", rng.choice([2, 3]), rng.choice([0, 1, 2]), rng.randint(1101, 1401))
    if kind == "reference":
        return _case("", "solve", rng.choice(["pore", "pack"]),
                     [_log_int(rng, 16, 64) for _ in range(3)], 0.5, "reference",
                     rng.choice([1, 2, 3]), rng.randrange(5), rng.randint(5, 31), True)
    if kind == "mixed":
        size = [_log_int(rng, 32, 288) for _ in range(3)]
        most = 3e11 / (FLOPS_PER_VOXEL * phi * math.prod(size))
        return _case("", "solve", medium, size, phi, "mixed", rng.choice([2, 3]),
                     rng.randrange(5), rng.randint(101, max(151, min(1101, int(most)))),
                     rng.random() < 0.5)
    size = [_log_int(rng, 32, 128) for _ in range(3)]
    solver = rng.choice([2, 3]) if kind == "jacobi" else rng.choice([1, 2, 3])
    return _case("", "solve", medium, size, phi, kind, solver, rng.randrange(5),
                 rng.randint(101, 501), rng.random() < 0.5)


# ------------------------------------------------------------------ media
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _pore(nx, ny, nz, seed):
    """Straight pore along z of about 0.42 of the narrower side's length."""
    r = random.Random(seed)
    rad = 0.42 * min(nx, ny) - r.uniform(0.0, 0.05 * min(nx, ny))
    cx, cy = (nx - 1) / 2 + r.uniform(-1, 1), (ny - 1) / 2 + r.uniform(-1, 1)
    y, x = np.mgrid[0:ny, 0:nx]
    solid = (x - cx) ** 2 + (y - cy) ** 2 > rad * rad
    return np.ascontiguousarray(np.broadcast_to(solid, (nz, ny, nx)).astype(np.uint8))


def _pack(nx, ny, nz, phi, seed):
    """Periodic overlapping spheres, radii U[4, 10], Poisson-many for porosity phi."""
    g = _gen(seed)
    mean_vol = 4 / 3 * math.pi * (10.0 ** 4 - 4.0 ** 4) / 4 / 6
    n = max(1, int(round(-math.log(phi) * nx * ny * nz / mean_vol)))
    solid = torch.zeros(nz, ny, nx, dtype=torch.uint8, device="cuda")
    size = torch.tensor([nz, ny, nx], device="cuda")
    off = torch.arange(-11, 12, device="cuda")
    for a in range(0, n, 2048):  # bounded scratch
        m = min(2048, n - a)
        c = torch.rand(m, 3, generator=g, device="cuda", dtype=torch.float64) * size
        rad = 4 + 6 * torch.rand(m, generator=g, device="cuda", dtype=torch.float64)
        i = torch.floor(c).long()[:, :, None] + off          # voxel indices per axis
        d2 = (i + 0.5 - c[:, :, None]) ** 2
        inside = (d2[:, 0, :, None, None] + d2[:, 1, None, :, None] + d2[:, 2, None, None, :]
                  <= (rad * rad)[:, None, None, None])
        i = i % size[None, :, None]
        lin = (i[:, 0, :, None, None] * ny + i[:, 1, None, :, None]) * nx + i[:, 2, None, None, :]
        solid.view(-1)[lin[inside]] = 1
    return solid.cpu().numpy()


def _gauss(nx, ny, nz, phi, seed, sigma=3.0):
    """Lowest phi quantile of Gaussian-filtered white noise (periodic)."""
    f = torch.randn(nz, ny, nx, generator=_gen(seed), device="cuda")
    h = torch.fft.rfftn(f)
    for ax, n in enumerate((nz, ny, nx)):
        k = torch.fft.rfftfreq(n) if ax == 2 else torch.fft.fftfreq(n)
        w = torch.exp(-2 * (math.pi * sigma * k) ** 2).cuda()
        h *= w.view([-1 if a == ax else 1 for a in range(3)])
    f = torch.fft.irfftn(h, s=(nz, ny, nx)).view(-1)
    thr = torch.sort(f[:: max(1, f.numel() // 4_000_000)])[0]
    thr = thr[int(phi * (thr.numel() - 1))]
    return (f > thr).to(torch.uint8).view(nz, ny, nx).cpu().numpy()


def _medium(kind, nx, ny, nz, phi, seed):
    if kind == "pore":
        return _pore(nx, ny, nz, seed)
    return _pack(nx, ny, nz, phi, seed) if kind == "pack" else _gauss(nx, ny, nz, phi, seed)


def _requests(case):
    """The server case's requests: sizes, media, porosities, walls (no seed)."""
    lo, hi, n = case["nx"], case["ny"], case["nz"]
    r = random.Random(case["mix"])
    out = []
    for k in range(n):
        size = [_log_int(r, lo, hi) for _ in range(3)]
        phi = min(0.6, max(0.2, case["porosity"] + r.uniform(-0.1, 0.15)))
        out.append({"medium": "pack" if k % 2 else "gauss", "size": size, "porosity": phi,
                    "bc": r.choice([0, 1, 2])})
    return out


def _geometries(case, seed):
    if case["kind"] == "server":
        return [_medium(q["medium"], *q["size"], q["porosity"], seed * 101 + k)
                for k, q in enumerate(_requests(case))]
    return [_medium(case["medium"], case["nx"], case["ny"], case["nz"], case["porosity"], seed)]


def _params(case, bc):
    kw = {"solving_algorithm": case["solver"], "boundary_method": bc, "voxel_size": VOXEL,
          "max_iter": case["iters"], "eps": case.get("eps", 1e-6)}
    if case["sweep"] == "mixed":
        kw["precision"] = "mixed"
    elif case["sweep"] != "redblack":  # red-black is the default order
        kw["order"] = case["sweep"]
    return kw


# ------------------------------------------------------------------ the calls
def prepare(case, seed):
    geoms = _geometries(case, seed)
    if case["kind"] == "server":
        reqs = _requests(case)
        params = []
        for q, g in zip(reqs, geoms):
            p = pm.default_params(**_params(case, q["bc"]))
            params.append(p)
        return {"case": case, "geoms": geoms, "params": params,
                "server": pm.Server("mixed", max_resident=case["slots"], autotune=1)}
    if case["kind"] == "tensor":
        return {"case": case, "geom": geoms[0],
                "params": pm.default_params(**_params(case, case["bc"]))}
    return {"case": case, "problem": pm.Problem(geoms[0], **_params(case, case["bc"]))}


def _result(r):
    return {"k": np.array([r.wk13, r.wk23, r.wk33]), "velocity": np.array([r.wmax_velz,
            r.wmean_velz]), "permeability": r.permeability, "conv": r.conv,
            "porosity": r.porosity, "iterations": int(r.iterations), "sweeps": int(r.sweeps),
            "converged": int(r.converged)}


def run(state):
    case = state["case"]
    if case["kind"] == "server":
        s = state["server"]
        at = {s.submit(g, p): k for k, (g, p) in enumerate(zip(state["geoms"], state["params"]))}
        out = [None] * len(at)
        active = 1
        while active:
            active = s.step()
            for c in s.poll():
                out[at[c.ticket]] = c.result
        return _table([_result(r) for r in out])
    if case["kind"] == "tensor":
        K, res = pm.solve_tensor(state["geom"], state["params"])
        return dict(_table([_result(r) for r in res]), K=K)
    pr = state["problem"]
    pr.reset()
    out = _result(pr.solve())
    if case["fields"]:
        out["u"], out["v"], out["w"], out["p"] = pr.fields()
    return out


def _table(rows):
    """The results of several solves, one array per quantity."""
    return {k: np.array([r[k] for r in rows]) for k in rows[0]}


def work(case):
    """Geometry in, results (and fields) out, and the sweeps' arithmetic."""
    if case["kind"] == "server":
        vox = fluid = 0
        for q in _requests(case):
            n = q["size"][0] * q["size"][1] * q["size"][2]
            vox += n
            fluid += q["porosity"] * n
        return {"bytes": vox, "flops": FLOPS_PER_VOXEL * fluid * 1101}
    vox = case["nx"] * case["ny"] * case["nz"]
    sweeps = case["iters"] * (3 if case["kind"] == "tensor" else 1)
    return {"bytes": vox * (1 + (32 if case["fields"] else 0)),
            "flops": FLOPS_PER_VOXEL * case["porosity"] * vox * sweeps}


# ------------------------------------------------------------------ 64-bit check
def _axis_cases(solid, ax):
    """Neighbourhood case (1..6) along one axis of every interior voxel."""
    n = [s - 4 for s in solid.shape]

    def at(d):
        return solid[tuple(slice(2 + (d if a == ax else 0), 2 + (d if a == ax else 0) + n[a])
                           for a in range(3))]

    ll, l, r, rr = at(-2), at(-1), at(1), at(2)
    c = torch.full(n, 6, dtype=torch.int64, device=solid.device)
    c = torch.where(l & r, 1, c)
    c = torch.where(l & ~r, torch.where(rr, 2, 4), c)
    return torch.where(~l & r, torch.where(ll, 3, 5), c)


#: per case: centre, second left, left, right, second right
_COEF = [[0] * 5, [-8, 0, 0, 0, 0], [-16 / 3, 0, 0, 8 / 3, 0], [-16 / 3, 0, 8 / 3, 0, 0],
         [-5, 0, 0, 2, -1 / 5], [-5, -1 / 5, 2, 0, 0], [-2, 0, 1, 1, 0]]


class _Dense:
    """The iteration on dense padded double arrays (axes z, y, x; halo 2)."""

    def __init__(self, geom, bc, solver):
        g = torch.from_numpy(geom).cuda() != 0
        self.n = nz, ny, nx = g.shape
        self.per = per = (bc <= 2, bc == 0, bc == 0)
        self.solver = solver
        pad = torch.zeros(nz + 4, ny + 4, nx + 4, dtype=torch.bool, device="cuda")
        self.inner = (slice(2, nz + 2), slice(2, ny + 2), slice(2, nx + 2))
        pad[self.inner] = g
        self._halo(pad)
        self.fluid = ~g
        self.padded_fluid = ~pad
        cs = [_axis_cases(pad, a) for a in range(3)]
        tab = torch.tensor(_COEF, dtype=torch.float64, device="cuda")
        self.coef = [[tab[:, k][c] for k in range(5)] for c in cs]
        self.lsolid = [(c == 1) | (c == 2) | (c == 4) for c in cs]
        z = torch.zeros(nz + 4, ny + 4, nx + 4, dtype=torch.float64, device="cuda")
        # pressure: nz + 2 at the first interior plane down to 3 at the last
        ramp = torch.arange(nz, device="cuda", dtype=torch.float64)
        p = torch.full_like(z, 0.0)
        p[self.inner] = torch.where(self.fluid, (nz + 2 - ramp)[:, None, None], 0.0)
        for a in range(3):
            if not per[a]:
                for s in (slice(0, 2), slice(self.n[a] + 2, None)):
                    p[tuple(s if b == a else slice(None) for b in range(3))] = -1.0
        self.f = [z, z.clone(), z.clone(), p]
        self._halo(p)
        self._planes(p)
        p[self.last] = torch.where(self.padded_fluid[self.last], 3.0, p[self.last])

    @property
    def last(self):
        return (self.n[0] + 1,) + self.inner[1:]

    def _halo(self, f):
        for a in range(3):
            if not self.per[a]:
                continue
            n = self.n[a]
            idx = [slice(None)] * 3
            src = [slice(None)] * 3
            for to, frm in ((slice(0, 2), slice(n, n + 2)), (slice(n + 2, n + 4), slice(2, 4))):
                idx[a], src[a] = to, frm
                f[tuple(idx)] = f[tuple(src)]

    def _planes(self, p):
        """Reapplied pressure on the z halo planes next to the domain."""
        for z, val in ((1, self.n[0] + 2.0), (self.n[0] + 2, 2.0)):
            at = (z,) + self.inner[1:]
            p[at] = torch.where(self.padded_fluid[at], val, p[at])

    def _at(self, f, ax, d):
        return f[tuple(slice(2 + (d if a == ax else 0), 2 + (d if a == ax else 0) + self.n[a])
                       for a in range(3))]

    def update(self, f):
        """New values of every interior voxel from the padded fields f."""
        u, v, w, p = f
        pc = p[self.inner].clone()
        pc[-1] = 3.0  # the reapplied pressure of the last plane
        new = []
        div = None
        for ax, q in ((2, u), (1, v), (0, w)):
            c = self._at(q, ax, 0)
            s = self._at(q, ax, -1) - 2 * c + self._at(q, ax, 1)
            for b in range(3):
                if b == ax:
                    continue
                k = self.coef[b]
                s = s + k[0] * c
                for j, d in ((1, -2), (2, -1), (3, 1), (4, 2)):
                    s = s + k[j] * self._at(q, b, d)
            dp = torch.where(self.lsolid[ax], 0.0, pc - self._at(p, ax, -1))
            if self.solver == 3:
                x = (1 - OMEGA) * c + OMEGA * (s / RE - dp) * DT
            else:
                x = torch.where(self.lsolid[ax], 0.0, c + (s / RE - dp) * DT)
            x = torch.where(self.fluid, x, 0.0)
            t = self._at(q, ax, 1) - (c if self.solver == 1 else x)
            div = t if div is None else div + t
            new.append(x)
        new.append(torch.where(self.fluid, pc - C2 * DT * div, 0.0))
        return new

    def put(self, f, new):
        for q, x in zip(f, new):
            q[self.inner] = x
            self._halo(q)
        self._planes(f[3])

    def sweep(self, f, redblack):
        if not redblack:
            self.put(f, self.update(f))
            return
        z, y, x = (torch.arange(n, device="cuda") for n in self.n)
        red = ((z[:, None, None] + y[:, None] + x) & 1) == 0
        new = self.update(f)
        for q, a in zip(f, new):  # interior neighbours see new red, halos the old iterate
            q[self.inner] = torch.where(red, a, q[self.inner])
        black = self.update(f)
        self.put(f, [torch.where(red, a, b) for a, b in zip(new, black)])

    def sweeps(self, redblack):
        """A function that does one sweep, replayed from a graph."""
        side = torch.cuda.Stream()
        keep = [q.clone() for q in self.f]
        with torch.cuda.stream(side):
            self.sweep(self.f, redblack)
        side.synchronize()
        for q, k in zip(self.f, keep):
            q.copy_(k)
        del keep
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            self.sweep(self.f, redblack)
        return g.replay

    def result(self, swept, conv, perm, check, converged):
        u, v, w = (q[self.inner][self.fluid] for q in self.f[:3])
        nfl = int(self.fluid.sum())
        phi = nfl / self.fluid.numel()
        k = [float(q.sum()) / nfl / RE * phi * VOXEL ** 2 for q in (u, v, w)]
        return {"k": np.array(k), "velocity": np.array([max(0.0, float(w.max())) * VOXEL,
                float(w.sum()) / nfl * VOXEL]), "permeability": perm, "conv": conv,
                "porosity": phi, "iterations": check, "sweeps": swept, "converged": converged}

    def fields(self):
        out = [q[self.inner].cpu().numpy().copy() for q in self.f]
        out[3][-1][self.fluid[-1].cpu().numpy()] = 3.0
        return out

    def solve(self, iters, eps, redblack):
        """calc_flow: a check every 100 iterations from iteration 1100 on."""
        step = self.sweeps(redblack)
        conv, perm, check, done = 1.0 + eps, 0.0, 0, 0
        for it in range(iters):
            step()
            if it > 1000 and it % 100 == 0:
                cur = float(self.f[2][self.inner][self.fluid].sum()) / int(self.fluid.sum()) / RE
                conv, perm, check = abs(cur - perm) / cur, cur, it
                if not conv >= eps:
                    done = 1
                    break
        return self.result(it + 1, conv, perm, check, done)

    def solve_in_place(self, iters, eps):
        """The reference program's order: every voxel in place, x fastest."""
        nz, ny, nx = self.n
        py, pz = nx + 4, (nx + 4) * (ny + 4)
        z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda") for n in self.n),
                                 indexing="ij")
        plane = (x + y + z)[self.fluid]
        at = ((z + 2) * pz + (y + 2) * py + x + 2)[self.fluid]
        lin = ((z * ny + y) * nx + x)[self.fluid]
        order = torch.argsort(plane, stable=True)
        cut = torch.bincount(plane, minlength=nx + ny + nz - 2).cumsum(0).tolist()
        steps = (1, py, pz)
        flat = [q.view(-1) for q in self.f]
        parts = []
        for a, b in zip([0] + cut[:-1], cut):
            if a == b:
                continue
            i, k = at[order[a:b]], lin[order[a:b]]
            parts.append((i, [[t.reshape(-1)[k] for t in self.coef[2 - ax]] for ax in range(3)],
                          [self.lsolid[2 - ax].reshape(-1)[k] for ax in range(3)]))
        for _ in range(iters):
            for i, coef, ls in parts:
                pc = flat[3][i]
                div = 0.0
                new = []
                for ax in range(3):
                    q = flat[ax]
                    c = q[i]
                    s = q[i - steps[ax]] - 2 * c + q[i + steps[ax]]
                    for b in range(3):
                        if b != ax:
                            k, t = coef[b], steps[b]
                            s = (s + k[0] * c + k[1] * q[i - 2 * t] + k[2] * q[i - t]
                                 + k[3] * q[i + t] + k[4] * q[i + 2 * t])
                    dp = torch.where(ls[ax], 0.0, pc - flat[3][i - steps[ax]])
                    if self.solver == 3:
                        xn = (1 - OMEGA) * c + OMEGA * (s / RE - dp) * DT
                    else:
                        xn = torch.where(ls[ax], 0.0, c + (s / RE - dp) * DT)
                    div = div + q[i + steps[ax]] - (c if self.solver == 1 else xn)
                    new.append(xn)
                new.append(pc - C2 * DT * div)
                for q, xn in zip(flat, new):
                    q[i] = xn
            for q in self.f:
                self._halo(q)
            self._planes(self.f[3])
            self.f[3][self.last] = torch.where(self.fluid[-1], 3.0, self.f[3][self.last])
        return self.result(iters, 1.0 + eps, 0.0, 0, 0)


def _cost(voxels, sweeps):
    """Seconds of a 64-bit dense solve, roughly."""
    return sweeps * (2.5e-4 + voxels * 3.5e-10)


def exact(case, seed):
    iters, eps = case["iters"], case.get("eps", 1e-6)
    if case["kind"] == "server":
        reqs = _requests(case)
        if sum(_cost(math.prod(q["size"]), iters) for q in reqs) > 18:
            return None
        return _table([_Dense(g, q["bc"], case["solver"]).solve(iters, eps, False)
                       for g, q in zip(_geometries(case, seed), reqs)])
    geom = _geometries(case, seed)[0]
    if case["kind"] == "tensor":
        if 3 * _cost(geom.size, iters) > 18:
            return None
        rows, K = [], np.zeros((3, 3))
        # flow along x, y, z: z' is the flow axis, x' and y' follow it cyclically
        for flow, perm in ((0, (2, 0, 1)), (1, (1, 2, 0)), (2, (0, 1, 2))):
            g = np.ascontiguousarray(geom.transpose(perm))
            rows.append(_Dense(g, case["bc"], case["solver"]).solve(iters, eps, False))
            # axes (x', y', z') of the rotated sample in the original's numbering
            K[[2 - perm[2], 2 - perm[1], 2 - perm[0]], flow] = rows[-1]["k"]
        return dict(_table(rows), K=K)
    if case["sweep"] == "reference":
        if iters * sum(geom.shape) * 6e-4 > 18:
            return None
        d = _Dense(geom, case["bc"], case["solver"])
        out = d.solve_in_place(iters, eps)
    else:
        twice = 2 if case["sweep"] == "redblack" else 1
        if twice * _cost(geom.size, iters) > 18:
            return None
        d = _Dense(geom, case["bc"], case["solver"])
        out = d.solve(iters, eps, case["sweep"] == "redblack")
    if case["fields"]:
        out["u"], out["v"], out["w"], out["p"] = d.fields()
    return out
