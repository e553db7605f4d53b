"""The work the library is timed on: whole calls through its public entry points.

Four kinds of call, as the library's users make them:

  step   the drop-in C-ABI, as a simulation code drives it once per time step: positions,
         h, velocities and accelerations up from page-locked host arrays, the density and
         smoothing-length solve with its gradient sweep, the thermodynamic state up, the
         force pass, every result slot down
  batch  many independent sets solved together: upload, density, download
  serve  a burst of requests to the running server, some of them continuing a set that
         stays on the device; all results waited for
  order  the allocation-free Hilbert keys and sort order of a device-resident set

Particle sets are the repository's workloads, generated here: the close-packed lattice with
1% of its smoothing lengths off (what a run starts from), the same lattice slightly drifted
with smoothing lengths near convergence (what a run hands over between steps), uniform
random particles in the unit periodic box, and Plummer spheres with scattered h.
"""
import math

import numpy as np
import torch

from cosmosphere_b200 import capi

GAMMA, BETA, ALPHAU, TOLH = 5.0 / 3.0, 2.0, 1.0, 1e-4
UNIT_BOX = [0.0, 1.0, 0.0, 1.0, 0.0, 1.0]
EPS = 2.220446049250313e-16


def listed():
    step = lambda name, gen, n, **kw: {"name": name, "kind": "step", "gen": gen, "n": n, "quintic": False,
                                       "mixed": False, "disc": False, **kw}
    return [
        # the smallest set a driver runs: launches and host round trips are its whole cost
        step("lattice_8", "lattice", 672),
        # a small periodic box, random (Poisson) neighbours: every h has to move
        step("box_20k", "box", 20011),
        # an ordinary disc / sphere run: open, centrally concentrated, disc viscosity
        step("plummer_120k_disc", "plummer", 120017, disc=True),
        # an ordinary periodic box in the mixed-precision form
        step("box_300k_mixed", "box", 300007, mixed=True),
        # the headline workload (lattice 100, 1% jiggle, 1.403 M particles), a run's first step
        step("lattice_100", "lattice", 1403000),
        # the same in the mixed-precision form
        step("lattice_100_mixed", "lattice", 1403000, mixed=True),
        # the same set in mid-run: drifted positions, h from the previous step
        step("lattice_100_warm", "warm", 1403000),
        # the largest single set: Plummer sphere, quintic kernel, h scattered log-normally
        step("plummer_2m_quintic", "plummer", 2000000, quintic=True),
        # ensembles of boxes and spheres, sizes log-uniform over the range users batch
        {"name": "batch_24", "kind": "batch", "nsets": 24, "nmin": 10000, "nmax": 120000, "sizes": 42, "mixed": False},
        {"name": "batch_40_mixed", "kind": "batch", "nsets": 40, "nmin": 10000, "nmax": 300000, "sizes": 43,
         "mixed": True},
        # a burst on the server: new sets of every kind and continuations of some
        {"name": "serve_10", "kind": "serve", "nreq": 10, "ncont": 4, "nmin": 5000, "nmax": 200000, "sizes": 42},
        # a tree code's own key sort, near the largest set the fixed scratch takes
        {"name": "order_500k", "kind": "order", "n": 500009},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "batch", "serve", "order"], weights=[7, 3, 1, 1])[0]
    if kind == "step":
        gen = rng.choice(["lattice", "warm", "box", "plummer"])
        quintic = rng.random() < 0.3
        n = _log_uniform(rng, 700 if gen in ("lattice", "warm") else 5000, 1000000 if gen == "plummer" else 1500000)
        return {"kind": "step", "gen": gen, "n": n, "quintic": quintic, "mixed": rng.random() < 0.3,
                "disc": rng.random() < 0.25}
    if kind == "batch":
        nmin = _log_uniform(rng, 5000, 20000)
        return {"kind": "batch", "nsets": rng.randint(5, 40), "nmin": nmin, "nmax": _log_uniform(rng, 2 * nmin, 150000),
                "sizes": rng.randrange(1 << 30), "mixed": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": "serve", "nreq": rng.randint(4, 10), "ncont": rng.randint(1, 4), "nmin": 5000,
                "nmax": _log_uniform(rng, 20000, 200000), "sizes": rng.randrange(1 << 30)}
    return {"kind": "order", "n": _log_uniform(rng, 1000, 524288)}


# ------------------------------------------------------------------ particle sets
def _lattice_dims(n):
    """The close-packed lattice of about n particles: its particles per side, rows, layers."""
    npx = max(4, int(round((n / 1.403) ** (1.0 / 3.0))))
    return npx, int(npx * 2.0 / math.sqrt(3.0)), int(npx * 3.0 / math.sqrt(6.0))


def _count(gen, n):
    if gen in ("lattice", "warm"):
        npx, ny, nz = _lattice_dims(n)
        return npx * ny * nz
    return n


def _set(gen, n, quintic, seed):
    """One particle set: pos (3, n), h (n), vel and acc (3, n), thermo (4, n), pmass, box, hfact."""
    rng = np.random.default_rng([int(seed), int(n), ["lattice", "warm", "box", "plummer", "sphere"].index(gen)])
    hfact = 1.0 if quintic else 1.2
    box, u0, vsig = None, 1.0, 0.1
    if gen in ("lattice", "warm"):
        npx, ny, nz = _lattice_dims(n)
        n = npx * ny * nz
        dx = 1.0 / npx
        dy, dz = dx * math.sqrt(3.0) / 2.0, dx * math.sqrt(6.0) / 3.0
        k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(npx), indexing="ij")
        pos = np.stack([(i * dx + ((j + k) % 2) * 0.5 * dx).ravel(), (j * dy + (k % 2) * dy / 3.0).ravel(),
                        (k * dz).ravel()])
        if gen == "lattice":
            h = np.full(n, hfact * dx)
            few = rng.permutation(n)[: max(1, n // 100)]
            h[few] *= rng.uniform(0.65, 1.35, few.size)
        else:
            # h of the lattice's own density (sqrt(2) particles per dx^3), a step's drift off
            pos += 0.03 * dx * rng.standard_normal((3, n))
            h = hfact * dx / 2.0 ** (1.0 / 6.0) * (1.0 + 0.01 * rng.standard_normal(n))
    elif gen == "box":
        box = list(UNIT_BOX)
        pos = rng.random((3, n))
        h = hfact * n ** (-1.0 / 3.0) * rng.uniform(0.8, 1.2, n)
    else:
        # Plummer sphere (scale radius 1, total mass 1) inside r < 20; |v| = 0.5 v_circ; h off
        # log-normally (plummer) or by up to 20% (sphere, the ensembles' own)
        top = (20.0 ** 3) / (1.0 + 20.0 ** 2) ** 1.5
        r = 1.0 / np.sqrt((rng.random(n) * top) ** (-2.0 / 3.0) - 1.0)
        mu, phi = rng.uniform(-1.0, 1.0, n), rng.uniform(0.0, 2.0 * math.pi, n)
        s = np.sqrt(1.0 - mu * mu)
        pos = r * np.stack([s * np.cos(phi), s * np.sin(phi), mu])
        dens = 3.0 / (4.0 * math.pi) * (1.0 + r * r) ** -2.5 / top
        h = hfact * (n * dens) ** (-1.0 / 3.0)
        h = h * (np.exp(0.3 * rng.standard_normal(n)) if gen == "plummer" else rng.uniform(0.8, 1.2, n))
        u0, vsig = 0.05, 0.5 * np.sqrt(r * r / (1.0 + r * r) ** 1.5 / 3.0)
    vel = vsig * rng.standard_normal((3, n))
    acc = 0.1 * rng.standard_normal((3, n))
    pmass = 1.0 / n
    u = u0 * rng.uniform(0.9, 1.1, n)
    rho = pmass * (hfact / h) ** 3
    thermo = np.stack([(GAMMA - 1.0) * u / rho, np.sqrt(GAMMA * (GAMMA - 1.0) * u), rng.uniform(0.1, 1.0, n), u])
    return {"n": n, "pos": pos, "h": h, "vel": vel, "acc": acc, "thermo": thermo, "pmass": pmass, "box": box,
            "hfact": hfact}


def _batch_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    return np.rint(np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["nsets"]))).astype(int)


def _batch_sets(case, seed):
    """Even sets in the unit periodic box, odd ones open Plummer spheres."""
    return [_set("sphere" if k % 2 else "box", int(n), False, seed * 1000 + k)
            for k, n in enumerate(_batch_sizes(case))]


def _serve_plan(case):
    """(generator, n) of each new request, and the requests the continuations extend."""
    rng = np.random.default_rng(case["sizes"])
    sizes = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["nreq"]))
    new = [(["lattice", "box", "plummer"][k % 3], int(round(v))) for k, v in enumerate(sizes)]
    return new, [int(v) for v in rng.permutation(case["nreq"])[: min(case["ncont"], case["nreq"])]]


def _serve_sets(case, seed):
    new, cont = _serve_plan(case)
    sets = [_set(g, n, False, seed * 1000 + k) for k, (g, n) in enumerate(new)]
    for p in sets:
        p["dt"] = 0.1 * float(np.min(p["h"] / p["thermo"][1]))
    return sets, cont


# ------------------------------------------------------------------ prepare and run
def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


_server = []


def prepare(case, seed):
    if case["kind"] == "step":
        p = _set(case["gen"], case["n"], case["quintic"], seed)
        for k in ("pos", "h", "vel", "acc", "thermo"):
            p[k] = _pinned(p[k])
        n = p["n"]
        return {"case": case, "c": capi.Cosmo(case["quintic"]), "p": p,
                "out": {k: _pinned(np.zeros((nc, n))) for k, nc in
                        (("h", 1), ("dens", 2), ("grad", 3), ("force", 6))}}
    if case["kind"] == "batch":
        sets = [{"x": p["pos"][0], "y": p["pos"][1], "z": p["pos"][2], "h": p["h"], "pmass": p["pmass"],
                 "box": p["box"]} for p in _batch_sets(case, seed)]
        return {"case": case, "c": capi.Cosmo(), "b": capi.Batch(sets)}
    if case["kind"] == "serve":
        if not _server:
            capi.Cosmo().set_precision(False)
            _server.append(capi.Server(slots=4, budget_gb=60.0))
        sets, cont = _serve_sets(case, seed)
        req = [({"x": p["pos"][0], "y": p["pos"][1], "z": p["pos"][2], "vx": p["vel"][0], "vy": p["vel"][1],
                 "vz": p["vel"][2], "h": p["h"], "pmass": p["pmass"]}, p["thermo"], p["box"], p["dt"]) for p in sets]
        return {"case": case, "server": _server[0], "req": req, "cont": cont}
    p = _set("plummer", case["n"], False, seed)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return {"case": case, "c": capi.Cosmo(), "x": dev(p["pos"][0]), "y": dev(p["pos"][1]), "z": dev(p["pos"][2]),
            "h": dev(p["h"]), "keys": torch.empty(case["n"], dtype=torch.int64, device="cuda"),
            "order": torch.empty(case["n"], dtype=torch.int32, device="cuda")}


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        c, p, out = state["c"], state["p"], state["out"]
        n = p["n"]
        c.set_precision(case["mixed"])
        c.arrays_init(n)
        c.upload(capi.POS, p["pos"], n)
        c.upload(capi.HSML, p["h"], n)
        c.upload(capi.VEL, p["vel"], n)
        c.upload(capi.ACCEL, p["acc"], n)
        c.density(n, p["pmass"], periodic_box=p["box"], tolh=TOLH, hfact=p["hfact"])
        c.upload(capi.THERMO, p["thermo"], n, sorted_=True)
        c.force(n, p["pmass"], beta=BETA, alphau=ALPHAU, disc=1 if case["disc"] else 0)
        c.download(capi.HSML, n, out["h"])
        c.download(capi.DENS_OUT, n, out["dens"])
        c.download(capi.GRAD_OUT, n, out["grad"])
        c.download(capi.FORCE_OUT, n, out["force"])
        return out
    if case["kind"] == "batch":
        state["c"].set_precision(case["mixed"])
        b = state["b"]
        b.upload()
        b.density(tolh=TOLH, hfact=1.2, final_rho=True)
        h, rho, gradh = b.download()
        return {"h": np.concatenate(h), "rho": np.concatenate(rho), "gradh": np.concatenate(gradh)}
    if case["kind"] == "serve":
        s = state["server"]
        ids = [s.submit(p, th, box=box, tolh=TOLH, hfact=1.2, beta=BETA, alphau=ALPHAU, keep=True)
               for p, th, box, _ in state["req"]]
        more = [s.cont(ids[k], state["req"][k][3]) for k in state["cont"]]
        out = [s.wait(r)[1] for r in ids + more]
        for r in ids:
            s.release(r)
        return out
    n = case["n"]
    state["c"].hilbert_order_noalloc(n, *(state[k].data_ptr() for k in ("x", "y", "z", "h", "keys", "order")))
    return {"keys": state["keys"], "order": state["order"]}


# ------------------------------------------------------------------ the work of one pass
# Per particle of a step: 14 doubles up, 12 down (through the host's arrays, once each).
# Flops: the accepted pairs' arithmetic of one Newton evaluation at least (30 a pair), the
# gradient sweep (80) and the force pass (110), at the neighbour count of the kernel.
def _pairs(n, quintic):
    return n * 4.0 / 3.0 * math.pi * (3.0 if quintic else 2.4) ** 3


def work(case):
    if case["kind"] == "step":
        n = _count(case["gen"], case["n"])
        return {"bytes": 26 * 8 * n, "flops": 220 * _pairs(n, case["quintic"])}
    if case["kind"] == "batch":
        n = int(_batch_sizes(case).sum())
        return {"bytes": 7 * 8 * n, "flops": 60 * _pairs(n, False)}
    if case["kind"] == "serve":
        new, cont = _serve_plan(case)
        sizes = [_count(g, n) for g, n in new]
        more = sum(sizes[k] for k in cont)
        return {"bytes": 8 * (23 * sum(sizes) + 12 * more), "flops": 220 * _pairs(sum(sizes) + more, False)}
    return {"bytes": (4 * 8 + 8 + 4) * case["n"], "flops": 0}


# ------------------------------------------------------------------ 64-bit values
# Plain torch on the same inputs: cell grids for the neighbours (one per band of h, so that
# a wide range of h keeps its cells small), sums by index_add_.
class _Near:
    """For particles i with search radius R h_i: chunks (i, j, dx, dy, dz, r2) with r < R h_i."""

    def __init__(self, pos, box, R):
        self.pos, self.R = pos, R
        self.len = None if box is None else torch.tensor([box[1] - box[0], box[3] - box[2], box[5] - box[4]],
                                                         dtype=torch.float64, device=pos.device)
        self.lo = pos.amin(1) if box is None else torch.tensor(box[0::2], dtype=torch.float64, device=pos.device)
        self.span = pos.amax(1) - self.lo if box is None else self.len

    def __call__(self, idx, h, most=24_000_000):
        hi = h[idx]
        band = torch.floor(torch.log(hi / hi.min()) / math.log(1.25)).to(torch.int64)
        for b in torch.unique(band).tolist():
            yield from self._band(idx[band == b], h, most)

    def _band(self, idx, h, most):
        pos, dev = self.pos, self.pos.device
        cell = float(h[idx].max()) * self.R * (1.0 + 1e-9)
        nc = torch.clamp(torch.floor(self.span / cell), 1, 1 << 20).to(torch.int64)
        size = self.span / nc
        if self.len is not None and int(nc.min()) < 3:
            nc = torch.ones_like(nc)          # the box is a few cells wide: one cell, all pairs
            size = self.span / nc
        ic = torch.minimum(((pos - self.lo[:, None]) / size[:, None]).to(torch.int64).clamp_(min=0), (nc - 1)[:, None])
        key, order = torch.sort((ic[0] * nc[1] + ic[1]) * nc[2] + ic[2])
        offs = [(0, 0, 0)] if int(nc.max()) == 1 else [(a, b, c) for a in (-1, 0, 1) for b in (-1, 0, 1)
                                                      for c in (-1, 0, 1)]
        first, count = [], []
        for o in offs:
            c = ic[:, idx] + torch.tensor(o, device=dev)[:, None]
            if self.len is not None:
                c = c % nc[:, None]
            ok = ((c >= 0) & (c < nc[:, None])).all(0)
            k = (c[0] * nc[1] + c[1]) * nc[2] + c[2]
            a = torch.searchsorted(key, k)
            first.append(a)
            count.append(torch.where(ok, torch.searchsorted(key, k, right=True) - a, 0))
        first, count = torch.stack(first, 1), torch.stack(count, 1)
        ends = torch.cumsum(count.sum(1), 0)
        done, at = 0, 0
        while at < idx.numel():
            to = int(torch.searchsorted(ends, torch.tensor(done + most, device=dev)))
            to = min(max(to, at + 1), idx.numel())
            cnt = count[at:to].reshape(-1)
            tot = int(cnt.sum())
            row = torch.repeat_interleave(torch.arange(cnt.numel(), device=dev), cnt)
            start = torch.cumsum(cnt, 0) - cnt
            j = order[first[at:to].reshape(-1)[row] + torch.arange(tot, device=dev) - start[row]]
            i = idx[at:to][row // len(offs)]
            d = pos[:, i] - pos[:, j]
            if self.len is not None:
                d = d - self.len[:, None] * torch.round(d / self.len[:, None])
            r2 = (d * d).sum(0)
            m = r2 < (self.R * h[i]) ** 2
            yield i[m], j[m], d[0][m], d[1][m], d[2][m], r2[m]
            done, at = int(ends[to - 1]), to


def _kernel(q, quintic):
    """W and dW/dq, unnormalised, for q inside the support."""
    if quintic:
        a, b, c = torch.clamp(3 - q, min=0), torch.clamp(2 - q, min=0), torch.clamp(1 - q, min=0)
        return a ** 5 - 6 * b ** 5 + 15 * c ** 5, -5 * a ** 4 + 30 * b ** 4 - 75 * c ** 4
    a, b = torch.clamp(2 - q, min=0), torch.clamp(1 - q, min=0)
    return 0.25 * a ** 3 - b ** 3, -0.75 * a ** 2 + 3 * b ** 2


def _norm(quintic):
    return 1.0 / (120.0 * math.pi) if quintic else 1.0 / math.pi


def _sums(near, idx, h, quintic):
    rho, gra = torch.zeros_like(h), torch.zeros_like(h)
    for i, _, _, _, _, r2 in near(idx, h):
        q = torch.sqrt(r2) / h[i]
        w, dw = _kernel(q, quintic)
        rho.index_add_(0, i, w)
        gra.index_add_(0, i, -q * dw - 3.0 * w)
    return rho[idx], gra[idx]


def _density(near, h, pmass, hfact, quintic):
    """The Newton-Raphson solve: converged h."""
    h = h.clone()
    idx = torch.arange(h.numel(), device=h.device)
    for _ in range(100):
        sr, sg = _sums(near, idx, h, quintic)
        hi = h[idx]
        rho, gra = sr * _norm(quintic) * pmass / hi ** 3, sg * _norm(quintic) * pmass / hi ** 4
        rhoh = pmass * (hfact / hi) ** 3
        dh = -hi / (3.0 * rhoh)
        om = 1.0 - dh * gra
        new = hi - (rhoh - rho) * dh / torch.where(om > 0, om, torch.abs(om + 1e-300))
        new = torch.minimum(torch.maximum(new, 0.8 * hi), 1.2 * hi)
        h[idx] = new
        idx = idx[~(torch.abs((new - hi) / hi) < TOLH)]
        if not idx.numel():
            return h
    return None


def _step(pos, h, vel, acc, thermo, pmass, box, hfact, quintic, disc):
    """One density + force step: (h, dens (2, n), grad (3, n), force (6, n))."""
    R, norm = (3.0 if quintic else 2.0), _norm(quintic)
    near = _Near(pos, box, R)
    h = _density(near, h, pmass, hfact, quintic)
    if h is None:
        return None
    n = h.numel()
    every = torch.arange(n, device=h.device)
    z = lambda k: torch.zeros((k, n), dtype=torch.float64, device=h.device)
    sr, sg = _sums(near, every, h, quintic)
    rho, gra = sr * norm * pmass / h ** 3, sg * norm * pmass / h ** 4
    pro2, cs, alpha, u = thermo
    rhoh = pmass * (hfact / h) ** 3
    om = 1.0 + h / (3.0 * rhoh) * gra
    oinv = torch.where(om > 0, 1.0 / om, torch.ones_like(om))
    grk, pr, auterm = norm * oinv / h ** 4, pro2 * rhoh * rhoh, 0.5 * pmass / rhoh * ALPHAU
    dv, da, rm, divs = z(9), z(9), z(6), z(1)[0]
    f, f4, vs, divf = z(3), z(1)[0], z(1)[0], z(1)[0]
    for i, j, dx, dy, dz, r2 in near(every, h):
        m = r2 > 0
        i, j, dx, dy, dz, r2 = i[m], j[m], dx[m], dy[m], dz[m], r2[m]
        r = torch.sqrt(r2)
        _, dw = _kernel(r / h[i], quintic)
        e = [dx / r, dy / r, dz / r]
        d = [dx, dy, dz]
        dvel = [vel[k][i] - vel[k][j] for k in range(3)]
        dacc = [acc[k][i] - acc[k][j] for k in range(3)]
        for a in range(3):
            for b in range(3):
                dv[3 * a + b].index_add_(0, i, dvel[a] * e[b] * dw * pmass)
                da[3 * a + b].index_add_(0, i, dacc[a] * e[b] * dw * pmass)
        for k, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
            rm[k].index_add_(0, i, -d[a] * e[b] * dw * pmass)
        pv = dvel[0] * e[0] + dvel[1] * e[1] + dvel[2] * e[2]
        divs.index_add_(0, i, pv * dw * pmass)
        # the pair's terms with W at h_i: the i-side terms act on i, the same as j-side terms on j
        top = torch.maximum(torch.clamp(cs[i] - BETA * pv, min=0), torch.clamp(cs[j] - BETA * pv, min=0))
        vs.scatter_reduce_(0, i, top, "amax")
        vs.scatter_reduce_(0, j, top, "amax")
        if disc:
            near_v = torch.where(pv < 0, alpha[i] * cs[i] - BETA * pv, alpha[i] * cs[i])
            q = -0.5 / rhoh[i] * near_v * (h[i] / r) * pv
            diss = -0.5 * pmass / rhoh[i] * alpha[i] * cs[i] * (h[i] / r) * pv * pv
        else:
            q = torch.where(pv < 0, -0.5 / rhoh[i] * torch.clamp(alpha[i] * cs[i] - BETA * pv, min=0) * pv,
                            torch.zeros_like(pv))
            diss = pmass * q * pv
        g = dw * grk[i]
        gp = pmass * (pro2[i] + q) * g
        for k in range(3):
            f[k].index_add_(0, i, -gp * e[k])
            f[k].index_add_(0, j, gp * e[k])
        cond = torch.sqrt(torch.abs(pr[i] - pr[j]) * 2.0 / (rhoh[i] + rhoh[j])) * (u[i] - u[j]) * auterm[i] * g
        f4.index_add_(0, i, pmass * pro2[i] * pv * g + diss * g + cond)
        f4.index_add_(0, j, -cond)
        divf.index_add_(0, i, pmass * dw * pv)
    # the gradient sweep's finish: linear-exact velocity and acceleration gradients
    omg = 1.0 + h / (3.0 * rho) * gra
    term = norm * torch.where(omg > 0, 1.0 / omg, torch.ones_like(omg)) / h ** 4 / rho
    M = torch.stack([torch.stack([rm[0], rm[1], rm[2]]), torch.stack([rm[1], rm[3], rm[4]]),
                     torch.stack([rm[2], rm[4], rm[5]])]).permute(2, 0, 1)
    inv = torch.linalg.inv(M)
    gv = -torch.einsum("anp,npb->anb", dv.reshape(3, 3, n).permute(0, 2, 1), inv).permute(0, 2, 1)
    ga = -torch.einsum("anp,npb->anb", da.reshape(3, 3, n).permute(0, 2, 1), inv).permute(0, 2, 1)
    gf = gv.float().double()
    curl = (gf[2][1] - gf[1][2]) ** 2 + (gf[0][2] - gf[2][0]) ** 2 + (gf[1][0] - gf[0][1]) ** 2
    comp = torch.clamp(-(gf[0][0] + gf[1][1] + gf[2][2]), min=0) ** 2
    xi = torch.where(comp + curl > EPS, comp / (comp + curl), torch.ones_like(comp))
    ddt = ga[0][0] + ga[1][1] + ga[2][2] - (gv[0][0] ** 2 + gv[1][1] ** 2 + gv[2][2] ** 2 + 2.0 * (
        gv[0][1] * gv[1][0] + gv[0][2] * gv[2][0] + gv[1][2] * gv[2][1]))
    return (h, torch.stack([rho, gra]), torch.stack([-divs * term, xi, ddt]),
            torch.stack([f[0], f[1], f[2], f4, vs, -divf * norm * oinv / h ** 4 / rhoh]))


def _host(*arrays):
    return [a.cpu().numpy() for a in arrays]


def _exact_set(p, quintic, disc):
    d = {k: torch.from_numpy(np.ascontiguousarray(p[k])).cuda() for k in ("pos", "h", "vel", "acc", "thermo")}
    return _step(d["pos"], d["h"], d["vel"], d["acc"], d["thermo"], p["pmass"], p["box"], p["hfact"], quintic, disc)


def exact(case, seed):
    if case["kind"] == "order" or (case["kind"] == "step" and case["gen"] == "plummer" and case["n"] > 250000):
        return None
    if case["kind"] == "step":
        r = _exact_set(_set(case["gen"], case["n"], case["quintic"], seed), case["quintic"], case["disc"])
        if r is None:
            return None
        h, dens, grad, force = _host(*r)
        return {"h": h[None, :], "dens": dens, "grad": grad, "force": force}
    if case["kind"] == "batch":
        out = []
        for p in _batch_sets(case, seed):
            near = _Near(torch.from_numpy(p["pos"]).cuda(), p["box"], 2.0)
            h = _density(near, torch.from_numpy(p["h"]).cuda(), p["pmass"], 1.2, False)
            if h is None:
                return None
            sr, sg = _sums(near, torch.arange(h.numel(), device=h.device), h, False)
            out.append(_host(h, sr * _norm(False) * p["pmass"] / h ** 3, sg * _norm(False) * p["pmass"] / h ** 4))
        return {k: np.concatenate([o[a] for o in out]) for a, k in enumerate(("h", "rho", "gradh"))}
    sets, cont = _serve_sets(case, seed)
    for p in sets:
        p["acc"] = np.zeros_like(p["vel"])   # the server takes no accelerations
    first = [_exact_set(p, False, False) for p in sets]
    more = []
    for k in cont:
        p = sets[k]
        if first[k] is None:
            return None
        p["pos"] = p["pos"] + p["vel"] * p["dt"]
        if p["box"] is not None:
            p["pos"] = np.where(p["pos"] >= 1.0, p["pos"] - 1.0, np.where(p["pos"] < 0.0, p["pos"] + 1.0, p["pos"]))
        p["h"] = first[k][0].cpu().numpy()
        more.append(_exact_set(p, False, False))
    if any(r is None for r in first + more):
        return None
    return [dict(zip(("h", "dens", "grad", "force"), _host(*r))) for r in first + more]
