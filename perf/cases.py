"""The calls a program makes on this engine, at the sizes it makes them, for timing and comparison.

A case describes a handle (which system, how many particles, precision) and
what one pass does with it through readdygpu_b200.Engine:

  edits        apply_edits with that many deletions and as many new particles
  upload       set_particles from the host buffers
  steps        step(steps)
  observables  forces(), metrics() and an RDF frame
  rdf          an RDF frame, 200 bins over 0-20 nm
  (always)     get_particles into the program's page-locked buffers

Systems ("system"): the particle types, potentials, densities and box shapes
of readdygpu_b200.configs at any size.

  plain    2 species, harmonic repulsion, one periodic cube (configuration 1)
  batch    "systems" such cubes of 500 .. 20,000 particles, sizes and volume
           fractions drawn as in configuration 4
  mixed    4 species, repulsion + weak attraction, a disk, z open (2)
  spheres  identical spheres at volume fraction 0.30 (3)
  vesicle  3 species in a spherical membrane, all axes open (5)

"tuned": the program calls autotune() once after its first upload, as the
JNI frame loop does; otherwise the handle keeps its default search.
"""
import math

import numpy as np
import torch

import readdygpu_b200 as R
from readdygpu_b200 import configs

RDF_BINS, RDF_MAX = 200, 20.0           # the RDF of configuration 3
OBS_BINS, OBS_MAX = 100, 12.0           # a several-species RDF frame
SKIN = 1.4                              # pair-list margin of exact()


def _case(name, system, n, precision, steps, systems=1, **more):
    c = {"system": system, "n": n, "systems": systems, "precision": precision, "steps": steps, "tuned": True,
         "upload": False, "edits": 0, "rdf": False, "observables": False}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a program that handles reactions after every step: the smallest call
        _case("step1_plain_1k_f32c", "plain", 1000, "f32c", 1),
        # the drop-in's frame on the smallest configuration, FP64 as the Java core computes
        _case("frame_plain_1k_f64", "plain", 1000, "f64", 100),
        # a script that never calls autotune: short calls on the default search, an odd size
        _case("default_plain_8k_f32c", "plain", 7919, "f32c", 100, tuned=False),
        # the drop-in's frame at the size of the largest system of the ensemble
        _case("frame_plain_20k_f64", "plain", 20000, "f64", 100),
        # the reaction loop: edits on the device, a short frame, positions to the host
        _case("reactions_plain_30k_f32c", "plain", 30011, "f32c", 10, edits=24),
        # observables of a several-species run, evaluated every 10 steps
        _case("observables_vesicle_60k_f64", "vesicle", 60013, "f64", 10, observables=True),
        # a host-driven frame: upload, 100 steps, download; open z, weak attraction, disk
        _case("upload_mixed_100k_f32c", "mixed", 100000, "f32c", 100, upload=True),
        # the vesicle's production frame
        _case("frame_vesicle_250k_f32c", "vesicle", 250000, "f32c", 100),
        # the sphere fluid with its RDF every 100 steps
        _case("rdf_spheres_1m_f32c", "spheres", 1000000, "f32c", 100, rdf=True),
        # a small ensemble in FP64
        _case("batch_64_f64", "batch", 0, "f64", 100, systems=64),
        # an ensemble driven from the host with short frames
        _case("upload_batch_160_f32c", "batch", 0, "f32c", 20, systems=160, upload=True),
        # the full ensemble: the largest call
        _case("frame_batch_512_f32c", "batch", 0, "f32c", 100, systems=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: any system, size, precision and kind of pass."""
    system = rng.choice(["plain", "plain", "mixed", "spheres", "vesicle", "batch", "batch"])
    precision = rng.choice(["f32c", "f32c", "f64"])
    top = {"plain": 120000, "mixed": 120000, "spheres": 1000000, "vesicle": 250000, "batch": 0}[system]
    if precision == "f64":
        top //= 2
    n = _log(rng, 500, top) if top else 0
    if system == "mixed":
        n = max(n, 2000)
    systems = _log(rng, 4, 400 if precision == "f32c" else 160) if system == "batch" else 1
    kind = rng.choice(["frame", "frame", "short", "upload", "rdf", "edits", "observables"])
    if system == "batch" and kind in ("edits", "rdf", "observables"):
        kind = "frame"
    if system == "mixed":                # clusters as it runs: every pass starts over
        kind = "upload"
    c = _case(None, system, n, precision, _log(rng, 20, 100), systems=systems)
    c["tuned"] = kind == "edits" or rng.random() < 0.85
    if not c["tuned"]:
        c["n"], c["systems"] = min(n, 60000), min(systems, 40)
    if kind == "short":
        c["steps"] = _log(rng, 1, 12)
    elif kind == "upload":
        c["upload"] = True
    elif kind == "rdf":                  # a periodic box wider than 2.5 times the range
        c["rdf"], c["n"] = True, max(c["n"], 2000)
    elif kind == "edits":
        c["system"], c["n"], c["edits"], c["steps"] = "plain", _log(rng, 2000, 60000), _log(rng, 2, 60), 10
    elif kind == "observables":
        c["n"], c["observables"], c["steps"] = min(n, 60000), True, 10
    return c


# ---- inputs -----------------------------------------------------------------

def _cube(n, density):
    return R.float_exact_box((n / density) ** (1.0 / 3.0))


def _sized(w, L):
    """The configuration's system in a periodic cube of edge L."""
    w.system.lo, w.system.hi = (0.0, 0.0, 0.0), (L, L, L)
    return w.system


def _ensemble(systems):
    """Particle numbers and box edges of an ensemble's systems, the same for every seed."""
    rng = np.random.default_rng(systems)
    Ns = np.rint(np.exp(rng.uniform(math.log(500), math.log(20000), systems))).astype(np.int64)
    vbar = 4.0 / 3.0 * math.pi * (1.5 ** 3 + 2.0 ** 3) / 2.0
    return Ns, [_cube(a, phi / vbar) for a, phi in zip(Ns, rng.uniform(0.1, 0.3, systems))]


def _inputs(case, seed):
    """(system, boxes or None, offsets or None, xyz, types), coordinates in FP32 as the frames of the reference."""
    rng = np.random.default_rng([seed, case["n"], case["systems"]])
    kind, n = case["system"], case["n"]
    boxes = offsets = None
    if kind == "plain":
        L = _cube(n, 1000 / 50.0 ** 3)
        sys_ = _sized(configs.config1(4), L)
        xyz, types = rng.uniform(0, L, (n, 3)), (np.arange(n) % 2).astype(np.int32)
    elif kind == "batch":
        Ns, Ls = _ensemble(case["systems"])
        sys_ = _sized(configs.config1(4), 1.0)
        boxes = [((0.0, 0.0, 0.0), (L, L, L), (1, 1, 1), seed * 1000003 + k) for k, L in enumerate(Ls)]
        offsets = np.concatenate([[0], np.cumsum(Ns)]).astype(np.int64)
        xyz = rng.uniform(0, 1, (int(offsets[-1]), 3)) * np.repeat(Ls, Ns)[:, None]
        types = np.concatenate([(np.arange(a) >= a // 2).astype(np.int32) for a in Ns])
    elif kind == "mixed":
        # configuration 2's density: the box shrinks with the particle number
        h = R.float_exact_box(200.0 * (n / 100000.0) ** (1.0 / 3.0))
        sys_ = configs.config2(4).system
        sys_.lo, sys_.hi = (-h, -h, -0.5 * h), (h, h, 0.5 * h)
        sys_.external[0].radius = 0.75 * h
        xyz = rng.uniform(sys_.lo, sys_.hi, (n, 3))
        types = (np.arange(n) * 4 // n).astype(np.int32)
    elif kind == "spheres":
        L = _cube(n, 0.30 / (4.0 / 3.0 * math.pi * 8.0))
        sys_ = configs.config3(1, rsa=lambda *a: np.zeros((1, 3))).system
        sys_.hi = (L, L, L)
        # a cubic lattice with every site shaken, without overlap at full occupancy
        m = math.ceil(n ** (1.0 / 3.0))
        site = rng.permutation(m ** 3)[:n]
        ijk = np.stack([site % m, (site // m) % m, site // (m * m)], 1)
        xyz = (ijk + 0.5) * (L / m) + rng.uniform(-0.3, 0.3, (n, 3))
        types = np.zeros(n, np.int32)
    else:
        # configuration 5's density and shell share
        f = (n / 250000.0) ** (1.0 / 3.0)
        radius = 120.0 * f
        sys_ = configs.config5(8, n_shell=2).system
        h = R.float_exact_box(radius + 10.0)
        sys_.lo, sys_.hi = (-h, -h, -h), (h, h, h)
        for e in sys_.external:
            e.radius = radius
        shell = max(1, int(n * 0.06))
        u = rng.normal(size=(n, 3))
        u /= np.linalg.norm(u, axis=1, keepdims=True)
        r = np.full(n, radius)
        r[: n - shell] = (radius - 1.0) * rng.uniform(0, 1, n - shell) ** (1.0 / 3.0)
        xyz = u * r[:, None]
        types = np.concatenate([np.arange(n - shell) % 2, np.full(shell, 2)]).astype(np.int32)
    xyz = xyz.astype(np.float32)
    for a in range(3):
        if boxes is None and sys_.periodic[a]:
            top = np.float32(sys_.hi[a])
            xyz[:, a][xyz[:, a] >= top] = np.float32(sys_.lo[a])
    if boxes is not None:
        top = np.repeat(np.float32(Ls), Ns)[:, None]
        xyz[xyz >= top] = 0.0
    return sys_, boxes, offsets, xyz, types


def _edits(case, sys_, seed):
    """One frame's reaction edits: rows (id, new type, x, y, z, index); deletions, then as many new particles."""
    k, rng = case["edits"], np.random.default_rng([seed, 77])
    e = np.zeros((2 * k, 6), np.float32)
    e[:k, 1] = -1
    e[:k, 5] = rng.choice(case["n"], k, replace=False)
    e[k:, 1] = rng.integers(0, sys_.n_types, k)
    e[k:, 2:5] = rng.uniform(sys_.lo, sys_.hi, (k, 3))
    e[k:, 5] = -1
    return e


def _seed64(seed):
    return 1000 + seed


def prepare(case, seed):
    sys_, boxes, offsets, xyz, types = _inputs(case, seed)
    real = np.float32 if case["precision"] == "f32c" else np.float64
    n = types.size
    pinned = torch.cuda.is_available()

    def host(shape, dtype, fill=None):
        a = torch.empty(shape, dtype=dtype, pin_memory=pinned).numpy()
        if fill is not None:
            a[...] = fill
        return a

    ft = torch.float32 if real is np.float32 else torch.float64
    s = {"case": case, "offsets": offsets,
         "x": host((n, 3), ft), "t": host((n,), torch.int32),
         "x0": host((n, 3), ft, xyz), "t0": host((n,), torch.int32, types),
         "edits": _edits(case, sys_, seed) if case["edits"] else None}
    e = R.Engine(sys_, precision=case["precision"], seed=_seed64(seed), boxes=boxes)
    e.set_particles(s["x0"], s["t0"], offsets=offsets)
    if case["tuned"]:
        e.autotune()
    s["engine"] = e
    return s


def run(s):
    e, case = s["engine"], s["case"]
    out = {}
    if case["upload"]:
        e.set_particles(s["x0"], s["t0"], offsets=s["offsets"])
    if case["edits"]:
        e.apply_edits(s["edits"])
    e.step(case["steps"])
    out["xyz"], out["types"] = e.get_particles(s["x"], s["t"])
    if case["rdf"]:
        counts, _ = e.rdf(RDF_BINS, RDF_MAX, accumulate=False)
        out["rdf"] = counts.view(np.int64)
    if case["observables"]:
        out["forces"], out["energy"] = e.forces()
        m = e.metrics()
        out["msd"] = np.array(m["msd"])
        counts, _ = e.rdf(OBS_BINS, OBS_MAX, accumulate=False)
        out["rdf"] = counts.view(np.int64)
    return out


# particles per nm^3 and the mean cutoff [nm], for the pair work
_DENSITY = {"plain": (0.008, 3.5), "batch": (0.008, 3.5), "mixed": (0.003125, 3.8), "spheres": (0.00895, 4.0),
            "vesicle": (0.0345, 2.1)}


def work(case):
    """Bytes: a step depends on every neighbour's last position, so each step reads and writes the 32-byte
    state of each particle once; uploads, downloads and observables once.  Operations: 30 per pair within the
    cutoff (each particle's own sum) and 150 for a particle's noise and update; 10 per RDF pair."""
    n = case["n"]
    if case["system"] == "batch":
        n = int(_ensemble(case["systems"])[0].sum())
    real = 4 if case["precision"] == "f32c" else 8
    frame = n * (3 * real + 4)
    rho, rc = _DENSITY[case["system"]]
    pairs = rho * 4.0 / 3.0 * math.pi * rc ** 3
    b = n * 64.0 * case["steps"] + frame * (2 if case["upload"] else 1)
    f = n * (30.0 * pairs + 150.0) * case["steps"]
    rmax = RDF_MAX if case["rdf"] else (OBS_MAX if case["observables"] else 0.0)
    if rmax:
        b += n * 4.0 * real
        f += 0.5 * n * rho * 4.0 / 3.0 * math.pi * rmax ** 3 * 10.0
    if case["observables"]:
        b += 2 * n * 32.0 + n * 24.0
        f += n * 30.0 * pairs
    return {"bytes": b, "flops": f}


# ---- the same pass in 64 bits, plain torch ----------------------------------

def _philox(c0, c1, step, key):
    """Philox4x32-10 words of the counters (c0, c1, step, 0); int64 tensors that hold 32-bit words."""
    mask = 0xFFFFFFFF

    def mul(m, c):
        p = m * (c & 0xFFFF)
        q = m * (c >> 16) + (p >> 16)
        return q >> 16, ((q & 0xFFFF) << 16) | (p & 0xFFFF)

    c = [c0, c1, torch.full_like(c0, step & mask), torch.zeros_like(c0)]
    k0, k1 = key & mask, (key >> 32) & mask
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return c


def _normals(index, key, step):
    u = [(w.double() + 0.5) * 2.0 ** -32 for w in _philox(index, torch.zeros_like(index), step, key)]
    ra, rb = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    a, b = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return torch.stack([ra * torch.cos(a), ra * torch.sin(a), rb * torch.cos(b)], 1)


class _Exact:
    """Brownian dynamics of one case in 64 bits: coordinates relative to the box, pairs from a cell grid."""

    def __init__(self, sys_, boxes, offsets, xyz, types, seed, device):
        self.sys, self.device = sys_, device
        d = lambda a, t=torch.float64: torch.as_tensor(np.asarray(a), dtype=t, device=device)  # noqa: E731
        n = types.size
        if boxes is None:
            boxes, offsets = [(sys_.lo, sys_.hi, sys_.periodic, seed)], np.array([0, n])
        counts = np.diff(offsets)
        which = np.repeat(np.arange(len(boxes)), counts)
        self.lo_s = d([b[0] for b in boxes])
        self.L_s = d([b[1] for b in boxes]) - self.lo_s
        self.per = d(boxes[0][2])
        self.sys_of = d(which, torch.int64)
        self.index = d(np.arange(n) - np.asarray(offsets)[which], torch.int64)
        self.key = d(np.array([b[3] for b in boxes], np.int64)[which], torch.int64)
        self.types = d(types, torch.int64)
        self.x = d(xyz) - self.lo_s[self.sys_of]
        self.x0 = self.x.clone()
        self.L = self.L_s[self.sys_of]
        S = sys_.n_types
        r0 = np.array([[sys_.pair_r0(i, j) for j in range(S)] for i in range(S)])
        self.hr0, self.k = d(r0).reshape(-1), sys_.pair[0].k
        self.cut = np.array(r0)
        self.weak = None
        for p in sys_.pair[1:]:
            on = np.zeros((S, S))
            for i, j in p.type_pairs:
                on[i, j] = on[j, i] = 1
                self.cut[i, j] = self.cut[j, i] = max(self.cut[i, j], p.r0 + p.length)
            self.weak = (d(on).reshape(-1) > 0, p)
        self.a = d([t.D * sys_.dt / (sys_.kB * sys_.T) for t in sys_.types])
        self.b = d([math.sqrt(2.0 * t.D * sys_.dt) for t in sys_.types])
        self.prad = d([t.radius for t in sys_.types])
        self.pairs = None
        self.step_no = 0

    def wrap(self):
        w = torch.floor(self.x / self.L) * self.per
        self.x = self.x - w * self.L
        return w

    def disp(self, i, j):
        dx = self.x[i] - self.x[j]
        return dx - torch.round(dx / self.L[i]) * self.L[i] * self.per

    def find_pairs(self):
        """Pairs i < j closer than the largest cutoff + SKIN."""
        r = float(self.cut.max()) + SKIN
        nc = torch.clamp(torch.floor(self.L_s / r), min=1).long()
        base = torch.cumsum(nc.prod(1), 0) - nc.prod(1)
        n3 = nc[self.sys_of]
        c = torch.clamp((self.x / self.L * n3).long(), min=0)
        c = torch.minimum(c, n3 - 1)
        flat = lambda q: base[self.sys_of] + (q[:, 2] * n3[:, 1] + q[:, 1]) * n3[:, 0] + q[:, 0]  # noqa: E731
        cell = flat(c)
        order = torch.argsort(cell)
        total = int(nc.prod(1).sum())
        count = torch.bincount(cell, minlength=total)
        start = torch.cumsum(count, 0) - count
        got = []
        few = (n3 < 3).any()
        for o in range(27):
            off = torch.tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device=self.device)
            q = c + off
            ok = ((q >= 0) & (q < n3) | (self.per > 0)).all(1)
            if few:                      # an axis of fewer than 3 cells reaches each of them once
                ok &= ~((n3 < 3) & ((q < 0) | (q >= n3))).any(1)
            cq = flat(torch.remainder(q, n3))
            m = torch.where(ok, count[cq], torch.zeros_like(cq))
            i = torch.repeat_interleave(torch.arange(len(m), device=self.device), m)
            first = torch.cumsum(m, 0) - m
            j = order[start[cq[i]] + torch.arange(len(i), device=self.device) - first[i]]
            keep = i < j
            i, j = i[keep], j[keep]
            keep = self.disp(i, j).square().sum(1) < r * r
            got.append(torch.stack([i[keep], j[keep]]))
        self.pairs = torch.cat(got, 1)
        self.ref = self.x.clone()
        self.tt = self.types[self.pairs[0]] * self.sys.n_types + self.types[self.pairs[1]]

    def forces(self):
        moved = None
        if self.pairs is not None:
            dx = self.x - self.ref
            dx = dx - torch.round(dx / self.L) * self.L * self.per
            moved = float(dx.square().sum(1).max().sqrt())
        if moved is None or moved > 0.5 * SKIN:
            self.find_pairs()
        i, j = self.pairs
        d = self.disp(i, j)
        r = d.square().sum(1).sqrt()
        over = r - self.hr0[self.tt]
        zero = torch.zeros_like(r)
        pre = torch.where((over < 0) & (r > 0), self.k * over / r, zero)
        e = torch.where(over < 0, 0.5 * self.k * over * over, zero).sum()
        if self.weak is not None:
            on, p = self.weak
            w, q, dep = on[self.tt], (2.0 / p.length) ** 2, p.depth
            s = r - p.r0
            z1, z2, z3 = s < 0, (s >= 0) & (s < 0.5 * p.length), (s >= 0.5 * p.length) & (s < p.length)
            f = torch.where(z1, p.k * s / r, torch.where(z2, dep * q * s / r, torch.where(
                z3, -dep * q * (s - p.length) / r, zero)))
            v = torch.where(z1, 0.5 * p.k * s * s - dep, torch.where(z2, 0.5 * dep * q * s * s - dep, torch.where(
                z3, -0.5 * dep * q * (s - p.length) ** 2, zero)))
            pre = pre + torch.where(w, f, zero)
            e = e + torch.where(w, v, zero).sum()
        F = torch.zeros_like(self.x)
        fd = -pre[:, None] * d
        F.index_add_(0, i, fd)
        F.index_add_(0, j, -fd)
        for p in self.sys.external:
            on = torch.zeros(self.sys.n_types, dtype=torch.bool, device=self.device)
            on[p.types] = True
            w = on[self.types].double()
            cen = torch.as_tensor(p.center, dtype=torch.float64, device=self.device) - self.lo_s[0]
            rel = self.x - cen
            pr = self.prad[self.types]
            if p.kind == R._abi.P1_DISK:            # attractive, normal z
                h, flat = rel[:, 2], rel.clone()
                flat[:, 2] = 0
                din = flat.square().sum(1).sqrt() + pr
                out = torch.clamp(din - p.radius, min=0)
                g = -(p.k * out / din)[:, None] * flat
                g[:, 2] -= p.k * h
                e = e + (w * 0.5 * p.k * (h * h + out * out)).sum()
            else:
                dist = rel.square().sum(1).sqrt()
                if p.subtype == "membrane":
                    rr, rad = dist - p.radius, dist
                else:
                    rr, rad = torch.clamp(dist + pr - p.radius, min=0), dist + pr
                g = -(p.k * rr / rad)[:, None] * rel
                e = e + (w * 0.5 * p.k * rr * rr).sum()
            F = F + w[:, None] * g
        return F, float(e)

    def step(self, n):
        for _ in range(n):
            F, _ = self.forces()
            xn = _normals(self.index, self.key, self.step_no)
            self.x = self.x + self.a[self.types][:, None] * F + self.b[self.types][:, None] * xn
            w = self.wrap()
            self.x0 = self.x0 - w * self.L          # keeps x - x0 the unwrapped displacement
            self.step_no += 1

    def edit(self, rows):
        rows = torch.as_tensor(rows, dtype=torch.float64, device=self.device)
        gone, new = rows[rows[:, 5] >= 0, 5].long(), rows[rows[:, 1] >= 0]
        keep = torch.ones(len(self.x), dtype=torch.bool, device=self.device)
        keep[gone] = False
        x = new[:, 2:5] - self.lo_s[0]
        self.x, self.x0 = torch.cat([self.x[keep], x]), torch.cat([self.x0[keep], x])
        self.types = torch.cat([self.types[keep], new[:, 1].long()])
        n = len(self.x)
        self.index = torch.arange(n, device=self.device)
        self.sys_of, self.key = torch.zeros_like(self.index), self.key[:1].expand(n)
        self.L, self.pairs = self.L_s[self.sys_of], None

    def absolute(self):
        return (self.x + self.lo_s[self.sys_of]).cpu().numpy()


def exact(case, seed):
    """The first pass on new inputs; None for the whole-number outputs, and where it would take too long."""
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    if work(case)["flops"] > (1.2e11 if device.type == "cuda" else 1.5e9):
        return None
    sys_, boxes, offsets, xyz, types = _inputs(case, seed)
    m = _Exact(sys_, boxes, offsets, xyz, types, _seed64(seed), device)
    if case["edits"]:
        m.edit(_edits(case, sys_, seed))
    m.step(case["steps"])
    out = {"xyz": m.absolute(), "types": None}
    if case["rdf"]:
        out["rdf"] = None
    if case["observables"]:
        F, e = m.forces()
        d2 = (m.x - m.x0).square().sum(1)
        out["forces"], out["energy"] = F.cpu().numpy(), e
        out["msd"] = np.array([float(d2[m.types == t].mean()) for t in range(sys_.n_types)])
        out["rdf"] = None
    return out
