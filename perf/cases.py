"""Performance cases of the slab-stepping core, over the range that its users run.

Every case goes through the package's public entry points: `_core.CudaSolver(...).run` (the drop-in
solver, FP64 or complex64 fields), `fast.run_3d` (the facade, set-up included),
`batch.Batch2D.solve_packed` (many uneven 2D solves at once) and `serve.Server` (requests). Sizes
are those of the repository's workloads (bwpm_b200/workloads.py), tests and benchmark, and generic
ones between them. Results of complex64 fields, which the entry points widen on return, are
returned as complex64.
"""

from __future__ import annotations

import numpy as np
import torch

from bwpm_b200 import workloads as wl

LAMBDA_UM = 0.633
BATCH_SIZES = wl.BATCH_SIZES
# run-time lengths of the served stream (2, 3 and 5 only), small to large
SERVED_SIZES = (1080, 1536, 2187, 1200, 2430, 1024, 3072, 1620)


def listed() -> list[dict]:
    return [
        # A short 2D chain, FP64: the smallest call (parameter sweeps, the adapter's estimates);
        # launches and latency are all there is.
        {"name": "line256_fp64", "kind": "line", "ny": 256, "nz": 40, "iters": 1, "prec": 64,
         "body": "facet"},
        # The planar 5 µm slab of the repository's 2D workload (1024 points, 250 slabs, 8
        # iterations), the drop-in's ordinary 2D solve: long, nearly always one pass per step.
        {"name": "slab1024_fp64", "kind": "line", "ny": 1024, "nz": 250, "iters": 8, "prec": 64,
         "body": "slab"},
        # A long line behind a tilted face, FP64: several passes on many steps, reflections.
        {"name": "line4096_fp64", "kind": "line", "ny": 4096, "nz": 300, "iters": 2, "prec": 64,
         "body": "facet"},
        # An uneven length of the served stream (2·3⁵·5), complex64 fields through the solver.
        {"name": "line2430_c64", "kind": "line", "ny": 2430, "nz": 300, "iters": 2, "prec": 32,
         "body": "lens"},
        # A Born chain (δn on every slab, GMRES per step) at the workload's line length, FP64.
        {"name": "born4096_fp64", "kind": "born", "ny": 4096, "nz": 24, "iters": 2, "prec": 64},
        # A 3D volume at the microlens workload's lateral size, FP64: the drop-in's 3D solve.
        {"name": "plane512_fp64", "kind": "plane", "ny": 512, "nx": 512, "nz": 60, "iters": 2,
         "prec": 64, "body": "lens"},
        # An uneven, odd 3D plane (3·5³ × 2·5³), FP64: sizes no kernel is compiled for.
        {"name": "plane375x250_fp64", "kind": "plane", "ny": 375, "nx": 250, "nz": 50, "iters": 1,
         "prec": 64, "body": "facet"},
        # The microlens workload's lateral size in complex64.
        {"name": "plane512_c64", "kind": "plane", "ny": 512, "nx": 512, "nz": 100, "iters": 2,
         "prec": 32, "body": "lens"},
        # The largest served plane in complex64.
        {"name": "plane1024_c64", "kind": "plane", "ny": 1024, "nx": 1024, "nz": 40, "iters": 2,
         "prec": 32, "body": "facet"},
        # A whole facade call, set-up included: a new 3D problem each time, host labels.
        {"name": "facade256_fp64", "kind": "facade", "ny": 256, "nx": 256, "nz": 100, "iters": 1,
         "prec": 64, "body": "lens"},
        # The batched engine end to end: uneven 2D solves of every compiled length, host to host.
        {"name": "batch33", "kind": "batch", "count": 33, "nz_lo": 60, "nz_hi": 360, "iters": 2},
        # The request loop: uneven 2D and 3D requests submitted at once, results collected.
        {"name": "served10", "kind": "served", "count2d": 8, "count3d": 2, "nz": 200, "iters": 1},
    ]


def _smooth(rng, lo: int, hi: int) -> int:
    """A lateral size with prime factors up to 7, log-uniform in [lo, hi]."""
    want = lo * (hi / lo) ** rng.random()
    best = None
    for v in range(lo, hi + 1):
        m = v
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1 and (best is None or abs(v - want) < abs(best - want)):
            best = v
    return best


def draw(rng) -> dict:
    kind = rng.choice(["line", "line", "line", "born", "plane", "plane", "plane", "facade",
                       "batch", "served"])
    prec = rng.choice([64, 32])
    body = rng.choice(["facet", "lens"])
    if kind == "line":
        ny = rng.choice([_smooth(rng, 128, 6000), rng.choice(BATCH_SIZES)])
        nz = int(20 * 15 ** rng.random()) + rng.randrange(7)
        return {"kind": kind, "ny": ny, "nz": nz, "iters": rng.randrange(3), "prec": prec,
                "body": body}
    if kind == "born":
        return {"kind": kind, "ny": rng.choice([_smooth(rng, 256, 4096), 1024, 2048]),
                "nz": rng.randrange(6, 25), "iters": rng.randrange(3), "prec": prec}
    if kind in ("plane", "facade"):
        sizes = [n for n in wl.SERVED_3D_LATERAL if n <= (1024 if prec == 32 else 512)]
        top = 1024 if prec == 32 else 560
        if kind == "facade":
            sizes, top = [256, 384], 400
        if rng.random() < 0.5:
            ny = nx = rng.choice(sizes)
        else:
            ny, nx = _smooth(rng, 120, top), _smooth(rng, 120, top)
        cells = (24e6 if kind == "plane" else 6e6) / (ny * nx)
        nz = max(12, min(100, int(cells * (0.4 + 0.6 * rng.random()))))
        return {"kind": kind, "ny": ny, "nx": nx, "nz": nz, "iters": rng.randrange(3),
                "prec": prec, "body": body}
    if kind == "batch":
        lo = rng.randrange(20, 100)
        return {"kind": kind, "count": rng.randrange(8, 34), "nz_lo": lo,
                "nz_hi": lo + rng.randrange(40, 260), "iters": rng.randrange(1, 3)}
    return {"kind": kind, "count2d": rng.randrange(3, 9), "count3d": rng.randrange(3),
            "nz": rng.randrange(80, 200), "iters": rng.randrange(1, 3)}


# ---- inputs -------------------------------------------------------------------------------------


def _volume(ny, nx, nz, body, rng) -> dict:
    """Grid, materials, body (a geometry of bwpm_b200.workloads) and incident field of one solve.
    The seed moves the beam, the materials and the tilt; the sizes and the shape of the work stay."""
    lam = LAMBDA_UM * 1e-3
    flat = nx == 1
    dy = lam / (8 if flat else 6)
    dx = 1.0 if flat else dy
    dz = lam / (10 if flat else 8)
    k0 = wl.k0_of(LAMBDA_UM)
    y, x = wl.centred(ny, dy), wl.centred(nx, dx)
    g = {"nz": nz, "ny": ny, "nx": nx, "dz": dz, "dy": dy, "dx": dx, "base": nz // 3 * dz}
    n = 1.45 + 0.05 * rng.random()
    if body == "facet":  # a tilted fibre facet
        g.update(kind="tilted_facet", tan_tilt=float(np.tan(np.deg2rad(1.0 + 0.1 * rng.random()))))
    elif body == "lens":  # an array of spherical caps
        sag = min(4e-3, 0.3 * nz * dz)
        pitch = max(24e-3, 4 * sag)
        g.update(kind="lens_array", pitch=pitch, sag=sag,
                 radius=((pitch / 2) ** 2 + sag**2) / (2 * sag))
    else:  # a planar slab
        g.update(kind="tilted_slab", tan_tilt=0.0, back=(nz // 3 + int(round(5e-3 / dz))) * dz)
    w0 = ny * dy / 8
    off = w0 * 0.2 * (rng.random() - 0.5)
    theta = np.deg2rad(4.0) * rng.random()
    prof = np.exp(-(((y - off) / w0) ** 2) + 1j * k0 * np.sin(theta) * y)[:, None]
    mask = wl.absorbing_mask_1d(y, ny * dy / 10)[:, None]
    field = np.zeros((ny, nx, 2), np.complex128)
    if flat:  # TE or TM
        field[..., rng.integers(2)] = prof
        mask = None if body == "slab" else mask
    else:
        wx = nx * dx / 8
        prof = prof * np.exp(-((x / wx) ** 2))[None, :]
        field[..., 0], field[..., 1] = prof, (0.2 + 0.2 * rng.random()) * 1j * prof
        mask = mask * wl.absorbing_mask_1d(x, nx * dx / 10)[None, :]
    return {"ny": ny, "nx": nx, "dy": dy, "dx": dx, "dz": dz, "k0": k0,
            "indices": np.array([1.0 + 0j, n + 0j]), "geometry": g, "before": 1.0 + 0j,
            "mask": mask, "field": field}


def _born(ny, nz, rng) -> dict:
    """A homogeneous host with a Gaussian random δn on every slab, tilted plane wave."""
    lam = LAMBDA_UM * 1e-3
    dy, dz, k0 = lam / 8, lam / 10, wl.k0_of(LAMBDA_UM)
    host = 1.5
    dn = wl.gaussian_random_field(rng, nz, ny, dz, dy, 0.5e-3, 0.01)
    ky = 2 * np.pi * np.fft.fftfreq(ny, d=dy)
    ky = ky[np.argmin(np.abs(ky - host * k0 * np.sin(np.deg2rad(8.0 + 4.0 * rng.random()))))]
    field = np.zeros((ny, 1, 2), np.complex128)
    field[:, 0, rng.integers(2)] = np.exp(1j * ky * wl.centred(ny, dy))
    return {"ny": ny, "nx": 1, "dy": dy, "dx": 1.0, "dz": dz, "k0": k0,
            "indices": np.array([host + 0j]), "labels": np.zeros((nz, ny, 1), np.int32),
            "before": host + 0j, "mask": None, "field": field,
            "fluctuation": dn.astype(np.complex128)[:, :, None]}


def _labels(v) -> np.ndarray:
    if "labels" not in v:
        v["labels"] = wl.geometry_labels(v["geometry"]).astype(np.int32)
    return v["labels"]


def _sizes(case) -> list[tuple[int, int, int, str]]:
    """(ny, nx, nz, body) of the solves of a batch or served case."""
    if case["kind"] == "batch":
        span = case["nz_hi"] - case["nz_lo"]
        return [(BATCH_SIZES[i % len(BATCH_SIZES)], 1, case["nz_lo"] + (i * 97) % (span + 1),
                 ("facet", "lens")[i % 2]) for i in range(case["count"])]
    out = [(SERVED_SIZES[i % len(SERVED_SIZES)], 1, case["nz"] + 23 * i, ("lens", "facet")[i % 2])
           for i in range(case["count2d"])]
    return out + [((256, 384)[i % 2],) * 2 + (case["nz"] // 3, "lens")
                  for i in range(case["count3d"])]


def _inputs(case, seed) -> list[dict]:
    rng = np.random.default_rng(seed)
    if case["kind"] == "born":
        return [_born(case["ny"], case["nz"], rng)]
    if case["kind"] in ("batch", "served"):
        return [_volume(*s, rng) for s in _sizes(case)]
    return [_volume(case["ny"], case.get("nx", 1), case["nz"], case["body"], rng)]


# ---- what a program holds, and one pass --------------------------------------------------------


def prepare(case, seed):
    from bwpm_b200 import _core, batch, serve
    from bwpm_b200.model import Bidirectional3D, Grid3D

    vs = _inputs(case, seed)
    v = vs[0]
    state = {"case": case}
    kind = case["kind"]
    if kind in ("line", "born"):
        state["solver"] = _core.CudaSolver(
            v["ny"], 1, v["dy"], v["dx"], v["dz"], v["k0"], v["indices"], _labels(v), v["before"],
            v["mask"], 0, fluctuation=v.get("fluctuation"), precision=case["prec"])
        state["field"] = v["field"]
    elif kind == "plane":
        state["solver"] = _core.CudaSolver.from_geometry(
            v["ny"], v["nx"], v["dy"], v["dx"], v["dz"], v["k0"], v["indices"], v["geometry"],
            v["before"], v["mask"], 0, precision=case["prec"])
        state["field"] = v["field"]
    elif kind == "facade":
        state["volume"] = Bidirectional3D(
            Grid3D(v["nx"], v["ny"], v["dx"], v["dy"], v["dz"], LAMBDA_UM), list(v["indices"]),
            _labels(v), v["before"], v["mask"])
        state["field"] = v["field"]
    elif kind == "batch":
        b = batch.Batch2D(0)
        for u in vs:
            b.add(u["ny"], u["dy"], u["dz"], u["k0"], u["indices"], _labels(u), u["before"],
                  u["mask"], u["field"], case["iters"])
        b.prepare()
        # page-locked host buffers, as a program that solves again and again keeps them
        fields = torch.empty(b.packed_size, dtype=torch.complex128, pin_memory=True).numpy()
        fields[:] = np.concatenate([u["field"].reshape(-1) for u in vs])
        state.update(batch=b, fields=fields,
                     out=torch.empty(2 * b.packed_size, dtype=torch.complex128,
                                     pin_memory=True).numpy())
    else:
        state["server"] = serve.Server(0)
        state["problems"] = [
            wl.Problem(u["ny"], u["nx"], u["dy"], u["dx"], u["dz"], u["k0"], u["indices"],
                       _labels(u) if u["nx"] == 1 else None, u["before"], u["mask"], u["field"],
                       case["iters"], geometry=u["geometry"]) for u in vs]
    return state


def _typed(a, prec):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t if prec == 64 else t.to(torch.complex64)


def run(state):
    from bwpm_b200 import fast

    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        state["batch"].solve_packed(state["fields"], state["out"])
        return _typed(state["out"], 32)
    if kind == "served":
        s = state["server"]
        tickets = [s.submit(p) for p in state["problems"]]
        results = [s.result(t) for t in tickets]
        return {"transmitted": [_typed(r["transmitted"], 32) for r in results],
                "reflected": [_typed(r["reflected"], 32) for r in results]}
    if kind == "facade":
        r = fast.run_3d(state["volume"], state["field"], case["iters"], backend="cuda",
                        precision=case["prec"])
        return {"transmitted": _typed(r.transmitted, case["prec"]),
                "reflected": _typed(r.reflected, case["prec"])}
    r = state["solver"].run(state["field"], case["iters"], [])
    return {"transmitted": _typed(r["transmitted"], case["prec"]),
            "reflected": _typed(r["reflected"], case["prec"])}


def work(case) -> dict:
    """One forward and one inverse transform of both components per slab and sweep, with the 2×2
    operator product (one component in the batched and served 2D solves, whose other is zero);
    bytes: labels, incident field, results."""
    if case["kind"] in ("batch", "served"):
        sizes = _sizes(case)
    else:
        sizes = [(case["ny"], case.get("nx", 1), case["nz"], "")]
    flops = bytes_ = 0.0
    for ny, nx, nz, _ in sizes:
        n = ny * nx
        comps = 1 if case["kind"] in ("batch", "served", "line") and nx == 1 else 2
        sweeps = 2 * case["iters"] if case["iters"] else 1
        per = comps * (10 * n * np.log2(n) + (6 if nx == 1 else 14) * n)
        if case["kind"] == "born":
            # the Cayley step's operator at least once per slab and sweep: three components in
            # and back, beside the source terms of the back-scatter (two Gauss points) of a
            # bidirectional run
            per += 3 * 10 * n * np.log2(n) * (3 if case["iters"] else 1)
        flops += sweeps * nz * per
        field = 2 * n * 16
        bytes_ += 3 * field + nz * n
    return {"bytes": float(bytes_), "flops": float(flops)}


# ---- 64-bit values: the method in plain torch ---------------------------------------------------


class _Exact:
    """The bidirectional wave propagation method in complex128: per slab the transmission and
    reflection operators of every label pair applied in the angular spectrum, selected per pixel."""

    def __init__(self, v):
        self.v = v
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        freq = lambda n, d: 2 * np.pi * torch.fft.fftfreq(n, d=d, dtype=torch.float64)  # noqa: E731
        self.ky, self.kx = (a.to(self.dev) for a in torch.meshgrid(
            freq(v["ny"], v["dy"]), freq(v["nx"], v["dx"]), indexing="ij"))
        self.kp2 = self.kx**2 + self.ky**2
        self.tables = {}
        self.labels = _labels(v)
        self.dl = torch.from_numpy(self.labels).to(self.dev)
        self.mask = None if v["mask"] is None else self._t(v["mask"])[..., None]
        # the distinct label pairs of every step (−1: the medium before the volume)
        lab = self.labels.reshape(self.labels.shape[0], -1)
        prev = np.vstack([np.full((1, lab.shape[1]), -1, lab.dtype), lab[:-1]])
        self.pairs = [[divmod(int(c), 4096) for c in np.unique((a.astype(np.int64) + 1) * 4096 + b)]
                      for a, b in zip(prev, lab)]

    def _t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def fft(self, e):
        return torch.fft.fft2(e, dim=(0, 1))

    def ifft(self, s):
        return torch.fft.ifft2(s, dim=(0, 1))

    def index(self, label):
        return complex(self.v["before"] if label < 0 else self.v["indices"][label])

    def kz(self, n):
        k0 = self.v["k0"]
        n2k2 = complex(n * n * k0 * k0)
        q = n2k2 - self.kp2.to(torch.complex128)
        q = torch.where(q.abs() <= 1e-12 * abs(n2k2), torch.zeros_like(q), q)
        kz = torch.sqrt(q)
        flip = (kz.imag < 0) | ((kz.imag == 0) & (kz.real < 0))
        kz = torch.where(flip, -kz, kz)
        return torch.where(kz.abs() < 1e-12 * k0, torch.full_like(kz, 1e-12j * k0), kz)

    def operator(self, reflect, backward, nr, ns):
        """(m00, m01, m11) of the transition nr → ns, propagation included."""
        key = (reflect, backward, nr, ns)
        if key in self.tables:
            return self.tables[key]
        k0, dz = self.v["k0"], self.v["dz"]
        a, b = self.kz(nr), self.kz(ns)
        kx, ky, kp2 = self.kx, self.ky, self.kp2
        flat = kp2 == 0
        safe = torch.where(flat, torch.ones_like(kp2), kp2)
        if reflect:
            s = (a - b) / (a + b)
            p = (ns * ns * a - nr * nr * b) / (ns * ns * a + nr * nr * b)
            # s keeps its direction; p: E⊥ along k⊥ turns over
            along, across = -p * (a * a + kp2) / (nr * k0) ** 2, s
            phase = torch.exp(2j * a * dz) if backward else 1.0
        else:
            s = 2 * a / (a + b)
            p = 2 * nr * ns * a / (ns * ns * a + nr * nr * b)
            along, across = p * (a * b + b * kp2 / a) / (nr * ns * k0 * k0), s
            phase = torch.exp(1j * (a if backward else b) * dz)
        along = torch.where(flat, across, along)
        m00 = (along * kx * kx + across * ky * ky) / safe
        m01 = (along - across) * kx * ky / safe
        m11 = (along * ky * ky + across * kx * kx) / safe
        m00, m11 = torch.where(flat, across, m00), torch.where(flat, across, m11)
        m01 = torch.where(flat, torch.zeros_like(m01), m01)
        self.tables[key] = got = tuple(m * phase for m in (m00, m01, m11))
        return got

    def apply(self, spec, p, reflect, backward):
        out = torch.zeros_like(spec)
        for r1, s in self.pairs[p]:
            r = r1 - 1
            nr, ns = self.index(s if backward else r), self.index(r if backward else s)
            if reflect and nr == ns:
                continue
            m00, m01, m11 = self.operator(reflect, backward, nr, ns)
            e = self.ifft(torch.stack([m00 * spec[..., 0] + m01 * spec[..., 1],
                                       m01 * spec[..., 0] + m11 * spec[..., 1]], -1))
            if len(self.pairs[p]) == 1:
                return e
            here = self.dl[p] == s
            if p > 0:
                here = here & (self.dl[p - 1] == r)
            out = torch.where(here[..., None], e, out)
        return out

    # weak fluctuations: Born terms of one slab

    def born(self, p):
        h, k0, dz = self.index(int(self.labels[p].flat[0])), self.v["k0"], self.v["dz"]
        kz = self.kz(h)
        k2 = (h * k0) ** 2
        prop = (self.kp2 < abs(k2)) & ((k2 - self.kp2).abs() > 1e-12 * abs(k2))
        pot = 2 * h * k0 * k0 * self._t(self.v["fluctuation"][p])
        green = torch.where(prop, 1j * dz / (2 * kz), torch.zeros_like(kz))
        return kz, k2, prop, pot, green

    def scatter(self, s, b, d, dist=0.0):
        """F{V·F⁻¹(Ŝ⊥, Ŝ_z)} of the waves in direction d, moved by `dist` first."""
        kz, _, prop, pot, _ = b
        ez = -d * (self.kx * s[..., 0] + self.ky * s[..., 1]) / kz
        w = torch.stack([s[..., 0], s[..., 1], ez], -1) * torch.exp(1j * kz * dist)[..., None]
        w = torch.where(prop[..., None], w, torch.zeros_like(w))
        return self.fft(pot[..., None] * self.ifft(w))

    def radiate(self, w, b, d, phase=1.0):
        kz, k2, _, _, green = b
        lon = (self.kx * w[..., 0] + self.ky * w[..., 1] + d * kz * w[..., 2]) / k2
        return torch.stack([w[..., 0] - self.kx * lon, w[..., 1] - self.ky * lon],
                           -1) * (green * phase)[..., None]

    def increment(self, spec, b, d):
        """F⁻¹{P_½^{±} y} with (1 − G/2) y = G P_½ Ê, by fixed-point iteration."""
        kz, _, prop, _, _ = b
        half = torch.where(prop, torch.exp(0.5j * kz * self.v["dz"]), torch.zeros_like(kz))
        back = half if d > 0 else torch.where(
            prop, torch.exp(-0.5j * kz * self.v["dz"]), torch.zeros_like(kz))
        rhs = self.radiate(self.scatter(spec * half[..., None], b, d), b, d)
        y, size = rhs, float(torch.linalg.vector_norm(rhs))
        for _ in range(200):
            new = rhs + 0.5 * self.radiate(self.scatter(y, b, d), b, d)
            step = float(torch.linalg.vector_norm(new - y))
            y = new
            if step <= 1e-16 * size:
                break
        return self.ifft(y * back[..., None])

    def emission(self, spec, b, d):
        """Waves radiated against direction d, at that edge of the slab (two Gauss points)."""
        dz, total = self.v["dz"], 0.0
        for g in ((1 - 3**-0.5) / 2, (1 + 3**-0.5) / 2):
            w = self.scatter(spec, b, d, (g if d > 0 else 1 - g) * dz)
            total = total + self.radiate(
                w, b, -d, 0.5 * torch.exp(-1j * d * b[0] * (1 - g) * dz))
        return self.ifft(total)

    def solve(self, iterations):
        v = self.v
        nz = self.labels.shape[0]
        born = v.get("fluctuation") is not None
        face = [any(self.index(r1 - 1) != self.index(s) for r1, s in ps) for ps in self.pairs]
        src_f, src_b, born_f, born_b = {}, {}, {}, {}
        inp = self._t(v["field"])
        masked = lambda e: e if self.mask is None else e * self.mask  # noqa: E731
        e = back = None
        for it in range(max(iterations, 1)):
            e = inp
            for p in range(nz):
                spec = self.fft(e)
                if iterations and face[p]:
                    src_b[p] = self.apply(spec, p, True, False)
                e = masked(self.apply(spec, p, False, False))
                if it and face[p]:
                    e = e + src_f[p]
                if born:
                    b = self.born(p)
                    e = e + masked(self.increment(spec, b, 1))
                    if iterations:
                        born_b[p] = self.emission(spec, b, 1)
                    if it:
                        e = e + born_f[p]
            if not iterations:
                return e, torch.zeros_like(e)
            back = torch.zeros_like(inp)
            for p in range(nz - 1, -1, -1):
                if born:
                    back = back + born_b[p]
                spec = self.fft(back)
                if born:
                    b = self.born(p)
                    born_f[p] = self.emission(spec, b, -1)
                    spec = self.fft(back + self.increment(spec, b, -1))
                if face[p]:
                    src_f[p] = self.apply(spec, p, True, True)
                back = masked(self.apply(spec, p, False, True))
                if face[p]:
                    back = back + src_b[p]
        return e, back


def exact(case, seed):
    vs = _inputs(case, seed)
    got = [[a.cpu() for a in _Exact(v).solve(case["iters"])] for v in vs]
    if case["kind"] == "batch":
        return torch.cat([torch.cat([t.reshape(-1), r.reshape(-1)]) for t, r in got])
    if case["kind"] == "served":
        shape = lambda a: a[:, 0] if a.shape[1] == 1 else a  # noqa: E731
        return {"transmitted": [shape(t) for t, _ in got], "reflected": [shape(r) for _, r in got]}
    return {"transmitted": got[0][0], "reflected": got[0][1]}
