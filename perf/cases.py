"""Measured workloads of the non-uniform FFT operator.

Each case is one pass through the public entry points (``Plan``,
``NUFFTOp``, ``cg_sense``, ``NUFFT``, ``BatchedOperator``) at sizes that MRI
reconstructions use: 2-D radial and spiral acquisitions, 3-D kooshballs and
slabs, one coil to 32 coils, with and without coil maps and density weights,
power-of-two and other grids.  ``exact`` restates the operator in float64
with torch alone.

Case fields: ``kind`` (pair: forward and adjoint; fwd; adj; cg; grad; host;
batch), image size ``nx, ny, nz`` (nz 0: 2-D), ``coils``, trajectory
``traj`` with ``lines`` x ``points`` samples, ``osf``, ``kw``, ``sw``,
``maps`` and ``dens`` (coil maps / density weights in use).
"""
import math

import numpy as np
import torch

import gpunufft_b200 as G
from gpunufft_b200.autograd import NUFFT
from gpunufft_b200.batch import BatchedOperator
from gpunufft_b200.cg_sense import cg_sense


def _case(name, kind, dims, coils, traj, lines, points, osf=2.0, kw=3, sw=8,
          maps=True, dens=True, **more):
    c = dict(kind=kind, nx=dims[0], ny=dims[1],
             nz=dims[2] if len(dims) > 2 else 0, coils=coils, traj=traj,
             lines=lines, points=points, osf=osf, kw=kw, sw=sw, maps=maps,
             dens=dens, **more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a single-coil 2-D radial frame: the smallest call, as in real-time
        # display or one coil of a pipeline; latency and launches count
        _case("pair_2d128_c1", "pair", (128, 128), 1, "radial", 64, 256,
              maps=False),
        # multi-coil 2-D radial gridding reconstruction with coil combine
        _case("adj_2d256_c16", "adj", (256, 256), 16, "radial", 402, 512),
        # spiral data simulation / residual: odd coil count, per-coil
        # images, wide kernel, fractional oversampling (grid 220 x 220)
        _case("fwd_2d160_spiral_c11", "fwd", (160, 160), 11, "spiral", 24,
              1667, osf=1.375, kw=5, maps=False, dens=False),
        # iterative multi-coil reconstruction (CG-SENSE), the whole solve
        _case("cg_2d256_c16", "cg", (256, 256), 16, "radial", 202, 512,
              iters=10),
        # 3-D kooshball of everyday size on a grid that is not a power of
        # two (192 cubed), both directions of an iterative solver
        _case("fwd_3d96_c16", "fwd", (96, 96, 96), 16, "koosh", 2048, 256),
        _case("adj_3d96_c16", "adj", (96, 96, 96), 16, "koosh", 2048, 256),
        # ragged slab: three different axes, wide kernel, low oversampling,
        # few coils, per-coil images
        _case("adj_3dslab_c6", "adj", (176, 144, 52), 6, "koosh", 1201, 255,
              osf=1.5, kw=5, maps=False),
        # the large 3-D reconstruction: 128 cubed, 32 coils, 2.1 M samples,
        # both directions
        _case("fwd_3d128_c32", "fwd", (128, 128, 128), 32, "koosh", 8192,
              256),
        _case("adj_3d128_c32", "adj", (128, 128, 128), 32, "koosh", 8192,
              256),
        # training step through the differentiable operator: gradients of
        # the image and of the trajectory
        _case("grad_2d320_c8", "grad", (320, 320), 8, "spiral", 32, 2500,
              osf=1.6, kw=4, dens=False),
        # host arrays through the binding-compatible class with its default
        # (texture) kernel: the call a user of the upstream binding makes
        _case("host_3d64_c8", "host", (64, 64, 64), 8, "koosh", 1024, 128),
        # a batch of uneven 2-D spirals (many slices or patients at once)
        _case("batch_spirals12", "batch", (320, 320), 32, "spiral", 48,
              2500, kw=5, maps=True, dens=False, n=12, shapes=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair", "fwd", "adj", "fwd", "adj", "fwd", "adj", "cg",
                       "grad", "host", "batch"])
    if kind == "batch":
        return _case(None, "batch", (320, 320), 32, "spiral", 48, 2500, kw=5,
                     dens=False, n=rng.randint(4, 14),
                     shapes=rng.randint(10, 10 ** 6))
    three = kind in ("fwd", "adj", "pair", "host") and rng.random() < 0.6
    kw = rng.choice([3, 3, 3, 4, 5])
    osf = rng.choice([2.0, 2.0, 1.5, 1.25, round(rng.uniform(1.25, 2.0), 2)])
    maps, dens = rng.random() < 0.7, rng.random() < 0.6
    even = ~1 if rng.random() < 0.75 else ~0  # odd image sides now and then
    if three:
        base = _log(rng, 32, 128)
        dims = tuple(max(24, min(128, int(base * rng.choice(
            [1.0, 1.0, 1.0, 0.75, 0.5, rng.uniform(0.4, 1.0)])))) & even
            for _ in range(3))
        n = max(dims)
        lines, points = _log(rng, 200, 60 * n), rng.randint(n, 2 * n)
        coils = rng.choice([1, 2, 4, 5, 8, 12, 16, 24, 32,
                            rng.randint(1, 32)])
        if kind == "host":
            lines, coils = min(lines, 1500), min(coils, 8)
        # no more work than the largest listed case
        coils = min(coils, max(1, int(50e6 // (lines * points))))
        if kw > 3:
            coils = min(coils, max(1, int(20e6 // (lines * points))))
        vol = dims[0] * dims[1] * dims[2] * osf ** 3
        coils = min(coils, max(1, int(400e6 // vol)))
        traj = "koosh"
    else:
        base = _log(rng, 64, 384)
        dims = (base & even, (base if rng.random() < 0.7 else
                              max(48, int(base * rng.uniform(0.5, 1.0)))) &
                even)
        traj = rng.choice(["radial", "spiral"])
        lines, points = rng.randint(16, 420), rng.randint(200, 520)
        if traj == "spiral":
            lines, points = rng.randint(8, 48), rng.randint(1200, 2600)
        coils = rng.choice([1, 4, 8, 16, 32, rng.randint(1, 32)])
    more = {}
    if kind == "cg":
        maps, coils, more = True, max(2, min(coils, 16)), dict(iters=5)
        dims = (max(dims), max(dims))
        if max(dims) > 256:
            dims = (256, 256)
        osf = 2.0
    return _case(None, kind, dims, coils, traj, lines, points, osf, kw, 8,
                 maps, dens, **more)


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _dims(case):
    return ((case["nx"], case["ny"], case["nz"]) if case["nz"] else
            (case["nx"], case["ny"]))


def _trajectory(case, rng):
    """Float32 (dim, M) coordinates in [-0.5, 0.5) and density weights."""
    L, P = case["lines"], case["points"]
    r = (np.arange(P) - P // 2) / P
    off = rng.uniform(0, 2 * np.pi)
    golden = (math.sqrt(5.0) - 1.0) / 2.0
    if case["traj"] == "radial":
        a = off + np.arange(L) * np.pi * golden
        t = np.stack([np.outer(np.cos(a), r), np.outer(np.sin(a), r)])
        d = np.broadcast_to(np.abs(r) + 0.5 / P, (L, P))
    elif case["traj"] == "koosh":
        i = np.arange(L) + 0.5
        z = 1.0 - 2.0 * i / L
        a = off + 2.0 * np.pi * golden * i
        s = np.sqrt(1.0 - z * z)
        u = np.stack([s * np.cos(a), s * np.sin(a), z])
        t = u[:, :, None] * r[None, None, :]
        d = np.broadcast_to(r * r + (0.5 / P) ** 2, (L, P))
    else:  # variable-density spiral
        u = np.arange(P) / P
        turns = 6.0 + 8.0 * rng.uniform()
        rad = 0.499 * u ** 1.6
        th = off + 2 * np.pi * (turns * u[None] +
                                np.arange(L)[:, None] / L)
        t = np.stack([rad * np.cos(th), rad * np.sin(th)])
        d = np.broadcast_to(rad + 0.5 / P, (L, P))
    t = np.clip(t.reshape(t.shape[0], -1), -0.5, np.nextafter(0.5, 0))
    d = d.reshape(-1) / d.max()
    return (np.ascontiguousarray(t, np.float32),
            np.ascontiguousarray(d, np.float32))


def _generator(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + 7919 * salt + 12345) % (1 << 62))
    return g


def _grids(shape):
    return torch.meshgrid(*[(torch.arange(n, device="cuda") - n // 2) / n
                            for n in shape], indexing="ij")


def _maps(shape, coils, gen):
    """Smooth Gaussian-profile coil maps with random centres and phases."""
    ax = _grids(shape)
    out = torch.empty((coils,) + tuple(shape), dtype=torch.complex64,
                      device="cuda")
    p = torch.rand((coils, 2 * len(shape) + 1), generator=gen,
                   device="cuda").cpu().tolist()
    for c in range(coils):
        r2 = sum((a - (p[c][i] - 0.5) * 1.2) ** 2 for i, a in enumerate(ax))
        ph = sum(a * (p[c][len(shape) + i] * 6 - 3)
                 for i, a in enumerate(ax)) + 6.28 * p[c][-1]
        out[c] = torch.polar(torch.exp(-2.0 * r2), ph)
    norm = out.abs().square().sum(0).sqrt().clamp_min(1e-3)
    return out / norm


def _images(shape, n, gen):
    """Blobs with phase and a little noise, n images."""
    ax = _grids(shape)
    out = torch.empty((n,) + tuple(shape), dtype=torch.complex64,
                      device="cuda")
    for c in range(n):
        p = torch.rand((6, 8), generator=gen, device="cuda").cpu().tolist()
        im = torch.zeros(shape, device="cuda")
        for q in p:
            r2 = sum(((a - (q[i] - 0.5) * 0.6) / (0.08 + 0.25 * q[3 + i])) ** 2
                     for i, a in enumerate(ax))
            im += (q[6] + 0.2) * (r2 < 1)
        ph = sum(a * (p[0][i] * 3) for i, a in enumerate(ax))
        out[c] = torch.polar(im, ph)
    out += 0.02 * torch.randn(out.shape, generator=gen, device="cuda",
                              dtype=torch.complex64)
    return out


def _kspace(traj, coils, width, gen):
    """Noise with the radial decay of k-space data."""
    r = torch.from_numpy(np.sqrt((traj.astype(np.float64) ** 2).sum(0))).cuda()
    decay = (1.0 / (1.0 + 0.25 * r * width)).float()
    return torch.randn((coils, traj.shape[1]), generator=gen, device="cuda",
                       dtype=torch.complex64) * decay


def _spirals(case):
    """The instances of a batch: 96..320 squared, 8-32 coils, 10k-120k
    samples, oversampling 1.25-2, kernel width 3-5."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["n"]):
        n = int(rng.choice([96, 160, 256, 320]))
        lines = int(rng.integers(8, 49))
        out.append(_case(None, "pair", (n, n), int(rng.integers(8, 33)),
                         "spiral", lines,
                         int(rng.integers(10_000, 120_001)) // lines,
                         osf=float(np.round(rng.uniform(1.25, 2.0), 2)),
                         kw=int(rng.integers(3, 6)), dens=False))
    return out


def _inputs(case, seed):
    rng = np.random.default_rng(int(seed) + 17)
    gen = _generator(seed)
    dims = _dims(case)
    shape = dims[::-1]
    traj, dens = _trajectory(case, rng)
    C = case["coils"]
    d = dict(traj=traj, dens=dens if case["dens"] else None, dims=dims,
             shape=shape)
    d["maps"] = _maps(shape, C, gen) if case["maps"] else None
    d["k"] = _kspace(traj, C, max(dims), gen)
    d["x"] = _images(shape, 1 if case["maps"] else C, gen)
    if case["maps"]:
        d["x"] = d["x"][0]
    return d


def _plan(case, d):
    return G.Plan(d["traj"], d["dims"], case["kw"], case["sw"], case["osf"],
                  d["dens"],
                  None if d["maps"] is None else d["maps"].cpu().numpy())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        subs = _spirals(case)
        ins = [_inputs(c, seed * 100 + i) for i, c in enumerate(subs)]
        plans = [_plan(c, d) for c, d in zip(subs, ins)]
        op = BatchedOperator(plans, [c["coils"] for c in subs])
        return dict(kind=kind, op=op, plans=plans, x=[d["x"] for d in ins],
                    k=[d["k"] for d in ins])
    d = _inputs(case, seed)
    s = dict(kind=kind, case=dict(case))
    if kind in ("fwd", "pair"):
        s["x"] = d["x"]
    if kind in ("adj", "pair", "cg"):
        s["k"] = d["k"]
    if kind == "grad":
        s["x"] = d["x"].requires_grad_()
        s["g"] = d["k"]
        s["t"] = torch.from_numpy(d["traj"]).cuda().requires_grad_()
        s["op"] = NUFFT(d["dims"], case["kw"], case["sw"], case["osf"],
                        d["maps"], d["dens"])
        s["op"].plan_for(s["t"])
    elif kind == "host":
        s["op"] = G.NUFFTOp(d["traj"], list(d["dims"]), case["coils"],
                            None if d["maps"] is None
                            else d["maps"].cpu().numpy(), d["dens"],
                            case["kw"], case["sw"], case["osf"])
        s["x"], s["k"] = d["x"].cpu().numpy(), d["k"].cpu().numpy()
    else:
        s["plan"] = _plan(case, d)
    return s


def run(s):
    kind = s["kind"]
    if kind == "fwd":
        return s["plan"].forward(s["x"])
    if kind == "adj":
        return s["plan"].adjoint(s["k"])
    if kind == "pair":
        return s["plan"].forward(s["x"]), s["plan"].adjoint(s["k"])
    if kind == "cg":
        return cg_sense(s["plan"], s["k"], maxit=s["case"]["iters"])
    if kind == "grad":
        y = s["op"](s["x"], s["t"])
        gx, gt = torch.autograd.grad(y, (s["x"], s["t"]), s["g"])
        return y.detach(), gx, gt
    if kind == "host":
        return s["op"].op(s["x"]), s["op"].adj_op(s["k"])
    return list(s["op"].forward(s["x"])), list(s["op"].adjoint(s["k"]))


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def work(case):
    if case["kind"] == "batch":
        ws = [work(c) for c in _spirals(case)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    dims = _dims(case)
    dim, C, kw = len(dims), case["coils"], case["kw"]
    M = case["lines"] * case["points"]
    N = math.prod(dims)
    grid = [int(np.float32(n) * np.float32(case["osf"])) for n in dims]
    # pruned transforms: lines of the axes in the order x, y, z
    fft = 0.0
    for a in range(dim):
        lines = math.prod(grid[:a]) * math.prod(dims[a + 1:])
        fft += lines * 5.0 * grid[a] * math.log2(max(2, grid[a]))
    flops = C * (4.0 * M * kw ** dim + fft + 14.0 * N)
    maps = 8 * C * N if case["maps"] else 0
    img = 8 * N * (1 if case["maps"] else C)
    sample = 4 * dim + (4 if case["dens"] else 0)
    bytes_ = maps + img + 8 * C * M + sample * M
    times = {"pair": 2, "host": 2, "grad": 3,
             "cg": 1 + 2 * case.get("iters", 0)}.get(case["kind"], 1)
    return {"bytes": float(bytes_ * times), "flops": float(flops * times)}


def tolerance(case):
    # 32-bit sums and transforms.  Measured against float64: 2e-7 to 9e-7
    # for single calls and gradients, 2e-6 for a ten-iteration solve (the
    # iterations amplify rounding) and 2.3e-6 for the batch (prime grid
    # sides, whose transforms run as convolutions).
    if case["kind"] in ("cg", "batch"):
        return {"rel": 1e-5}
    return {"rel": 4e-6}


# --------------------------------------------------------------------------
# the operator in float64
# --------------------------------------------------------------------------
def _i0(x):
    """Modified Bessel I0 by Abramowitz & Stegun 9.8.1 / 9.8.2 (the
    polynomials that define the operator's kernel)."""
    ax = np.abs(x)
    y = (ax / 3.75) ** 2
    lo = 1 + y * (3.5156229 + y * (3.0899424 + y * (1.2067492 + y * (
        0.2659732 + y * (0.360768e-1 + y * 0.45813e-2)))))
    q = 3.75 / np.maximum(ax, 1e-9)
    hi = np.exp(ax) / np.sqrt(np.maximum(ax, 1e-9)) * (
        0.39894228 + q * (0.1328592e-1 + q * (0.225319e-2 + q * (
            -0.157565e-2 + q * (0.916281e-2 + q * (-0.2057706e-1 + q * (
                0.2635537e-1 + q * (-0.1647633e-1 + q * 0.392377e-2))))))))
    return np.where(ax < 3.75, lo, hi)


class _Exact:
    """The operator restated: Kaiser-Bessel weights from the nearest entry
    of the operator's table (selected in float32, as the operator selects
    them), everything else in float64."""

    def __init__(self, case, d):
        f = np.float32
        self.dims, self.kw, self.osf = d["dims"], case["kw"], case["osf"]
        self.dim = len(self.dims)
        osf, kw, sw = f(self.osf), self.kw, case["sw"]
        self.grid = [int(f(f(n) * osf)) for n in self.dims]
        gmax = max(self.grid)
        radius = kw / 2.0 / gmax
        self.rsq = f(radius * radius)
        L = int(int(math.floor(float(f(0.91) / f(osf * f(0.001))))) *
                float(f(kw)) * 0.5)
        t = f(f(kw) / osf * f(osf - f(0.5)))
        self.beta = float(f(f(math.pi) * np.sqrt(f(t * t - f(0.8)))))
        r = np.sqrt(np.arange(L) / float(L - 1)).astype(f).astype(np.float64)
        lut = _i0(self.beta * np.sqrt(np.maximum(1 - r * r, 0))) / _i0(
            np.float64(self.beta))
        lut[0], lut[-1] = 1.0, 0.0
        self.lut = lut.astype(f).astype(np.float64)
        self.mult = f((L - 1) * (1.0 / (radius * radius)))
        self.aniso = [f(f(g) / f(gmax)) for g in self.grid]
        self.crop = [int(f(f(n) * f(osf - f(1)) / f(2))) for n in self.dims]
        self.traj = d["traj"]
        self.M = self.traj.shape[1]
        self.cells, self.w, self.dist = [], [], []
        for a in range(self.dim):
            c, w, e = self._axis(self.traj[a], a, sw)
            self.cells.append(torch.from_numpy(c).cuda())
            self.w.append(torch.from_numpy(w).cuda())
            self.dist.append(torch.from_numpy(e).cuda())
        self.sd = (None if d["dens"] is None else
                   torch.from_numpy(d["dens"]).cuda().double().sqrt())
        self.maps = d["maps"]
        self.deapo = torch.ones((), dtype=torch.float64, device="cuda")
        for a in range(self.dim):
            c, w, _ = self._axis(np.zeros(1, f), a, 8)
            n = np.arange(self.dims[a])
            k = (n + self.crop[a] + self.grid[a] // 2) % self.grid[a]
            ph = 2j * np.pi * np.outer(k, c[0]) / self.grid[a]
            m = torch.from_numpy(np.abs((np.exp(ph) * w[0]).sum(1))).cuda()
            self.deapo = (1 / m).reshape((-1,) + (1,) * a) * self.deapo

    def _axis(self, c, a, sw):
        """Wrapped cells, weights and distances of one axis, (M, kw + 2)."""
        f = np.float32
        g, kw = self.grid[a], self.kw
        p = (c * f(g)).astype(np.float64) + 0.5 * g
        rounded = np.copysign(np.floor(np.abs(p) + 0.5), p)
        top = math.ceil(float(f(g)) / sw) - 1
        sec = np.clip(np.floor(rounded / sw), 0, top).astype(np.int64)
        center = sec * sw + sw // 2
        pad = sw + 2 * (kw // 2)
        off = pad // 2
        pos = (c.astype(np.float64) * g + 0.5 * g).astype(f)
        pos = (pos - center.astype(f)) + f(off)
        kr = f(kw / 2.0)
        lo = np.maximum(np.ceil(pos - kr).astype(np.int64), 0)
        hi = np.maximum(np.floor(pos + kr).astype(np.int64), 0)
        hi = np.where(hi >= pad - 1, pad - 1, hi)
        lo = np.where(lo >= pad - 1, int(pad - 1 - 2 * float(kr)), lo)
        i = lo[:, None] + np.arange(kw + 2)[None]
        ok = i <= hi[:, None]
        gc = i + center[:, None] - off
        d = ((gc.astype(f) / f(g) - f(0.5)) - c[:, None]) * self.aniso[a]
        d2 = d * d
        ok &= d2 < self.rsq
        x = (d2 * self.mult).astype(f)
        at = np.floor(x)
        at = (at + (x - at >= f(0.5))).astype(np.int64)
        w = np.where(ok, self.lut[np.clip(at, 0, len(self.lut) - 1)], 0.0)
        return np.mod(gc, g), w, np.where(ok, d, 0).astype(np.float64)

    def _stencil(self, derivative=None):
        """Flat cells and weights of the footprint, one (cells, weights)
        pair of (M,) vectors at a time."""
        ws = list(self.w)
        if derivative is not None:
            a, R2, d = derivative, float(self.rsq), self.dist[derivative]
            s = (1 - d * d / R2).clamp_min(0).sqrt()
            b = math.pi * math.sqrt(max(
                (self.kw / float(np.float32(self.osf)) *
                 (float(np.float32(self.osf)) - 0.5)) ** 2 - 0.8, 0))
            i0 = float(torch.special.i0(torch.tensor(b, dtype=torch.float64)))
            q = torch.where(s > 1e-12, torch.special.i1(b * s) /
                            s.clamp_min(1e-12), torch.full_like(s, b / 2))
            q = b * q / (i0 * R2) * d * float(self.aniso[a])
            # outside the kernel's support the weight and its slope vanish
            ws[a] = torch.where(d != 0, q, torch.zeros_like(q))
        K = self.kw + 2
        live = [[k for k in range(K)
                 if bool((ws[a][:, k] != 0).any())] for a in range(self.dim)]
        for z in (live[2] if self.dim == 3 else [None]):
            for y in live[1]:
                zy = self.cells[1][:, y]
                wzy = ws[1][:, y]
                if z is not None:
                    zy = zy + self.cells[2][:, z] * self.grid[1]
                    wzy = wzy * ws[2][:, z]
                for x in live[0]:
                    yield (zy * self.grid[0] + self.cells[0][:, x],
                           wzy * ws[0][:, x])

    def _shape(self):
        return tuple(self.grid[::-1])

    def spectrum(self, x):
        """Oversampled spectrum of one coil image, flat."""
        pad = torch.zeros(self._shape(), dtype=torch.complex128, device="cuda")
        sl = tuple(slice(o, o + n) for o, n in zip(self.crop[::-1],
                                                   self.dims[::-1]))
        pad[sl] = x * self.deapo
        ax = tuple(range(self.dim))
        pad = torch.roll(pad, [-(g // 2) for g in self._shape()], ax)
        h = torch.fft.fftn(pad)
        h = torch.roll(h, [-((g + 1) // 2) for g in self._shape()], ax)
        return torch.view_as_real(h.reshape(-1) / math.sqrt(
            math.prod(self.grid)))

    def interpolate(self, h, derivative=None):
        out = torch.zeros((self.M, 2), dtype=torch.float64, device="cuda")
        for cell, w in self._stencil(derivative):
            out += h[cell] * w[:, None]
        out = torch.view_as_complex(out)
        return out if self.sd is None else out * self.sd

    def coil_image(self, x, c):
        x = x.to(torch.complex128)
        return x[c] if self.maps is None else x * self.maps[c]

    def forward(self, x, coils):
        return torch.stack([self.interpolate(self.spectrum(
            self.coil_image(x, c))) for c in range(coils)])

    def adjoint(self, k):
        outs = []
        total = 0
        ax = tuple(range(self.dim))
        sl = tuple(slice(o, o + n) for o, n in zip(self.crop[::-1],
                                                   self.dims[::-1]))
        for c in range(k.shape[0]):
            v = k[c].to(torch.complex128)
            if self.sd is not None:
                v = v * self.sd
            v = torch.view_as_real(v.contiguous())
            h = torch.zeros((math.prod(self.grid), 2), dtype=torch.float64,
                            device="cuda")
            for cell, w in self._stencil():
                h.index_add_(0, cell, v * w[:, None])
            h = torch.view_as_complex(h).reshape(self._shape())
            shift = [-(g // 2) for g in self._shape()]
            im = torch.fft.ifftn(torch.roll(h, shift, ax), norm="forward")
            im = torch.roll(im, shift, ax)[sl] * self.deapo / math.sqrt(
                math.prod(self.grid))
            if self.maps is None:
                outs.append(im)
            else:
                total = total + self.maps[c].conj().to(torch.complex128) * im
        return torch.stack(outs) if self.maps is None else total


def _np(t):
    return t.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        fs, as_ = [], []
        for i, c in enumerate(_spirals(case)):
            d = _inputs(c, seed * 100 + i)
            e = _Exact(c, d)
            fs.append(_np(e.forward(d["x"], c["coils"])))
            as_.append(_np(e.adjoint(d["k"])))
        return fs, as_
    if kind == "host":
        return None  # hardware texture filtering: no 64-bit counterpart
    d = _inputs(case, seed)
    e = _Exact(case, d)
    C = case["coils"]
    if kind == "fwd":
        return _np(e.forward(d["x"], C))
    if kind == "adj":
        return _np(e.adjoint(d["k"]))
    if kind == "pair":
        return _np(e.forward(d["x"], C)), _np(e.adjoint(d["k"]))
    if kind == "grad":
        y = e.forward(d["x"], C)
        gx = e.adjoint(d["k"])
        gt = torch.zeros((e.dim, e.M), dtype=torch.float64, device="cuda")
        for c in range(C):
            h = e.spectrum(e.coil_image(d["x"], c))
            u = d["k"][c].to(torch.complex128)
            for a in range(e.dim):
                gt[a] += (u.conj() * e.interpolate(h, a)).real
        return _np(y), _np(gx), _np(gt)
    # the CG-SENSE iteration in float64
    rhs = e.adjoint(d["k"])
    x = torch.zeros_like(rhs)
    r, p = rhs.clone(), rhs.clone()
    rr = torch.vdot(r.reshape(-1), r.reshape(-1)).real
    for _ in range(case["iters"]):
        ap = e.adjoint(e.forward(p, C))
        a = rr / torch.vdot(p.reshape(-1), ap.reshape(-1))
        x = x + a * p
        r = r - a * ap
        new = torch.vdot(r.reshape(-1), r.reshape(-1)).real
        p = r + (new / rr) * p
        rr = new
    return _np(x)
