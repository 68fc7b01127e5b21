"""The workloads the library's speed is measured on: what callers have it do, over the sizes they do it at.

A case is one call pattern of the public API on one seeded batch of curves:

  call        what a pass runs
  host        createArclengthTable, getAllCurveArclengths, arclengthReverse with host arrays in and out (the reference's
              own way of calling)
  device      the same work between device buffers (arclengthReverseInto on CUDA tensors)
  graph       the table and the sampling as one captured step (stepGraph)
  end_to_end  a context created from page-locked host arrays, table, sampling back to host memory, context destroyed
  f32         float curve data, positions and results (the reference's DataType = float)
  noalloc     total lengths without device allocations (gcv_bspline_lengths_noalloc)
  gradients   one training batch of the start-depth network: forward, loss, gradients
  bundle      B-spline dataset files parsed and normalised on the GPU (bundle.load_device)

and a curve family (the generators follow gcurval_gb300/datasets.py, on the GPU so that they are quick):

  ellipses        2D, axes U[0.1, 10], any rotation and centre
  uniform_cubics  2D clamped uniform cubics, random-walk control points
  spatial         3D, degree 3 or 5, 32-256 control points, random interior knots
  uneven          20 % ellipses, 80 % B-splines of degree 2-5 in 2D / 3D, 4-4,096 control points (log-uniform), 5 %
                  near-duplicate interior knots; 16-8,192 samples per curve (log-uniform)
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import gcurval_gb300 as g
from gcurval_gb300 import bundle, datasets, learned

TWO_PI = 2.0 * math.pi


# ---------------------------------------------------------------- the cases
def listed():
    plain, mixed = "plain", "mixed"
    return [
        # a tool that places a few points on a handful of outlines: launches, synchronisations and host work only
        dict(name="ellipses_64_host", call="host", family="ellipses", curves=64, samples=100, precision=plain,
             rtol=1e-10, what="us", spacing="even"),
        # the ellipse sample at its usual size
        dict(name="ellipses_4096", call="device", family="ellipses", curves=4096, samples=1000, precision=plain,
             rtol=1e-10, what="us", spacing="even"),
        # the B-spline sample at its usual size: uniform planar cubics
        dict(name="cubics_10k", call="device", family="uniform_cubics", curves=10000, ctrl=64, samples=1024,
             precision=plain, rtol=1e-10, what="us", spacing="even"),
        # tool paths in space, full precision, points at unordered positions
        dict(name="spatial_points", call="device", family="spatial", curves=1237, samples=333, precision=plain,
             rtol=1e-10, what="points", spacing="random"),
        # the spatial batch in mixed precision
        dict(name="spatial_mixed", call="device", family="spatial", curves=50000, samples=2048, precision=mixed,
             rtol=1e-8, what="us", spacing="even"),
        # one drawing's curves: a small uneven batch, one launch per curve code and phase
        dict(name="uneven_301", call="device", family="uneven", curves=301, precision=mixed, rtol=5e-9, what="us",
             spacing="even", network=False),
        # a service's large uneven batch, resident, with the start-depth network, as one captured step
        dict(name="uneven_network_graph", call="graph", family="uneven", curves=100000, precision=mixed, rtol=5e-9,
             what="us", spacing="even", network=True),
        # the same kind of batch arriving in host memory and going back there, one context per batch
        dict(name="uneven_end_to_end", call="end_to_end", family="uneven", curves=3000, precision=mixed, rtol=5e-9,
             what="points", spacing="even", network=False),
        # float data at the reference's float tolerance
        dict(name="cubics_f32", call="f32", family="uniform_cubics", curves=3001, ctrl=64, samples=500,
             precision=mixed, rtol=1e-6, what="points", spacing="even"),
        # lengths only, inside another library's allocator
        dict(name="cubics_noalloc", call="noalloc", family="uniform_cubics", curves=16384, ctrl=64, rtol=1e-10),
        # one batch of the network's training
        dict(name="network_gradients", call="gradients", rows=8192),
        # four dataset files of a thousand curves
        dict(name="bundle_4x1000", call="bundle", files=4, curves=1000),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    call = rng.choice(["host", "device", "device", "device", "device", "graph", "end_to_end", "f32", "noalloc",
                       "gradients", "bundle"])
    if call == "gradients":
        return dict(call=call, rows=_log_int(rng, 256, 8192))
    if call == "bundle":
        return dict(call=call, files=rng.randint(1, 4), curves=_log_int(rng, 50, 1000))
    if call == "noalloc":
        ctrl = _log_int(rng, 8, 200)
        return dict(call=call, family="uniform_cubics", curves=_log_int(rng, 100, 1_000_000 // (ctrl - 3)), ctrl=ctrl,
                    rtol=1e-10)
    if call == "f32":
        return dict(call=call, family="uniform_cubics", curves=_log_int(rng, 50, 10000), ctrl=_log_int(rng, 8, 128),
                    samples=_log_int(rng, 16, 1024), precision="mixed", rtol=1e-6,
                    what=rng.choice(["us", "points"]), spacing=rng.choice(["even", "random"]))
    family = rng.choice(["ellipses", "uniform_cubics", "spatial", "uneven"])
    if call == "graph":
        family = "uneven"
    precision = rng.choice(["plain", "mixed"])
    most = {"ellipses": 8192, "uniform_cubics": 16000, "spatial": 5000, "uneven": 2000}[family]
    if precision == "mixed":
        most = {"spatial": 40000, "uneven": 50000}.get(family, most)
    if call in ("host", "end_to_end"):
        most = min(most, 2000)
    c = dict(call=call, family=family, curves=_log_int(rng, 16, most), precision=precision,
             rtol=1e-10 if precision == "plain" else rng.choice([5e-9, 1e-8]),
             what=rng.choice(["us", "us", "points"]), spacing=rng.choice(["even", "even", "random"]))
    if family == "uniform_cubics":
        c["ctrl"] = _log_int(rng, 8, 128)
    if family == "uneven":
        c["network"] = precision == "mixed" and rng.random() < 0.5
    else:
        c["samples"] = _log_int(rng, 16, 2048)
    return c


# ------------------------------------------------------------------- inputs
def _off(lengths):
    return torch.nn.functional.pad(torch.cumsum(lengths, 0), (1, 0))


def _within(lengths):
    """0, 1, .., lengths[i] - 1 for every i, and the owners i."""
    owner = torch.repeat_interleave(torch.arange(lengths.numel(), device=lengths.device), lengths)
    return torch.arange(owner.numel(), device=lengths.device) - _off(lengths)[owner], owner


def _curves(case, gen):
    """The batch's arrays on the GPU: kind, degree, dim, knot_off, knots, ctrl_off, ctrl, counts."""
    dev = gen.device
    fam, n = case["family"], case["curves"]

    def uni(m, lo=0.0, hi=1.0):
        return torch.rand(m, generator=gen, device=dev, dtype=torch.float64) * (hi - lo) + lo

    def log_int(m, lo, hi):
        return torch.exp(uni(m, math.log(lo), math.log(hi + 1))).floor().long().clamp_(lo, hi)

    bs = torch.ones(n, dtype=torch.bool, device=dev)
    full = lambda v: torch.full((n,), v, dtype=torch.long, device=dev)  # noqa: E731
    degree, dim, nc, sigma, counts = full(3), full(2), full(5), 1.0, full(case.get("samples", 1))
    if fam == "ellipses":
        bs, degree = ~bs, full(0)
    elif fam == "uniform_cubics":
        nc = full(case["ctrl"])
    elif fam == "spatial":
        degree, dim, sigma = torch.where(uni(n) < 0.5, 3, 5), full(3), 0.5
        nc = torch.randint(32, 257, (n,), generator=gen, device=dev)
    else:
        bs = uni(n) >= 0.2
        degree = torch.where(bs, torch.randint(2, 6, (n,), generator=gen, device=dev), 0)
        dim = torch.where(bs, torch.randint(2, 4, (n,), generator=gen, device=dev), 2)
        nc = torch.maximum(log_int(n, 4, 4096), degree + 1)
        # the quantiles of the log-uniform distribution in a random order: every batch has as many samples
        q = (torch.arange(n, device=dev, dtype=torch.float64) + 0.5) / n
        counts = torch.exp(math.log(16) + q * math.log(8193 / 16)).long()[torch.randperm(n, generator=gen, device=dev)]
    # knots: clamped, interior ones even or sorted U(0, 1) (normalised exponential spacings)
    nk = torch.where(bs, nc + degree + 1, 2)
    j, owner = _within(nk)
    m = nc - degree - 1  # interior knots
    ko = _off(nk)
    i = (j - degree[owner]).clamp(min=0)
    if fam == "uniform_cubics":
        knots = torch.minimum(i.double() / (m + 1)[owner].double(), torch.ones((), dtype=torch.float64, device=dev))
    else:
        e = -torch.log1p(-uni(j.numel()))
        inside = (i > 0) & (i <= m[owner] + 1)
        cs = torch.cumsum(torch.where(inside, e, 0.0), 0)
        cs = cs - torch.where(ko[:-1] > 0, cs[ko[:-1] - 1], 0.0)[owner]
        knots = cs / cs[ko[1:] - 1][owner].clamp(min=1e-300)
        if fam == "uneven":  # near-duplicates: the previous knot plus 1e-6, kept in order
            pick = (uni(j.numel()) < 0.05) & (i > 1) & (i <= m[owner])
            knots = torch.where(pick, torch.minimum(knots.roll(1) + 1e-6, knots.roll(-1)), knots)
        knots = torch.where(i > m[owner], 1.0, torch.where(i == 0, 0.0, knots))
    if fam in ("ellipses", "uneven"):
        knots = torch.where(bs[owner], knots, j.double() * TWO_PI)
    # control values: random walks, or a, b, rotation, centre
    cl = torch.where(bs, nc * dim, 5)
    j, owner = _within(cl)
    co = _off(cl)
    step = torch.randn(j.numel(), 1, generator=gen, device=dev, dtype=torch.float64)[:, 0] * sigma
    step = torch.where(j < dim[owner], 0.0, step)
    ctrl = torch.empty_like(step)
    for d in (2, 3):
        sel = (dim[owner] == d) & bs[owner]
        if bool(sel.any()):
            w = torch.cumsum(step[sel].view(-1, d), 0)
            first = (j[sel].view(-1, d)[:, 0] == 0).long()
            ctrl[sel] = (w - w[first.bool()][torch.cumsum(first, 0) - 1]).reshape(-1)
    if fam in ("ellipses", "uneven"):
        u = uni(j.numel())
        lo = torch.tensor([0.1, 0.1, 0.0, -100.0, -100.0], dtype=torch.float64, device=dev)
        hi = torch.tensor([10.0, 10.0, TWO_PI, 100.0, 100.0], dtype=torch.float64, device=dev)
        k = j.clamp(max=4)
        ctrl = torch.where(bs[owner], ctrl, lo[k] + u * (hi - lo)[k])
    return dict(kind=bs.to(torch.uint8), degree=degree.to(torch.uint8), dim=dim.to(torch.uint8), knot_off=ko,
                knots=knots, ctrl_off=co, ctrl=ctrl, counts=counts.to(torch.int32))


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    b = _curves(case, gen)
    if case["call"] == "noalloc":
        return b
    n = b["counts"].long()
    j, owner = _within(n)
    if case["spacing"] == "even":
        b["pos"] = j.double() / (n - 1).clamp(min=1)[owner].double()
    else:
        b["pos"] = torch.rand(j.numel(), generator=gen, device="cuda", dtype=torch.float64)
    if case["call"] == "f32":
        for k in ("knots", "ctrl", "pos"):
            b[k] = b[k].float()
    return b


def _training_rows(case, seed):
    """Feature rows and labels with the spread that knot intervals of uneven batches have."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = case["rows"]
    r = lambda *s: torch.rand(*s, generator=gen, device="cuda")  # noqa: E731
    p = torch.randint(2, 6, (n, 1), generator=gen, device="cuda")
    edge = (0.1 + r(n, 5)) * (torch.arange(5, device="cuda") < p)
    cos = torch.where(torch.arange(4, device="cuda") < p - 1, 2 * r(n, 4) - 1, torch.ones(()).cuda())
    X = torch.cat([p * 0.2, torch.randint(0, 2, (n, 1), generator=gen, device="cuda").float(),
                   edge / edge.sum(1, keepdim=True), cos, 0.5 * r(n, 1), 0.25 * torch.randn(n, 2, generator=gen, device="cuda"),
                   0.5 * r(n, 1), torch.full((n, 1), 0.83, device="cuda")], 1)
    depth = (r(n) ** 3 * 6).to(torch.int32)
    share = 0.1 + r(n, 4)
    t = (torch.arange(8, device="cuda") + 0.5) / 4 - 1 + 0.1 * torch.randn(n, 8, generator=gen, device="cuda")
    return X.float().contiguous(), depth, (share / share.sum(1, keepdim=True)).contiguous(), t.contiguous()


def _bundle_files(case, seed):
    """Dataset files: cubics of 4-12 points, coordinates and knots with six digits."""
    rng = np.random.default_rng(seed)
    files = []
    for _ in range(case["files"]):
        out = []
        for nc in rng.permutation(4 + np.arange(case["curves"]) % 9):
            xy = 10.0 + np.cumsum(rng.normal(0.0, 2.0, (2, nc)), axis=1)
            kv = np.concatenate([np.zeros(4), np.sort(rng.random(nc - 4)), np.ones(4)])
            out += ["3 %d %d" % (nc, nc + 4)] + [" ".join(["%.6g" % v for v in row]) for row in (xy[0], xy[1], kv)] + [""]
        files.append("\n".join(out).encode())
    return files


def prepare(case, seed):
    call = case["call"]
    if call == "bundle":
        return dict(call=call, files=_bundle_files(case, seed))
    if call == "gradients":
        return dict(call=call, rows=_training_rows(case, seed),
                    trainer=learned.Trainer(case["rows"], weights=learned.load_model()))
    b = _inputs(case, seed)
    s = dict(call=call, n=case["curves"], b=b)
    if call == "noalloc":
        s.update(ko=b["knot_off"].int(), lengths=torch.empty(case["curves"], dtype=torch.float64, device="cuda"),
                 rtol=case["rtol"])
        torch.cuda.synchronize()
        return s
    s["what"] = g.GCV_RETURN_US if case["what"] == "us" else g.GCV_RETURN_POINTS
    opts = dict(precision=g.GCV_MIXED if case["precision"] == "mixed" else g.GCV_PLAIN_FP64, rtol=case["rtol"],
                learned=bool(case.get("network")))
    width = 1 if case["what"] == "us" else int(b["dim"].max())
    total = int(b["counts"].sum())
    curve = ("kind", "degree", "dim", "knot_off", "knots", "ctrl_off", "ctrl")
    if call == "end_to_end":
        h = {k: v.cpu().numpy() for k, v in b.items()}
        for k in ("knots", "ctrl", "pos"):
            h[k] = g.pinned_copy(h[k])
        s.update(batch=datasets.CurveBatch(*[h[k] for k in curve], h["counts"]), counts=h["counts"], pos=h["pos"],
                 opts=dict(opts, host_in_place=True), b=None,
                 weights=learned.load_model() if opts["learned"] else None, out=g.pinned_empty(total * width))
        return s
    if call == "f32":
        s["calc"] = g.ArclengthCalculateGpu.bsplines(3, 2, b["knot_off"].int(), b["knots"], b["ctrl"], **opts)
    else:
        s["calc"] = g.ArclengthCalculateGpu.from_device_batch(*[b[k] for k in curve], **opts)
    if opts["learned"]:
        s["calc"].set_learned_model(learned.load_model())
    if call == "host":
        s.update(counts=b["counts"].cpu().numpy(), pos=b["pos"].cpu().numpy())
    else:
        real = torch.float32 if call == "f32" else torch.float64
        s.update(counts=b["counts"], pos=b["pos"], out=torch.empty(total * width, dtype=real, device="cuda"),
                 lengths=torch.empty(case["curves"], dtype=real, device="cuda"))
    torch.cuda.synchronize()
    return s


# --------------------------------------------------------------------- a pass
def run(s):
    call = s["call"]
    if call == "bundle":
        return bundle.load_device(s["files"])
    if call == "gradients":
        return s["trainer"].gradients(*s["rows"])
    if call == "noalloc":
        capped = ctypes.c_int64()
        p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        lib = g.load()
        st = lib.gcv_bspline_lengths_noalloc(s["n"], 3, 2, p(s["ko"]), p(s["b"]["knots"]), p(s["b"]["ctrl"]), s["rtol"],
                                             30, p(s["lengths"]), None, ctypes.byref(capped))
        if st != 0:
            raise g.GcvError(st, lib.gcv_last_error().decode())
        return s["lengths"]
    if call == "end_to_end":
        with g.ArclengthCalculateGpu.from_batch(s["batch"], **s["opts"]) as calc:
            if s["weights"] is not None:
                calc.set_learned_model(s["weights"])
            calc.createArclengthTable()
            lengths = calc.getAllCurveArclengths()
            calc.arclengthReverseInto(s["counts"], s["pos"], s["out"], True, s["what"])
        return lengths, s["out"]
    calc = s["calc"]
    if call == "graph":
        calc.stepGraph(s["counts"], s["pos"], s["out"], True, s["what"])
        return calc.getAllCurveArclengths(s["lengths"]), s["out"]
    calc.createArclengthTable()
    if call == "host":
        lengths = calc.getAllCurveArclengths()
        return lengths, calc.arclengthReverse(s["counts"], s["pos"], True, g.GCV_HOST, s["what"]).numpy().reshape(-1)
    lengths = calc.getAllCurveArclengths(s["lengths"])
    calc.arclengthReverseInto(s["counts"], s["pos"], s["out"], True, s["what"])
    return lengths, s["out"]


# ----------------------------------------------------------------------- work
def work(case):
    """Each input read and each output written once; one 15-node panel per knot interval and one 8-node sum per sample
    (2 D p multiply-adds and a norm per node): the least the adaptive method can do."""
    call = case["call"]
    if call == "gradients":
        n = case["rows"]
        params = 16 * 128 + 2 * 128 * 128 + 128 * 32
        return dict(bytes=4.0 * (n * (16 + 1 + 4 + 8) + 2 * params), flops=6.0 * n * params)
    if call == "bundle":
        values = case["files"] * case["curves"] * (3 * 8 + 4)  # 8 points a curve on average
        return dict(bytes=values * (8.0 + 8.0), flops=8.0 * values)
    fam, n = case["family"], case["curves"]
    p, d, nc = {"ellipses": (1, 2, 2), "uniform_cubics": (3, 2, case.get("ctrl", 0)), "spatial": (4, 3, 144),
                "uneven": (3.5, 2.5, 0.8 * 590 + 0.4)}[fam]
    samples = n * (1311 if fam == "uneven" else case.get("samples", 0))
    width = d if case.get("what") == "points" else 1
    real = 4.0 if call == "f32" else 8.0
    node = 2 * d * p + 2 * d
    intervals = n * (1 if fam == "ellipses" else nc - p)
    return dict(bytes=real * (n * (nc * (1 + d) + p + 1) + samples * (1 + width) + n),
                flops=15.0 * intervals * node + 8.0 * samples * node)


# ------------------------------------------------- the same outputs in 64 bits
_X, _W = (torch.from_numpy(a) for a in np.polynomial.legendre.leggauss(12))


def _de_boor(win, pts, t, q, at):
    """Degree q de Boor at t [n, m]: points pts [n, q + 1, D], knots win[:, j + at] = U[span - q + j]."""
    d = [pts[:, j, None, :] for j in range(q + 1)]
    for r in range(1, q + 1):
        for j in range(q, r - 1, -1):
            a, b = win[:, j + at, None], win[:, j + at + q + 1 - r, None]
            al = ((t - a) / (b - a))[..., None]
            d[j] = (1 - al) * d[j - 1] + al * d[j]
    return d[q].expand(-1, t.shape[1], -1)


class _Splines:
    """The knot intervals of positive width of some B-splines of one degree and dimension."""

    def __init__(self, b, curves, p, D):
        ko, co = b["knot_off"][curves], b["ctrl_off"][curves]
        j, o = _within((b["knot_off"][curves + 1] - ko) - 2 * p - 1)
        at = ko[o] + j + p
        t0, t1 = b["knots"][at], b["knots"][at + 1]
        keep = t1 > t0
        j, o, at = j[keep], o[keep], at[keep]
        self.owner, self.t0, self.t1, self.p = o, t0[keep], t1[keep], p
        self.win = b["knots"][at[:, None] + torch.arange(-p + 1, p + 1, device=at.device)]
        i = co[o][:, None] + (j[:, None] + torch.arange(p + 1, device=at.device)) * D
        self.pts = b["ctrl"][i[..., None] + torch.arange(D, device=at.device)]
        den = self.win[:, p:] - self.win[:, :p]
        q = p * (self.pts[:, 1:] - self.pts[:, :-1]) / den[..., None]
        # dC/dv as a polynomial in the local variable v in [-1, 1]: from its values at p points
        v = torch.cos((torch.arange(p, device=at.device, dtype=torch.float64) + 0.5) * (math.pi / p))
        hw = 0.5 * (self.t1 - self.t0)
        val = _de_boor(self.win, q, self.t0[:, None] + (v + 1) * hw[:, None], p - 1, 0) * hw[:, None, None]
        inv = torch.linalg.inv(torch.stack([v ** k for k in range(p)], 1))
        self.c = torch.einsum("kj,njd->nkd", inv, val)

    def take(self, s):
        return self.c[s]

    @staticmethod
    def speed(c, v):
        s = 0
        for d in range(c.shape[2]):
            x = c[:, -1, d, None].expand_as(v)
            for k in range(c.shape[1] - 2, -1, -1):
                x = x * v + c[:, k, d, None]
            s = s + x * x
        return s.sqrt()

    def points(self, s, t):
        return _de_boor(self.win[s], self.pts[s], t[:, None], self.p, -1)[:, 0]


class _Ellipses:
    def __init__(self, b, curves):
        self.prm = b["ctrl"][b["ctrl_off"][curves][:, None] + torch.arange(5, device=curves.device)]
        self.owner = torch.arange(curves.numel(), device=curves.device)
        self.t0 = torch.zeros(curves.numel(), dtype=torch.float64, device=curves.device)
        self.t1 = self.t0 + TWO_PI

    def take(self, s):
        return self.prm[s]

    @staticmethod
    def speed(c, v):
        t = (v + 1) * math.pi
        return math.pi * torch.hypot(c[:, :1] * t.sin(), c[:, 1:2] * t.cos())

    def points(self, s, t):
        a, b, r, cx, cy = self.prm[s].unbind(1)
        x, y = a * t.cos(), b * t.sin()
        return torch.stack([r.cos() * x - r.sin() * y + cx, r.sin() * x + r.cos() * y + cy], 1)


def _gauss(f, c, a, b):
    h = 0.5 * (b - a)
    return (f.speed(c, (a + h)[:, None] + h[:, None] * _X.to(a.device)) * _W.to(a.device)).sum(1) * h


def _solve(f, n_curves, target_of, counts):
    """Lengths, and interval and parameter of every sample, by bisection of the intervals to 1e-13 and Newton."""
    dev = f.t0.device
    seg = torch.arange(f.t0.numel(), device=dev)
    a = torch.full((seg.numel(),), -1.0, dtype=torch.float64, device=dev)
    b = -a
    whole = val = _gauss(f, f.take(seg), a, b)
    done = []
    for level in range(60):
        c, m = f.take(seg), 0.5 * (a + b)
        lo, hi = _gauss(f, c, a, m), _gauss(f, c, m, b)
        ok = (lo + hi - val).abs() <= 1e-13 * whole[seg]
        done += [(seg[ok], a[ok], m[ok], lo[ok]), (seg[ok], m[ok], b[ok], hi[ok])]
        if bool(ok.all()) or level == 59:
            break
        k = ~ok
        seg, a, b, val = torch.cat([seg[k]] * 2), torch.cat([a[k], m[k]]), torch.cat([m[k], b[k]]), torch.cat([lo[k], hi[k]])
    seg, a, b, val = (torch.cat(x) for x in zip(*done))
    o = torch.argsort(a)
    o = o[torch.argsort(seg[o], stable=True)]
    seg, a, b, val = seg[o], a[o], b[o], val[o]
    cum = torch.cumsum(val, 0)
    first = torch.searchsorted(f.owner[seg].contiguous(), torch.arange(n_curves + 1, device=dev))
    base = torch.nn.functional.pad(cum, (1, 0))[first]
    lengths = torch.zeros(n_curves, dtype=torch.float64, device=dev).index_add_(0, f.owner[seg], val)
    if counts is None:
        return lengths, None, None
    target, owner = target_of(lengths)
    leaf = torch.searchsorted(cum, base[owner] + target)
    leaf = torch.minimum(torch.maximum(leaf, first[owner]), first[owner + 1] - 1)
    r = target - (cum[leaf] - val[leaf] - base[owner])
    s, lo, hi = seg[leaf], a[leaf], b[leaf]
    left, c = lo, f.take(s)
    v = lo + (hi - lo) * (r / val[leaf]).clamp(0, 1)
    for _ in range(12):
        F = _gauss(f, c, left, v) - r
        lo, hi = torch.where(F < 0, v, lo), torch.where(F > 0, v, hi)
        nv = v - F / f.speed(c, v[:, None])[:, 0]
        nv = torch.where((nv >= lo) & (nv <= hi), nv, 0.5 * (lo + hi))
        moved = float((nv - v).abs().max()) if v.numel() else 0.0
        v = nv
        if moved < 1e-15:
            break
    t0, t1 = f.t0[s], f.t1[s]
    hw = 0.5 * (t1 - t0)
    return lengths, s, torch.where(v <= 0, t0 + (v + 1) * hw, t1 + (v - 1) * hw)


def _exact_curves(case, b):
    b = {k: v.double() if v.is_floating_point() else v for k, v in b.items()}
    n = case["curves"]
    counts = None if case["call"] == "noalloc" else b["counts"].long()
    degree, dim = b["degree"].long(), b["dim"].long()
    code = torch.where(b["kind"] == 0, 0, degree * 4 + dim)
    lengths = torch.zeros(n, dtype=torch.float64, device="cuda")
    width = 1 if case.get("what", "us") == "us" else int(dim.max())
    off = None if counts is None else _off(counts)
    out = None if counts is None else torch.zeros(int(off[-1]), width, dtype=torch.float64, device="cuda")
    size = (b["knot_off"][1:] - b["knot_off"][:-1]) + (0 if counts is None else counts)
    for cd in code.unique().tolist():
        curves = (code == cd).nonzero()[:, 0]
        part = torch.cumsum(size[curves], 0) // 1_000_000
        for k in part.unique().tolist():
            sel = curves[part == k]
            f = _Ellipses(b, sel) if cd == 0 else _Splines(b, sel, cd // 4, cd % 4)
            if counts is not None:
                j, o = _within(counts[sel])
                at = off[sel][o] + j

            def target_of(lens):
                return b["pos"][at] * lens[o], o

            lengths[sel], s, u = _solve(f, sel.numel(), target_of, counts)
            if counts is not None:
                if case["what"] == "us":
                    out[at, 0] = u
                else:
                    q = f.points(s, u)
                    out[at, :q.shape[1]] = q
    return lengths if counts is None else (lengths, out.reshape(-1))


def _exact_gradients(case, seed):
    X, depth, share, t = _training_rows(case, seed)
    w = torch.from_numpy(learned.load_model()).double().cuda().requires_grad_()
    at, h = 0, X.double()
    for k, m in ((16, 128), (128, 128), (128, 128), (128, 32)):
        h = h @ w[at:at + k * m].view(k, m) + w[at + k * m:at + k * m + m]
        at += k * m + m
        if m == 128:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    ls = torch.log_softmax(h[:, 13:17], 1)
    parts = torch.stack([torch.nn.functional.cross_entropy(h[:, :13], depth.long()), -(share.double() * ls).sum(1).mean(),
                         0.5 * (h[:, 17:25] - t.double()).square().sum(1).mean()])
    parts.sum().backward()
    return w.grad, parts.detach()


def _exact_bundle(case, seed):
    knots, ctrl, nk, nc = [], [], [], []
    for text in _bundle_files(case, seed):
        v, i = np.array(text.split(), dtype=np.float64), 0
        while i < v.size:
            m, k = int(v[i + 1]), int(v[i + 2])
            q = np.stack([v[i + 3:i + 3 + m], v[i + 3 + m:i + 3 + 2 * m]], axis=1)
            q = q - q.mean(axis=0)
            ctrl.append((q / np.abs(q).max()).reshape(-1))
            knots.append(v[i + 3 + 2 * m:i + 3 + 2 * m + k])
            nk.append(k)
            nc.append(2 * m)
            i += 3 + 2 * m + k
    return None, None, None, None, np.concatenate(knots), None, np.concatenate(ctrl)


def exact(case, seed):
    if case["call"] == "bundle":
        return _exact_bundle(case, seed)
    if case["call"] == "gradients":
        return _exact_gradients(case, seed)
    return _exact_curves(case, _inputs(case, seed))
