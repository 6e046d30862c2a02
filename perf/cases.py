"""Workloads of the compact-difference operators, as a solver's program calls them.

``listed()`` names twelve of them and ``draw`` makes more of the same kinds:
operator sweeps along x, y and z (cd06 / cd10 derivatives, the cf90 filter;
periodic lines and lines with one-sided, symmetric or antisymmetric closures),
field operators that sum several derivatives, a differentiated loss, a batch
of uneven fields replayed from a CUDA graph, and the staggered scheme.  Extents
run from 24 to 1024 points along each axis, odd ones included, and fields from
2^15 to 2^27 points; everything is FP64, as the library is.

A case is a dict of plain values:

    what    "sweep", "vector", "adjoint", "batch" or "stagg"
    scheme  "cd06", "cd10" or "cf90"    (sweep)
    order   1 or 2, the derivative      (sweep)
    n       "n1 n2 n3", x first
    per     one letter per axis: p periodic, w with walls    (stagg: z alone)
    bc      "bc1 bcn" of x, y and z: the closures of an axis with walls

``exact`` restates the schemes as dense line operators: band matrices and
stencils in numpy's extended precision, D = A^-1 B rounded to 64 bits, applied
by matrix products.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import padeops_b200 as pb
from padeops_b200 import field_ops
from padeops_b200.autograd import compact_op
from padeops_b200.batch import Batch
from padeops_b200.operators import Derivatives, Filters
from padeops_b200.stagg import cd06stagg

FILTER, D1, D2 = 0, 1, 2
MIN_POINTS, MAX_POINTS = 2 ** 15, 2 ** 27
BATCH_DIMS = (32, 48, 64, 96, 128, 192, 256, 384)
STAGG_OPS = ("ddz_E2C", "ddz_C2E", "d2dz2_C2C", "InterpZ_E2C", "InterpZ_C2E")


# ---- the cases --------------------------------------------------------------------
def listed():
    zero = "0 0 0 0 0 0"
    return [
        # a solver's smallest production-like grid: three calls of a few microseconds each
        {"name": "cd06_periodic_64", "what": "sweep", "scheme": "cd06", "order": 1, "n": "64 64 64", "per": "ppp",
         "bc": zero},
        # a ragged debugging grid, every axis with walls: latency, partial tiles, short odd lines
        {"name": "cd10_walls_50x33x40", "what": "sweep", "scheme": "cd10", "order": 1, "n": "50 33 40", "per": "www",
         "bc": "0 0 1 -1 0 1"},
        # isotropic turbulence in a periodic box on one GPU: first and second derivatives, and the filter that
        # such a solver applies to every field each time step
        {"name": "cd10_periodic_512", "what": "sweep", "scheme": "cd10", "order": 1, "n": "512 512 512", "per": "ppp",
         "bc": zero},
        {"name": "cd10_second_periodic_512", "what": "sweep", "scheme": "cd10", "order": 2, "n": "512 512 512",
         "per": "ppp", "bc": zero},
        {"name": "cf90_periodic_512", "what": "sweep", "scheme": "cf90", "order": 0, "n": "512 512 512", "per": "ppp",
         "bc": zero},
        # a channel: periodic along and across, one-sided closures at the walls
        {"name": "cd06_channel_1024x512x256", "what": "sweep", "scheme": "cd06", "order": 1, "n": "1024 512 256",
         "per": "ppw", "bc": zero},
        {"name": "cd10_channel_1024x512x256", "what": "sweep", "scheme": "cd10", "order": 1, "n": "1024 512 256",
         "per": "ppw", "bc": zero},
        # odd extents (no axis of which the copy engine can move), walls on every axis, the filter
        {"name": "cf90_walls_255x127x191", "what": "sweep", "scheme": "cf90", "order": 0, "n": "255 127 191",
         "per": "www", "bc": "0 0 0 -1 1 1"},
        # right-hand side of a flow solver: divergence of a vector field and laplacian of a scalar, accumulated
        {"name": "vector_384x256x192", "what": "vector", "n": "384 256 192", "per": "ppw", "bc": "0 0 0 0 1 -1"},
        # a differentiated mismatch of two operators: loss, residual and gradient
        {"name": "adjoint_256", "what": "adjoint", "n": "256 256 256"},
        # many uneven fields (multiblock grid), one CUDA-graph replay
        {"name": "batch_32_fields", "what": "batch", "fields": 32, "cap": 1 << 27, "pick": 4},
        # staggered wall-normal operators of an incompressible solver (cell and edge grids)
        {"name": "stagg_192x192x256", "what": "stagg", "n": "192 192 256", "per": "w", "top": 1, "bot": -1},
    ]


def _extent(rng):
    v = int(round(math.exp(rng.uniform(math.log(24), math.log(1024)))))
    r = rng.random()
    if r < 0.35:
        v = max(24, v // 16 * 16)
    elif r < 0.65:
        v |= 1
    return min(v, 1024)


def _shape(rng, most=MAX_POINTS):
    while True:
        n = [_extent(rng) for _ in range(3)]
        if MIN_POINTS <= n[0] * n[1] * n[2] <= most:
            return " ".join(str(v) for v in n)


def draw(rng):
    per = "".join(rng.choice("pw") for _ in range(3))
    bc = " ".join(str(rng.choice((0, 0, 1, -1))) for _ in range(6))
    r = rng.random()
    if r < 0.64:
        scheme, order = rng.choice((("cd06", 1), ("cd10", 1), ("cd10", 2), ("cf90", 0)))
        if scheme == "cd06":
            bc = "0 0 0 0 0 0"  # its closures are fixed at init
        return {"what": "sweep", "scheme": scheme, "order": order, "n": _shape(rng), "per": per, "bc": bc}
    if r < 0.74:
        return {"what": "vector", "n": _shape(rng, MAX_POINTS // 4), "per": per, "bc": bc}
    if r < 0.84:
        return {"what": "adjoint", "n": _shape(rng, MAX_POINTS // 4)}
    if r < 0.92:
        return {"what": "batch", "fields": rng.randint(8, 64), "cap": rng.choice((1 << 22, 1 << 24, 1 << 26)),
                "pick": rng.randint(0, 9999)}
    return {"what": "stagg", "n": _shape(rng, MAX_POINTS // 4), "per": rng.choice("pw"), "top": rng.choice((1, -1)),
            "bot": rng.choice((1, -1))}


def _sizes(case):
    return [int(v) for v in case["n"].split()]


def _periodic(case):
    return [v == "p" for v in case["per"]]


def _closures(case):
    v = [int(b) for b in case["bc"].split()]
    return [(v[0], v[1]), (v[2], v[3]), (v[4], v[5])]


# ---- inputs -----------------------------------------------------------------------
def _spacing(n, periodic):
    return 2 * math.pi / n if periodic else 1.0 / (n - 1)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed) % (2 ** 63))


def _field(gen, shape, per):
    """Random-phase field of energy spectrum k^-5/3 up to 2/3 of the resolved wavenumbers, unit RMS,
    plus a cubic along every axis that is not periodic (walls then see values of their own)."""
    n3, n2, n1 = shape
    dev = gen.device

    def freq(n, real=False):
        k = torch.fft.rfftfreq(n, 1.0 / n, dtype=torch.float64, device=dev) if real else \
            torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev)
        return k

    k2 = freq(n3)[:, None, None] ** 2 + freq(n2)[None, :, None] ** 2 + freq(n1, True)[None, None, :] ** 2
    amp = torch.where((k2 >= 1) & (k2 <= (max(shape) / 3.0) ** 2), k2.clamp(min=1.0) ** (-11.0 / 12.0),
                      torch.zeros((), dtype=torch.float64, device=dev))
    del k2
    phase = torch.rand(amp.shape, dtype=torch.float64, device=dev, generator=gen).mul_(2 * math.pi)
    f = torch.fft.irfftn(torch.polar(amp, phase), s=shape)
    del amp, phase
    f /= f.square().mean().sqrt()
    for ax, (n, p) in enumerate(zip((n1, n2, n3), per)):
        if not p:
            c = torch.rand(4, dtype=torch.float64, device=dev, generator=gen) * 2 - 1
            t = torch.linspace(0, 1, n, dtype=torch.float64, device=dev)
            poly = c[0] + t * (c[1] + t * (c[2] + t * c[3]))
            f += poly.reshape([-1 if d == 2 - ax else 1 for d in range(3)])
    return f.contiguous()


def _torch_shape(case):
    n1, n2, n3 = _sizes(case)
    return (n3, n2, n1)


def _derivatives(case, methods):
    der = Derivatives()
    n, per = _sizes(case), _periodic(case)
    der.init(*n, *[_spacing(a, p) for a, p in zip(n, per)], *per, *methods)
    return der


def _batch_plan(case):
    """The batch's items: (shape, scheme, periodic, axis) each, from the case alone."""
    rng = np.random.default_rng([case["pick"], case["fields"]])
    out, total = [], 0
    while len(out) < case["fields"]:
        shape = tuple(int(v) for v in rng.choice(BATCH_DIMS, 3))
        item = (shape, "cd10" if rng.integers(2) else "cd06", bool(rng.integers(2)), int(rng.integers(1, 4)))
        pts = shape[0] * shape[1] * shape[2]
        # an even share each, on average: what is left is never spent on one field
        if pts <= max(2 * (case["cap"] - total) // (case["fields"] - len(out)), 32 ** 3):
            out.append(item)
            total += pts
    return out


def _inputs(case, seed):
    gen = _generator(seed)
    what = case["what"]
    if what == "sweep":
        return [_field(gen, _torch_shape(case), _periodic(case))]
    if what == "vector":
        return [_field(gen, _torch_shape(case), _periodic(case)) for _ in range(4)]
    if what == "adjoint":
        return [_field(gen, _torch_shape(case), [True, True, False]) for _ in range(2)]
    if what == "batch":
        return [_field(gen, shape, [periodic] * 3) for shape, _, periodic, _ in _batch_plan(case)]
    n1, n2, n = _sizes(case)
    edges, cells = (_field(gen, (m, n2, n1), [True] * 3) for m in (n + 1, n))
    if case["per"] == "p":
        edges[n] = edges[0]
    return [edges, cells]


def prepare(case, seed):
    what, x = case["what"], _inputs(case, seed)
    st = {"case": case, "x": x}
    if what == "sweep":
        if case["scheme"] == "cf90":
            st["op"] = Filters()
            st["op"].init(*_sizes(case), *["cf90"] * 3, *_periodic(case))
        else:
            st["op"] = _derivatives(case, [case["scheme"]] * 3)
        st["out"] = [torch.empty_like(x[0]) for _ in range(3)]
    elif what == "vector":
        st["op"] = _derivatives(case, ["cd10"] * 3)
        st["out"] = [torch.empty_like(x[0]) for _ in range(2)]
    elif what == "adjoint":
        n1, _, n3 = _sizes(case)
        opx, opz = pb.cd10(), pb.cd06()
        assert opx.init(n1, _spacing(n1, True), True) == 0 and opz.init(n3, _spacing(n3, False), False) == 0
        st["op"] = (opx, opz)
        x[0].requires_grad_(True)
    elif what == "batch":
        items, ops = [], {}
        for f, (shape, scheme, periodic, axis) in zip(x, _batch_plan(case)):
            n = shape[3 - axis]
            key = (scheme, n, periodic)
            if key not in ops:
                ops[key] = pb.cd10() if scheme == "cd10" else pb.cd06()
                assert ops[key].init(n, _spacing(n, periodic), periodic) == 0
            items.append((ops[key], D1, axis, f, torch.empty_like(f), 0, 0))
        st["out"] = [it[4] for it in items]
        st["op"] = Batch(items)
        st["op"].set_graph_branches(4)  # what tune.tune_batch picks for such batches
        st["op"].run_graph()  # captures the graph
    else:
        n1, n2, n = _sizes(case)
        op = cd06stagg()
        if case["per"] == "p":
            assert op.init(n, 2 * math.pi / n) == 0
        else:
            assert op.init(n, 1.0 / n, case["top"] == 1, case["bot"] == 1) == 0
        st["op"] = op
        st["out"] = [torch.empty_like(x[1] if op.sizes(name)[1] == n else x[0]) for name in STAGG_OPS]
    return st


def run(state):
    case, x, op = state["case"], state["x"], state["op"]
    what = case["what"]
    if what == "sweep":
        f, (a, b, c) = x[0], state["out"]
        if case["scheme"] == "cf90":
            calls = (op.filterx, op.filtery, op.filterz)
        elif case["order"] == 1:
            calls = (op.ddx, op.ddy, op.ddz)
        else:
            calls = (op.d2dx2, op.d2dy2, op.d2dz2)
        for call, out, bc in zip(calls, (a, b, c), _closures(case)):
            call(f, out, *bc)
        return [a, b, c]
    if what == "vector":
        div, lap = state["out"]
        bcs = _closures(case)
        field_ops.divergence(op, x[0], x[1], x[2], div, *bcs)
        field_ops.laplacian(op, x[3], lap, *bcs)
        return [div, lap]
    if what == "adjoint":
        u, g = x
        u.grad = None
        res = compact_op(op[0], D1, 1, u) + compact_op(op[1], D1, 3, u) - g
        loss = 0.5 * res.square().sum()
        loss.backward()
        return [loss.detach(), res.detach(), u.grad]
    if what == "batch":
        op.run_graph()
        return list(state["out"])
    n1, n2, n = _sizes(case)
    for name, out in zip(STAGG_OPS, state["out"]):
        getattr(op, name)(x[1] if op.sizes(name)[0] == n else x[0], out, n1, n2)
    return list(state["out"])


# ---- cost -------------------------------------------------------------------------
# flops per point: stencil, and the two sweeps of a tridiagonal or pentadiagonal solve
_FLOPS = {("cd06", 1): 6 + 5, ("cd10", 1): 9 + 9, ("cd10", 2): 13 + 9, ("cf90", 0): 13 + 9}


def work(case):
    """Every application reads its field and writes its result once (an accumulated one also reads it)."""
    what = case["what"]
    if what == "batch":
        plan = _batch_plan(case)
        pts = sum(a * b * c for (a, b, c), _, _, _ in plan)
        return {"bytes": 16 * pts, "flops": sum(a * b * c * _FLOPS[s, 1] for (a, b, c), s, _, _ in plan)}
    pts = math.prod(_sizes(case))
    if what == "sweep":
        return {"bytes": 3 * 16 * pts, "flops": 3 * pts * _FLOPS[case["scheme"], case["order"]]}
    if what == "vector":  # four fields in, two results out
        return {"bytes": 8 * 6 * pts, "flops": pts * 3 * (_FLOPS["cd10", 1] + _FLOPS["cd10", 2])}
    if what == "adjoint":  # two operators, two adjoints, g, residual and gradient
        return {"bytes": (4 * 16 + 3 * 8) * pts, "flops": pts * 2 * (_FLOPS["cd10", 1] + _FLOPS["cd06", 1] + 3)}
    return {"bytes": len(STAGG_OPS) * 16 * pts, "flops": len(STAGG_OPS) * 11 * pts}


def tolerance(case):
    """About four times the distance between this library and ``exact`` measured over the ranges above: at
    most 1.2e-13 for the filter (the condition number of its matrix is near 2000), 2.5e-15 for first
    derivatives, 4.6e-15 for second ones, 6.2e-15 through a gradient; the spread comes from the rounding of
    differences of neighbouring values, which grows with the extents."""
    if case["what"] == "sweep" and case["scheme"] == "cf90":
        return {"rel": 5e-13}
    if case["what"] in ("adjoint", "vector") or case.get("order") == 2:
        return {"rel": 3e-14}
    return {"rel": 2e-14}


# ---- the schemes in plain numpy / torch -------------------------------------------------
_LD = np.longdouble


def _ld(*v):
    return [_LD(a) for a in v]


def _interior(scheme, order):
    """(left-hand side half band [1, alpha, beta], stencil half widths, parity of the stencil)."""
    one = _LD(1)
    if scheme == "cd06":
        return [one, one / 3], [_LD(0), _LD(7) / 9, one / 36], -1
    if scheme == "cd10" and order == 1:
        return [one, one / 2, one / 20], [_LD(0), _LD(17) / 24, _LD(101) / 600, one / 600], -1
    if scheme == "cd10":
        a, b, c = _LD(1065) / 1798, _LD(1038) / 899 / 4, _LD(79) / 1798 / 9
        return [one, _LD(334) / 899, _LD(43) / 1798], [-2 * (a + b + c), a, b, c], 1
    return ([one, _LD("0.66624"), _LD("0.16688")],
            [_LD("0.99965"), _LD("0.66652"), _LD("0.16674"), _LD("0.00004"), _LD("-0.000005")], 1)


def _one_sided(scheme, order):
    """Closure rows of a one-sided left end: [({offset: left-hand side}, {offset: stencil})], from the wall in.
    Each row may be scaled freely (both sides alike)."""
    one = _LD(1)
    sym = lambda *h: {o: h[abs(o)] for o in range(-len(h) + 1, len(h))}  # noqa: E731
    anti = lambda *h: {o: (h[abs(o) - 1] if o > 0 else -h[abs(o) - 1])  # noqa: E731
                       for o in range(-len(h), len(h) + 1) if o}
    ahead = lambda *h: dict(enumerate(h))  # noqa: E731
    first = ({0: one, 1: _LD(3)}, ahead(-_LD(17) / 6, _LD(3) / 2, _LD(3) / 2, -one / 6))
    second = (sym(one, one / 4), anti(_LD(3) / 4))
    if scheme == "cd06":
        ah, q, s = one / 3, _LD(3) / 2, -one / 6
        app = ((40 * ah - 1) * q + 7 * (4 * ah - 1) * s) / (16 * (ah + 2) * q + 8 * (1 - 4 * ah) * s)
        return [first, second, (sym(one, app), anti((app + 2) / 3, (4 * app - 1) / 12))]
    if scheme == "cd10" and order == 1:
        q, s = _LD(3) / 2, -one / 6
        qh, rh, sh = _LD(17) / 24, _LD(101) / 600, one / 600
        a4 = (8 * rh - 175 * sh) / (18 * rh - 550 * sh)
        b4, q4, r4, s4 = (8 * a4 - 3) / 20, (12 - 7 * a4) / 12, (568 * a4 - 183) / 600, (9 * a4 - 4) / 300
        t1 = s * (rh + 2 * sh) - q * (qh + rh + sh)
        t2 = qh + rh - sh * (q4 / s4 - 1)
        a3 = ((17 * t1) / (72 * (q + s) * t2) - _LD(8) / 9) / ((19 * t1) / (24 * (q + s) * t2) - one / 3)
        return [first, second,
                (sym(one, a3, (3 * a3 - 1) / 12), anti((8 - 3 * a3) / 9, (57 * a3 - 17) / 72)),
                (sym(one, a4, b4), anti(q4, r4, s4))]
    if scheme == "cd10":
        al, a3 = _LD(11), _LD(344) / 1179
        qa, qb = (696 - 1191 * a3) / 428, (2454 * a3 - 294) / 535 / 4
        w2 = 4 * (1 - one / 10) / 3
        return [({0: one, 1: al}, ahead((11 * al + 35) / 12, -(5 * al + 26) / 3, (al + 19) / 2, (al - 14) / 3,
                                        (11 - al) / 12)),
                (sym(one, one / 10), sym(-2 * w2, w2)),
                (sym(one, a3, (38 * a3 - 9) / 214), sym(-2 * (qa + qb), qa, qb))]
    return [({0: one}, {0: one}),
            (sym(one, _LD("0.4997")), sym(*_ld("0.9997", "0.49985"))),
            (sym(one, *_ld("0.66624", "0.16688")), sym(*_ld("0.99952", "0.66656", "0.1668"))),
            (sym(one, *_ld("0.66624", "0.16688")), sym(*_ld("0.99968", "0.66652", "0.16672", "0.00004")))]


def _at_line(i, n, periodic, left, right):
    """Point i of a line of n points carried on beyond its ends: (index, sign); left and right are the
    signs of a mirror about the end points (0: nothing lies beyond)."""
    if periodic:
        return i % n, 1
    if i < 0:
        return -i, left
    if i >= n:
        return 2 * (n - 1) - i, right
    return i, 1


def _at_half(i, n, periodic, left, right):
    """The same for cells, whose mirrors lie half a cell beyond the end points."""
    if periodic:
        return i % n, 1
    if i < 0:
        return -1 - i, left
    if i >= n:
        return 2 * n - 1 - i, right
    return i, 1


def _solve_rows(lhs, B, at, periodic, special):
    """A^-1 B in extended precision: A has the symmetric band lhs, its rows closed by `at`, except the rows
    of `special` ({row: [(column, coefficient)]})."""
    n, m = B.shape[0], len(lhs) - 1
    if periodic:
        k = np.arange(n)
        angle = (np.outer(k, k) % n) * (2 * np.arccos(_LD(-1)) / n)
        c = np.cos(angle)
        inv = (c @ (1 / (lhs[0] + sum(2 * v * c[:, j % n] for j, v in enumerate(lhs) if j)))) / n
        first = sum(B[0, j] * np.roll(inv, j) for j in np.nonzero(B[0])[0])  # circulant: one row tells all
        return np.stack([np.roll(first, i) for i in range(n)])
    band = np.zeros((n, 2 * m + 1), _LD)
    for i in range(n):
        row = special.get(i)
        if row is None:
            row = [(j, s * lhs[abs(o)]) for o in range(-m, m + 1) for j, s in (at(i + o),)]
        for j, c in row:
            band[i, j - i + m] += c
    B = B.copy()
    for i in range(n):  # elimination of the band, all right-hand sides at once
        for k in range(1, m + 1):
            if i + k < n and band[i + k, m - k] != 0:
                w = band[i + k, m - k] / band[i, m]
                hi = min(m, n - 1 - i)
                band[i + k, m - k:m - k + hi + 1] -= w * band[i, m:m + hi + 1]
                B[i + k] -= w * B[i]
    for i in range(n - 1, -1, -1):
        for k in range(1, m + 1):
            if i + k < n:
                B[i] -= band[i, m + k] * B[i + k]
        B[i] /= band[i, m]
    return B


@functools.lru_cache(maxsize=64)
def _dense(scheme, order, n, dx, periodic, bc1, bcn):
    """D = A^-1 B of one line, float64, computed in extended precision."""
    lhs, rhs, parity = _interior(scheme, order)
    w = len(rhs) - 1
    B = np.zeros((n, n), _LD)
    for i in range(n):
        for o in range(-w, w + 1):
            j, s = _at_line(i + o, n, periodic, bc1, bcn)
            B[i, j] += s * rhs[abs(o)] * (parity if o < 0 else 1)
    special = {}
    if not periodic:
        flip = 1 if parity > 0 else -1  # the line read from its other end
        for r, (a, b) in enumerate(_one_sided(scheme, order)):
            if bc1 == 0:
                special[r] = [(r + o, c) for o, c in a.items()]
                B[r] = 0
                for o, c in b.items():
                    B[r, r + o] = c
            if bcn == 0:
                i = n - 1 - r
                special[i] = [(i - o, c) for o, c in a.items()]
                B[i] = 0
                for o, c in b.items():
                    B[i, i - o] = flip * c
    # a mirrored field's result has the operator's parity about the same point
    D = _solve_rows(lhs, B, lambda i: _at_line(i, n, periodic, bc1 * parity, bcn * parity), periodic, special)
    return (D * (_LD(1) / _LD(dx)) ** order).astype(np.float64)


@functools.lru_cache(maxsize=64)
def _dense_stagg(name, n, dx, periodic, bot, top):
    """The same for a staggered operator between cells (n) and edges (n + 1; a periodic line's last edge
    repeats its first)."""
    one = _LD(1)
    src, dst = ("E", "C") if name.endswith("E2C") else (("C", "E") if name.endswith("C2E") else ("C", "C"))
    if name.startswith("ddz"):
        lhs, taps, order, parity = [one, _LD(9) / 62], [_LD(63) / 62, _LD(17) / 62 / 3], 1, -1
    elif name.startswith("d2"):
        lhs, order, parity = [one, _LD(2) / 11], 2, 1
        taps = [_LD(12) / 11, _LD(3) / 11 / 4]
    else:
        lhs, taps, order, parity = [one, _LD(3) / 10], [_LD(3) / 4, one / 20], 0, 1
    sizes = {"C": n, "E": n if periodic else n + 1}
    where = {"C": _at_half, "E": _at_line}
    nin, nout = sizes[src], sizes[dst]
    B = np.zeros((nout, nin), _LD)
    for i in range(nout):
        if src == dst:
            pairs = [(i + o, taps[abs(o) - 1]) for o in (-2, -1, 1, 2)] + [(i, -2 * (taps[0] + taps[1]))]
        else:  # taps at half cells: cell i lies between edges i and i + 1
            up = i + 1 if dst == "C" else i
            pairs = [(up + k, taps[k]) for k in (0, 1)] + [(up - 1 - k, parity * taps[k]) for k in (0, 1)]
        for j, c in pairs:
            jj, s = where[src](j, nin, periodic, bot, top)
            B[i, jj] += s * c
    D = _solve_rows(lhs, B, lambda i: where[dst](i, nout, periodic, bot * parity, top * parity), periodic, {})
    D = (D * (_LD(1) / _LD(dx)) ** order).astype(np.float64)
    if periodic and src == "E":
        D = np.concatenate([D, np.zeros((nout, 1))], axis=1)
    if periodic and dst == "E":
        D = np.concatenate([D, D[:1]], axis=0)
    return D


def _apply(D, f, axis):
    """D along x (1), y (2) or z (3) of an (n3, n2, n1) field."""
    D = torch.from_numpy(D).to(f.device)
    if axis == 1:
        return f @ D.T
    if axis == 2:
        return torch.matmul(D, f)
    return (D @ f.reshape(f.shape[0], -1)).reshape(D.shape[0], *f.shape[1:])


def exact(case, seed):
    what, x = case["what"], _inputs(case, seed)

    def line(scheme, order, axis, bc=(0, 0)):
        n, p = _sizes(case)[axis - 1], _periodic(case)[axis - 1]
        bc = (0, 0) if p or scheme == "cd06" else bc
        return _dense(scheme, order, n, 1.0 if order == 0 else _spacing(n, p), p, *bc)

    if what == "sweep":
        return [_apply(line(case["scheme"], case["order"], ax, _closures(case)[ax - 1]), x[0], ax)
                for ax in (1, 2, 3)]
    if what == "vector":
        # divergence takes the negated closures of its direction: the components are odd where a scalar is even
        neg = [tuple(-b for b in bc) for bc in _closures(case)]
        div = sum(_apply(line("cd10", 1, ax, neg[ax - 1]), x[ax - 1], ax) for ax in (2, 1, 3))
        lap = sum(_apply(line("cd10", 2, ax, _closures(case)[ax - 1]), x[3], ax) for ax in (2, 1, 3))
        return [div, lap]
    if what == "adjoint":
        u, g = x
        n1, _, n3 = _sizes(case)
        dx = _dense("cd10", 1, n1, _spacing(n1, True), True, 0, 0)
        dz = _dense("cd06", 1, n3, _spacing(n3, False), False, 0, 0)
        res = _apply(dx, u, 1) + _apply(dz, u, 3) - g
        grad = _apply(np.ascontiguousarray(dx.T), res, 1) + _apply(np.ascontiguousarray(dz.T), res, 3)
        return [0.5 * res.square().sum(), res, grad]
    if what == "batch":
        out = []
        for f, (shape, scheme, periodic, axis) in zip(x, _batch_plan(case)):
            n = shape[3 - axis]
            out.append(_apply(_dense(scheme, 1, n, _spacing(n, periodic), periodic, 0, 0), f, axis))
        return out
    n, periodic = _sizes(case)[2], case["per"] == "p"
    h = 2 * math.pi / n if periodic else 1.0 / n
    out = []
    for name in STAGG_OPS:
        D = _dense_stagg(name, n, h, periodic, case["bot"], case["top"])
        out.append(_apply(D, x[0] if D.shape[1] == n + 1 else x[1], 3))
    return out
