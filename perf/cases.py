"""Timed cases of the grid-transfer path, through the package's public calls.

Three kinds of case:

* ``boxes``: independent box-pairs, each with arrays of its own, run as the
  plain drop-in (one ``transfer_data`` per pair) or as one uploaded ``Batch``.
  ``ops`` names the operators, dealt out to the pairs in turn; the region of
  every pair is ``ex`` x ``ey`` x ``ez`` points, or drawn per axis from
  ``lo`` .. ``hi`` with the seed ``geom``.
* ``levels``: nested vertex-centred hierarchies (``nested``), run as one phase
  of ``BergerOliger`` (a batch over all grid functions), as a whole coarse
  step replayed from a CUDA graph, or as the plain drop-in's calls of one step.
* ``served``: a burst of requests to the ``Server`` of an ``Ensemble``.

Fields are sums of smooth separable bumps plus 1e-6 of noise.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import carpet_b200 as cb
from carpet_b200 import bo, hierarchy, serve, transfer
from carpet_b200.amr import BergerOliger, Storage

DT = 1.0 / 64  # coarse time step; the time-interpolated cases sit between two levels

# operator: (operator type, centring, order_space, fine-to-coarse?)
OPS = {
    "copy": (cb.OP_LAGRANGE, cb.VERTEX, 1),
    "vc1": (cb.OP_LAGRANGE, cb.VERTEX, 1),
    "vc3": (cb.OP_LAGRANGE, cb.VERTEX, 3),
    "vc5": (cb.OP_LAGRANGE, cb.VERTEX, 5),
    "eno": (cb.OP_ENO, cb.VERTEX, 3),
    "cc1": (cb.OP_LAGRANGE, cb.CELL, 1),
    "cc3": (cb.OP_LAGRANGE, cb.CELL, 3),
    "cc5": (cb.OP_LAGRANGE, cb.CELL, 5),
    "cceno": (cb.OP_ENO, cb.CELL, 3),
    "mono": (transfer.OP_LAGRANGE_MONOTONE, cb.VERTEX, 5),
    "inject": (cb.OP_LAGRANGE, cb.VERTEX, 1),
    "avg": (cb.OP_LAGRANGE, cb.CELL, 1),
    "avg3": (cb.OP_LAGRANGE, cb.CELL, 3),
    "avg5": (cb.OP_LAGRANGE, cb.CELL, 5),
}
RESTRICT = ("inject", "avg", "avg3", "avg5")


def listed():
    return [
        # one ghost face of a small component through the drop-in call: the
        # smallest call there is, bound by the call and the launch
        dict(name="plain_ghost_face33", kind="boxes", form="plain", ops="copy", pairs=1, ex=3, ey=33, ez=33,
             ntl=1, fp="exact"),
        # the two-level 33^3 hierarchy of the drop-in test: every call of a
        # coarse step (order-3 boundary prolongation, injection, ghost sync)
        dict(name="plain_twolevel33", kind="levels", form="plain", nlevels=2, n=33, px=2, py=1, pz=1, ghost=3,
             buffer=3, order=3, ngf=1),
        # one boundary slab of one 64^3 component, order 5 in space and
        # quadratic in time, as the drop-in makes it
        dict(name="plain_slab64_o5_3tl", kind="boxes", form="plain", ops="vc5", pairs=1, ex=64, ey=12, ez=52,
             ntl=3, fp="exact"),
        # a newly refined 161^3 box filled by one drop-in call
        dict(name="plain_fill161_o5", kind="boxes", form="plain", ops="vc5", pairs=1, ex=161, ey=161, ez=161,
             ntl=1, fp="exact"),
        # the boundary prolongation of one refined level between two coarse
        # times: 129^3 in 8 components, 25 grid functions, order 5, 3 timelevels
        dict(name="phase_prolong_3tl", kind="levels", form="phase", phase="prolong", tl=3, nlevels=2, n=129, px=2,
             py=2, pz=2, ghost=3, buffer=9, order=5, ngf=25, fp="exact"),
        # the ghost sync of the same level
        dict(name="phase_sync", kind="levels", form="phase", phase="sync", tl=1, nlevels=2, n=129, px=2, py=2,
             pz=2, ghost=3, buffer=9, order=5, ngf=25, fp="exact"),
        # the whole coarse step of the five-level hierarchy, one graph replay
        dict(name="step_5levels", kind="levels", form="step", nlevels=5, n=129, px=2, py=2, pz=2, ghost=3,
             buffer=9, order=5, ngf=25, fp="exact"),
        # 256 uneven pairs of mixed operators in one batch (40% vertex order
        # 5, 20% vertex ENO, 20% cell order 3, 20% cell averaging)
        dict(name="uneven_256", kind="boxes", form="batch", ops="vc5,eno,cc3,vc5,avg", pairs=256, lo=16, hi=96,
             geom=3, ntl=1, fp="exact"),
        # the fill of the moved boxes of a regrid, fused multiply-adds
        dict(name="regrid_fill_fma", kind="boxes", form="batch", ops="vc5", pairs=32, lo=81, hi=161, geom=5, ntl=1,
             fp="fma"),
        # cell-centred and limited transport operators of a hydro evolution,
        # the boundary prolongation side
        dict(name="hydro_prolong", kind="boxes", form="batch", ops="cceno,cc5,mono,cc3", pairs=64, lo=16, hi=96,
             geom=7, ntl=1, fp="exact"),
        # ... and the restriction side: averaging and the higher orders
        dict(name="hydro_restrict", kind="boxes", form="batch", ops="avg,avg3,avg5", pairs=96, lo=16, hi=64,
             geom=9, ntl=1, fp="exact"),
        # a burst of requests from 20 small three-level hierarchies
        dict(name="served_burst", kind="served", nhier=20, lo=24, hi=64, ngf=4, requests=512, geom=11),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["plain", "plain", "batch", "batch", "hydro", "phase", "step", "served"])
    if what == "plain":
        op = rng.choice(["copy", "vc1", "vc3", "vc5", "vc5", "eno", "cc3", "cceno", "inject", "avg"])
        ext = [_log(rng, 3, 161) for _ in range(3)]
        return dict(kind="boxes", form="plain", ops=op, pairs=rng.randint(1, 6), ex=ext[0], ey=ext[1], ez=ext[2],
                    ntl=rng.choice([1, 3]) if op in ("copy", "vc1", "vc3", "vc5", "cc3") else 1,
                    fp=rng.choice(["exact", "exact", "fma"]))
    if what in ("batch", "hydro"):
        many = ["copy", "vc1", "vc3", "vc5", "eno", "cc1", "cc3", "cc5", "inject", "avg"] if what == "batch" else \
            ["cceno", "cc5", "mono", "avg", "avg3", "avg5"]
        lo = rng.randint(3, 40)
        return dict(kind="boxes", form="batch", ops=",".join(rng.sample(many, rng.randint(1, 4))),
                    pairs=_log(rng, 4, 256), lo=lo, hi=lo + rng.randint(1, 56), geom=rng.randint(0, 1 << 20),
                    ntl=rng.choice([1, 1, 3]) if what == "batch" else 1, fp=rng.choice(["exact", "exact", "fma"]))
    px, py, pz = rng.choice([(2, 1, 1), (1, 2, 1), (1, 1, 2), (2, 2, 1), (2, 2, 2)])
    shape = dict(px=px, py=py, pz=pz, ghost=3, order=5)
    if what == "phase":
        ph = rng.choice(["prolong", "prolong", "sync", "restrict"])
        return dict(kind="levels", form="phase", phase=ph, tl=rng.choice([1, 3]) if ph == "prolong" else 1,
                    nlevels=2, n=4 * rng.randint(14, 32) + 1, buffer=rng.choice([3, 6, 9]),
                    ngf=_log(rng, 1, 25), fp=rng.choice(["exact", "exact", "fma"]), **shape)
    if what == "step":
        return dict(kind="levels", form="step", nlevels=rng.randint(2, 4), n=4 * rng.randint(14, 32) + 1,
                    buffer=rng.choice([3, 6, 9]), ngf=_log(rng, 1, 12), fp="exact", **shape)
    return dict(kind="served", nhier=rng.randint(4, 20), lo=24, hi=rng.randint(32, 64), ngf=rng.randint(1, 4),
                requests=_log(rng, 32, 512), geom=rng.randint(0, 1 << 20))


# ---------------------------------------------------------------- box-pairs
class _Box:
    """one box-pair's geometry: source and destination extents, the region"""

    def __init__(self, op, ext, rng):
        self.op, self.ext = op, ext
        lo = [int(rng.integers(-20, 21)) for _ in range(3)]  # odd and even starts
        up = [lo[d] + ext[d] - 1 for d in range(3)]
        if op == "copy":
            # the ghost face of one component from another's interior
            self.reg = (*lo, *up, 1, 1, 1)
            self.src = (*[v - 3 for v in lo], *[v + 3 for v in up], 1, 1, 1)
            self.dst = (*[v - 2 for v in lo], *[v + 4 for v in up], 1, 1, 1)
        elif op in ("vc1", "vc3", "vc5", "eno", "mono"):
            w = {"vc1": 2, "vc3": 3, "vc5": 4, "eno": 3, "mono": 4}[op]
            self.reg = (*lo, *up, 1, 1, 1)
            self.src = (*[2 * (v // 2 - w) for v in lo], *[2 * (v // 2 + w) for v in up], 2, 2, 2)
            self.dst = (*[v - 2 for v in lo], *[v + 2 for v in up], 1, 1, 1)
        elif op in ("cc1", "cc3", "cc5", "cceno"):
            lo, up = [2 * v + 1 for v in lo], [2 * v + 1 for v in up]
            self.reg = (*lo, *up, 2, 2, 2)
            self.src = (*[4 * ((v - 2) // 4 - 4) + 2 for v in lo], *[4 * ((v - 2) // 4 + 5) + 2 for v in up], 4, 4, 4)
            self.dst = (*[v - 4 for v in lo], *[v + 4 for v in up], 2, 2, 2)
        elif op == "inject":
            lo, up = [2 * v for v in lo], [2 * v for v in up]
            self.reg = (*lo, *up, 2, 2, 2)
            self.src = (*[v - 2 for v in lo], *[v + 3 for v in up], 1, 1, 1)
            self.dst = (*[v - 4 for v in lo], *[v + 4 for v in up], 2, 2, 2)
        else:
            lo, up = [4 * v + 2 for v in lo], [4 * v + 2 for v in up]
            self.reg = (*lo, *up, 4, 4, 4)
            self.src = (*[v - 7 for v in lo], *[v + 7 for v in up], 2, 2, 2)
            self.dst = (*[v - 4 for v in lo], *[v + 4 for v in up], 4, 4, 4)

    @staticmethod
    def shape(b):
        n = [(b[3 + d] - b[d]) // b[6 + d] + 1 for d in range(3)]
        return n[2], n[1], n[0]

    @staticmethod
    def padded(b):
        nz, ny, nx = _Box.shape(b)
        return nz, ny, nx + (nx & 1)


def _boxes(case):
    ops = case["ops"].split(",")
    rng = np.random.default_rng(case.get("geom", 1))
    out = []
    for i in range(case["pairs"]):
        op = ops[i % len(ops)]
        if "lo" in case:
            ext = [int(v) for v in rng.integers(case["lo"], case["hi"] + 1, 3)]
        else:
            ext = [case["ex"], case["ey"], case["ez"]]
        if op in RESTRICT and "lo" in case:
            ext = [max(1, v // 2) for v in ext]  # coarse points under a fine box of that extent
        out.append(_Box(op, ext, rng))
    return out


def _ntl(case, op):
    return case["ntl"] if op in ("copy", "vc1", "vc3", "vc5", "cc1", "cc3", "cc5") else 1


def _offsets(shapes):
    """start of every array in a pool, 256 bytes apart at least"""
    offs, n = [], 0
    for z, y, x in shapes:
        offs.append(n)
        n += (z * y * x + 31) // 32 * 32
    return offs, n


def _bump(gen, shape, device):
    """a sum of four separable bumps over a (z, y, x) array, plus noise"""
    prm = torch.rand((3, 4, 2), generator=gen, dtype=torch.float64)
    ax = []
    for d, n in enumerate(shape):
        u = torch.arange(n, dtype=torch.float64) / 64.0
        c, w = prm[d, :, :1] * 1.5, 0.1 + 0.5 * prm[d, :, 1:]
        ax.append(torch.exp(-(((u[None] - c) / w) ** 2)))
    amp = 2.0 * torch.rand(4, generator=gen, dtype=torch.float64) - 1.0
    z, y, x = (a.to(device) for a in ax)
    return torch.einsum("kz,ky,kx->zyx", z * amp.to(device)[:, None], y, x)


def _fields(case, seed, device="cuda"):
    """the pools a boxes case works on: sources per timelevel, destination"""
    boxes = _boxes(case)
    gen = torch.Generator().manual_seed(int(seed))
    noise = torch.Generator(device=device).manual_seed(int(seed) + 1)
    so, sn = _offsets([_Box.padded(b.src) for b in boxes])
    do, dn = _offsets([_Box.padded(b.dst) for b in boxes])
    ntl = max(_ntl(case, b.op) for b in boxes)
    srcs = []
    for t in range(ntl):
        p = torch.randn(sn, generator=noise, dtype=torch.float64, device=device).mul_(1e-6)
        srcs.append(p)
    for b, o in zip(boxes, so):
        sh = _Box.padded(b.src)
        v = _bump(gen, sh, device)
        for t in range(_ntl(case, b.op)):
            srcs[t][o:o + v.numel()].view(sh).add_(v, alpha=1.0 - 0.125 * t)
    return boxes, so, do, srcs, torch.zeros(dn, dtype=torch.float64, device=device)


def _times(ntl):
    return ([0.0], 0.0, 0) if ntl == 1 else ([0.0, -DT, -2 * DT][:ntl], -DT / 2, ntl - 1)


def _prepare_boxes(case, seed):
    boxes, so, do, srcs, dst = _fields(case, seed)
    calls = []
    for b, s, d in zip(boxes, so, do):
        op, cent, order = OPS[b.op]
        ss, ds = _Box.padded(b.src), _Box.padded(b.dst)
        n, m = ss[0] * ss[1] * ss[2], ds[0] * ds[1] * ds[2]
        ntl = _ntl(case, b.op)
        times, time, order_time = _times(ntl)
        calls.append(dict(dst=cb.Data(b.dst, dst[d:d + m].view(ds)),
                          srcs=[cb.Data(b.src, srcs[t][s:s + n].view(ss)) for t in range(ntl)],
                          times=times, dstbox=b.reg, srcbox=b.reg if b.op == "copy" else b.src, time=time,
                          order_space=order, order_time=order_time, op=op, cent=cent, high=b.op))
    state = dict(form=case["form"], out=dst, srcs=srcs, calls=calls, fma=case["fp"] == "fma")
    cb.set_fp_mode(state["fma"])
    if case["form"] == "batch":
        batch = cb.Batch()
        for c in calls:
            high = c.pop("high")
            cb.set_restriction(high in ("avg3", "avg5"), int(high[-1]) if high in ("avg3", "avg5") else 1)
            batch.add(**c)
        cb.set_restriction(False)
        batch.upload()
        state["batch"] = batch
    else:
        for c in calls:
            c.pop("high")
    cb.set_fp_mode(False)
    return state


def _run_boxes(state):
    if state["form"] == "batch":
        state["batch"].launch()
    else:
        if state["fma"]:
            cb.set_fp_mode(True)
        for c in state["calls"]:
            cb.transfer_data(**c)
        if state["fma"]:
            cb.set_fp_mode(False)
    return state["out"]


def _box_work(b, ntl):
    """bytes (each input read once, each output written once) and operations
    of a separable evaluation that keeps the operator's order of sums"""
    m = [(b.reg[3 + d] - b.reg[d]) // b.reg[6 + d] + 1 for d in range(3)]
    npts = m[0] * m[1] * m[2]
    if b.op in ("copy", "inject"):
        return 8 * npts * (1 + ntl), npts * (2 * ntl - 1 if ntl > 1 else 0)
    if b.op in ("avg", "avg3", "avg5"):
        return 72 * npts, npts * {"avg": 16, "avg3": 128, "avg5": 77}[b.op]
    taps = {"vc1": 2, "vc3": 4, "vc5": 6, "eno": 4, "cc1": 2, "cc3": 4, "cc5": 6, "cceno": 4, "mono": 6}[b.op]
    cell = b.op.startswith("cc")
    coarse = [v // 2 + taps for v in m]
    odd = m if cell else [v // 2 for v in m]
    if b.op == "mono":  # one chain of 6, 36 or 216 terms for one, two or three odd axes: not separable
        even = [v - o for v, o in zip(m, odd)]
        ops = 11 * (odd[0] * even[1] * even[2] + even[0] * odd[1] * even[2] + even[0] * even[1] * odd[2]) \
            + 71 * (odd[0] * odd[1] * even[2] + odd[0] * even[1] * odd[2] + even[0] * odd[1] * odd[2]) \
            + 431 * odd[0] * odd[1] * odd[2]
        return 8 * npts + 8 * coarse[0] * coarse[1] * coarse[2], ops
    sums = odd[0] * coarse[1] * coarse[2] + m[0] * odd[1] * coarse[2] + m[0] * m[1] * odd[2]
    ops = ntl * sums * (2 * taps - 1) + (npts * (2 * ntl - 1) if ntl > 1 else 0)
    return 8 * npts + 8 * ntl * coarse[0] * coarse[1] * coarse[2], ops


# ---- the same in plain torch
def _lagrange(nodes, x):
    c = []
    for i, a in enumerate(nodes):
        v = 1.0
        for j, b in enumerate(nodes):
            if j != i:
                v *= (x - b) / (a - b)
        c.append(v)
    return c


def _matrix(op, b, d, device):
    """the linear 1-D operator along axis d: (region points, source points)"""
    n = (b.reg[3 + d] - b.reg[d]) // b.reg[6 + d] + 1
    ns = (b.src[3 + d] - b.src[d]) // b.src[6 + d] + 1
    a = np.zeros((n, ns))
    for i in range(n):
        x = b.reg[d] + i * b.reg[6 + d]
        p = (x - b.src[d]) / b.src[6 + d]  # position in source points
        if op in ("copy", "inject"):
            a[i, round(p)] = 1.0
            continue
        k = {"vc1": 2, "vc3": 4, "vc5": 6, "mono": 6, "cc1": 2, "cc3": 4, "cc5": 6, "avg": 2, "avg3": 4, "avg5": 6}[op]
        if op in ("vc1", "vc3", "vc5", "mono") and p == round(p):
            a[i, round(p)] = 1.0
            continue
        j0 = math.floor(p) - k // 2 + 1
        a[i, j0:j0 + k] = _lagrange([j - p for j in range(j0, j0 + k)], 0.0)
    return torch.from_numpy(a).to(device)


def _axes(v, fn):
    """fn on x, then y, then z (each as the last axis)"""
    for d in range(3):
        v = fn(v.movedim(2 - d, -1), d).movedim(-1, 2 - d)
    return v


def _coarse_index(b, d, device):
    """coarse base and parity of every region point along axis d"""
    n = (b.reg[3 + d] - b.reg[d]) // b.reg[6 + d] + 1
    half = b.reg[6 + d] // 2 if b.op == "cceno" else 0
    s = (b.reg[d] - b.src[d] + half) // b.reg[6 + d] + torch.arange(n, device=device)
    return s // 2, s % 2


def _eno(v, c, par):
    q1, q2, q3, q4 = (v[..., (c + k).clamp(0, v.shape[-1] - 1)] for k in (-1, 0, 1, 2))
    dl, dr = q1 + q3 - 2 * q2, q2 + q4 - 2 * q3
    r = torch.where(dl.abs() < dr.abs(), -q1 + 6 * q2 + 3 * q3, 3 * q2 + 6 * q3 - q4) / 8
    r = torch.where(((r - q2) * (q3 - r) < 0) | (dl * dr <= 0), (q2 + q3) / 2, r)
    return torch.where(par == 1, r, q2)


def _cceno(v, c, par):
    # f0 the cell itself, f1 the neighbour on the fine point's side
    side = 2 * par - 1
    f = {k: v[..., c + k * side] for k in (-2, -1, 0, 1, 2)}
    first = (f[1] + 3 * f[0]) / 4
    near, away = f[1] - 2 * f[0] + f[-1], f[2] - 2 * f[1] + f[0]
    # the two three-point stencils that hold the nearest two cells
    r = torch.where(away.abs() < near.abs(), (-3 * f[2] + 14 * f[1] + 21 * f[0]) / 32,
                    (5 * f[1] + 30 * f[0] - 3 * f[-1]) / 32)
    r = torch.where(away * near <= 0, first, r)
    return torch.where((r - f[0]) * (f[1] - r) < 0, first, r)


def _exact_box(b, srcs):
    dev = srcs[0].device
    if b.op == "eno" or b.op == "cceno":
        rule = _eno if b.op == "eno" else _cceno
        return _axes(srcs[0], lambda v, d: rule(v, *_coarse_index(b, d, dev)))
    lin = [_axes(s, lambda v, d: v @ _matrix(b.op, b, d, dev).T) for s in srcs]
    if len(lin) > 1:
        t, at, _ = _times(len(lin))
        return sum(w * v for w, v in zip(_lagrange(t, at), lin))
    if b.op != "mono":
        return lin[0]
    (cx, px), (cy, py), (cz, pz) = (_coarse_index(b, d, dev) for d in range(3))
    near = [srcs[0][cz + i * pz][:, cy + j * py][:, :, cx + k * px]
            for i in (0, 1) for j in (0, 1) for k in (0, 1)]
    near = torch.stack(near)
    out = (lin[0] > near.amax(0)) | (lin[0] < near.amin(0))
    return torch.where(out, near.mean(0), lin[0])


def exact(case, seed):
    if case["kind"] != "boxes":
        return None  # hierarchies: their region lists are the package's own
    boxes, so, do, srcs, dst = _fields(case, seed)
    for b, s, d in zip(boxes, so, do):
        ss, ds = _Box.padded(b.src), _Box.padded(b.dst)
        nz, ny, nx = _Box.shape(b.src)
        v = [srcs[t][s:s + ss[0] * ss[1] * ss[2]].view(ss)[:, :, :nx] for t in range(_ntl(case, b.op))]
        r = _exact_box(b, v)
        o = [(b.reg[k] - b.dst[k]) // b.dst[6 + k] for k in range(3)]
        m = r.shape
        dst[d:d + ds[0] * ds[1] * ds[2]].view(ds)[o[2]:o[2] + m[0], o[1]:o[1] + m[1], o[0]:o[0] + m[2]] = r
    return dst


# ---------------------------------------------------------------- hierarchies
def _parts(case):
    return case["px"], case["py"], case["pz"]


def _nested(case):
    parts = _parts(case)
    if case["form"] == "plain":  # one coarse component, the refined level split
        parts = [(1, 1, 1)] + [parts] * (case["nlevels"] - 1)
    return hierarchy.nested(case["nlevels"], case["n"], parts=parts, ghost=case["ghost"], buffer=case["buffer"],
                            order=case["order"])


def _fill(st, seed):
    gen = torch.Generator().manual_seed(int(seed))
    noise = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    for l, pools in enumerate(st.pools):
        for t, pool in enumerate(pools):
            torch.randn(pool.shape, generator=noise, dtype=torch.float64, device="cuda", out=pool)
            pool.mul_(1e-6)
            by_gf = pool.view(st.ngf, -1)
            amp = (1.0 + torch.rand(st.ngf, generator=gen, dtype=torch.float64)).cuda()
            for d in st.data[l][t][0]:
                o = (d.tensor.data_ptr() - pool.data_ptr()) // 8
                v = _bump(gen, tuple(d.tensor.shape), "cuda").reshape(-1)
                by_gf[:, o:o + v.numel()].addcmul_(amp[:, None], v[None])


def _phase_keys(case, keys):
    if case["form"] != "phase":
        return keys
    return [next(k for k in keys if k[0] == case["phase"] and k[3] == case["tl"]
                 and k[1] == (0 if case["phase"] == "restrict" else 1))]


def _prepare_levels(case, seed):
    h = _nested(case)
    st = Storage(h, case["ngf"], 3)
    _fill(st, seed)
    cb.set_fp_mode(case.get("fp") == "fma")
    form = case["form"]
    b = BergerOliger(h, st, order_space=case["order"], groups=2 if form == "step" and case["ngf"] > 1 else 1)
    keys = _phase_keys(case, b.step_phases())
    state = dict(form=form, st=st, bo=b, keys=keys, out=[p for pools in st.pools for p in pools])
    if form == "plain":
        state["calls"] = [c for k in keys for c in _plain_calls(b, k)]
    else:
        b.autotune([k for k in keys if k[0] == "prolong"], reps=2)
        if form == "step":
            state["stream"] = s = torch.cuda.Stream()
            s.wait_stream(torch.cuda.current_stream())
            b.run(keys, s)  # builds and uploads what the capture records
            s.synchronize()
            _fill(st, seed)
            state["graph"] = g = cb.Graph()
            with g.capture(s):
                b.run(keys, s)
            torch.cuda.synchronize()
        else:
            b.batch(keys[0])
            _fill(st, seed)  # the tuning launches wrote
    cb.set_fp_mode(False)
    return state


def _plain_calls(b, key):
    """the drop-in's calls of a phase, one per box-pair and grid function"""
    kind, l, rots, ntl = key
    pairs, ld, ls = bo.phase_pairs(b.h, key)
    dst = b.st.data[ld][bo.pool_index(rots[0], 0, 3)]
    rs = rots[-1]
    srcs = [b.st.data[ls][bo.pool_index(rs, t, 3)] for t in range(3 if kind == "prolong" else 1)]
    times, time = bo.prolong_times(ntl) if kind == "prolong" else ([0.0], 0.0)
    return [dict(dst=dst[g][p.dst_comp], srcs=[s[g][p.src_comp] for s in srcs], times=times, dstbox=p.dstbox,
                 srcbox=p.srcbox, time=time, order_space=b.order_space if kind != "sync" else 1,
                 order_time=2 if kind == "prolong" else 0)
            for g in range(b.st.ngf) for p in pairs]


def _run_levels(state):
    if state["form"] == "plain":
        for c in state["calls"]:
            cb.transfer_data(**c)
    elif state["form"] == "phase":
        state["bo"].batch(state["keys"][0]).launch()
    else:
        s = state["stream"]
        s.wait_stream(torch.cuda.current_stream())
        state["graph"].launch(s)
        torch.cuda.current_stream().wait_stream(s)
    return state["out"]


def _levels_work(case):
    h = _nested(case)
    keys = _phase_keys(case, bo.step_phases(case["nlevels"], 3, [0] * case["nlevels"]))
    nbytes, _ = bo.step_totals(h, keys, case["order"])
    ops = 0
    for k in keys:
        if k[0] == "prolong":
            pairs, _, ls = bo.phase_pairs(h, k)
            ops += sum(bo.fp64_ops("prolong", k[3], p.dstbox, h.levels[ls].comps[p.src_comp].exterior, case["order"])
                       for p in pairs)
    return dict(bytes=nbytes * case["ngf"], flops=ops * case["ngf"])


# ---------------------------------------------------------------- served
def _ensemble(case, server, seed):
    ens = serve.Ensemble(server, nhier=case["nhier"], size_range=(case["lo"], case["hi"]), ngf=case["ngf"],
                         seed=case["geom"], fill_seed=int(seed) % (1 << 30))
    keys, _ = serve.poisson_trace(ens, 1e5, case["requests"], seed=case["geom"] + 1)
    return ens, keys


def _prepare_served(case, seed):
    server = serve.Server(max_requests=1 << 23)  # the table keeps every request of a server's life
    server.set_config(1)
    ens, keys = _ensemble(case, server, seed)
    server.start()
    torch.cuda.synchronize()
    out = [p for m in ens.members for p in (lev[0] for lev in m.storage.pools)]
    return dict(server=server, ens=ens, ops=serve.ops_for(ens.ops, keys), at=[0.0] * len(keys), out=out)


def _run_served(state):
    state["server"].replay(state["ops"], state["at"])
    state["server"].drain()
    return state["out"]


def _served_work(case):
    rng = np.random.default_rng(case["geom"])
    hs = []
    for _ in range(case["nhier"]):
        n = [int(((int(rng.integers(case["lo"], case["hi"] + 1)) - 1 + 3) // 4) * 4 + 1) for _ in range(3)]
        hs.append(hierarchy.nested(3, n, parts=(2, 1, 1), ghost=3, buffer=3, order=5))

    class _E:  # the part of an ensemble that the trace reads
        members = [type("M", (), dict(hier=h, retired=False)) for h in hs]

    keys, _ = serve.poisson_trace(_E, 1e5, case["requests"], seed=case["geom"] + 1)
    nbytes = ops = 0
    for m, what, l in keys:
        k = {"sync": ("sync", l, (0,), 1), "prolong": ("prolong", l, (0, 0), 3), "restrict": ("restrict", l, (0, 0), 1)}
        pairs, _, ls = bo.phase_pairs(hs[m], k[what])
        for p in pairs:
            nbytes += bo.algorithmic_bytes(what, k[what][3], p.dstbox, hs[m].levels[ls].comps[p.src_comp].exterior)
            ops += bo.fp64_ops(what, k[what][3], p.dstbox, hs[m].levels[ls].comps[p.src_comp].exterior)
    return dict(bytes=nbytes * case["ngf"], flops=ops * case["ngf"])


# ---------------------------------------------------------------- the three calls
def prepare(case, seed):
    return {"boxes": _prepare_boxes, "levels": _prepare_levels, "served": _prepare_served}[case["kind"]](case, seed)


def run(state):
    if "server" in state:
        return _run_served(state)
    return _run_boxes(state) if "calls" in state and "keys" not in state else _run_levels(state)


def work(case):
    if case["kind"] == "boxes":
        w = [_box_work(b, _ntl(case, b.op)) for b in _boxes(case)]
        return dict(bytes=sum(x[0] for x in w), flops=sum(x[1] for x in w))
    return _levels_work(case) if case["kind"] == "levels" else _served_work(case)
