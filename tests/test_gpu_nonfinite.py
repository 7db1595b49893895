"""Sources that hold infinities, NaN, signed zeros, subnormals and values near
the overflow: every operator family against the oracle, per box and batched,
in both floating-point modes.  A sum that the tile forms for a point that is
not stored, or from a value that the point's stencil does not hold, must not
reach a stored value.  Values agree bit for bit, NaN as such (their sign and
payload are the processor's)."""
import numpy as np
import pytest

from oracle.binding import CELL, OP_ENO, OP_LAGRANGE, OP_LAGRANGE_MONOTONE, VERTEX, Port

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FAMILIES = [("vc", OP_LAGRANGE, VERTEX, o) for o in (1, 3, 5, 7, 9, 11)] + [("vc", OP_ENO, VERTEX, 3)] + \
    [("cc", OP_LAGRANGE, CELL, o) for o in range(6)] + [("cc", OP_ENO, CELL, 3), ("cc", OP_ENO, CELL, 5),
    ("vc", OP_LAGRANGE_MONOTONE, VERTEX, 5), ("copy", OP_LAGRANGE, VERTEX, 1), ("copy", OP_ENO, VERTEX, 3),
    ("inject", OP_LAGRANGE, VERTEX, 1), ("avg", OP_LAGRANGE, CELL, 1), ("avg", OP_LAGRANGE, CELL, 3),
    ("avg", OP_LAGRANGE, CELL, 5)]
SHAPES = [((17, 15, 9), (1, 1, 1)), ((33, 6, 11), (0, 1, 0)), ((3, 20, 5), (1, 0, 1))]
SPECIAL = [np.inf, -np.inf, np.nan, 0.0, -0.0, 5e-324, -1e-310, 1.6e308, -1.7e308]


def _boxes(kind, n, off):
    if kind == "vc":
        lo = [16 + o for o in off]
        up = [a + m - 1 for a, m in zip(lo, n)]
        return (*lo, *up, 1, 1, 1), (*[2 * (a // 2 - 6) for a in lo], *[2 * (b // 2 + 7) for b in up], 2, 2, 2)
    if kind == "cc":
        lo = [2 * (8 + o) + 1 for o in off]
        up = [a + 2 * (m - 1) for a, m in zip(lo, n)]
        return (*lo, *up, 2, 2, 2), (*[4 * ((a - 2) // 4 - 5) + 2 for a in lo], *[4 * ((b - 2) // 4 + 6) + 2 for b in up], 4, 4, 4)
    if kind == "copy":
        return (*off, *[o + m - 1 for o, m in zip(off, n)], 1, 1, 1), (-2, -2, -2, *[m + 2 for m in n], 1, 1, 1)
    if kind == "inject":
        lo, up = [2 * o for o in off], [2 * (o + m - 1) for o, m in zip(off, n)]
        return (*lo, *up, 2, 2, 2), (-2, -2, -2, *[v + 3 for v in up], 1, 1, 1)
    lo, up = [4 * o + 2 for o in off], [4 * (o + m - 1) + 2 for o, m in zip(off, n)]
    return (*lo, *up, 4, 4, 4), (*[v - 7 for v in lo], *[v + 7 for v in up], 2, 2, 2)


def _shape(b):
    return tuple((b[5 - d] - b[2 - d]) // b[8 - d] + 1 for d in range(3))


def _same(got, want):
    nan = np.isnan(want)
    return np.array_equal(nan, np.isnan(got)) and \
        np.array_equal(got[~nan].view(np.uint64), want[~nan].view(np.uint64))


@pytest.mark.parametrize("fma", [False, True], ids=["exact", "fma"])
@pytest.mark.parametrize("kind,op,cent,order", FAMILIES)
def test_nonfinite_sources(kind, op, cent, order, fma):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200 as cb
    port = Port()
    rng = np.random.default_rng(31 * order + 7 * op + cent)
    high = kind == "avg" and order > 1
    many = kind in ("vc", "cc", "copy") and op != OP_LAGRANGE_MONOTONE and order < 7
    for setter in (port.set_restriction, cb.set_restriction):
        setter(high, order if high else 1)
    cb.set_fp_mode(fma)
    try:
        for ntl in (1, 3) if many else (1,):
            times, time = [1.0, 0.75, 0.5][:ntl], 1.0 if ntl == 1 else 0.875
            b, todo = cb.Batch(), []
            for n, off in SHAPES:
                for share in (0.003, 0.05):
                    reg, sb = _boxes(kind, n, off)
                    shape = _shape(sb)
                    srcs = []
                    for _ in range(ntl):
                        s = rng.standard_normal(shape)
                        at = rng.random(shape) < share
                        s[at] = rng.choice(SPECIAL, int(at.sum()))
                        srcs.append(s)
                    want = np.zeros(_shape(reg))
                    sbox = reg if kind == "copy" else sb
                    port.transfer(op, cent, want, reg, srcs, sb, times, reg, sbox, time, order, ntl - 1, fma=fma)
                    pad = ((0, 0), (0, 0), (0, shape[2] & 1))
                    dev = [cb.Data(sb, torch.from_numpy(np.pad(s, pad)).cuda()) for s in srcs]
                    out = [cb.Data(reg, torch.zeros(want.shape, dtype=torch.float64, device="cuda")) for _ in range(2)]
                    cb.transfer_data(out[0], dev, times, reg, sbox, time, order, ntl - 1, op=op, cent=cent)
                    b.add(out[1], dev, times, reg, sbox, time, order, ntl - 1, op=op, cent=cent)
                    todo.append((reg, share, out, want, dev))
            b.upload()
            b.launch()
            b.check()
            torch.cuda.synchronize()
            assert any(np.isnan(want).any() for _, _, _, want, _ in todo)
            for reg, share, out, want, _ in todo:
                for i, o in enumerate(out):
                    assert _same(o.tensor.cpu().numpy(), want), (reg, share, ntl, i)
    finally:
        cb.set_fp_mode(False)
        for setter in (port.set_restriction, cb.set_restriction):
            setter(False, 1)
