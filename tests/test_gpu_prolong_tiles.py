"""Prolongation tiles at the edges of their shapes, batched and per box.

The tile shape of a prolongation follows the region (widths balanced over it,
even source positions in y and z), the destination's alignment (tiles that
start at 32-byte sectors, or two points further in every other row) and the
number of tiles of the launch.  Every operator family is compared bit for bit
with the oracle over regions around those shapes: one tile and one point more,
full 16-point tiles that start at odd and even source positions, destination
rows of every pitch modulo a sector, and regions thinner than a stencil.
"""
import numpy as np
import pytest

from oracle.binding import CELL, OP_ENO, OP_LAGRANGE, VERTEX, Port

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FAMILIES = [("vc", OP_LAGRANGE, VERTEX, 1), ("vc", OP_LAGRANGE, VERTEX, 3), ("vc", OP_LAGRANGE, VERTEX, 5),
            ("vc", OP_ENO, VERTEX, 3)] + [("cc", OP_LAGRANGE, CELL, o) for o in range(6)] + [
            ("cc", OP_ENO, CELL, 3), ("cc", OP_ENO, CELL, 5)]
# region extents; offsets (odd and even starts); destination margins, which
# set the row and plane pitches and the first point's place in a sector
SHAPES = [((16, 16, 6), (0, 0, 0), (0, 0, 0)), ((17, 15, 9), (1, 1, 1), (3, 1, 0)),
          ((32, 5, 7), (2, 1, 0), (0, 3, 1)), ((33, 2, 66), (3, 0, 1), (2, 0, 2)),
          ((48, 33, 3), (2, 1, 1), (2, 2, 0)), ((64, 12, 13), (0, 0, 1), (4, 0, 0)),
          ((47, 9, 10), (3, 1, 0), (1, 2, 1)), ((1, 40, 1), (1, 0, 1), (1, 1, 1))]


@pytest.fixture(scope="module")
def cb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200
    return carpet_b200


def _case(kind, n, off, margin, rng):
    """(region, source bbox, destination bbox): strides 2/1 (vertex) or 4/2"""
    if kind == "vc":
        lo = [8 + o for o in off]
        reg = (*lo, *[a + m - 1 for a, m in zip(lo, n)], 1, 1, 1)
        src = (*[2 * (a // 2 - 4) for a in lo], *[2 * (b // 2 + 4) for b in reg[3:6]], 2, 2, 2)
        dst = (*[a - m for a, m in zip(lo, margin)], *[b + m for b, m in zip(reg[3:6], margin)], 1, 1, 1)
    else:
        lo = [2 * (8 + o) + 1 for o in off]
        reg = (*lo, *[a + 2 * (m - 1) for a, m in zip(lo, n)], 2, 2, 2)
        src = (*[4 * ((a - 2) // 4 - 5) + 2 for a in lo], *[4 * ((b - 2) // 4 + 6) + 2 for b in reg[3:6]], 4, 4, 4)
        dst = (*[a - 2 * m for a, m in zip(lo, margin)], *[b + 2 * m for b, m in zip(reg[3:6], margin)], 2, 2, 2)
    return reg, src, dst


def _shape(b):
    return tuple((b[5 - d] - b[2 - d]) // b[8 - d] + 1 for d in range(3))


def _pad(a, even):
    """x padded to an even length (16-byte rows) or left as it is"""
    if not even or a.shape[2] % 2 == 0:
        return a
    out = np.full(a.shape[:2] + (a.shape[2] + 1,), np.nan)
    out[:, :, :a.shape[2]] = a
    return out


@pytest.mark.parametrize("fma", [False, True])
@pytest.mark.parametrize("kind,op,cent,order", FAMILIES)
def test_tile_edges(cb, kind, op, cent, order, fma):
    port = Port()
    rng = np.random.default_rng(100 * order + 7 * op + cent)
    times3 = [1.0, 0.75, 0.5]
    for ntl, even in ((1, True), (3, True), (2, True), (1, False)):
        time, ot = (1.0, 0) if ntl == 1 else (0.875, ntl - 1)
        todo = []
        for n, off, margin in SHAPES:
            reg, sb, db = _case(kind, n, off, margin, rng)
            srcs = [rng.standard_normal(_shape(sb)) for _ in range(3)]
            want = np.full(_shape(db), np.nan)
            port.transfer(op, cent, want, db, srcs, sb, times3, reg, sb, time, order, ot, fma=fma)
            dev = [cb.Data(sb, torch.from_numpy(_pad(s, even).copy()).cuda()) for s in srcs]
            out = [cb.Data(db, torch.from_numpy(_pad(np.full(_shape(db), np.nan), even).copy()).cuda())
                   for _ in range(2)]
            todo.append((reg, sb, dev, out, want))
        cb.set_fp_mode(fma)
        try:
            b = cb.Batch()
            for reg, sb, dev, out, _ in todo:
                b.add(out[0], dev, times3, reg, sb, time, order, ot, op=op, cent=cent)
                cb.transfer_data(out[1], dev, times3, reg, sb, time, order, ot, op=op, cent=cent)
            for cfg in range(5):
                b.set_config(cfg)
                b.upload()
                b.launch()
                b.check()
                torch.cuda.synchronize()
                for reg, sb, dev, out, want in todo:
                    for o in (out if cfg == 0 else out[:1]):
                        got = o.tensor.cpu().numpy()[:, :, :want.shape[2]]
                        assert np.array_equal(got.view(np.uint64), want.view(np.uint64)), (reg, ntl, even, cfg)
                    out[0].tensor.fill_(float("nan"))
        finally:
            cb.set_fp_mode(False)
