"""Copies, restrictions and monotone prolongations at the edges of their tiles.

Copies go point by point or, for rows of 16 values and more, by whole 32-byte
sectors of the destination (a batch chooses by its share of narrow boxes, and
fetches its destinations ahead when it copies more than L2 keeps); the
higher-order restrictions march tiles of rows; the monotone prolongation walks
rows by parity; one large prolongation alone is staged by TMA.  Each is
compared bit for bit with the oracle over whole destination arrays, in a batch
and by a call of its own.
"""
import numpy as np
import pytest

from oracle.binding import CELL, OP_ENO, OP_LAGRANGE, OP_LAGRANGE_MONOTONE, VERTEX, Port

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# region extents; margins of the destination and of the source below and above
# (they set the pitches and the first value's place in a sector)
COPIES = [((15, 3, 2), (0, 1), (1, 0)), ((16, 4, 3), (0, 0), (0, 0)), ((17, 3, 5), (1, 0), (2, 1)),
          ((18, 2, 3), (2, 1), (3, 2)), ((19, 5, 1), (3, 2), (0, 1)), ((33, 8, 9), (1, 1), (1, 2)),
          ((35, 1, 17), (2, 3), (2, 0)), ((130, 7, 3), (3, 3), (1, 1)), ((64, 16, 8), (4, 0), (0, 4))]
NARROW = [((3, 40, 21), (0, 1), (1, 0)), ((1, 33, 9), (2, 2), (0, 3))]
RESTRICT = [((16, 8, 4), 0), ((17, 9, 5), 1), ((15, 7, 3), 2), ((33, 8, 17), 1), ((1, 1, 1), 0),
            ((31, 16, 16), 3), ((2, 17, 33), 2), ((64, 49, 22), 0), ((65, 48, 23), 1)]
MONO = [((8, 6, 5), (0, 0, 0)), ((9, 7, 6), (1, 1, 1)), ((33, 2, 3), (1, 0, 1)), ((1, 1, 1), (1, 1, 1)),
        ((2, 31, 1), (0, 1, 0)), ((67, 9, 10), (0, 1, 1)), ((64, 33, 4), (1, 0, 0))]


@pytest.fixture(scope="module")
def cb():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200
    return carpet_b200


def _shape(b):
    return tuple((b[5 - d] - b[2 - d]) // b[8 - d] + 1 for d in range(3))


def _dev(cb, a, bbox):
    return cb.Data(bbox, torch.from_numpy(a.copy()).cuda())


def _check(cb, todo, times, time, order, ot, op, cent, fma):
    """todo: (region, source bbox, destination bbox); one batch of all pairs
    and a call for each pair, bit for bit against the oracle"""
    port = Port()
    rng = np.random.default_rng(len(todo) + 10 * order + ot)
    port.set_restriction(*_check.restriction)
    cb.set_restriction(*_check.restriction)
    cb.set_fp_mode(fma)
    try:
        b, res = cb.Batch(), []
        for reg, sb, db in todo:
            srcs = [rng.standard_normal(_shape(sb)) for _ in times]
            want = np.full(_shape(db), np.nan)
            port.transfer(op, cent, want, db, srcs, sb, times, reg, sb, time, order, ot, fma=fma)
            dev = [_dev(cb, s, sb) for s in srcs]
            out = [_dev(cb, np.full(_shape(db), np.nan), db) for _ in range(2)]
            b.add(out[0], dev, times, reg, sb, time, order, ot, op=op, cent=cent)
            cb.transfer_data(out[1], dev, times, reg, sb, time, order, ot, op=op, cent=cent)
            res.append((reg, out, want, dev))
        b.upload()
        b.launch()
        b.check()
        torch.cuda.synchronize()
        for reg, out, want, _ in res:
            for o in out:
                assert np.array_equal(o.tensor.cpu().numpy().view(np.uint64), want.view(np.uint64)), reg
    finally:
        cb.set_fp_mode(False)
        cb.set_restriction(False, 1)
        port.set_restriction(False, 1)


_check.restriction = (False, 1)


def _copy(n, dm, sm):
    lo = (5, 6, 7)
    up = [a + m - 1 for a, m in zip(lo, n)]
    def box(m):
        return (*[a - m[0] for a in lo], *[b + m[1] for b in up], 1, 1, 1)
    return (*lo, *up, 1, 1, 1), box(sm), box(dm)


@pytest.mark.parametrize("fma", [False, True])
@pytest.mark.parametrize("op,ntl", [(OP_LAGRANGE, 1), (OP_LAGRANGE, 2), (OP_LAGRANGE, 3), (OP_ENO, 3)])
def test_copies(cb, op, ntl, fma):
    times, ot = [1.0, 0.75, 0.5], max(ntl - 1, 0)
    time = 1.0 if ntl == 1 else 0.875
    wide = [_copy(*c) for c in COPIES]
    for todo in (wide, wide + [_copy(*c) for c in NARROW] * 12, wide[:1], wide[2:3]):
        _check(cb, todo, times, time, 1, ot, op, VERTEX, fma)


def test_large_copies(cb):
    todo = [_copy((150, 149, 141), (1, 0), (0, 2)), _copy((17, 129, 40), (3, 1), (1, 1)), _copy((64, 8, 8), (0, 0), (0, 0))]
    assert 16 * sum(np.prod(_shape(t[0])) for t in todo) >= 48 << 20
    _check(cb, todo, [0.0], 0.0, 1, 0, OP_LAGRANGE, VERTEX, False)


@pytest.mark.parametrize("fma", [False, True])
@pytest.mark.parametrize("order", [3, 5])
def test_restriction_tiles(cb, order, fma, monkeypatch):
    monkeypatch.setattr(_check, "restriction", (True, order))
    reach, todo = 1 if order == 3 else 2, []
    for n, m in RESTRICT:
        lo = [4 * a + 2 for a in (3, 4, 5)]
        up = [a + 4 * (k - 1) for a, k in zip(lo, n)]
        todo.append(((*lo, *up, 4, 4, 4),
                     (*[a - 1 - 2 * (reach + m) for a in lo], *[b + 1 + 2 * (reach + m // 2) for b in up], 2, 2, 2),
                     (*[a - 4 * m for a in lo], *[b + 4 * (m // 2) for b in up], 4, 4, 4)))
    _check(cb, todo, [0.0], 0.0, 1, 0, OP_LAGRANGE, CELL, fma)


def _prolong(n, off, margin=0):
    lo = [8 + o for o in off]
    up = [a + m - 1 for a, m in zip(lo, n)]
    return ((*lo, *up, 1, 1, 1), (*[2 * (a // 2 - 4) for a in lo], *[2 * (b // 2 + 4) for b in up], 2, 2, 2),
            (*[a - margin for a in lo], *[b + margin for b in up], 1, 1, 1))


@pytest.mark.parametrize("fma", [False, True])
@pytest.mark.parametrize("ntl", [1, 3])
def test_monotone_rows(cb, ntl, fma):
    times, time = [1.0, 0.75, 0.5], 1.0 if ntl == 1 else 0.875
    todo = [_prolong(n, off, m) for m, (n, off) in enumerate(MONO)]
    _check(cb, todo, times, time, 5, ntl - 1, OP_LAGRANGE_MONOTONE, VERTEX, fma)


@pytest.mark.parametrize("op,cent,order,ntl,n", [
    (OP_LAGRANGE, VERTEX, 5, 3, (99, 87, 85)), (OP_LAGRANGE, VERTEX, 3, 1, (131, 130, 127)),
    (OP_LAGRANGE, CELL, 4, 1, (130, 129, 128)), (OP_ENO, CELL, 3, 1, (129, 128, 131))])
def test_one_large_box(cb, op, cent, order, ntl, n):
    assert ntl * np.prod(n) >= 8 << 18
    times, time = [1.0, 0.75, 0.5], 1.0 if ntl == 1 else 0.875
    if cent == VERTEX:
        todo = [_prolong(n, (1, 0, 1), 1)]
    else:
        lo = [2 * (8 + o) + 1 for o in (1, 0, 1)]
        up = [a + 2 * (m - 1) for a, m in zip(lo, n)]
        todo = [((*lo, *up, 2, 2, 2),
                 (*[4 * ((a - 2) // 4 - 5) + 2 for a in lo], *[4 * ((b - 2) // 4 + 6) + 2 for b in up], 4, 4, 4),
                 (*[a - 2 for a in lo], *[b + 2 for b in up], 2, 2, 2))]
    # an even source pitch is what the TMA boxes take; both are compared
    reg, sb, db = todo[0]
    _check(cb, [(reg, sb, db), (reg, (*sb[:3], sb[3] + sb[6], *sb[4:]), db)], times, time, order, ntl - 1,
           op, cent, False)
