"""A served launch of more kinds of kernel than a server slot has side streams:
its segments share the streams, one after another on each.  One operation of
every prolongation family with one to three timelevels, copies, injection and
averaging is served several times and compared bit for bit with plain calls of
its pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIDE_STREAMS = 24


def _pairs(cb):
    """(op, centring, order, timelevels, region, source box)"""
    reg, src = (1, 0, 1, 20, 12, 9, 1, 1, 1), (-8, -8, -8, 30, 22, 18, 2, 2, 2)
    creg, csrc = (1, 3, 1, 41, 21, 19, 2, 2, 2), (-18, -18, -18, 62, 42, 42, 4, 4, 4)
    out = []
    for ntl in (1, 2, 3):
        out += [(cb.OP_LAGRANGE, cb.VERTEX, o, ntl, reg, src) for o in (1, 3, 5)]
        out += [(cb.OP_ENO, cb.VERTEX, 3, ntl, reg, src)]
        out += [(cb.OP_LAGRANGE, cb.CELL, o, ntl, creg, csrc) for o in range(6)]
        out += [(cb.OP_ENO, cb.CELL, o, ntl, creg, csrc) for o in (3, 5)]
        out += [(cb.OP_LAGRANGE, cb.VERTEX, 1, ntl, reg, (*[v - 2 for v in reg[:3]], *[v + 2 for v in reg[3:6]], 1, 1, 1))]
    out += [(cb.OP_LAGRANGE, cb.VERTEX, 1, 1, (0, 0, 0, 16, 8, 6, 2, 2, 2), (-2, -2, -2, 19, 11, 9, 1, 1, 1)),
            (cb.OP_LAGRANGE, cb.CELL, 1, 1, (2, 2, 2, 34, 22, 18, 4, 4, 4), (-5, -5, -5, 43, 31, 27, 2, 2, 2))]
    return out


def test_more_segments_than_side_streams():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200 as cb
    from carpet_b200.serve import SERVE_BATCHED, Server
    cb.set_fp_mode(False)
    gen = torch.Generator(device="cuda").manual_seed(5)
    b, todo, times = cb.Batch(), [], [0.0, -0.125, -0.25]
    for op, cent, order, ntl, reg, src in _pairs(cb):
        srcs = [cb.Data(src) for _ in range(ntl)]
        for s in srcs:
            s.tensor.normal_(generator=gen)
        want, got = cb.Data(reg), cb.Data(reg)
        want.tensor.fill_(float("nan"))
        got.tensor.fill_(float("nan"))
        box = reg if src[6] == reg[6] else src
        at, ot = (0.0, 0) if ntl == 1 else (-0.0625, ntl - 1)
        cb.transfer_data(want, srcs, times[:ntl], reg, box, at, order, ot, op=op, cent=cent)
        b.add(got, srcs, times[:ntl], reg, box, at, order, ot, op=op, cent=cent)
        todo.append((want, got, srcs))
    b.upload()
    assert b.kernels() > SIDE_STREAMS + 1
    torch.cuda.synchronize()
    sv = Server(mode=SERVE_BATCHED)
    sv.set_config(1)
    op_id = sv.define(0, b)
    for _ in range(5):
        sv.submit(op_id)
    sv.drain()
    assert sv.report()["requests"] == 5
    sv.close()
    for i, (want, got, _) in enumerate(todo):
        x, y = (t.tensor.cpu().numpy().view(np.uint64) for t in (want, got))
        assert np.array_equal(x, y), _pairs(cb)[i]
