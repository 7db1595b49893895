"""Lists of the no-allocation form whose prolongations are cut differently.

A list's prolongation tiles are cut in z by what the whole list takes: one
pair into the shortest chunks, many pairs into whole lengths, lists between by
the waves that their tiles run in.  Every list is compared bit for bit with the
same pairs as plain calls, copies and restrictions (tiled on their own) among
them.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# (region extent, kind): thin and long ones, one point, odd starts
PAIRS = [((64, 12, 52), "vc5"), ((5, 7, 3), "vc1"), ((33, 33, 33), "cc3"), ((17, 3, 70), "copy"), ((1, 1, 1), "vc5"),
         ((16, 16, 9), "inject"), ((40, 2, 129), "eno")]


def _pair_type():
    from carpet_b200._lib import cgx_array

    class cgx_pair(C.Structure):
        _fields_ = [("op", C.c_int), ("cent", C.c_int), ("dst", cgx_array), ("srcs", cgx_array * 3), ("times", C.c_double * 3),
                    ("nsrc", C.c_int), ("dstbox", C.c_int * 9), ("srcbox", C.c_int * 9), ("has_slab", C.c_int),
                    ("slab_offset", C.c_int * 3), ("time", C.c_double), ("order_space", C.c_int), ("order_time", C.c_int)]
    return cgx_pair


def _case(n, kind, i):
    lo = [i % 3, (i + 1) % 2, i % 2]
    up = [a + m - 1 for a, m in zip(lo, n)]
    if kind == "copy":
        reg = (*lo, *up, 1, 1, 1)
        return reg, (*[v - 3 for v in lo], *[v + 3 for v in up], 1, 1, 1), reg
    if kind == "inject":
        reg = (*[2 * v for v in lo], *[2 * v for v in up], 2, 2, 2)
        return reg, (*[2 * v - 2 for v in lo], *[2 * v + 3 for v in up], 1, 1, 1), reg
    if kind == "cc3":
        reg = (*[2 * v + 1 for v in lo], *[2 * v + 1 for v in up], 2, 2, 2)
        return reg, (*[4 * (v // 2 - 4) + 2 for v in lo], *[4 * (v // 2 + 5) + 2 for v in up], 4, 4, 4), reg
    reg = (*lo, *up, 1, 1, 1)
    return reg, (*[2 * (v // 2 - 4) for v in lo], *[2 * (v // 2 + 4) for v in up], 2, 2, 2), reg


@pytest.mark.parametrize("npairs,ntl", [(1, 1), (7, 3), (19, 1), (70, 3)])
def test_lists_agree_with_plain_calls(npairs, ntl):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200 as cb
    from carpet_b200._lib import lib
    cb.set_fp_mode(False)
    order = {"vc5": (cb.OP_LAGRANGE, cb.VERTEX, 5), "vc1": (cb.OP_LAGRANGE, cb.VERTEX, 1), "eno": (cb.OP_ENO, cb.VERTEX, 3),
             "cc3": (cb.OP_LAGRANGE, cb.CELL, 3), "copy": (cb.OP_LAGRANGE, cb.VERTEX, 1), "inject": (cb.OP_LAGRANGE, cb.VERTEX, 1)}
    gen = torch.Generator(device="cuda").manual_seed(npairs)
    times = [0.0, -0.125, -0.25]
    recs, plain, listed, keep = (_pair_type() * npairs)(), [], [], []
    for i in range(npairs):
        n, kind = PAIRS[i % len(PAIRS)]
        op, cent, o = order[kind]
        reg, sb, db = _case(n, kind, i)
        t = 1 if kind == "inject" else ntl
        srcs = [cb.Data(sb) for _ in range(t)]
        for s in srcs:
            s.tensor.normal_(generator=gen)
        box = reg if kind == "copy" else sb
        a, b = cb.Data(db), cb.Data(db)
        a.tensor.fill_(float("nan"))
        b.tensor.fill_(float("nan"))
        at, ot = (0.0, 0) if t == 1 else (-0.0625, t - 1)
        cb.transfer_data(a, srcs, times[:t], reg, box, at, o, ot, op=op, cent=cent)
        r = recs[i]
        r.op, r.cent, r.dst, r.nsrc, r.time, r.order_space, r.order_time = op, cent, b.cgx(), t, at, o, ot
        for k, s in enumerate(srcs):
            r.srcs[k], r.times[k] = s.cgx(), times[k]
        r.dstbox[:], r.srcbox[:] = reg, box
        plain.append(a)
        listed.append(b)
        keep += srcs
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.cgx_transfer_pairs_noalloc(recs, npairs, s) == 0, lib.cgx_last_error()
    assert lib.cgx_noalloc_check(s) == 0
    for i, (a, b) in enumerate(zip(plain, listed)):
        x, y = a.tensor.cpu().numpy().view(np.uint64), b.tensor.cpu().numpy().view(np.uint64)
        assert np.array_equal(x, y), (i, PAIRS[i % len(PAIRS)])
