"""The packed record of a plain call: its layout is cgx_pair's, and calls that
cannot be packed take the general path (checked without a device)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def T():
    try:
        from carpet_b200 import transfer
    except ImportError as e:
        pytest.skip(str(e))
    return transfer


def _pair_struct():
    from carpet_b200._lib import cgx_array

    class cgx_pair(C.Structure):
        _fields_ = [("op", C.c_int), ("cent", C.c_int), ("dst", cgx_array), ("srcs", cgx_array * 3),
                    ("times", C.c_double * 3), ("nsrc", C.c_int), ("dstbox", C.c_int * 9), ("srcbox", C.c_int * 9),
                    ("has_slab", C.c_int), ("slab_offset", C.c_int * 3), ("time", C.c_double),
                    ("order_space", C.c_int), ("order_time", C.c_int)]
    return cgx_pair


@pytest.mark.parametrize("nsrc", [1, 2, 3])
@pytest.mark.parametrize("slab", [None, (1, -2, 3)])
def test_record_layout(T, monkeypatch, nsrc, slab):
    cgx_pair = _pair_struct()
    assert T._PAIR.size == C.sizeof(cgx_pair)
    seen = []
    monkeypatch.setattr(T, "lib", type("L", (), dict(
        cgx_transfer_pair=staticmethod(lambda rec, s: seen.append((cgx_pair.from_buffer_copy(rec), s)) or 0)))())
    dst = T.Data((0, 0, 0, 6, 4, 3, 1, 1, 1), device="cpu")
    srcs = [T.Data((-2, -2, -2, 8 + 2 * t, 8, 8, 2, 2, 2), device="cpu") for t in range(nsrc)]
    box, sbox = np.array((1, 0, 1, 5, 3, 2, 1, 1, 1)), (-2, -2, -2, 8, 8, 8, 2, 2, 2)
    T.transfer_data(dst, srcs, [1.0, 0.5, 0.25], box, sbox, 0.75, 5, 2, slab_offset=slab, stream=77)
    (p, s), = seen
    assert s == 77 and (p.op, p.cent, p.nsrc) == (T.OP_LAGRANGE, T.VERTEX, nsrc)
    for a, d in zip([p.dst, *p.srcs[:nsrc]], [dst, *srcs]):
        assert (a.data, tuple(a.padext), list(a.bbox)) == (d.tensor.data_ptr(), d.padext, d.extent)
    assert list(p.times)[:nsrc] == [1.0, 0.5, 0.25][:nsrc]
    assert tuple(p.dstbox) == tuple(box) and tuple(p.srcbox) == sbox
    assert (p.time, p.order_space, p.order_time) == (0.75, 5, 2)
    assert (p.has_slab, tuple(p.slab_offset)) == ((0, (0, 0, 0)) if slab is None else (1, slab))


def test_unpackable_calls_take_the_general_path(T, monkeypatch):
    general = []
    monkeypatch.setattr(T, "lib", type("L", (), dict(
        cgx_transfer=staticmethod(lambda *a: general.append(a) or 0),
        cgx_transfer_pair=staticmethod(lambda *a: pytest.fail("packed"))))())
    d = T.Data((0, 0, 0, 6, 4, 3, 1, 1, 1), device="cpu")
    box = (0, 0, 0, 6, 4, 3, 1, 1, 1)
    T.transfer_data(d, [d] * 4, [0.0, -1.0, -2.0, -3.0], box, box, -0.5, 1, 3, stream=1)  # four timelevels
    T.transfer_data(d, [d], [0.0], tuple(float(v) for v in box), box, 0.0, 1, 0, stream=1)  # floats for indices
    assert [a[5] for a in general] == [4, 1]
