"""The C entry cgx_copy (gdata::copy_data) against the Python call of the same
name, which goes through the general entry: both centrings, every stride
relation, a slab offset."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# centring, region, source box, slab offset
CASES = [("VERTEX", (1, 0, 1, 20, 9, 6, 1, 1, 1), (-2, -2, -2, 24, 13, 9, 1, 1, 1), None),
         ("VERTEX", (1, 0, 1, 20, 9, 6, 1, 1, 1), (-2, -2, -2, 24, 13, 9, 1, 1, 1), (2, -1, 1)),
         ("VERTEX", (1, 0, 1, 20, 9, 6, 1, 1, 1), (-4, -4, -4, 26, 14, 12, 2, 2, 2), None),
         ("VERTEX", (0, 0, 0, 16, 8, 6, 2, 2, 2), (-2, -2, -2, 19, 11, 9, 1, 1, 1), None),
         ("CELL", (1, 3, 1, 41, 21, 19, 2, 2, 2), (-18, -18, -18, 62, 42, 42, 4, 4, 4), None),
         ("CELL", (2, 2, 2, 34, 22, 18, 4, 4, 4), (-5, -5, -5, 43, 31, 27, 2, 2, 2), None)]


@pytest.mark.parametrize("cent,reg,src,slab", CASES)
def test_c_entry_equals_python_call(cent, reg, src, slab):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200 as cb
    from carpet_b200._lib import box9, ints3, lib
    cent = getattr(cb, cent)
    s = cb.Data(src)
    s.tensor.normal_(generator=torch.Generator(device="cuda").manual_seed(3))
    out = [cb.Data(reg), cb.Data(reg)]
    for o in out:
        o.tensor.fill_(float("nan"))
    cb.copy_data(out[0], s, reg, src, cent=cent, slab_offset=slab)
    d, a = out[1].cgx(), s.cgx()
    rc = lib.cgx_copy(cb.OP_LAGRANGE, cent, C.byref(d), C.byref(a), box9(reg), box9(src), ints3(slab),
                      C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, lib.cgx_last_error()
    torch.cuda.synchronize()
    x, y = (o.tensor.cpu().numpy() for o in out)
    assert np.isfinite(x[..., :(reg[3] - reg[0]) // reg[6] + 1]).all()
    assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
