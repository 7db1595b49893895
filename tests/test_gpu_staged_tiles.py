"""Transfers through per-timelevel temporaries whose timelevels are tiled
differently.

With four or five timelevels every timelevel is prolongated into a temporary
of its own.  A plain call tiles a large one for tensor copies where its base
lies on 16 bytes and for plain loads where it does not, so one call can hold
both; each stage has to be launched with the tile count of its own form.  One
timelevel lies 8 bytes off, first, in the middle or last; the result is
compared bit for bit with the oracle, per box and batched.
"""
import numpy as np
import pytest

from oracle.binding import OP_LAGRANGE, VERTEX, Port

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _off(a, off):
    """a device copy of a whose base lies ``off`` doubles into its buffer"""
    buf = torch.empty(a.size + 2, dtype=torch.float64, device="cuda")
    v = buf[off:off + a.size].view(a.shape)
    v.copy_(torch.from_numpy(a))
    return v


@pytest.mark.parametrize("order_time,odd", [(3, 0), (3, 3), (4, 2), (4, 4)])
def test_one_unaligned_timelevel(order_time, odd):
    import carpet_b200 as cb
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, ntl = 129, order_time + 1  # 129^3 points: over the size from which single boxes are staged by tensor copies
    reg = (1, 0, 1, n, n - 1, n, 1, 1, 1)
    src = (-4, -4, -4, n + 5, n + 5, n + 5, 2, 2, 2)
    dst = (-1, 0, 1, n + 2, n - 1, n, 1, 1, 1)
    sshape = tuple((src[5 - d] - src[2 - d]) // 2 + 1 for d in range(3))
    dshape = tuple(dst[5 - d] - dst[2 - d] + 1 for d in range(3))
    rng = np.random.default_rng(17 * order_time + odd)
    srcs = [rng.standard_normal(sshape) for _ in range(ntl)]
    times = [1.0 - t / 8 for t in range(ntl)]
    time = 1.0 - 1.0 / 16
    want = np.full(dshape, np.nan)
    Port().transfer(OP_LAGRANGE, VERTEX, want, dst, srcs, src, times, reg, src, time, 1, order_time)
    pad = (0, (-sshape[2]) % 2)
    dev = [cb.Data(src, _off(np.pad(s, ((0, 0), (0, 0), pad)), int(t == odd))) for t, s in enumerate(srcs)]
    assert [d.tensor.data_ptr() % 16 for d in dev] == [8 * (t == odd) for t in range(ntl)]
    out = [cb.Data(dst, torch.full(dshape, np.nan, dtype=torch.float64, device="cuda")) for _ in range(2)]
    cb.transfer_data(out[0], dev, times, reg, src, time, 1, order_time)
    b = cb.Batch()
    b.add(out[1], dev, times, reg, src, time, 1, order_time)
    b.launch_per_box()
    b.check()
    torch.cuda.synchronize()
    for o in out:
        assert np.array_equal(o.tensor.cpu().numpy().view(np.uint64), want.view(np.uint64))
