"""Batched copies of several timelevels on both sides of the rule that sends
them point by point (few points) or by whole destination sectors (many): the
same regions, bit for bit against the oracle, with odd row pitches, rows that
start at every place in a sector, and both kinds of three-timelevel
interpolation."""
import numpy as np
import pytest

from oracle.binding import OP_ENO, OP_LAGRANGE, VERTEX, Port

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FEW = [((97, 5, 3), 0), ((18, 40, 9), 1), ((130, 7, 30), 2), ((33, 33, 33), 3)]
MANY = FEW + [((141, 140, 139), 1)]  # 2.7 million points more


@pytest.mark.parametrize("op", [OP_LAGRANGE, OP_ENO])
@pytest.mark.parametrize("shapes", [FEW, MANY], ids=["points", "sectors"])
@pytest.mark.parametrize("ntl", [2, 3])
def test_copies_of_several_timelevels(shapes, op, ntl):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200 as cb
    cb.set_fp_mode(False)
    rng = np.random.default_rng(len(shapes) + ntl)
    times, time = [1.0, 0.75, 0.5][:ntl], 0.9
    b, todo = cb.Batch(), []
    for n, margin in shapes:
        reg = (0, 0, 0, *[m - 1 for m in n], 1, 1, 1)
        db = (-margin, 0, 0, n[0] + 1, n[1], n[2], 1, 1, 1)
        sb = (-1, 0, -margin, n[0] + margin, n[1], n[2], 1, 1, 1)
        shape = lambda x: tuple(x[5 - d] - x[2 - d] + 1 for d in range(3))  # noqa: E731
        srcs = [rng.standard_normal(shape(sb)) for _ in range(ntl)]
        want = np.full(shape(db), np.nan)
        Port().transfer(op, VERTEX, want, db, srcs, sb, times, reg, reg, time, 3, ntl - 1)
        out = cb.Data(db, torch.full(shape(db), np.nan, dtype=torch.float64, device="cuda"))
        dev = [cb.Data(sb, torch.from_numpy(s).cuda()) for s in srcs]
        b.add(out, dev, times, reg, reg, time, 3, ntl - 1, op=op)
        todo.append((out, want, dev))
    b.upload()
    b.launch()
    b.check()
    for out, want, _ in todo:
        assert np.array_equal(out.tensor.cpu().numpy().view(np.uint64), want.view(np.uint64))
