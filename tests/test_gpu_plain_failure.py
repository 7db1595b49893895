"""Failure detection of plain calls, without a GPU fault.

A large plain prolongation is staged by tensor copies and waits for them, for
about a second at most.  The library's failure-injection hook leaves one stage
out, so that the wait runs out: the plain-call check has to report it once, and
the next call has to be right.  A plain call may also be the first use of the
device by the library, inside a stream capture.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle.binding import CELL, OP_ENO, OP_LAGRANGE, VERTEX, Port

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EDEVICE = 5
N = 129  # 129^3 points: over the size from which single boxes are staged by tensor copies


def _call(op, cent, order):
    """source, destination, region and expected values of one large box"""
    if cent == VERTEX:
        reg, src, dst = (0, 0, 0, N - 1, N - 1, N - 1, 1, 1, 1), (-6, -6, -6, N + 7, N + 7, N + 7, 2, 2, 2), \
            (-1, -1, -1, N, N, N, 1, 1, 1)
    else:
        reg, src, dst = (1, 1, 1, 2 * N - 1, 2 * N - 1, 2 * N - 1, 2, 2, 2), \
            (-14, -14, -14, 2 * N + 16, 2 * N + 16, 2 * N + 16, 4, 4, 4), (-1, -1, -1, 2 * N + 1, 2 * N + 1, 2 * N + 1, 2, 2, 2)
    shape = lambda b: tuple((b[5 - d] - b[2 - d]) // b[8 - d] + 1 for d in range(3))  # noqa: E731
    s = np.random.default_rng(order).standard_normal(shape(src))
    s = np.pad(s, ((0, 0), (0, 0), (0, s.shape[2] & 1)))
    want = np.full(shape(dst), np.nan)
    Port().transfer(op, cent, want, dst, [s], src, [0.0], reg, src, 0.0, order, 0)
    return reg, src, dst, s, want


@pytest.mark.parametrize("op,cent,order", [(OP_LAGRANGE, VERTEX, 1), (OP_LAGRANGE, CELL, 3), (OP_ENO, CELL, 5)])
def test_plain_wait_runs_out_and_is_reported(op, cent, order):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import carpet_b200 as cb
    from carpet_b200._lib import lib
    cb.set_fp_mode(False)
    reg, sb, db, s, want = _call(op, cent, order)
    src = cb.Data(sb, torch.from_numpy(s).cuda())
    dst = cb.Data(db, torch.full(want.shape, np.nan, dtype=torch.float64, device="cuda"))
    cb.check_transfers()
    assert lib.cgx_debug_skip_tma_plane(1) == 0
    try:
        cb.transfer_data(dst, [src], [0.0], reg, sb, 0.0, order, 0, op=op, cent=cent)
        with pytest.raises(cb.CgxError) as e:
            cb.check_transfers()
        assert e.value.code == EDEVICE
    finally:
        lib.cgx_debug_skip_tma_plane(0)
    cb.check_transfers()  # the report has cleared it
    cb.transfer_data(dst, [src], [0.0], reg, sb, 0.0, order, 0, op=op, cent=cent)
    cb.check_transfers()
    assert np.array_equal(dst.tensor.cpu().numpy().view(np.uint64), want.view(np.uint64))


FIRST_USE = """
import torch, carpet_b200 as cb
n = {n}
src = cb.Data((-6, -6, -6, n + 7, n + 7, n + 7, 2, 2, 2))
src.tensor.normal_()
out = [cb.Data((0, 0, 0, n, n, n, 1, 1, 1)) for _ in range(2)]
args = ([src], [0.0], (0, 0, 0, n - 1, n - 1, n - 1, 1, 1, 1), src.extent, 0.0, 5, 0)
for d in out:
    d.tensor.zero_()
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    cb.transfer_data(out[0], *args)
g.replay()
cb.transfer_data(out[1], *args)
cb.check_transfers()
torch.cuda.synchronize()
assert torch.equal(out[0].tensor, out[1].tensor) and out[0].tensor.abs().sum() > 0
print("first use in a capture ok")
"""


def test_first_use_inside_a_capture():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", FIRST_USE.format(n=N)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "first use in a capture ok" in r.stdout, r.stderr
