"""A map's occupancy needs no GPU call: it can be asked for while a graph is being captured and in a
forked child, and it is the grid as it was when the map was made."""
import os
import signal

import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("form", [np.ascontiguousarray, np.asfortranarray])
def test_occupancy_without_the_gpu(rl, form):
    occ = W.rect_disk_map(121, 3)[:, :77]
    rows = form(occ.T.copy())
    maps = [rl.PyOMap(rows) for _ in range(3)]
    rows[...] = 1
    x = torch.zeros(8, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x += 1
        inside = maps[0].occupancy.copy()
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(inside, occ) and float(x.sum()) == 8.0
    pid = os.fork()
    if pid == 0:   # host work only, and no way back into the test runner
        signal.alarm(20)
        ok = np.array_equal(maps[1].occupancy, occ) and maps[1].isOccupied(0, 0) == bool(occ[0, 0])
        os._exit(0 if ok else 1)
    assert os.waitstatus_to_exitcode(os.waitpid(pid, 0)[1]) == 0
    assert np.array_equal(maps[2].occupancy, occ)
