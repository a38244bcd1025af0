"""Tuning against what a call picks without a schedule: it is among the candidates, and whatever is kept gives
the same bits, in the fused update, the other calls and batches."""
import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind,n,na", [("rm", 2100, 150), ("rm", 300, 21), ("cddt", 2800, 100), ("glt", 5500, 48), ("bl", 2000, 132)])
def test_tuned_calls(rl, kind, n, na):
    occ = W.corridor_map(300, 8)
    om = rl.PyOMap(np.ascontiguousarray(occ.T))
    make = {"rm": lambda: rl.PyRayMarchingGPU(om, 90.0), "cddt": lambda: rl.PyCDDTCast(om, 90.0, 72),
            "glt": lambda: rl.PyGiantLUTCast(om, 90.0, 36), "bl": lambda: rl.PyBresenhamsLine(om, 90.0)}[kind]
    fs = W.free_cell_queries(occ, n, 9)
    ins = torch.from_numpy(np.stack([fs[:, 1], fs[:, 0], fs[:, 2]], 1).astype(np.float32)).cuda()
    ang = torch.from_numpy(W.laser_angles(na)).cuda()
    obs = torch.linspace(1, 80, na, device="cuda")

    def results(m):
        w, r, q = (torch.full((k,), -1.0, dtype=d, device="cuda") for k, d in ((n, torch.float64), (n * na, torch.float32), (n, torch.float32)))
        m.calc_range_repeat_angles_eval_sensor_model(ins, ang, obs, w)
        m.calc_range_repeat_angles(ins, ang, r)
        m.calc_range_many(ins, q)
        torch.cuda.synchronize()
        return w, r, q

    m = make()
    m.set_sensor_model(W.sensor_table(91) ** 0.2)
    exp = results(m)
    m.autotune(ins, ang, obs, torch.empty(n, dtype=torch.float64, device="cuda"))
    table = m.autotune_results()
    own = [t for t in table if t[0][1:] == (0, 0, 0) and t[0][0] != 3]
    assert len(own) == 1 and own[0][1] > 0 and sum(t[2] is not None for t in table) == 3
    assert all(torch.equal(a, b) for a, b in zip(results(m), exp))
    sched = m.schedule()
    assert any(t[2] is not None and t[0][0] == sched[0] and t[0][2:] == sched[2:] for t in table)
    m.set_schedule(*sched)
    assert all(torch.equal(a, b) for a, b in zip(results(m), exp))


def test_tuned_batch(rl):
    filters, exp = [], []
    for side, n, na, mr, seed in ((256, 700, 61, 100.0, 3), (400, 90, 300, 150.0, 4), (128, 33, 7, 60.0, 5)):
        wl = W.batch_filter(W.FilterSpec(side, n, na, mr, seed))
        m = rl.PyRayMarching(rl.PyOMap(np.ascontiguousarray(wl.occ.T)), wl.max_range)
        m.set_sensor_model(wl.table)
        t = [torch.from_numpy(a).cuda() for a in (wl.ins, wl.angles, wl.obs)]
        w = torch.zeros(len(wl.ins), dtype=torch.float64, device="cuda")
        m.calc_range_repeat_angles_eval_sensor_model(*t, w)
        exp.append(w.clone())
        filters.append((m, *t, w))
    batch = rl.PyFilterBatch(filters)
    batch.autotune()
    for f in filters:
        f[4].fill_(-1.0)
    batch.run()
    torch.cuda.synchronize()
    assert all(torch.equal(f[4], e) for f, e in zip(filters, exp))
