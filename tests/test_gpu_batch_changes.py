"""Batches whose methods change between runs: another sensor model, of another size, and another trig override."""
import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kinds", [("rm", "rm"), ("bl", "cddt")])
def test_another_sensor_model_between_runs(rl, kinds):
    """Every run takes the tables that the per-filter calls take at that moment."""
    occ = W.rect_disk_map(200, 17)
    om = rl.PyOMap(np.ascontiguousarray(occ.T))
    make = {"rm": lambda: rl.PyRayMarching(om, 80.0), "bl": lambda: rl.PyBresenhamsLine(om, 80.0),
            "cddt": lambda: rl.PyCDDTCast(om, 80.0, 72)}
    fs = W.free_cell_queries(occ, 150, 18)
    ins = np.stack([fs[:, 1], fs[:, 0], fs[:, 2]], 1).astype(np.float32)
    ang, obs = W.laser_angles(37), np.linspace(2, 78, 37).astype(np.float32)
    methods = [make[k]() for k in kinds]
    for m in methods:
        m.set_sensor_model(W.sensor_table(81))
    dev = [torch.from_numpy(a).cuda() for a in (ins, ang, obs)]
    outs = [torch.zeros(len(ins), dtype=torch.float64, device="cuda") for _ in methods]
    batch = rl.PyFilterBatch([(m, *dev, w) for m, w in zip(methods, outs)])
    seen = []
    for which, size in ((None, 0), (1, 57), (0, 130), (1, 81), (1, 40)):
        if which is not None:
            methods[which].set_sensor_model(W.sensor_table(size) ** 0.5)
        batch.run()
        torch.cuda.synchronize()
        for m, w in zip(methods, outs):
            exp = np.empty(len(ins))
            m.calc_range_repeat_angles_eval_sensor_model(ins, ang, obs, exp)
            assert np.array_equal(w.cpu().numpy().view(np.uint64), exp.view(np.uint64)), (which, size)
        seen.append(outs[1].cpu().numpy().copy())
    assert not np.array_equal(seen[0], seen[1]) and not np.array_equal(seen[3], seen[4])
