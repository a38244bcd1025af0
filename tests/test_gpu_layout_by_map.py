"""Ray marching without a schedule on maps with few equal-step runs (oblique walls) and with many: the
ranges and weights of every explicit layout."""
import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def oblique_map(side):
    """Walls two cells thick along lines at 19, 31 and 67 degrees."""
    x, y = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    occ = np.zeros((side, side), np.uint8)
    for deg, gap in ((19.0, 83.0), (31.0, 131.0), (67.0, 97.0)):
        t = np.deg2rad(deg)
        occ |= (np.mod(x * np.cos(t) + y * np.sin(t), gap) < 2.0).astype(np.uint8)
    rng = np.random.default_rng(5)
    for cx, cy in rng.integers(0, side, (side // 8, 2)):   # doors
        occ[max(cx - 6, 0):cx + 6, max(cy - 6, 0):cy + 6] = 0
    return occ


@pytest.mark.parametrize("occ", [oblique_map(300), W.corridor_map(512, 3), np.ones((40, 40), np.uint8), np.zeros((9, 70), np.uint8)],
                         ids=["oblique", "corridor", "full", "empty"])
def test_layouts_agree(rl, occ):
    m = rl.PyRayMarchingGPU(rl.PyOMap(np.ascontiguousarray(occ.T)), 120.0)
    m.set_sensor_model(W.sensor_table(121))
    rng = np.random.default_rng(1)
    n, na = 1500, 40   # repeat-angle and fused calls in the ranges where the runs may be chosen
    ins = np.stack([rng.uniform(-3, occ.shape[0] + 3, n), rng.uniform(-3, occ.shape[1] + 3, n), rng.uniform(-4, 4, n)], 1)
    ins = torch.from_numpy(ins.astype(np.float32)).cuda()
    angles = torch.linspace(-2.3, 2.3, na, device="cuda")
    obs = torch.linspace(1.0, 119.0, na, device="cuda")

    def run():
        r, q = torch.zeros(n * na, device="cuda"), torch.zeros(n, device="cuda")
        w, v = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
        m.calc_range_many(ins, q)
        m.calc_range_repeat_angles(ins, angles, r)
        m.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, w)
        rl.PyFilterBatch([(m, ins, angles, obs, v)]).run()
        torch.cuda.synchronize()
        return r, q, w, v

    got = run()
    for layout in (0, 4, 5):
        m.set_schedule(layout, 0, 0, 0)
        assert all(torch.equal(a, b) for a, b in zip(got, run())), layout
