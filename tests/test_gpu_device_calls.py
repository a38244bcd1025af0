"""Calls on CUDA tensors through the C entry points against the checked Python path: the same results,
the same refusals, the caller's current stream."""
import numpy as np
import pytest

from range_libc_gb300 import _lib, workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def setup(rl):
    occ = W.rect_disk_map(200, 17)
    m = rl.PyRayMarchingGPU(rl.PyOMap(np.ascontiguousarray(occ.T)), 90.0)
    m.set_sensor_model(W.sensor_table(91))
    rng = np.random.default_rng(3)
    ins = np.stack([rng.uniform(5, 195, 50), rng.uniform(5, 195, 50), rng.uniform(-3, 3, 50)], 1).astype(np.float32)
    put = lambda x: torch.from_numpy(x).cuda()  # noqa: E731
    obs = rng.uniform(1, 80, 20).astype(np.float32)
    return m, put(ins), put(np.linspace(-2, 2, 20, dtype=np.float32)), put(obs)


def run(m, ins, angles, obs):
    n, na = len(ins), len(angles)
    r = torch.full((n * na + 3,), -7.0, device="cuda")
    q, w, v = torch.zeros(n, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    m.calc_range_repeat_angles(ins, angles, r)
    m.calc_range_many(ins, q)
    m.eval_sensor_model(obs, r, w, na, n)
    m.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, v)
    return r, q, w, v


def test_same_as_checked_path(setup, monkeypatch):
    m, ins, angles, obs = setup
    assert _lib.fast() is not None
    a = run(m, ins, angles, obs)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        b = run(m, ins, angles, obs)
    side.synchronize()
    c = run(m, torch.nn.Parameter(ins), angles, obs)   # a subclass: by the checked path
    monkeypatch.setattr(_lib, "_fast", False)
    d = run(m, ins, angles, obs)
    for x in (b, c, d):
        assert all(torch.equal(p, q) for p, q in zip(a, x))


def test_empty(setup):
    m, ins, angles, obs = setup
    run(m, ins[:0], angles, obs)


@pytest.mark.parametrize("fast", [True, False])
def test_refusals(setup, monkeypatch, fast):
    m, ins, angles, obs = setup
    if not fast:
        monkeypatch.setattr(_lib, "_fast", False)
    out = torch.zeros(1000, device="cuda")
    w = torch.zeros(50, dtype=torch.float64, device="cuda")
    for bad in (lambda: m.calc_range_many(ins, out),                                  # fewer rows than outs
                lambda: m.calc_range_many(ins.double(), out[:50]),
                lambda: m.calc_range_many(ins, out[:100:2]),
                lambda: m.calc_range_many(ins[0], out[:3]),
                lambda: m.calc_range_many(ins, np.zeros(50, np.float32)),
                lambda: m.calc_range_repeat_angles(ins, angles, out[:999]),
                lambda: m.calc_range_repeat_angles(ins, angles.cpu().numpy(), out),
                lambda: m.eval_sensor_model(obs, out, w.float(), 20, 50),
                lambda: m.eval_sensor_model(obs, out[:999], w, 20, 50),
                lambda: m.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs[:19], w),
                lambda: m.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, w[:49])):
        with pytest.raises(ValueError):
            bad()
    with pytest.raises(TypeError):
        m.calc_range_many(ins.cpu(), out[:50])
