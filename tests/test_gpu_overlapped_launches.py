"""Kernels that are launched while the one before drains: long chains of calls whose results feed the
next call, on one stream and across streams, and the same chains captured into a graph."""
import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", params=["rm", "cddt", "glt"])
def setup(rl, request):
    occ = W.rect_disk_map(256, 23)
    om = rl.PyOMap(np.ascontiguousarray(occ.T))
    m = {"rm": lambda: rl.PyRayMarchingGPU(om, 90.0), "cddt": lambda: rl.PyCDDTCast(om, 90.0, 108),
         "glt": lambda: rl.PyGiantLUTCast(om, 90.0, 36)}[request.param]()
    m.set_sensor_model(W.sensor_table(91))
    rng = np.random.default_rng(3)
    ins = np.stack([rng.uniform(5, 250, 4000), rng.uniform(5, 250, 4000), rng.uniform(-3, 3, 4000)], 1).astype(np.float32)
    return m, torch.from_numpy(ins).cuda(), torch.linspace(-2, 2, 61, device="cuda")


def chain(m, ins, angles, bufs, side=None):
    """obs = the first pose's ranges; weights and the next poses hang on the call before."""
    ranges, obs, q, w, w2, cur = bufs
    cur.copy_(ins)
    n, na = len(ins), len(angles)
    for _ in range(6):
        m.calc_range_repeat_angles(cur, angles, ranges)
        obs.copy_(ranges[:na])
        m.eval_sensor_model(obs, ranges, w, na, n)
        if side is not None:
            main = torch.cuda.current_stream()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                m.calc_range_many(cur, q)
            m.calc_range_repeat_angles_eval_sensor_model(cur, angles, obs, w2)
            main.wait_stream(side)
        else:
            m.calc_range_many(cur, q)
            m.calc_range_repeat_angles_eval_sensor_model(cur, angles, obs, w2)
        cur[:, 2] += q * 0.01
    return ranges, q, w, w2, cur


def bufs(n, na):
    f = lambda *s, dtype=torch.float32: torch.zeros(*s, dtype=dtype, device="cuda")  # noqa: E731
    return f(n * na), f(na), f(n), f(n, dtype=torch.float64), f(n, dtype=torch.float64), f(n, 3)


def stepwise(m, ins, angles, b):
    """The same chain, every call waited for."""
    real = {k: getattr(m, k) for k in ("calc_range_repeat_angles", "eval_sensor_model", "calc_range_many",
                                       "calc_range_repeat_angles_eval_sensor_model")}

    class Waiting:
        def __getattr__(self, k):
            def call(*a):
                torch.cuda.synchronize()
                real[k](*a)
                torch.cuda.synchronize()
            return call
    return [x.clone() for x in chain(Waiting(), ins, angles, b)]


@pytest.mark.parametrize("two_streams", [False, True])
def test_chains(setup, two_streams):
    m, ins, angles = setup
    exp = stepwise(m, ins, angles, bufs(len(ins), len(angles)))
    side = torch.cuda.Stream() if two_streams else None
    for _ in range(3):
        got = chain(m, ins, angles, bufs(len(ins), len(angles)), side)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, exp))


@pytest.mark.parametrize("two_streams", [False, True])
def test_captured_chains(setup, two_streams):
    m, ins, angles = setup
    exp = stepwise(m, ins, angles, bufs(len(ins), len(angles)))
    b = bufs(len(ins), len(angles))
    side = torch.cuda.Stream() if two_streams else None
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        chain(m, ins, angles, b, side)
    torch.cuda.current_stream().wait_stream(s)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = chain(m, ins, angles, b, side)
    for _ in range(3):
        for x in b:
            x.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, e) for a, e in zip(got, exp))
