"""CDDT queries by the table's index, and the heading wraps done in float.

The wraps of discretize_theta (RangeLib.h:1287-1340, 1834-1867) add or subtract a double constant and
round to float; add_2pi and sub_2pi (rlc_cast.cu) do the same with float pairs on the intervals tested
here for every float.  On the GPU, queries without a schedule go by the index: against the binary
search and the oracle, on the table's own zero points, at bucket and quad edges, off the map, and on
loaded tables that can or cannot have an index.
"""
import math

import numpy as np
import pytest

from range_libc_gb300 import workloads as W

K2PI = 6.28318530718            # RangeLib.h:61
HI = np.float32(float.fromhex("0x1.921fb6p+2"))
LO = np.float32(float.fromhex("-0x1.777a22p-23"))


def _two_sum(a, b):
    s = a + b
    bb = s - a
    return s, (a - (s - bb)) + (b - bb)


def _floats(lo, hi, step=1):
    a, b = np.float32(lo).view(np.uint32), np.float32(hi).view(np.uint32)
    for u in range(int(a), int(b) + 1, 1 << 23):
        yield np.arange(u, min(u + (1 << 23), int(b) + 1), step, dtype=np.uint32).view(np.float32)


def test_add_2pi_every_float():
    assert HI == np.float32(K2PI) and LO == np.float32(K2PI - float(HI))
    for t in _floats(2.0 ** -16, 16.0):
        t = -t
        s, e = _two_sum(t, HI)
        far = np.abs(s) >= np.float32(2.0 ** -10)
        t, s, e = t[far], s[far], e[far]
        assert np.array_equal((s + (e + LO)).view(np.uint32), (t.astype(np.float64) + K2PI).astype(np.float32).view(np.uint32))


def test_sub_2pi_every_float():
    for t in _floats(np.nextafter(HI, np.float32(0)), 64.0):
        t = t[t.astype(np.float64) > K2PI]
        s, e = _two_sum(t, -HI)
        assert np.array_equal((s + (e - LO)).view(np.uint32), (t.astype(np.float64) - K2PI).astype(np.float32).view(np.uint32))


# ---------------------------------------------------------------- GPU
def _bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


def _queries(occ, seed):
    """Free and occupied poses, cell corners and centres with axis headings (on zero points exactly),
    far off the map, huge and infinite coordinates and headings, NaN."""
    rng = np.random.default_rng(seed)
    W_, H_ = occ.shape
    q = np.empty((12000, 3), np.float32)
    q[:, 0], q[:, 1] = rng.uniform(-4, W_ + 4, len(q)), rng.uniform(-4, H_ + 4, len(q))
    q[:, 2] = rng.uniform(-20, 20, len(q))
    q[2000:6000, :2] = np.floor(q[2000:6000, :2]) + 0.5
    q[3000:7000, 2] = rng.integers(-8, 9, 4000) * np.float32(math.pi / 4)
    q[6000:7000, :2] = np.floor(q[6000:7000, :2])
    q[7000:7200, :2] *= 1000.0
    q[7200:7210] = [[np.inf, 3, 0], [3, np.inf, 1], [-np.inf, 2, 2], [2, -np.inf, 3], [np.nan, 1, 1], [1, np.nan, 1],
                    [1, 1, np.nan], [3e38, 3e38, 0.5], [5, 5, 1e4], [5, 5, -1e4]]
    q[7210:7300, 2] = rng.uniform(-2e-4, 2e-4, 90)
    return q


def _check(rl, g, q, exp=None):
    """No schedule (the index) against the binary search, in grid coordinates."""
    a, b = np.full(len(q), -1, np.float32), np.full(len(q), -2, np.float32)
    for out, fresh in ((a, True), (b, False)):
        if not fresh:
            g.set_schedule(0, 0, 0, 0)
        rl._lib.call("rlc_calc_range_many", g.handle, q.ctypes.data, out.ctypes.data, len(q), rl._lib.RLC_NO_WORLD, None)
    same = (_bits(a) == _bits(b)) | (np.isnan(a) & np.isnan(b))
    assert same.all(), (int((~same).sum()), q[~same][:3], a[~same][:3], b[~same][:3])
    if exp is not None:
        assert np.array_equal(_bits(a), _bits(exp))


@pytest.mark.gpu
@pytest.mark.parametrize("td", [2, 3, 16, 107, 108])
@pytest.mark.parametrize("prune", [False, True])
@pytest.mark.parametrize("name", ["small", "rect", "wide", "empty", "full", "corridor"])
def test_index_equals_binary_search(rl, oracle_mod, name, td, prune):
    occ = {"small": (np.random.default_rng(3).random((5, 6)) < 0.3).astype(np.uint8),
           "rect": W.rect_disk_map(200, 21), "wide": np.ascontiguousarray(W.rect_disk_map(512, 22)[:130, :450]),
           "empty": np.zeros((40, 25), np.uint8), "full": np.ones((70, 130), np.uint8),
           "corridor": W.corridor_map(400, 24)}[name]
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    g = rl.PyCDDTCast(m, 90.0, td)
    if prune:
        g.prune()
    q = _queries(occ, td)
    fin = np.isfinite(q).all(1) & (np.abs(q[:, 2]) < 50) & (np.abs(q[:, :2]) < 1e4).all(1)
    h = rl.PyCDDTCast(m, 90.0, td)
    if prune:
        h.prune()
    _check(rl, g, q)
    ref = oracle_mod.OracleMethod(occ, "pcddt" if prune else "cddt", 90.0, td=td)
    out = np.empty(int(fin.sum()), np.float32)
    h.calc_range_many(q[fin], out)
    assert np.array_equal(_bits(out), _bits(ref.calc_range_many(q[fin])))


@pytest.mark.gpu
@pytest.mark.parametrize("change", ["thinned", "doubled", "one_bin", "upper_slices", "infinite", "unsorted"])
def test_index_of_a_loaded_table(rl, change):
    """Tables from outside: fewer zero points, repeated ones, a crowded bin, slices past td / 2 filled;
    and two that cannot have an index and are searched as before."""
    occ = W.rect_disk_map(150, 33)
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    td = 24
    src = rl.PyCDDTCast(m, 80.0, td)
    widths, trans, n, z = src.table()
    bins = np.split(z, np.cumsum(n)[:-1])
    rng = np.random.default_rng(5)
    if change == "thinned":
        bins = [b[::3] for b in bins]
    elif change == "doubled":
        bins = [np.repeat(b, 2) for b in bins]
    elif change == "one_bin":
        k = int(np.argmax(n))
        bins = [np.sort(rng.uniform(-50, 200, 5000)).astype(np.float32) if i == k else b for i, b in enumerate(bins)]
    elif change == "upper_slices":
        lo = int(widths[:td // 2].sum())
        bins = [b if i < lo else np.sort(rng.uniform(-150, 150, 3)).astype(np.float32) for i, b in enumerate(bins)]
    elif change == "infinite":
        bins = [np.append(b, np.float32(np.inf)) if len(b) else b for b in bins]
    else:
        bins = [b[::-1] for b in bins]
    ln = np.array([len(b) for b in bins], np.int64)
    g = rl.PyCDDTCast(m, 80.0, td)
    g.load_table(trans, ln, np.concatenate(bins))
    _check(rl, g, _queries(occ, 6))


@pytest.mark.gpu
def test_batch_after_the_table_changed(rl):
    """A batch made before its CDDT method was pruned takes up the new table at its next run."""
    torch = pytest.importorskip("torch")
    occ = W.rect_disk_map(200, 44)
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    g = rl.PyCDDTCast(m, 90.0, 36)
    table = W.sensor_table(91) ** 0.3
    g.set_sensor_model(table)
    fs = W.free_cell_queries(occ, 200, 45)
    ins = np.stack([fs[:, 1], fs[:, 0], fs[:, 2]], 1).astype(np.float32)
    ang, obs = W.laser_angles(41), np.linspace(1, 80, 41).astype(np.float32)
    t = [torch.from_numpy(a).cuda() for a in (ins, ang, obs)]
    w = torch.zeros(200, dtype=torch.float64, device="cuda")
    batch = rl.PyFilterBatch([(g, *t, w)])
    batch.run()
    g.prune()
    w.fill_(-1.0)
    batch.run()
    torch.cuda.synchronize()
    exp = np.empty(200)
    g.calc_range_repeat_angles_eval_sensor_model(ins, ang, obs, exp)
    assert np.array_equal(w.cpu().numpy().view(np.uint64), exp.view(np.uint64))
