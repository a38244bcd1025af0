"""The sensor model's kernels at the sizes where they change shape.

eval_sensor_model takes 32 particles per block and 32 beams per chunk; the fused update of 256 K rays
or more (no schedule set; ray marching from 2,000 particles x 128 beams, tables from 48 beams) takes
up to 32 particles per block through chunks of beams, with table factors or bins in shared memory.  Both must give the oracle's weights bit for bit, and a call without a
schedule those of the same call with one.
"""
import os

import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint64)


@pytest.fixture(scope="module")
def small(rl, oracle_mod):
    occ = W.rect_disk_map(256, 61)
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    g = rl.PyRayMarching(m, 100.0)
    ref = oracle_mod.OracleMethod(occ, "rm", 100.0, world=m.world)
    table = W.sensor_table(101) ** 0.25
    g.set_sensor_model(table)
    ref.set_sensor_model(table)
    return g, ref


@pytest.mark.parametrize("n", [1, 31, 32, 33, 70])
@pytest.mark.parametrize("na", [0, 1, 31, 32, 33, 64, 65, 300])
def test_eval_sensor_model_edges(small, n, na):
    g, ref = small
    rng = np.random.default_rng(n * 1000 + na)
    obs = rng.uniform(-5, 120, na).astype(np.float32)
    ranges = rng.uniform(-5, 120, n * na).astype(np.float32)
    ranges[rng.random(n * na) < 0.01] = np.inf
    w = np.full(n, -1.0)
    g.eval_sensor_model(obs, ranges, w, na, n)
    exp = ref.eval_sensor_model(obs, ranges, na, n) if na else np.ones(n)
    assert np.array_equal(_bits(w), _bits(exp))


# particles per block 2, 3, 8 (factors), 9 and 17 (bins) on 152 SMs, a last block of one particle, a
# chunk's last beam alone, several chunks, two waves of blocks
@pytest.mark.parametrize("n,na", [(2000, 132), (2049, 512), (2049, 513), (2433, 433), (5461, 193), (9728, 129),
                                   (9729, 128), (3000, 1081), (20673, 137), (39000, 192),
                                   (5500, 48), (250, 1081)])
@pytest.mark.parametrize("kind", ["rm", "cddt", "glt"])
def test_wide_fused_update(rl, oracle_mod, kind, n, na):
    side, mr = 300, 60.0
    occ = np.ascontiguousarray(W.rect_disk_map(side, 62)[:, :250])
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    cls = {"rm": rl.PyRayMarching, "cddt": rl.PyCDDTCast, "glt": rl.PyGiantLUTCast}[kind]
    g = cls(m, mr) if kind == "rm" else cls(m, mr, 36)
    table = W.sensor_table(int(mr) + 1) ** (8.0 / na)
    g.set_sensor_model(table)
    rng = np.random.default_rng(n + na)
    ins = np.empty((n, 3), np.float32)
    ins[:, 0], ins[:, 1] = rng.uniform(-10, 260, n), rng.uniform(-10, 310, n)   # some off the map
    ins[:, 2] = rng.uniform(-4, 4, n)
    ins[::701, rng.integers(0, 3)] = np.nan
    angles = W.laser_angles(na)
    obs = rng.uniform(0, mr, na).astype(np.float32)
    w = np.full(n, -1.0)
    g.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, w)
    assert g.schedule() == (0, 256, 0, 0)
    g.set_schedule(0, 0, 0, 0)
    exp = np.empty(n)
    g.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, exp)
    assert np.array_equal(_bits(w), _bits(exp))
    if kind == "rm":   # the host's cos/sin on both sides
        h = cls(m, mr)
        h.set_sensor_model(table)
        _, trig = oracle_mod.world_rays(m.world, ins, angles)
        h.set_trig_override(trig)
        h.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, w)
    if kind != "glt":
        ref = oracle_mod.OracleMethod(occ, kind, mr, td=36, world=m.world)
        ref.set_sensor_model(table)
        exp = ref.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, nthreads=NT)
        assert np.array_equal(_bits(w), _bits(exp))


@pytest.mark.parametrize("scale", [1, 40])   # a few particles per tile, and 16
def test_wide_batch(rl, oracle_mod, scale):
    """A batch without a schedule against per-filter calls: tiles of 2 to 16 particles, chunks with one
    beam, filters without particles or beams, poses off the map, ranges kept, cos/sin given."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(70 + scale)
    filters, host = [], []
    sizes = [(700, 129), (1, 300), (33, 1), (0, 50), (5, 0), (900, 128), (1300, 61)]
    for k, (n, na) in enumerate(sizes):
        n *= scale
        mr = 50.0 + 9 * k
        occ = np.ascontiguousarray(W.rect_disk_map(256, 80 + k)[:, :200 + k])
        m = rl.PyOMap(np.ascontiguousarray(occ.T))
        g = rl.PyRayMarching(m, mr)
        table = W.sensor_table(int(mr) + 1) ** 0.1
        g.set_sensor_model(table)
        ins = np.empty((n, 3), np.float32)
        ins[:, 0], ins[:, 1] = rng.uniform(-5, 210, n), rng.uniform(-5, 260, n)
        ins[:, 2] = rng.uniform(-7, 7, n)
        ins[::97, 2] = np.nan
        angles = W.laser_angles(na) if na else np.zeros(0, np.float32)
        obs = rng.uniform(0, mr, na).astype(np.float32)
        if k == 5:
            g.set_trig_override(oracle_mod.world_rays(m.world, ins, angles)[1])
        t = [torch.from_numpy(a).cuda() for a in (ins, angles, obs)]
        filters.append((g, *t, torch.full((n,), -1.0, dtype=torch.float64, device="cuda"),
                        torch.full((n * na,), -1.0, device="cuda") if k % 2 == 0 else None))
        host.append((ins, angles, obs, n, na))
    batch = rl.PyFilterBatch(filters)
    for _ in range(2):
        batch.run()
    torch.cuda.synchronize()
    assert batch.schedule() == (0, 0, 256, 0) and batch.product_mode() == "overlapped"
    first = [f[4].clone() for f in filters]
    for f, (ins, angles, obs, n, na) in zip(filters, host):
        g = f[0]
        g.set_schedule(0, 0, 0, 0)
        if n:
            w = np.empty(n)
            g.calc_range_repeat_angles_eval_sensor_model(ins, angles, obs, w)
            assert np.array_equal(_bits(f[4].cpu().numpy()), _bits(w)), (n, na)
        if f[5] is not None and n and na:
            r = np.empty(n * na, np.float32)
            g.calc_range_repeat_angles(ins, angles, r)
            assert np.array_equal(f[5].cpu().numpy().view(np.uint32), r.view(np.uint32)), (n, na)
    for separate in (False, True):   # the schedules that a caller can ask for afterwards
        batch.set_product_mode(separate)
        batch.run()
        torch.cuda.synchronize()
        assert all(torch.equal(a, f[4]) for a, f in zip(first, filters))
