"""Bresenham's walk in blocks of steps over the free-distance map, against the oracle.

Walks shorter than a block, ending at and around block edges, through free spaces around the map's
largest free distance, along walls and axes, from off the map, off its edge, and far away; the fused
update of a wide block too.
"""
import os

import numpy as np
import pytest

from range_libc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


def _maps():
    rng = np.random.default_rng(12)
    one = np.zeros((260, 190), np.uint8)
    one[130, 95] = 1
    dots = (rng.random((151, 233)) < 0.0008).astype(np.uint8)
    lines = np.zeros((200, 200), np.uint8)
    lines[::66, :] = 1
    lines[:, ::67] = 1
    return {"empty": np.zeros((300, 64), np.uint8), "one": one, "dots": dots, "lines": lines,
            "thin": np.ascontiguousarray(W.rect_disk_map(256, 5)[:, :3]), "rects": W.rect_disk_map(256, 6)}


MAPS = _maps()


def _queries(occ, seed):
    rng = np.random.default_rng(seed)
    W_, H_ = occ.shape
    q = np.empty((3000, 3), np.float32)   # world frame of an identity map: x is the second index
    q[:, 0], q[:, 1] = rng.uniform(-1, H_ + 1, len(q)), rng.uniform(-1, W_ + 1, len(q))
    q[:, 2] = rng.uniform(-7, 7, len(q))
    q[500:1000, 2] = rng.integers(-4, 5, 500) * np.float32(np.pi / 2)
    q[1000:1300, 2] = rng.integers(-4, 5, 300) * np.float32(np.pi / 4)
    q[800:1200, :2] = np.floor(q[800:1200, :2]) + rng.choice([0.0, 0.5, 0.99993896], (400, 1))
    q[1300:1500, :2] = rng.uniform(-80, 400, (200, 2))
    q[1500:1510, 0] = [1e6, -1e6, 4194303.5, -4194304.0, 4194305.0, 2e7, -3e9, np.inf, np.nan, 3e38]
    return q


@pytest.mark.parametrize("name", list(MAPS))
@pytest.mark.parametrize("mr", [0.0, 0.4, 1.0, 7.5, 9.0, 10.2, 17.0, 26.5, 64.0, 66.0, 131.0, 700.0])
def test_walks(rl, oracle_mod, name, mr):
    occ = MAPS[name]
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    g = rl.PyBresenhamsLine(m, mr)
    ref = oracle_mod.OracleMethod(occ, "bl", mr, world=m.world)
    q = _queries(occ, int(mr * 10))
    ok = np.isfinite(q).all(1) & (np.abs(q[:, :2]) < 1e7).all(1)   # beyond, the reference's loop need not end
    _, trig = oracle_mod.world_rays(m.world, q)
    g.set_trig_override(trig)
    out = np.empty(len(q), np.float32)
    g.calc_range_many(q, out)
    g.set_trig_override(trig[ok])
    got = np.empty(int(ok.sum()), np.float32)
    g.calc_range_many(q[ok], got)
    exp = ref.calc_range_many(q[ok], nthreads=NT)
    assert np.array_equal(got.view(np.uint32), exp.view(np.uint32))
    assert np.array_equal(out[ok].view(np.uint32), exp.view(np.uint32))
    assert np.all(out[~ok][np.abs(q[~ok][:, 0]) > 1e8] == np.float32(mr))


def test_wide_fused_update_bl(rl, oracle_mod):
    occ = MAPS["rects"]
    m = rl.PyOMap(np.ascontiguousarray(occ.T))
    g = rl.PyBresenhamsLine(m, 70.0)
    ref = oracle_mod.OracleMethod(occ, "bl", 70.0, world=m.world)
    table = W.sensor_table(71) ** 0.1
    g.set_sensor_model(table)
    ref.set_sensor_model(table)
    fs = W.free_cell_queries(occ, 2051, 45)
    ins = np.stack([fs[:, 1], fs[:, 0], fs[:, 2]], 1).astype(np.float32)
    ang, obs = W.laser_angles(131), np.linspace(1, 69, 131).astype(np.float32)
    _, trig = oracle_mod.world_rays(m.world, ins, ang)
    g.set_trig_override(trig)
    w = np.empty(len(ins))
    g.calc_range_repeat_angles_eval_sensor_model(ins, ang, obs, w)
    exp = ref.calc_range_repeat_angles_eval_sensor_model(ins, ang, obs, nthreads=NT)
    assert np.array_equal(w.view(np.uint64), exp.view(np.uint64))
