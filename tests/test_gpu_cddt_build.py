"""CDDT construction against the oracle's table where its passes can go wrong: grids that no word
divides, bins of every sorting size and beyond, slices too wide for shared memory; and the float form
of the projection's (int)(v +- 0.00001)."""
import numpy as np
import pytest


def _trunc_off(v, plus):
    """trunc_off of rlc_cddt.cu: (result, whether float decided)."""
    whole = np.trunc(v).astype(np.float32)
    frac = v - whole
    d = np.float32(1) - frac if plus else frac
    f = (v >= 0) & (v < 8388608) & ~((d > np.float32(0.9e-5)) & (d < np.float32(1.1e-5)))
    w = whole.astype(np.int64)
    keep = (d >= np.float32(1e-5)) | ((not plus) & (w == 0))
    return np.where(keep, w, w + (1 if plus else -1)), f


@pytest.mark.parametrize("plus", [False, True])
def test_trunc_off(plus):
    rng = np.random.default_rng(2)
    vs = [rng.uniform(0, s, 200000).astype(np.float32) for s in (1.0, 8.0, 3000.0, 70000.0, 8388608.0)]
    for w in (0.0, 1.0, 2.0, 3.0, 17.0, 255.0, 256.0, 4096.0, 40000.0, 100000.0, 8388607.0):
        vs.append((w + np.linspace(-3e-5, 3e-5, 20001)).astype(np.float32))
        b = np.float32(w).view(np.int32)
        vs.append((b + np.arange(-2000, 2001)).astype(np.int32).view(np.float32) if w else np.arange(0, 4000, dtype=np.int32).view(np.float32))
    v = np.concatenate(vs)
    got, f = _trunc_off(v, plus)
    exp = np.trunc(v.astype(np.float64) + (0.00001 if plus else -0.00001)).astype(np.int64)
    assert f.mean() > 0.5
    assert np.array_equal(got[f], exp[f])


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,fill,td", [(1, 1, 1.0, 4), (9, 7, 0.5, 6), (64, 64, 0.3, 10), (131, 77, 0.5, 18), (900, 41, 0.5, 12),
                                         (37, 1200, 0.05, 9), (26001, 3, 0.4, 6)])
def test_table(rl, oracle_mod, W, H, fill, td):
    rng = np.random.default_rng(W * H)
    occ = (rng.random((W, H)) < fill).astype(np.uint8)
    ref = oracle_mod.OracleMethod(occ, "cddt", 300.0, td=td)
    rw, rt, rlen, rz = ref.cddt_table()
    m = rl.PyCDDTCast(rl.PyOMap(np.ascontiguousarray(occ.T)), 300.0, td)
    w, t, n, z = m.table()
    assert np.array_equal(w, rw) and np.array_equal(t, rt)
    assert np.array_equal(n, rlen)
    assert np.array_equal(z, rz)
