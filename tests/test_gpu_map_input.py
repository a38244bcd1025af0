"""PyOMap(ndarray) packs the array's own memory on the device: every order, stride and type it
accepts gives grid[x][y] = arr[y, x] != 0, as do the layouts built from it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forms(a):
    """The same array in C order, Fortran order, as strided and reversed views, and read-only."""
    big = np.zeros((a.shape[0] * 2, a.shape[1] * 3), a.dtype)
    big[::2, ::3] = a
    frozen = a.copy()
    frozen.flags.writeable = False
    off = np.zeros(a.size + 3, a.dtype)[3:].reshape(a.shape)   # a base that is not 8-byte aligned
    off[...] = a
    return [np.ascontiguousarray(a), np.asfortranarray(a), big[::2, ::3], np.asfortranarray(big)[::2, ::3],
            a[::-1, ::-1][::-1, ::-1], frozen, off]


@pytest.mark.parametrize("shape", [(1, 1), (3, 17), (8, 8), (13, 64), (64, 13), (40, 72), (72, 40)])
@pytest.mark.parametrize("dtype", [np.bool_, np.uint8, np.int8, np.int64, np.float32])
def test_every_form_of_an_array(rl, oracle_mod, shape, dtype):
    rng = np.random.default_rng(shape[0] * 100 + shape[1])
    a = np.where(rng.random(shape) < 0.3, rng.integers(1, 120, shape), 0).astype(dtype)
    exp = (a != 0).T
    for k, form in enumerate(_forms(a)):
        m = rl.PyOMap(form)
        assert (m.width(), m.height()) == exp.shape and not m.error()
        assert m.occupancy.dtype == np.uint8 and np.array_equal(m.occupancy, exp), k
        assert m.isOccupied(exp.shape[0] - 1, 0) == bool(exp[-1, 0])
    dt = np.empty(exp.shape, np.float32)
    rl._lib.call("rlc_map_distance_transform", m.handle, dt.ctypes.data_as(rl._lib._f32p))
    assert np.array_equal(dt.view(np.uint32), oracle_mod.edt(exp.astype(np.uint8)).view(np.uint32))
