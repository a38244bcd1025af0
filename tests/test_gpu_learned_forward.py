"""The fused forward pass at the edges of its tiles and of its grid (two tiles of 128 rays per SM and
round): the same bits as the layer-by-layer path."""
import pytest

from test_gpu_learned import learned_setup  # noqa: F401

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [1, 127, 128, 129, 151 * 128 + 1, 152 * 128, 152 * 128 + 1, 303 * 128 + 77, 304 * 128,
                               304 * 128 + 1, 457 * 128 - 5])
def test_fused_forward_at_grid_edges(rl, learned_setup, n):  # noqa: F811
    _, _, rm = learned_setup
    L = rl.PyLearnedRM(rm, seed=9)
    L.train(steps=3, batch=1024)
    xyt, _, _ = L.sample_rays(n, seed=n)
    assert torch.equal(L.predict(xyt), L.predict(xyt, layered=True))


@pytest.mark.parametrize("na", [1, 7, 30, 31, 32, 33, 108])
def test_fused_forward_of_shared_positions(rl, learned_setup, na):  # noqa: F811
    """Runs of rays from one position (features of x and y computed once where a warp's rays have at most two)."""
    _, _, rm = learned_setup
    L = rl.PyLearnedRM(rm, seed=9)
    L.train(steps=3, batch=1024)
    poses, _, _ = L.sample_rays(5000 // na + 1, seed=na)
    xyt = poses.repeat_interleave(na, dim=0)
    xyt[:, 2] += torch.linspace(-2.0, 2.0, na, device=xyt.device).repeat(len(poses))
    xyt = xyt[3:].contiguous()
    assert torch.equal(L.predict(xyt), L.predict(xyt, layered=True))
