"""Gradients and training of the learned surrogate at the edges of their splits: one tile of rays,
batches that no split divides, several splits of unequal length; and that a run repeats bit for bit."""
import numpy as np
import pytest

from test_gpu_learned import KFEAT, KHID, bf16, cpu_gradients, learned_setup  # noqa: F401

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n", [128, 384, 640, 20096])
def test_gradients_at_split_edges(rl, learned_setup, n):  # noqa: F811
    _, _, rm = learned_setup
    L = rl.PyLearnedRM(rm, seed=7)
    xyt, t, _ = L.sample_rays(n, seed=n)
    g, loss = L.gradients(xyt, t)
    g2, loss2 = L.gradients(xyt, t)
    assert np.array_equal(g, g2) and loss == loss2
    X = L.features(xyt).float().cpu().numpy()
    exp, exp_loss = cpu_gradients(L.params(), X, t.cpu().numpy())
    assert abs(loss - exp_loss) <= 1e-3 * max(1.0, abs(exp_loss))
    off = 0
    for l in range(4):   # the bounds of the 256- and 2,048-ray cases
        for size in (KHID * (KFEAT if l == 0 else KHID), KHID):
            a, b = g[off:off + size], exp[off:off + size]
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b) + 1e-9, (l, size)
            off += size
    assert np.linalg.norm(g[off:] - exp[off:]) <= 1e-3 * np.linalg.norm(exp[off:]) + 1e-9


def test_training_repeats(rl, learned_setup):  # noqa: F811
    _, _, rm = learned_setup
    runs = []
    for _ in range(2):
        L = rl.PyLearnedRM(rm, seed=5)
        loss = L.train(steps=25, batch=1152, seed=9)
        runs.append((loss, L.params()))
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][1], runs[1][1])


@pytest.mark.parametrize("a_t,b_t", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (384, 512, 576), (128, 256, 4160)])
@pytest.mark.parametrize("shift", [0, 1])   # operands off the tile loads' 16 bytes
def test_transposed_operands(rl, M, N, K, a_t, b_t, shift):
    """Small whole numbers: products and sums are exact in float32."""
    rng = np.random.default_rng(M + N + K)
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    b = rng.integers(-3, 4, (N, K)).astype(np.float32)
    dev = torch.device("cuda:0")

    def put(x, t):
        flat = np.ascontiguousarray(x.T if t else x).reshape(-1)
        at = shift if t else 0
        buf = torch.zeros(flat.size + 8, dtype=torch.bfloat16, device=dev)
        buf[at:at + flat.size] = torch.from_numpy(flat).to(dev).to(torch.bfloat16)
        return buf[at:at + flat.size]

    c = rl.tc_gemm(put(a, a_t), put(b, b_t), M, N, K, bool(a_t), bool(b_t))
    torch.cuda.synchronize()
    assert np.array_equal(c.cpu().numpy(), a @ b.T)


@pytest.mark.parametrize("K", [128, 384, 640, 4224])   # stages of 128 K: fewer than, as many as and more than the ring
def test_transposed_operands_long_stages(rl, K):
    """Small whole numbers: products and sums are exact in float32."""
    M, N = 256, 256
    rng = np.random.default_rng(K)
    a = rng.integers(-3, 4, (M, K)).astype(np.float32)
    b = rng.integers(-3, 4, (N, K)).astype(np.float32)
    put = lambda x: torch.from_numpy(np.ascontiguousarray(x.T)).cuda().to(torch.bfloat16)  # noqa: E731
    c = rl.tc_gemm(put(a), put(b), M, N, K, True, True)
    torch.cuda.synchronize()
    assert np.array_equal(c.cpu().numpy(), a @ b.T)
