"""push_pull more than once for the same batch: every call applies the gradients it is given, to keys seen once and to
keys with runs of any length, and what is held back for the owner counts all of them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from gpu_world import GpuWorld  # noqa: E402

WORLDS = [(1, "none"), (2, "inproc"), (2, "p2p"), (3, "p2p")]


@pytest.mark.parametrize("nrank,exchange", WORLDS)
@pytest.mark.parametrize("width", [8, 128])
def test_every_call_applies_its_gradients(nrank, exchange, width):
    # nothing is cached, learning rate 1, whole-number gradients: rows are minus the sums, whatever the order
    N, B = 400, 2500
    rng = np.random.RandomState(width)
    root = rng.randint(nrank, size=N).astype(np.uint8)
    gw = GpuWorld(nrank, N, width, 0, 0, 1.0, root, [np.flatnonzero(root == r) for r in range(nrank)], exchange=exchange)
    runs = [1, 2, 32, 33, 64, 256, 257, 500]
    keys, want = [], np.zeros((N, width), dtype=np.float32)
    for r in range(nrank):
        hot = np.repeat(rng.permutation(N)[:len(runs)], runs)
        keys.append(rng.permutation(np.concatenate([hot, rng.randint(N, size=B - len(hot))])))
    every = [rng.permutation(N) for _ in range(nrank)]
    gw.preprocess(keys)
    gw.push_pull(None)
    gw.preprocess(every)
    for _ in range(3):
        grads = [rng.randint(-8, 9, size=(B, width)).astype(np.float32) for _ in range(nrank)]
        got = gw.push_pull(grads)
        for r in range(nrank):
            np.add.at(want, keys[r], -grads[r])
        for r in range(nrank):
            assert np.array_equal(got[r], want[every[r]])
    count = np.zeros(N, dtype=np.int64)
    for r in range(nrank):
        np.add.at(count, keys[r], 3)
    for r in range(nrank):
        version, stored = gw.get(r, "version"), gw.get(r, "stored_keys")
        assert np.array_equal(version, count[stored])
    gw.close()


@pytest.mark.parametrize("exchange", ["inproc", "p2p"])
def test_push_decision_counts_both_calls(exchange):
    # rank 0 caches key 5 of rank 1 and may hold back 10 updates: 4 + 4 of one batch, pushed with the 4 of the next
    N, W = 16, 4
    root = np.array([0] * 4 + [1] * 12, dtype=np.uint8)
    gw = GpuWorld(2, N, W, 100, 10, 1.0, root, [np.arange(8), np.flatnonzero(root == 1)], exchange=exchange)
    a, other = np.full(4, 5), np.array([0, 1, 2, 3])
    g = [np.ones((4, W), dtype=np.float32), np.zeros((4, W), dtype=np.float32)]
    held = lambda: int(gw.get(0, "updates")[np.flatnonzero(gw.get(0, "stored_keys") == 5)[0]])  # noqa: E731
    gw.preprocess([a, other])
    gw.push_pull(None)
    gw.preprocess([a, other])
    gw.push_pull(g)
    assert held() == 4
    gw.push_pull(g)
    assert held() == 8
    gw.preprocess([a, other])
    gw.push_pull(g)  # 8 + 4 > 10
    assert held() == 0
    owner = np.flatnonzero(gw.get(1, "stored_keys") == 5)[0]
    assert int(gw.get(1, "version")[owner]) == 12
    assert np.array_equal(gw.get_f32(1, "embedding")[owner], np.full(W, -12, dtype=np.float32))
    gw.close()
