"""Steps as a training loop takes them: nothing is looked at in between but the pulled rows (any look at a table drains its
streams), so work of one step overlaps the next.  State is compared once, at the end."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from gpu_world import _parallel, assert_index_parity, assert_state_parity  # noqa: E402
from test_gpu_parity import make_worlds  # noqa: E402


def _push_pull(gw, grads):
    """gw.push_pull without draining the device: the inputs are ready when torch's own stream is."""
    if gw.buffers != "device":
        return gw.push_pull(grads)
    dsts = [torch.full((max(b, 1), gw.width), float("nan"), device=gw.dev) for b in gw._batch]
    grads = [None] * gw.nrank if grads is None else [torch.from_numpy(g).to(gw.dev) for g in grads]
    torch.cuda.current_stream().synchronize()
    _parallel([lambda r=r: gw.tables[r].push_pull(grads[r], dsts[r]) for r in range(gw.nrank)])
    return [d[:b].cpu().numpy() for d, b in zip(dsts, gw._batch)]


def _run(gw, ow, plan, batch, seed=0):
    """plan: a letter per step - t(rain), s(erve: no gradients), 2 (preprocess twice, then train), e(mpty batch, train),
    x (a key outside the table, refused; then train).  batch(step, rank) -> keys."""
    rng = np.random.RandomState(seed)
    n, W = gw.nrank, gw.width
    last = [np.zeros(0, dtype=np.int64)] * n
    for step, what in enumerate(plan):
        keys = [batch(step, r) for r in range(n)]
        if what == "e":
            keys = [k[:0] for k in keys]
        if what == "x":
            bad = [k.copy() for k in keys]
            bad[0][len(bad[0]) // 2] = gw.length
            with pytest.raises(RuntimeError, match="outside"):
                gw.preprocess(bad)
            ow.preprocess([k[:0] for k in keys])  # the refused batch stands there empty
            last = [k[:0] for k in keys]
        if what == "2":
            for w in (gw, ow):
                w.preprocess(keys)
            last, keys = keys, [k[::-1].copy() for k in keys]
        for w in (gw, ow):
            w.preprocess(keys)
        grads = None if what == "s" else [rng.normal(0, 1, size=(len(k), W)).astype(np.float32) for k in last]
        got, want = _push_pull(gw, grads), ow.push_pull(grads)
        for r in range(n):
            assert np.array_equal(got[r], want[r]), f"step {step} ({what}) rank {r}"
        last = keys
    assert_state_parity(gw, ow)
    for w in (gw, ow):
        w.preprocess(last)
    assert_index_parity(gw, ow)
    gw.close()


PLANS = ["sttttttt", "ssstttsst", "st2tts2t", "setstets", "tttstttt"]


@pytest.mark.parametrize("plan", PLANS + ["stxtsxtt"])
@pytest.mark.parametrize("keys_on_device", [True, False])
# one cluster; the largest cluster and the smallest batch of the multi-launch form in turn; several tiles of 4 and 8
@pytest.mark.parametrize("sizes", [(700, 500), (65_536, 65_537), (300_000, 470_000)])
def test_single_rank(oracle_mod, plan, keys_on_device, sizes):
    N, W = 20_000, 4
    rng = np.random.RandomState(len(plan) + sizes[0])
    gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.1, np.zeros(N, dtype=np.uint8), [rng.permutation(N)],
                         keys_on_device=keys_on_device)
    _run(gw, ow, plan, lambda step, r: (rng.zipf(1.3, size=sizes[step % 2]) * 7919) % N)


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("buffers,B,W", [("pinned", 300, 16), ("pinned", 4000, 64), ("pinned", 9000, 256), ("pageable", 4000, 64)])
def test_host_buffers(oracle_mod, plan, buffers, B, W):
    N = 3 * B
    rng = np.random.RandomState(B)
    gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.1, np.zeros(N, dtype=np.uint8), [np.arange(N)], buffers=buffers,
                         keys_on_device=False)
    _run(gw, ow, plan, lambda step, r: np.where(rng.rand(B) < 0.6, rng.randint(N // 40, size=B), rng.randint(N, size=B)))


@pytest.mark.parametrize("plan", PLANS)
@pytest.mark.parametrize("exchange", ["inproc", "p2p"])
@pytest.mark.parametrize("nrank,B,W,bound", [(2, 2000, 16, 0), (2, 2000, 128, 3), (2, 80_000, 4, 3), (3, 1500, 32, 2)])
def test_ranks(oracle_mod, plan, exchange, nrank, B, W, bound):
    N = 6000
    rng = np.random.RandomState(nrank * 10 + bound)
    root = rng.randint(nrank, size=N).astype(np.uint8)
    storage = [np.flatnonzero((root == r) | (rng.rand(N) < 0.3)) for r in range(nrank)]
    gw, ow = make_worlds(oracle_mod, nrank, N, W, bound, bound, 0.1, root, storage, exchange=exchange, keys_on_device=False)
    _run(gw, ow, plan, lambda step, r: (rng.zipf(1.2, size=B) * 31) % N)


@pytest.mark.parametrize("n", [9, 100, 70_000])
@pytest.mark.parametrize("bad", [-1, 5000, 1 << 40])
def test_bad_host_key_anywhere(oracle_mod, n, bad):
    # the copy of a host batch finds it - in its vector body, its tail, its second piece - the batch is refused, and the
    # step after it is exact
    N, W = 5000, 4
    gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.1, np.zeros(N, dtype=np.uint8), [np.arange(N)], keys_on_device=False)
    rng = np.random.RandomState(n)
    places = [p for p in (0, 7, 8, n - 1, 65_535, 65_536, 69_999) if p < n]
    last = np.zeros(0, dtype=np.int64)
    for p in places:
        good = rng.randint(N, size=n)
        keys = good.copy()
        keys[p] = bad
        with pytest.raises(RuntimeError, match="outside"):
            gw.preprocess([keys])
        ow.preprocess([last[:0]])
        for k in (good, rng.randint(N, size=300)):
            for w in (gw, ow):
                w.preprocess([k])
            g = None if k is good else [rng.normal(0, 1, size=(len(last), W)).astype(np.float32)]
            assert np.array_equal(_push_pull(gw, g)[0], ow.push_pull(g)[0])
            last = k
    assert_state_parity(gw, ow)
    gw.close()


@pytest.mark.parametrize("pinned", [False, True])
def test_bad_host_key_with_ranks(oracle_mod, pinned):
    # the ranks are in step: the key is reported by its rank's push_pull, and the next steps are exact
    N, W, n = 5000, 4, 70_000
    root = (np.arange(N) % 2).astype(np.uint8)
    storage = [np.flatnonzero(root == r) for r in range(2)]
    gw, ow = make_worlds(oracle_mod, 2, N, W, 0, 0, 0.1, root, storage, exchange="p2p", keys_on_device=False)
    rng = np.random.RandomState(3)
    keys = [rng.randint(N, size=n) for _ in range(2)]
    keys[0][66_000] = -1
    gw.preprocess([torch.from_numpy(k).pin_memory().numpy() if pinned else k for k in keys])
    with pytest.raises(RuntimeError, match="outside"):
        gw.push_pull(None)
    last = None
    for step in range(3):
        keys = [rng.randint(N, size=2000) for _ in range(2)]
        for w in (gw, ow):
            w.preprocess(keys)
        g = None if last is None else [rng.normal(0, 1, size=(2000, W)).astype(np.float32) for _ in range(2)]
        got, want = _push_pull(gw, g), ow.push_pull(g)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        last = keys
    assert_state_parity(gw, ow)
    gw.close()
