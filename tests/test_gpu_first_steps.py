"""The first steps of a fresh table: what a step of this size needs is there after the first pull - nothing is allocated in
the steps that follow, and the first one with gradients launches what every later one launches."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402
from gpu_world import GpuWorld, _parallel  # noqa: E402


def _steps(nrank, n, width, keys_on_device):
    """(kernels launched, free device memory afterwards) of five steps of a fresh table, the first without gradients."""
    rows = 500_000
    root = (np.arange(rows) % nrank).astype(np.uint8)
    gw = GpuWorld(nrank, rows, width, 0, 0, 0.1, root, [np.flatnonzero(root == r) for r in range(nrank)],
                  exchange="p2p")
    rng = np.random.RandomState(n)
    keys = [[rng.randint(rows, size=n).astype(np.int64) for _ in range(nrank)] for _ in range(2)]
    if keys_on_device:
        keys = [[torch.from_numpy(k).cuda() for k in b] for b in keys]
    grads = [torch.zeros((n, width), device="cuda") for _ in range(nrank)]
    out = [torch.zeros((n, width), device="cuda") for _ in range(nrank)]
    got = []
    for step in range(5):
        torch.cuda.synchronize()
        before = hb.lib().hctr_launch_count()
        _parallel([lambda r=r: gw.tables[r].preprocess(keys[step & 1][r], n) for r in range(nrank)])
        _parallel([lambda r=r: gw.tables[r].push_pull(grads[r] if step else None, out[r]) for r in range(nrank)])
        launches = hb.lib().hctr_launch_count() - before
        torch.cuda.synchronize()
        got.append((launches, torch.cuda.mem_get_info()[0]))
    gw.close()
    return got


@pytest.mark.parametrize("keys_on_device", [True, False])
@pytest.mark.parametrize("nrank,n", [(1, 20_000), (1, 600_000), (2, 300_000)])
def test_nothing_is_left_for_the_first_gradients(nrank, n, keys_on_device):
    _steps(nrank, n, 8, keys_on_device)  # (the driver loads kernels when they are first used)
    steps = _steps(nrank, n, 8, keys_on_device)
    assert len({free for _, free in steps}) == 1
    assert len({launches for launches, _ in steps[1:]}) == 1


def test_a_serving_loop_does_not_group_its_batches():
    rows, n = 10_000, 5000
    gw = GpuWorld(1, rows, 8, 0, 0, 0.1, np.zeros(rows, dtype=np.uint8), [np.arange(rows)])
    t, keys, out = gw.tables[0], torch.arange(n, device="cuda"), torch.zeros((n, 8), device="cuda")
    count = []
    for _ in range(4):
        before = hb.lib().hctr_launch_count()
        t.preprocess(keys, n)
        t.push_pull(None, out)
        count.append(hb.lib().hctr_launch_count() - before)
    assert count[0] == 3 and count[1:] == [2, 2, 2]  # key ingest and expansion; the first pull may open a training loop
    gw.close()
