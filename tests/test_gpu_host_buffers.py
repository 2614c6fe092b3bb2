"""Keys, gradients and rows in host memory that is laid out in unusual ways: at addresses that are no multiple of an
element's size (fields of a packed record), or rows that take the gradients' place."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402


def _table(rows, width, lr=1.0):
    t = hb.Table(0, 1, 0, "127.0.0.1", 0, rows, width, 0, 0, np.zeros(rows, dtype=np.uint8), np.arange(rows),
                 (hb.INIT_ZERO, 0, 0), lr, 0)
    emb = np.arange(rows * width, dtype=np.float32).reshape(rows, width) % 251
    t.set_embedding(emb)
    return t, emb


def _host(a, pinned, shift=0):
    """A copy of `a` in host memory `shift` bytes behind the start of an allocation: (owner, address, view)."""
    raw = torch.zeros(a.nbytes + 64, dtype=torch.uint8)
    raw = raw.pin_memory() if pinned else raw
    view = raw.numpy()[shift:shift + a.nbytes]
    view[:] = np.frombuffer(a.tobytes(), dtype=np.uint8)
    return raw, raw.data_ptr() + shift, view


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("n,width", [(1, 4), (300, 12), (20_000, 4), (20_000, 32), (70_001, 4)])
def test_host_buffers_at_odd_addresses(n, width, pinned):
    rows = 5000
    t, emb = _table(rows, width)
    rng = np.random.RandomState(n)
    batch = [rng.randint(rows, size=n).astype(np.int64) for _ in range(2)]
    grad = rng.randint(-4, 5, size=(n, width)).astype(np.float32)
    for step in range(2):
        keys = _host(batch[step], pinned, 3)
        grads = _host(grad, pinned, 1)
        out = _host(np.zeros((n, width), dtype=np.float32), pinned, 2)
        t.preprocess(keys[1], n)
        keys[2][:] = 255  # the caller's buffer is free as soon as preprocess is back
        t.push_pull(grads[1] if step else None, out[1])
        if step:
            np.add.at(emb, batch[0], -grad)
        assert np.array_equal(np.frombuffer(out[2].tobytes(), dtype=np.float32).reshape(n, width), emb[batch[step]])
    t.close()


@pytest.mark.parametrize("n", [1, 70_001])
def test_device_keys_at_an_odd_address(n):
    t, emb = _table(5000, 4)
    keys = np.random.RandomState(n).randint(5000, size=n).astype(np.int64)
    raw = torch.zeros(8 * n + 64, dtype=torch.uint8, device="cuda")
    raw[4:4 + 8 * n] = torch.from_numpy(np.frombuffer(keys.tobytes(), dtype=np.uint8).copy()).cuda()
    out = torch.zeros((n, 4), device="cuda")
    torch.cuda.synchronize()
    t.preprocess(raw.data_ptr() + 4, n)
    t.push_pull(None, out)
    assert np.array_equal(out.cpu().numpy(), emb[keys])
    t.close()


@pytest.mark.parametrize("n,width", [(300, 16), (4000, 64), (20_000, 128)])  # copied, split in two, in pieces
@pytest.mark.parametrize("shift", [0, 7, -3000])
def test_rows_take_the_place_of_the_gradients(n, width, shift):
    # one pinned buffer for both directions, the rows `shift` floats behind the gradients
    rows = 3000
    t, emb = _table(rows, width)
    rng = np.random.RandomState(n)
    pinned = torch.zeros(n * width + 8000).pin_memory()
    buf, at = pinned.numpy(), 4000
    batch = None
    for step in range(4):
        keys = rng.randint(rows, size=n) if step % 2 else rng.randint(rows // 2, size=n)
        grad = rng.randint(-4, 5, size=(n, width)).astype(np.float32)
        buf[at:at + n * width] = grad.reshape(-1)
        t.preprocess(keys, n)
        t.push_pull(pinned.data_ptr() + 4 * at if step else None, pinned.data_ptr() + 4 * (at + shift))
        if step:
            np.add.at(emb, batch, -grad)
        assert np.array_equal(buf[at + shift:at + shift + n * width].reshape(n, width), emb[keys])
        batch = keys
    t.close()
