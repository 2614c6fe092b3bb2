"""The key ingest that is launched before its keys are staged: chunks that arrive one by one, that will not come and that do
not come in time (the kernel then says so and returns), on caller-owned buffers; and tables whose ingest gives up, or whose
launches wait for their kernels, against the oracle."""
import ctypes
import os
import subprocess
import sys
import time

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
vp, sz, u32 = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_uint32
CHUNK, LOST = 1000, 0xffffffff


@pytest.mark.parametrize("width", [4, 8])
@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 9000])
@pytest.mark.parametrize("lost", ["none", "last", "never"])
def test_chunks(n, width, lost):
    L = hb.lib()
    L.hctr_ingest_keys_following.argtypes = [vp, ctypes.c_int, vp, sz, vp, u32, vp, sz, vp, vp, vp, u32, vp, u32, vp]
    dev, length, epoch = torch.device("cuda:0"), 70_000, 5
    rng = np.random.RandomState(n)
    keys = rng.randint(length, size=n)
    row_of = rng.permutation(length).astype(np.int32)
    dt = torch.int32 if width == 4 else torch.int64
    src = torch.zeros(n, dtype=dt).pin_memory()
    progress = torch.full((1,), (epoch - 1) << 32 | n).pin_memory()  # (an earlier call's)
    gave_up = torch.zeros(1, dtype=torch.int32).pin_memory()
    seen = torch.full((1,), (epoch - 1) << 32 | n, device=dev)
    dst = torch.full((n,), -7, dtype=torch.int64, device=dev)
    rows = torch.full((n,), -7, dtype=torch.int32, device=dev)
    meta = torch.full((9,), 3, dtype=torch.int32, device=dev)
    row_d = torch.from_numpy(row_of).to(dev)
    torch.cuda.synchronize()
    starts = list(range(0, n, CHUNK))
    # a chunk that is not coming in time ends the wait after a millisecond; the others get as long as they need
    limit = 1000 if lost == "never" else 1_000_000
    if lost == "never":  # (all but the last are there beforehand)
        src.copy_(torch.from_numpy(keys).to(dt))
        progress[0] = epoch << 32 | starts[-1]
    assert L.hctr_ingest_keys_following(src.data_ptr(), width, dst.data_ptr(), n, meta.data_ptr(), 9, row_d.data_ptr(),
                                        length, rows.data_ptr(), progress.data_ptr(), seen.data_ptr(), epoch,
                                        gave_up.data_ptr(), limit, None) == 0
    if lost != "never":
        for at in starts:
            part = slice(at, min(n, at + CHUNK))
            src[part] = torch.from_numpy(keys[part]).to(dt)
            progress[0] = epoch << 32 | (LOST if lost == "last" and at == starts[-1] else part.stop)
    torch.cuda.synchronize()
    assert int(gave_up[0]) == (1 if lost == "never" else 0)
    got, at = dst.cpu().numpy(), rows.cpu().numpy()
    for first in range(0, n, 1024):  # a block takes all of its keys or none
        block = slice(first, min(n, first + 1024))
        if got[block][0] != -7:
            assert np.array_equal(got[block], keys[block]) and np.array_equal(at[block], row_of[keys[block]])
        else:
            assert (got[block] == -7).all() and (at[block] == -7).all()
    there = int((got != -7).sum())
    if lost == "none":
        assert there == n
    elif lost == "never":
        assert there == starts[-1] // 1024 * 1024
    else:  # (a block that looks late finds that the rest is lost)
        assert there <= starts[-1]
    assert not bool(meta.any())


def test_the_limit_is_for_the_next_keys():
    """Twelve chunks, the last of them long after the limit has passed since the launch, but none of them late by itself."""
    L = hb.lib()
    L.hctr_ingest_keys_following.argtypes = [vp, ctypes.c_int, vp, sz, vp, u32, vp, sz, vp, vp, vp, u32, vp, u32, vp]
    dev, n, limit = torch.device("cuda:0"), 12 * 4096, 0.2
    keys = torch.arange(n)
    src, progress, gave_up = keys.int().pin_memory(), torch.zeros(1, dtype=torch.int64).pin_memory(), torch.zeros(1).int().pin_memory()
    seen, dst = torch.zeros(1, dtype=torch.int64, device=dev), torch.zeros(n, dtype=torch.int64, device=dev)
    rows, meta = torch.zeros(n, dtype=torch.int32, device=dev), torch.zeros(9, dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    assert L.hctr_ingest_keys_following(src.data_ptr(), 4, dst.data_ptr(), n, meta.data_ptr(), 9, None, n, rows.data_ptr(),
                                        progress.data_ptr(), seen.data_ptr(), 3, gave_up.data_ptr(), int(limit * 1e6), None) == 0
    for chunk in range(12):
        time.sleep(limit / 4)
        progress[0] = 3 << 32 | (chunk + 1) * 4096
    torch.cuda.synchronize()
    assert int(gave_up[0]) == 0 and torch.equal(dst.cpu(), keys) and torch.equal(rows.cpu(), keys.int())


def test_a_waiting_ingest_leaves_room_for_other_streams():
    """A kernel whose blocks need an empty SM (a tile of the grouping: 1024 threads) runs while the ingest of a batch that would
    fill every SM waits for its keys."""
    from test_gpu_group_keys import GroupArgs

    L = hb.lib()
    L.hctr_ingest_keys_following.argtypes = [vp, ctypes.c_int, vp, sz, vp, u32, vp, sz, vp, vp, vp, u32, vp, u32, vp]
    L.hctr_group_keys.argtypes = [ctypes.POINTER(GroupArgs), vp]
    dev, n, m, length = torch.device("cuda:0"), 1_300_000, 1000, 5000

    def z(count, dt=torch.int32):
        return torch.zeros(count, dtype=dt, device=dev)

    keys = torch.arange(n) % length
    src, progress, gave_up = keys.int().pin_memory(), torch.zeros(1, dtype=torch.int64).pin_memory(), torch.zeros(1).int().pin_memory()
    seen, dst, rows, meta = z(1, torch.int64), z(n, torch.int64), z(n), z(9)
    t = dict(keys=keys[:m].to(dev), owner_of=z(length, torch.uint8), pos_row=z(m), pairs0=z(m, torch.int64), pairs1=z(m, torch.int64),
             sort_keys=z(m), tile_counts=z(512 * 256), hist=z(2048), tile_flags=z(1024), chain_scratch=z(512), uniq=z(m, torch.int64),
             uniq_owner=z(m, torch.uint8), uniq_row=z(m), run_start=z(m + 1), sorted_pos=z(m), idx_map=z(m), chunk_key=z(m),
             heavy_list=z(m), meta=z(6))
    a = GroupArgs(batch=m, length=length, nrank=1, epoch=1, **{k: v.data_ptr() for k, v in t.items()})
    first, other = torch.cuda.Stream(), torch.cuda.Stream()
    assert L.hctr_group_keys(ctypes.byref(a), other.cuda_stream) == 0  # (loads the kernel)
    torch.cuda.synchronize()
    assert L.hctr_ingest_keys_following(src.data_ptr(), 4, dst.data_ptr(), n, meta.data_ptr(), 9, None, length, rows.data_ptr(),
                                        progress.data_ptr(), seen.data_ptr(), 3, gave_up.data_ptr(), 1_000_000,
                                        first.cuda_stream) == 0
    time.sleep(0.01)
    assert L.hctr_group_keys(ctypes.byref(a), other.cuda_stream) == 0
    done = other.record_event()
    until = time.time() + 0.3
    while not done.query() and time.time() < until:
        time.sleep(0.001)
    ran = done.query()
    progress[0] = 3 << 32 | n
    torch.cuda.synchronize()
    assert ran and int(gave_up[0]) == 0
    assert torch.equal(dst.cpu(), keys) and torch.equal(rows.cpu(), keys.int()) and int(t["meta"][0]) == m


def _steps(oracle_mod, sizes, bad=(), width=32):
    """Training and serving steps with pageable keys, against the oracle; a batch of `bad` has one key out of range.  Returns how
    the keys were ingested."""
    from test_gpu_parity import assert_state_parity, make_worlds

    N, W = 60_000, width
    rng = np.random.RandomState(3)
    gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.5, np.zeros(N, dtype=np.uint8), [rng.permutation(N)],
                         keys_on_device=False)
    before = None
    for s, n in enumerate(sizes):
        keys = [rng.randint(N, size=n)]
        if s in bad:
            broken = keys[0].copy()
            broken[n - 1 - n // 3] = N
            with pytest.raises(RuntimeError, match="outside"):
                gw.preprocess([broken])
            before = None
            gw.push_pull(None)
            continue
        gw.preprocess(keys)
        ow.preprocess(keys)
        grads = None if before is None or s % 4 == 3 else [rng.normal(0, 1, size=(before, W)).astype(np.float32)]
        got, want = gw.push_pull(grads), ow.push_pull(grads)
        assert np.array_equal(got[0], want[0]), s
        before = n
    counts = gw.tables[0].ingest_counts()
    assert_state_parity(gw, ow, exact=True)
    gw.close()
    return counts


SIZES = [40_000, 32_768, 32_767, 70_000, 45_057, 300, 50_000, 36_864, 140_001]


# No limit: the kernel gives up when it looks twice without a further chunk in between (2 us of copying), so it hardly ever keeps
# up; a second: it always does.
AT_ONCE, PATIENT = "0", "1000000"


@pytest.mark.parametrize("width,least", [(32, 32_768), (4, 65_536), (16, 49_152)])  # (3 MB of rows, else 65,536 keys)
def test_tables_keep_up(oracle_mod, monkeypatch, width, least):
    monkeypatch.setenv("HCTR_FOLLOW_LIMIT_US", PATIENT)
    sizes = SIZES + [least, least - 1]
    assert _steps(oracle_mod, sizes, width=width) == {"followed": sum(n >= least for n in sizes), "redone": 0, "not_started": 0}


def test_a_table_that_serves_does_not_follow(oracle_mod, monkeypatch):
    from test_gpu_parity import make_worlds

    monkeypatch.setenv("HCTR_FOLLOW_LIMIT_US", PATIENT)
    N, W, n = 60_000, 32, 40_000
    rng = np.random.RandomState(7)
    gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.5, np.zeros(N, dtype=np.uint8), [np.arange(N)], keys_on_device=False)
    followed = []
    for grads in (False, False, False, False, True, True):
        keys = [rng.randint(N, size=n)]
        gw.preprocess(keys)
        ow.preprocess(keys)
        grad = [rng.normal(0, 1, size=(n, W)).astype(np.float32)] if grads else None
        assert np.array_equal(gw.push_pull(grad)[0], ow.push_pull(grad)[0])
        followed.append(gw.tables[0].ingest_counts()["followed"])
    assert followed == [1, 2, 2, 2, 2, 3]  # (two pulls in a row are how it is told)
    gw.close()


def test_tables_give_up(oracle_mod, monkeypatch):
    monkeypatch.setenv("HCTR_FOLLOW_LIMIT_US", AT_ONCE)
    counts = _steps(oracle_mod, SIZES * 4)
    assert counts["redone"] >= 1
    # given up is not given up for good
    assert counts["followed"] + counts["not_started"] >= 4


def test_bad_key(oracle_mod):
    _steps(oracle_mod, SIZES + SIZES, bad=(3, 10))


@pytest.mark.parametrize("limit", [PATIENT, AT_ONCE])
def test_two_batches_in_a_row(oracle_mod, monkeypatch, limit):
    from test_gpu_parity import make_worlds

    monkeypatch.setenv("HCTR_FOLLOW_LIMIT_US", limit)
    N, W, redone = 60_000, 32, 0
    for seed in range(6):
        rng = np.random.RandomState(seed)
        gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.5, np.zeros(N, dtype=np.uint8), [np.arange(N)], keys_on_device=False)
        for n in (50_000, 80_000):
            keys = [rng.randint(N, size=n)]
            gw.preprocess(keys)
            ow.preprocess(keys)
        grad = [rng.normal(0, 1, size=(50_000, W)).astype(np.float32)]
        assert np.array_equal(gw.push_pull(grad)[0], ow.push_pull(grad)[0])
        redone += gw.tables[0].ingest_counts()["redone"]
        gw.close()
    assert (redone > 0) == (limit == AT_ONCE)


@pytest.mark.parametrize("limit", [PATIENT, AT_ONCE])
def test_gradients_and_rows_in_pinned_memory(oracle_mod, monkeypatch, limit):
    """The step that writes rows while gradients still come in reads the batch's rows earlier than the others."""
    from test_gpu_parity import make_worlds

    monkeypatch.setenv("HCTR_FOLLOW_LIMIT_US", limit)
    N, W, redone = 60_000, 32, 0
    for seed in range(6):
        rng = np.random.RandomState(seed)
        gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.5, np.zeros(N, dtype=np.uint8), [np.arange(N)], keys_on_device=False,
                             buffers="pinned")
        before = None
        for n in (20_000, 50_000):  # (only the second one is followed)
            keys = [rng.randint(N, size=n)]
            gw.preprocess(keys)
            ow.preprocess(keys)
            grad = None if before is None else [rng.normal(0, 1, size=(before, W)).astype(np.float32)]
            assert np.array_equal(gw.push_pull(grad)[0], ow.push_pull(grad)[0])
            before = n
        redone += gw.tables[0].ingest_counts()["redone"]
        gw.close()
    assert (redone > 0) == (limit == AT_ONCE)


def test_launches_that_wait_for_their_kernels():
    code = ("import sys; sys.path[:0] = [%r, %r]\n"
            "from oracle import build, hetu_oracle\n"
            "import test_gpu_following_ingest as t\n"
            "c = t._steps(hetu_oracle, t.SIZES * 3)\n"
            "assert c['followed'] == 0 and c['not_started'] >= 3, c\nprint('same')\n" % (ROOT, os.path.join(ROOT, "tests")))
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, CUDA_LAUNCH_BLOCKING="1"), cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
