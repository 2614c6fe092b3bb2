"""hctr_group_keys (stable radix grouping of a batch) on caller-owned buffers against numpy, at the sizes where it
changes: inside one tile, full tiles, the last batch of the one-launch form and the first of the multi-launch form,
with runs around the list thresholds, one key filling the batch, and keys out of range."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402

vp, sz, u32 = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_uint32
LIGHT, LONG, CHUNK, TILES = 32, 256, 32, 256


class GroupArgs(ctypes.Structure):  # field order of hctr_group_args
    _fields_ = [("keys", vp), ("batch", sz), ("length", sz), ("nrank", ctypes.c_int), ("owner_of", vp),
                ("pos_row", vp), ("pairs0", vp), ("pairs1", vp), ("sort_keys", vp), ("tile_counts", vp), ("hist", vp),
                ("tile_flags", vp), ("chain_scratch", vp), ("epoch", u32), ("uniq", vp), ("uniq_owner", vp),
                ("uniq_row", vp), ("run_start", vp), ("sorted_pos", vp), ("idx_map", vp), ("chunk_key", vp),
                ("heavy_list", vp), ("meta", vp)]


@pytest.mark.parametrize("length,nrank", [(200, 1), (70_000, 3), (1 << 22, 1), (40_000_000, 5)])
@pytest.mark.parametrize("batch", [0, 1, 31, 33, 8193, 16_385, 32_769, 65_536, 65_537, 114_689, 200_001])
def test_grouping_matches_numpy(batch, length, nrank):
    L = hb.lib()
    L.hctr_group_keys.argtypes = [ctypes.POINTER(GroupArgs), vp]
    L.hctr_group_index_map.argtypes = [vp, vp, vp, vp, vp]
    L.hctr_group_fits.argtypes = [sz, sz, ctypes.c_int]
    assert L.hctr_group_fits(batch, length, nrank) == 1
    dev = torch.device("cuda:0")
    rng = np.random.RandomState(batch % 1000 + nrank)
    owner = rng.randint(nrank, size=length).astype(np.uint8)

    def z(n, dt):
        return torch.zeros(max(int(n), 1), dtype=dt, device=dev)

    cap = batch // CHUNK + 2
    t = dict(owner_of=torch.from_numpy(owner).to(dev), pairs0=z(batch, torch.int64), pairs1=z(batch, torch.int64),
             sort_keys=z(batch, torch.int32), tile_counts=z(512 * TILES, torch.int32), hist=z(2048, torch.int32),
             tile_flags=z(4 * TILES, torch.int32), chain_scratch=z(2 * TILES, torch.int32), uniq=z(batch, torch.int64),
             uniq_owner=z(batch, torch.uint8), uniq_row=z(batch, torch.int32), run_start=z(batch + 1, torch.int32),
             sorted_pos=z(batch, torch.int32), idx_map=z(batch, torch.int32), chunk_key=z(cap, torch.int32),
             heavy_list=z(cap, torch.int32), meta=z(4 + nrank + 1, torch.int32))
    for epoch, kind in enumerate(("skewed", "uniform", "one key", "invalid keys"), 1):
        keys = (rng.zipf(1.2, size=batch) - 1 + rng.randint(length)) % length
        if kind == "uniform":
            keys = rng.randint(length, size=batch)
        elif kind == "one key":
            keys[:] = length - 1
        for run, key in ((32, 3), (33, 4), (256, 5), (257, 6)):  # runs around the two list thresholds
            if kind == "uniform" and batch >= 8191:
                keys[keys == key] = 7
                keys[rng.choice(np.flatnonzero(keys > 7), run, replace=False)] = key
        bad = np.zeros(batch, dtype=bool)
        if kind == "invalid keys" and batch:
            bad = rng.rand(batch) < 0.3
            keys[bad] = rng.choice([-1, length, 1 << 40], size=int(bad.sum()))
        pos_row = rng.randint(1 << 30, size=batch).astype(np.int32)
        if batch:  # equal keys have equal rows
            _, first, inv = np.unique(keys, return_index=True, return_inverse=True)
            pos_row = pos_row[first][inv].astype(np.int32)
        kd, pd = torch.from_numpy(keys.astype(np.int64)).to(dev), torch.from_numpy(pos_row).to(dev)
        t["meta"].zero_()
        a = GroupArgs(keys=kd.data_ptr(), pos_row=pd.data_ptr(), batch=batch, length=length, nrank=nrank, epoch=epoch,
                      **{k: v.data_ptr() for k, v in t.items()})
        assert L.hctr_group_keys(ctypes.byref(a), None) == 0
        torch.cuda.synchronize()
        h = {k: v.cpu().numpy() for k, v in t.items()}
        good = np.flatnonzero(~bad)
        uk = np.unique(keys[good])
        uk = uk[np.lexsort((uk, owner[uk]))]
        U, meta = len(uk), h["meta"]
        assert meta[0] == U and meta[1] == (1 if bad.any() else 0)
        assert np.array_equal(h["uniq"][:U], uk)
        if nrank > 1:
            assert np.array_equal(h["uniq_owner"][:U], owner[uk])
        assert np.array_equal(meta[4:4 + nrank + 1], np.searchsorted(owner[uk], np.arange(nrank + 1)))
        place = {int(k): i for i, k in enumerate(uk)}
        idx = np.array([place[int(k)] for k in keys[good]], dtype=np.int64)
        exp_map = np.full(batch, -1, dtype=np.int64)
        exp_map[good] = idx
        assert np.array_equal(h["idx_map"][:batch], exp_map)
        pos = good[np.argsort(idx, kind="stable")]
        assert np.array_equal(h["sorted_pos"][:len(good)], pos)
        runs = np.concatenate([[0], np.cumsum(np.bincount(idx, minlength=U))]).astype(np.int64)
        assert np.array_equal(h["run_start"][:U + 1], runs)
        assert np.array_equal(h["uniq_row"][:U], pos_row[pos[runs[:-1]]])
        chunks = (len(good) + CHUNK - 1) // CHUNK
        exp_chunk = np.searchsorted(runs[:-1], np.arange(chunks + 1) * CHUNK)
        exp_chunk[chunks] = U
        assert np.array_equal(h["chunk_key"][:chunks + 1], exp_chunk)
        long_, very = np.flatnonzero(np.diff(runs) > LIGHT), np.flatnonzero(np.diff(runs) > LONG)
        assert meta[2] == len(long_) and meta[3] == len(very)
        assert np.array_equal(np.sort(h["heavy_list"][:len(long_)]), long_)
        back = h["heavy_list"][batch // 32 + 2 - len(very):batch // 32 + 2]
        assert np.array_equal(np.sort(back), very)
        if not bad.any():
            t["idx_map"].fill_(-7)
            assert L.hctr_group_index_map(t["meta"].data_ptr(), t["run_start"].data_ptr(), t["sorted_pos"].data_ptr(),
                                          t["idx_map"].data_ptr(), None) == 0
            torch.cuda.synchronize()
            assert np.array_equal(t["idx_map"].cpu().numpy()[:batch], exp_map)
        assert int(t["hist"].abs().sum()) == 0


def test_batch_beyond_the_grouping_limit(oracle_mod):
    # more keys than hctr_group_keys serves: the bitmap ranking makes the runs, hctr_run_chunks what the reduction needs
    from test_gpu_parity import make_worlds, run_steps

    N, W, B = 50_000, 2, 8192 * TILES + 5
    gw, ow = make_worlds(oracle_mod, 1, N, W, 0, 0, 0.5, np.zeros(N, dtype=np.uint8), [np.arange(N)])
    rng = np.random.RandomState(9)
    keys = rng.randint(N, size=B)
    keys[rng.rand(B) < 0.02] = 77
    grads = [None, [rng.normal(0, 1, size=(B, W)).astype(np.float32)]]
    run_steps(gw, ow, [[keys], [rng.randint(N, size=1000)]], grads)
    gw.close()


@pytest.mark.parametrize("width", [1, 2, 6, 12, 31, 32, 33, 60, 64, 66, 128, 130, 200, 516, 1030])
def test_reduction_run_lengths(oracle_mod, width):
    # runs on both sides of every limit of the reduction (short / long / very long, tiles of its rings), keys seen
    # once between them, at widths of every element size and number of lanes
    from test_gpu_parity import make_worlds, run_steps

    N = 3000
    gw, ow = make_worlds(oracle_mod, 1, N, width, 0, 0, 0.5, np.zeros(N, dtype=np.uint8),
                         [np.random.RandomState(4).permutation(N)])
    rng = np.random.RandomState(width)
    runs = [1, 2, 3, 4, 5, 31, 32, 33, 39, 40, 41, 63, 64, 65, 96, 255, 256, 257, 383, 384, 385, 511, 512, 640, 1300]
    key = np.repeat(rng.permutation(N)[:len(runs)], runs)
    b0 = np.concatenate([key, rng.randint(N, size=900)])
    rng.shuffle(b0)
    b1 = np.full(300, 11)
    batches = [[b0], [b1], [np.arange(N)]]
    grads = [None] + [[rng.normal(0, 1, size=(len(b[0]), width)).astype(np.float32)] for b in batches[:-1]]
    run_steps(gw, ow, batches, grads)
    gw.close()


@pytest.mark.parametrize("width,scale", [(300, 1), (258, 1), (301, 1), (64, 4)])
def test_host_gradients_in_pieces(oracle_mod, width, scale):
    # gradients in pinned host memory, large enough to come in several pieces: short, long and very long runs that end
    # in each piece, keys that span the pieces, and keys the batch before did not contain
    from test_gpu_parity import make_worlds, run_steps

    N = 9000 * scale
    gw, ow = make_worlds(oracle_mod, 1, N, width, 0, 0, 0.1, np.zeros(N, dtype=np.uint8), [np.arange(N)],
                         buffers="pinned", keys_on_device=False)
    rng = np.random.RandomState(width)
    runs = [1] * 800 * scale + [2, 3, 31, 32, 33, 64, 65, 255, 256, 257, 700]

    def batch():
        ids, parts = rng.permutation(N), []
        for i in range(4):  # a part of the batch with keys of its own
            part = np.repeat(ids[i * len(runs):(i + 1) * len(runs)], runs)
            parts.append(rng.permutation(np.concatenate([part, ids[-40:]])))
        return np.concatenate(parts)

    batches = [[batch()] for _ in range(3)] + [[np.arange(N)]]
    grads = [None] + [[rng.normal(0, 1, size=(len(b[0]), width)).astype(np.float32)] for b in batches[:-1]]
    run_steps(gw, ow, batches, grads)
    gw.close()


@pytest.mark.parametrize("width", [1, 3, 4, 6, 10, 12, 50, 64, 100, 128, 132, 258])
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 37, 4097, 60_001])
def test_expand_local(batch, width):
    L = hb.lib()
    L.hctr_expand_rows_local.argtypes = [sz, sz, vp, vp, vp, vp]
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev)
    g.manual_seed(batch + width)
    emb = torch.randn((3000, width), generator=g, device=dev)
    rows = torch.randint(3000, (batch,), generator=g, device=dev, dtype=torch.int32)
    rows[batch // 2] = -1  # no row: zeros
    guard = torch.full((batch + 1, width), float("nan"), device=dev)
    for dst in (guard[:batch], guard.reshape(-1)[1:1 + batch * width].reshape(batch, width)):  # the second misaligned
        guard.fill_(float("nan"))
        assert L.hctr_expand_rows_local(batch, width, rows.data_ptr(), emb.data_ptr(), dst.data_ptr(), None) == 0
        torch.cuda.synchronize()
        want = emb[rows.clamp(min=0).long()]
        want[batch // 2] = 0
        assert torch.equal(dst, want)
        assert int(torch.isnan(guard).sum()) == width
