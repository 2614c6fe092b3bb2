"""A grouping whose bounded wait ran out (HCTR_ERR_TIMEOUT in the batch's meta words) leaves a batch without keys behind:
whatever it did not write is neither looked at nor passed on, and nobody downstream updates, sends or lists anything.
No wait runs out here: the error bit is set beforehand, and the buffers hold numbers that would be out of range."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402
from test_gpu_group_keys import CHUNK, TILES, GroupArgs  # noqa: E402

vp, sz, u32 = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_uint32
TIMEOUT = 8


class LocalReduceArgs(ctypes.Structure):  # field order of hctr_local_reduce_args
    _fields_ = [("batch", sz), ("width", sz), ("neg_lr", ctypes.c_float), ("grad", vp), ("run_start", vp),
                ("sorted_pos", vp), ("chunk_key", vp), ("heavy_list", vp), ("uniq_row", vp), ("meta", vp),
                ("embedding", vp), ("version", vp), ("err", vp)]


def _group(L, dev, batch, length, nrank, broken):
    """Arrays of a grouping of random keys; `broken` sets the error bit before the launches."""
    rng = np.random.RandomState(batch % 1000 + nrank)

    def full(n, dt, v=-1):
        return torch.full((max(int(n), 1),), v, dtype=dt, device=dev)

    i64, i32 = torch.int64, torch.int32
    keys = torch.from_numpy((rng.zipf(1.2, size=batch) - 1) % length).to(dev)
    t = dict(owner_of=torch.from_numpy(rng.randint(nrank, size=length).astype(np.uint8)).to(dev),
             pairs0=full(batch, i64), pairs1=full(batch, i64), sort_keys=full(batch, i32),
             tile_counts=full(512 * TILES, i32), hist=full(2048, i32, 0), tile_flags=full(4 * TILES, i32, 0),
             chain_scratch=full(2 * TILES, i32, 0), uniq=full(batch, i64), uniq_owner=full(batch, torch.uint8, 0),
             uniq_row=full(batch, i32), run_start=full(batch + 1, i32), sorted_pos=full(batch, i32),
             idx_map=full(batch, i32, -7), chunk_key=full(batch // CHUNK + 2, i32), heavy_list=full(batch // CHUNK + 2, i32),
             meta=full(4 + nrank + 1, i32, 0))
    if broken:
        t["meta"][1] = TIMEOUT
    rows = keys.to(i32)
    a = GroupArgs(keys=keys.data_ptr(), pos_row=rows.data_ptr(), batch=batch, length=length, nrank=nrank, epoch=1,
                  **{k: v.data_ptr() for k, v in t.items()})
    assert L.hctr_group_keys(ctypes.byref(a), None) == 0
    torch.cuda.synchronize()
    return keys, t


@pytest.mark.parametrize("nrank", [1, 3])
@pytest.mark.parametrize("batch", [65_537, 200_001, 500_003, 950_001])  # 1, 2, 8 and 8 pairs per thread, several launches
def test_broken_passes_leave_a_batch_without_keys(batch, nrank):
    L = hb.lib()
    L.hctr_group_keys.argtypes = [ctypes.POINTER(GroupArgs), vp]
    dev = torch.device("cuda:0")
    _, t = _group(L, dev, batch, 70_000, nrank, broken=True)
    meta = t["meta"].cpu().numpy()
    assert meta[1] == TIMEOUT and not meta[[0, 2, 3]].any() and not meta[4:].any()
    assert int(t["run_start"][0]) == 0 and int(t["chunk_key"][0]) == 0
    assert bool((t["idx_map"] == -1).all())
    pos = t["sorted_pos"]
    assert int(pos.min()) >= 0 and int(pos.max()) < batch
    assert int(t["hist"].abs().sum()) == 0  # at rest for the next batch


@pytest.mark.parametrize("width", [1, 6, 64, 128])
def test_reduction_of_a_broken_batch_updates_nothing_and_says_so(width):
    L = hb.lib()
    L.hctr_group_keys.argtypes = [ctypes.POINTER(GroupArgs), vp]
    L.hctr_grad_reduce_local.argtypes = [ctypes.POINTER(LocalReduceArgs), vp]
    L.hctr_grad_reduce_window.argtypes = [ctypes.POINTER(LocalReduceArgs), u32, u32, vp]
    dev = torch.device("cuda:0")
    batch, length = 3000, 2000
    _, t = _group(L, dev, batch, length, 1, broken=False)
    grad = torch.ones((batch, width), device=dev)
    emb, version = torch.zeros((length, width), device=dev), torch.zeros(length, dtype=torch.int64, device=dev)
    err = torch.zeros(1, dtype=torch.int32, device=dev)
    names = ("run_start", "sorted_pos", "chunk_key", "heavy_list", "uniq_row", "meta")
    a = LocalReduceArgs(batch=batch, width=width, neg_lr=-1.0, grad=grad.data_ptr(), embedding=emb.data_ptr(),
                        version=version.data_ptr(), err=err.data_ptr(), **{k: t[k].data_ptr() for k in names})
    t["meta"][1] = TIMEOUT  # as a wait of group_finish leaves it: everything else in place
    for call in (lambda: L.hctr_grad_reduce_local(ctypes.byref(a), None),
                 lambda: L.hctr_grad_reduce_window(ctypes.byref(a), 0, batch, None)):
        err.zero_()
        torch.cuda.synchronize()
        assert call() == 0
        torch.cuda.synchronize()
        assert int(err[0]) == TIMEOUT
        assert not bool(emb.any()) and not bool(version.any())
    t["meta"][1] = 0
    err.zero_()
    torch.cuda.synchronize()
    assert L.hctr_grad_reduce_local(ctypes.byref(a), None) == 0
    torch.cuda.synchronize()
    assert int(err[0]) == 0 and int(version.sum()) == batch and float(emb.sum()) == -batch * width


def test_readers_of_a_broken_batch_find_no_keys():
    L = hb.lib()
    L.hctr_group_keys.argtypes = [ctypes.POINTER(GroupArgs), vp]
    L.hctr_group_index_map.argtypes = [vp, vp, vp, vp, vp]
    L.hctr_run_chunks.argtypes = [sz, vp, vp, vp, vp, vp]
    L.hctr_last_seen.argtypes = [sz, vp, vp, vp, vp, vp, vp, vp]
    L.hctr_pack_counts.argtypes = [vp, vp, ctypes.c_int, vp, vp]
    dev = torch.device("cuda:0")
    batch, nrank = 3000, 3
    keys, t = _group(L, dev, batch, 2000, nrank, broken=False)
    t["meta"][1] = TIMEOUT
    p = {k: v.data_ptr() for k, v in t.items()}
    t["idx_map"].fill_(-7)
    t["chunk_key"].fill_(-1)
    seen = torch.zeros(batch, dtype=torch.int32, device=dev)
    counts = torch.full((2 * nrank,), -1, dtype=torch.int32, device=dev)
    torch.cuda.synchronize()
    assert L.hctr_group_index_map(p["meta"], p["run_start"], p["sorted_pos"], p["idx_map"], None) == 0
    assert L.hctr_run_chunks(batch, p["run_start"], p["chunk_key"], p["heavy_list"], p["meta"], None) == 0
    assert L.hctr_last_seen(batch, keys.data_ptr(), p["uniq"], p["meta"], p["run_start"], p["sorted_pos"],
                            seen.data_ptr(), None) == 0
    assert L.hctr_pack_counts(p["meta"], None, nrank, counts.data_ptr(), None) == 0
    torch.cuda.synchronize()
    assert bool((t["idx_map"] == -7).all()) and bool((t["chunk_key"] == -1).all())
    assert bool((seen == -1).all())  # HCTR_NEVER
    assert not bool(counts.any())
