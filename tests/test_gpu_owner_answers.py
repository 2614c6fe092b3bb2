"""What a rank asks the owners, and the owner's staleness test and row gather where the queries change their share per warp: fewer than a warp each, a
remainder, more than one round of 32, with the rank's own (unanswered) queries in front of, between and behind the others.
Oracle: numpy."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402
from hetuctr_b200.owner_replay import Box, Ctx, cnt_words  # noqa: E402

vp, sz, i64, u32 = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_longlong, ctypes.c_uint32
NEVER = np.iinfo(np.int64).min
WARPS = 148 * 32


@pytest.mark.parametrize("rank", [0, 1, 2])
@pytest.mark.parametrize("width", [3, 32, 132])
@pytest.mark.parametrize("counts", [(0, 0, 0), (1, 5, 0), (700, 40, 301), (WARPS * 4 + 1, 9, WARPS), (40, WARPS * 20, WARPS * 14)])
def test_queries(counts, width, rank):
    L = hb.lib()
    L.hctr_p2p_stale_gather.argtypes = [vp, u32, vp, sz, sz, vp, vp, i64, vp]
    dev, n, rows, cached, bound = torch.device("cuda:0"), 3, 5000, 100, 2
    rng = np.random.RandomState(width + rank)
    cap = max(max(counts), 1)
    length = rows
    row_of = rng.permutation(rows).astype(np.int32)
    owned = np.flatnonzero(row_of >= cached)
    emb = torch.randn((rows, width), device=dev)
    version = rng.randint(0, 9, size=rows)

    def z(m, dt, v=0):
        return torch.full((m,), v, dtype=dt, device=dev)

    boxes = [dict(hdr=z(n * 16, torch.int32), qkey=z(n * cap, torch.int64), qver=z(n * cap, torch.int64),
                  pkey=z(n * cap, torch.int64), pupd=z(n * cap, torch.int64), pval=z(n, torch.float32),
                  flag=z(n * cap, torch.uint8, 0), rver=z(n * cap, torch.int64, -1),
                  rval=torch.full((n * cap, width), float("nan"), device=dev)) for _ in range(n)]
    keys = [rng.choice(owned, size=c) for c in counts]
    vers = [np.where(rng.rand(c) < 0.2, NEVER, rng.randint(0, 9, size=c)) for c in counts]
    for s in range(n):
        boxes[rank]["qkey"][s * cap:s * cap + counts[s]] = torch.from_numpy(keys[s]).to(dev)
        boxes[rank]["qver"][s * cap:s * cap + counts[s]] = torch.from_numpy(vers[s]).to(dev)
    names = [f[0] for f in Box._fields_]
    raw = np.array([[b[k].data_ptr() for k in names] for b in boxes], dtype=np.uint64)
    box_d = torch.from_numpy(raw.view(np.int64)).to(dev)
    cnt = np.zeros(cnt_words(n), dtype=np.int32)
    cnt[:n] = counts
    cnt[3 * n:4 * n + 1] = np.concatenate([[0], np.cumsum(counts)])
    cnt_d, err = torch.from_numpy(cnt).to(dev), z(1, torch.int32)
    ver_d, row_d = torch.from_numpy(version).to(dev), torch.from_numpy(row_of).to(dev)
    c = Ctx(nrank=n, rank=rank, cap=cap, width=width, box=box_d.data_ptr(), cnt_in=cnt_d.data_ptr(), err=err.data_ptr(),
            timeout_ns=10 ** 9)
    torch.cuda.synchronize()
    assert L.hctr_p2p_stale_gather(ctypes.byref(c), 7, row_d.data_ptr(), length, cached, emb.data_ptr(),
                                   ver_d.data_ptr(), bound, None) == 0
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    e = emb.cpu().numpy()
    for s in range(n):
        b, m = boxes[s], counts[s]
        flag = b["flag"].cpu().numpy()[rank * cap:rank * cap + m]
        rval = b["rval"].cpu().numpy()[rank * cap:rank * cap + m]
        rver = b["rver"].cpu().numpy()[rank * cap:rank * cap + m]
        at = row_of[keys[s]]
        stale = (vers[s] == NEVER) | (vers[s] + bound < version[at])
        if s == rank:
            stale[:] = False
        assert np.array_equal(flag, stale.astype(np.uint8))
        assert np.array_equal(rval[stale], e[at[stale]]) and np.isnan(rval[~stale]).all()
        assert np.array_equal(rver[stale], version[at[stale]]) and (rver[~stale] == -1).all()
        assert int(b["hdr"][rank * 16 + 8]) == 7


@pytest.mark.parametrize("lost", [False, True])
def test_queries_of_a_rank(lost):
    """Own keys are counted and not written; one that is not stored here is reported, as its owner would."""
    L = hb.lib()
    L.hctr_p2p_query_send.argtypes = [vp, vp, sz, vp, vp, vp, vp, u32, vp, vp]
    dev, n, rank, cap, rows = torch.device("cuda:0"), 3, 1, 2000, 4000
    rng = np.random.RandomState(4)
    counts = [700, 1100, 1]
    seg, U = np.r_[0, np.cumsum(counts)], sum(counts)
    owner = np.repeat(np.arange(n), counts)
    uniq, version = rng.permutation(100_000)[:U], rng.randint(0, 99, size=rows)
    row = rng.permutation(rows)[:U]
    row[(owner != rank) & (rng.rand(U) < 0.5)] = -1
    if lost:
        row[seg[rank] + 1050] = -1
    put = lambda a, dt: torch.from_numpy(np.ascontiguousarray(a).astype(dt)).to(dev)  # noqa: E731
    boxes = [dict(hdr=torch.zeros(n * 16, dtype=torch.int32, device=dev), qkey=torch.full((n * cap,), -5, device=dev),
                  qver=torch.full((n * cap,), -5, device=dev)) for _ in range(n)]
    raw = np.array([[b[k].data_ptr() if k in b else 0 for k, _ in Box._fields_] for b in boxes], dtype=np.uint64)
    box_d, cnt, err = torch.from_numpy(raw.view(np.int64)).to(dev), put(np.zeros(cnt_words(n)), np.int32), put([0], np.int32)
    meta = put(np.r_[U, 0, 0, 0, seg], np.int32)
    d = [put(uniq, np.int64), put(owner, np.uint8), put(row, np.int32), put(version, np.int64)]
    c = Ctx(nrank=n, rank=rank, cap=cap, width=4, box=box_d.data_ptr(), cnt_in=cnt.data_ptr(), err=err.data_ptr(),
            timeout_ns=10 ** 9)
    assert L.hctr_p2p_query_send(ctypes.byref(c), meta.data_ptr(), U, *[t.data_ptr() for t in d], 9, None, None) == 0
    torch.cuda.synchronize()
    assert int(err[0]) == (2 if lost else 0)  # HCTR_ERR_NOT_OWNER
    for p, b in enumerate(boxes):
        hdr = b["hdr"].cpu().numpy()[rank * 16:]
        assert (hdr[0], hdr[1], hdr[2]) == (9, counts[p], 0)
        key, ver = (b[k].cpu().numpy() for k in ("qkey", "qver"))
        at = slice(rank * cap, rank * cap + counts[p])
        if p != rank:
            mine = slice(seg[p], seg[p + 1])
            assert np.array_equal(key[at], uniq[mine])
            assert np.array_equal(ver[at], np.where(row[mine] >= 0, version[row[mine]], NEVER))
            key[at] = ver[at] = -5
        assert (key == -5).all() and (ver == -5).all()
