"""The reduction of tables with peers through the C-ABI: long runs around a stage of rows, a chunk of positions and the ring, with
each size of stage (the GPU to itself or shared, beside the short runs or on one stream).  Oracle: numpy, sums in batch order,
bit-exact."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import hetuctr_b200 as hb  # noqa: E402

vp, sz = ctypes.c_void_p, ctypes.c_size_t


class Args(ctypes.Structure):
    _fields_ = [("n_unique", sz), ("width", sz), ("n_cached", sz), ("neg_lr", ctypes.c_float), ("grad", vp), ("run_start", vp),
                ("sorted_pos", vp), ("heavy_list", vp), ("n_heavy", sz), ("uniq", vp), ("uniq_row", vp), ("need_push", vp),
                ("push_slot", vp), ("embedding", vp), ("version", vp), ("pending", vp), ("pending_cnt", vp), ("push_key", vp),
                ("push_updates", vp), ("push_val", vp), ("work_counter", vp), ("p2p", vp), ("uniq_owner", vp),
                ("push_base", vp), ("side_stream", vp), ("fork_event", vp), ("join_event", vp)]


@pytest.mark.parametrize("forked,shared", [(True, 0), (True, 1), (False, 0), (False, 1)])
@pytest.mark.parametrize("width", [3, 64, 127, 128, 132, 256, 512, 1100])
def test_stage_sizes(width, forked, shared):
    L = hb.lib()
    reduce = L.hctr_grad_reduce_apply_pack_shared if shared else L.hctr_grad_reduce_apply_pack
    reduce.argtypes = [vp, vp]
    rng = np.random.RandomState(width)
    dev, rows = torch.device("cuda:0"), 400
    fits = {max(1, s // (4 * width)) for s in (8192, 16384, 32768)}  # rows of a stage
    lens = [1, 32, 33, 255, 256, 2047, 2048, 2049] + [n * k + d for n in fits for k in (1, 3, 4) for d in (-1, 0, 1)]
    lens = np.array([x for x in lens if 0 < x < 3000] + [34] * 150)  # (more long runs than there are blocks)
    U, B = len(lens), int(lens.sum())
    run = np.r_[0, np.cumsum(lens)]
    pos = np.concatenate([np.sort(p) for p in np.split(rng.permutation(B), run[1:-1])])
    uniq = rng.permutation(rows)[:U].astype(np.int64)
    pushed = rng.rand(U) < 0.5
    urow = np.where(pushed, -1, uniq)
    slot = np.r_[0, np.cumsum(pushed)]
    heavy = rng.permutation(np.flatnonzero(lens > 32))
    grad, emb = rng.normal(size=(B, width)).astype(np.float32), rng.normal(size=(rows, width)).astype(np.float32)

    def t(x, dt=None):
        return torch.from_numpy(np.ascontiguousarray(x if dt is None else x.astype(dt))).to(dev)

    d = dict(grad=t(grad), run_start=t(run, np.int32), sorted_pos=t(pos, np.int32), heavy_list=t(heavy, np.int32), uniq=t(uniq),
             uniq_row=t(urow, np.int32), need_push=t(pushed, np.int32), push_slot=t(slot, np.int32), embedding=t(emb),
             version=torch.zeros(rows, dtype=torch.int64, device=dev), pending=torch.zeros(4, device=dev),
             pending_cnt=torch.zeros(4, dtype=torch.int64, device=dev),
             push_key=torch.full((U,), -1, dtype=torch.int64, device=dev),
             push_updates=torch.zeros(U, dtype=torch.int64, device=dev), push_val=torch.zeros((U, width), device=dev),
             work_counter=torch.zeros(2, dtype=torch.int32, device=dev), uniq_owner=t(pushed, np.uint8),
             push_base=torch.zeros(2, dtype=torch.int32, device=dev))
    s, side, ev = torch.cuda.Stream(), torch.cuda.Stream(), [torch.cuda.Event() for _ in range(2)]
    for e in ev:
        e.record(s)
    torch.cuda.synchronize()
    a = Args(n_unique=U, width=width, neg_lr=-0.25, n_heavy=len(heavy), **{k: v.data_ptr() for k, v in d.items()})
    if forked:
        a.side_stream, a.fork_event, a.join_event = side.cuda_stream, ev[0].cuda_event, ev[1].cuda_event
    assert reduce(ctypes.byref(a), s.cuda_stream) == 0
    torch.cuda.synchronize()
    sums = np.zeros((U, width), np.float32)
    for u in range(U):
        for p in pos[run[u]:run[u + 1]]:
            sums[u] += grad[p]
    sums *= np.float32(-0.25)
    mine = ~pushed
    want, ver = emb.copy(), np.zeros(rows, np.int64)
    want[uniq[mine]] += sums[mine]
    ver[uniq[mine]] = lens[mine]
    assert np.array_equal(d["embedding"].cpu().numpy(), want)
    assert np.array_equal(d["version"].cpu().numpy(), ver)
    n = int(pushed.sum())
    assert np.array_equal(d["push_val"].cpu().numpy()[:n], sums[pushed])
    assert np.array_equal(d["push_key"].cpu().numpy()[:n], uniq[pushed])
    assert np.array_equal(d["push_updates"].cpu().numpy()[:n], lens[pushed])
