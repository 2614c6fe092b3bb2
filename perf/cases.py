"""Timing cases of the embedding table: one step of a training or serving loop, through the public `hetuCTR` module
(single-rank tables) and `hetuctr_b200.Table` (ranks that share this process).

A pass is what a user's program does for one batch: `preprocess(keys)` and `push_pull(gradients of the batch before,
rows of this one)`; serving passes no gradients.  Every state alternates between two batches, so that a pass pulls rows
the passes before it have updated.  Shapes are those of `hetuctr_b200.workloads.CONFIGS`, of the tests and of the
benchmark; keys are drawn per field from a bounded power law over a geometric vocabulary split, or uniformly.
"""
import itertools
import math
import os
import threading

import numpy as np
import torch

import hetuctr_b200
from hetuctr_b200.workloads import CONFIGS, field_vocab

_job = itertools.count(20001)  # thread ranks of one job find each other by this number
_PRIME = 2147483647  # larger than any vocabulary: rank * _PRIME mod v is a bijection of [0, v)


def _case(name, rows, width, samples, fields, alpha, train=True, keys="device", buffers="device", nrank=1, cache=0.0,
          pull=0, push=0, lr=0.01):
    return dict(name=name, rows=rows, width=width, samples=samples, fields=fields, alpha=alpha, train=train, keys=keys,
                buffers=buffers, nrank=nrank, cache=cache, pull=pull, push=push, lr=lr)


def listed():
    c1, c2, c4 = CONFIGS["cfg1_plumbing"], CONFIGS["cfg2_hybrid"], CONFIGS["cfg4_stress"]
    c3, c5 = CONFIGS["cfg3_large"], CONFIGS["cfg5_sweep"]
    return [
        # one request of an online ranking service: a single sample's keys, straight from the request handler
        _case("serve_1x26_w16", c1["rows"], 16, 1, 26, 0.0, train=False, keys="host"),
        # offline scoring / evaluation over a full-size batch
        _case("serve_8192x26_w128", c2["rows"], 128, 8192, 26, c2["alpha"], train=False),
        # a small model: few samples, a row width that is no multiple of four
        _case("train_333x17_w50", 1_200_000, 50, 333, 17, 1.1),
        # config 1, keys from a host array as the reference's driver script passes them
        _case("train_1024x26_w16", c1["rows"], c1["width"], c1["samples"], 26, 0.0, keys="host", lr=c1["lr"]),
        # the reference benchmark's default step: 2048 samples, rows of 128, host keys
        _case("train_2048x26_w128", c2["rows"], 128, 2048, 26, c2["alpha"], keys="host"),
        # config 2 on one GPU: the headline step
        _case("train_8192x26_w128", c2["rows"], 128, 8192, 26, c2["alpha"]),
        # config 5's shape on a quarter of its table: wide rows
        _case("train_4096x26_w256", c5["rows"] // 4, 256, c5["samples"], 26, c5["alpha"]),
        # one GPU's eighth of config 3: many fields, very hot keys
        _case("train_16384x39_w64", c3["rows"] // 8, 64, c3["samples"], 39, c3["alpha"]),
        # config 4: narrow rows, keys almost all distinct
        _case("train_32768x26_w32", c4["rows"], 32, c4["samples"], 26, 0.0, lr=c4["lr"]),
        # a trainer whose model runs elsewhere: keys, gradients and rows in pinned host memory
        _case("train_host_2048x26_w128", 4_000_000, 128, 2048, 26, c2["alpha"], keys="pinned", buffers="pinned"),
        # two ranks of a job with a cache of non-owned rows kept exact (thread ranks sharing this GPU)
        _case("ranks2_2048x26_w128", 4_000_000, 128, 2048, 26, c2["alpha"], nrank=2, cache=0.1),
        # the same with bounded staleness and keys almost all distinct
        _case("ranks2_8192x26_w32", 10_000_000, 32, 8192, 26, 0.0, nrank=2, cache=0.05, pull=10, push=10, lr=0.05),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train"] * 6 + ["serve"] * 3 + ["host"] + ["ranks"] * 2)
    width = _log(rng, 4, 512)
    if rng.random() < 0.7:
        width = max(4, width // 4 * 4)
    fields = rng.randint(1, 39)
    # keys and elements of a batch stay within the largest listed step of the same kind
    most_keys, most_elems = {"host": (53_248, 53_248 * 128), "ranks": (212_992, 53_248 * 128)}.get(kind, (638_976, 8192 * 26 * 128))
    most = max(1, min(16384, most_keys // fields, most_elems // (fields * width)))
    samples = _log(rng, 1, most)
    rows = _log(rng, 10_000, min(33_762_577 if kind in ("train", "serve") else 10_000_000, 12_000_000_000 // (4 * width)))
    rows = max(rows, 40)
    alpha = 0.0 if rng.random() < 0.3 else round(rng.uniform(1.02, 1.3), 3)
    ranks = kind == "ranks"
    stale = rng.choice([0, 0, 2, 10]) if ranks else 0
    c = _case("", rows, width, samples, fields, alpha, train=kind != "serve",
              keys="pinned" if kind == "host" else rng.choice(["host", "device", "device"]),
              buffers="pinned" if kind == "host" else "device", nrank=2 if ranks else 1,
              cache=round(rng.uniform(0.02, 0.3), 3) if ranks else 0.0, pull=stale, push=stale, lr=0.01)
    del c["name"]
    return c


def _keys(case, gen):
    """One sample-major batch of int64 keys on the GPU."""
    n, f, rows = case["samples"], case["fields"], case["rows"]
    if case["alpha"] == 0.0:
        return torch.randint(rows, (n * f,), generator=gen, device="cuda")
    vocab = field_vocab(rows, f, 0.8 if f > 26 else 0.7)
    v = torch.from_numpy(vocab).cuda()
    base = torch.cumsum(v, 0) - v
    u = torch.rand((n, f), generator=gen, device="cuda", dtype=torch.float64)
    e = 1.0 - case["alpha"]  # inverse of the continuous power law on [1, v + 1)
    rank = ((1.0 - u * (1.0 - (v + 1.0) ** e)) ** (1.0 / e)).long() - 1
    rank = torch.minimum(rank.clamp_(min=0), v - 1)
    return (base + rank * _PRIME % v).reshape(-1).contiguous()


def _where(t, place):
    return t if place == "device" else t.cpu().pin_memory() if place == "pinned" else t.cpu()


def _tables(case):
    """The table of every rank."""
    m, n, rows = hetuctr_b200.hetuCTR, case["nrank"], case["rows"]
    rng = np.random.RandomState(7)
    root = np.zeros(rows, dtype=np.uint8) if n == 1 else rng.randint(n, size=rows).astype(np.uint8)
    job, out, errors = next(_job), [None] * n, []
    hot = None
    if n > 1:
        # hottest keys of every field, where the power law puts them
        vocab = field_vocab(rows, case["fields"], 0.8 if case["fields"] > 26 else 0.7)
        base = np.cumsum(vocab) - vocab
        top = np.minimum(vocab, max(1, int(rows * case["cache"] / case["fields"])))
        hot = np.concatenate([b + np.arange(t) * _PRIME % v for b, t, v in zip(base, top, vocab)])

    if n == 1:
        init = m.Initializer(m.InitType.Normal, 0.0, 0.1)
        return [m.HetuTable(rank=0, nrank=1, device_id=0, ip="127.0.0.1", port=job, length=rows, width=case["width"],
                            pull_bound=case["pull"], push_bound=case["push"], root_arr=root,
                            storage_arr=np.arange(rows), init=init, learning_rate=case["lr"], verbose=0)]

    def make(r):  # the constructor meets the other ranks: one thread each
        keep = np.union1d(np.flatnonzero(root == r), hot)
        try:
            out[r] = hetuctr_b200.Table(r, n, 0, "inproc", job, rows, case["width"], case["pull"], case["push"], root,
                                        keep, (hetuctr_b200.INIT_NORMAL, 0.0, 0.1), case["lr"], 0)
        except Exception as e:  # noqa: BLE001 - raised again below
            errors.append(e)

    old = os.environ.get("HCTR_EXCHANGE")
    os.environ["HCTR_EXCHANGE"] = "p2p"  # the exchange of a job with one process per GPU
    try:
        threads = [threading.Thread(target=make, args=(r,)) for r in range(n)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        os.environ.pop("HCTR_EXCHANGE")
        if old is not None:
            os.environ["HCTR_EXCHANGE"] = old
    if errors:
        raise errors[0]
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n, b, w = case["nrank"], case["samples"] * case["fields"], case["width"]
    hetuctr_b200.hetuCTR.seed(0)
    s = {"tables": _tables(case), "n": b, "step": 0, "train": case["train"]}
    s["keys"] = [[_where(_keys(case, gen), case["keys"]) for _ in range(2)] for _ in range(n)]
    s["grads"] = [[_where(torch.randn((b, w), generator=gen, device="cuda") * 0.01, case["buffers"])
                   for _ in range(2)] if case["train"] else [None, None] for _ in range(n)]
    s["rows"] = [_where(torch.zeros((b, w), device="cuda"), case["buffers"]) for _ in range(n)]
    torch.cuda.synchronize()
    _step(s, train=False)  # the loop is running: one batch is open and its gradients come with the next pass
    return s


def _step(s, train):
    i = s["step"] & 1
    s["step"] += 1
    tables, keys, rows = s["tables"], s["keys"], s["rows"]
    grads = [g[1 - i].data_ptr() if train else 0 for g in s["grads"]]
    if len(tables) == 1:
        tables[0].preprocess(keys[0][i].data_ptr(), s["n"])
        tables[0].push_pull(grads[0], rows[0].data_ptr())
        return rows[0]
    for w in [t.async_preprocess(k[i].data_ptr(), s["n"]) for t, k in zip(tables, keys)]:
        w.wait()
    for w in [t.async_push_pull(g, d.data_ptr()) for t, g, d in zip(tables, grads, rows)]:
        w.wait()
    return rows


def run(state):
    return _step(state, state["train"])


def _distinct(case):
    """Expected number of distinct keys of a batch."""
    n, f, rows = case["samples"], case["fields"], case["rows"]
    if case["alpha"] == 0.0:
        return rows * -math.expm1(n * f * math.log1p(-1.0 / rows)) if rows > 1 else 1.0
    total, e = 0.0, 1.0 - case["alpha"]
    for v in field_vocab(rows, f, 0.8 if f > 26 else 0.7):
        edge = np.unique(np.concatenate([np.arange(min(v, 1024)), np.geomspace(1, v, 2000).astype(np.int64), [v]]))
        lo, hi = edge[:-1] + 1.0, edge[1:] + 1.0
        mass = (lo ** e - hi ** e) / (1.0 - (v + 1.0) ** e)
        cnt = hi - lo
        total += float(np.sum(cnt * -np.expm1(n * np.log1p(-np.minimum(mass / cnt, 1 - 1e-12)))))
    return total


def work(case):
    """Keys, rows of the distinct keys and pulled rows; with gradients: every gradient row once, and every distinct
    key's row and version read and written.  A row of another rank is also written for its owner and read there, and
    the other way round."""
    b, d, u = case["samples"] * case["fields"], 4 * case["width"], _distinct(case)
    n, away = case["nrank"], 1.0 - 1.0 / case["nrank"]
    nbytes = 8 * b + (4 + d) * u + d * b
    if case["train"]:
        nbytes += d * b + (2 * d + 16) * u + away * u * 2 * d
    nbytes += away * u * 2 * d
    flops = (b + u) * case["width"] if case["train"] else 0
    return {"bytes": n * nbytes, "flops": n * flops}


def tolerance(case):
    """Serving copies rows; training sums 32-bit gradients."""
    return {"rel": 1e-5} if case["train"] else "exact"
