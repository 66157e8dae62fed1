"""Performance cases of the engine: the calls its users make, over the range
of sizes they make them at.

Kinds of case (`case["kind"]`):

  collective  one collective over P virtual ranks through a Comm, on the
              default engine or on the one that follows the reference's
              schedule step by step ("pipelined").  Rows are packed, so an
              odd count gives rows that start off the 16-byte grid.
  batch       many independent collectives of uneven P, size, operation and
              element type in one launch (Batch).
  links       per-link byte counts of a schedule on a torus (link_bytes).
  training    forward and backward of the variant picker's network
              (MLP.gradients).

`count` has the meaning of the collective's own argument: the vector per rank
for allreduce and bcast, the received block per rank for reduce_scatter, the
sent block for allgather and alltoall.
"""
import math
import random

import numpy as np
import torch

import bine_trees_fugaku_b200 as bine

_TORCH = {"int32": torch.int32, "int64": torch.int64, "float32": torch.float32, "float64": torch.float64}
_CODE = {"int32": bine.INT32, "int64": bine.INT64, "float32": bine.FLOAT, "float64": bine.DOUBLE}
_SIZE = {"int32": 4, "int64": 8, "float32": 4, "float64": 8}
_LARGEST = 1 << 30  # bytes that a drawn collective or batch reads and writes, at most


def _collective(name, coll, P, count, dtype, engine="fused"):
    return {"name": name, "kind": "collective", "coll": coll, "P": P, "count": count, "dtype": dtype, "engine": engine}


def listed():
    return [
        # The smallest calls: a few KiB per rank, where the launch and the
        # chain of dependent additions are all there is.
        _collective("allreduce_f32_small", "allreduce", 16, 1024, "float32"),
        # The headline workload of the benchmark: 4 MiB per rank, 2 GiB moved.
        _collective("allreduce_i32_headline", "allreduce", 256, 1 << 20, "int32"),
        # Float sums in the reference's order at a rank count that is not a
        # power of two (blocks start anywhere in the row), 2 MiB per rank.
        _collective("allreduce_f32_p384", "allreduce", 384, 1 << 19, "float32"),
        # A gradient-like vector whose length is not a multiple of 4: packed
        # rows of odd length.
        _collective("allreduce_f32_ragged", "allreduce", 96, 262147, "float32"),
        # Sharded reduction, 8 MiB in and 128 KiB out per rank.
        _collective("reduce_scatter_f32", "reduce_scatter", 64, 32768, "float32"),
        # Gathering 32 KiB shards at a rank count that is not a power of two.
        _collective("allgather_i64", "allgather", 96, 4096, "int64"),
        # Broadcast of a medium vector (512 KiB).
        _collective("bcast_i64", "bcast", 256, 65536, "int64"),
        # Transpose-like exchange of blocks of odd length (40 KB).
        _collective("alltoall_i32_ragged", "alltoall", 64, 10001, "int32"),
        # The reference's own schedule, step by step, 1 MiB per rank.
        _collective("pipelined_allreduce_f32", "allreduce", 256, 262144, "float32", "pipelined"),
        # 512 mixed collectives in one launch, rows of 64 B to 64 KiB.
        {"name": "batch_512", "kind": "batch", "items": 512, "max_bytes": 65536, "layout": 2024},
        # Link loads of the bandwidth-optimal allreduce on a 4096-node torus.
        {"name": "links_allreduce_64x64", "kind": "links", "coll": "allreduce", "variant": "B", "dims": "64x64",
         "ports": 1, "count": 262144},
        # One gradient of the picker's network at its training batch.
        {"name": "picker_gradients", "kind": "training", "batch": 256, "in": 16, "out": 144},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["collective", "pipelined", "batch", "links", "training"], [10, 3, 2, 2, 1])[0]
    if kind in ("collective", "pipelined"):
        engine = "fused" if kind == "collective" else "pipelined"
        coll = rng.choice(["allreduce", "allreduce", "allreduce", "reduce_scatter", "allgather", "bcast", "alltoall"])
        dtype = rng.choice(["int32", "int64", "float32", "float32", "float32", "float64"])
        # Schedules with wrong results or deadlocks in the reference at
        # other rank counts are refused: powers of two there, even counts
        # for allreduce, any count where no schedule is followed.
        free = engine == "fused" and (coll in ("allgather", "bcast", "alltoall") or dtype.startswith("int"))
        if free:
            P = _log_int(rng, 4, 512)
        elif coll == "allreduce":
            P = 2 * _log_int(rng, 2, 256 if engine == "fused" else 128)
        else:
            P = 1 << rng.randint(2, 9 if engine == "fused" else 7)
        size = _SIZE[dtype]
        # Bytes of the largest row per rank, 32 B to 4 MiB.
        row = _log_int(rng, 32, 4 << 20)
        per_rank = row // size if coll in ("allreduce", "bcast") else row // (size * P)
        count = max(1, min(per_rank, _LARGEST // (2 * size * P * (1 if coll in ("allreduce", "bcast") else P))))
        if rng.random() < 0.5:  # whole 16-byte vectors, or any length
            count = max(1, count * size // 16) * 16 // size
        if coll == "allreduce" and not free:
            count = max(count, P)  # the bandwidth-optimal schedules need a block per rank
        return {k: v for k, v in _collective("", coll, P, count, dtype, engine).items() if k != "name"}
    if kind == "batch":
        return {"kind": "batch", "items": _log_int(rng, 16, 1024), "max_bytes": _log_int(rng, 1024, 32768),
                "layout": rng.randrange(1 << 20)}
    if kind == "links":
        coll, variant = rng.choice([("allreduce", "B"), ("allreduce", "L"), ("allgather", "VEC_DOUBLING_CONT_PERMUTE")])
        dims = [1 << rng.randint(1, 6)] * rng.choice([2, 3])
        dims[rng.randrange(len(dims))] = 1 << rng.randint(1, 6)
        while math.prod(dims) > 4096:
            dims[dims.index(max(dims))] //= 2
        return {"kind": "links", "coll": coll, "variant": variant, "dims": "x".join(map(str, dims)),
                "ports": rng.choice([1, 1, 2 * len(dims)]), "count": _log_int(rng, 1 << 16, 1 << 22)}
    return {"kind": "training", "batch": 16 * _log_int(rng, 1, 32), "in": 16 * rng.randint(1, 4), "out": 16 * rng.randint(1, 16)}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) % (1 << 62))
    return g


def _values(shape, dtype, g):
    """int32 U[-1000, 1000], int64 U[-2^40, 2^40], floats N(0, 1)."""
    if dtype == "int32":
        return torch.randint(-1000, 1001, shape, dtype=torch.int32, device="cuda", generator=g)
    if dtype == "int64":
        return torch.randint(-(1 << 40), (1 << 40) + 1, shape, dtype=torch.int64, device="cuda", generator=g)
    return torch.randn(shape, dtype=_TORCH[dtype], device="cuda", generator=g)


def _rows(case):
    """Elements per rank of the input and output rows."""
    P, n = case["P"], case["count"]
    return {"allreduce": (n, n), "bcast": (n, n), "reduce_scatter": (n * P, n), "allgather": (n, n * P),
            "alltoall": (n * P, n * P)}[case["coll"]]


def _batch_items(case):
    """(operation, P, count, float?) per item: P ~ U[4, 512], the larger row
    per rank log-uniform from 64 B, half allreduce, a quarter each
    reduce_scatter and allgather, half float32; whole 16-byte vectors."""
    r = random.Random(case["layout"])
    items = []
    for _ in range(case["items"]):
        P = r.randint(4, 512)
        coll = r.choices(["allreduce", "reduce_scatter", "allgather"], [2, 1, 1])[0]
        row = math.exp(r.uniform(math.log(64), math.log(case["max_bytes"])))
        count = max(4, int(row / (4 if coll == "allreduce" else 4 * P)) // 4 * 4)
        items.append((coll, P, count, r.random() < 0.5))
    return items


def _batch_sizes(coll, P, count):
    """Input and output elements of one item."""
    return {"allreduce": (P * count, P * count), "reduce_scatter": (P * P * count, P * count),
            "allgather": (P * count, P * P * count)}[coll]


def _batch_inputs(case, seed):
    g = _generator(seed)
    n = {"int32": 0, "float32": 0}
    for coll, P, count, is_float in _batch_items(case):
        n["float32" if is_float else "int32"] += _batch_sizes(coll, P, count)[0]
    return {k: _values((max(4, v),), k, g) for k, v in n.items()}


def _training_inputs(case, seed):
    g = _generator(seed)
    n = case["batch"]
    x = torch.randn((n, case["in"]), device="cuda", generator=g)
    t = torch.randn((n, case["out"]), device="cuda", generator=g)
    # A call's arms are a part of all arms: the rest is masked out.
    mask = (torch.rand((n, case["out"]), device="cuda", generator=g) < 0.3).float()
    mask[:, 0] = 1
    return x, t, mask


def _training_params(case, seed):
    """Weights as after some training: He-like scale, non-zero biases."""
    rng = np.random.default_rng(seed)
    layout = bine.mlp_layout(case["in"], 256, case["out"])
    p = np.zeros((layout[-1][1] + layout[-1][2] + 15) // 16 * 16, np.float32)
    for w, b, nout, nin in layout:
        p[w:w + nout * nin] = rng.standard_normal(nout * nin) * math.sqrt(2.0 / nin)
        p[b:b + nout] = rng.standard_normal(nout) * 0.1
    return p, layout


def prepare(case, seed):
    kind = case["kind"]
    stream = torch.cuda.current_stream()
    if kind == "collective":
        P, (si, so) = case["P"], _rows(case)
        comm = bine.Comm(P)
        comm.set_stream(stream)
        comm.set_engine(case["engine"])
        x = _values((P, si), case["dtype"], _generator(seed))
        y = x if case["coll"] == "bcast" else torch.zeros((P, so), dtype=_TORCH[case["dtype"]], device="cuda")
        state = {"case": case, "comm": comm, "x": x, "y": y, "code": _CODE[case["dtype"]]}
        # A program calls a collective of one shape many times: the plan is
        # made by the first call (on other data, so that no result is ready).
        if case["coll"] == "bcast":
            keep = x.clone()
            run(state)
            x.copy_(keep)
        else:
            run(state)
            y.zero_()
        return state
    if kind == "batch":
        pools = _batch_inputs(case, seed)
        items, outs, at = [], {}, {"int32": [0, 0], "float32": [0, 0]}
        sizes = _batch_items(case)
        for k in pools:
            total = sum(_batch_sizes(c, P, n)[1] for c, P, n, f in sizes if f == (k == "float32"))
            outs[k] = torch.zeros(max(4, total), dtype=_TORCH[k], device="cuda")
        for coll, P, count, is_float in sizes:
            k = "float32" if is_float else "int32"
            si, so = _batch_sizes(coll, P, count)
            a, b = at[k]
            items.append((coll, pools[k][a:a + si], outs[k][b:b + so], count, _CODE[k], P))
            at[k] = [a + si, b + so]
        return {"case": case, "batch": bine.Batch(items), "in": pools, "out": outs, "stream": stream}
    if kind == "links":
        dims = [int(d) for d in case["dims"].split("x")]
        comm = bine.Comm(math.prod(dims), dims)
        comm.set_stream(stream)
        comm.set_ports(case["ports"])
        comm.set_algo(case["coll"], case["variant"])
        out = torch.zeros(comm.nranks * len(dims) * 2, dtype=torch.int64, device="cuda")
        # The message size asked about: up to a half more than the case's.
        count = case["count"] + random.Random(seed).randrange(case["count"] // 2)
        return {"case": case, "comm": comm, "out": out, "count": count}
    x, t, mask = _training_inputs(case, seed)
    mlp = bine.MLP(case["in"], 256, case["out"], case["batch"])
    mlp.set_params(_training_params(case, seed)[0])
    return {"case": case, "mlp": mlp, "x": x, "t": t, "mask": mask}


def run(state):
    case = state["case"]
    if case["kind"] == "collective":
        state["comm"].run(case["coll"], state["x"], state["y"], case["count"], state["code"])
        return state["y"]
    if case["kind"] == "batch":
        state["batch"].launch(state["stream"])
        return state["out"]
    if case["kind"] == "links":
        state["comm"].link_bytes(case["coll"], state["count"], bine.INT32, state["out"])
        return state["out"]
    grads, loss = state["mlp"].gradients(state["x"], state["t"], state["mask"])
    return {"grads": grads, "loss": loss}


def work(case):
    if case["kind"] == "collective":
        P, size, (si, so) = case["P"], _SIZE[case["dtype"]], _rows(case)
        if case["coll"] == "bcast":
            return {"bytes": P * so * size, "flops": 0}
        adds = (P - 1) * si if case["coll"] in ("allreduce", "reduce_scatter") else 0
        return {"bytes": P * (si + so) * size, "flops": adds}
    if case["kind"] == "batch":
        total = [_batch_sizes(c, P, n) for c, P, n, _ in _batch_items(case)]
        return {"bytes": 4 * sum(a + b for a, b in total), "flops": 0}
    if case["kind"] == "links":
        dims = [int(d) for d in case["dims"].split("x")]
        return {"bytes": 8 * math.prod(dims) * len(dims) * 2, "flops": 0}
    n, layers = case["batch"], [(case["in"], 256), (256, 256), (256, 256), (256, case["out"])]
    weights = sum(a * b + b for a, b in layers)
    macs = 3 * sum(a * b for a, b in layers) - case["in"] * 256  # no gradient of the input
    return {"bytes": 4 * (2 * weights + n * (case["in"] + 2 * case["out"])), "flops": 2 * n * macs}


def exact(case, seed):
    if case["kind"] == "collective":
        if not case["dtype"].startswith("float"):
            return None  # whole numbers: the same or wrong
        P, n, (si, _) = case["P"], case["count"], _rows(case)
        x = _values((P, si), case["dtype"], _generator(seed))
        if case["coll"] in ("allreduce", "reduce_scatter"):
            total = torch.zeros(si, dtype=torch.float64, device="cuda")
            for row in x:
                total += row
            return total.expand(P, n) if case["coll"] == "allreduce" else total.view(P, n)
        x = x.double()
        if case["coll"] == "allgather":
            return x.reshape(1, -1).expand(P, -1)
        if case["coll"] == "bcast":
            return x[:1].expand(P, n)
        return x.view(P, P, n).transpose(0, 1).reshape(P, P * n)
    if case["kind"] == "batch":
        pool, outs, a = _batch_inputs(case, seed)["float32"], [], 0
        for coll, P, count, is_float in _batch_items(case):
            if not is_float:
                continue
            si, so = _batch_sizes(coll, P, count)
            x = pool[a:a + si].view(P, -1).double()
            a += si
            outs.append({"allreduce": lambda: x.sum(0).expand(P, -1), "reduce_scatter": lambda: x.sum(0),
                         "allgather": lambda: x.reshape(1, -1).expand(P, -1)}[coll]().reshape(-1))
        out = torch.cat(outs) if outs else torch.zeros(4, dtype=torch.float64, device="cuda")
        return {"int32": None, "float32": out}
    if case["kind"] == "links":
        return None  # whole numbers
    x, t, mask = (v.double() for v in _training_inputs(case, seed))
    p, layout = _training_params(case, seed)
    p = torch.from_numpy(p).double().cuda().requires_grad_()
    a = x
    for l, (w, b, nout, nin) in enumerate(layout):
        a = a @ p[w:w + nout * nin].view(nout, nin).T + p[b:b + nout]
        if l + 1 < len(layout):
            a = torch.nn.functional.gelu(a)
    loss = ((mask * (a - t)) ** 2).sum() / (mask != 0).sum()
    loss.backward()
    return {"grads": p.grad.cpu().numpy(), "loss": float(loss)}
