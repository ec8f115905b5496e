"""Performance cases of the collectives on one GPU.

Every case runs through the calls an application makes: ``mccs_b200.Communicator`` collectives on
service memory (planned by the daemon; launched by the client library for a communicator of one rank,
by the daemon for ranks that share the GPU), the ``mccs_b200.ops`` functions on ordinary tensors (what
the ``torch.distributed`` backend is made of), and ``ops.local_all_reduce_no_alloc``.

A case is a dict:
  path      "comm" (service memory), "staged" (ordinary tensors), "local" (no daemon)
  coll      "all_reduce", "all_gather", "reduce_scatter"
  ranks     ranks of the communicator, all of them driven by this process on cuda:0
  tenants   communicators that issue the same work side by side
  calls     collectives each rank issues in a pass, all of them in one group
  dtype, count   element type and count as the call takes it: elements per rank (all_reduce, all_gather),
            per block (reduce_scatter)
  op        reduction operator
  in_place  whether input and output are the same memory
  offset    elements between the start of the allocation and the first element used
"""
import atexit
import os
import tempfile
import threading

import torch

os.environ.setdefault("MCCS_LOG", "warn")

import mccs_b200 as M  # noqa: E402
from mccs_b200 import ops  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32, "f64": torch.float64,
          "i32": torch.int32, "u8": torch.uint8}
SIZE = {"bf16": 2, "f16": 2, "f32": 4, "f64": 8, "i32": 4, "u8": 1}
MIB = 1 << 20


def _case(path="comm", coll="all_reduce", ranks=2, tenants=1, calls=1, dtype="f32", count=1, op="sum", in_place=False, offset=0):
    return {"path": path, "coll": coll, "ranks": ranks, "tenants": tenants, "calls": calls, "dtype": dtype, "count": count,
            "op": op, "in_place": in_place, "offset": offset}


def listed():
    def named(name, **kw):
        return dict(_case(**kw), name=name)

    return [
        # the repository's benchmark as it runs on one GPU: one rank, 512 MiB of bf16, out of place
        named("one_rank_512m_bf16", ranks=1, dtype="bf16", count=256 * MIB),
        # one rank, a small message: what a call costs from Python to the kernel when the library launches it
        named("one_rank_64k_f32", ranks=1, dtype="f32", count=16384),
        # a 25 MB gradient bucket in an ordinary tensor, as torch DDP hands it to the torch.distributed backend
        named("staged_25m_f32", path="staged", ranks=1, dtype="f32", count=6553600),
        # the smallest message of the evaluation sweep, eight ranks: latency and launches
        named("all_reduce_8x32k_bf16", ranks=8, dtype="bf16", count=16384),
        # a 25 MB gradient bucket of mccs_b200.parallel.DataParallel: in place, average
        named("bucket_4x25m_bf16_avg", ranks=4, dtype="bf16", count=13107200, op="avg", in_place=True),
        # the multi-tenant evaluation: each tenant's iteration is 16 back-to-back fp32 AllReduces of 8 MiB
        named("tenants_2x2_16x8m_f32", ranks=2, tenants=2, calls=16, dtype="f32", count=2 * MIB),
        # all gradients of the VGG trace in one AllReduce: 574,668,960 bytes on four ranks
        named("all_reduce_4x574m_f32", ranks=4, dtype="f32", count=143667240),
        # a view that starts at an odd element and has an odd length (a slice of a flat parameter buffer)
        named("all_reduce_8x_ragged_f16", ranks=8, dtype="f16", count=1000003, offset=3),
        # AllGather, 64 MiB gathered on every one of eight ranks
        named("all_gather_8x8m_bf16", coll="all_gather", ranks=8, dtype="bf16", count=4 * MIB),
        # AllGather of byte strings whose length is no multiple of anything (serialised objects)
        named("all_gather_4x_ragged_u8", coll="all_gather", ranks=4, dtype="u8", count=1000003),
        # the ReduceScatter of a 25 MB sharded gradient bucket (mccs_b200.parallel.ShardedDataParallel)
        named("reduce_scatter_8x25m_bf16", coll="reduce_scatter", ranks=8, dtype="bf16", count=1638400, op="avg"),
        # partial results of eight workers of one GPU summed without daemon or allocation
        named("local_8x32m_bf16", path="local", ranks=8, dtype="bf16", count=16 * MIB),
    ]


_MOST_BYTES = 4_500_000_000      # below the largest listed case
_MOST_RAGGED = 64 * MIB         # odd offsets and lengths are met in small and medium messages


def draw(rng):
    path = rng.choice(["comm"] * 7 + ["staged"] + ["local"] * 2)
    if path == "local":
        coll = "all_reduce"
    elif path == "staged":
        coll = rng.choice(["all_reduce", "all_gather", "reduce_scatter"])
    else:
        coll = rng.choice(["all_reduce"] * 5 + ["all_gather"] * 3 + ["reduce_scatter"] * 2)
    ranks = 1 if path == "staged" else rng.choice([2, 2, 3, 4, 4, 5, 6, 7, 8, 8] + ([] if path == "local" else [1, 1]))
    if path == "local":
        dtype = rng.choice(["bf16", "f16", "f32"])
    elif coll == "all_gather":
        dtype = rng.choice(["bf16", "f32", "u8"])
    else:
        dtype = rng.choice(["bf16"] * 3 + ["f32"] * 3 + ["f16"] * 2 + ["i32", "f64"])
    floating = dtype not in ("i32", "u8")
    op, in_place = "sum", False
    if path == "comm" and coll != "all_gather":
        op = rng.choice(["sum", "sum", "avg", "max"]) if floating else rng.choice(["sum", "max"])
        in_place = ranks > 1 and op in ("avg", "max") and rng.random() < 0.5     # repeated passes keep such values in range
    elif path == "comm":
        in_place = ranks > 1 and rng.random() < 0.3
    ragged = rng.random() < 0.3
    offset = rng.choice([0, 1, 3, 5]) if ragged else 0
    calls = tenants = 1
    if path == "comm" and ranks > 1 and rng.random() < 0.2:
        calls = rng.choice([2, 4, 8])
    case = _case(path, coll, ranks, tenants, calls, dtype, 1, op, in_place, offset)
    most = _MOST_RAGGED if ragged else _MOST_BYTES
    top = min(512 * MIB, most * SIZE[dtype] / work(case)["bytes"])      # bytes per rank (per block for reduce_scatter)
    low = 8192
    nbytes = low * (max(top, low) / low) ** rng.random()
    count = max(1, int(nbytes / SIZE[dtype]))
    case["count"] = count | 1 if ragged else max(1, count // 64) * 64
    return case


def _units(case):
    """Elements one rank's input and output hold."""
    n, c = case["ranks"], case["count"]
    return (c * n if case["coll"] == "reduce_scatter" else c), (c * n if case["coll"] == "all_gather" else c)


def work(case):
    n, esz, (i, o) = case["ranks"], SIZE[case["dtype"]], _units(case)
    if case["in_place"] and case["coll"] == "all_gather":
        o -= case["count"]      # a rank's own block is in its place already
    times = case["tenants"] * case["calls"]
    # elements that have to be reduced: once on the GPU, however many ranks receive them
    reduced = 0 if case["coll"] == "all_gather" else case["count"] * (n if case["coll"] == "reduce_scatter" else 1)
    return {"bytes": times * n * (i + o) * esz, "flops": times * (n - 1) * reduced}


def tolerance(case):
    if case["coll"] == "all_gather" or case["ranks"] == 1 or case["op"] == "max" or case["dtype"] in ("i32", "u8"):
        return "exact"
    # fp32 accumulation; 16-bit results are rounded once
    return {"rel": {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5, "f64": 1e-12}[case["dtype"]]}


# -- what a program keeps: the daemon's connection and one communicator per group of ranks -----------
_comms = {}


def _communicators(ranks, tenant):
    if not _comms:
        prefix = tempfile.mkdtemp(prefix="mccs-perf-")
        # launch = "client": the library launches its own kernels where it can, as in a process outside the daemon
        M.init(M.daemon.start_embedded(prefix=prefix, listen_port=0, extra='launch = "client"'))
        atexit.register(M.daemon.stop_embedded)
        if M.backend() != "cuda":
            raise RuntimeError("the daemon did not come up on the CUDA backend")
    key = (ranks, tenant)
    if key not in _comms:
        made, errors = [None] * ranks, []

        def join(r):      # a communicator exists once every rank has joined
            try:
                torch.cuda.set_device(0)
                made[r] = M.Communicator(7000 + 100 * tenant + ranks, r, ranks, device=0)
            except Exception as e:  # noqa: BLE001
                errors.append(e)

        threads = [threading.Thread(target=join, args=(r,)) for r in range(ranks)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        if errors:
            raise errors[0]
        _comms[key] = made
    return _comms[key]


def _fill(t, gen):
    if t.dtype.is_floating_point:
        t.uniform_(-1, 1, generator=gen)
    else:
        t.random_(0, 200 if t.dtype == torch.uint8 else 1000, generator=gen)


def _buffer(numel, case):
    dtype, off = DTYPES[case["dtype"]], case["offset"]
    if case["path"] == "comm":
        b = M.Buffer((numel + off) * SIZE[case["dtype"]], 0)
        return _holding(b.tensor(dtype, numel + off)[off:], b)
    return _holding(torch.empty(numel + off, dtype=dtype, device="cuda:0")[off:], None)


def _holding(tensor, buffer):
    """The tensor with a reference to the service memory under it: an output that is kept longer than
    its state must not outlive the allocation."""
    tensor.service_buffer = buffer
    return tensor


def prepare(case, seed):
    torch.cuda.set_device(0)
    gen = torch.Generator(device="cuda:0").manual_seed(1000003 * seed + 17)
    state = {"case": case, "calls": [], "out": []}
    n, (i, o) = case["ranks"], _units(case)
    for t in range(case["tenants"]):
        comms = [None] * n if case["path"] == "local" else _communicators(n, t)
        for _ in range(case["calls"]):
            send, recv = [], []
            for r in range(n):
                if not case["in_place"]:
                    s, d = _buffer(i, case), _buffer(o, case)
                elif case["coll"] == "all_gather":
                    d = _buffer(o, case)
                    s = _holding(d[r * i:(r + 1) * i], d.service_buffer)
                else:
                    s = _buffer(i, case)
                    d = s if case["coll"] == "all_reduce" else _holding(s[r * o:(r + 1) * o], s.service_buffer)
                _fill(s, gen)
                send.append(s)
                recv.append(d)
            state["calls"].append((comms, send, recv))
            state["out"] += recv
    return state


def _collective(case, comm, send, recv):
    if case["coll"] == "all_reduce":
        comm.all_reduce(send, recv, op=case["op"])
    elif case["coll"] == "all_gather":
        comm.all_gather(send, recv)
    else:
        comm.reduce_scatter(send, recv, op=case["op"])


def run(state):
    case = state["case"]
    if case["path"] == "local":
        for _, send, recv in state["calls"]:
            ops.local_all_reduce_no_alloc(send, recv)
    elif case["path"] == "staged":
        for comms, send, recv in state["calls"]:
            if case["coll"] == "all_reduce":
                ops.all_reduce(comms[0], send[0], recv[0], op=case["op"])
            elif case["coll"] == "all_gather":
                ops.all_gather(comms[0], send[0], recv[0])
            else:
                ops.reduce_scatter(comms[0], send[0], recv[0], op=case["op"])
    elif case["ranks"] == 1 and case["calls"] == 1 and case["tenants"] == 1:
        comms, send, recv = state["calls"][0]
        _collective(case, comms[0], send[0], recv[0])
    else:
        with M.group():     # one thread drives every rank
            for comms, send, recv in state["calls"]:
                for comm, s, d in zip(comms, send, recv):
                    _collective(case, comm, s, d)
    return state["out"]
