"""The kernels that carry every rank of a communicator on one GPU (csrc/kernels/one_gpu.cuh)
through the service, at the sizes where they can go wrong: around a 16-byte pack, a tile of a CTA
and a grid of many tiles, buffers at other 16-byte phases, in place, and a grid bounded by an
operator's CTA limit. Sums accumulate in fp32 (fp64 for doubles) in rank order and are rounded
once, so the result differs from the fp64 sum by at most n - 1 roundings of partial sums below n
in magnitude plus the final rounding."""
import threading
import time

import pytest
import torch

from helpers import fresh_comm_id, run_ranks

pytestmark = pytest.mark.gpu

#: unit roundoff (2^-p for a significand of p bits, the implicit one among them) of the accumulator
#: and of the result type: p = 24 for fp32, 8 for bf16, 11 for fp16, 53 for fp64
ROUND = {torch.float32: (2.0**-24, 2.0**-24), torch.bfloat16: (2.0**-24, 2.0**-8), torch.float16: (2.0**-24, 2.0**-11),
         torch.float64: (2.0**-53, 2.0**-53)}


def _input(dtype, count, seed):
    g = torch.Generator().manual_seed(seed)
    if dtype.is_floating_point:
        return (torch.rand(count, generator=g) * 2 - 1).to(dtype)
    return torch.randint(-50, 50, (count,), generator=g).to(dtype)


def _case(M, coll, n, dtype, count, op="sum", offset=0, recv_offset=None, in_place=False, ctas=0):
    cid, esz = fresh_comm_id(), torch.empty((), dtype=dtype).element_size()
    recv_offset = offset if recv_offset is None else recv_offset
    n_in = count * n if coll == "reduce_scatter" else count
    n_out = count * n if coll == "all_gather" else count

    def rank_fn(r):
        torch.cuda.set_device(0)
        torch.cuda.set_stream(torch.cuda.Stream())
        a, b = M.Buffer((n_in + offset) * esz, 0), M.Buffer((n_out + recv_offset + 16) * esz, 0)
        whole = b.tensor(dtype, n_out + recv_offset + 16)
        whole.fill_(7)
        d = whole[recv_offset:recv_offset + n_out]
        s = a.tensor(dtype, n_in + offset)[offset:]
        if in_place:
            s, d = {"all_reduce": (s, s), "reduce_scatter": (s, s[r * count:(r + 1) * count]),
                    "all_gather": (d[r * count:(r + 1) * count], d)}[coll]
        x = _input(dtype, n_in, 31 * r + count % 1000)
        s.copy_(x)
        c = M.Communicator(cid, r, n, device=0)
        if ctas and r == 0:
            assert M.reconfigure(M.daemon.embedded_admin_port(), [{"communicator_id": cid, "ctas": ctas}])["status"] == "ok"
        if coll == "all_reduce":
            c.all_reduce(s, d, op=op)
        elif coll == "reduce_scatter":
            c.reduce_scatter(s, d, op=op)
        else:
            c.all_gather(s, d)
        torch.cuda.synchronize()
        got, plan, q = d.cpu(), c.last_plan(), c.query()
        guards = bool((whole[:recv_offset] == 7).all()) and bool((whole[recv_offset + n_out:] == 7).all())
        c.destroy()
        return x, got, plan[0], q, guards

    outs = run_ranks(n, rank_fn)
    xs = torch.stack([o[0] for o in outs])
    for r, (_, got, plan, q, guards) in enumerate(outs):
        assert plan == "one_gpu" and guards and q["device_error"] == 0 and q["async_error"] == 0
        if coll == "all_gather":
            assert torch.equal(got, xs.reshape(-1))
            continue
        mine = xs if coll == "all_reduce" else xs[:, r * count:(r + 1) * count]
        wide = mine.double() if dtype.is_floating_point else mine.to(torch.int64)
        if op == "max":
            assert torch.equal(got, wide.max(0).values.to(dtype))
        elif not dtype.is_floating_point:
            assert torch.equal(got.to(torch.int64), wide.sum(0))
        else:
            want = wide.sum(0) / (n if op == "avg" else 1)
            acc, res = ROUND[dtype]
            # n - 1 additions of values below n (and, for avg, a multiplication), then one rounding of
            # the result. The factor 1/n of avg is an fp32 number for every type: 2^-24 of the result.
            bound = (n + 1) * n * acc + want.abs() * (res * 1.01 + (2.0**-24 if op == "avg" else 0.0))
            assert bool(((got.double() - want).abs() <= bound).all()), f"{coll} n={n} {dtype} count={count} offset={offset}"


@pytest.mark.parametrize("coll", ["all_reduce", "reduce_scatter", "all_gather"])
@pytest.mark.parametrize("n", [2, 3, 4, 7, 8])
def test_one_gpu_sizes_and_phases(service, coll, n):
    M = service
    assert M.backend() == "cuda"
    for count in (1, 8, 129, 4096 + 8, 300_007, 1 << 20):
        _case(M, coll, n, torch.bfloat16, count)
    _case(M, coll, n, torch.float32, 65_539, offset=3)                       # one phase everywhere
    _case(M, coll, n, torch.float16, 100_003, offset=3, recv_offset=0)       # sources shifted against destinations
    _case(M, coll, n, torch.uint8, 70_001, offset=5, recv_offset=2) if coll == "all_gather" else \
        _case(M, coll, n, torch.int32, 40_001, op="max", offset=1, recv_offset=2)
    _case(M, coll, n, torch.float64, 20_001, in_place=True, op="avg")
    _case(M, coll, n, torch.float32, 1 << 20, ctas=2)                        # bounded grid: many tiles per CTA


@pytest.mark.parametrize("dtype", [torch.int8, torch.uint8, torch.int64])
def test_one_gpu_integer_types(service, dtype):
    _case(service, "all_reduce", 4, dtype, 10_007, op="max")
    _case(service, "reduce_scatter", 8, dtype, 4_099, op="max")


@pytest.mark.parametrize("coll,n", [("all_reduce", 2), ("all_reduce", 8), ("reduce_scatter", 4), ("all_gather", 3)])
def test_one_gpu_groups_in_one_launch(service, coll, n):
    """Collectives of one group may share a launch: different lengths (below a pack, around a tile,
    ragged), and calls that have to run in order: a chain in place, and one that reads what the
    chain left with other ranks. In odd rounds the communicator is paused until the whole group
    waits, in even ones products queued in front keep the GPU busy while it is posted."""
    M = service
    torch.cuda.set_device(0)
    counts = [4096, 1, 300_008, 65_536, 8, 77, 4096, 1 << 20, 4096, 4096]
    cid, comms = fresh_comm_id(), [None] * n
    run_ranks(n, lambda r: comms.__setitem__(r, M.Communicator(cid, r, n, device=0)))
    keep = []

    def per_rank(count):
        bufs = [M.Buffer(count * 4, 0) for _ in range(n)]
        keep.extend(bufs)
        return [b.tensor(torch.float32, count) for b in bufs]

    pairs = [(per_rank(c * (n if coll == "reduce_scatter" else 1)), per_rank(c * (n if coll == "all_gather" else 1))) for c in counts]
    chain, last = per_rank(50_000), per_rank(50_000)
    big = torch.randn(4096, 4096, device="cuda")
    for it in range(4):
        for k, (send, _) in enumerate(pairs):
            for r in range(n):
                send[r].copy_(torch.arange(send[r].numel(), device="cuda") % 13 + r + k + it)   # sums of small whole numbers are exact
        for r in range(n):
            chain[r].fill_(1.0)
        if it % 2:
            assert M.daemon.embedded_admin({"cmd": "pause", "communicator_id": cid})["status"] == "ok"
            threading.Timer(0.1, lambda: M.daemon.embedded_admin({"cmd": "resume", "communicator_id": cid})).start()
        else:
            for _ in range(6):
                torch.mm(big, big)
        with M.group():
            for send, recv in pairs:
                for r in range(n):
                    getattr(comms[r], coll)(send[r], recv[r])
            for _ in range(3):
                for r in range(n):
                    comms[r].all_reduce(chain[r])
            for r in range(n):
                comms[r].all_reduce(chain[(r + 1) % n], last[r])
        for k, (send, recv) in enumerate(pairs):
            count = counts[k]
            whole = torch.cat(send) if coll == "all_gather" else torch.stack(send).sum(0)
            for r in range(n):
                want = whole[r * count:(r + 1) * count] if coll == "reduce_scatter" else whole
                assert torch.equal(recv[r], want), f"{coll} n={n} member {k} ({count})"
        for r in range(n):
            assert bool((chain[r] == float(n) ** 3).all()) and bool((last[r] == float(n) ** 4).all())
    for _ in range(200):         # the daemon counts a launch's members once it has seen the completion word
        q = comms[0].query()
        if q["launched"] == q["completed"]:
            break
        time.sleep(0.01)
    assert q["async_error"] == 0 and q["device_error"] == 0 and q["launched"] == q["completed"] == 4 * (len(counts) + 4)
    stats = M.daemon.embedded_admin({"cmd": "stats"})["stats"]["communicators"][str(cid)]
    assert stats["fused_members"] >= 2 * len(counts)      # both paused rounds: every independent call shared a launch
    for c in comms:
        c.destroy()
