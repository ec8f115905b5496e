"""Clients inside the daemon's process whose ranks share a GPU: the daemon launches on the
caller's stream when all ranks are on one, and orders the callers' streams itself when they are
not. Long-running work is queued in front of every collective and a consumer behind it, on the
same stream, on changing streams, on one stream per rank, with a deferred wait and with
``Communicator.wait`` from another stream: whatever is not ordered reads poisoned values."""
import threading

import pytest
import torch

from helpers import fresh_comm_id, run_ranks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["one_stream", "changing", "per_rank", "deferred", "wait_elsewhere"])
@pytest.mark.parametrize("n", [1, 2, 4])
def test_collectives_are_ordered_with_the_callers_streams(service, n, mode):
    M, count = service, 1 << 20
    torch.cuda.set_device(0)
    cid, comms = fresh_comm_id(), [None] * n
    threads = [threading.Thread(target=lambda r=r: comms.__setitem__(r, M.Communicator(cid, r, n, device=0))) for r in range(n)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    bufs = [(M.Buffer(count * 4, 0), M.Buffer(count * 4, 0)) for _ in range(n)]
    send = [a.tensor(torch.float32, count) for a, _ in bufs]
    recv = [b.tensor(torch.float32, count) for _, b in bufs]
    streams = [torch.cuda.Stream() for _ in range(max(n, 3))]
    other = torch.cuda.Stream()
    big = torch.randn(4096, 4096, device="cuda")
    bad = torch.zeros((), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for c in comms:
        c.set_deferred_wait(mode == "deferred")
    for it in range(12):
        used = [streams[r if mode == "per_rank" else it % 3 if mode == "changing" else 0] for r in range(n)]
        for r in range(n):
            used[r].wait_stream(torch.cuda.default_stream())     # the previous round's consumers
            with torch.cuda.stream(used[r]):
                for _ in range(3):
                    torch.mm(big, big)                           # the inputs exist only after this
                send[r].fill_(float(it + r))
                recv[r].fill_(-1.0)
        with M.group():
            for r in range(n):
                comms[r].all_reduce(send[r], recv[r], stream=used[r])
        for r in range(n):
            reader = other if mode in ("deferred", "wait_elsewhere") else used[r]
            if reader is other:
                comms[r].wait(other)
            with torch.cuda.stream(reader):
                wrong = (recv[r] != float(n * it + n * (n - 1) // 2)).sum()
            torch.cuda.default_stream().wait_stream(reader)
            bad += wrong
    torch.cuda.synchronize()
    assert int(bad) == 0
    for c in comms:
        q = c.query()
        assert q["async_error"] == 0 and q["device_error"] == 0
        c.destroy()


def test_kernels_that_wait_for_one_another_on_callers_streams(service):
    """The cooperative kernels may end without their completion word, so streams and the release of memory follow
    an event behind them: mixed with the one-pass kernels on changing streams, read after
    ``Communicator.wait`` elsewhere, and freed while queued (the free returns when the kernel has ended)."""
    M, count, n = service, 1 << 18, 2
    torch.cuda.set_device(0)
    cid, comms = fresh_comm_id(), [None] * n
    run_ranks(n, lambda r: comms.__setitem__(r, M.Communicator(cid, r, n, device=0)))
    streams, other = [torch.cuda.Stream() for _ in range(2)], torch.cuda.Stream()
    bufs = [M.Buffer(count * 4, 0) for _ in range(2 * n)]
    x, y = ([b.tensor(torch.float32, count) for b in bufs[i::2]] for i in range(2))
    for it, algo in enumerate(["ar_twoshot", "auto", "auto", "ar_twoshot", "ar_ring", "auto", "ar_twoshot", "ar_oneshot"] * 2):
        for t in x + y:
            t.fill_(-1.0)
        torch.cuda.synchronize()
        stream = streams[it // 2 % 2] if it % 4 else streams[0]
        with torch.cuda.stream(stream):
            torch.cuda._sleep(4_000_000)
            for r in range(n):
                x[r].fill_(float(it + r))
        with M.group():
            for r in range(n):
                comms[r].all_reduce(x[r], y[r], algo=algo, stream=stream)
        assert algo == "auto" or comms[0].last_plan()[0] == algo
        comms[it % 2].wait(other)
        with torch.cuda.stream(other):
            seen = [t.clone() for t in y]
        torch.cuda.synchronize()
        assert all(bool((t == float(2 * it + 1)).all()) for t in seen), (it, algo, seen[0][:4].tolist())
    for algo in ("ar_twoshot", "auto"):
        extra = [M.Buffer(count * 4, 0) for _ in range(n)]
        with torch.cuda.stream(streams[0]):
            torch.cuda._sleep(100_000_000)       # about 50 ms
        with M.group():
            for r in range(n):
                comms[r].all_reduce(x[r], extra[r].tensor(torch.float32, count), algo=algo, stream=streams[0])
        assert not streams[0].query()
        extra[0].free()
        assert streams[0].query()
        extra[1].free()
    for c in comms:
        q = c.query()
        assert q["async_error"] == 0 and q["device_error"] == 0
        c.destroy()


FUSED = r"""
import os, threading
import torch
import mccs_b200 as M

torch.cuda.set_device(0)
M.init(M.daemon.start_embedded(prefix=f"/tmp/mccs-fused-streams-{os.getpid()}", listen_port=-1, extra="fuse_allreduce = 4"))
n, count, comms = 2, 1 << 20, [None, None]
ts = [threading.Thread(target=lambda r=r: comms.__setitem__(r, M.Communicator(41, r, n, device=0))) for r in range(n)]
[t.start() for t in ts]
[t.join() for t in ts]
bufs = [M.Buffer(count * 4, 0) for _ in range(4 * n)]
a, ra, b, rb = ([x.tensor(torch.float32, count) for x in bufs[i::4]] for i in range(4))
s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
for it in range(6):
    for r in range(n):
        a[r].fill_(float(it + r)); b[r].fill_(float(10 * it + r)); ra[r].fill_(-1.0); rb[r].fill_(-1.0)
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(20_000_000)        # the launch cannot run before this has ended
    # held back until the whole group waits: its two calls go out in one launch
    assert M.daemon.embedded_admin({"cmd": "pause", "communicator_id": 41})["status"] == "ok"
    threading.Timer(0.1, lambda: M.daemon.embedded_admin({"cmd": "resume", "communicator_id": 41})).start()
    with M.group():
        for r in range(n):
            comms[r].all_reduce(a[r], ra[r], algo="ar_twoshot", stream=s1)
        for r in range(n):
            comms[r].all_reduce(b[r], rb[r], algo="ar_twoshot", stream=s2)
    seen = []
    for stream, out, want in ((s1, ra, 2 * it + 1), (s2, rb, 20 * it + 1)):
        with torch.cuda.stream(stream):
            seen += [(x.clone(), float(want)) for x in out]
    torch.cuda.synchronize()
    for k, (x, want) in enumerate(seen):
        assert bool((x == want).all()), (it, k, x[:4].tolist(), want)
stats = M.daemon.embedded_admin({"cmd": "stats"})["stats"]["communicators"]["41"]
assert stats["fused_members"] == 12, stats
for c in comms:
    c.destroy()
M.finalize()
M.daemon.stop_embedded()
print("OK")
"""


def test_members_of_a_fused_launch_on_streams_of_their_own():
    """With ``fuse_allreduce`` one launch carries calls that were given different streams: each of them waits for it."""
    import os
    import subprocess
    import sys

    from helpers import REPO
    p = subprocess.run([sys.executable, "-c", FUSED], env=dict(os.environ, PYTHONPATH=REPO), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("OK"), p.stdout[-2000:] + p.stderr[-3000:]


@pytest.mark.parametrize("n", [1, 2])
def test_streams_destroyed_while_their_collective_waits(service, n):
    """A stream may be destroyed while work is queued on it, and its handle given to the next one: the next
    collective and whoever waits for the communicator are still behind the old stream's."""
    import ctypes
    M, count, cid, comms = service, 1 << 20, fresh_comm_id(), [None] * n
    torch.cuda.set_device(0)
    run_ranks(n, lambda r: comms.__setitem__(r, M.Communicator(cid, r, n, device=0)))
    bufs = [M.Buffer(count * 4, 0) for _ in range(3 * n)]
    x, y, z = ([b.tensor(torch.float32, count) for b in bufs[i::3]] for i in range(3))
    lib, other, handles = ctypes.CDLL("libcuda.so.1"), torch.cuda.Stream(), []

    def create():
        s = ctypes.c_void_p()
        assert lib.cuStreamCreate(ctypes.byref(s), 1) == 0
        handles.append(s.value)
        return s, torch.cuda.ExternalStream(s.value)

    def reduce(src, dst, stream):
        with M.group():
            for r in range(n):
                comms[r].all_reduce(src[r], dst[r], stream=stream)

    for it in range(12):
        for r in range(n):
            y[r].fill_(-1.0)
            z[r].fill_(-1.0)
        torch.cuda.synchronize()
        old, stream = create()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(10_000_000)
            for r in range(n):
                x[r].fill_(float(it + r))
        reduce(x, y, stream)
        assert lib.cuStreamDestroy_v2(old) == 0
        new, stream = create()
        if it % 2:
            reduce(y, z, stream)
            with torch.cuda.stream(stream):
                seen = [t.clone() for t in z]
        else:
            comms[0].wait(stream)
            with torch.cuda.stream(stream):
                seen = [t.clone() for t in y]
        torch.cuda.synchronize()
        want = float(n * it + n * (n - 1) // 2) * (n if it % 2 else 1)
        assert all(bool((t == want).all()) for t in seen), (it, want, seen[0][:4].tolist())
        assert lib.cuStreamDestroy_v2(new) == 0
    print(f"{len(handles) - len(set(handles))} of {len(handles)} handles were given out again")
    for c in comms:
        c.destroy()


TIMED_OUT = r"""
import ctypes, os, threading, time
import torch
import mccs_b200 as M

torch.cuda.set_device(0)
M.init(M.daemon.start_embedded(prefix=f"/tmp/mccs-given-up-{os.getpid()}", listen_port=-1))
lib, count = ctypes.CDLL("libcuda.so.1"), 1 << 20

def create():
    s = ctypes.c_void_p()
    assert lib.cuStreamCreate(ctypes.byref(s), 1) == 0
    return s, torch.cuda.ExternalStream(s.value)

def timed_out(call):
    try:
        call()
    except M.MccsError as e:
        assert e.code == -6, e
        return
    raise AssertionError("the call came back")

def communicators(cid, n):
    comms = [None] * n
    ts = [threading.Thread(target=lambda r=r: comms.__setitem__(r, M.Communicator(cid, r, n, device=0))) for r in range(n)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    return comms

def pause(cid, on):
    assert M.daemon.embedded_admin({"cmd": "pause" if on else "resume", "communicator_id": cid})["status"] == "ok"

other = torch.cuda.Stream()
for cid, n, grouped in ((51, 2, False), (52, 2, True), (53, 1, False), (54, 1, True)):
    comms = communicators(cid, n)
    bufs = [M.Buffer(count * 4, 0) for _ in range(2 * n)]
    x, y = ([b.tensor(torch.float32, count) for b in bufs[i::2]] for i in range(2))
    for t in x:
        t.fill_(1.0)
    with M.group():                                    # loads the kernel (which waits for a busy GPU)
        for r in range(n):
            comms[r].all_reduce(x[r], y[r])
    for it in range(3):
        for t in y:
            t.fill_(-1.0)
        torch.cuda.synchronize()
        raw, stream = create()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_500_000_000)           # outlasts the call's patience: the input exists only after it
            x[0].fill_(float(it + 1))
        def first():
            if grouped:
                with M.group():
                    comms[0].all_reduce(x[0], y[0], stream=stream)
            else:
                comms[0].all_reduce(x[0], y[0], stream=stream)
        if n == 1:
            pause(cid, True)
        timed_out(first)                               # no peer (or a paused communicator)
        assert lib.cuStreamDestroy_v2(raw) == 0        # the caller is done with its stream
        raw2, stream2 = create()
        if n == 1:
            pause(cid, False)
        else:
            with torch.cuda.stream(stream2):
                x[1].fill_(10.0)
            comms[1].all_reduce(x[1], y[1], stream=stream2)
            with torch.cuda.stream(stream2):
                seen = y[1].clone()
        comms[0].flush()                               # the request was carried out all the same
        comms[0].wait(other)
        with torch.cuda.stream(other):
            mine = y[0].clone()
        torch.cuda.synchronize()
        want = float(it + 1) + (10.0 if n == 2 else 0.0)
        assert bool((mine == want).all()), (cid, it, mine[:4].tolist(), want)
        if n == 2:
            assert bool((seen == want).all()), (cid, it, seen[:4].tolist(), want)
        assert lib.cuStreamDestroy_v2(raw2) == 0
    # and the communicator goes on as before
    for t in x:
        t.fill_(1.0)
    with M.group():
        for r in range(n):
            comms[r].all_reduce(x[r], y[r])
    assert all(bool((t == float(n)).all()) for t in y)
    for c in comms:
        c.destroy()
M.finalize()
M.daemon.stop_embedded()
print("OK")
"""


def test_a_call_that_timed_out_gives_its_stream_back():
    """A call that ends without its answer leaves its request behind, but not the caller's stream: the stream can be
    destroyed, and the collective still runs behind what had been queued on it when the peers arrive."""
    import os
    import subprocess
    import sys

    from helpers import REPO
    p = subprocess.run([sys.executable, "-c", TIMED_OUT], env=dict(os.environ, PYTHONPATH=REPO, MCCS_WC_TIMEOUT_MS="300"),
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("OK"), p.stdout[-2000:] + p.stderr[-3000:]


@pytest.mark.parametrize("n", [1, 2])
def test_a_named_stream_under_capture_is_refused(service, n):
    """The refusal of graph capture looks at the stream the collective is given, not only at the current one."""
    M = service
    torch.cuda.set_device(0)
    cid, comms = fresh_comm_id(), [None] * n
    run_ranks(n, lambda r: comms.__setitem__(r, M.Communicator(cid, r, n, device=0)))
    bufs = [M.Buffer(4096, 0) for _ in range(n)]
    x = [b.tensor(torch.float32) for b in bufs]
    for t in x:
        t.fill_(1.0)
    scratch = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="relaxed")
        scratch.add_(1.0)
        with torch.cuda.stream(torch.cuda.Stream()):
            for c, t in zip(comms, x):
                with pytest.raises(M.MccsError, match="-9"):
                    c.all_reduce(t, stream=stream)
        graph.capture_end()
    with M.group():
        for c, t in zip(comms, x):
            c.all_reduce(t)
    graph.replay()
    torch.cuda.synchronize()
    assert all(bool((t == float(n)).all()) for t in x) and bool((scratch == 1.0).all())
    for c in comms:
        q = c.query()
        assert q["async_error"] == 0 and q["device_error"] == 0
        c.destroy()
