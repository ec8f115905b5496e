"""The functions of ``mccs_b200.ops`` on a communicator of one rank and ordinary CUDA tensors: one copy
kernel from tensor to tensor where that is the same as the staged form (copy into the communicator's
arena, collective there, copy out), the staged form everywhere else."""
import ctypes
import os
import subprocess
import sys

import pytest
import torch

from helpers import REPO, fresh_comm_id

pytestmark = pytest.mark.gpu


@pytest.fixture
def comm(service):
    torch.cuda.set_device(0)
    c = service.Communicator(fresh_comm_id(), 0, 1, device=0)
    yield c
    torch.cuda.synchronize()
    c.destroy()


def _collectives():
    from mccs_b200 import ops
    return [ops.all_reduce, ops.all_gather, ops.reduce_scatter]


@pytest.mark.parametrize("shift", [1, 3, 4, 4096, 999_999])
@pytest.mark.parametrize("count", [5, 1000, 1_000_003])
def test_tensors_that_overlap_in_part(comm, count, shift):
    """Shifted by ``shift`` elements in both directions, as if the input had been copied first; neighbours
    that only touch are no overlap."""
    for fn in _collectives():
        for up in (True, False):
            base = torch.arange(count + shift, dtype=torch.float32, device="cuda")
            lo, hi = base[:count], base[shift:]
            send, recv = (lo, hi) if up else (hi, lo)
            want = send.clone()
            rest = base[:shift].clone() if up else base[count:].clone()
            fn(comm, send, recv)
            assert torch.equal(recv, want), f"{fn.__name__} up={up}"
            kept = min(shift, count)       # what lies outside the output is untouched
            assert torch.equal(base[:kept] if up else base[-kept:], rest[:kept] if up else rest[-kept:])


def test_the_c_call_refuses_partial_overlap(comm):
    from mccs_b200 import _lib
    lib, x = _lib.shim(), torch.arange(4096, dtype=torch.uint8, device="cuda")
    assert lib.mccsCommTakesAnyMemory(comm._h) == 1
    stream = torch.cuda.current_stream().cuda_stream
    call = lambda a, b, n: lib.mccsCommSelfCopy(comm._h, x.data_ptr() + a, x.data_ptr() + b, n, stream)  # noqa: E731
    assert call(0, 1, 100) == -1 and call(1, 0, 100) == -1 and call(0, 99, 100) == -1
    assert call(0, 100, 100) == 0 and call(0, 0, 100) == 0
    torch.cuda.synchronize()
    assert torch.equal(x[100:200], x[:100]) and int(x[200]) == 200


GROUP = r"""
import os, sys, threading
import torch
import mccs_b200 as M
from mccs_b200 import ops

def check(comm, pause):
    # In each pass the input is a temporary whose block the allocator hands out again at once, and the
    # output is read within the group: both are right only if the input was read during the call.
    for fn in (ops.all_reduce, ops.all_gather, ops.reduce_scatter):
        for it in range(8):
            a = torch.full((1 << 20,), float(it + 1), device="cuda")
            out = torch.zeros(1 << 20, device="cuda")
            if pause and it == 0:
                pause()
            with M.group():
                t = a * 2
                at = t.data_ptr()
                fn(comm, t, out)
                del t
                b = torch.full((1 << 20,), -1.0, device="cuda")
                reused = b.data_ptr() == at
                seen = out.clone()
            torch.cuda.synchronize()
            assert bool((out == 2.0 * (it + 1)).all()) and bool((seen == out).all()), (fn.__name__, it, reused)

torch.cuda.set_device(0)
mode = sys.argv[1]
M.init(M.daemon.start_embedded(prefix=f"/tmp/mccs-group-{os.getpid()}", listen_port=-1,
                               extra='launch = "client"\nfuse_allreduce = 4' if mode == "client" else ""))
comm = M.Communicator(31, 0, 1, device=0)
assert comm.launch_mode == mode
def pause():       # the communicator answers nothing for a while
    assert M.daemon.embedded_admin({"cmd": "pause", "communicator_id": 31})["status"] == "ok"
    threading.Timer(0.2, lambda: M.daemon.embedded_admin({"cmd": "resume", "communicator_id": 31})).start()
check(comm, pause)
comm.destroy()
M.finalize()
M.daemon.stop_embedded()
print("OK")
"""


@pytest.mark.parametrize("mode", ["daemon", "client"])
def test_inside_a_group_the_input_is_read_during_the_call(mode):
    p = subprocess.run([sys.executable, "-c", GROUP, mode], env=dict(os.environ, PYTHONPATH=REPO), capture_output=True, text=True, timeout=300)
    assert p.returncode == 0 and p.stdout.strip().endswith("OK"), p.stdout[-2000:] + p.stderr[-3000:]


def test_views_whose_bytes_are_not_their_values(comm):
    """Negative views (lazy, contiguous) keep their sign as input and as output; a conjugate view cannot be
    gathered as bytes and is refused."""
    from mccs_b200 import ops
    x = torch.arange(1000.0, device="cuda")
    for fn in _collectives():
        if fn.__name__ != "all_gather":        # bytes of a negative view: refused like those of a conjugate one
            out = torch.zeros_like(x)
            fn(comm, torch._neg_view(x), out)
            assert torch.equal(out, -x)
            store = torch.zeros_like(x)
            fn(comm, x, torch._neg_view(store))
            assert torch.equal(store, -x)
    z = torch.randn(64, dtype=torch.complex64, device="cuda")
    for send in (z.conj(), torch._neg_view(x)):
        with pytest.raises(RuntimeError):
            ops.all_gather(comm, send, torch.empty_like(send))
    out = torch.empty_like(z)
    ops.all_gather(comm, z, out)               # without the view it is plain memory
    assert torch.equal(out, z)


def test_service_memory_is_named_to_the_daemon(service):
    """Two tensors in service memory go out as an ordinary collective, whose request keeps the allocations from
    being released while it waits; with a tensor of the caller's own it is the direct copy. (Seen at
    stand-ins for the C functions: nothing is launched.)"""
    from mccs_b200 import _lib
    mod, called = _lib.calls(), []
    gather = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_void_p] * 3, ctypes.c_size_t, ctypes.c_int, ctypes.c_void_p)(
        lambda c, s, d, n, algo, st: called.append(("gather", s, d, n)) or 0)
    copy = ctypes.CFUNCTYPE(ctypes.c_int, *[ctypes.c_void_p] * 3, ctypes.c_size_t, ctypes.c_void_p)(
        lambda c, s, d, n, st: called.append(("copy", s, d, n)) or 0)
    any_memory = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p)(lambda c: 1)
    torch.cuda.set_device(0)
    bufs = [service.Buffer(4096, 0) for _ in range(2)]
    a, b = (x.tensor(torch.float32) for x in bufs)
    short, x = bufs[1].tensor(torch.int16), torch.zeros(1024, device="cuda")
    try:
        _lib.bind_calls(mod, mccsAllGatherEx=gather, mccsCommSelfCopy=copy, mccsCommTakesAnyMemory=any_memory)
        calls = mod.CommCalls()
        calls._attach(1, 0, 1)
        assert calls.self_copy(a, b, None) is True and called.pop() == ("gather", a.data_ptr(), b.data_ptr(), 4096)
        assert calls.self_copy(a, x, None) is True and called.pop() == ("copy", a.data_ptr(), x.data_ptr(), 4096)
        assert calls.self_copy(x, b, None) is True and called.pop() == ("copy", x.data_ptr(), b.data_ptr(), 4096)
        assert calls.self_copy(bufs[0].tensor(torch.int16), short, None) is False and not called    # no collective of this type
    finally:
        _lib.bind_calls(mod)


def test_autograd_sees_the_write(comm):
    """What ``copy_`` into the output did: its version goes up (a tensor saved for backward that was overwritten
    is an error, not a wrong gradient), a leaf that requires grad is refused, gradients pass through."""
    x = torch.ones(1000, device="cuda")
    for fn in _collectives():
        a = torch.full((1000,), 3.0, device="cuda", requires_grad=True)
        b = a * 2
        y = (b * b).sum()
        version = b._version
        with torch.no_grad():
            fn(comm, x, b)
        assert b._version > version and torch.equal(b, x)
        with pytest.raises(RuntimeError, match="inplace operation"):
            y.backward()
        if fn.__name__ != "all_gather":        # (that one stores through a view of the bytes, which autograd does not follow)
            with pytest.raises(RuntimeError):
                fn(comm, x, a)
            assert bool((a == 3.0).all())
        with torch.no_grad():
            fn(comm, x, a)
        assert torch.equal(a.detach(), x)
        with torch.inference_mode():
            frozen = torch.zeros(1000, device="cuda")
            fn(comm, x, frozen)
            assert torch.equal(frozen, x)
        if fn.__name__ != "all_gather":
            with pytest.raises(RuntimeError, match="[Ii]nference"):
                fn(comm, x, frozen)
    from mccs_b200 import ops
    w = torch.ones(1000, device="cuda", requires_grad=True)
    out = torch.zeros(1000, device="cuda")
    (ops.all_reduce(comm, w * 5, out) * 2).sum().backward()
    assert torch.equal(w.grad, torch.full_like(w, 10.0))


def test_a_collective_given_another_stream(comm):
    """Input and output stay in the order of the current stream, however far behind the named one is."""
    side = torch.cuda.Stream()
    for it, fn in enumerate(_collectives()):
        recv = torch.zeros(1 << 20, device="cuda")
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)          # about 10 ms
        send = torch.full((1 << 20,), float(it + 1), device="cuda")
        fn(comm, send, recv, stream=side)
        seen = recv.clone()
        send.fill_(-1.0)
        torch.cuda.synchronize()
        assert bool((seen == float(it + 1)).all()) and torch.equal(recv, seen), fn.__name__


def test_unknown_names_are_refused(comm):
    from mccs_b200 import ops
    x, y = torch.ones(8, device="cuda"), torch.zeros(8, device="cuda")
    for fn in _collectives():
        with pytest.raises(KeyError):
            fn(comm, x, y, algo="no_such_kernel")
    for fn in (ops.all_reduce, ops.reduce_scatter):
        with pytest.raises(KeyError):
            fn(comm, x, y, op="no_such_operator")
    torch.cuda.synchronize()
    assert not bool(y.any())
