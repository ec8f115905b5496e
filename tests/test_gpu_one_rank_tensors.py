"""The functions of ``mccs_b200.ops`` on a communicator of one rank and ordinary CUDA tensors: one copy
kernel from tensor to tensor where that is the same as the staged form (copy into the communicator's
arena, collective there, copy out), the staged form everywhere else."""
import pytest
import torch

from helpers import fresh_comm_id

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
