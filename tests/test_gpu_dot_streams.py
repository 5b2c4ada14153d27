"""Column dot products that one thread queues on two streams without waiting.

They overlap on the device, so each stream needs its own partial sums and ticket;
the sums run in a fixed order and equal those of calls one after another bit for
bit.  Many streams go through the bounded set of scratch buffers."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dot(torch, lib, x, y, out):
    assert lib.kmsd_column_dot(C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), x.shape[0], x.shape[1],
                               C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0


@pytest.mark.parametrize("streams,b", [(2, 16), (2, 3), (40, 8)])
def test_dots_on_several_streams_of_one_thread(cuda, streams, b):
    from kubomsd_b200 import _abi
    torch, lib = cuda, _abi.require_library()
    n = 200_000
    g = torch.Generator(device="cuda").manual_seed(streams)
    x, y = (torch.randn((n, b), dtype=torch.complex128, device="cuda", generator=g) for _ in range(2))
    xs = [x * (1 + i) for i in range(4)]
    want = torch.zeros((4, b), dtype=torch.complex128, device="cuda")
    for i in range(4):
        _dot(torch, lib, xs[i], y, want[i])
        torch.cuda.synchronize()
    ref = torch.stack([(v.conj() * y).sum(0) for v in xs])
    assert float((want - ref).abs().max()) <= 1e-10 * float(ref.abs().max() + n ** .5)
    got = torch.zeros((200, b), dtype=torch.complex128, device="cuda")
    pool = [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    for i in range(200):
        with torch.cuda.stream(pool[i % streams]):
            _dot(torch, lib, xs[i % 4], y, got[i])
    torch.cuda.synchronize()
    assert torch.equal(got, want.repeat(50, 1))


def test_captured_dot_after_calls_outside(cuda):
    """A capture allocates nothing: any earlier call of the thread that needed as much
    scratch is enough, on whatever stream; replays beside later calls are unchanged."""
    from kubomsd_b200 import _abi
    torch, lib = cuda, _abi.require_library()
    x, y = (torch.randn((50_000, 4), dtype=torch.complex128, device="cuda") for _ in range(2))
    want, got, other = (torch.zeros(4, dtype=torch.complex128, device="cuda") for _ in range(3))
    _dot(torch, lib, x, y, want)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _dot(torch, lib, x, y, got)
    big = torch.randn((60_000, 64), dtype=torch.complex128, device="cuda")
    for _ in range(3):
        got.zero_()
        graph.replay()
        _dot(torch, lib, big, big, torch.zeros(64, dtype=torch.complex128, device="cuda"))
        _dot(torch, lib, x, y, other)
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(other, want)
