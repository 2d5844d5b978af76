"""spgemm_batched_raw's order of host calls with device operands: the arrays
that torch has to copy (strided ones) are copied on torch's stream, so the wait
for that stream has to come after the last copy of all instances of A and B and
before the library reads them.  On the CPU with stand-ins for the tensors,
torch's stream and the library."""
import pytest
import torch

from tilespgemm_gb300 import _abi, api


class _Tensor:
    """A device array that notes when torch would queue a copy of it."""
    is_cuda = True

    def __init__(self, events, name, dtype, n, strided, device="cuda:0"):
        self.events, self.name, self.dtype, self.n, self.strided, self.device = events, name, dtype, n, strided, device
        self.shape = (n,)

    def contiguous(self):
        if self.strided:
            self.events.append(("copy", self.device))
        return self

    def numel(self):
        return self.n

    def data_ptr(self):
        return 4096


class _Lib:
    def __init__(self, events):
        self.events = events

    def tsg_spgemm_batched(self, *a):
        self.events.append(("call", None))
        return _abi.OK

    def tsg_stream_wait(self, *a):
        self.events.append(("wait", "cuda:0"))
        return _abi.OK


@pytest.mark.parametrize("op", ["AA", "AB"])
@pytest.mark.parametrize("strided", [(0,), (1,), (3,), (0, 1, 3), ()])
@pytest.mark.parametrize("devices", [1, 2])
def test_no_copy_after_the_last_wait(monkeypatch, op, strided, devices):
    events = []

    class Stream:
        def __init__(self, device):
            self.device, self.cuda_stream = device, 0

        def synchronize(self):
            events.append(("wait", self.device))

    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: Stream(device))
    monkeypatch.setattr(api, "lib", lambda: _Lib(events))
    ctx = object.__new__(api.Context)
    ctx.handle = None

    def matrix(i):
        dev = f"cuda:{i % devices}"
        s = i in strided
        return api.CSR(4, 4, _Tensor(events, "rp", torch.int64, 5, s, dev), _Tensor(events, "col", torch.int32, 4, s, dev),
                       _Tensor(events, "val", torch.float64, 4, s, dev))

    ctx.spgemm_batched_raw([matrix(i) for i in range(4)], [matrix(i) for i in range(4)] if op == "AB" else None, op=op)
    kinds = [k for k, _ in events]
    assert kinds.count("call") == 1 and kinds[-1] == "call"
    assert kinds.count("copy") == 3 * len(strided) * (2 if op == "AB" else 1)
    for d in {f"cuda:{i}" for i in range(devices)}:
        waits = [t for t, e in enumerate(events) if e == ("wait", d)]
        assert waits, "operands of this device were never waited for"
        assert all(t < waits[-1] for t, e in enumerate(events) if e == ("copy", d))
