"""Host side of the operators' grouped kernels: scratch, remembered facts, refusals (no GPU)."""

import contextlib
import ctypes
from types import SimpleNamespace

import torch


def test_calls_in_flight_together_do_not_share_scratch(monkeypatch):
    """A second call of the same shape on the same stream, made while the first is still enqueueing
    its launches (another host thread: the library call releases the interpreter lock), must not
    be handed the first one's scratch.  The library is a stand-in that makes that second call."""
    from keep_b200 import _lib, prefill

    nbytes, seen = 4096, []
    rows = torch.zeros((2, 256), dtype=torch.bfloat16)
    codes, scales = torch.zeros((1, 32, 32), dtype=torch.uint16), torch.ones((1, 32, 1), dtype=torch.float16)
    table, rhs = torch.full((256,), 0x11111111, dtype=torch.int32), torch.zeros(2, dtype=torch.int32)

    def project(args, stream):
        first = not seen
        seen.append(ctypes.cast(args.workspace, ctypes.c_void_p).value)
        assert args.workspace_bytes >= nbytes
        if first:
            assert prefill.tensor_core_projection(rows, codes, scales, table, rhs) is not None
        return 0

    fake = SimpleNamespace(keepvq_grouped_projection=project)
    monkeypatch.setattr(_lib, "load", lambda: fake)
    monkeypatch.setattr(prefill, "_scratch_bytes", lambda routes, in_dim: nbytes)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    prefill.tensor_core_projection(rows, codes, scales, table, rhs)
    assert len(seen) == 2 and abs(seen[0] - seen[1]) >= nbytes


def test_the_answer_about_a_table_survives_an_eviction(monkeypatch):
    """Whether a table's nibbles are all odd is remembered for a few tables; another thread may evict
    the entry between its insertion and the answer."""
    from keep_b200 import prefill

    class Forgetful(dict):
        def __setitem__(self, key, value):
            pass

    monkeypatch.setattr(prefill, "_all_odd", Forgetful())
    assert prefill._table_all_odd(torch.full((256,), 0x11111111, dtype=torch.int32)) is True
    assert prefill._table_all_odd(torch.full((256,), 0x11111112, dtype=torch.int32)) is False


def test_a_call_that_the_library_will_refuse_prepares_nothing(monkeypatch):
    """8-bit calls of few routes belong to the general kernel: neither scratch nor outputs are
    allocated, nor the library called, to find that out."""
    from keep_b200 import prefill

    rows, codes = torch.zeros((6, 256), dtype=torch.bfloat16), torch.zeros((64, 32, 32), dtype=torch.uint8)
    scales, table, rhs = torch.ones((64, 32, 1), dtype=torch.float16), torch.zeros(256, dtype=torch.int32), torch.zeros(6, dtype=torch.int32)

    def prepared(*args, **kwargs):
        raise AssertionError("prepared a call")

    monkeypatch.setattr(torch.cuda, "current_stream", prepared)
    monkeypatch.setattr(torch, "empty", prepared)
    assert prefill.tensor_core_projection(rows, codes, scales, table, rhs, code_bits=8) is None


def test_the_routes_of_a_single_matrix_outlive_any_caller(monkeypatch):
    """The expert indices of a single matrix's routes belong to no caller, stream or tracer: a call made
    under a tracing mode (or on a stream that is gone) must not leave its own behind for the next."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    from keep_b200 import _lib, kernels, prefill

    held, seen = (ctypes.c_uint32 * 64)(), []

    def zero_routes(address, count):
        address._obj.value, count._obj.value = ctypes.addressof(held), 64
        return 0

    def project(rows, routes, *rest, **named):
        seen.append(rest[7])
        return torch.empty(routes)

    monkeypatch.setattr(_lib, "load", lambda: SimpleNamespace(keepvq_zero_routes=zero_routes))
    monkeypatch.setattr(prefill, "project", project)
    monkeypatch.setattr(kernels, "_zero_routes", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())

    def call(routes):
        rows = torch.zeros((routes, 256), dtype=torch.bfloat16)
        codes, scales = torch.zeros((32, 32), dtype=torch.uint16), torch.ones((32, 1), dtype=torch.float16)
        kernels._one_matrix(rows, codes, scales, torch.zeros(256, dtype=torch.int32), 16, (routes, 32))
        return seen[-1]

    with FakeTensorMode():
        call(3)
    rhs = call(3)
    assert rhs.data_ptr()
    assert list((ctypes.c_uint32 * 3).from_address(rhs.data_ptr())) == [0, 0, 0]
    assert call(65).numel() == 65 and not call(65).any()  # more than the library holds
