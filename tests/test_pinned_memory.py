"""Pinned buffers whose copies PyTorch's host allocator does not hear of: nobody gets their memory while a copy is on its way."""
import contextlib
import gc
import types

import pytest
import torch

import helpers

LONG = 300_000_000            # clock cycles: some 0.15 s of the stream


def _others(n):
    """Tensors that take whatever pinned memory of this size is free."""
    return [torch.full((n,), -1, dtype=torch.int32, pin_memory=True) for _ in range(6)]


@pytest.mark.gpu
def test_a_buffer_that_goes_waits_for_its_last_copy():
    from pulsar_b200 import ops
    values = torch.arange(72, dtype=torch.int32, device="cuda")
    buf = ops.Pinned(72, torch.int32)
    torch.cuda._sleep(LONG)
    buf.from_device(values, 72)
    del buf
    others = _others(72)
    torch.cuda.synchronize()
    assert all(bool((t == -1).all()) for t in others)


@pytest.mark.gpu
def test_a_buffer_is_read_and_written_in_the_stream():
    from pulsar_b200 import ops
    buf, dev = ops.Pinned(8, torch.int32), torch.zeros(8, dtype=torch.int32, device="cuda")
    buf.host[:] = torch.arange(8, dtype=torch.int32)
    buf.to_device(dev, 5)
    dev += 10
    buf.wait()
    buf.from_device(dev, 3)
    buf.wait()
    assert buf.host.tolist() == [10, 11, 12, 3, 4, 5, 6, 7] and dev.tolist() == [10, 11, 12, 13, 14, 10, 10, 10]


@pytest.mark.gpu
def test_an_engine_that_goes_with_a_pass_in_flight(tmp_path):
    """``step`` returns with the next pass on the device; its report lands in memory that is nobody else's."""
    from pulsar_b200.engine.engine import Engine
    raw, seed, page = helpers.TINY["B"]
    helpers.make_folder(str(tmp_path), raw, seed)
    eng = Engine(str(tmp_path), dict(dtype="float32", page_size=page, num_pages=32, max_sessions=2, max_running=2, max_chunk_size=8,
                                     device="cuda:0", eos_id=-1))
    draw = eng.sampler.sample_on_device

    def slow(*args, **kw):
        torch.cuda._sleep(LONG)
        return draw(*args, **kw)
    eng.sampler.sample_on_device = slow
    eng.feed(eng.create_session([3, 14, 15]), [], 8)
    assert len(eng.step(1)) == 1 and eng._inflight is not None
    del eng, draw, slow
    gc.collect()
    others = _others(72)
    torch.cuda.synchronize()
    assert all(bool((t == -1).all()) for t in others)


@pytest.mark.parametrize("current", [0, 1])
def test_copies_are_in_the_stream_of_the_tensors_device(current, monkeypatch):
    """A runner on one device while another is the current one (the CUDA calls are the test's own)."""
    from pulsar_b200 import ops
    at, copies, marks = [current], [], []

    @contextlib.contextmanager
    def device(where):
        before, at[0] = at[0], where.index
        yield
        at[0] = before
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(ops, "_device", lambda: at[0])
    monkeypatch.setattr(ops, "_raw_stream", lambda index: 100 + index)
    monkeypatch.setattr(ops, "current_stream", lambda: 100 + at[0])
    monkeypatch.setattr(ops, "fn", lambda name: lambda *args: copies.append((name, at[0], args[-1])) or 0)
    buf = ops.Pinned.__new__(ops.Pinned)
    buf.host = torch.zeros(8, dtype=torch.int32)
    buf.event = types.SimpleNamespace(record=marks.append, synchronize=lambda: None)
    dev = types.SimpleNamespace(is_cuda=True, device=torch.device("cuda:1"), dtype=torch.int32, numel=lambda: 8, is_contiguous=lambda: True,
                                data_ptr=lambda: 4096, element_size=lambda: 4)
    buf.to_device(dev, 8)
    buf.from_device(dev, 4)
    assert copies == [("pb_copy", 1, 101)] * 2 and marks == [101, 101] and at[0] == current
