"""Pinned buffers whose copies PyTorch's host allocator does not hear of: nobody gets their memory while a copy is on its way."""
import gc

import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu

LONG = 300_000_000            # clock cycles: some 0.15 s of the stream


def _others(n):
    """Tensors that take whatever pinned memory of this size is free."""
    return [torch.full((n,), -1, dtype=torch.int32, pin_memory=True) for _ in range(6)]


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
