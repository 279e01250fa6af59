"""Fused steps of several decoders on one GPU take turns (their CTAs wait for one another, so two such kernels must not
share the device). On the CPU: who waits for what, over streams and events that keep a log and refuse what CUDA refuses.
On the GPU: decoders that step in threads of their own give what each gives alone."""

import contextlib
import functools
import threading
import time
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from cohere_inference_b200 import stream_decoder as sd

DEV = 97  # a device index no real decoder of this process has


class _Stream:
    def __init__(self):
        self.ops, self.waits, self.capturing = [], [], False

    def wait_event(self, ev):
        if ev.in_capture and not self.capturing:
            raise RuntimeError("an event of a capture: this stream would be pulled into it")
        if self.capturing and not ev.in_capture:
            raise RuntimeError("dependency created on uncaptured work in another stream")
        self.waits.append((ev.stream, ev.at))

    def synchronize(self):
        pass


class _Event:
    def __init__(self, *a, **k):
        self.stream, self.at, self.in_capture = None, 0, False

    def record(self, stream):
        self.stream, self.at, self.in_capture = stream, len(stream.ops), stream.capturing


@pytest.fixture
def decoders(monkeypatch):
    """make(fused buckets) -> a StreamDecoder without its GPU side: a step of bucket b appends b to its stream's log."""
    current = []

    @contextlib.contextmanager
    def on(stream):
        current.append(stream)
        yield
        current.pop()

    @contextlib.contextmanager
    def capture(graph, pool=None, stream=None):
        stream.capturing = True
        with on(stream):
            yield
        stream.capturing = False
    cuda = torch.cuda
    for name, fake in (("Event", _Event), ("stream", on), ("graph", capture), ("device", contextlib.nullcontext),
                       ("graph_pool_handle", lambda: None), ("CUDAGraph", SimpleNamespace),
                       ("is_current_stream_capturing", lambda: current[-1].capturing)):
        monkeypatch.setattr(cuda, name, fake)
    for name in ("range_push", "range_pop"):
        monkeypatch.setattr(cuda.nvtx, name, lambda *a: None)

    def make(fused):
        d = object.__new__(sd.StreamDecoder)
        d.stream, d.device, d.buckets = _Stream(), SimpleNamespace(index=DEV), (8, 128)
        d._fused_ws, d.use_graphs, d.graphs = dict.fromkeys(fused), False, {}
        d._fused_done = _Event()
        d.plan = SimpleNamespace(fused_ws=[b + 1 in fused or None for b in range(16)])
        d.reset = d.check_status = lambda: None
        d.during_capture = lambda: None

        def step(b):
            d.stream.ops.append(b if b > 16 or d.plan.fused_ws[b - 1] else (b, "kernel sequence"))
            if d.stream.capturing:
                d.during_capture()
        d._step = step
        return d
    yield make
    for table in (v for v in vars(sd.StreamDecoder).values() if isinstance(v, dict)):
        table.pop(DEV, None)


def test_a_step_during_another_decoders_capture_stays_out_of_it(decoders):
    """One decoder is built while another one serves, each in its own thread: between any two calls of the capture the
    other decoder may step."""
    serving, built = decoders((8,)), decoders((8,))
    serving.step(8)
    built.during_capture = lambda: serving.step(8)
    built._capture()
    assert serving.stream.ops == [8, 8, 8] and built.stream.ops == [128, 128, 8, 8]
    serving.step(8)
    assert built.stream.waits and not any(s is built.stream and at > 3 for s, at in serving.stream.waits)


def test_a_decoder_without_fused_steps_takes_no_turn(decoders):
    serving, other = decoders((8,)), decoders(())
    serving.step(8)
    other._capture()
    other.step(8)
    serving.step(8)
    assert not other.stream.waits and not serving.stream.waits


def test_a_turn_is_waited_for_up_to_the_fused_step_only(decoders):
    """What the other decoder has been given besides (its steps of 128 rows) goes on beside this one's."""
    a, b = decoders((8,)), decoders((8,))
    for bucket in (8, 8, 128, 128, 128):
        a.step(bucket)
    b.step(8)
    assert b.stream.waits == [(a.stream, 2)]
    b.step(8)
    b.step(128)
    assert len(b.stream.waits) == 1  # still its turn
    a.step(8)
    assert a.stream.waits == [(b.stream, 2)]


def test_a_step_inside_a_callers_capture_takes_no_turn_and_is_not_fused(decoders):
    """Nobody takes the turn when the caller's graph is replayed, so what it holds must not need one."""
    a, b = decoders((8,)), decoders((8,))
    a.step(8)
    with torch.cuda.graph(None, stream=b.stream):
        b.step(8)
        b.step(8)
    assert b.stream.ops == [(8, "kernel sequence")] * 2 and not b.stream.waits
    a.step(8)
    b.step(8)
    assert a.stream.ops == [8, 8] and b.stream.ops[2:] == [8] and not a.stream.waits
    assert b.stream.waits == [(a.stream, 2)]


# ---- on the GPU -----------------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=1)
def _model():
    from cohere_inference_b200.synth import synthetic_model
    return synthetic_model(3, layers=2, bias_std=0.05).cuda()


def _decoder(**kw):
    return sd.StreamDecoder(_model(), int8=True, max_new_tokens=64, max_prompt=16, max_audio_s=10.0, eos=-1, **kw)


def _admit(dec, seed, rows=8):
    """`rows` seeded requests of 48 new tokens each; returns the bucket."""
    rng = np.random.default_rng(seed)
    lens = rng.integers(20, 100, rows).tolist()
    memory = torch.from_numpy(rng.standard_normal((sum(lens), 1024)).astype(np.float32)).cuda()
    with torch.cuda.stream(dec.stream):
        dec.fill_cross(memory, lens, list(range(rows)))
    dec.admit(list(range(rows)), [torch.from_numpy(rng.integers(0, 16384, 8)) for _ in lens], lens, [48] * rows)
    return dec.set_active(list(range(rows)))


def _tokens(dec, rows=8):
    dec.check_status()
    return dec.out[:rows, :56].cpu().numpy()


@functools.lru_cache(maxsize=None)
def _alone(seed):
    dec = _decoder(slots=8, buckets=(8,))
    b = _admit(dec, seed)
    for _ in range(55):
        dec.step(b)
    return _tokens(dec)


@pytest.mark.gpu
def test_decoders_that_step_in_their_own_threads():
    decs = [_decoder(slots=8, buckets=(8,)) for _ in range(2)]
    buckets = [_admit(d, seed) for seed, d in enumerate(decs)]

    def serve(d, b):
        for _ in range(60):  # a row that has ended stays as it is
            d.step(b)
    threads = [threading.Thread(target=serve, args=a) for a in zip(decs, buckets)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for seed, d in enumerate(decs):
        assert d.launches(8) == 1 and np.array_equal(_tokens(d), _alone(seed))


@pytest.mark.gpu
def test_a_decoder_built_while_another_one_steps():
    first = _decoder(slots=8, buckets=(8,))
    b, stop = _admit(first, 0), threading.Event()

    def serve():
        while not stop.is_set():
            first.step(b)
            time.sleep(2e-4)
    t = threading.Thread(target=serve)
    t.start()
    try:
        second = _decoder(slots=16, buckets=(1, 2, 4, 8, 16))
    finally:
        stop.set()
        t.join()
    b2 = _admit(second, 1)
    for _ in range(55):
        first.step(b)
        second.step(b2)
    assert np.array_equal(_tokens(first), _alone(0)) and np.array_equal(_tokens(second), _alone(1))


@pytest.mark.gpu
def test_a_fused_step_does_not_wait_for_another_decoders_larger_steps():
    a, b = _decoder(slots=128, buckets=(8, 128)), _decoder(slots=8, buckets=(8,))
    small = _admit(b, 1)
    large = _admit(a, 0, rows=128)
    torch.cuda.synchronize()
    a.step(8)
    for _ in range(500):
        a.step(large)
    b.step(small)
    b.stream.synchronize()
    assert not a.stream.query()  # hundreds of its steps of 128 rows are still to come
    for _ in range(54):
        b.step(small)
    assert np.array_equal(_tokens(b), _alone(1))
    a.check_status()


@pytest.mark.gpu
def test_a_replay_inside_a_callers_capture_stays_refused():
    first, dec = _decoder(slots=8, buckets=(8,)), _decoder(slots=8, buckets=(8,))
    first.step(_admit(first, 1))
    b = _admit(dec, 0)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="during capturing stage"), torch.cuda.graph(torch.cuda.CUDAGraph(), stream=dec.stream):
        dec.step(b)
    for _ in range(55):
        first.step(b)
        dec.step(b)
    assert np.array_equal(_tokens(dec), _alone(0))


@pytest.mark.gpu
def test_a_callers_capture_holds_the_kernel_sequence():
    first, dec = _decoder(slots=8, buckets=(8,)), _decoder(slots=8, buckets=(8,), graphs=False)
    first.step(_admit(first, 1))  # the newest turn is another decoder's
    b = _admit(dec, 0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=dec.stream):
        dec.step(b)
    with torch.cuda.stream(dec.stream):
        for i in range(55):
            graph.replay() if i % 2 else dec.step(b)
    # the two ways round differently, so tokens may part where two logits are as good as equal: the first ones may not
    assert np.array_equal(_tokens(dec)[:, :16], _alone(0)[:, :16]) and int(dec.pos.sum()) == 8 * 55
