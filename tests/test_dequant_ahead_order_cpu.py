"""The order of the two-stream hand-over in ``linear.DequantAhead``, on a model of streams and events (no GPU).

Streams are lists of operations; an event remembers the operation it was recorded behind, and a wait makes everything launched later
on the waiting stream come after that. From these the test derives which operation is certain to finish before which, and asks it
of every pair that touches one buffer."""
from types import SimpleNamespace

import pytest
import torch

from owl_engine_b200.ops import linear
from owl_engine_b200.utils.ledger import DeviceLedger


_dense_scratch = linear._dense_scratch


class _Buffer(torch.Tensor):
    def record_stream(self, stream):
        pass


class _Ledger(DeviceLedger):
    def alloc(self, *a, **kw):
        return super().alloc(*a, **kw).as_subclass(_Buffer)


class _Model:
    """``drop``: the number of the wait that is left out (an oracle that must then find a race)."""

    def __init__(self, drop=None):
        self.drop, self.waits, self.before, self.touch = drop, 0, [], []
        model = self

        class Stream:
            def __init__(self, device=None):
                self.last, self.cuda_stream = None, self

            def wait(self, op):
                model.waits += 1
                if op is not None and model.waits - 1 != model.drop:
                    self.last = model.op([self.last, op])

            def wait_event(self, ev):
                self.wait(ev.at)

            def wait_stream(self, other):
                self.wait(other.last)

        class Event:
            at = None

            def record(self, stream):
                self.at = stream.last
        self.main = Stream()
        self.cuda = SimpleNamespace(Stream=Stream, Event=Event, current_stream=lambda device=None: self.main, current_device=lambda: 0,
                                    OutOfMemoryError=MemoryError, memory_allocated=lambda dev: 0,
                                    get_device_properties=lambda dev: SimpleNamespace(total_memory=1 << 40))

    def op(self, after):
        self.before.append(set().union(*({a} | self.before[a] for a in after if a is not None), set()))
        return len(self.before) - 1

    def run(self, stream, buffer, writes):
        stream.last = self.op([stream.last])
        self.touch.append((stream.last, buffer, writes))

    def races(self):
        out = []
        for i, (a, buf_a, wa) in enumerate(self.touch):
            for b, buf_b, wb in self.touch[:i]:
                if buf_a == buf_b and (wa or wb) and b not in self.before[a]:
                    out.append((b, a))
        return out


def _run(monkeypatch, drop=None, streams=False):
    m = _Model(drop)
    led = _Ledger("cpu")

    class Torch:
        cuda = m.cuda

        def __getattr__(self, name):
            return getattr(torch, name)
    monkeypatch.setattr(linear, "torch", Torch())
    monkeypatch.setattr(linear, "ledger_for", lambda dev: led)
    monkeypatch.setattr(linear, "_scratch", {})
    monkeypatch.setattr(linear, "_ahead", {})
    monkeypatch.setattr(linear, "_dense_scratch", lambda n, k, device, dtype, scratch=_dense_scratch: scratch(n, k, "cpu:0", dtype))
    monkeypatch.setattr(linear.K, "w4_dequant", lambda w, out, on=None: m.run(m.main if on is None else on, out.data_ptr(), True) or out)
    monkeypatch.setattr(linear.gemm_tc, "f16_gemm", lambda x, w, out: m.run(m.main, w.data_ptr(), False) or out)
    ws = [SimpleNamespace(n=n, k=16, layout="slice") for n in (64, 32, 64, 16, 48)]
    ahead = linear.DequantAhead("cpu:0")
    x, out = torch.empty(300, 16, dtype=torch.float16), torch.empty(300, 64, dtype=torch.bfloat16)
    for chunk in range(3):
        if streams and chunk:
            m.main = m.cuda.Stream()                              # every chunk on a stream of its own
        assert ahead.start(ws)
        for w in ws:
            linear.w4_gemm(w, x, out, ahead=ahead)
    assert ahead.start(ws)                                        # a chunk that ends after two projections ...
    for w in ws[:2]:
        linear.w4_gemm(w, x, out, ahead=ahead)
    for w in ws[2:]:                                              # ... and the scratch's next users
        linear.w4_gemm(w, x, out)
    assert m.touch and len({b for _, b, _ in m.touch}) == 2
    return m


@pytest.mark.parametrize("streams", [False, True])
def test_every_use_of_a_buffer_is_ordered(monkeypatch, streams):
    assert not _run(monkeypatch, streams=streams).races()


def test_the_model_sees_a_missing_wait(monkeypatch):
    """Leaving out one wait at a time: the race it opens is seen, but for the waits that others cover: the very first, which has
    nothing before it, and in each of the four chunks that before the second dequantisation (its buffer's last product lies before
    the chunk, and the first dequantisation has waited for that)."""
    n = _run(monkeypatch).waits
    seen = [bool(_run(monkeypatch, drop=i).races()) for i in range(n)]
    assert sum(seen) == n - 5, seen
