"""The drop-in `run(...)` where no GPU is needed: how it sets up and shares its handles."""
import contextlib
import re
import threading
import time
from pathlib import Path
from types import SimpleNamespace

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def test_option_matches_the_header(pkg):
    txt = (ROOT / "include" / "moe_fp8_b200.h").read_text()
    value = re.search(r"MOE_FP8_B200_OPT_SCALES_IN_PLACE\s*=\s*(\d+)", txt).group(1)
    assert int(value) == pkg._lib.OPT_SCALES_IN_PLACE


class FakeStream:
    def __init__(self, log, name, stream_id, capturing=False):
        self.log, self.name, self.stream_id, self.capturing = log, name, stream_id, capturing
        self.cuda_stream = 1000 + stream_id

    def wait_stream(self, other):
        self.log.append(f"{self.name} behind {other.name}")

    def wait_event(self, event):
        self.log.append(f"{self.name} behind {event}")

    def record_event(self):
        self.log.append(f"event on {self.name}")
        return f"event of {self.name}"


class FakeTensor:
    is_cuda, device = True, SimpleNamespace(index=0)

    def __init__(self, *shape):
        self.shape = shape


class FakeLayer:
    """Stands in for MoeLayer; a handle is not thread-safe, so neither is this."""
    pause = 0.0

    def __init__(self, log, max_tokens):
        self.log, self.max_tokens, self.inside, self.overlaps = log, max_tokens, 0, 0

    def set_scales_in_place(self, on):
        pass

    def run(self, *args, stream=None):
        self.inside += 1
        self.overlaps += self.inside != 1
        time.sleep(self.pause)
        self.log.append("run")
        self.inside -= 1

    def close(self):
        self.overlaps += self.inside != 0
        self.log.append("close")


@pytest.fixture
def fakes(pkg, monkeypatch):
    """(call the drop-in `run` with T tokens on a stream, log, layers made)"""
    from fp8_moe_dev_b200 import op
    log, made, here = [], [], threading.local()

    def make(max_tokens, *rest):
        made.append(FakeLayer(log, max_tokens))
        return made[-1]

    @contextlib.contextmanager
    def on(stream):
        before, here.stream = here.stream, stream
        yield
        here.stream = before

    monkeypatch.setattr(op, "_layers", {})
    monkeypatch.setattr(op, "MoeLayer", make)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: here.stream)
    monkeypatch.setattr(torch.cuda, "stream", on)
    monkeypatch.setattr(op, "_raw_stream", lambda dev: here.stream.cuda_stream, raising=False)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: here.stream.capturing)

    def call(stream, T=16):
        here.stream = stream
        pkg.run(FakeTensor(T, 256), None, None, None, FakeTensor(32, 1, 1), None, None, None, 0, 2.5, None)

    return call, log, made


def test_streams_take_turns(fakes):
    call, log, made = fakes
    default, own, foreign = FakeStream(log, "default", 0), FakeStream(log, "own", 3), FakeStream(log, "foreign", 64)
    graph = FakeStream(log, "graph", 5, capturing=True)
    for s in (default, default, own, foreign, foreign, default, graph, default):
        call(s)
    assert log == ["run", "run", "own behind default", "run", "foreign behind own", "run", "event on foreign", "run",
                   "event on foreign", "default behind event of foreign", "run", "run", "run"]
    log.clear()
    graph.capturing = False
    call(graph)
    call(own, T=17)   # a larger batch: the old handle's end waits for the device, nothing else to wait for
    assert log == ["graph behind default", "run", "close", "run"] and len(made) == 2


def test_threads_take_turns(fakes):
    call, log, made = fakes
    FakeLayer.pause = 0.0005
    try:
        def work(i):
            stream = FakeStream([], f"s{i}", 2 * i + 1)
            for k in range(20):
                call(stream, T=16 + 8 * (i % 3) + k)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    finally:
        FakeLayer.pause = 0.0
    assert log.count("run") == 120 and sum(layer.overlaps for layer in made) == 0
    assert log.count("close") == len(made) - 1
