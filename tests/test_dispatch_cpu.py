"""CPU: the rules that pick a form for a call, and what they take into account besides sizes."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def in_a_process_of_its_own(code):
    """Settings of torch that cannot be taken back stay out of the other tests."""
    done = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.parametrize("setting,tf32", [
    ("m.fp32_precision = 'tf32'", True), ("m.allow_tf32 = True", True), ("torch.backends.fp32_precision = 'tf32'", True), ("m.allow_tf32 = True; m.fp32_precision = 'ieee'", False)])
def test_tf32_is_read_through_either_interface(setting, tf32):
    """The rule for f32 products reads the precision however a program has set it; torch's older getter raises after some of these."""
    in_a_process_of_its_own(f"import torch; from lit_llama_b200 import mixers; m = torch.backends.cuda.matmul\n{setting}\nassert mixers._tf32_products() is {tf32}")


def test_f32_products_of_no_entries_or_too_many_rows_stay_with_the_library():
    """Products that the tensor-core kernel refuses: a sum over nothing is zeros, and rows past its grid (16 * 65535) are products like others."""
    import torch
    from lit_llama_b200 import mixers

    w, rows = torch.empty(64, 256), 16 * 65535
    assert mixers._f32_sizes(torch.empty(rows, 256), w) and not mixers._f32_sizes(torch.empty(rows + 1, 256), w)
    assert not mixers._f32_sizes(torch.empty(1024, 0), torch.empty(1024, 0))


@pytest.mark.parametrize("rows,outputs,k,taken", [
    (256, 1024, 1024, True), (255, 1024, 1024, False), (8, 32768, 1024, True), (7, 65536, 1024, False), (256, 1024, 768, True), (256, 1024, 760, False),
    (272, 1024, 384, True), (8, 65536, 384, True), (8, 65536, 376, False), (48, 32000, 256, True), (47, 32000, 256, False), (272, 1024, 256, True),
    (74, 8192, 248, True), (73, 8192, 128, False), (100, 8200, 128, False), (586, 1024, 128, True), (4096, 4096, 120, False)])
def test_f32_products_on_both_sides_of_the_line(rows, outputs, k, taken):
    """Rows, k, results and products from which the tensor-core form is the faster one."""
    import torch
    from lit_llama_b200 import mixers

    assert mixers._f32_sizes(torch.empty(rows, k), torch.empty(outputs, k)) is taken


@pytest.mark.parametrize("x,w,taken", [
    ("wide[:, :1024]", "w", True), ("wide[:, 4:1028]", "w", True), ("wide[:, 2:1026]", "w", False), ("wide[:, :1020]", "w[:, :1020]", False),
    ("wide[:, :1024]", "w.t()", False), ("wide.t()[:300, :1024]", "w", False), ("odd[:, :1024]", "w", False), ("wide[:, :1024]", "odd[:, :1024]", False),
    ("wide[:1, :1024].expand(300, 1024)", "w", False), ("wide[:, :1024].double()", "w.double()", False), ("wide[:, :1024]", "w.bfloat16()", False), ("wide[0, :1024]", "w", False),
    ("wide[None, :, :1024]", "w", False), ("wide[:, :512]", "w", False)])
def test_f32_products_by_layout(x, w, taken):
    """Column slices on 16-byte boundaries are taken; other offsets, k not in groups of 8, transposed, repeated, broadcast and narrower operands are not."""
    import torch
    from lit_llama_b200 import mixers

    names = {"wide": torch.empty(1200, 1200), "w": torch.empty(1024, 1024), "odd": torch.empty(1024, 1029)}
    assert mixers._f32_sizes(eval(x, names), eval(w, names)) is taken


def test_calls_that_torch_follows_stay_with_torch():
    """Forward-mode derivatives, function transforms, tracing and modes see a product only where it is torch's; a default device does not count."""
    import torch
    from lit_llama_b200 import mixers
    from torch.utils.flop_counter import FlopCounterMode

    x, seen = torch.zeros(2, 2), []

    def look(t):
        seen.append(mixers._followed())
        return t + 1

    look(x)
    with torch.device("cpu"):
        look(x)
    assert seen == [False, False]
    with torch.autograd.forward_ad.dual_level():
        look(x)
    torch.vmap(look)(x)
    torch.jit.trace(look, x, check_trace=False)
    with FlopCounterMode(display=False):
        look(x)
    assert seen[2:] and all(seen[2:])


# ---------------------------------------------------------------------------- the engine's recorded portions, with the graph and the device stubbed
class _Model:
    vocab, dtype, portion_graph_safe, capture_layers = 8, None, True, None

    def __init__(self):
        import torch

        self.dtype, self.device = torch.float32, torch.device("cpu")
        self.weight = torch.ones(2)

    def state_specs(self):
        return {}

    def forward_portion(self, tokens, ctx, want=None):
        import torch

        return torch.full((0 if want is None else want.numel(), self.vocab), float(tokens.sum()) * float(self.weight[0]))


class _Graph:
    def __init__(self, body, log):
        self.body, self.log, self.out = body, log, body()
        log.append("recorded")

    def replay(self):
        self.log.append("replayed")
        self.out.copy_(self.body())


@pytest.fixture
def stubbed(monkeypatch):
    import torch
    from lit_llama_b200 import Engine, replay

    class Log(list):
        pass

    log = Log()

    def record(stream, pool, body):
        log.fails = getattr(log, "fails", 0) - 1
        if log.fails >= 0:
            raise RuntimeError("out of memory")
        g = _Graph(body, log)
        return g, g.out

    monkeypatch.setattr(replay, "record", record)
    monkeypatch.setattr(replay, "recording_stream", lambda *a: None)
    monkeypatch.setattr(torch.backends.cuda, "preferred_blas_library", lambda: 0)      # asks the driver
    for name, value in (("is_current_stream_capturing", False), ("synchronize", None), ("graph_pool_handle", (0, 1))):
        monkeypatch.setattr(torch.cuda, name, lambda *a, value=value, **k: value)
    return Engine(_Model(), n_slots=1, device="cpu"), log


def _feed(engine, T):
    out = engine.step([{"id": "r", "tokens": [1] * T, "want": [T - 1]}], end=["r"])[0]
    assert float(out[0, 0]) == T * float(engine.model.weight[0])


@pytest.mark.parametrize("lengths,random,recordings,replays", [(4, False, 4, 2980), (8, False, 4, 1480), (20, False, 4, 560), (50, False, 4, 200), (50, True, 6, 150)])
def test_mixed_lengths_are_not_recorded_again_and_again(stubbed, lengths, random, recordings, replays):
    """3000 portions of lengths in rotation or at random: a few recordings, and every portion of a length that has one is a replay."""
    import random as R

    engine, log = stubbed
    rng = R.Random(1)
    for i in range(3000):
        _feed(engine, 2 + (rng.randrange(lengths) if random else i % lengths))
    assert log.count("recorded") <= recordings and log.count("replayed") >= replays and len(engine._sightings.counts) <= 512


def test_a_length_that_comes_much_more_often_takes_a_graph_over(stubbed):
    """Four lengths with graphs, then one other alone: it has a graph within 200 portions, and the least frequent of the four has none."""
    engine, log = stubbed
    for i in range(100):
        _feed(engine, 2 + i % 4 if i % 5 else 2)
    assert log.count("recorded") == 4
    for _ in range(200):
        _feed(engine, 9)
    assert log.count("recorded") == 5 and (9, 1) in {k[:2] for k in engine._portions} and len(engine._portions) == 4
    engine.portion_graphs = 0
    _feed(engine, 11)


@pytest.mark.parametrize("T", [1, 7])
@pytest.mark.parametrize("fails", [1, 3])
def test_a_step_that_cannot_be_recorded_runs_eagerly(stubbed, T, fails):
    """A recording that fails leaves the eager step in its place, is tried again, and after three times no more."""
    engine, log = stubbed
    log.fails = fails
    for _ in range(12):
        _feed(engine, T)
    assert log.count("recorded") == (1 if fails == 1 else 0) and engine._failed_recordings == fails
    assert log.count("replayed") == (9 if fails == 1 else 0)


def test_portions_under_other_settings_are_not_replayed(stubbed, monkeypatch):
    """A model that refuses TF32 refuses it where its portion has a graph as well, and has the graph again when the setting is taken back."""
    import torch

    engine, log = stubbed
    run, m = type(engine.model).forward_portion, torch.backends.cuda.matmul

    def refusing(self, *a):
        if torch.backends.cuda.matmul.allow_tf32:
            raise RuntimeError("TF32")
        return run(self, *a)

    monkeypatch.setattr(_Model, "forward_portion", refusing)
    for _ in range(5):
        _feed(engine, 7)
    m.allow_tf32 = True
    try:
        with pytest.raises(RuntimeError, match="TF32"):
            _feed(engine, 7)
    finally:
        m.allow_tf32 = False
    before = log.count("replayed")
    engine.step([], end=["r"])
    _feed(engine, 7)
    assert before == 3 and log.count("replayed") == 4 and log.count("recorded") == 1


@pytest.mark.parametrize("change", ["m.weight = torch.full((2,), 3.0)", "m.weight.data = torch.full((2,), 3.0)", "m.layers[0].scale = 3.0", "m.layers[0] = m.Layer(3.0)",
                                    "m.layers[0].table['b'] = (torch.full((2,), 3.0),)", "m.layers.append(m.Layer(1.0))"])
def test_portions_with_other_weights_are_recorded_again(stubbed, change):
    """Tensors and values that a program has put in the place of those the model had, at any depth: the next portion has them, and recording begins anew.  New contents
    of the same tensor are no reason for one."""
    import torch

    class Layer:
        def __init__(self, scale):
            self.scale, self.table = scale, {"b": (torch.ones(2),)}

    engine, log = stubbed
    m = engine.model
    m.Layer, m.layers = Layer, [Layer(1.0)]
    for _ in range(5):
        _feed(engine, 7)
    m.weight.fill_(2.0)
    _feed(engine, 7)
    assert log.count("recorded") == 1 and log.count("replayed") == 4
    exec(change)
    for _ in range(5):
        _feed(engine, 7)
    assert log.count("recorded") == 2 and log.count("replayed") == 6


def test_attention_without_room_runs_the_form_that_needs_none(monkeypatch):
    """A portion in f32 asks for up to 128 MB it can do without: where that does not fit, the call is made without it."""
    import types

    import torch
    from lit_llama_b200 import _seqlib as S
    from lit_llama_b200 import mixers

    seen = []
    monkeypatch.setattr(S, "lib", lambda: types.SimpleNamespace(b2l_seq_block_attention_work_floats=lambda a: 1 << 20,
                                                                b2l_seq_block_attention=lambda a, s: seen.append((a._obj.work, a._obj.work_floats)) or 0))

    def none_left(*a, **k):
        raise torch.OutOfMemoryError("CUDA out of memory")

    monkeypatch.setattr(torch, "empty", none_left)
    mixers.local_attention(S.AttnArgs(), types.SimpleNamespace(meta=torch.zeros(2), stream=None))
    assert seen == [(None, 0)]


def test_an_owner_collected_while_a_stream_is_handed_out(monkeypatch):
    """Engines are collected at any moment, also while their thread takes a stream from the list: its stream is given back without waiting for itself."""
    import contextlib
    import threading

    import torch
    from lit_llama_b200 import replay

    class Owner:
        pass

    class Streams(dict):
        def get(self, key):
            gone.clear()                                     # the collector runs here
            return dict.get(self, key)

    gone, free = [Owner()], Streams()
    monkeypatch.setattr(replay, "_free", free)
    monkeypatch.setattr(torch.cuda, "device", lambda i: contextlib.nullcontext())
    monkeypatch.setattr(torch.cuda, "synchronize", lambda i: None)
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda at, device: at)
    free[0] = [11]
    first, taken = Owner(), []
    kept = gone[0]
    assert replay.recording_stream(kept, torch.device("cuda", 0)) == 11
    gone[:] = [kept]
    del kept
    free[0] = [12]
    t = threading.Thread(target=lambda: taken.append(replay.recording_stream(first, torch.device("cuda", 0))), daemon=True)
    t.start()
    t.join(20)
    assert not t.is_alive() and taken and sorted(free[0] + taken) == [11, 12]
