"""Decode steps replayed from CUDA graphs (llm_decoder.engine.DecodeSteps) against the same steps run launch by launch: the same
kernels on the same numbers, so the logits agree to the last bit except where a kernel's work split depends on the bound of the
lengths (bfloat16 sums in another order: 2e-2 of the logits' spread, as for this precision elsewhere)."""
import random

import pytest
import torch

from oracle import domilix_ref, dubarax_ref, gunulorn_ref, hybrid_ref, namudra_ref, tiradra_ref


def _pair(config, W, **kw):
    """Two engines over equal models; the second never captures."""
    import llm_decoder as ld
    a, b = (ld.Engine(ld.HybridDecoder(config, W, "bfloat16", **kw)) for _ in range(2))
    a._decode.PATIENCE = 2
    b._decode.serves = lambda *_a: False
    return a, b


def _config(name):
    if name == "tiradra":
        R = tiradra_ref
        c = R.make_config([R.attention_layer(dim=64, heads=4, kv_heads=2), R.latent_layer()], loop={"start": 0, "stop": 2, "times": 2})
    elif name == "namudra":
        R = namudra_ref
        c = R.make_config([R.retention_layer(ff=32)], streams=2)
    else:
        R = dubarax_ref
        c = R.make_config([R.attention_layer(mlp=R.moe_mlp()), R.mamba_layer(mlp=R.moe_mlp())])
    return c, R.random_weights(c, 3)


def _close(x, y):
    assert torch.isfinite(x).all() and (x - y).abs().max() < 2e-2 * y.abs().max(), (x - y).abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["tiradra", "namudra", "dubarax"])
def test_replayed_steps_equal_launched_ones(name):
    """Requests of unequal length decode together, some end and others take their slots, the number of sequences changes, a step is
    skipped by one of them, and the lengths cross the bound of 256."""
    config, W = _config(name)
    a, b = _pair(config, W, max_tokens=2048, max_seqs=4)
    g = torch.Generator().manual_seed(1)
    tok = lambda n=1: torch.randint(0, config["vocab"], (n,), generator=g).tolist()  # noqa: E731
    both = lambda entries: (a.step(entries), b.step(entries))  # noqa: E731
    _close(*both([(0, tok(7), [6]), (1, tok(250), [249]), (2, tok(1), [0])]))
    for k in range(12):
        _close(*both([(i, tok(), [0]) for i in (0, 1, 2)]))
    assert a._decode._graphs
    for e in (a, b):
        e.finish(0)
    _close(*both([(3, tok(30), [29]), (1, tok(), [0])]))            # a prompt beside a decoded token: launched
    for k in range(4):
        _close(*both([(i, tok(), [0]) for i in (3, 1, 2)]))         # the slot of request 0
        _close(*both([(i, tok(), [0]) for i in (2, 3)]))
        x, y = both([(i, tok(), [0] if i == 2 else []) for i in (2, 3)])
        assert x.shape[0] == 1
        _close(x, y)
    with pytest.raises(ValueError):
        a.step([(2, [1], [1])])


@pytest.mark.gpu
def test_replaced_weights_hooks_and_streams():
    """A weight replaced by another tensor, or given other storage, is seen by the next step; results of earlier steps stay; steps on
    changing streams keep their order; a hook makes steps run launch by launch."""
    config, W = _config("tiradra")
    a, b = _pair(config, W, max_tokens=512, max_seqs=2)
    step = lambda t: (a.step([(0, [t], [0]), (1, [t + 1], [0])]), b.step([(0, [t], [0]), (1, [t + 1], [0])]))  # noqa: E731
    first = [step(t) for t in range(4)]
    kept = [x.clone() for x, _y in first]
    for m in (a.model, b.model):
        m.head = m.head * 0.5
    x, y = step(5)
    _close(x, y)
    for _ in range(4):
        _close(*step(6))
    for m in (a.model, b.model):
        m.head.data = m.head.data * 3.0
    for _ in range(4):
        _close(*step(7))
    for m in (a.model, b.model):
        m.head.mul_(0.25)                       # in place: the graph reads the new numbers
    _close(*step(8))
    assert all(torch.equal(p, x) for p, (x, _y) in zip(kept, first))
    s = torch.cuda.Stream()
    for k in range(6):
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s if k % 2 else torch.cuda.current_stream()):
            _close(*step(9 + k))
        torch.cuda.current_stream().wait_stream(s)
    calls = []
    a.model.layer_hook = b.model.layer_hook = lambda x: calls.append(1)
    _close(*step(20))
    assert calls


@pytest.mark.gpu
def test_functions_in_place_of_methods_and_failed_captures():
    """A method replaced on the instance is called in every step; a capture that fails leaves the step to launches."""
    config, W = _config("tiradra")
    a, b = _pair(config, W, max_tokens=256, max_seqs=1)
    calls, real = [], a.model._linear
    a.model._linear = lambda *args, **kw: (calls.append(1), real(*args, **kw))[1]
    for k in range(6):
        n = len(calls)
        _close(a.step([(0, [k], [0])]), b.step([(0, [k], [0])]))
        assert len(calls) > n
    del a.model._linear

    def fails(*_a):
        raise RuntimeError("no capture")
    a._decode._capture = fails
    for k in range(6):
        _close(a.step([(0, [k + 9], [0])]), b.step([(0, [k + 9], [0])]))
    assert not a._decode._graphs


def _design(name):
    """A model of every design, with the head sizes of the shared-out kernels where the design has such layers, and without."""
    if name == "megusun":
        R = hybrid_ref
        c = R.make_config([R.attention_layer(mlp=R.moe_mlp()), R.mingru_layer(mlp=R.dense_mlp())])
    elif name == "domilix":
        R = domilix_ref
        c = R.make_config([R.latent_layer(mlp=R.dense_mlp()), R.latent_layer(heads=20, dim=16, rot_dim=16, kv_rank=128, mlp=R.moe_mlp()),
                           R.latent_layer(kv_from=0, mlp=R.dense_mlp())])
    elif name == "gunulorn":
        R = gunulorn_ref
        c = R.make_config([R.conv_layer(dim=64, vdim=128, mlp=R.dense_mlp()), R.window_layer(dim=64, vdim=64, mlp=R.moe_mlp()),
                           R.conv_layer(mlp=R.dense_mlp())])
    elif name == "dubarax":
        R = dubarax_ref
        c = R.make_config([R.attention_layer(dim=64, vdim=64, window=300, mlp=R.moe_mlp()), R.parallel_layer(mlp=R.moe_mlp()), R.mamba_layer(mlp=R.moe_mlp())])
    elif name == "namudra":
        R = namudra_ref
        c = R.make_config([R.window_layer(), R.latent_layer(), R.latent_layer(dim=16, rot_dim=16, kv_rank=256), R.retention_layer(dim=64, vdim=64)])
    else:
        R = tiradra_ref
        c = R.make_config([R.attention_layer(dim=128, heads=4, kv_heads=2), R.latent_layer(dim=16, rot_dim=16, kv_rank=128), R.latent_layer()])
    return c, R.random_weights(c, 5)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["megusun", "domilix", "dubarax", "gunulorn", "namudra", "tiradra"])
def test_a_replayed_step_gives_the_bits_of_a_launched_one(name):
    """A request's logits do not depend on how many steps of a kind the engine has run: contexts of unequal length, past the bounds from
    which kernels cut their keys, growing over a multiple of 256 and of 512."""
    config, W = _design(name)
    a, b = _pair(config, W, max_tokens=4096, max_seqs=4)
    a._decode.GAP = 0
    g = torch.Generator().manual_seed(2)
    tok = lambda n=1: torch.randint(0, config["vocab"], (n,), generator=g).tolist()  # noqa: E731
    both = lambda entries: (a.step(entries), b.step(entries))  # noqa: E731
    both([(0, tok(762), [761]), (1, tok(90), [89]), (2, tok(20), [19]), (3, tok(506), [505])])
    replays = 0
    for ids in ((0, 1, 2), (3,), (3, 1)):
        for k in range(12):
            x, y = both([(i, tok(), [0]) for i in ids])
            assert torch.equal(x, y), (ids, k, (x - y).abs().max())
        replays += sum(k[0] == len(ids) for k in a._decode._graphs)
    assert replays >= 3


class _Held:
    """Stands in for streams, events, graphs and batches: takes every call and has every attribute."""
    rows = 1

    def __getattr__(self, _name):
        return _Held()

    def __call__(self, *_a, **_kw):
        return _Held()

    def __enter__(self):
        return self

    def __exit__(self, *_exc):
        return False


def _host_only(monkeypatch):
    """DecodeSteps over stand-ins: its bookkeeping without a GPU.  The current stream is steps.on, captures are noted in steps.noted."""
    from llm_decoder import engine
    steps = engine.DecodeSteps(_Held())
    steps.on, steps.noted, steps.now = _Held(), [], 0
    monkeypatch.setattr(torch.cuda, "Event", lambda *_a: _Held())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *_a: steps.on)
    monkeypatch.setattr(engine, "DecodeBatch", lambda *_a: _Held())
    steps.model.device, steps.model.runs = torch.device("cpu"), []
    st = steps.model.states = _Held()
    st.length, st.advance, st._tables, st.track_tokens = lambda _s: 100, lambda _e: (), [], False
    steps._lane = _Held()
    steps._watched = lambda: ([], ())
    steps._same = lambda _w: True
    steps._capture = lambda g, _stream: (steps.noted.append(steps.now), g.update(graph=_Held(), logits=torch.zeros(1), want=None, watched=None))
    return steps


@pytest.mark.parametrize("kinds", [9, 21, 64])
@pytest.mark.parametrize("order", ["in turn", "at random", "walk"])
def test_captures_of_many_kinds_are_few(monkeypatch, kinds, order):
    """Numbers of sequences that change from step to step, more of them than graphs are kept: a capture costs up to 30 launched steps, so
    no more than one in 64 steps captures, none where the kept ones keep coming back, and kept ones are replayed."""
    steps = _host_only(monkeypatch)
    r, n, replayed = random.Random(3), kinds // 2, 0
    for steps.now in range(6000):
        if order == "in turn":
            n = steps.now % kinds
        elif order == "at random":
            n = r.randrange(kinds)
        elif r.random() < 0.2:
            n = min(max(n + r.choice((-1, 1)), 0), kinds - 1)
        replayed += steps.step([(i, [0]) for i in range(n + 1)]) is not None
    caught = steps.noted
    assert len(steps._graphs) <= steps.MOST
    assert order != "in turn" or len(caught) == steps.MOST
    assert all(b - a >= 64 for a, b in zip(caught, caught[1:])), caught
    assert replayed > 6000 * min(1.0, steps.MOST / kinds) * 0.5, replayed


def test_replays_of_an_engine_follow_one_another(monkeypatch):
    """All graphs of an engine share the scratch of the stream they were captured on: a replay waits for the last one on another stream,
    of whatever kind, and the buffers a replay reads are kept for the streams that replay."""
    from llm_decoder import engine
    steps = _host_only(monkeypatch)
    steps.PATIENCE = steps.GAP = 0
    log, held = [], []

    class Stream:
        def wait_event(self, event):
            log.append(("wait", self, event.by))

    class Event:
        by = None

        def record(self, stream):
            self.by = stream

    class Batch(_Held):
        def __init__(self, *_a):
            self.streams = []
            held.append(self)

        def used_on(self, stream):
            self.streams.append(stream)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(engine, "DecodeBatch", Batch)
    lane = object.__new__(engine._Lane)
    lane.side, lane.lock, lane._event, lane._stream = _Held(), _Held(), Event(), None
    steps._lane = lane
    a, b = Stream(), Stream()
    for steps.on, n in ((a, 1), (a, 2), (b, 1), (b, 1), (b, 2), (a, 2), (a, 1)):
        assert steps.step([(i, [0]) for i in range(n)]) is not None
    assert log == [("wait", b, a), ("wait", a, b)]
    assert held[0].streams == [a, b, a] and held[1].streams == [a, b, a]


@pytest.mark.gpu
def test_capture_streams_are_nobody_elses():
    """No stream that a program gets is one that graphs were captured on, and engines capture on different ones."""
    config, W = _config("tiradra")
    sides = []
    for _ in range(3):
        a, b = _pair(config, W, max_tokens=64, max_seqs=1)
        for k in range(5):
            _close(a.step([(0, [k], [0])]), b.step([(0, [k], [0])]))
        sides.append(a._decode._lane.side.cuda_stream)
    assert len(set(sides)) == 3
    assert not set(sides) & {torch.cuda.Stream().cuda_stream for _ in range(70)}


@pytest.mark.parametrize("kind", [RuntimeError, ValueError, AssertionError, KeyError])
def test_any_error_of_a_capture_leaves_the_step_to_launches(monkeypatch, kind):
    """The sequences have advanced by then: the step runs launch by launch, once, and its kind is not captured again."""
    steps = _host_only(monkeypatch)
    steps.PATIENCE = steps.GAP = 0
    advanced = []
    steps.model.states.advance = lambda entries: advanced.append(entries) or ()
    steps.model.forward = lambda *_a: "launched"

    def fails(*_a):
        steps.noted.append(1)
        raise kind("no capture")
    steps._capture = fails
    assert steps.step([(0, [1])]) == "launched"
    assert steps.step([(0, [1])]) is None and len(advanced) == 1 and len(steps.noted) == 1

    def broken(*_a):
        raise kind("neither")
    steps.model.forward = broken
    with pytest.raises(kind):
        steps.step([(0, [1]), (1, [1])])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", [RuntimeError, ValueError])
def test_a_capture_that_stops_half_way(monkeypatch, kind):
    """An error in the middle of a real capture ends it; this and all later steps give the launched results, and another kind of step is
    captured and replayed."""
    from llm_decoder.hybrid import HybridDecoder
    config, W = _config("tiradra")
    a, b = _pair(config, W, max_tokens=256, max_seqs=2)
    a._decode.GAP = 0
    real, raised = HybridDecoder._linear, []

    def linear(self, *args, **kw):
        if torch.cuda.is_current_stream_capturing():
            raised.append(len(raised))
            if len(raised) == 4:
                raise kind("in the middle")
        return real(self, *args, **kw)
    monkeypatch.setattr(HybridDecoder, "_linear", linear)
    for k in range(6):
        _close(a.step([(0, [k], [0])]), b.step([(0, [k], [0])]))
    assert len(raised) == 4 and not a._decode._graphs
    for k in range(6):
        _close(a.step([(i, [k + i], [0]) for i in (0, 1)]), b.step([(i, [k + i], [0]) for i in (0, 1)]))
    assert len(a._decode._graphs) == 1


def test_a_model_put_in_the_place_of_another(monkeypatch):
    """Steps run on the engine's model and states of the moment."""
    import contextlib
    import llm_decoder as ld
    from llm_decoder import engine
    monkeypatch.setattr(engine._cabi, "on_device", lambda _d: contextlib.nullcontext())

    class Model:
        def __init__(self, name, states):
            self.device, self.vocab, self.states, self.name = torch.device("cpu"), 3, states, name

        def forward(self, *_a):
            return self.name

    class Steps(engine.DecodeSteps):
        def serves(self, *_a):
            return True

        def step(self, _entries):
            return self.model.name
    states = _Held()
    states.alloc = lambda: 0
    e = ld.Engine(Model("first", states))
    e._decode = Steps(e.model)
    assert e.step([(0, [1], [0])]) == "first"
    e.model = Model("second", states)
    assert e.step([(0, [1], [0])]) == "second"


def test_a_run_with_lost_waits_hands_out_no_tokens(monkeypatch):
    """The scheduler asks for waits that ran out before it hands out a request's tokens."""
    import contextlib
    import llm_decoder as ld
    from llm_decoder import engine
    lost = [5]
    monkeypatch.setattr(engine._cabi, "lost_waits", lambda: lost[0])
    monkeypatch.setattr(engine._cabi, "on_device", lambda _d: contextlib.nullcontext())
    monkeypatch.setattr(ld.Scheduler, "_sample", lambda _self, logits: torch.zeros(logits.shape[0], dtype=torch.int32))
    e = _Held()
    e.model, e.states = _Held(), _Held()
    e.model.device, e.states.max_seqs, e.states.tile_size = torch.device("cuda"), 4, 16
    e.has, e.states.free_tokens = lambda _r: False, lambda: 1 << 20
    e.step = lambda entries: torch.zeros(sum(len(w) for _r, _t, w in entries), 7)
    s = ld.Scheduler(e)
    rid = s.add_request([1, 2, 3], 4)
    assert s.run()[rid] == [1, 2, 3, 0, 0, 0, 0]        # lost before this scheduler was made
    rid = s.add_request([1, 2], 3)
    s.step()
    lost[0] += 1
    with pytest.raises(RuntimeError):
        s.run()
    assert rid not in s.done
