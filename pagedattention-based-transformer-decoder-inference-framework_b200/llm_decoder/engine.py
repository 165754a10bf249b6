"""Engine and Scheduler for the config-driven models (hybrid.HybridDecoder).

Engine.step(entries) is THE step function: every entry brings the next tokens of one request (a prompt portion of
any length, or one decoded token); all entries run as one ragged batch through the model from the K/V pages and state
slots earlier steps left.  A request is admitted (state slot) at its first entry, may sit out steps, and gives back its
slot and pages with `finish`.

Scheduler is continuous batching on top of it: waiting requests are admitted while slots and pool tokens last, prompts
are fed in chunks under a per-step token budget next to the running requests' single decode tokens, and the next token
of every request whose last fed token ended its prompt (or was a decoded token) is sampled on the device with the
framework's samplers (greedy pa_argmax_f32; temperature / top-k / top-p through llm_decoder.sampling)."""
import collections
import ctypes
import threading
import types

import torch

from . import _cabi
from .host_stage import to_device as _to_device
from .hybrid import HybridDecoder
from .seq_state import DecodeBatch


class _Lane:
    """A stream that graphs are captured on, and the order of their replays.  The vendor products captured on a stream share the
    library's scratch of that stream, so the replays of a lane follow one another, whatever streams they are issued on; and a lane's stream
    is nobody else's, so that no launched product uses that scratch.  An engine has a lane of its own up to the EACH-th of a device."""
    EACH = 8
    _lock, _lanes, _next = threading.Lock(), {}, {}

    def __init__(self, device):
        raw = ctypes.c_void_p()
        _cabi.check(_cabi.lib().pa_stream_create(ctypes.byref(raw)), "pa_stream_create")
        self.side, self.lock = torch.cuda.ExternalStream(raw.value, device=device), threading.Lock()
        self._event, self._stream = torch.cuda.Event(), None

    @classmethod
    def of(cls, device):
        with cls._lock:
            at = torch.cuda.current_device()
            lanes, i = cls._lanes.setdefault(at, []), cls._next.get(at, 0)
            cls._next[at] = i + 1
            if len(lanes) < cls.EACH:
                lanes.append(cls(device))
            return lanes[i % cls.EACH]

    def before(self, stream):
        if self._stream is not None and self._stream != stream:
            stream.wait_event(self._event)

    def after(self, stream):
        self._event.record(stream)
        self._stream = stream


class DecodeSteps:
    """Steps that decode one token of each of n sequences, as CUDA graphs: such a step is some dozens of launches of a few
    microseconds each, and issuing them takes several times as long as running them (8 sequences, 4 layers of width 1024: 1.0 ms
    launch by launch, 0.3 ms replayed).  A graph belongs to a number of sequences and a bound of their lengths (see _bound).
    A capture costs as much as 6 to 30 launched steps, so the first PATIENCE steps of a kind run launch by launch; from then on a
    step writes its tokens, slots and positions into the graph's buffers and replays it.  Where more kinds come up than graphs are kept,
    captures stay rare: one in GAP steps at most, a graph gives way only after IDLE steps without a replay, and a kind that was captured
    before has to come up twice as often as the last time.

    A graph holds the addresses of the model's weights and caches.  It keeps those tensors alive, and before every replay every
    attribute of the model, its layers, their parts and the caches has to be the very object it was at the capture: anything that
    was replaced since makes the step run launch by launch and be captured anew."""
    MOST, SEQS = 8, 256                     # graphs kept; sequences of a step
    PATIENCE, GAP, IDLE = 16, 64, 256       # in steps, see above

    def __init__(self, model):
        self.model, self._lane = model, None
        self._graphs = collections.OrderedDict()        # kind -> graph, the one whose replay is longest ago first
        self._seen, self._caught = {}, {}               # kind -> launched steps since its last capture; captures
        self._now, self._last = 0, None                 # steps so far; the step of the last capture

    def _due(self, key):
        """Whether a step of a kind without a graph captures one."""
        seen = self._seen.get(key, 0)
        due = (seen >= self.PATIENCE << min(self._caught.get(key, 0), 20) and
               (self._last is None or self._now - self._last >= self.GAP) and
               (len(self._graphs) < self.MOST or self._now - next(iter(self._graphs.values()))["used"] >= self.IDLE))
        if not due:
            if len(self._seen) > 64 * self.MOST:        # kinds that came up now and then
                self._seen.clear()
                self._caught.clear()
            self._seen[key] = seen + 1
        return due

    def serves(self, entries, wanted_rows):
        m = self.model
        return (type(m) is HybridDecoder and len(entries) <= self.SEQS and m.act_dtype == torch.bfloat16 and m.device.type == "cuda" and
                m.layer_hook is None and
                len(wanted_rows) == len(entries) and all(len(t) == 1 for _s, t in entries) and
                not torch.cuda.is_current_stream_capturing())

    def _bound(self, longest):
        """The bound of the lengths that the launches of a graph are made for: a power of two from 512 on.  Equal shares of the keys
        follow from the lengths alone, so these launches give the bits of launches made for the exact lengths; the kernels that cut
        keys by the longest context do so from 513 keys on, by its multiples of 256 and up to 64 of them: where a layer runs on
        those, the bound lies between the same multiples."""
        if 512 < longest < 64 * 256 and any(getattr(mixer, "cuts_keys", False) for _L, mixer, _pass in self.model.runs):
            return longest // 256 * 256 + 255
        bound = 512
        while bound < longest:
            bound *= 2
        return bound

    def _watched(self):
        """What a forward pass reads: [(owner's dict, its size, [(key, value, address of a tensor)])] and the runs."""
        seen, out = set(), []
        todo = [self.model, self.model.states] + self.model.states._kv + [k.page_table_ for k in self.model.states._kv]
        for L, mixer, _pass in self.model.runs:
            todo += [L, mixer, L.ff]
        while todo:
            o = todo.pop()
            d = o if isinstance(o, dict) else getattr(o, "__dict__", None)
            if d is None or id(d) in seen:
                continue
            seen.add(id(d))
            out.append((d, len(d), [(k, v, v.data_ptr() if isinstance(v, torch.Tensor) else None) for k, v in d.items()]))
            todo += [v for k, v in d.items() if k in ("core", "left", "right", "shared", "mixer", "ff")]
        return out, tuple(self.model.runs)

    def _same(self, watched):
        dicts, runs = watched
        now = self.model.runs
        return (len(now) == len(runs) and all(a is b for a, b in zip(now, runs)) and
                all(len(d) == n and all(d.get(k) is v and (p is None or v.data_ptr() == p) for k, v, p in items) for d, n, items in dicts))

    def step(self, entries):
        """Logits [n, vocab] of the step, or None where it is to run launch by launch."""
        m, st = self.model, self.model.states
        bound = self._bound(max((st.length(s) for s, _t in entries), default=0) + 1)
        key = (len(entries), bound)
        self._now += 1
        g = self._graphs.get(key)
        if g is not None and not self._same(g["watched"]):
            del self._graphs[key]
            g = None
        if g is None and not self._due(key):
            return None
        if g is None and any(isinstance(v, (types.FunctionType, types.MethodType)) for _d, _n, items in self._watched()[0] for _k, v, _p in items):
            return None         # a function put in the place of a method may do more than launch kernels
        if self._lane is None:
            self._lane = _Lane.of(m.device)
        if g is None:
            g = dict(batch=DecodeBatch(len(entries), bound, m.device, st.track_tokens), graph=None, stream=None)
        stream = torch.cuda.current_stream(m.device)
        with self._lane.lock:
            self._lane.before(stream)           # the last replay, on another stream, still reads the buffers
            if g["stream"] != stream:           # ... and this one may when the graph is dropped
                g["stream"] = stream
                g["batch"].used_on(stream)
            g["batch"].fill(*st.advance(entries))
            for kv in st._tables:
                kv.page_table_.flush()          # no update of a table belongs into the graph
            if g["graph"] is None:
                try:
                    self._capture(g, stream)
                except Exception:           # memory, a call that cannot be captured: this kind stays with launches, which raise
                                            # what was not the capture's fault
                    self._seen[key] = -(1 << 60)
                    return m.forward(g["batch"], g["batch"].seq_start)
                while len(self._graphs) >= self.MOST:
                    self._graphs.popitem(last=False)
                self._graphs[key], self._last = g, self._now
                self._seen[key], self._caught[key] = 0, self._caught.get(key, 0) + 1
            self._graphs.move_to_end(key)
            g["used"] = self._now
            g["graph"].replay()
            out = g["logits"].clone()
            self._lane.after(stream)
        return out

    def _capture(self, g, stream):
        m = self.model
        side, graph = self._lane.side, torch.cuda.CUDAGraph()
        side.wait_stream(stream)
        with torch.cuda.stream(side):
            graph.capture_begin(capture_error_mode="thread_local")
            try:
                logits = m.forward(g["batch"], g["batch"].seq_start)
            finally:
                graph.capture_end()
        stream.wait_stream(side)
        g.update(graph=graph, logits=logits, watched=self._watched())


class Engine:
    def __init__(self, model):
        self.model = model
        self.states = model.states
        self._slot = {}          # request id -> slot
        self._decode = DecodeSteps(model)

    def live(self):
        return list(self._slot)

    def has(self, rid):
        return rid in self._slot

    def length(self, rid):
        return self.states.length(self._slot[rid])

    def step(self, entries):
        """entries: [(request id, token ids, wanted indices into these tokens)].  Returns float logits
        [total wanted, vocab] (device) in entry / wanted order."""
        batch_entries, want, row0 = [], [], 0
        for rid, toks, wanted in entries:
            if not len(toks):
                continue
            if rid not in self._slot:
                self._slot[rid] = self.states.alloc()
            batch_entries.append((self._slot[rid], toks))
            for w in wanted:
                if not 0 <= int(w) < len(toks):
                    raise ValueError("wanted index outside the entry's tokens")
                want.append(row0 + int(w))
            row0 += len(toks)
        dev = self.model.device
        if not batch_entries:
            return torch.empty((0, self.model.vocab), dtype=torch.float32, device=dev)
        with _cabi.on_device(dev):
            if self._decode.model is not self.model:
                self._decode = DecodeSteps(self.model)
            if self.model.states is self.states and self._decode.serves(batch_entries, want) and want == list(range(row0)):
                logits = self._decode.step(batch_entries)
                if logits is not None:
                    return logits
            batch = self.states.make_batch(batch_entries)
            want_rows = _to_device(torch.tensor(want, dtype=torch.int32), dev)
            return self.model.forward(batch, want_rows)

    def finish(self, rid):
        slot = self._slot.pop(rid, None)
        if slot is not None:
            self.states.free(slot)


class _Request:
    def __init__(self, rid, prompt, max_new_tokens):
        self.rid, self.prompt, self.max_new = rid, list(prompt), int(max_new_tokens)
        self.fed = 0            # prompt tokens already given to the engine
        self.out = []           # generated tokens
        self.pending = None     # a sampled token not yet fed


class Scheduler:
    def __init__(self, engine, max_batch_tokens=2048, temperature=1.0, top_k=0, top_p=1.0, eos_token_id=-1, seed=0):
        self.engine = engine
        self.max_batch_tokens = int(max_batch_tokens)
        self.temperature, self.top_k, self.top_p = float(temperature), int(top_k), float(top_p)
        self.eos = int(eos_token_id)
        self.waiting = collections.deque()
        self.running = []
        self.done = {}
        self._next = 0
        self._lost = self._lost_waits()
        self._gen = None
        if self.top_k > 0 or self.top_p < 1.0:
            self._gen = torch.Generator(device=engine.model.device)
            self._gen.manual_seed(int(seed))

    def add_request(self, prompt, max_new_tokens, rid=None):
        if not len(prompt):
            raise ValueError("empty prompt")
        rid = self._next if rid is None else rid
        self._next += 1
        self.waiting.append(_Request(rid, prompt, max_new_tokens))
        return rid

    def _lost_waits(self):
        dev = self.engine.model.device
        if dev.type != "cuda":
            return 0
        with _cabi.on_device(dev):
            return _cabi.lost_waits()

    def _tiles(self, n):
        ts = self.engine.states.tile_size
        return (n + ts - 1) // ts * ts

    def _sample(self, logits):
        """logits [n, vocab] float -> [n] int32 next ids, on the device."""
        n, V = logits.shape
        ids = torch.empty(n, dtype=torch.int32, device=logits.device)
        lib = _cabi.lib()
        if self._gen is None:
            _cabi.check(lib.pa_argmax_f32(logits.data_ptr(), n, V, 1.0, 1, ids.data_ptr(), _cabi.stream()), "pa_argmax_f32")
            return ids
        from . import sampling
        probs = sampling.softmax_temperature(logits.contiguous(), self.temperature)
        sampling.apply_topk_topp_filter(probs, self.top_k, self.top_p, -1, 0.0)
        u = torch.rand(n, device=logits.device, generator=self._gen)
        sampling.sample_from_probs(probs, u, out=ids)
        return ids

    def step(self):
        """One engine step.  Returns False when nothing is left to do."""
        st = self.engine.states
        # admit: a request needs a slot and room for its whole prompt and output (it is never evicted half-way)
        reserved = sum(self._tiles(len(r.prompt) + r.max_new) - self._tiles(self.engine.length(r.rid) if self.engine.has(r.rid) else 0)
                       for r in self.running)
        while self.waiting and len(self.running) < st.max_seqs:
            r = self.waiting[0]
            need = self._tiles(len(r.prompt) + r.max_new)
            if reserved + need > st.free_tokens():
                if not self.running:
                    raise RuntimeError("request does not fit the cache pool")
                break
            reserved += need
            self.running.append(self.waiting.popleft())
        if not self.running:
            return False
        budget = self.max_batch_tokens
        entries, owners = [], []
        for r in self.running:                      # decode tokens first: one each
            if r.pending is not None and budget > 0:
                entries.append((r.rid, [r.pending], [0]))
                owners.append(r)
                r.pending = None
                budget -= 1
        for r in self.running:                      # then prompt portions under what is left of the budget
            if r.fed < len(r.prompt) and budget > 0:
                n = min(budget, len(r.prompt) - r.fed)
                toks = r.prompt[r.fed:r.fed + n]
                r.fed += n
                budget -= n
                last = r.fed == len(r.prompt)
                entries.append((r.rid, toks, [n - 1] if last else []))
                if last:
                    owners.append(r)
        logits = self.engine.step(entries)
        if owners:
            ids = self._sample(logits).cpu().tolist()
            ended = [len(r.out) + 1 >= r.max_new or int(t) == self.eos for r, t in zip(owners, ids)]
            if any(ended) and self._lost_waits() != self._lost:     # asked before tokens are handed out: the GPU is idle here anyway
                raise RuntimeError("a kernel gave up on a wait: logits of this run are not valid")
            for r, t, end in zip(owners, ids, ended):
                r.out.append(int(t))
                if end:
                    self.engine.finish(r.rid)
                    self.done[r.rid] = r.prompt + r.out
                    self.running.remove(r)
                else:
                    r.pending = int(t)
        return bool(self.running or self.waiting)

    def run(self):
        while self.step():
            pass
        return self.done


def generate(model, prompts, max_new_tokens, **kw):
    """Greedy (or sampled) generation of several prompts of any lengths through Engine + Scheduler; returns
    prompt + generated ids per prompt."""
    sch = Scheduler(Engine(model), **kw)
    rids = [sch.add_request(p, max_new_tokens) for p in prompts]
    done = sch.run()
    return [done[r] for r in rids]
