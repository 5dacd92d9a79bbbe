"""CUDA graphs of a model's forward and backward launches.

A micro-step of a small batch is bound by the host: a 12-layer GPT-2 issues about 260 kernel launches of a few microseconds each, and the
launcher takes longer than the kernel (forward + backward of 4 x 64 tokens of GPT-2 124M: 4.5 ms launched, 1.3 ms replayed).
``StepGraphs.run`` executes a launch sequence eagerly the first two times it sees its key and from the third time on replays a graph of it.

What makes a replay equal to the eager call: the sequence only reads and writes buffers that the model owns (inputs are copied into them
before), all scalar arguments are part of the key, and the addresses of every parameter, gradient and activation buffer and of the rotary
table are compared.  The scratch buffers of the operators are shared by all callers and replaced when one needs a larger one, so a graph keeps those that its own operators took.
"""
import contextlib
import gc
import threading

import torch

from ..ops import kernels


class _NoCollection:
    """Garbage collection is off while any thread is inside (the switch is the process's, captures are each thread's); the last one out puts back
    what the first one found."""

    def __init__(self):
        self._lock, self._inside, self._was_on = threading.Lock(), 0, False

    def __enter__(self):
        with self._lock:
            if self._inside == 0:
                self._was_on = gc.isenabled()
                gc.disable()
            self._inside += 1

    def __exit__(self, *exc):
        with self._lock:
            self._inside -= 1
            if self._inside == 0 and self._was_on:
                gc.enable()


_no_collection = _NoCollection()


class Inline:
    """Launches outside a capture: everything in one stream, in the order of the calls."""

    def fork(self):
        return contextlib.nullcontext()

    fork_sums = fork

    def other(self, t):
        return t

    def mark_sums(self):
        return None

    def read(self, *buffers):
        pass

    free = read

    def join(self, mark=None):
        pass


class Side:
    """Two more branches of the graph that is being captured, for launches whose results the chain of the backward pass does not read: one for gradients of
    weights, one for the small sums (gradients of biases and of the norms' parameters).  A small batch leaves most SMs idle in every kernel of that chain.
    ``fork()`` / ``fork_sums()``: the launches inside the block follow all launches of the main branch so far; ``join(mark_sums())``: the launches of
    the main branch from here on follow the sums given up to the mark, ``join()``: everything the side branches have been given.
    ``read(buffer)`` notes that the launches given to them so far read it, ``free(buffer)`` joins those: before the main branch writes it again.

    Forward and backward of GPT-2 124M at 4 x 64 tokens 1372 us with one branch that is joined at the end of every layer, 1335 us with two, 1310 with the priority of
    ``_capture``, 1280 since a join adds no edge that is there already (with everything recomputed and 2 x 64 tokens 1370, -, 1390, 1355)."""

    def __init__(self, stream, sums):
        self.stream, self.sums = stream, sums
        self._forks = {}                   # of the two, those that have work of this capture: how often they were given some
        self._joined = {}                  # and how much of it the main branch follows
        self._others = {}
        self._readers = {}

    def other(self, t):
        """A second buffer like ``t``, in the memory of the graph: the main branch writes it while the side branch still reads ``t``.  It gives ``t`` for itself.
        Outside a capture, where nothing is read late, both are ``t``."""
        if t.data_ptr() not in self._others:
            o = torch.empty_like(t)
            self._others[t.data_ptr()], self._others[o.data_ptr()] = o, t
        return self._others[t.data_ptr()]

    def _fork(self, stream):
        self._forks[stream] = self._forks.get(stream, 0) + 1
        stream.wait_event(torch.cuda.current_stream().record_event())
        return torch.cuda.stream(stream)

    def fork(self):
        return self._fork(self.stream)

    def fork_sums(self):
        return self._fork(self.sums)

    def _mark(self, stream):
        return stream, self._forks[stream], stream.record_event()

    def mark_sums(self):
        return self._mark(self.sums)

    def join(self, *marks):
        # a launch with an edge from another branch does not start under the one before it: none for what the main branch follows already
        for stream, forks, event in marks or [self._mark(s) for s in self._forks]:
            if self._joined.get(stream, 0) < forks:
                self._joined[stream] = forks
                torch.cuda.current_stream().wait_event(event)

    def read(self, *buffers):
        marks = [self._mark(s) for s in self._forks]
        for t in buffers:
            self._readers[t.data_ptr()] = marks

    def free(self, *buffers):
        for t in buffers:
            marks = self._readers.pop(t.data_ptr(), None)
            if marks:
                self.join(*marks)


class StepGraphs:
    # sequences longer than this many tokens are bound by the GPU (at 4096 tokens GPT-2 124M computes as long as the host takes to launch)
    MAX_TOKENS = 4096
    # distinct sequences kept per model; more than these (many micro-step indices, many sequence lengths) run eagerly
    MAX_GRAPHS = 16

    def __init__(self):
        self._entries = {}
        self.side = Inline()               # where the launches beside the main chain go

    def __reduce__(self):
        return StepGraphs, ()              # a copied or unpickled model captures graphs of its own buffers

    def clear(self):
        self._entries.clear()

    def run(self, model, tokens, key, fn):
        """``fn()`` issues the launches; ``key`` holds every argument they depend on besides the model's buffers."""
        if tokens > self.MAX_TOKENS or model.device.type != "cuda" or model.dtype != torch.bfloat16 or not model.use_graphs \
                or torch.cuda.is_current_stream_capturing():
            return fn()
        buffers = [model.params_flat, *model.params.values(), model.inputs, model.targets, *model.acts.values()]
        if getattr(model, "freqs", None) is not None:
            buffers.append(model.freqs)                        # rotary table
        if model.grads is not None:
            buffers += [model.grads_flat, *model.grads.values()]
        addresses = tuple(t.data_ptr() for t in buffers)
        e = self._entries.get(key)
        if e is None or e["addresses"] != addresses:
            if e is None and len(self._entries) >= self.MAX_GRAPHS:
                return fn()
            e = self._entries[key] = {"addresses": addresses, "seen": 0, "graph": None, "tokens": tokens}
        e["seen"] += 1
        if e["seen"] <= 2:
            return fn()
        if e["graph"] is None:
            self._capture(model, e, fn)
        e["graph"].replay()
        kernels.count_launches(e["launches"])

    @staticmethod
    def _capture(model, e, fn):
        # the chain in a stream of higher priority: its blocks come first wherever an SM gets free, those of the side branches take what it leaves.  Pays as long
        # as the side branches are the smaller part, and they grow with the tokens and the square of the channels.  GPT-2's layers, us, without / with the priority, 12 of 768
        # channels: 64 tokens 1163 / 1147, 512 1581 / 1545, 1024 2375 / 2289, 1536 2671 / 2648; 8 of 1280: 64 1089 / 1042, 1024 2454 / 2395, 1536 2680 / 2651; 4 of 2048: 64
        # 928 / 884, 512 1390 / 1368, but 768 1791 / 1800; 3 of 2560: 256 1138 / 1124, 384 1324 / 1327, 1536 3240 / 3434; 2 of 4096: 128 1220 / 1208, 256 1359 / 1387, 512 2044 /
        # 2125; two LLaMA layers' worth of wide weight gradients over 128 tokens 1279 / 1307.  The models say up to how many tokens (LLaMA: none)
        first = 0 < e.get("tokens", 0) <= getattr(model, "chain_first_tokens", 0)
        graph, chain = torch.cuda.CUDAGraph(), torch.cuda.Stream(device=model.device, **({"priority": -1} if first else {}))
        before = kernels.launch_count()
        # a collection inside the capture could find a dropped model, and the graphs it held cannot be freed by a thread that captures
        with torch.cuda.stream(chain), kernels.scratch_taken() as scratch, _no_collection:
            # other threads (watchdog, data loader) may use the device meanwhile
            graph.capture_begin(capture_error_mode="thread_local")
            model.step_graphs.side = Side(torch.cuda.Stream(device=model.device), torch.cuda.Stream(device=model.device))
            try:
                fn()
            finally:
                model.step_graphs.side = Inline()
                graph.capture_end()
        e["launches"] = kernels.launch_count() - before
        kernels.count_launches(-e["launches"])                 # captured, not launched
        e["scratch"] = scratch
        e["graph"] = graph
