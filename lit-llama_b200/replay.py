"""Steps recorded as CUDA graphs: the stream they are recorded on, the recording, and which portions are worth one."""
import ctypes as C
import threading
import types
import weakref
from typing import Callable, Collection, Dict, Hashable, List, Optional, Tuple

import torch

from . import _seqlib as S

_lock = threading.RLock()                 # an owner may be collected, and give back, while its thread is inside
_free: Dict[int, List[int]] = {}          # device -> recording streams whose owners are gone


def recording_stream(owner, device: torch.device) -> torch.cuda.Stream:
    """A stream that no other living owner records on.  The library's products have a workspace per thread and stream, and a graph keeps the one of the
    stream it was recorded on: graphs of two owners may run at the same time, so theirs must differ.  Streams (and their workspaces) of owners that are
    gone are given out again, after the graphs they were for have run."""
    index = device.index if device.index is not None else torch.cuda.current_device()
    with torch.cuda.device(index):
        with _lock:
            at = _free[index].pop() if _free.get(index) else None
        if at is None:
            p = C.c_void_p()
            S.check(S.lib().b2l_seq_stream_create(C.byref(p)), "b2l_seq_stream_create")
            at = p.value
        else:
            torch.cuda.synchronize(index)
    weakref.finalize(owner, _give_back, index, at).atexit = False
    return torch.cuda.ExternalStream(at, device=torch.device("cuda", index))


def _give_back(index: int, at: int) -> None:
    with _lock:
        _free.setdefault(index, []).append(at)


def record(stream: torch.cuda.Stream, pool, body: Callable[[], torch.Tensor]) -> Tuple[torch.cuda.CUDAGraph, torch.Tensor]:
    """What body() launches as a graph (not run), with its temporaries in `pool` (None: one of its own), and body()'s result.  Only this thread's calls count
    as part of the recording: another thread may allocate, launch or record meanwhile."""
    with torch.cuda.device(stream.device), torch.cuda.stream(stream):
        torch.cuda.current_blas_handle()                 # the thread's handle and its workspace for this stream are there before the recording
        try:
            return _recorded(pool, body)
        except RuntimeError:
            # a recording that a call has broken off leaves torch's random numbers waiting for its end; one that ends takes them out of that
            _recorded(None, lambda: torch.zeros(1, device=stream.device))
            raise


def _recorded(pool, body):
    g = torch.cuda.CUDAGraph()
    g.capture_begin(pool=pool, capture_error_mode="thread_local")
    try:
        out = body()
    finally:
        g.capture_end()
    return g, out


def settings() -> tuple:
    """What torch's products look at besides their operands: a recording has the forms that were chosen under the settings of its time."""
    m = torch.backends.cuda.matmul
    return (m.fp32_precision == "tf32", m.allow_bf16_reduced_precision_reduction, m.allow_fp16_accumulation, torch.backends.cuda.preferred_blas_library(),
            torch.are_deterministic_algorithms_enabled(), torch.is_autocast_enabled("cuda"))


class Held:
    """What recordings have taken from Python objects: the tensors (a graph has their addresses) and values that lie in their attributes, lists and dicts.
    `unchanged` says whether all are where they were; new contents of a tensor are no change.  It takes some 0.1 us for each."""

    def __init__(self, *roots) -> None:
        self.lists, self.values, self.tensors, seen, todo = [], [], [], set(), list(roots)
        while todo:
            o = todo.pop()
            box = o if isinstance(o, (dict, list, tuple)) else getattr(o, "__dict__", None)
            if box is None or id(box) in seen or isinstance(o, (type, types.ModuleType, types.FunctionType)):
                continue
            seen.add(id(box))
            if not isinstance(box, dict):
                self.lists.append((box, len(box)))
            for key, v in box.items() if isinstance(box, dict) else enumerate(box):
                if isinstance(v, torch.Tensor):
                    self.tensors.append((box, key, weakref.ref(v), v.data_ptr()))      # weak: weights that are replaced are free to go
                else:
                    self.values.append((box, key, v))
                    todo.append(v)

    def unchanged(self) -> bool:
        try:
            return (all(box[key] is v for box, key, v in self.values) and all(len(box) == n for box, n in self.lists)
                    and all((t := box[key]) is held() and t.data_ptr() == at for box, key, held, at in self.tensors))
        except (KeyError, IndexError, AttributeError):
            return False


class Sightings:
    """How often portions of a kind have come lately, and from that which are recorded.  A recording takes 0.5 ms more than its portion run eagerly and
    saves 0.4 ms whenever it is replayed (four layers of width 1024; both grow with the layers).  While there is room a kind is recorded once it has
    come `after` times; then only one that comes more than twice as often as the rarest that has a graph, and LEAD times more: lengths that take turns
    keep the graphs they have, and a recording is spread over more than LEAD portions.  Counts outlive the graphs and are halved every HALF portions."""

    HALF, LEAD = 256, 32

    def __init__(self) -> None:
        self.counts: Dict[Hashable, int] = {}
        self.total = 0

    def worth(self, key: Hashable, kept: Collection[Hashable], after: int, room: int) -> Tuple[bool, Optional[Hashable]]:
        """One more portion of kind `key`, while those of `kept` have graphs: whether it is recorded now, and the graph that goes for it."""
        self.total += 1
        if self.total % self.HALF == 0:
            self.counts = {k: n // 2 for k, n in self.counts.items() if n > 1}
        n = self.counts[key] = self.counts.get(key, 0) + 1
        if key in kept or n <= after or room <= 0:
            return False, None
        if len(kept) < room:
            return True, None
        rarest = min(kept, key=lambda k: self.counts.get(k, 0))
        return n > 2 * self.counts.get(rarest, 0) + self.LEAD, rarest
