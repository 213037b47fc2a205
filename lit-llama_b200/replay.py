"""Steps recorded as CUDA graphs: the stream they are recorded on, and the recording."""
import ctypes as C
import threading
import weakref
from typing import Callable, Dict, List, Tuple

import torch

from . import _seqlib as S

_lock = threading.Lock()
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
    weakref.finalize(owner, _give_back, index, at)
    return torch.cuda.ExternalStream(at, device=torch.device("cuda", index))


def _give_back(index: int, at: int) -> None:
    with _lock:
        _free.setdefault(index, []).append(at)


def record(stream: torch.cuda.Stream, pool, body: Callable[[], torch.Tensor]) -> Tuple[torch.cuda.CUDAGraph, torch.Tensor]:
    """What body() launches as a graph (not run), with its temporaries in `pool` (None: one of its own), and body()'s result.  Only this thread's calls count
    as part of the recording: another thread may allocate, launch or record meanwhile."""
    g = torch.cuda.CUDAGraph()
    with torch.cuda.device(stream.device), torch.cuda.stream(stream):
        torch.cuda.current_blas_handle()                 # the thread's handle and its workspace for this stream are there before the recording
        g.capture_begin(pool=pool, capture_error_mode="thread_local")
        try:
            out = body()
        finally:
            g.capture_end()
    return g, out
