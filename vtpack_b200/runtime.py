"""Device-side plumbing shared by the op wrappers: dtype codes, the current CUDA
stream as a raw pointer, cached scratch buffers (PyTorch owns all device memory;
the library never allocates), and the captured launch sequences the models replay."""
import threading
import weakref
from collections import OrderedDict
from operator import attrgetter, getitem, is_

import torch

from . import _lib


def dtype_code(t: torch.dtype) -> int:
    if t == torch.float32:
        return _lib.VTP_F32
    if t == torch.bfloat16:
        return _lib.VTP_BF16
    raise TypeError(f"vtpack_b200 supports float32 and bfloat16, got {t}")


def stream_ptr(device=None) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError("vtpack_b200 ops run on CUDA tensors only (there is no CPU path)")


def ptr(t):
    return None if t is None else t.data_ptr()


_scratch = {}       # (device type, index, use) -> buffer
_scratch_gen = {}   # (device type, index, use) -> how many times the buffer was replaced
_scratch_users = {}  # (device type, index, use) -> streams that have been handed the current buffer


def scratch(device, nbytes: int, use: str = "block") -> torch.Tensor:
    """A uint8 buffer of at least nbytes on `device`, grown on demand and reused.

    One buffer per device and use, shared by every block / model forward on it: forwards that can run at
    the same time (two streams, two host threads) would overwrite each other's intermediates, so
    run the forwards of one device on one stream at a time.  When the buffer has to grow, the old
    one is handed back to the allocator only after the streams it was given to have finished
    their queued work; CUDA graphs captured against it are invalid from then on
    (``scratch_generation`` changes)."""
    key = (device.type, device.index, use)
    buf = _scratch.get(key)
    cur = torch.cuda.current_stream(device)
    if buf is None or buf.numel() < nbytes:
        if buf is not None:
            for st in _scratch_users.get(key, ()):
                buf.record_stream(st)          # kernels queued on st may still be using the old buffer
        buf = torch.empty(max(int(nbytes), 1), dtype=torch.uint8, device=device)
        _scratch[key] = buf
        _scratch_gen[key] = _scratch_gen.get(key, 0) + 1
        _scratch_users[key] = []
    users = _scratch_users.setdefault(key, [])
    if all(u.cuda_stream != cur.cuda_stream for u in users):
        users.append(cur)
    return buf


def scratch_generation(device, use: str = "block") -> int:
    """Changes whenever the device's scratch buffer is replaced by a larger one."""
    return _scratch_gen.get((device.type, device.index, use), 0)


_version_of = attrgetter("_version")


class ParamWatch:
    """Tells whether a module's parameters are still the ones seen before, without walking the module tree: a
    snapshot of every owner's parameters and submodules is compared by identity, then versions and addresses.
    ``generation()`` returns a number that changes with any replacement, in-place update or move of a parameter,
    plain tensors in a parameter's place (``torch.func.functional_call`` puts them there) among them
    (48 us for a 12-block model where building a key from ``module.parameters()`` takes 320 us)."""

    def __init__(self, module):
        self._module = weakref.ref(module)    # (the module owns the watch)
        self._gen = 0
        self._kept = None

    def generation(self) -> int:
        try:
            same = self._kept is not None and all(map(is_, map(getitem, self._owners, self._names), self._kept))
        except KeyError:                      # a parameter or submodule was removed
            same = False
        if not same:
            dicts = [d for m in self._module().modules() for d in (m._modules, m._parameters)]
            self._owners = [d for d in dicts for _ in d]
            self._names = [n for d in dicts for n in d]
            self._kept = [v for d in dicts for v in d.values()]
            self._params = [v for v in self._kept if isinstance(v, torch.Tensor)]
            self._state = None
        state = (list(map(_version_of, self._params)), list(map(torch.Tensor.data_ptr, self._params)))
        if state != self._state:
            self._state = state
            self._gen += 1
        return self._gen


class LaunchPlans:
    """Captured launch sequences (CUDA graphs) of one model's forward, one per call shape: replaying one removes the
    host work of its launches and the gaps between them.  A shape is captured when it is seen for the second
    time, so a shape or a set of weights that is used once never pays for it; at most ``most`` are kept, the
    least recently used one goes first, and they go with the model."""

    def __init__(self, most=8):
        self.most = most
        self._plans = OrderedDict()
        self._lock = threading.Lock()

    def __reduce__(self):                     # graphs hold device addresses: copies of the model make their own
        return (LaunchPlans, (self.most,))

    def clear(self):
        with self._lock:
            self._plans.clear()

    def get(self, key, valid, capture):
        """The plan for `key`: None the first time, then ``capture()``'s result, made again when ``valid(plan)``
        says that the kept one no longer fits."""
        if torch.cuda.is_current_stream_capturing():
            return None                       # the caller is recording a graph of its own
        with self._lock:
            if key not in self._plans:
                self._plans[key] = None
                while len(self._plans) > self.most:
                    self._plans.popitem(last=False)
                return None
            plan = self._plans[key]
            self._plans.move_to_end(key)
            if plan is None or not valid(plan):
                plan = self._plans[key] = capture()
            return plan


def capture_launches(device, launch):
    """A CUDA graph of the kernels that ``launch(stream pointer)`` launches; nothing runs."""
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream(device)
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="thread_local")
        try:
            launch(side.cuda_stream)
        finally:
            graph.capture_end()
    return graph
