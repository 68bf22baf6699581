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


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)     # (absent from builds of torch without CUDA)


def stream_ptr(device=None) -> int:
    """The current stream of `device` as the library takes it.  Asked for its number only: making the Stream object costs
    4 us, as much as the launch that follows."""
    if _raw_stream is None:
        return torch.cuda.current_stream(device).cuda_stream
    index = None if device is None else torch.device(device).index
    return _raw_stream(torch.cuda.current_device() if index is None else index)


def require_cuda(*tensors):
    for t in tensors:
        if t is not None and not t.is_cuda:
            raise RuntimeError("vtpack_b200 ops run on CUDA tensors only (there is no CPU path)")


def ptr(t):
    return None if t is None else t.data_ptr()


_scratch = {}       # (device type, index, use) -> buffer
_scratch_gen = {}   # (device type, index, use) -> how many times the buffer was replaced
_scratch_users = {}  # (device type, index, use) -> {stream number: stream} that have been handed the current buffer


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
    if buf is None or buf.numel() < nbytes:
        if buf is not None:
            for st in _scratch_users.get(key, {}).values():
                buf.record_stream(st)          # kernels queued on st may still be using the old buffer
        buf = torch.empty(max(int(nbytes), 1), dtype=torch.uint8, device=device)
        _scratch[key] = buf
        _scratch_gen[key] = _scratch_gen.get(key, 0) + 1
        _scratch_users[key] = {}
    users = _scratch_users.setdefault(key, {})
    number = stream_ptr(device)
    if number not in users:
        users[number] = torch.cuda.current_stream(device)
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
    host work of its launches and the gaps between them.  At most ``most`` are kept, the least recently used one goes
    first, and they go with the model.

    A shape is captured at its ``earn``-th call, and after twice as many each time its plan has been dropped for others':
    calls are counted for the last 8 ``most`` shapes.  A capture costs 0.7 to 1.9 ms, a replay saves 25 us (DeiT-Ti, one
    image) to 300 us (PVT-small, 33), so a shape that is rarely seen should not pay for one.  Mean of a call, waited
    for, with no plans / captured at the second sighting among the last ``most`` shapes / this rule: batches of 1 to 12
    at random, 400 calls, DeiT-Ti 678 / 872 / 697 us, PVT-tiny 971 / 1226 / 967 us; of 1 to 48, 800 calls, 889 / 1023 / 927
    and 1285 / 1406 / 1303 us; 7 images 400 times, 678 / 650 / 657 and 999 / 761 / 763 us."""

    def __init__(self, most=8, earn=8):
        self.most, self.earn = most, earn
        self._plans = OrderedDict()           # shape -> plan
        self._calls = OrderedDict()           # shape -> [calls without a plan, calls that earn one]
        self._lock = threading.Lock()

    def __reduce__(self):                     # graphs hold device addresses: copies of the model make their own
        return (LaunchPlans, (self.most, self.earn))

    def clear(self):
        with self._lock:
            self._plans.clear()
            self._calls.clear()

    def get(self, key, valid, capture):
        """The plan for `key`: None until the shape has earned one, then ``capture()``'s result, made again when
        ``valid(plan)`` says that the kept one no longer fits."""
        if torch.cuda.is_current_stream_capturing():
            return None                       # the caller is recording a graph of its own
        with self._lock:
            plan = self._plans.get(key)
            if plan is None:
                calls = self._calls.setdefault(key, [0, self.earn])
                self._calls.move_to_end(key)
                while len(self._calls) > 8 * self.most:
                    self._calls.popitem(last=False)
                calls[0] += 1
                if calls[0] < calls[1]:
                    return None
                calls[:] = [0, 2 * calls[1]]          # should the plan be dropped for others, the next one is dearer
            if plan is None or not valid(plan):
                plan = self._plans[key] = capture()
            self._plans.move_to_end(key)
            while len(self._plans) > self.most:
                self._plans.popitem(last=False)
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
