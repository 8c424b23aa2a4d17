"""What a compiled call did, written down so that later calls need no Python (``csrc/replay.cpp``).

``record`` runs a recorded schedule once more while two observers look on: every call of an exported launch function goes
through ``native.recorder()``, every torch call through a dispatch mode. When all that happened on the device was launches of
functions in ``LAUNCHES`` and allocations, and every pointer that they were given lies in an argument, in a tensor that the run
allocated or in one that outlives the recording, the launches serve later calls of the same signature with other pointers. Otherwise
(torch kernels, reads on the host, random numbers, meshes, operations of other modules, shared results) the schedule keeps being run by
Python. ``graph_call`` does the same for a schedule that was captured into a CUDA graph.
"""
from __future__ import annotations

import ctypes
import os

import torch
from torch.utils._python_dispatch import TorchDispatchMode, _get_current_dispatch_mode

from .. import config, native
from ..core.common import pytree
from ..core.tensor.api import Tensor
from ..core.tensor.impl import TensorImpl

# launch functions: all of their effects are on the device and on the stream that is their last argument
LAUNCHES = frozenset("""nb_gemm_bf16 nb_gemm_dual_bf16 nb_attn_fwd nb_attn_bwd nb_layernorm_fwd nb_layernorm_bwd nb_colsum nb_colsum_group nb_softmax
    nb_lse_pick_fwd nb_lse_pick_bwd nb_adamw nb_adamw_group nb_adam_hyper nb_mean_diff nb_sgd nb_embedding_gather nb_embedding_scatter_add
    nb_cast nb_activation nb_nf4_dequant nb_nf4_dequant_codes nb_pool2d_fwd nb_pool2d_bwd nb_pool2d_select nb_conv2d_direct nb_conv_flip
    nb_conv2d_wgrad_direct nb_sgemm nb_sum_slices nb_binary nb_unary nb_reduce nb_cumsum""".split())
# functions of sizes alone
QUERIES = frozenset("""nb_layernorm_bwd_nblocks nb_colsum_nparts nb_conv2d_wgrad_slices nb_sgemm_slices nb_reduce_splits
    nb_embedding_scatter_work""".split())
# switches that the wrappers read on every call
ENVIRONMENT = ("NABLA_B200_DISABLE_NATIVE", "NABLA_B200_ATTENTION", "NABLA_B200_ATTENTION_BWD", "NABLA_B200_ELEMENTWISE", "NABLA_B200_LN_BWD",
               "NABLA_B200_OPTIMIZER_STREAM", "NABLA_B200_TAPE")
_ALLOCATIONS = frozenset(("aten::empty", "aten::empty_strided", "aten::empty_like", "aten::new_empty"))
_VIEWS = frozenset(("aten::view", "aten::_unsafe_view", "aten::_reshape_alias", "aten::permute", "aten::transpose", "aten::t", "aten::unsqueeze",
                    "aten::squeeze", "aten::expand", "aten::as_strided", "aten::slice", "aten::select", "aten::alias", "aten::detach"))
MAX_SCRATCH = 256 << 20       # above, the device's time is far more than the host's, and pieces fit where one block may not
INT, FLOAT, DOUBLE, POINTER, STREAM, BLOB = range(6)
_POINTER_TYPES = (ctypes.c_void_p,)

_module = None


def module():
    """The extension, or None where it is not built, or not for this Python and torch (then Python replays)."""
    global _module
    if _module is None:
        _module = _load() or False
    return _module or None


def _load():
    import importlib.machinery
    import importlib.util
    import warnings

    from ..csrc.build import replay_built_for

    path = native.lib_path("libnb_replay.so")
    if not path.exists():
        return None
    loader = importlib.machinery.ExtensionFileLoader("libnb_replay", str(path))
    try:
        m = importlib.util.module_from_spec(importlib.util.spec_from_file_location("libnb_replay", str(path), loader=loader))
        loader.exec_module(m)
        if m.built_for != replay_built_for():
            raise ImportError(f"it was built for {m.built_for}, this is {replay_built_for()}")
        m.classes(Tensor, TensorImpl)
    except (ImportError, OSError, AttributeError, TypeError) as e:
        warnings.warn(f"{path.name} cannot be used, compiled calls are replayed by Python (python -m nabla_b200.csrc.build builds it anew): {e}")
        return None
    return m


class _Refused(Exception):
    pass


def tree_of(td) -> tuple:
    """A structure as ``replay.cpp`` reads it; registered containers are refused."""
    kinds = {"leaf": b"x", "none": b"n", "list": b"l", "tuple": b"t", "dict": b"d"}
    if td.kind not in kinds:
        raise _Refused(f"a container of type {td.kind}")
    return (kinds[td.kind], tuple(td.meta) if td.kind == "dict" else None, tuple(tree_of(c) for c in td.children))


class _Recorder(TorchDispatchMode):
    """Allocations, launches and the first thing that speaks against a tape."""

    def __init__(self):
        super().__init__()
        self.why = None
        self.allocated: list[tuple[int, int]] = []      # first byte and the one behind the last; not kept alive
        self.launches: list[tuple] = []           # (name, function, argument types, arguments, code, allocations so far)

    def refuse(self, why: str) -> None:
        self.why = self.why or why

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        out = func(*args, **(kwargs or {}))
        name = func.name().split(".")[0]
        if name in _ALLOCATIONS:
            if not (isinstance(out, torch.Tensor) and out.is_cuda and out.layout == torch.strided):
                self.refuse(f"{name} elsewhere than on the GPU")
            else:
                self.allocated.append(_span(out))
        elif name not in _VIEWS:
            self.refuse(name)
        return out

    def function(self, name: str, fn):
        """``fn`` of a library as the wrappers call it while this recorder is on."""
        if name in QUERIES:
            return fn
        if name not in LAUNCHES:
            self.refuse(name)
            return fn

        def launch(*args):
            rc = fn(*args)
            self.launches.append((name, fn, fn.argtypes, args, rc, len(self.allocated)))
            return rc

        return launch

    def library(self, lib):
        return _Library(self, lib)


class _Library:
    def __init__(self, recorder, lib):
        self._recorder, self._lib = recorder, lib

    def __getattr__(self, name):
        return self._recorder.function(name, getattr(self._lib, name))


def _span(t: torch.Tensor) -> tuple[int, int]:
    s = t.untyped_storage()
    return s.data_ptr(), s.data_ptr() + s.nbytes()


def _value(arg) -> int:
    v = arg.value if isinstance(arg, ctypes._SimpleCData) else arg
    return int(v or 0)


def can_record(rec) -> bool:
    """Is this a call whose launches all go through the wrappers that are observed? A recording of which none is says so once (``rec.tape``)."""
    if not _recordable(rec):
        rec.tape = False
        return False
    return (module() is not None and os.environ.get("NABLA_B200_TAPE", "1") != "0" and not rec.arena_blocks
            and not torch.cuda.is_current_stream_capturing() and _get_current_dispatch_mode() is None
            and not config.get_flag("VERIFY_EAGER_SHAPES"))


def _recordable(rec) -> bool:
    """What of it the recording decides."""
    def own(op) -> bool:
        m = type(op).__module__
        return m.startswith(("nabla_b200.ops.", "nabla_b200.nn.finetune.")) and not m.endswith((".custom", ".custom_op", ".communication")) \
            and ".communication." not in m

    return bool(not rec.host_sync and not rec.side_steps and not any(rec.donated)
                and rec.placeholders and all(p.sharding is None and p.device.label == "gpu" for p in rec.placeholders)
                and all(own(n.op) and all(o is None or o.sharding is None for o in n.outputs()) for n in rec.nodes))


def _leaves(tensors) -> list:
    return [(im._shape, im._dtype, im.batch_dims, im._device, im._buffers[0]) for im in (t._impl for t in tensors)]


def _environment() -> list:
    return [(n.encode(), os.environ[n].encode() if n in os.environ else None) for n in ENVIRONMENT]


def _device(tensors) -> int:
    dev = {t._impl._buffers[0].device for t in tensors}
    if len(dev) != 1 or any(len(t._impl._buffers) != 1 or t._impl.sharding is not None for t in tensors):
        raise _Refused("arguments on several devices")
    index = dev.pop().index
    if index != torch.cuda.current_device():
        raise _Refused("not the current device")
    return index


def record(rec, tensors: list, tds: tuple, run, collect):
    """Run the schedule (``run``), collect its result, and return (result, tape or None, why not)."""
    r = _Recorder()
    native.set_recorder(r)
    try:
        with r:
            run()
    finally:
        native.set_recorder(None)
    result_buffers = [list(i._buffers) if i is not None else None for i in rec.out_impls]
    result = collect()
    try:
        if r.why:
            raise _Refused(r.why)
        return result, _tape(rec, tensors, tds, r, result_buffers), None
    except _Refused as e:
        return result, None, str(e)


def _captured(rec) -> list[TensorImpl]:
    """Tensors that the function found outside of its arguments, and its numbers."""
    placeholders = {id(p) for p in rec.placeholders}
    return list({id(a): a for n in rec.nodes for a in n.input_impls() if id(a) not in placeholders and a.output_refs is None and a._buffers}.values())


def _constants(rec) -> list[torch.Tensor]:
    """Tensors that outlive the recording's calls: captured by the function, made with the plan, or the library's own."""
    from ..nn.finetune import qlora

    out = [b for a in _captured(rec) for b in a._buffers]
    out += [b for o in rec.constants for b in o._buffers]
    out += list(native._status.values())
    out += list(qlora._CODEBOOKS.values())
    return [t for t in out if t.is_cuda and t.numel()]


def _tape(rec, tensors, tds, r: _Recorder, result_buffers):
    device = _device(tensors)
    bases = [t._impl._buffers[0] for t in tensors]
    spans = [_extent(t) for t in bases]
    if any(len(a._buffers) != 1 for a in _captured(rec)):
        raise _Refused("a captured tensor in pieces")
    constants = [_span(t) for t in _constants(rec)]
    order = sorted(s for s in spans if s[0] != s[1])
    if any(a[1] > b[0] for a, b in zip(order, order[1:])) or any(lo < s[1] and s[0] < hi for s in order for lo, hi in constants):
        raise _Refused("arguments that share memory")       # of this call; the next may be told apart
    allocated = r.allocated
    # results: whole allocations of this run, one each
    outs, result_of = [], {}
    n_in = len(tensors)
    for k, (impl, static, bufs) in enumerate(zip(rec.out_impls, rec.out_static, result_buffers)):
        if impl is None:
            outs.append((static,))
            continue
        (b,) = bufs if len(bufs) == 1 else (None,)
        if b is None:
            raise _Refused("a result in pieces")
        lo, hi = _span(b)
        own = [i for i, s in enumerate(allocated) if s == (lo, hi) and lo != hi]
        if not own or b.storage_offset() or b.data_ptr() != lo or own[-1] in result_of or _extent(b) != (lo, lo + _dense_bytes(b)) \
                or not _is_whole(b, hi - lo):
            raise _Refused("a result that shares its memory")
        result_of[own[-1]] = n_in + k
        outs.append((b, TensorImpl.result_like(impl, [b])))
    # an address belongs to the latest allocation in front of the launch, then to an argument, then to what outlives the call
    uses: dict[int, list[int]] = {}
    found: list[tuple] = []

    def place(p: int, upto: int, at: int):
        for i in range(upto - 1, -1, -1):
            lo, hi = allocated[i]
            if lo <= p < hi:
                uses.setdefault(i, []).append(at)
                return ("alloc", i, p - lo)
        for i, (lo, hi) in enumerate(spans):
            if lo <= p < hi:
                return ("in", i, p - lo)
        if any(lo <= p < hi for lo, hi in constants):
            return None
        raise _Refused("a pointer of unknown origin")

    for at, (name, fn, types, args, rc, upto) in enumerate(r.launches):
        if len(types) != len(args):
            raise _Refused(f"arguments of {name}")
        row = []
        for k, (ty, arg) in enumerate(zip(types, args)):
            if ty is ctypes.c_float:
                row.append((FLOAT, float(arg)))
            elif ty is ctypes.c_double:
                row.append((DOUBLE, float(arg)))
            elif ty not in _POINTER_TYPES:
                row.append((INT, _value(arg)))
            elif k == len(args) - 1:
                row.append((STREAM,))
            elif isinstance(arg, ctypes.Array):
                patches = []
                if arg._type_ in _POINTER_TYPES:
                    for j, v in enumerate(arg):
                        w = place(v, upto, at) if v else None
                        if w is not None:
                            patches.append((j * ctypes.sizeof(arg._type_), w))
                row.append((BLOB, bytes(arg), patches))
            else:
                p = _value(arg)
                w = place(p, upto, at) if p else None
                row.append((INT, p) if w is None else (POINTER, w))
        found.append((ctypes.cast(fn, ctypes.c_void_p).value, rc, name.encode(), row))
    # scratch: what is neither argument nor result, each from its first to its last launch, in one block
    blocks, scratch = {}, 0
    for i in sorted(i for i in uses if i not in result_of):
        size = -(-(allocated[i][1] - allocated[i][0]) // 512) * 512
        first, last = min(uses[i]), max(uses[i])
        lo = 0
        for at_, n, f, l in sorted(blocks.values()):
            if f <= last and first <= l and at_ < lo + size and lo < at_ + n:
                lo = at_ + n
        blocks[i] = (lo, size, first, last)
        scratch = max(scratch, lo + size)
    if scratch > MAX_SCRATCH:
        raise _Refused(f"{scratch} bytes of scratch")
    n_bases = n_in + len(outs)

    def base(w) -> tuple[int, int]:
        kind, i, off = w
        if kind == "in":
            return i, off - (bases[i].data_ptr() - spans[i][0])
        return (result_of[i], off) if i in result_of else (n_bases, blocks[i][0] + off)

    launches = []
    for address, rc, name, row in found:
        out = []
        for e in row:
            if e[0] == POINTER:
                out.append((POINTER, *base(e[1])))
            elif e[0] == BLOB:
                out.append((BLOB, e[1], [(at, *base(w)) for at, w in e[2]]))
            else:
                out.append(e)
        launches.append((address, rc, name, out))
    return module().make((tuple(tree_of(td) for td in tds), _leaves(tensors), _environment(), device, config.is_deterministic(), launches,
                          scratch, outs, tree_of(rec.out_treedef), None, [a for a in _captured(rec) if a.literal is None], rec.owned or []))


def _extent(t: torch.Tensor) -> tuple[int, int]:
    """First byte of a tensor and the one behind its last."""
    if not t.numel():
        return t.data_ptr(), t.data_ptr()
    lo = hi = t.data_ptr()
    for n, s in zip(t.shape, t.stride()):
        hi += (n - 1) * s * t.element_size()
    return lo, hi + t.element_size()


def _dense_bytes(t: torch.Tensor) -> int:
    return t.numel() * t.element_size()


def _is_whole(t: torch.Tensor, nbytes: int) -> bool:
    from ..native.kernels import _is_dense

    return _is_dense(t) and _dense_bytes(t) == nbytes


def graph_call(rec, tensors: list, tds: tuple):
    """A tape of a schedule in a CUDA graph: copies in, the graph, copies out. None where torch makes some of the copies."""
    try:
        if module() is None or os.environ.get("NABLA_B200_TAPE", "1") == "0" or any(rec.donated) or rec.static_ptrs \
                or any(c is not None for c in rec.out_cached):
            return None
        device = _device(tensors)
        ins, outs_ = rec.copy_in, rec.copy_out
        if not all(ins.plain) or not all(outs_.plain) or outs_.all_sizes is None or len(ins.fixed) != len(tensors) \
                or any(t._impl._buffers[0].stride() != s for t, s in zip(tensors, ins.strides)):
            return None
        outs, k = [], 0
        for impl, static, bufs in zip(rec.out_impls, rec.out_static, rec.static_outputs):
            if impl is None:
                outs.append((static,))
                continue
            if len(bufs) != 1:
                return None
            outs.append((bufs[0], TensorImpl.result_like(impl, list(bufs))))
            k += 1
        if k != len(outs_.fixed):
            return None
        from ..native.kernels import _L

        address = ctypes.cast(_L().nb_copy_batch, ctypes.c_void_p).value
        graph = (rec.cuda_graph.replay, address, [(t.data_ptr(), n) for t, n in zip(ins.fixed, ins.size)],
                 [(t.data_ptr(), n) for t, n in zip(outs_.fixed, outs_.size)])
        return module().make((tuple(tree_of(td) for td in tds), _leaves(tensors), _environment(), device, config.is_deterministic(), [], 0, outs,
                              tree_of(rec.out_treedef), graph, [], [*ins.fixed, *outs_.fixed, *(rec.owned or [])]))
    except _Refused:
        return None
