"""Plan construction with peephole fusion.

``build_plan`` turns a topologically ordered node list into steps. Patterns recognised on
CUDA bf16 tensors:

* ``matmul -> add(bias row) [-> relu | gelu]`` where the intermediates have no other
  consumer: one tcgen05 GEMM launch with the bias/activation epilogue
  (replaces the composition of nabla/nn/functional/layers.py:30-35).

* ``matmul | linear (no bias) -> all_reduce(sum) | reduce_scatter`` on a mesh that runs one
  process per GPU: one launch of the fused GEMM + collective kernel (tiles are reduced over
  NVLink while later tiles are still being multiplied).
* ``linear (+bias) | matmul -> add(residual)``: the residual is added in the GEMM epilogue (compiled replays).
* ``x @ w [+ b] + (h @ v) [* a power of two]`` with a K of h of up to 256 (a frozen weight and its adapter): one launch, whose accumulator takes both
  products (compiled replays).
* ``matmul -> mul(one element)`` and ``mul(one element) -> matmul ...`` (the scale of a LoRA adapter and its gradient): the
  factor is applied in the GEMM epilogue (compiled replays).
* ``layer norm backward -> add``: the gradient that joins dx is added in the same pass (compiled replays).
* ``linear`` with an activation whose pre-activation nobody reads (inference): it is not written (compiled replays).
* ``matmul -> dact_mul`` (backward of linear + relu/gelu): the activation derivative is applied in
  the GEMM epilogue.
* ``sub -> [mul with itself ->] sums over all axes -> division by a number``: the mean of a cross-entropy or a squared error, one
  launch that also leaves the difference where the backward reads it (compiled replays).
* ``x * y + x * y`` (the gradient of a square): one pass (compiled replays).
* ``add(number) -> adam_hyper``: the step count and what follows from it, one launch (compiled replays).
* compiled replays with donated optimizer state: ``matmul -> all_reduce(dp) -> adam_wstep`` becomes a
  GEMM that writes its (unreduced) weight gradient into a symmetric arena plus one kernel that sums
  the ranks' gradients while reading them and applies AdamW in place (``gemm_to_arena`` /
  ``adamw_reduce`` steps, set up by ``transforms/compile.py``).
* ``all_gather(rows) -> linear | matmul [-> dact_mul]``: one launch that pulls the peers' rows while the tensor
  cores already work on the rows that are there; the gathered tensor is still produced.
* ``conv2d -> relu`` whose pre-activation is read by nothing but the relu's derivative, and ``max pooling backward -> relu's derivative``:
  one launch each (compiled replays).
* ``zeros -> scatter-add``: the gradient of an embedding table without the table of zeros.
* ``gather -> add`` of a tensor over the trailing dims (token plus position embedding): one pass (compiled replays).
* ``adamw_group``: the updates of small parameters with the same hyperparameters, one launch at the end of a compiled
  schedule (grouped by ``transforms/compile.py``).
* ``sum -> sum ...`` over neighbouring axes: one reduction over the joined axes, where ``kernels.joined_sum`` takes it.

Every other node is a plain 'op' step. Fusion never changes which tensors exist: fused-away
intermediates that are still referenced are simply not fusable.
"""
from __future__ import annotations

import math
import os

import torch

from ..tensor.impl import TensorImpl
from .tracing import OpNode


_FUSE_RESIDUAL = os.environ.get("NABLA_B200_FUSE_RESIDUAL", "0") == "1"


def enabled() -> bool:
    return os.environ.get("NABLA_B200_NO_PLAN", "0") != "1"


def _single_consumer_map(nodes: list[OpNode], targets) -> dict[int, list[int]]:
    cons: dict[int, list[int]] = {}
    for ni, n in enumerate(nodes):
        for a in n.arg_leaves:
            if isinstance(a, TensorImpl):
                cons.setdefault(id(a), []).append(ni)
    return cons


def build_plan(nodes: list[OpNode], targets: list[TensorImpl], private: bool = False):
    """``private``: nobody outside ``nodes`` can ask for an intermediate later (a compiled recording), so values that
    autodiff traced through may be fused away too when no node reads them."""
    from .engine import Plan

    cons = _single_consumer_map(nodes, targets)
    target_ids = {id(t) for t in targets}
    pos = {id(n): i for i, n in enumerate(nodes)}
    used = [False] * len(nodes)
    steps = []
    producer: dict[int, int] = {}
    for ni, nd in enumerate(nodes):
        for o_ in nd.outputs():
            if o_ is not None:
                producer[id(o_)] = ni

    def sole_output(n: OpNode):
        outs = n.outputs()
        return outs[0] if len(outs) == 1 else None

    def fusable_intermediate(impl: TensorImpl) -> bool:
        # only this plan consumes it, exactly once; not requested by the caller; not traced
        return (impl is not None and id(impl) not in target_ids and not impl.is_traced
                and len(cons.get(id(impl), [])) == 1 and impl.sharding is None and impl.batch_dims == 0)

    def private_intermediate(impl: TensorImpl) -> bool:
        return (impl is not None and id(impl) not in target_ids and len(cons.get(id(impl), [])) == 1
                and impl.sharding is None and impl.batch_dims == 0)

    def heads_epilogue(j: int) -> bool:
        """Is product ``j`` to be fused with the activation gradient or the bias behind it?"""
        o = sole_output(nodes[j])
        if _is_local_gemm(nodes[j]) and _dact_consumer(nodes[j], nodes, cons, target_ids, used) is not None:
            return True
        if not fusable_intermediate(o):
            return False
        k = cons[id(o)][0]
        return not used[k] and nodes[k].op.name == "add" and _is_bias_add(nodes[k], o)

    for i, n in enumerate(nodes):
        if used[i]:
            continue
        chain = None
        if n.op.name == "matmul" and _is_cuda_bf16_2d(n):
            o = sole_output(n)
            if fusable_intermediate(o):
                j = cons[id(o)][0]
                m = nodes[j]
                if not used[j] and m.op.name == "add" and _is_bias_add(m, o):
                    chain = [i, j]
                    o2 = sole_output(m)
                    if fusable_intermediate(o2):
                        k = cons[id(o2)][0]
                        a = nodes[k]
                        if not used[k] and a.op.name in ("relu", "gelu") and not (
                                a.op.name == "gelu" and a.kwargs.get("approximate", "none") not in ("none", "tanh")):
                            chain = [i, j, k]
        kind = "linear_epilogue"
        if chain is None and private and n.op.name == "linear" and n.kwargs.get("activation") in ("relu", "gelu", "gelu_tanh") \
                and _is_plain_gemm(n) and len(n.outputs()) == 2 and n.outputs()[0] is not None:
            z = n.outputs()[1]
            if z is None or (id(z) not in target_ids and not cons.get(id(z))):
                chain = [i]
                kind = "linear_act"
        if chain is None and private and n.op.name == "gather" and _is_table_gather(n):
            o = sole_output(n)
            if private_intermediate(o):
                j = cons[id(o)][0]
                m = nodes[j]
                if not used[j] and m.op.name == "add" and _is_trailing_add(m, o):
                    chain = [i, j]
                    kind = "gather_add"
        if chain is None and n.op.name == "full":
            # zeros -> scatter-add (the gradient of an embedding): the kernel writes every row once and
            # takes no base at all, so the zeros are neither written nor read
            o = sole_output(n)
            if fusable_intermediate(o) and _is_zero_table(n, o):
                j = cons[id(o)][0]
                if not used[j] and _is_scatter_add_into(nodes[j], o):
                    chain = [i, j]
                    kind = "scatter_zeros"
        if chain is None and private and n.op.name == "conv2d":
            k = _relu_behind(n, nodes, cons, target_ids)
            if k is not None and not used[k]:
                used[i] = used[k] = True
                steps.append((i, ("conv_relu", (i, k))))
                continue
        if chain is None and private and n.op.name == "pool2d_bwd" and n.kwargs.get("mode") == "max" and _is_plain_gpu(n):
            o = sole_output(n)
            if private_intermediate(o):
                k = cons[id(o)][0]
                d = nodes[k]
                x = n.input_impls()[0]
                if not used[k] and d.op.name == "dact_mul" and d.kwargs.get("activation") == "relu" and d.input_impls()[0] is o \
                        and len(d.input_impls()) == 2:
                    z = d.input_impls()[1]
                    p = nodes[producer[id(x)]] if id(x) in producer else None
                    if z is x or (p is not None and p.op.name == "relu" and p.input_impls()[0] is z):
                        chain = [i, k]
                        kind = "pool_bwd_relu"
        if chain is None and private and n.op.name == "sub":
            idxs = _mean_of_difference(i, nodes, cons, target_ids, used, producer, private_intermediate)
            if idxs is not None:
                for c in idxs:
                    used[c] = True
                steps.append((i, ("mean_diff", tuple(idxs))))       # where the difference was made: others may read it
                continue
        if chain is None and private and n.op.name == "mul" and _is_plain_binary(n):
            # x * y + x * y
            o = sole_output(n)
            if private_intermediate(o):
                k = cons[id(o)][0]
                a_ = nodes[k]
                if not used[k] and a_.op.name == "add" and _is_plain_binary(a_):
                    other = [x for x in a_.input_impls() if x is not o]
                    j = producer.get(id(other[0]), -1) if len(other) == 1 else -1
                    if j > i and not used[j] and nodes[j].op.name == "mul" and private_intermediate(other[0]) \
                            and {id(x) for x in nodes[j].input_impls()} == {id(x) for x in n.input_impls()} and len(nodes[j].input_impls()) == 2:
                        chain = [i, j, k]
                        kind = "twice_product"
        if chain is None and private and n.op.name == "add" and _is_plain_binary(n):
            # step + 1 -> [lr, 1 - b1^t, 1 - b2^t, 1]
            o = sole_output(n)
            j = min(cons.get(id(o), [i])) if o is not None else i
            if j != i and not used[j] and nodes[j].op.name == "adam_hyper" and _is_counted_step(n, o):
                used[i] = used[j] = True
                steps.append((i, ("next_step", (i, j))))
                continue
        if chain is None and n.op.name == "reduce_sum" and _is_plain_sum(n) \
                and n.kwargs["axis"] < len(n.input_impls()[0]._shape) - 1:
            # sums over neighbouring axes, one after the other (``sum(axis=(0, 1, 2))``): one reduction over
            # as many joined axes as the kernels' rule takes, without the partial results and their rounding.
            # Not where the last axis is among them: one long row would be left to one warp
            from ...native import kernels

            idxs, lo, hi = [i], n.kwargs["axis"], n.kwargs["axis"]
            x0 = n.input_impls()[0]
            last_axis, joined = len(x0._shape) - 1, 1
            while True:
                o = sole_output(nodes[idxs[-1]])
                if not fusable_intermediate(o):
                    break
                j = cons[id(o)][0]
                m = nodes[j]
                if used[j] or m.op.name != "reduce_sum" or not _is_plain_sum(m) or m.kwargs["axis"] not in (lo - 1, lo) \
                        or (m.kwargs["axis"] == lo and hi + 1 == last_axis):
                    break
                if m.kwargs["axis"] == lo:
                    hi += 1
                else:
                    lo -= 1
                idxs.append(j)
                if kernels.joined_sum(math.prod(x0._shape[:lo]), math.prod(x0._shape[lo:hi + 1]), math.prod(x0._shape[hi + 1:]),
                                      x0.dtype.to_torch()):
                    joined = len(idxs)
            if joined > 1:
                chain = idxs[:joined]
                kind = "sum_axes"
        if chain is None and n.op.name == "matmul" and _is_local_gemm(n):
            dk = _dact_consumer(n, nodes, cons, target_ids, used)
            if dk is not None:
                chain = [i, dk]
                kind = "gemm_dact"
        if chain is None and private and n.op.name in ("matmul", "linear"):
            dual = _sum_of_products(i, nodes, cons, used, producer, private_intermediate, heads_epilogue)
            if dual is not None:
                chain = dual
                kind = _DUAL[len(dual) - 3]
        if chain is None and private and n.op.name == "matmul" and _is_cuda_bf16_2d(n):
            # x @ w * s with one element s
            o = sole_output(n)
            if private_intermediate(o):
                j = cons[id(o)][0]
                if not used[j] and nodes[j].op.name == "mul" and _scalar_factor(nodes[j], o) is not None:
                    chain = [i, j]
                    kind = "gemm_scale"
        if chain is None and private and n.op.name == "mul":
            # x * s with one element s, read by nothing but GEMMs, none of which takes more than this pass into its own epilogue
            o = sole_output(n)
            readers = cons.get(id(o), []) if o is not None else []
            if readers and id(o) not in target_ids and o.sharding is None and not o.batch_dims and len(set(readers)) == len(readers) \
                    and any(_scalar_factor(n, x) is not None for x in n.input_impls()) \
                    and all(not used[j] and nodes[j].op.name == "matmul" and _is_cuda_bf16_2d(nodes[j]) and not heads_epilogue(j) for j in readers):
                used[i] = True
                for j in readers:
                    used[j] = True
                    steps.append((j, ("scale_gemm", (i, j))))
                continue
        if chain is None and private and n.op.name in ("linear", "matmul") and n.kwargs.get("activation") is None \
                and _is_plain_gemm(n):
            # a residual of the same shape goes into the epilogue; of two products that are added, into the one with more to
            # multiply
            o = sole_output(n)
            if private_intermediate(o):
                k = cons[id(o)][0]
                a_ = nodes[k]
                if not used[k] and a_.op.name == "add" and _same_layout_addend(a_, o):
                    other = [x for x in a_.input_impls() if x is not o][0]
                    p = nodes[producer[id(other)]] if id(other) in producer else None
                    if p is None or p.op.name not in ("linear", "matmul") or not _is_plain_gemm(p) or used[producer[id(other)]] \
                            or p.input_impls()[0]._shape[-1] <= n.input_impls()[0]._shape[-1]:
                        chain = [i, k]
                        kind = "gemm_residual"
        if chain is None and private and n.op.name == _LN_BWD_NAME and _is_plain_ln_bwd(n):
            o = n.outputs()[0]
            if private_intermediate(o):
                k = cons[id(o)][0]
                a_ = nodes[k]
                if not used[k] and a_.op.name == "add" and _same_layout_addend(a_, o):
                    other = [x for x in a_.input_impls() if x is not o][0]
                    # the step runs where the layer norm's does, so that dgamma and dbeta are no later than before
                    if producer.get(id(other), -1) < i:
                        used[i] = used[k] = True
                        steps.append((i, ("ln_bwd_add", (i, k))))
                        continue
        if chain is None and _FUSE_RESIDUAL and n.op.name == "linear" and n.kwargs.get("activation") is None \
                and _is_local_linear(n):
            # y = x @ w + b followed by "+ residual" of the same shape: the residual is added in the epilogue
            o = sole_output(n)
            if (o is not None and id(o) not in target_ids and len(cons.get(id(o), [])) == 1 and o.batch_dims == 0
                    and not (o.sharding is not None and o.sharding.partial_sum_axes)):
                k = cons[id(o)][0]
                a_ = nodes[k]
                if not used[k] and a_.op.name == "add" and _same_layout_addend(a_, o):
                    chain = [i, k]
                    kind = "gemm_residual"
        if chain is None and n.op.name in ("matmul", "linear") and _is_partial_gemm(n):
            o = sole_output(n)
            # a traced product may stay an unrealized promise: no backward rule reads its value
            if o is not None and id(o) not in target_ids and len(cons.get(id(o), [])) == 1 and o.batch_dims == 0:
                j = cons[id(o)][0]
                m = nodes[j]
                if not used[j] and m.op.name == "all_reduce" and _is_sum_over_partials(m, o):
                    chain = [i, j]
                    kind = "gemm_all_reduce"
                elif not used[j] and m.op.name == "reduce_scatter" and _is_scatter_of_partials(m, o):
                    chain = [i, j]
                    kind = "gemm_reduce_scatter"
                    # + bias row and + residual fold into the pass that sums the partial row blocks
                    cur = sole_output(m)
                    for want in ("bias", "residual"):
                        if cur is None or id(cur) in target_ids or len(cons.get(id(cur), [])) != 1 or cur.batch_dims:
                            break
                        k = cons[id(cur)][0]
                        a = nodes[k]
                        if used[k] or a.op.name != "add" or _rs_addend(a, cur) != want:
                            if want == "bias":
                                continue          # no bias: the next add may still be the residual
                            break
                        chain.append(k)
                        cur = sole_output(a)
        if chain is None and n.op.name == "all_gather" and _is_row_gather(n):
            o = sole_output(n)
            users = cons.get(id(o), []) if o is not None else []
            if o is not None and users and o.batch_dims == 0:
                j = min(users)
                m = nodes[j]
                if not used[j] and m.op.name in ("matmul", "linear") and _is_gathered_gemm(m, o):
                    # the GEMM may move up to right after its other inputs exist, but not past
                    # another user of the gathered tensor
                    ready = i
                    for x in m.input_impls():
                        if x is not o and id(x) in producer:
                            ready = max(ready, producer[id(x)])
                    idxs = [i, j]
                    dk = _dact_consumer(m, nodes, cons, target_ids, used)
                    if dk is not None:
                        z = nodes[dk].input_impls()[1]
                        zr = producer.get(id(z), -1)
                        if max(ready, zr) < j:
                            ready = max(ready, zr)
                            idxs.append(dk)
                    if ready < j and all(u > ready for u in users):
                        for c_ in idxs:
                            used[c_] = True
                        steps.append((ready + 0.5, ("all_gather_gemm", tuple(idxs))))
                        continue
        if chain is not None:
            # schedule at the position of the LAST node of the chain
            last = chain[-1]
            for c in chain:
                used[c] = True
            steps.append((last, (kind, tuple(chain))))
        else:
            used[i] = True
            steps.append((i, ("op", (i,))))
    steps.sort(key=lambda s: s[0])
    return Plan([s for _, s in steps], len(nodes))


def _is_cuda_bf16_2d(n: OpNode) -> bool:
    ins = n.input_impls()
    if len(ins) != 2:
        return False
    a, b = ins
    if a.sharding is not None or b.sharding is not None or a.batch_dims or b.batch_dims:
        return False
    from ...types import DType

    return (a.device.label == "gpu" and a.dtype is DType.bfloat16 and b.dtype is DType.bfloat16
            and len(b._shape) == 2 and len(a._shape) >= 2)


def _is_plain_gpu(n: OpNode) -> bool:
    """Unsharded fp32 / bf16 GPU operands of one type and the result too."""
    from ...types import DType

    xs = [*n.input_impls(), *n.outputs()]
    return all(x is not None and x.sharding is None and not x.batch_dims and x.device.label == "gpu" and x.dtype is xs[0].dtype for x in xs) \
        and xs[0].dtype in (DType.bfloat16, DType.float32)


def _relu_behind(n: OpNode, nodes, cons, target_ids) -> int | None:
    """The relu behind ``n`` when its result z is read by nothing else but derivatives of a relu: those ask whether z is above 0,
    which the relu's own result answers as well, so z need not exist."""
    outs = n.outputs()
    z = outs[0] if len(outs) == 1 else None
    if z is None or id(z) in target_ids or not _is_plain_gpu(n):
        return None
    relus = []
    for j in dict.fromkeys(cons.get(id(z), [])):
        m = nodes[j]
        if m.op.name == "relu" and len(m.input_impls()) == 1:
            relus.append(j)
        elif not (m.op.name == "dact_mul" and m.kwargs.get("activation") == "relu" and m.input_impls()[1] is z and m.input_impls()[0] is not z):
            return None
    return relus[0] if len(relus) == 1 and nodes[relus[0]].outputs()[0] is not None else None


def _is_plain_binary(n: OpNode) -> bool:
    """Two unsharded fp32 / bf16 GPU operands of the result's type."""
    from ...types import DType

    ins, outs = n.input_impls(), n.outputs()
    o = outs[0] if len(outs) == 1 else None
    return (len(ins) == 2 and o is not None and o.sharding is None and not o.batch_dims and o.dtype in (DType.bfloat16, DType.float32)
            and all(x.sharding is None and not x.batch_dims and x.device.label == "gpu" and x.dtype is o.dtype and x.device == o.device
                    for x in ins))


def _mean_of_difference(i: int, nodes, cons, target_ids, used, producer, private_intermediate) -> list[int] | None:
    """[sub, (mul,) reduce_sum..., div | divide_by_count] when node ``i`` begins a mean over all elements of ``a - b`` or of its
    square, whose sums nobody else reads. The difference itself may have other readers where it is squared."""
    n = nodes[i]
    if not _is_plain_binary(n):
        return None
    a, b = n.input_impls()
    d = n.outputs()[0]
    numel = math.prod(int(s) for s in d._shape)
    if tuple(a._shape) != tuple(b._shape) or not 0 < numel <= 1 << 18 or not d._shape:
        return None
    idxs, cur = [i], d
    readers = cons.get(id(d), [])
    squares = [j for j in dict.fromkeys(readers) if nodes[j].op.name == "mul" and all(x is d for x in nodes[j].input_impls())]
    if squares:
        if len(squares) != 1 or used[squares[0]]:
            return None
        idxs.append(squares[0])
        cur = nodes[squares[0]].outputs()[0]
    while True:
        if not private_intermediate(cur):
            return None
        j = cons[id(cur)][0]
        m = nodes[j]
        if used[j]:
            return None
        if m.op.name == "reduce_sum" and _is_plain_sum(m):
            idxs.append(j)
            cur = m.outputs()[0]
            if cur is None:
                return None
            continue
        if len(cur._shape) or cur is d:
            return None
        if m.op.name == "divide_by_count" and m.outputs()[0] is not None:
            return idxs + [j]
        if m.op.name == "div" and _is_plain_binary(m) and m.input_impls()[0] is cur and m.input_impls()[1].literal is not None \
                and not m.input_impls()[1]._shape:
            return idxs + [j]
        return None


_DUAL = ("gemm+gemm_residual", "gemm_scale+gemm_residual")       # a sum of two products, without a factor and with one


def _sum_of_products(i: int, nodes, cons, used, producer, private_intermediate, heads_epilogue) -> list[int] | None:
    """[small product, (its scale,) large product, add] in the order of the schedule when product ``i`` is one of two that are added. The
    small one has the shorter K, of up to 256, and perhaps a one-element factor behind it; nobody else reads either."""
    def branch(j: int):
        # (nodes from the product to what is added, the value that is added)
        if used[j] or nodes[j].op.name not in ("matmul", "linear") or nodes[j].kwargs.get("activation") is not None or not _is_plain_gemm(nodes[j]) \
                or heads_epilogue(j):
            return None
        o = nodes[j].outputs()[0]
        if not private_intermediate(o):
            return None
        k = cons[id(o)][0]
        if not used[k] and nodes[k].op.name == "mul" and _scalar_factor(nodes[k], o) is not None:
            v = nodes[k].outputs()[0]
            return ([j, k], v) if private_intermediate(v) else None
        return [j], o

    mine = branch(i)
    if mine is None:
        return None
    path, value = mine
    k = cons[id(value)][0]
    add = nodes[k]
    if used[k] or add.op.name != "add" or not _same_layout_addend(add, value):
        return None
    other = [x for x in add.input_impls() if x is not value][0]
    j = producer.get(id(other), -1)
    if j >= 0 and nodes[j].op.name == "mul" and not used[j]:
        firsts = [producer[id(x)] for x in nodes[j].input_impls() if id(x) in producer and _scalar_factor(nodes[j], x) is not None]
        j = firsts[0] if len(firsts) == 1 else -1
    theirs = branch(j) if j >= 0 and j != i else None
    if theirs is None or theirs[1] is not other:
        return None
    small, large = sorted((path, theirs[0]), key=lambda p: int(nodes[p[0]].input_impls()[0]._shape[-1]))
    depth = int(nodes[small[0]].input_impls()[0]._shape[-1])
    if depth > 256 or len(large) > 1 or len(nodes[small[0]].input_impls()) > 2 \
            or depth >= int(nodes[large[0]].input_impls()[0]._shape[-1]):
        return None
    return small + large + [k]


def _is_power_of_two(x) -> bool:
    """A number that scales bf16 values without rounding them."""
    return x is not None and 2.0 ** -64 <= x <= 2.0 ** 64 and math.frexp(x)[0] == 0.5


def _is_counted_step(add: OpNode, o: TensorImpl) -> bool:
    """``add`` of a number to the one fp32 element of a step count."""
    from ...types import DType

    ins = add.input_impls()
    return (o.dtype is DType.float32 and not o._shape and not ins[0]._shape and not ins[1]._shape and ins[0] is not ins[1]
            and any(x.literal is not None for x in ins))


def _is_table_gather(n: OpNode) -> bool:
    """Rows of an unsharded fp32 / bf16 GPU table."""
    from ...types import DType

    ins = n.input_impls()
    return (len(ins) == 2 and n.kwargs.get("axis") == 0 and not n.kwargs.get("bd", 0) and len(ins[0]._shape) == 2
            and all(x.sharding is None and not x.batch_dims for x in ins) and ins[0].device.label == "gpu"
            and ins[0].dtype in (DType.bfloat16, DType.float32))


def _is_trailing_add(add: OpNode, x: TensorImpl) -> bool:
    """``x`` plus a tensor of its dtype over its trailing dims (the last one at least)."""
    ins = add.input_impls()
    if len(ins) != 2:
        return False
    other = ins[1] if ins[0] is x else ins[0] if ins[1] is x else None
    if other is None or other is x or other.sharding is not None or other.batch_dims or other.dtype is not x.dtype \
            or other.device != x.device or len(other._shape) > len(x._shape):
        return False
    shp = tuple(other._shape)
    while len(shp) > 1 and shp[0] == 1:
        shp = shp[1:]
    return len(shp) >= 1 and tuple(x._shape)[len(x._shape) - len(shp):] == shp


def _is_zero_table(n: OpNode, o: TensorImpl) -> bool:
    from ...types import DType

    v = n.kwargs.get("value")
    return (isinstance(v, (int, float)) and v == 0 and o.device.label == "gpu" and len(o._shape) == 2
            and o.dtype in (DType.bfloat16, DType.float32))


def _is_scatter_add_into(n: OpNode, table: TensorImpl) -> bool:
    if n.op.name != "scatter" or n.kwargs.get("mode") != "add" or n.kwargs.get("axis") != 0 or n.kwargs.get("bd", 0):
        return False
    ins = n.input_impls()
    return len(ins) == 3 and ins[0] is table and all(x is not table for x in ins[1:]) \
        and all(x.sharding is None and not x.batch_dims for x in ins)


def _is_plain_sum(n: OpNode) -> bool:
    """Unsharded floating-point GPU sum that drops its axis."""
    from ...types import DType

    ins = n.input_impls()
    return (len(ins) == 1 and ins[0].sharding is None and not ins[0].batch_dims and ins[0].device.label == "gpu"
            and ins[0].dtype in (DType.bfloat16, DType.float32) and not n.kwargs.get("keepdims", False)
            and set(n.kwargs) <= {"axis", "keepdims"} and n.kwargs["axis"] >= 0)


def _is_local_gemm(n: OpNode) -> bool:
    """bf16 GPU ``x @ w`` (w 2-D) whose product needs no collective."""
    ins = n.input_impls()
    if len(ins) != 2:
        return False
    a, b = ins
    outs = n.outputs()
    o = outs[0] if len(outs) == 1 else None
    if o is None or (o.sharding is not None and o.sharding.partial_sum_axes):
        return False
    from ...types import DType

    return (a.device.label == "gpu" and a.dtype is DType.bfloat16 and b.dtype is DType.bfloat16
            and len(b._shape) == 2 and len(a._shape) >= 2 and a.batch_dims == 0 and b.batch_dims == 0)


def _is_local_linear(n: OpNode) -> bool:
    ins = n.input_impls()
    if len(ins) not in (2, 3):
        return False
    a, b = ins[0], ins[1]
    from ...types import DType

    return (a.device.label == "gpu" and a.dtype is DType.bfloat16 and b.dtype is DType.bfloat16
            and len(b._shape) == 2 and len(a._shape) >= 2 and a.batch_dims == 0 and b.batch_dims == 0)


def _is_plain_gemm(n: OpNode) -> bool:
    """Unsharded bf16 GPU ``x @ w [+ b]`` (w 2-D)."""
    ins = n.input_impls()
    from ...types import DType

    return (len(ins) in (2, 3) and all(x.sharding is None and not x.batch_dims and x.device.label == "gpu" for x in ins)
            and all(x.dtype is DType.bfloat16 for x in ins[:2]) and len(ins[1]._shape) == 2 and len(ins[0]._shape) >= 2)


def _scalar_factor(mul: OpNode, x: TensorImpl) -> TensorImpl | None:
    """The one-element GPU tensor that ``mul`` multiplies the bf16 tensor ``x`` with, if that is what it does."""
    from ...types import DType

    ins = mul.input_impls()
    if len(ins) != 2 or x.dtype is not DType.bfloat16:
        return None
    other = ins[1] if ins[0] is x else ins[0] if ins[1] is x else None
    outs = mul.outputs()
    o = outs[0] if len(outs) == 1 else None
    if other is None or other is x or o is None or other.sharding is not None or other.batch_dims or x.sharding is not None \
            or x.batch_dims or other.device != x.device or other.dtype is not x.dtype or tuple(o._shape) != tuple(x._shape) \
            or any(int(d) != 1 for d in other._shape) or all(int(d) == 1 for d in x._shape):
        return None
    return other


_LN_BWD_NAME = "layer_norm_bwd"


def _is_plain_ln_bwd(n: OpNode) -> bool:
    ins = n.input_impls()
    return (len(ins) in (4, 5) and all(x.sharding is None and not x.batch_dims and x.device.label == "gpu" for x in ins)
            and ins[0].dtype is ins[1].dtype)


def _same_layout_addend(add: OpNode, x: TensorImpl) -> bool:
    ins = add.input_impls()
    if len(ins) != 2:
        return False
    other = ins[1] if ins[0] is x else ins[0] if ins[1] is x else None
    if other is None or other is x or other.batch_dims or other.dtype is not x.dtype or other.device != x.device \
            or tuple(other._shape) != tuple(x._shape):
        return False
    sa = [tuple(d.axes) for d in other.sharding.dim_specs] if other.sharding is not None else None
    sb = [tuple(d.axes) for d in x.sharding.dim_specs] if x.sharding is not None else None
    if sa != sb:
        return False
    return not (other.sharding is not None and other.sharding.partial_sum_axes)


def _dact_consumer(mm: OpNode, nodes, cons, target_ids, used) -> int | None:
    """Index of the ``dact_mul`` node that is the only reader of ``mm``'s product, if any."""
    outs = mm.outputs()
    o = outs[0] if len(outs) == 1 else None
    if o is None or id(o) in target_ids or o.batch_dims or len(cons.get(id(o), [])) != 1:
        return None
    if mm.kwargs.get("activation") is not None or len(mm.input_impls()) != 2:
        return None
    k = cons[id(o)][0]
    d = nodes[k]
    if used[k] or d.op.name != "dact_mul" or d.kwargs.get("activation") not in ("relu", "gelu", "gelu_tanh"):
        return None
    ins = d.input_impls()
    if len(ins) != 2 or ins[0] is not o or ins[1] is o or tuple(ins[1]._shape) != tuple(o._shape):
        return None
    return k


def _is_partial_gemm(n: OpNode) -> bool:
    """bf16 ``x @ w`` on a one-process-per-GPU mesh whose product is a pending partial sum."""
    ins = n.input_impls()
    if len(ins) != 2 or n.kwargs.get("activation") is not None:
        return False
    a, b = ins
    outs = n.outputs()
    o = outs[0] if len(outs) == 1 else None
    if o is None or o.sharding is None or not o.sharding.partial_sum_axes or not o.sharding.mesh.is_distributed:
        return False
    from ...types import DType

    if not (a.device.label == "gpu" and a.dtype is DType.bfloat16 and b.dtype is DType.bfloat16
            and len(b._shape) == 2 and len(a._shape) >= 2 and a.batch_dims == 0 and b.batch_dims == 0):
        return False
    from ...parallel import symm

    return symm.is_ready()


def _is_sum_over_partials(m: OpNode, mm_out: TensorImpl) -> bool:
    axes = set(m.kwargs.get("reduce_axes", ()))
    if m.kwargs.get("reduce_op", "sum") != "sum" or not axes:
        return False
    sp = mm_out.sharding
    if _group_size(sp.mesh, axes) <= 1:
        return False           # a group of one rank: the all-reduce is the identity, keep the plain GEMM
    # a plain sum of the partial products: no dim of the operand is split over the reduced axes
    return axes <= set(sp.partial_sum_axes) and not any(set(d.axes) & axes for d in sp.dim_specs)


def _group_size(mesh, axes) -> int:
    n = 1
    for a in axes:
        n *= mesh.get_axis_size(a)
    return n


def _is_scatter_of_partials(m: OpNode, mm_out: TensorImpl) -> bool:
    axes = set(m.kwargs.get("scatter_axes", ()))
    dim = m.kwargs.get("dim")
    sp = mm_out.sharding
    if not axes or dim is None or dim >= len(mm_out._shape) - 1 or _group_size(sp.mesh, axes) <= 1:
        return False
    return axes <= set(sp.partial_sum_axes) and not any(set(d.axes) & axes for d in sp.dim_specs)


def _rs_addend(add: OpNode, x: TensorImpl) -> str | None:
    """What ``add`` adds to the reduce-scatter result ``x``: 'bias' (one row, no split dims),
    'residual' (same shape and layout) or None."""
    ins = add.input_impls()
    if len(ins) != 2:
        return None
    other = ins[1] if ins[0] is x else ins[0] if ins[1] is x else None
    if other is None or other.batch_dims or other.dtype is not x.dtype:
        return None
    split = [tuple(d.axes) for d in other.sharding.dim_specs] if other.sharding is not None else []
    if len(other._shape) >= 1 and other._shape[-1] == x._shape[-1] and all(d == 1 for d in other._shape[:-1]) \
            and not any(split):
        return "bias"
    if tuple(other._shape) == tuple(x._shape) and other.sharding is not None and x.sharding is not None and \
            split == [tuple(d.axes) for d in x.sharding.dim_specs] and not other.sharding.partial_sum_axes:
        return "residual"
    return None


def _is_row_gather(n: OpNode) -> bool:
    ins = n.input_impls()
    if len(ins) != 1:
        return False
    x = ins[0]
    dim = n.kwargs.get("dim")
    if x.sharding is None or not x.sharding.mesh.is_distributed or dim is None or dim >= len(x._shape) - 1:
        return False
    if not x.sharding.dim_specs[dim].axes or x.sharding.partial_sum_axes or x.batch_dims:
        return False
    if _group_size(x.sharding.mesh, x.sharding.dim_specs[dim].axes) <= 1:
        return False
    from ...types import DType

    if not (x.device.label == "gpu" and x.dtype is DType.bfloat16):
        return False
    from ...parallel import symm

    return symm.is_ready()


def _is_gathered_gemm(m: OpNode, gathered: TensorImpl) -> bool:
    ins = m.input_impls()
    if len(ins) < 2 or ins[0] is not gathered or any(x is gathered for x in ins[1:]):
        return False
    w = ins[1]
    from ...types import DType

    if not (w.dtype is DType.bfloat16 and len(w._shape) == 2 and w.batch_dims == 0):
        return False
    act = m.kwargs.get("activation")
    return act in (None, "relu", "gelu", "gelu_tanh")


def _is_bias_add(m: OpNode, mm_out: TensorImpl) -> bool:
    ins = m.input_impls()
    if len(ins) != 2:
        return False
    other = ins[1] if ins[0] is mm_out else ins[0] if ins[1] is mm_out else None
    if other is None or other.sharding is not None or other.batch_dims:
        return False
    n = mm_out._shape[-1]
    shp = other._shape
    return len(shp) >= 1 and shp[-1] == n and all(d == 1 for d in shp[:-1]) and other.dtype is mm_out.dtype


def run_fused(kind: str, group: list[OpNode], keep_graph: bool = False, arena_blocks: dict | None = None) -> None:
    """``arena_blocks`` (compiled replays only): {id(impl): (arena, offset)} of gathered tensors
    that live in a symmetric arena; the replay frees them after their last use."""
    from .engine import store_outputs

    if kind == "linear_epilogue":
        from ... import native
        from ...native.gemm import gemm_bf16

        mm, add = group[0], group[1]
        act = group[2] if len(group) > 2 else None
        a, b = [x._buffers[0] for x in mm.input_impls()]
        if not native.use_native(a):
            for n_ in group:
                _plain(n_, keep_graph)
            return
        mm_out = mm.outputs()[0]
        bias_impl = [x for x in add.input_impls() if x is not mm_out][0]
        bias = bias_impl._buffers[0]
        epi = "bias" if act is None else act.op.name
        tanh = act is not None and act.op.name == "gelu" and act.kwargs.get("approximate", "none") == "tanh"
        a2 = a.reshape(-1, a.shape[-1])
        out = gemm_bf16(a2, b, bias=bias, epilogue=epi, gelu_tanh=tanh).reshape(*a.shape[:-1], b.shape[-1])
        last = group[-1]
        if keep_graph:
            o = last.outputs()[0]
            if o is not None:
                o._buffers = [out]
        else:
            store_outputs(last, [[out]])
        return
    if kind == "adamw_group":
        from ... import native

        leaves = [[x._buffers[0] for x in n_.input_impls()] for n_ in group]
        kw = group[0].kwargs
        outs = None
        if all(native.use_native(b[0]) for b in leaves):
            from ...native import kernels

            flags = [bool(n_.kwargs.get("inplace")) and all(t.is_contiguous() for t in (b[0], b[2], b[3])) for n_, b in zip(group, leaves)]
            corrected = kw.get("bias_correction", True)
            outs = kernels.adamw_group([(b[0], b[1], b[2], b[3], f) for b, f in zip(leaves, flags)], lr=kw["lr"], b1=kw["beta1"],
                                       b2=kw["beta2"], eps=kw["eps"], wd=kw["weight_decay"],
                                       step=kw.get("step_value") if corrected else None,
                                       hyper=leaves[0][4].contiguous() if len(leaves[0]) > 4 and corrected else None)
        for n_, o in zip(group, outs if outs is not None else group):
            if outs is not None:
                _store(n_, [[t] for t in o], keep_graph)
            else:
                _plain(n_, keep_graph)
        return
    if kind == "linear_act":
        from ... import native
        from ...native.gemm import gemm_bf16

        (lin,) = group
        ins = [x._buffers[0] for x in lin.input_impls()]
        x, w = ins[:2]
        act = lin.kwargs["activation"]
        if not native.use_native(x) or not x.numel():
            return _plain(lin, keep_graph)
        bias = ins[2] if len(ins) > 2 else torch.zeros(w.shape[-1], dtype=w.dtype, device=w.device)
        out = gemm_bf16(x.reshape(-1, x.shape[-1]), w, bias=bias, epilogue="relu" if act == "relu" else "gelu", gelu_tanh=act == "gelu_tanh")
        _store(lin, [[out.reshape(*x.shape[:-1], w.shape[-1])], None], keep_graph)
        return
    if kind == "bias_grads":
        from ... import native
        from ...native import kernels

        xs = [n_.input_impls()[0]._buffers[0] for n_ in group]
        if all(native.use_native(x) for x in xs):
            for n_, o in zip(group, kernels.colsum_group(xs)):
                _store(n_, [[o]], keep_graph)
        else:
            for n_ in group:
                _plain(n_, keep_graph)
        return
    if kind == "conv_relu":
        from ...ops.convolution import _conv_fwd, _own_kernels

        conv, relu = group
        ins = [t._buffers[0] for t in conv.input_impls()]
        if _own_kernels(ins[0]):
            out = _conv_fwd(ins[0], ins[1], ins[2] if len(ins) > 2 else None, conv.kwargs["stride"], conv.kwargs["padding"], relu=True)
            _store(conv, [[out]], keep_graph)           # for the relu's derivative, which is all that reads it
            _store(relu, [[out]], keep_graph)
        else:
            _plain(conv, keep_graph)
            _plain(relu, keep_graph)
        return
    if kind == "pool_bwd_relu":
        from ...native import kernels
        from ...ops.convolution import _fold
        from ...ops.pooling import _native_ok

        pool, dact = group
        x, dy = [t._buffers[0] for t in pool.input_impls()]
        (kh, kw), (sh, sw), (pt, pb, pl, pr) = pool.kwargs["kernel_size"], pool.kwargs["stride"], pool.kwargs["padding"]
        x4, dy4 = _fold(x)[0], _fold(dy)[0]
        if _native_ok(x4) and pt == pb and pl == pr and dy4.dtype == x4.dtype:
            _store(dact, [[kernels.pool2d_bwd(x4, dy4, kh, kw, sh, sw, pt, pl, "max", relu=True).reshape(x.shape)]], keep_graph)
        else:
            _plain(pool, keep_graph)
            _plain(dact, keep_graph)
        return
    if kind == "mean_diff":
        from ... import native
        from ...native import kernels

        sub, last = group[0], group[-1]
        a, b = [x._buffers[0] for x in sub.input_impls()]
        square = group[1].op.name == "mul"
        if native.use_native(a) and native.use_native(b) and a.device == b.device and kernels.elementwise_enabled():
            count = last.kwargs["count"] if last.op.name == "divide_by_count" else last.input_impls()[1]._buffers[0]
            d, out = kernels.mean_diff(a, b, square, count)
            _store(sub, [[d]], keep_graph)
            _store(last, [[out]], keep_graph)
        else:
            for n_ in group:
                _plain(n_, keep_graph)
        return
    if kind == "twice_product":
        from ... import native
        from ...native import kernels

        x, y = [t._buffers[0] for t in group[0].input_impls()]
        out = kernels.binary(x, y, "mul2") if native.use_native(x) else None
        if out is not None:
            _store(group[-1], [[out]], keep_graph)
        else:
            for n_ in group:
                _plain(n_, keep_graph)
        return
    if kind == "next_step":
        from ... import native
        from ...native import kernels

        add, hyper = group
        x, y = [t._buffers[0] for t in add.input_impls()]
        if native.use_native(x) and native.use_native(y) and x.device == y.device:
            step, out = kernels.adam_hyper(x, hyper.kwargs["lr"], hyper.kwargs["beta1"], hyper.kwargs["beta2"], plus=y)
            _store(add, [[step]], keep_graph)
            _store(hyper, [[out]], keep_graph)
        else:
            _plain(add, keep_graph)
            _plain(hyper, keep_graph)
        return
    if kind == "gather_add":
        from ... import native

        ga, add = group
        table, idx = [x._buffers[0] for x in ga.input_impls()]
        rows = ga.outputs()[0]
        other = [x for x in add.input_impls() if x is not rows][0]._buffers[0]
        out = None
        if native.use_native(table) and idx.numel() and table.numel():
            from ...native import kernels

            out = kernels.embedding_gather(table, idx, other)
        if out is not None:
            _store(add, [[out]], keep_graph)
        else:
            _plain(ga, keep_graph)
            _plain(add, keep_graph)
        return
    if kind == "scatter_zeros":
        from ... import native

        z, sc = group
        _, idx, upd = [x._buffers[0] if x._buffers else None for x in sc.input_impls()]
        shape, dt = tuple(sc.input_impls()[0]._shape), sc.input_impls()[0].dtype.to_torch()
        if native.use_native(upd) and upd.dim() and upd.shape[-1] == shape[1] and all(shape):
            from ...native import kernels

            _store(sc, [[kernels.embedding_scatter_add(None, idx, upd, shape[0], dt)]], keep_graph)
        else:
            _plain(z, keep_graph)
            _plain(sc, keep_graph)
        return
    if kind == "sum_axes":
        from ...native import kernels

        x = group[0].input_impls()[0]._buffers[0]
        lo = hi = group[0].kwargs["axis"]
        for n_ in group[1:]:
            if n_.kwargs["axis"] == lo:
                hi += 1
            else:
                lo -= 1
        out = kernels.reduce(x.contiguous().reshape(*x.shape[:lo], -1, *x.shape[hi + 1:]), lo, "sum") if x.numel() else None
        if out is not None:
            _store(group[-1], [[out]], keep_graph)
        else:
            for n_ in group:
                _plain(n_, keep_graph)
        return
    if kind in ("gemm_scale", "scale_gemm"):
        from ... import native
        from ...native.gemm import gemm_bf16

        mm, mul = group if kind == "gemm_scale" else (group[1], group[0])
        if kind == "gemm_scale":
            a, b = [x._buffers[0] for x in mm.input_impls()]
            factor = _scalar_factor(mul, mm.outputs()[0])
        else:
            factor = [f for f in (_scalar_factor(mul, x) for x in mul.input_impls()) if f is not None][0]
            scaled = [x for x in mul.input_impls() if x is not factor][0]
            product = mul.outputs()[0]
            a, b = [(scaled if x is product else x)._buffers[0] for x in mm.input_impls()]
        if native.use_native(a) and a.numel() and b.numel():
            out = gemm_bf16(a.reshape(-1, a.shape[-1]), b, alpha=factor._buffers[0]).reshape(*a.shape[:-1], b.shape[-1])
            _store(group[-1], [[out]], keep_graph)
        elif kind == "gemm_scale":
            _plain(mm, keep_graph)
            _plain(mul, keep_graph)
        else:
            _plain(mul, keep_graph)
            _plain(mm, keep_graph)
        return
    if kind == "ln_bwd_add":
        from ... import native
        from ...native import kernels

        ln, add = group
        dx_out = ln.outputs()[0]
        other = [x for x in add.input_impls() if x is not dx_out][0]._buffers[0]
        ins = [x._buffers[0] for x in ln.input_impls()]
        dy, x = ins[0], ins[1]
        if native.use_native(x) and x.numel() and x.dtype in (torch.bfloat16, torch.float32) and dy.dtype == x.dtype \
                and kernels.supports_rows(x, 2048):
            dx, dg, db = kernels.layernorm_bwd(dy, x, ins[4] if len(ins) > 4 else None, ins[2].reshape(-1), ins[3].reshape(-1), add=other)
            _store(ln, [None, [dg], [db]], keep_graph)
            _store(add, [[dx]], keep_graph)
        else:
            _plain(ln, keep_graph)
            _plain(add, keep_graph)
        return
    if kind in _DUAL:
        from ... import native
        from ...native import kernels
        from ...native.gemm import dual_takes, gemm_dual

        small, big, add = group[0], group[-2], group[-1]
        a2, b2 = [x._buffers[0] for x in small.input_impls()]
        ins = [x._buffers[0] for x in big.input_impls()]
        a, b = ins[:2]
        k, k2, n_out = a.shape[-1], a2.shape[-1], b.shape[-1]
        m = a.numel() // max(k, 1)
        # the thin operand takes a factor that does not round it; any other is applied to the fp32 product, in launches of their own
        factor = _scalar_factor(group[1], small.outputs()[0]) if len(group) == 4 else None
        if native.use_native(a) and a.numel() and b.numel() and dual_takes(m, n_out, k, k2) and (factor is None or _is_power_of_two(factor.literal)):
            a2 = a2.reshape(-1, k2)
            if factor is not None:
                if factor.literal != 1:
                    s = factor._buffers[0].reshape(())
                    scaled = kernels.binary(a2, s, "mul")
                    a2 = scaled if scaled is not None else a2 * s
            out = gemm_dual(a.reshape(-1, k), b, a2, b2, ins[2] if len(ins) > 2 else None)
            _store(add, [[out.reshape(*a.shape[:-1], n_out)]], keep_graph)
        else:
            if len(group) == 4:
                run_fused("gemm_scale", list(group[:2]), keep_graph)
            else:
                _plain(small, keep_graph)
            run_fused("gemm_residual", [big, add], keep_graph)
        return
    if kind == "gemm_residual":
        from ... import native
        from ...native.gemm import cluster_slices, gemm_bf16, residual_in_epilogue, split_k_factor

        lin, add = group
        ins = lin.input_impls()
        a, b = ins[0]._buffers[0], ins[1]._buffers[0]
        bias = ins[2]._buffers[0] if len(ins) > 2 else None
        lin_out = lin.outputs()[0]
        res = [x for x in add.input_impls() if x is not lin_out][0]._buffers[0]
        fits = native.use_native(a) and a.numel() > 0 and b.numel() > 0
        if fits:
            m, k, n_out = a.numel() // a.shape[-1], a.shape[-1], b.shape[-1]
            # (a product that is worth cutting into K slices in memory keeps its own launch: the slices are summed by another)
            fits = (bias is not None or split_k_factor(m, n_out, k) == 1) and (n_out % 8 == 0 or cluster_slices(m, n_out, k) > 1)
        if fits:
            res = res.reshape(-1, n_out)             # a copy where the rows are not in order: not before it is known to be of use
            fits = residual_in_epilogue(m, n_out, k, res)
        if fits:
            out = gemm_bf16(a.reshape(-1, k), b, bias=bias, aux="add", aux_in=res).reshape(*a.shape[:-1], n_out)
            _store(add, [[out]], keep_graph)
        else:
            _plain(lin, keep_graph)
            _plain(add, keep_graph)
        return
    if kind == "gemm_dact":
        from ... import native
        from ...native.gemm import gemm_bf16

        mm, da = group
        a, b = [x._buffers[0] for x in mm.input_impls()]
        z = da.input_impls()[1]._buffers[0]
        act = da.kwargs["activation"]
        if native.use_native(a) and a.numel() and b.numel():
            n_out = b.shape[-1]
            out = gemm_bf16(a.reshape(-1, a.shape[-1]), b, aux="drelu" if act == "relu" else "dgelu",
                            aux_in=z.reshape(-1, n_out), gelu_tanh=act == "gelu_tanh").reshape(*a.shape[:-1], n_out)
            _store(da, [[out]], keep_graph)
        else:
            _plain(mm, keep_graph)
            _plain(da, keep_graph)
        return
    if kind == "all_reduce_bucket":
        # many small partial sums over the same device group: one flat all-reduce
        from ...parallel import backend

        first = group[0]
        mesh = first.input_impls()[0].sharding.mesh
        axes = [x for x in mesh.axis_names if x in first.kwargs["reduce_axes"]]
        xs = [n_.input_impls()[0]._buffers[0] for n_ in group]
        flat = torch.cat([x.reshape(-1) for x in xs])
        red = backend.all_reduce(flat, mesh, axes, "sum")
        off = 0
        for n_, x in zip(group, xs):
            k = x.numel()
            _store(n_, [[red[off: off + k].view(x.shape)]], keep_graph)
            off += k
        backend.stats["bucketed_all_reduce"] = backend.stats.get("bucketed_all_reduce", 0) + len(group)
        return
    if kind == "gemm_to_arena":
        # weight gradient of a data-parallel replica group: keep it unreduced, in the arena; the
        # matching adamw_reduce step sums it over the group while it reads it
        from ...native.gemm import gemm_bf16
        from ...parallel import symm

        mm, ar = group
        a, b = [x._buffers[0] for x in mm.input_impls()]
        ar_out = ar.outputs()[0]
        mesh = ar.input_impls()[0].sharding.mesh
        axes = [x for x in mesh.axis_names if x in ar.kwargs["reduce_axes"]]
        arena = symm.arena(mesh, axes) if arena_blocks is not None else None
        m_rows = a.numel() // max(a.shape[-1], 1)
        nbytes = m_rows * b.shape[-1] * 2
        off = arena.alloc(nbytes) if (arena is not None and ar_out is not None and a.dim() == 2
                                      and os.environ.get("NABLA_B200_FUSE_DP_ADAMW", "0") == "1") else None
        if off is None:
            return run_fused("gemm_all_reduce", group, keep_graph, arena_blocks)
        out = arena.buf[off: off + nbytes].view(torch.bfloat16).view(m_rows, b.shape[-1])
        gemm_bf16(a, b, out=out)
        arena_blocks[id(ar_out)] = (arena, off)
        _store(ar, [[out]], keep_graph)
        return
    if kind == "adamw_reduce":
        from ...parallel import backend, symm

        (ad,) = group
        ins = ad.input_impls()
        blk = arena_blocks.get(id(ins[1])) if arena_blocks is not None else None
        if blk is None:
            return _plain(ad, keep_graph)
        kw = ad.kwargs
        p_, m_, v_ = ins[0]._buffers[0], ins[2]._buffers[0], ins[3]._buffers[0]
        hyper = ins[4]._buffers[0].contiguous() if (len(ins) > 4 and kw.get("bias_correction", True)) else None
        mesh, axes = arena_blocks[("dp_group", id(ad))]
        symm.adamw_reduce(p_, m_, v_, blk[1], mesh, axes, lr=kw["lr"], b1=kw["beta1"], b2=kw["beta2"], eps=kw["eps"],
                          wd=kw["weight_decay"], step=kw.get("step_value") if kw.get("bias_correction", True) else None,
                          hyper=hyper)
        backend.stats["fused_dp_adamw"] = backend.stats.get("fused_dp_adamw", 0) + 1
        _store(ad, [[p_], [m_], [v_]], keep_graph)
        return
    if kind == "gemm_all_reduce":
        from ...parallel import backend, symm

        mm, ar = group
        a, b = [x._buffers[0] for x in mm.input_impls()]
        mesh = mm.outputs()[0].sharding.mesh if mm.outputs()[0] is not None else ar.input_impls()[0].sharding.mesh
        axes = [x for x in mesh.axis_names if x in ar.kwargs["reduce_axes"]]
        split = 1
        if a.is_cuda and a.dim() == 2 and a.dtype == torch.bfloat16:
            from ...native.gemm import gemm_bf16, split_k_factor

            split = split_k_factor(a.shape[0], b.shape[-1], a.shape[1])
        if split > 1:
            # few output tiles and a very long K (weight gradients of a tensor-parallel shard): the
            # fused kernel's fixed 128 x 256 tiles would leave most SMs idle, so the product runs
            # as K slices on all SMs and the small result is all-reduced on its own
            out = backend.all_reduce(gemm_bf16(a, b), mesh, axes, "sum")
            backend.stats["split_k_gemm_all_reduce"] = backend.stats.get("split_k_gemm_all_reduce", 0) + 1
        elif symm.gemm_all_reduce_supported(a, b):
            out = symm.gemm_all_reduce(a, b, mesh, axes).clone().reshape(*a.shape[:-1], b.shape[-1])
            backend.stats["fused_gemm_all_reduce"] = backend.stats.get("fused_gemm_all_reduce", 0) + 1
        else:
            y = mm.op.kernel(a, b)
            out = backend.all_reduce(y, mesh, axes, "sum")
        if keep_graph:
            o = ar.outputs()[0]
            if o is not None:
                o._buffers = [out]
        else:
            store_outputs(ar, [[out]])
        return
    if kind == "gemm_reduce_scatter":
        from ...parallel import backend, symm

        mm, rs = group[0], group[1]
        a, b = [x._buffers[0] for x in mm.input_impls()]
        bias = resid = None
        cur = rs.outputs()[0]
        for add in group[2:]:
            other = [x for x in add.input_impls() if x is not cur][0]
            if _rs_addend(add, cur) == "bias":
                bias = other._buffers[0]
            else:
                resid = other._buffers[0]
            cur = add.outputs()[0]
        mesh = rs.input_impls()[0].sharding.mesh
        axes = [x for x in mesh.axis_names if x in rs.kwargs["scatter_axes"]]
        dim = rs.kwargs["dim"]
        world = 1
        for x in axes:
            world *= mesh.get_axis_size(x)
        lead = tuple(a.shape[:-1])
        inner = 1
        for d in lead[dim + 1:]:
            inner *= d
        m_total = 1
        for d in lead:
            m_total *= d
        cs = (lead[dim] // world) * inner if lead[dim] % world == 0 else 0
        if (symm.gemm_all_reduce_supported(a, b) and symm.chunked_supported(m_total, cs, world)
                and os.environ.get("NABLA_B200_FUSE_RS", "1") != "0"):
            y = symm.gemm_reduce_scatter(a, b, mesh, axes, cs, bias=bias, residual=resid)
            out = y.reshape(*lead[:dim], lead[dim] // world, *lead[dim + 1:], b.shape[-1])
            backend.stats["fused_gemm_reduce_scatter"] = backend.stats.get("fused_gemm_reduce_scatter", 0) + 1
            _store(group[-1], [[out]], keep_graph)
        else:
            for n_ in group:
                _plain(n_, keep_graph)
        return
    if kind == "all_gather_gemm":
        from ...parallel import backend, symm

        ag, mm = group[0], group[1]
        da = group[2] if len(group) > 2 else None
        x_impl = ag.input_impls()[0]
        x = x_impl._buffers[0]
        dim = ag.kwargs["dim"]
        mesh = x_impl.sharding.mesh
        axes = list(x_impl.sharding.dim_specs[dim].axes)
        world = 1
        for a_ in axes:
            world *= mesh.get_axis_size(a_)
        ins = mm.input_impls()
        w = ins[1]._buffers[0]
        bias = ins[2]._buffers[0] if len(ins) > 2 else None
        act = mm.kwargs.get("activation")
        lead = tuple(x.shape[:-1])
        cs = 1
        for d in lead[dim:]:
            cs *= d
        m_total = world * x.numel() // max(x.shape[-1], 1)
        k, n = x.shape[-1], w.shape[-1]
        even = all(s == x.shape[dim] for s in
                   [_local_extent(x_impl, dim, r) for r in mesh.group_of(mesh.rank, axes)])
        if (even and symm.chunked_supported(m_total, cs, world) and n % 8 == 0 and k % 8 == 0 and w.dim() == 2
                and m_total // world * k * 2 + 4096 <= symm.DEFAULT_BYTES - 65536
                and os.environ.get("NABLA_B200_FUSE_AG", "1") != "0"):
            epi = "none" if act is None else ("relu" if act == "relu" else "gelu")
            off = None
            ag_out = ag.outputs()[0]
            if arena_blocks is not None and ag_out is not None and os.environ.get("NABLA_B200_AG_PUSH", "1") != "0":
                ar = symm.arena(mesh, axes)
                if ar is not None:
                    off = ar.alloc(m_total * k * 2)
                    if off is not None:
                        arena_blocks[id(ag_out)] = (ar, off)
            dact = None
            if da is not None:
                dact = (da.input_impls()[1]._buffers[0], da.kwargs["activation"])
            res = symm.all_gather_gemm(x, w, mesh, axes, cs, bias=bias, epilogue=epi, gelu_tanh=act == "gelu_tanh",
                                       store_preact=act is not None, arena_off=off, dact=dact)
            full_shape = (*lead[:dim], lead[dim] * world, *lead[dim + 1:])
            _store(ag, [[res[0].reshape(*full_shape, k)]], keep_graph)
            outs = [[res[1].reshape(*full_shape, n)]]
            if act is not None:
                outs.append([res[2].reshape(*full_shape, n)])
            _store(da if da is not None else mm, outs, keep_graph)
            backend.stats["fused_all_gather_gemm"] = backend.stats.get("fused_all_gather_gemm", 0) + 1
        else:
            for n_ in group:
                _plain(n_, keep_graph)
        return
    raise ValueError(f"unknown fused step {kind}")


def _local_extent(impl: TensorImpl, dim: int, device_id: int) -> int:
    from ..sharding.spec import compute_local_shape

    return compute_local_shape(impl._shape, impl.sharding, device_id)[dim]


def _store(node: OpNode, outs, keep_graph: bool) -> None:
    from .engine import store_outputs

    if keep_graph:
        for i, ref in enumerate(node.out_refs):
            o = ref()
            if o is not None:
                o._buffers = outs[i]
    else:
        store_outputs(node, outs)


def _plain(node: OpNode, keep_graph: bool) -> None:
    _store(node, node.op.execute(node), keep_graph)
