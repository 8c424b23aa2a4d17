"""Python wrappers of the memory-bound fused kernels (``csrc/fused_kernels.cu``).

Inputs and outputs are torch CUDA tensors (bf16 or fp32, contiguous); scratch buffers come
from torch's caching allocator. ``launch_count`` counts kernel launches issued from here.
"""
from __future__ import annotations

import ctypes
import os

import torch

from . import load, ptr, recorder, stream_ptr

_lib = None
launch_count = 0
c_int, c_ll, c_f, c_vp, c_ull = ctypes.c_int, ctypes.c_longlong, ctypes.c_float, ctypes.c_void_p, ctypes.c_ulonglong


def _L():
    global _lib
    if _lib is None:
        lib = load("libnb_kernels.so")
        sig = {
            "nb_layernorm_fwd": [c_vp] * 6 + [c_int, c_int, c_f, c_int, c_vp],
            "nb_layernorm_bwd_nblocks": [c_int, c_int, c_int],
            "nb_layernorm_bwd": [c_vp] * 10 + [c_int, c_int, c_int, c_vp],
            "nb_colsum_nparts": [c_int] * 3,
            "nb_colsum": [c_vp] * 3 + [c_int] * 4 + [c_vp],
            "nb_colsum_group": [c_vp] * 5 + [c_int] * 3 + [c_vp],
            "nb_softmax": [c_vp, c_vp, c_int, c_int, c_int, c_int, c_vp],
            "nb_lse_pick_fwd": [c_vp] * 4 + [c_int, c_int, c_int, c_vp],
            "nb_lse_pick_bwd": [c_vp] * 6 + [c_int, c_int, c_int, c_vp],
            "nb_adamw": [c_vp] * 7 + [c_ll] + [c_f] * 8 + [c_vp, c_int, c_int, c_vp],
            "nb_adamw_group": [c_vp] * 8 + [c_int] + [c_f] * 8 + [c_vp, c_int, c_int, c_vp],
            "nb_adam_hyper": [c_vp] * 4 + [c_f, ctypes.c_double, ctypes.c_double, c_vp],
            "nb_mean_diff": [c_vp] * 4 + [c_ll, c_int, c_vp, c_f, c_int, c_vp],
            "nb_sgd": [c_vp] * 5 + [c_ll] + [c_f] * 4 + [c_int, c_int, c_vp],
            "nb_embedding_gather": [c_vp] * 4 + [c_int] * 5 + [c_vp],
            "nb_embedding_scatter_add": [c_vp] * 5 + [c_int] * 4 + [c_vp],
            "nb_embedding_scatter_sorted": [c_vp] * 5 + [c_int] * 4 + [c_vp],
            "nb_cast": [c_vp, c_vp, c_ll, c_int, c_int, c_vp],
            "nb_copy_batch": [c_vp, c_vp, c_vp, c_int, c_vp],
            "nb_activation": [c_vp] * 3 + [c_ll, c_int, c_int, c_int, c_vp],
            "nb_rng": [c_vp, c_ll, c_ull, c_ull, c_int, c_f, c_f, c_int, c_vp],
            "nb_dropout": [c_vp] * 3 + [c_ll, c_f, c_ull, c_ull, c_int, c_vp],
            "nb_rng_dev": [c_vp, c_ll, c_vp, c_ull, c_int, c_f, c_f, c_int, c_vp],
            "nb_dropout_dev": [c_vp] * 3 + [c_ll, c_f, c_vp, c_ull, c_int, c_vp],
            "nb_nf4_dequant": [c_vp] * 3 + [c_ll, c_int, c_int, c_vp],
            "nb_nf4_dequant_codes": [c_vp] * 4 + [c_ll, c_int, c_int, c_vp],
            "nb_pool2d_fwd": [c_vp, c_vp] + [c_int] * 14 + [c_vp],
            "nb_pool2d_bwd": [c_vp] * 3 + [c_int] * 15 + [c_vp],
            "nb_pool2d_select": [c_vp] * 3 + [c_int] * 13 + [c_vp],
            "nb_conv2d_direct": [c_vp] * 4 + [c_int] * 15 + [c_vp],
            "nb_conv_flip": [c_vp] * 2 + [c_int] * 5 + [c_vp],
            "nb_conv2d_wgrad_slices": [c_ll, c_int, c_int],
            "nb_conv2d_wgrad_direct": [c_vp] * 4 + [c_int] * 14 + [c_vp],
            "nb_sgemm_slices": [c_int] * 3,
            "nb_sgemm": [c_vp] * 5 + [c_int] * 3 + [c_ll] * 4 + [c_vp],
            "nb_sum_slices": [c_vp, c_vp, c_ll, c_int, c_int, c_vp],
            "nb_binary": [c_vp, c_vp, c_vp, c_ll, c_int, c_int, c_ll, c_int, c_int, c_vp],
            "nb_unary": [c_vp, c_vp, c_ll, c_int, c_int, c_vp],
            "nb_reduce": [c_vp, c_vp, c_vp, c_ll, c_ll, c_ll, c_int, c_int, c_vp],
            "nb_reduce_splits": [c_ll, c_ll, c_ll],
            "nb_cumsum": [c_vp, c_vp, c_ll, c_ll, c_ll, c_int, c_int, c_int, c_vp],
        }
        for name, args in sig.items():
            fn = getattr(lib, name)
            fn.argtypes = args
            fn.restype = c_int
        lib.nb_embedding_scatter_work.argtypes = [c_int] * 4
        lib.nb_embedding_scatter_work.restype = c_ll
        lib.nb_layernorm_bwd_two_kernels.argtypes = [c_int]
        lib.nb_layernorm_bwd_two_kernels.restype = None
        # NABLA_B200_LN_BWD=two_kernels: dx and dgamma / dbeta in separate passes instead of the one-pass
        # kernels, for comparisons (no row width needs them)
        lib.nb_layernorm_bwd_two_kernels(1 if os.environ.get("NABLA_B200_LN_BWD", "fused") == "two_kernels" else 0)
        _lib = lib
    r = recorder()
    return _lib if r is None else r.library(_lib)


def has(name: str) -> bool:
    """True when the native library is present (every kernel family ships in one library)."""
    try:
        _L()
        return True
    except Exception:
        return False


def _dt(t: torch.Tensor) -> int:
    if t.dtype == torch.bfloat16:
        return 1
    if t.dtype == torch.float32:
        return 0
    raise TypeError(f"native kernels take bf16 or fp32, got {t.dtype}")


def _ok(rc: int, what: str) -> None:
    global launch_count
    if rc != 0:
        raise RuntimeError(f"{what} failed with code {rc}")
    launch_count += 1


def supports_rows(x: torch.Tensor, d_limit: int = 4096) -> bool:
    v = 8 if x.dtype == torch.bfloat16 else 4
    return x.dtype in (torch.bfloat16, torch.float32) and x.shape[-1] % v == 0 and x.shape[-1] <= d_limit * (v // 4)


# ---------------------------------------------------------------- layer norm
def layernorm_fwd(x: torch.Tensor, gamma, beta, eps: float):
    D = x.shape[-1]
    x2 = x.contiguous().view(-1, D)
    rows = x2.shape[0]
    y = torch.empty_like(x2)
    mean = torch.empty(rows, dtype=torch.float32, device=x.device)
    rstd = torch.empty(rows, dtype=torch.float32, device=x.device)
    g = gamma.contiguous().to(x.dtype) if gamma is not None else None
    b = beta.contiguous().to(x.dtype) if beta is not None else None
    _ok(_L().nb_layernorm_fwd(ptr(x2), ptr(g), ptr(b), ptr(y), ptr(mean), ptr(rstd), rows, D, float(eps), _dt(x),
                              stream_ptr()), "layernorm_fwd")
    return y.view(x.shape), mean, rstd


def layernorm_bwd(dy: torch.Tensor, x: torch.Tensor, gamma, mean: torch.Tensor, rstd: torch.Tensor, add: torch.Tensor | None = None):
    """(dx, dgamma, dbeta); ``add`` (x's shape and dtype) is added to dx in the same pass."""
    global launch_count
    if add is not None:
        if add.device != x.device:
            raise RuntimeError("layernorm_bwd: expected all tensors to be on the same GPU")
        add = add.contiguous()
        if add.data_ptr() & 15 or os.environ.get("NABLA_B200_LN_BWD") == "two_kernels":
            dx, dgamma, dbeta = layernorm_bwd(dy, x, gamma, mean, rstd)
            return dx + add, dgamma, dbeta
    D = x.shape[-1]
    x2 = x.contiguous().view(-1, D)
    dy2 = dy.contiguous().view(-1, D)
    rows = x2.shape[0]
    dx = torch.empty_like(x2)
    dgamma = torch.empty(D, dtype=x.dtype, device=x.device)
    dbeta = torch.empty(D, dtype=x.dtype, device=x.device)
    nb = _L().nb_layernorm_bwd_nblocks(rows, D, _dt(x))
    partial = torch.empty((nb, 2, D), dtype=torch.float32, device=x.device)
    g = gamma.contiguous().to(x.dtype) if gamma is not None else None
    _ok(_L().nb_layernorm_bwd(ptr(dy2), ptr(x2), ptr(g), ptr(mean), ptr(rstd), ptr(add), ptr(dx), ptr(dgamma), ptr(dbeta),
                              ptr(partial), rows, D, _dt(x), stream_ptr()), "layernorm_bwd")
    launch_count += 2
    return dx.view(x.shape), dgamma, dbeta


def colsum_clusters(rows: int, N: int, dtype: torch.dtype) -> int:
    """Column sums by clusters of blocks, in one launch: 0 no, 1 in tiles of 8 vectors of columns, 2 of 32. One launch instead of slabs
    and their fold pays until the slabs' many more blocks do (us, slabs + fold, 8, 32; bf16 unless said): 512 x 256 4.1, 3.3, 3.5;
    2002 x 512 5.2, 3.5, 5.4; 2002 x 2048 5.7, 4.2, 5.4, fp32 5.7, 6.5, 5.1; 8192 x 512 5.9, 5.1, 10.9; 4096 x 8192 10.8, 13.2,
    9.0, fp32 25.7, 37, 30; 16384 x 8192 44, 55, 52; 65536 x 256 17, 18, 63. Fewer than 16 tiles of 32 vectors leave a third of the chip idle, which
    longer sums do not make up for: in chains 4096 x 3072 12.3, -, 13.6, fp32 4096 x 1536 11.3, -, 12.6, of 3000 rows 10.7, -, 10.8 and 9.5, -, 10.2. Rows that are not whole vectors took a
    cast, a sum and a cast, or in fp32 one sum: 512 x 10 5.4, 3.1, fp32 3.0, 2.9; 512 x 1 fp32 2.2, 2.9; 3000 x 777 24, 9.8, 5.6, fp32 11.6,
    8.9, 4.7. Of whole vectors no value goes through more additions that round than as slabs (counted for every number of rows and slabs); of
    others the sums are as near to 64 bits as the cast's."""
    v = 8 if dtype == torch.bfloat16 else 4
    if rows > 8192:
        return 0
    if N % v:
        if v == 4 and N < 8:
            return 0
        return 1 if N <= 64 else 2 if rows <= 4096 else 0
    if rows >= 4096 and N // v < 32:
        return 0                                     # tall and narrow: slabs of a few rows at a time
    if -(-N // (8 * v)) <= 40:
        return 1
    return 2 if rows <= (4096 if N >= 16 * 32 * v else 2500) and N <= (8192 if v == 8 else 2048) else 0


def colsum_group(xs: list[torch.Tensor], out_dtype: torch.dtype | None = None, wide: bool = False) -> list[torch.Tensor]:
    """``colsum`` of several matrices of one type in one launch (per 32), by clusters of blocks: no scratch, no fold."""
    global launch_count
    n = len(xs)
    xs = [x.contiguous().view(-1, x.shape[-1]) for x in xs]
    outs = [torch.empty(x.shape[1], dtype=out_dtype or x.dtype, device=x.device) for x in xs]
    k = _L().nb_colsum_group((c_vp * n)(*[x.data_ptr() for x in xs]), (c_vp * n)(*[o.data_ptr() for o in outs]),
                             (c_int * n)(*[x.shape[0] for x in xs]), (c_int * n)(*[x.shape[1] for x in xs]),
                             (c_int * n)(*[_dt(o) for o in outs]), n, _dt(xs[0]), int(wide), stream_ptr())
    if k < 0:
        raise RuntimeError(f"colsum_group failed with code {k}")
    launch_count += k
    return outs


def colsum(x: torch.Tensor, out_dtype: torch.dtype | None = None) -> torch.Tensor:
    """Sum over all leading dims: (..., N) -> (N,)."""
    global launch_count
    N = x.shape[-1]
    x2 = x.contiguous().view(-1, N)
    rows = x2.shape[0]
    how = colsum_clusters(rows, N, x.dtype)
    if how:
        return colsum_group([x2], out_dtype, how == 2)[0]
    out = torch.empty(N, dtype=out_dtype or x.dtype, device=x.device)
    np_ = _L().nb_colsum_nparts(rows, N, _dt(x))
    partial = torch.empty((np_, N), dtype=torch.float32, device=x.device)
    _ok(_L().nb_colsum(ptr(x2), ptr(out), ptr(partial), rows, N, _dt(x), _dt(out), stream_ptr()), "colsum")
    launch_count += 1
    return out


# ---------------------------------------------------------------- softmax / cross entropy
def softmax(x: torch.Tensor, log: bool = False) -> torch.Tensor:
    D = x.shape[-1]
    x2 = x.contiguous().view(-1, D)
    y = torch.empty_like(x2)
    _ok(_L().nb_softmax(ptr(x2), ptr(y), x2.shape[0], D, int(log), _dt(x), stream_ptr()), "softmax")
    return y.view(x.shape)


def lse_pick_fwd(logits: torch.Tensor, targets: torch.Tensor):
    """Per row: (logsumexp(logits), logits[target] or 0 when the target is outside [0, D))."""
    D = logits.shape[-1]
    l2 = logits.contiguous().view(-1, D)
    t = targets.contiguous().view(-1).to(torch.int64)
    rows = l2.shape[0]
    lse = torch.empty(rows, dtype=torch.float32, device=logits.device)
    picked = torch.empty(rows, dtype=torch.float32, device=logits.device)
    _ok(_L().nb_lse_pick_fwd(ptr(l2), ptr(t), ptr(lse), ptr(picked), rows, D, _dt(logits), stream_ptr()), "lse_pick_fwd")
    return lse.view(targets.shape), picked.view(targets.shape)


def lse_pick_bwd(logits: torch.Tensor, targets: torch.Tensor, lse: torch.Tensor, g_lse, g_pick) -> torch.Tensor:
    D = logits.shape[-1]
    l2 = logits.contiguous().view(-1, D)
    t = targets.contiguous().view(-1).to(torch.int64)
    d = torch.empty_like(l2)
    gl = g_lse.reshape(-1).float().contiguous() if g_lse is not None else None
    gp = g_pick.reshape(-1).float().contiguous() if g_pick is not None else None
    _ok(_L().nb_lse_pick_bwd(ptr(l2), ptr(t), ptr(lse.reshape(-1).float().contiguous()), ptr(gl), ptr(gp), ptr(d),
                             l2.shape[0], D, _dt(logits), stream_ptr()), "lse_pick_bwd")
    return d.view(logits.shape)


# ---------------------------------------------------------------- optimizers
def adamw(p, g, m, v, *, lr, b1, b2, eps, wd, step: int | None = None, hyper: torch.Tensor | None = None,
          grad_scale: float = 1.0, inplace: bool = False):
    """Returns (p', m', v'). ``hyper`` = device tensor [lr, 1-b1^t, 1-b2^t, grad_scale] overrides
    the scalar arguments (lets a captured CUDA graph advance the step)."""
    p = p.contiguous()
    g = g.contiguous()
    po = p if inplace else torch.empty_like(p)
    mo = m if inplace else torch.empty_like(m)
    vo = v if inplace else torch.empty_like(v)
    bc1 = 1.0 - b1 ** step if step is not None else 1.0
    bc2 = 1.0 - b2 ** step if step is not None else 1.0
    _ok(_L().nb_adamw(ptr(p), ptr(g), ptr(m), ptr(v), ptr(po), ptr(mo), ptr(vo), p.numel(), float(lr), float(b1),
                      float(b2), float(eps), float(wd), float(bc1), float(bc2), float(grad_scale), ptr(hyper), _dt(p),
                      _dt(g), stream_ptr()), "adamw")
    return po, mo, vo


def adamw_group(leaves: list, *, lr, b1, b2, eps, wd, step: int | None = None, hyper: torch.Tensor | None = None):
    """``adamw`` of several small tensors that share their hyperparameters and types, in one launch per 48: ``leaves``
    holds (p, g, m, v, inplace); returns [(p', m', v')], or None (nothing updated) where a tensor is not 16-byte aligned
    or has more than 2^20 elements, which the kernel is not made for."""
    n = len(leaves)
    if any(leaf[0].numel() > 1 << 20 for leaf in leaves):
        return None
    ins, outs = [], []
    for p, g, m, v, inplace in leaves:
        p, g, m, v = p.contiguous(), g.contiguous(), m.contiguous(), v.contiguous()
        ins.append((p, g, m, v))
        outs.append((p, m, v) if inplace else (torch.empty_like(p), torch.empty_like(m), torch.empty_like(v)))
    cols = [(c_vp * n)(*[t[i].data_ptr() for t in ins]) for i in range(4)] + [(c_vp * n)(*[t[i].data_ptr() for t in outs]) for i in range(3)]
    if any((a or 0) & 15 for col in cols for a in col):
        return None
    bc1 = 1.0 - b1 ** step if step is not None else 1.0
    bc2 = 1.0 - b2 ** step if step is not None else 1.0
    sizes = (c_int * n)(*[t[0].numel() for t in ins])
    _ok(_L().nb_adamw_group(*cols, sizes, n, float(lr), float(b1), float(b2), float(eps), float(wd), float(bc1), float(bc2), 1.0,
                            ptr(hyper), _dt(ins[0][0]), _dt(ins[0][1]), stream_ptr()), "adamw_group")
    return outs


def adam_hyper(step: torch.Tensor, lr: float, b1: float, b2: float, plus: torch.Tensor | None = None):
    """[lr, 1 - b1^t, 1 - b2^t, 1] for the fp32 step count ``t`` on the device (one element). With ``plus`` (another such
    element) t is their sum, and (sum, vector) is returned."""
    out = torch.empty(4, dtype=torch.float32, device=step.device)
    total = torch.empty((), dtype=torch.float32, device=step.device) if plus is not None else None
    _ok(_L().nb_adam_hyper(ptr(step), ptr(plus), ptr(total), ptr(out), float(lr), float(b1), float(b2), stream_ptr()), "adam_hyper")
    return out if plus is None else (total, out)


def sgd(p, g, buf, *, lr, momentum=0.0, wd=0.0, grad_scale=1.0):
    p = p.contiguous()
    g = g.contiguous()
    po = torch.empty_like(p)
    bo = torch.empty_like(buf) if buf is not None else None
    _ok(_L().nb_sgd(ptr(p), ptr(g), ptr(buf), ptr(po), ptr(bo), p.numel(), float(lr), float(momentum), float(wd),
                    float(grad_scale), _dt(p), _dt(g), stream_ptr()), "sgd")
    return po, bo


# ---------------------------------------------------------------- embedding
def embedding_gather(table: torch.Tensor, ids: torch.Tensor, add: torch.Tensor | None = None) -> torch.Tensor | None:
    """Rows of ``table`` (vocab, D) by id. ``add``: a tensor over the trailing dims of the result (at least the
    last), added in the same pass; None when that pass does not take it (the caller then gathers and adds)."""
    if ids.device != table.device:
        raise RuntimeError("embedding: expected all tensors to be on the same GPU")
    period = 0
    if add is not None:
        shape = tuple(add.shape)
        while len(shape) > 1 and shape[0] == 1:
            shape = shape[1:]
        full = (*ids.shape, table.shape[1])
        if add.dtype != table.dtype or add.device != table.device or not shape or full[len(full) - len(shape):] != shape or not add.numel() \
                or not elementwise_enabled():
            return None
        add = add.contiguous()
        period = add.numel() // table.shape[1]
    table = table.contiguous()
    if add is not None and (add.data_ptr() | table.data_ptr()) & 15:
        return None
    flat = ids.contiguous().view(-1).to(torch.int64)
    D = table.shape[1]
    out = torch.empty((flat.numel(), D), dtype=table.dtype, device=table.device)
    _ok(_L().nb_embedding_gather(ptr(table), ptr(flat), ptr(add), ptr(out), flat.numel(), D, table.shape[0], period, _dt(table),
                                 stream_ptr()), "embedding_gather")
    return out.view(*ids.shape, D)


def embedding_scatter_add(base: torch.Tensor | None, ids: torch.Tensor, upd: torch.Tensor, vocab: int = 0,
                          dtype: torch.dtype | None = None) -> torch.Tensor:
    """base + scatter_add(ids, upd) with fp32 accumulation (embedding backward). ``base`` None: a table of
    ``vocab`` rows of zeros in ``dtype``, which is neither made nor read."""
    global launch_count
    from .. import config

    if ids.device != upd.device or (base is not None and base.device != upd.device):
        raise RuntimeError("embedding: expected all tensors to be on the same GPU")
    if base is None and config.is_deterministic():
        base = torch.zeros((vocab, upd.shape[-1]), dtype=dtype, device=upd.device)
    if base is not None:
        base = base.contiguous()
        vocab, dtype = base.shape[0], base.dtype
    V, D = vocab, upd.shape[-1]
    flat = ids.contiguous().view(-1).to(torch.int64)
    u = upd.contiguous().view(-1, D).to(dtype)

    if config.is_deterministic():
        # no atomics: stable sort of the ids, then one block per run of equal ids adds the run's rows
        # in their original order
        sorted_ids, perm = torch.sort(flat, stable=True)
        out = base.clone()
        _ok(_L().nb_embedding_scatter_sorted(ptr(sorted_ids), ptr(perm), ptr(u), ptr(base), ptr(out), flat.numel(), D, V,
                                             _dt(base), stream_ptr()), "embedding_scatter_sorted")
        launch_count += 1
        return out
    work = torch.empty(_L().nb_embedding_scatter_work(flat.numel(), D, V, _dt(u)), dtype=torch.int32, device=u.device)
    out = torch.empty((V, D), dtype=dtype, device=u.device)
    _ok(_L().nb_embedding_scatter_add(ptr(work), ptr(flat), ptr(u), ptr(base), ptr(out), flat.numel(), D, V, _dt(u),
                                      stream_ptr()), "embedding_scatter_add")
    launch_count += 1
    return out


def _is_dense(t: torch.Tensor) -> bool:
    """No gaps and no overlaps between the elements, in any order of the dims: one run of bytes."""
    want = 1
    for st, n in sorted((st, n) for st, n in zip(t.stride(), t.shape) if n != 1):
        if st != want:
            return False
        want *= n
    return True


class CopyBatch:
    """Copies between a fixed list of tensors and equally laid out ones that come with each call, all in one
    launch (or one per 128 tensors). ``shared``: callers may hold views of the fixed tensors' memory."""

    def __init__(self, fixed: list[torch.Tensor], shared: bool = False):
        from . import use_native

        n = len(fixed)
        self.dev = dev = torch.cuda.current_device()
        self.fixed = fixed
        self.strides = [t.stride() for t in fixed]
        self.fixed_ptrs = (c_vp * n)(*[t.data_ptr() for t in fixed])
        self.own = [t.data_ptr() for t in fixed]
        self.size = [t.numel() * t.element_size() for t in fixed]
        # what one launch can move: dense tensors of this device (a CPU scalar among the inputs is not one), and none
        # where the native kernels are switched off
        self.plain = [use_native(t) and t.device.index == dev and _is_dense(t) for t in fixed]
        self.storages = {t.untyped_storage().data_ptr() for t in fixed} if shared else None
        self.all_sizes = (c_ull * n)(*self.size) if all(self.plain) else None
        self.launches = -(-sum(1 for s in self.size if s) // 128)          # of a call that copies all of them

    def fresh(self) -> list[torch.Tensor]:
        """New tensors like the fixed ones with their contents: what was just allocated for the purpose needs none of the
        checks of ``run``."""
        global launch_count
        others = [torch.empty_like(t) for t in self.fixed]
        if self.all_sizes is None or not others or torch.cuda.current_device() != self.dev or any(
                o.stride() != s for o, s in zip(others, self.strides)):
            self.run(others, into_fixed=False)
            return others
        n = len(others)
        k = _L().nb_copy_batch((c_vp * n)(*[o.data_ptr() for o in others]), self.fixed_ptrs, self.all_sizes, n, stream_ptr())
        if k < 0:
            raise RuntimeError(f"copy_batch failed with code {k}")
        launch_count += k
        return others

    def run(self, others: list[torch.Tensor], into_fixed: bool) -> None:
        """``fixed <- others`` (``into_fixed``) or ``others <- fixed``. A pair that shares its storage is left
        alone; one whose layouts differ goes through torch's copy. A source that lies in the memory of the fixed
        tensors (a result of the captured step that comes back in another place) is copied aside first, so that
        every pair reads what was there before the call."""
        global launch_count
        own, copies = self.own, False
        n = len(own)
        rest = []                                           # pairs that torch copies
        if self.storages is not None and into_fixed:
            others = [o.clone() if o.data_ptr() != own[i] and o.untyped_storage().data_ptr() in self.storages else o
                      for i, o in enumerate(others)]
        ptrs, nbytes = (c_vp * n)(), (c_ull * n)()          # of this call: another thread may be in here too
        here = torch.cuda.current_device() == self.dev
        for i, (o, f, q, plain, stride, size) in enumerate(zip(others, self.fixed, own, self.plain, self.strides, self.size)):
            p = o.data_ptr()
            if p == q:
                continue
            if here and plain and o.dtype is f.dtype and o.stride() == stride and o.get_device() == self.dev:
                ptrs[i] = p
                nbytes[i] = size
                copies = copies or size > 0
            elif size:
                rest.append(i)
        for i in rest:
            self.fixed[i].copy_(others[i]) if into_fixed else others[i].copy_(self.fixed[i])
        if not copies:
            return
        dst, src = (self.fixed_ptrs, ptrs) if into_fixed else (ptrs, self.fixed_ptrs)
        k = _L().nb_copy_batch(dst, src, nbytes, n, stream_ptr())
        if k < 0:
            raise RuntimeError(f"copy_batch failed with code {k}")
        launch_count += k


def cast(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    x = x.contiguous()
    out = torch.empty(x.shape, dtype=dtype, device=x.device)
    _ok(_L().nb_cast(ptr(x), ptr(out), x.numel(), _dt(x), _dt(out), stream_ptr()), "cast")
    return out


ACT = {"relu": 0, "gelu": 1, "gelu_tanh": 2, "silu": 3}


def activation(z: torch.Tensor, mode: str) -> torch.Tensor:
    z = z.contiguous()
    out = torch.empty_like(z)
    _ok(_L().nb_activation(ptr(z), None, ptr(out), z.numel(), ACT[mode], 0, _dt(z), stream_ptr()), "activation")
    return out


def activation_bwd(z: torch.Tensor, dy: torch.Tensor, mode: str) -> torch.Tensor:
    z = z.contiguous()
    dy = dy.contiguous().to(z.dtype)
    out = torch.empty_like(z)
    _ok(_L().nb_activation(ptr(z), ptr(dy), ptr(out), z.numel(), ACT[mode], 1, _dt(z), stream_ptr()), "activation_bwd")
    return out


# ---------------------------------------------------------------- RNG
_rng_states: dict = {}      # device -> (int64[2] tensor [seed, draws so far], host epoch it was written for)


def rng_state(device) -> torch.Tensor:
    """This device's random-stream position ``[seed, draws so far]`` in device memory. The kernels
    read it when they run and a one-thread kernel advances it after each draw, so a CUDA-graph replay
    continues the stream instead of repeating it. Re-written from the host after every ``seed()``
    call (never during stream capture: run one uncaptured step first, which ``compile`` does)."""
    from ..core.graph.engine import GRAPH

    device = torch.device(device)
    epoch = (GRAPH.seed, getattr(GRAPH, "seed_epoch", 0))
    ent = _rng_states.get(device)
    if ent is None or ent[1] != epoch:
        if torch.cuda.is_current_stream_capturing():
            if ent is None:
                raise RuntimeError("random op inside CUDA-graph capture before the device stream state exists")
            return ent[0]
        t = ent[0] if ent is not None else torch.zeros(2, dtype=torch.int64, device=device)
        t.copy_(torch.tensor([GRAPH.seed & (2 ** 63 - 1), GRAPH.rng_counter], dtype=torch.int64))
        ent = (t, epoch)
        _rng_states[device] = ent
    return ent[0]


def rng_dev(shape, dtype: torch.dtype, device, salt: int, mode: str, a: float, b: float) -> torch.Tensor:
    """Uniform / gaussian tensor from this device's stream (``rng_state``), Philox in one kernel."""
    out = torch.empty(shape, dtype=dtype, device=device)
    st = rng_state(out.device)
    _ok(_L().nb_rng_dev(ptr(out), out.numel(), ptr(st), salt & (2 ** 64 - 1), 0 if mode == "uniform" else 1,
                        float(a), float(b), _dt(out), stream_ptr()), "rng")
    return out


def dropout_dev(x: torch.Tensor, p: float, salt: int):
    """Dropout whose mask comes from this device's stream (``rng_state``): ``(y, keep mask uint8)``."""
    x = x.contiguous()
    y = torch.empty_like(x)
    mask = torch.empty(x.shape, dtype=torch.uint8, device=x.device)
    st = rng_state(x.device)
    _ok(_L().nb_dropout_dev(ptr(x), ptr(y), ptr(mask), x.numel(), float(p), ptr(st), salt & (2 ** 64 - 1), _dt(x),
                            stream_ptr()), "dropout")
    return y, mask


def rng(shape, dtype: torch.dtype, device, seed: int, offset: int, mode: str, a: float, b: float) -> torch.Tensor:
    out = torch.empty(shape, dtype=dtype, device=device)
    _ok(_L().nb_rng(ptr(out), out.numel(), seed & (2 ** 64 - 1), offset & (2 ** 64 - 1), 0 if mode == "uniform" else 1,
                    float(a), float(b), _dt(out), stream_ptr()), "rng")
    return out


def dropout(x: torch.Tensor, p: float, seed: int, offset: int):
    x = x.contiguous()
    y = torch.empty_like(x)
    mask = torch.empty(x.shape, dtype=torch.uint8, device=x.device)
    _ok(_L().nb_dropout(ptr(x), ptr(y), ptr(mask), x.numel(), float(p), seed & (2 ** 64 - 1), offset & (2 ** 64 - 1),
                        _dt(x), stream_ptr()), "dropout")
    return y, mask


def nf4_dequant(packed: torch.Tensor, absmax: torch.Tensor, n: int, block: int, dtype: torch.dtype) -> torch.Tensor:
    out = torch.empty(n, dtype=dtype, device=packed.device)
    _ok(_L().nb_nf4_dequant(ptr(packed.contiguous()), ptr(absmax.contiguous().float()), ptr(out), n, block, _dt(out),
                            stream_ptr()), "nf4_dequant")
    return out


# ---------------------------------------------------------------- pooling / conv (NHWC)
def pool2d_fwd(x, kh, kw, sh, sw, ph, pw, mode: str):
    x = x.contiguous()
    N, H, W, C = x.shape
    OH = (H + 2 * ph - kh) // sh + 1
    OW = (W + 2 * pw - kw) // sw + 1
    y = torch.empty((N, OH, OW, C), dtype=x.dtype, device=x.device)
    _ok(_L().nb_pool2d_fwd(ptr(x), ptr(y), N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, 0 if mode == "avg" else 1,
                           _dt(x), stream_ptr()), "pool2d_fwd")
    return y


def pool2d_bwd(x, dy, kh, kw, sh, sw, ph, pw, mode: str, relu: bool = False):
    """``relu`` (max pooling): x is the output of a relu, whose derivative is applied to the gradient in the same pass."""
    x = x.contiguous()
    dy = dy.contiguous()
    N, H, W, C = x.shape
    _, OH, OW, _ = dy.shape
    dx = torch.empty_like(x)
    _ok(_L().nb_pool2d_bwd(ptr(x), ptr(dy), ptr(dx), N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw,
                           0 if mode == "avg" else 1, int(relu), _dt(x), stream_ptr()), "pool2d_bwd")
    return dx


def pool2d_select(x, t, kh, kw, sh, sw, ph, pw):
    """``out[window] = t[arg-max of x over the window]`` (NHWC; the tangent of max pooling)."""
    x = x.contiguous()
    t = t.contiguous().to(x.dtype)
    N, H, W, C = x.shape
    OH = (H + 2 * ph - kh) // sh + 1
    OW = (W + 2 * pw - kw) // sw + 1
    y = torch.empty((N, OH, OW, C), dtype=x.dtype, device=x.device)
    _ok(_L().nb_pool2d_select(ptr(x), ptr(t), ptr(y), N, H, W, C, OH, OW, kh, kw, sh, sw, ph, pw, _dt(x), stream_ptr()),
        "pool2d_select")
    return y


def conv_flip(w: torch.Tensor) -> torch.Tensor:
    """(R, S, C, F) filter -> (R, S, F, C), turned around in both of the first dims: the filter of the input gradient."""
    R, S, C, F = w.shape
    w = w.contiguous()
    out = torch.empty((R, S, F, C), dtype=w.dtype, device=w.device)
    _ok(_L().nb_conv_flip(ptr(w), ptr(out), R, S, C, F, _dt(w), stream_ptr()), "conv_flip")
    return out


def conv2d_direct(x, w, bias, stride, padding, relu: bool = False):
    """NHWC x RSCF direct convolution; padding = (top, bottom, left, right)."""
    x = x.contiguous()
    w = w.contiguous().to(x.dtype)
    N, H, W, C = x.shape
    R, S, _, F = w.shape
    pt, pb, pl, pr = padding
    OH = (H + pt + pb - R) // stride[0] + 1
    OW = (W + pl + pr - S) // stride[1] + 1
    y = torch.empty((N, OH, OW, F), dtype=x.dtype, device=x.device)
    b = bias.contiguous().to(x.dtype).view(-1) if bias is not None else None
    _ok(_L().nb_conv2d_direct(ptr(x), ptr(w), ptr(b), ptr(y), N, H, W, C, R, S, F, OH, OW, stride[0], stride[1], pt, pl,
                              int(relu), _dt(x), stream_ptr()), "conv2d_direct")
    return y


def conv2d_wgrad_direct(x, dy, w_shape, stride, padding):
    """Filter gradient of the NHWC x RSCF convolution: ``dw[r,s,c,f] = sum x[...] * dy[...]`` over
    the batch and all output pixels (deterministic, no atomics)."""
    global launch_count
    x = x.contiguous()
    dy = dy.contiguous().to(x.dtype)
    N, H, W, C = x.shape
    R, S, _, F = w_shape
    OH, OW = dy.shape[1], dy.shape[2]
    dw = torch.empty((R, S, C, F), dtype=x.dtype, device=x.device)
    slices = _L().nb_conv2d_wgrad_slices(N * OH * OW, R * S * C, F)
    part = torch.empty(slices * dw.numel(), dtype=torch.float32, device=x.device)
    _ok(_L().nb_conv2d_wgrad_direct(ptr(x), ptr(dy), ptr(dw), ptr(part), N, H, W, C, R, S, F, OH, OW, stride[0], stride[1],
                                    padding[0], padding[2], _dt(x), stream_ptr()), "conv2d_wgrad_direct")
    launch_count += 1
    return dw


def nf4_dequant_codes(codes: torch.Tensor, absmax: torch.Tensor, codebook: torch.Tensor, n: int, block: int,
                      dtype: torch.dtype) -> torch.Tensor:
    """``out[i] = codebook[codes[i]] * absmax[i // block]`` for one-code-per-byte NF4 weights, in one
    kernel; ``dtype`` fp32 or bf16."""
    out = torch.empty(n, dtype=dtype, device=codes.device)
    _ok(_L().nb_nf4_dequant_codes(ptr(codes.contiguous()), ptr(absmax.contiguous().float()),
                                  ptr(codebook.contiguous().float()), ptr(out), n, block, _dt(out), stream_ptr()),
        "nf4_dequant_codes")
    return out


def sgemm_pays(M: int, N: int, K: int) -> bool:
    """Where ``sgemm`` beats the library (us, library and this, over 45 sizes and both orders): few results of long sums. 256 x 10
    over 1568 21.7 and 6.9, 128 x 128 over 512 10.5 and 5.6, 256 x 100 over 256 6.8 and 5.7, over 2048 21.9 and 16.5; not 256 x
    256 over 256 (6.6 and 7.9), 1568 x 100 over 256 (7.4 and 14.1), 256 x 1568 over 10 (3.0 and 3.3), 8 x 1024 over 1024 (8.1 and 9.6)."""
    return min(M, N) > 8 and M * N <= 32768 and 256 <= K <= 4096


def sgemm_takes(a: torch.Tensor, b: torch.Tensor, bias: torch.Tensor | None = None) -> bool:
    """``sgemm_pays`` for the operands at hand. Of up to 16 rows the library has kernels of its own, quick (us, library and ``sgemm``) at rows along
    K times columns along K up to K = 512 (16 x 64 over 256 3.4, 5.4, over 512 5.1, 5.4, over 700 6.7, 6.3), at few columns of short sums (9 x 9
    over 256 4.1, 4.5; 12 x 45 6.4, 5.2; the first operand transposed, 16 x 64 over 400 5.7, 6.3) and at many of long ones (16 x 1000 over 512
    6.7, 7.1); a bias is a launch more there, so not with one. Over 70
    sizes of 9 to 32 rows in four orders: 0.85 to 6 times as fast as the library, with a bias 0.88 to 6.4, 7 of 552 below 0.95."""
    (M, K), N = a.shape, b.shape[1]
    if not sgemm_pays(M, N, K):
        return False
    if M > 16 or bias is not None:
        return True
    rows, columns = a.stride(1) == 1, b.stride(0) == 1        # along K
    if columns:
        return K > 512 or N >= 1000 if rows else N * K <= 800_000
    return N * K <= 400_000 and (K >= 512 or N > 64 or (rows and (M > 10 or K >= 320)))


def sgemm(a: torch.Tensor, b: torch.Tensor, bias: torch.Tensor | None = None) -> torch.Tensor | None:
    """``a @ b [+ bias]`` of small 2-D fp32 matrices of any strides on the CUDA cores; None for anything else."""
    if not (a.is_cuda and a.device == b.device and a.dim() == 2 and b.dim() == 2 and a.dtype == b.dtype == torch.float32
            and elementwise_enabled()):
        return None
    M, K, N = a.shape[0], a.shape[1], b.shape[1]
    if b.shape[0] != K or not 0 < M * N * K < 1 << 31 or M > 1 << 20 \
            or (bias is not None and (bias.numel() != N or bias.dtype != torch.float32 or bias.device != a.device)):
        return None
    z = _L().nb_sgemm_slices(M, N, K)
    out = torch.empty((M, N), dtype=torch.float32, device=a.device)
    part = torch.empty((z, M, N), dtype=torch.float32, device=a.device) if z > 1 else None
    bias = bias.reshape(-1).contiguous() if bias is not None else None
    _ok(_L().nb_sgemm(ptr(a), ptr(b), ptr(bias), ptr(out), ptr(part), M, N, K, a.stride(0), a.stride(1), b.stride(0), b.stride(1),
                      stream_ptr()), "sgemm")
    return out


def mean_diff(a: torch.Tensor, b: torch.Tensor, square: bool, count) -> tuple[torch.Tensor, torch.Tensor]:
    """(d, m): d = a - b, and m the sum of d (or of d * d) over all elements, divided by ``count`` (a number, or an element of a's type
    on the device), of two fp32 / bf16 tensors of one shape and type. The sum is kept in fp32 and rounded once."""
    a, b = a.contiguous(), b.contiguous()
    d = torch.empty_like(a)
    out = torch.empty((), dtype=a.dtype, device=a.device)
    on_device = isinstance(count, torch.Tensor)
    _ok(_L().nb_mean_diff(ptr(a), ptr(b), ptr(d), ptr(out), a.numel(), int(square), ptr(count if on_device else None),
                          0.0 if on_device else float(max(int(count), 1)), _dt(a), stream_ptr()), "mean_diff")
    return d, out


def sum_slices(part: torch.Tensor, out_dtype: torch.dtype) -> torch.Tensor:
    """Sum a contiguous fp32 tensor over its leading dim (the partial products of a split-K GEMM)."""
    s_ = part.shape[0]
    out = torch.empty(part.shape[1:], dtype=out_dtype, device=part.device)
    _ok(_L().nb_sum_slices(ptr(part), ptr(out), out.numel(), s_, _dt(out), stream_ptr()), "sum_slices")
    return out


# ---------------------------------------------------------------- pointwise / reduction families
BINARY_OPS = {"add": 0, "sub": 1, "mul": 2, "div": 3, "maximum": 4, "minimum": 5, "pow": 6, "mul2": 7}
UNARY_OPS = {"neg": 0, "abs": 1, "exp": 2, "log": 3, "sqrt": 4, "rsqrt": 5, "tanh": 6, "sigmoid": 7, "sin": 8, "cos": 9,
             "erf": 10, "log1p": 11, "floor": 12, "trunc": 13, "round": 14, "square": 15, "reciprocal": 16}
REDUCE_OPS = {"sum": 0, "max": 1, "min": 2, "mean": 3, "argmax": 4, "argmin": 5}
_FLOATS = (torch.float32, torch.bfloat16)


def elementwise_enabled() -> bool:
    import os

    return os.environ.get("NABLA_B200_ELEMENTWISE", "native") == "native"


def binary(a: torch.Tensor, b: torch.Tensor, op: str):
    """``a (op) b`` in one kernel when both are fp32 / bf16 CUDA tensors of one dtype and ``b`` (or
    ``a``) has the other's shape, is a single element, or is a vector over the trailing dims (bias
    style). Returns None for anything else (mixed dtypes, general broadcasting, integers): the caller
    then uses the framework's generic path."""
    if not (a.is_cuda and b.is_cuda and a.dtype == b.dtype and a.dtype in _FLOATS and elementwise_enabled()):
        return None
    swap = 0
    if a.numel() < b.numel():
        a, b, swap = b, a, 1
    if a.numel() == 0 or tuple(torch.broadcast_shapes(a.shape, b.shape)) != tuple(a.shape):
        return None
    v = 16 // a.element_size()
    if b.numel() == 1:
        mode, inner = 1, 1
    elif tuple(b.shape) == tuple(a.shape):
        mode, inner = 0, 1
    else:
        bs = tuple(b.shape)
        while bs and bs[0] == 1:
            bs = bs[1:]
        if not bs or tuple(a.shape[len(a.shape) - len(bs):]) != bs:
            return None
        mode, inner = 2, b.numel()
        if inner % v:
            return None
    a_c, b_c = a.contiguous(), b.contiguous()
    if (a_c.data_ptr() | b_c.data_ptr()) & 15:
        return None
    out = torch.empty_like(a_c)
    _ok(_L().nb_binary(ptr(a_c), ptr(b_c), ptr(out), a_c.numel(), BINARY_OPS[op], mode, inner, swap, _dt(a_c), stream_ptr()),
        "binary")
    return out


def unary(x: torch.Tensor, op: str):
    """``f(x)`` in one kernel for fp32 / bf16 CUDA tensors; None otherwise."""
    if not (x.is_cuda and x.dtype in _FLOATS and x.numel() and elementwise_enabled()):
        return None
    xc = x.contiguous()
    if xc.data_ptr() & 15:
        return None
    out = torch.empty_like(xc)
    _ok(_L().nb_unary(ptr(xc), ptr(out), xc.numel(), UNARY_OPS[op], _dt(xc), stream_ptr()), "unary")
    return out


def _outer_r_inner(x: torch.Tensor, axis: int):
    outer = 1
    for d in x.shape[:axis]:
        outer *= int(d)
    inner = 1
    for d in x.shape[axis + 1:]:
        inner *= int(d)
    return outer, int(x.shape[axis]), inner


def joined_sum(outer: int, rows: int, inner: int, dtype: torch.dtype) -> bool:
    """Whether one sum over ``rows`` = several neighbouring axes serves better than one sum per axis.

    Column sums of a tall narrow matrix (a convolution's bias gradient) always do: their chains of additions are
    short and they fill the chip (256 x 28 x 28 x 16 fp32 over its leading axes: 45 us as three sums, 13 as one).
    Otherwise fp32 stays with one sum per axis: each has R / 8 rows in a chain, one over all axes has the
    product (64 x 64 x 32768: 1.1e-7 from 64 bits as two sums, 4.1e-7 as one, 198 and 188 us), while bf16 loses a rounding
    of its partial results to 16 bits by joining, and joins where the one kernel has two blocks per SM or the
    tensor is small: 100 x 30 x 8192 81 -> 36 us, but 1000 x 1000 x 256, where 64 slabs of 2 column tiles are 128 blocks,
    243 as two sums and 566 as one, 1.4 M x 8 in two outer parts 56 and 196."""
    v = 8 if dtype == torch.bfloat16 else 4
    column_sums = outer == 1 and rows > 4096 and inner % v == 0 and inner <= 4096 * (v // 4)      # as in reduce()
    if column_sums and inner // v < 32:
        return True
    if dtype != torch.bfloat16:
        return False
    if outer * rows * inner <= 1 << 20 or (rows <= 256 and inner % v == 0 and outer * (inner // v) >= 148 * 256):
        return True
    if column_sums:
        blocks = -(-inner // (32 * v)) * _L().nb_colsum_nparts(rows, inner, 1)
    else:
        blocks = outer * -(-inner // 32) * _L().nb_reduce_splits(outer, rows, inner)
    return blocks >= 2 * 148


def reduce(x: torch.Tensor, axis: int, op: str, keepdims: bool = False):
    """sum / max / min / mean / argmax / argmin over one axis in one kernel (fp32 / bf16 CUDA, non-empty
    axis); None otherwise."""
    if not (x.is_cuda and x.dtype in _FLOATS and x.numel() and elementwise_enabled()):
        return None
    axis = axis % x.dim() if x.dim() else 0
    if x.dim() == 0:
        return None
    xc = x.contiguous()
    outer, r, inner = _outer_r_inner(xc, axis)
    if inner > 1 and op == "sum" and outer == 1 and r > 4096 and supports_rows(xc.reshape(r, inner)):
        # column sums of a tall 2-D matrix (bias-gradient shape) have their own slab kernel
        out = colsum(xc.reshape(r, inner), out_dtype=x.dtype)
        return out.reshape([1] + list(xc.shape[axis + 1:]) if keepdims else list(xc.shape[axis + 1:]))
    shape = list(xc.shape)
    if keepdims:
        shape[axis] = 1
    else:
        shape.pop(axis)
    out = torch.empty(shape, dtype=torch.int64 if op.startswith("arg") else x.dtype, device=x.device)
    splits = _L().nb_reduce_splits(outer, r, inner)
    scratch = torch.empty(outer * splits * inner * 3 + 1, dtype=torch.float32, device=x.device) if splits > 1 else None
    _ok(_L().nb_reduce(ptr(xc), ptr(out), ptr(scratch), outer, r, inner, REDUCE_OPS[op], _dt(xc), stream_ptr()), "reduce")
    return out


def cumsum(x: torch.Tensor, axis: int, exclusive: bool = False, reverse: bool = False):
    if not (x.is_cuda and x.dtype in _FLOATS and x.numel() and x.dim() and elementwise_enabled()):
        return None
    xc = x.contiguous()
    outer, r, inner = _outer_r_inner(xc, axis % x.dim())
    if outer * inner < 4096 and r > 2048:
        return None                      # a few long scans: the sequential-per-column kernel is the wrong tool
    out = torch.empty_like(xc)
    _ok(_L().nb_cumsum(ptr(xc), ptr(out), outer, r, inner, int(exclusive), int(reverse), _dt(xc), stream_ptr()), "cumsum")
    return out
