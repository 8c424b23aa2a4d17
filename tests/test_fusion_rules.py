"""Rules of the fused schedules of compiled recordings and of the wrappers around kernels, asked on the CPU: they look at
shapes, types and devices alone."""
import weakref
from types import SimpleNamespace

import pytest
import torch

from nabla_b200.core.graph import fusion
from nabla_b200.core.graph.tracing import OpNode
from nabla_b200.core.tensor.impl import TensorImpl
from nabla_b200.types import Device, DType

GPU, GPU1, HOST = Device("gpu", 0), Device("gpu", 1), Device("cpu", 0)


class _Graph:
    """Recorded nodes whose tensors have no values."""

    def __init__(self):
        self.nodes, self.keep = [], []

    def tensor(self, *shape, device=GPU, dtype=DType.bfloat16):
        t = TensorImpl(None, shape=shape, dtype=dtype, device=device)
        self.keep.append(t)
        return t

    def op(self, name, args, *shapes, dtype=DType.bfloat16, **kwargs):
        n = OpNode(SimpleNamespace(name=name), list(args), None, kwargs, kwargs)
        outs = [self.tensor(*s, dtype=dtype) for s in shapes]
        for o in outs:
            o.output_refs = n
        n.out_refs = [weakref.ref(o) for o in outs]
        self.nodes.append(n)
        return outs[0] if len(outs) == 1 else outs

    def plan(self, *targets):
        return [(kind, tuple(self.nodes[i].op.name for i in idxs))
                for kind, idxs in fusion.build_plan(self.nodes, list(targets), private=True).steps]


@pytest.mark.parametrize("device,fused", [(GPU, True), (GPU1, False), (HOST, False)])
@pytest.mark.parametrize("name", ["matmul", "linear"])
def test_residual_on_another_device_stays_an_add(name, device, fused):
    g = _Graph()
    y = g.op(name, [g.tensor(64, 32), g.tensor(32, 64)], (64, 64))
    z = g.op("add", [y, g.tensor(64, 64, device=device)], (64, 64))
    assert g.plan(z) == ([("gemm_residual", (name, "add"))] if fused else [("op", (name,)), ("op", ("add",))])


@pytest.mark.parametrize("device,fused", [(GPU, True), (GPU1, False), (HOST, False)])
def test_gradient_on_another_device_does_not_join_the_layer_norm(device, fused):
    g = _Graph()
    stat = lambda: g.tensor(64, dtype=DType.float32)  # noqa: E731
    dx, dg, db = g.op("layer_norm_bwd", [g.tensor(64, 32), g.tensor(64, 32), stat(), stat(), g.tensor(32)], (64, 32), (32,), (32,))
    z = g.op("add", [g.tensor(64, 32, device=device), dx], (64, 32))
    assert (g.plan(z, dg, db)[0][0] == "ln_bwd_add") == fused


@pytest.mark.parametrize("shape", [(1,), ()])
def test_a_factor_leaves_products_their_own_epilogues(shape):
    """Backward of gelu(x w1) w2 * s: the scaled gradient is read by two products, one of which ends in the gelu's gradient. That
    pass is over tokens x hidden, the factor's over tokens x dim."""
    g = _Graph()
    dy = g.op("mul", [g.tensor(64, 32), g.tensor(*shape)], (64, 32))
    dw = g.op("matmul", [g.tensor(128, 64), dy], (128, 32))
    dz = g.op("dact_mul", [g.op("matmul", [dy, g.tensor(32, 128)], (64, 128)), g.tensor(64, 128)], (64, 128), activation="gelu")
    assert g.plan(dw, dz) == [("op", ("mul",)), ("op", ("matmul",)), ("gemm_dact", ("matmul", "dact_mul"))]


def test_a_factor_leaves_products_their_bias_and_activation():
    g = _Graph()
    x = g.op("mul", [g.tensor(64, 32), g.tensor(1)], (64, 32))
    y = g.op("relu", [g.op("add", [g.op("matmul", [x, g.tensor(32, 128)], (64, 128)), g.tensor(1, 128)], (64, 128))], (64, 128))
    assert g.plan(y) == [("op", ("mul",)), ("linear_epilogue", ("matmul", "add", "relu"))]


def test_a_factor_of_plain_products_goes_into_their_epilogues():
    g = _Graph()
    x = g.op("mul", [g.tensor(1), g.tensor(64, 32)], (64, 32))
    y, z = g.op("matmul", [x, g.tensor(32, 128)], (64, 128)), g.op("matmul", [g.tensor(16, 64), x], (16, 32))
    assert g.plan(y, z) == [("scale_gemm", ("mul", "matmul"))] * 2


class _Fake:
    """A tensor of the GPU as far as a wrapper looks before it launches."""

    def __init__(self, *shape, dtype):
        self.shape, self.dtype, self.is_cuda, self.device = shape, dtype, True, torch.device("cuda", 0)

    def dim(self):
        return len(self.shape)

    def get_device(self):
        return 0


def test_wrappers_refuse_operands_on_the_host():
    from nabla_b200.native import gemm, kernels

    a, b = _Fake(64, 512, dtype=torch.float32), _Fake(512, 64, dtype=torch.float32)
    assert kernels.sgemm(a, b, torch.zeros(64)) is None                # the caller's torch call then raises
    x, w, host = _Fake(64, 32, dtype=torch.bfloat16), _Fake(32, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16)
    for args, kw in (((x, host), {}), ((x, w), {"bias": host[0]}), ((x, w), {"aux": "add", "aux_in": torch.zeros(64, 64, dtype=torch.bfloat16)}),
                     ((x, w), {"alpha": torch.ones(1)}), ((host.t(), host), {})):
        with pytest.raises(RuntimeError, match="same GPU"):
            gemm.gemm_bf16(*args, **kw)
    with pytest.raises(RuntimeError, match="same GPU"):
        kernels.layernorm_bwd(x, x, None, None, None, add=host)
    table, ids = _Fake(64, 32, dtype=torch.bfloat16), torch.zeros(5, dtype=torch.int64)
    with pytest.raises(RuntimeError, match="same GPU"):
        kernels.embedding_gather(table, ids)
    with pytest.raises(RuntimeError, match="same GPU"):
        kernels.embedding_scatter_add(None, ids, table, 64, torch.bfloat16)


def test_a_slice_count_that_could_not_be_asked_for_is_not_kept(monkeypatch):
    from nabla_b200 import native
    from nabla_b200.native import gemm

    answers = [0, 4, 1]
    monkeypatch.setattr(gemm, "_get", lambda: None)
    monkeypatch.setattr(native, "load", lambda name: SimpleNamespace(nb_gemm_slices=lambda *a: answers.pop(0)))
    sizes = (123457, 11, 13)                       # nobody else's
    assert [gemm.cluster_slices(*sizes) for _ in range(3)] == [1, 4, 4]


def test_a_group_with_a_large_tensor_is_left_to_single_updates():
    from nabla_b200.native import kernels

    leaves = [tuple(torch.zeros(n) for _ in range(4)) + (True,) for n in (8, (1 << 20) + 8)]
    assert kernels.adamw_group(leaves, lr=1e-3, b1=0.9, b2=0.99, eps=1e-8, wd=0.0, step=1) is None


@pytest.mark.parametrize("slices,shape,view,fused", [
    (1, (64, 512), lambda r: r, True), (1, (64, 77), lambda r: r, False), (1, (64, 515), lambda r: r[:, :512], False), (1, (65, 512), lambda r: r[1:], True),
    (1, (64, 513), lambda r: r.reshape(-1)[1:64 * 512 + 1].view(64, 512), False), (1, (512, 64), lambda r: r.t(), True), (1, (77, 64), lambda r: r.t(), False),
    (2, (64, 77), lambda r: r, True), (2, (64, 515), lambda r: r[:, :512], True)])
def test_residual_rows_that_the_epilogue_reads_in_pieces_of_two_bytes_are_added_behind_it(monkeypatch, slices, shape, view, fused):
    from nabla_b200.native import gemm

    monkeypatch.setattr(gemm, "cluster_slices", lambda *a: slices)
    r = view(torch.zeros(shape, dtype=torch.bfloat16))
    assert gemm.residual_in_epilogue(r.shape[0], r.shape[1], 512, r) == fused


@pytest.mark.parametrize("N,H,C,F,R,stride,fp32,bf16", [
    (256, 28, 1, 16, 3, 1, True, True), (256, 14, 16, 32, 3, 1, True, True), (256, 14, 16, 32, 1, 1, False, False),      # taps to share a band
    (64, 7, 16, 16, 3, 1, True, True), (256, 6, 16, 32, 3, 1, False, False), (100, 4, 24, 17, 3, 2, False, False),         # positions of a band
    (64, 6, 5, 4, 5, 1, True, True), (8, 4, 5, 9, 3, 1, False, False), (64, 6, 1, 48, 3, 1, False, False),
    (64, 28, 16, 32, 2, 2, False, False), (1, 224, 3, 16, 3, 2, True, False), (1, 224, 8, 16, 3, 2, False, False),         # what a slice stages
    (1, 112, 24, 17, 5, 1, False, False), (16, 28, 16, 17, 3, 1, False, False), (16, 28, 16, 20, 5, 1, True, True),        # dy one value at a time
    (64, 28, 16, 32, 3, 1, False, False), (1, 512, 64, 8, 7, 1, False, False)])                                              # a full chip; 48 KB
def test_filter_gradients_that_read_patches(N, H, C, F, R, stride, fp32, bf16):
    from nabla_b200.native import load

    o = (H + 2 * (R // 2) - R) // stride + 1
    ask = load("libnb_kernels.so").nb_conv2d_wgrad_patches
    assert [bool(ask(N, H, H, C, R, R, F, o, o, stride, stride, dtype)) for dtype in (0, 1)] == [fp32, bf16]


@pytest.mark.parametrize("N,E,C,F,R,stride,px", [
    (256, 28, 1, 16, 3, 1, 8), (256, 14, 16, 32, 3, 1, 8), (16, 16, 8, 32, 3, 1, 4), (1, 14, 16, 32, 3, 1, 0),                # blocks enough
    (256, 14, 16, 32, 1, 1, 8), (100, 32, 32, 32, 1, 2, 0), (100, 40, 12, 16, 2, 2, 0), (16, 128, 8, 16, 3, 2, 4),           # terms per value
    (64, 24, 32, 1, 1, 1, 0), (256, 12, 8, 33, 2, 1, 0), (256, 32, 12, 33, 3, 1, 8),                                          # results one by one
    (16, 40, 1, 32, 3, 1, 0), (100, 12, 1, 64, 3, 1, 0), (32, 112, 5, 20, 3, 1, 0), (128, 64, 1, 8, 3, 1, 8), (64, 56, 3, 32, 1, 1, 8),
    (100, 64, 5, 7, 7, 1, 8), (16, 112, 3, 64, 7, 2, 0), (64, 64, 64, 64, 5, 1, 0)])
def test_convolutions_that_read_patches(N, E, C, F, R, stride, px):
    from nabla_b200.native import load

    o = (E + 2 * (R // 2) - R) // stride + 1
    assert load("libnb_kernels.so").nb_conv2d_patches(N, E, E, C, R, R, F, o, o, stride, stride) == px


@pytest.mark.parametrize("M,N,K,orders", [            # (rows, rows), (columns, rows), (rows, columns), (columns, columns)
    (17, 64, 256, [True] * 4), (16, 64, 256, [True, False, False, True]), (10, 64, 256, [False, False, False, True]), (10, 64, 320, [True, False, False, True]),
    (10, 65, 256, [True, True, False, True]), (16, 64, 512, [True, True, False, True]), (16, 64, 513, [True] * 4), (16, 1000, 400, [True] * 4),
    (16, 1000, 401, [False, False, True, True]), (16, 1000, 801, [False, False, True, False]), (64, 8, 512, [False] * 4)])
def test_small_products_of_few_rows_that_the_library_has_kernels_for(M, N, K, orders):
    from nabla_b200.native import kernels

    for (ta, tb), takes in zip([(False, False), (True, False), (False, True), (True, True)], orders):
        a = torch.empty(K, M).t() if ta else torch.empty(M, K)
        b = torch.empty(N, K).t() if tb else torch.empty(K, N)
        assert kernels.sgemm_takes(a, b) == takes and kernels.sgemm_takes(a, b, torch.empty(N)) == kernels.sgemm_pays(M, N, K)


@pytest.mark.parametrize("rows,cols,bf16,how", [(2500, 3072, True, 2), (2501, 3072, True, 0), (4096, 4096, True, 2), (4097, 4096, True, 0), (2501, 1536, False, 0), (4096, 2048, False, 2),
                                                (4096, 2560, True, 1), (4096, 777, True, 2)])
def test_column_sums_go_by_clusters_where_these_fill_the_chip(rows, cols, bf16, how):
    from nabla_b200.native.kernels import colsum_clusters

    assert colsum_clusters(rows, cols, torch.bfloat16 if bf16 else torch.float32) == how


def test_factors_that_a_thin_operand_takes_do_not_round_it():
    """Beside a larger product a low-rank one is scaled before it: by powers of two alone, whose products with bf16 values are exact."""
    h = torch.randn(1000).bfloat16()
    for x, takes in ((1, True), (1.0, True), (2.0, True), (0.25, True), (0.75, False), (4 / 3, False), (-2.0, False), (0.0, False), (True, True), (None, False),
                     (float("inf"), False), (float("nan"), False), (2.0 ** 100, False), (10 ** 400, False)):
        assert fusion._is_power_of_two(x) is takes, x
        if takes:
            assert torch.equal((h * x).double(), h.double() * x)
