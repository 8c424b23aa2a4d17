"""Kernels and dispatch rules at the sizes where they can go wrong (tile edges, remainders, the smallest and
largest of a rule's range) against 64-bit torch results. Needs a B200 (sm_100a)."""
import os
import subprocess
import sys

import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu

# largest relative error (2-norm) of a result stored in the type: half a unit in the last place at most, and for
# fp32 the rounding of sums of a few hundred terms
STORED = {torch.bfloat16: 2.0 ** -8, torch.float32: 4e-6}


def _rel2(got, ref):
    got, ref = got.double(), ref.double()
    return ((got - ref).norm() / ref.norm().clamp_min(1e-30)).item()


@pytest.fixture(autouse=True)
def _check_status():
    yield
    from nabla_b200 import native

    torch.cuda.synchronize()
    native.check_status()


# ---------------------------------------------------------------- direct convolution
def _windows(x, R, S, stride, pad):
    """(N, OH, OW, R, S, C) windows of an NHWC tensor and which of their positions lie in the image."""
    pt, pb, pl, pr = pad

    def cut(t):
        t = TF.pad(t, (0, 0, pl, pr, pt, pb))
        return t.unfold(1, R, stride[0]).unfold(2, S, stride[1]).permute(0, 1, 2, 4, 5, 3)

    return cut(x), cut(torch.ones_like(x)) > 0


def _conv64(x, w, b, stride, pad):
    """Convolution and its terms for the filter gradient; a padded position is absent, not 0 * w."""
    win, ok = _windows(x.double(), w.shape[0], w.shape[1], stride, pad)
    terms = torch.where(ok.unsqueeze(-1), win.unsqueeze(-1) * w.double(), torch.zeros((), dtype=torch.float64, device=x.device))
    return terms.sum((3, 4, 5)) + b.double(), win, ok


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,H,W,C,F,R,S,stride,pad", [
    (1, 3, 3, 1, 1, 3, 3, (1, 1), (1, 1, 1, 1)), (2, 9, 7, 1, 8, 3, 3, (1, 1), (1, 1, 1, 1)), (3, 8, 8, 3, 9, 3, 3, (2, 1), (1, 1, 2, 0)),
    (2, 11, 11, 4, 16, 3, 3, (1, 1), (1, 1, 1, 1)), (2, 7, 13, 5, 17, 5, 2, (1, 2), (2, 2, 0, 1)), (4, 16, 16, 8, 33, 3, 3, (1, 1), (1, 1, 1, 1)),
    (1, 6, 6, 36, 12, 1, 1, (1, 1), (0, 0, 0, 0)), (5, 33, 33, 2, 4, 3, 3, (1, 1), (0, 0, 0, 0))])
def test_direct_convolution_and_filter_gradient(dtype, N, H, W, C, F, R, S, stride, pad):
    from nabla_b200.native import kernels

    torch.manual_seed(0)
    x = torch.randn(N, H, W, C, device="cuda").to(dtype)
    w = torch.randn(R, S, C, F, device="cuda").to(dtype)
    b = torch.randn(F, device="cuda").to(dtype)
    y = kernels.conv2d_direct(x, w, b, stride, pad)
    ref, win, _ = _conv64(x, w, b, stride, pad)
    assert y.shape == ref.shape and _rel2(y, ref) < STORED[dtype]
    dy = torch.randn(ref.shape, device="cuda").to(dtype)
    dw = kernels.conv2d_wgrad_direct(x, dy, tuple(w.shape), stride, pad)
    assert _rel2(dw, torch.einsum("nhwrsc,nhwf->rscf", win, dy.double())) < STORED[dtype]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,H,W,C,F,R,S,stride,pad", [
    (3, 14, 14, 16, 32, 3, 3, (1, 1), (1, 1, 1, 1)), (2, 14, 14, 32, 16, 3, 3, (1, 1), (1, 1, 1, 1)), (2, 28, 28, 1, 16, 3, 3, (1, 1), (1, 1, 1, 1)),
    (2, 15, 31, 3, 8, 3, 3, (1, 1), (1, 1, 1, 1)), (1, 32, 32, 8, 17, 3, 3, (1, 1), (2, 0, 0, 2)), (2, 29, 33, 4, 6, 3, 3, (2, 2), (1, 1, 1, 1)),
    (5, 8, 8, 12, 33, 1, 5, (1, 1), (0, 0, 2, 2)), (2, 16, 16, 5, 64, 2, 2, (1, 1), (0, 0, 0, 0)), (300, 16, 16, 8, 16, 3, 3, (1, 1), (1, 1, 1, 1)),
    (1, 64, 64, 4, 8, 3, 3, (1, 1), (1, 1, 1, 1)), (1, 3, 256, 4, 16, 3, 3, (1, 1), (1, 1, 1, 1)), (2, 20, 20, 36, 40, 3, 3, (1, 1), (1, 1, 1, 1))])
def test_direct_convolution_from_patches(dtype, N, H, W, C, F, R, S, stride, pad):
    """Bands of rows with and without a remainder, both counts of positions per thread, channels in fours and not, halos, strides,
    channel tiles with a remainder, filters and gradients that are not finite under padding; output and filter gradient."""
    from nabla_b200.native import kernels

    torch.manual_seed(0)
    x = torch.randn(N, H, W, C, device="cuda").to(dtype)
    w = torch.randn(R, S, C, F, device="cuda").to(dtype)
    b = torch.randn(F, device="cuda").to(dtype)
    ref, _, _ = _conv64(x, w, b, stride, pad)
    y = kernels.conv2d_direct(x, w, b, stride, pad)
    assert y.shape == ref.shape and _rel2(y, ref) < STORED[dtype]
    ref, _, _ = _conv64(x, w, torch.zeros_like(b), stride, pad)
    assert _rel2(kernels.conv2d_direct(x, w, None, stride, pad), ref) < STORED[dtype]
    _, win, ok = _conv64(x, w, b, stride, pad)
    dy = torch.randn(ref.shape, device="cuda").to(dtype)
    dw = kernels.conv2d_wgrad_direct(x, dy, tuple(w.shape), stride, pad)
    assert _rel2(dw, torch.einsum("nhwrsc,nhwf->rscf", win, dy.double())) < STORED[dtype]
    if N < 10:
        dy[0, 0, 0, F - 1], dy[N - 1, -1, -1, 0] = float("inf"), float("nan")
        ref = torch.where(ok.unsqueeze(-1), win.unsqueeze(-1) * dy.double()[:, :, :, None, None, None], torch.zeros((), dtype=torch.float64, device="cuda")).sum((0, 1, 2))
        dw = kernels.conv2d_wgrad_direct(x, dy, tuple(w.shape), stride, pad).double()
        fin = torch.isfinite(ref)
        assert torch.equal(torch.isfinite(dw), fin) and torch.equal(torch.isnan(dw), torch.isnan(ref)) and _rel2(dw[fin], ref[fin]) < STORED[dtype]
        w[0, 0, 0, F - 1], w[R - 1, S - 1, C - 1, 0] = float("inf"), float("nan")
        ref, _, _ = _conv64(x, w, b, stride, pad)
        y = kernels.conv2d_direct(x, w, b, stride, pad).double()
        ok = torch.isfinite(ref)
        assert torch.equal(torch.isfinite(y), ok) and torch.equal(torch.isnan(y), torch.isnan(ref)) and _rel2(y[ok], ref[ok]) < STORED[dtype]


def test_direct_convolution_skips_padding_under_infinite_operands():
    from nabla_b200.native import kernels

    torch.manual_seed(1)
    x = torch.randn(2, 6, 5, 4, device="cuda")
    w = torch.randn(3, 3, 4, 10, device="cuda")
    w[0, 1, 2, 3], w[2, 2, 0, 7] = float("inf"), float("nan")
    b = torch.zeros(10, device="cuda")
    y = kernels.conv2d_direct(x, w, b, (1, 1), (1, 1, 1, 1))
    ref, win, ok = _conv64(x, w, b, (1, 1), (1, 1, 1, 1))
    torch.testing.assert_close(y.double(), ref, rtol=1e-5, atol=1e-5, equal_nan=True)
    dy = torch.randn(2, 6, 5, 10, device="cuda")
    dy[0, 0, 0, 1], dy[1, 5, 4, 9] = float("inf"), float("nan")
    dw = kernels.conv2d_wgrad_direct(x, dy, tuple(w.shape), (1, 1), (1, 1, 1, 1))
    zero = torch.zeros((), dtype=torch.float64, device="cuda")
    ref = torch.where(ok.unsqueeze(-1), win.unsqueeze(-1) * dy.double()[:, :, :, None, None, None, :], zero).sum((0, 1, 2))
    torch.testing.assert_close(dw.double(), ref, rtol=1e-5, atol=1e-5, equal_nan=True)


@pytest.mark.parametrize("H,W,R,S,pad", [(1, 1 << 20, 2100, 1, (2099, 0, 0, 0)), (2, 4, 40000, 1, (39999, 0, 0, 0)), (1, 2, 1, 70000, (0, 0, 69999, 0))])
def test_direct_convolution_with_tall_and_wide_filters(H, W, R, S, pad):
    """Filter taps whose offset in the image passes 2^31 (only the last rows of the filter meet the image), and
    more rows and columns than 16 bits hold. Small whole values: every sum is exact."""
    from nabla_b200.native import kernels

    torch.manual_seed(1)
    x = torch.randint(-3, 4, (1, H, W, 1), device="cuda").float()
    w = torch.randint(-3, 4, (R, S, 1, 1), device="cuda").float()
    y = kernels.conv2d_direct(x, w, None, (1, 1), pad)
    dy = torch.randint(-1, 2, y.shape, device="cuda").float()
    dw = kernels.conv2d_wgrad_direct(x, dy, tuple(w.shape), (1, 1), pad)
    ref, ref_dw = torch.zeros_like(y, dtype=torch.float64), torch.zeros_like(w, dtype=torch.float64)
    for oh in range(y.shape[1]):
        for ow in range(y.shape[2]) if S > 1 else [slice(None)]:
            # the window's first row (column) lies pad above (left of) output row oh (column ow)
            rows = slice(max(0, pad[0] - oh), min(R, H + pad[0] - oh))
            top = rows.start - (pad[0] - oh)
            n = rows.stop - rows.start
            if S > 1:
                cols = slice(max(0, pad[2] - ow), min(S, W + pad[2] - ow))
                left, m = cols.start - (pad[2] - ow), cols.stop - cols.start
                part = x[0, top:top + n, left:left + m, 0].double()
                ref[0, oh, ow, 0] = (w[rows, cols, 0, 0].double() * part).sum()
                ref_dw[rows, cols, 0, 0] += part * dy[0, oh, ow, 0].double()
            else:
                part = x[0, top:top + n, :, 0].double()
                ref[0, oh, :, 0] = (w[rows, 0, 0, 0].double()[:, None] * part).sum(0)
                ref_dw[rows, 0, 0, 0] += (part * dy[0, oh, :, 0].double()).sum(1)
    assert torch.equal(y.double(), ref) and torch.equal(dw.double(), ref_dw)


@pytest.mark.parametrize("F", [32 * 65535, 32 * 65535 + 1, 3 * 32 * 65535 + 77])
def test_direct_convolution_to_more_channel_tiles_than_a_grid_holds_in_y(F):
    from nabla_b200.native import kernels

    x = torch.tensor([2.0, 3.0], device="cuda").view(1, 1, 2, 1)
    w = torch.randint(-3, 4, (1, 1, 1, F), device="cuda").float()
    y = kernels.conv2d_direct(x, w, None, (1, 1), (0, 0, 0, 0))
    assert torch.equal(y, x * w.view(F))


# ---------------------------------------------------------------- adds and factors that GEMMs and the layer norm take
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,D", [(1, 8), (5, 128), (777, 256), (9, 264), (33, 1000), (1001, 512), (300, 2048), (4, 1024)])
def test_layer_norm_backward_plus_a_gradient(dtype, rows, D):
    """dx + add, rounded once, by the kernel of narrow rows and the one of wide rows; dgamma and dbeta as without it."""
    from nabla_b200.native import kernels

    torch.manual_seed(rows)
    x, dy, add = (torch.randn(rows, D, device="cuda").to(dtype) for _ in range(3))
    g, b = torch.randn(D, device="cuda").to(dtype), torch.randn(D, device="cuda").to(dtype)
    _, mean, rstd = kernels.layernorm_fwd(x, g, b, 1e-5)
    plain, got = kernels.layernorm_bwd(dy, x, g, mean, rstd), kernels.layernorm_bwd(dy, x, g, mean, rstd, add=add)
    x64 = x.double().requires_grad_(True)
    ref, = torch.autograd.grad(TF.layer_norm(x64, (D,), g.double(), b.double()), x64, dy.double())
    assert _rel2(got[0], ref + add.double()) < STORED[dtype]
    assert torch.equal(got[1], plain[1]) and torch.equal(got[2], plain[2])


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (130, 64, 72), (257, 77, 200), (2048, 16, 6144), (16, 512, 2048), (300, 1024, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemm_with_a_factor_on_the_device(M, N, K, dtype):
    """Also where the product is cut into K slices, and beside a bias and a residual."""
    from nabla_b200.native.gemm import gemm_bf16

    torch.manual_seed(0)
    a, b = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
    s = torch.tensor([1.7], device="cuda").to(dtype)
    ref = (a.double() @ b.double()) * s.double()
    assert _rel2(gemm_bf16(a, b, alpha=s), ref) < STORED[torch.bfloat16]
    bias, res = torch.randn(N, device="cuda").bfloat16(), torch.randn(M, N, device="cuda").bfloat16()
    got = gemm_bf16(a, b, alpha=s, bias=bias, aux="add", aux_in=res)
    assert _rel2(got, ref + bias.double() + res.double()) < STORED[torch.bfloat16]


@pytest.mark.parametrize("tokens,dim,out,rank", [(100, 64, 192, 8), (333, 128, 77, 16), (1, 64, 64, 8), (2, 4096, 64, 8)])
def test_compiled_products_take_their_adds_and_factors(tokens, dim, out, rank):
    """x w + (x a) b s, a residual and a layer norm between them: values and gradients against 64 bits, with the steps that the
    schedule has to have; a product that is asked for on its own stays on its own."""
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    torch.manual_seed(tokens)
    mk = lambda *s: torch.randn(*s, device="cuda").mul(s[0] ** -0.5 if len(s) == 2 else 1.0).bfloat16()  # noqa: E731
    x, w, a, b = torch.randn(tokens, dim, device="cuda").bfloat16(), mk(dim, out), mk(dim, rank), mk(rank, out)
    g, be, w2, dy = mk(dim), mk(dim), mk(out, dim), torch.randn(tokens, dim, device="cuda").bfloat16()

    def layer(x, w, a, b, g, be, w2):
        h = F.layer_norm(x, g, be)
        y = h @ w + ((h @ a) @ b) * 0.75
        return x + F.linear(y, w2)

    def layer64(x, w, a, b, g, be, w2):
        h = TF.layer_norm(x, (dim,), g, be)
        return x + (h @ w + ((h @ a) @ b) * 0.75) @ w2

    args = (x, w, a, b, g, be, w2)
    ps = [t.double().requires_grad_(True) for t in args]
    y64 = layer64(*ps)
    want = [y64] + list(torch.autograd.grad(y64, ps, dy.double()))
    ts, dt = [nb.Tensor.from_torch(t) for t in args], nb.Tensor.from_torch(dy)

    def run(*ps):
        y, pull = nb.vjp(layer, *ps[:-1], create_graph=False)
        return (y, *pull(ps[-1]))

    f = nb.compile(run)
    for _ in range(2):
        for got, ref in zip(f(*ts, dt), want):
            assert _rel2(got.to_torch(), ref) < 2.5e-2          # five products of bf16 operands and results, 2^-9 each, in a chain
    plan = str(f.dump_plan())
    for kind in ("gemm_residual", "gemm_scale", "scale_gemm", "ln_bwd_add"):
        assert (kind in plan) or (tokens == 1 and kind == "gemm_residual"), (kind, plan)
    h = nb.compile(lambda x, w, r: (lambda p: (p, p + r))(x @ w))
    p, q = h(ts[0], ts[1], nb.Tensor.from_torch(mk(tokens, out)))
    assert "gemm_residual" not in str(h.dump_plan()) and _rel2(p.to_torch(), x.double() @ w.double()) < STORED[torch.bfloat16]


@pytest.mark.parametrize("kind", ["gemm_residual", "linear_epilogue", "gemm_dact"])
def test_compiled_products_without_native_kernels(kind, monkeypatch):
    """The switch that turns the native kernels off holds for the steps that fuse a product with what follows it."""
    import nabla_b200 as nb
    from nabla_b200.native import gemm
    from nabla_b200.nn import functional as F

    monkeypatch.setenv("NABLA_B200_DISABLE_NATIVE", "1")
    torch.manual_seed(0)
    x, w, w2, r, b = (torch.randn(*s, device="cuda").bfloat16() for s in ((48, 32), (32, 64), (64, 64), (48, 64), (1, 64)))

    def mlp(x, w, w2, r, b):
        return nb.vjp(lambda t: F.linear(F.linear(t, w, b, activation="gelu"), w2), x, create_graph=False)[1](r)[0]

    call, ref = {"gemm_residual": (lambda x, w, w2, r, b: x @ w + r, x.double() @ w.double() + r.double()),
                 "linear_epilogue": (lambda x, w, w2, r, b: nb.relu(x @ w + b), torch.relu(x.double() @ w.double() + b.double())),
                 "gemm_dact": (mlp, None)}[kind]
    if ref is None:
        x64 = x.double().requires_grad_(True)
        ref = torch.autograd.grad(TF.gelu(x64 @ w.double() + b.double()) @ w2.double(), x64, r.double())[0]
    f, n = nb.compile(call), gemm.launch_count
    args = [nb.Tensor.from_torch(t) for t in (x, w, w2, r, b)]
    for _ in range(2):
        assert _rel2(f(*args).to_torch(), ref) < 4 * STORED[torch.bfloat16]      # up to three roundings of a value and a product's
    assert kind in str(f.dump_plan()) and gemm.launch_count == n


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("M,N,K", [(9473, 72, 64), (9600, 200, 64), (9473, 264, 128), (4800, 456, 64), (9473, 8, 64), (300, 328, 64), (130, 1096, 2048), (257, 128, 2048), (9473, 77, 64), (300, 333, 64), (130, 77, 1800)])
def test_residual_in_wide_and_sliced_tiles(M, N, K, fp32):
    """Both epilogue groups read a residual: ends of their 64-column pairs, of tiles of every width and of K slices."""
    from nabla_b200.native.gemm import gemm_bf16

    torch.manual_seed(M + N)
    a, b, res = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, K), (K, N), (M, N)))
    bias = torch.randn(N, device="cuda")
    ref = a.double() @ b.double() + bias.double() + res.double()
    out = gemm_bf16(a, b, bias=bias, aux="add", aux_in=res, out_dtype=torch.float32 if fp32 else torch.bfloat16)
    # fp32: each MMA of 16 products cuts its sum by less than one unit in the last place
    err = (out.double() - ref).abs().max().item()
    assert err <= (K / 16 * 2.0 ** -23 + (0 if fp32 else 2.0 ** -8)) * ref.abs().max().item()


def test_threads_that_ask_first_agree_on_the_slices():
    """Eight threads of a new process plan their first product at the same time; each has to get what a later call gets."""
    code = """
import threading, torch
torch.zeros(1, device="cuda")
from nabla_b200.native import gemm, load
gemm._get()
ask = load("libnb_gemm.so").nb_gemm_slices
start, got = threading.Barrier(8), [None] * 8
def one(i):
    start.wait()
    got[i] = ask(64, 256, 8192)
threads = [threading.Thread(target=one, args=(i,)) for i in range(8)]
for t in threads: t.start()
for t in threads: t.join()
assert got == [ask(64, 256, 8192)] * 8 and got[0] > 1, got
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]


def test_operands_on_the_host_are_refused():
    """A residual of a compiled product and a bias that live on the host, where the fused kernels would take them."""
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    t = lambda *s, d="cuda", ty=torch.bfloat16: nb.Tensor.from_torch(torch.ones(*s, device=d, dtype=ty))  # noqa: E731
    f32 = torch.float32
    for call, args in ((lambda x, w, r: x @ w + r, (t(64, 32), t(32, 64), t(64, 64, d="cpu"))),
                       (lambda x, w, b: F.linear(x, w, b), (t(64, 32), t(32, 64), t(64, d="cpu"))),
                       (lambda x, w, b: F.linear(x, w, b), (t(64, 512, ty=f32), t(512, 64, ty=f32), t(64, d="cpu", ty=f32)))):
        for fn in (call, nb.compile(call)):
            with pytest.raises(RuntimeError):
                fn(*args).to_torch()


@pytest.mark.parametrize("M,N,K,sliced", [(2048, 16, 2048, True), (1, 512, 2048, True), (130, 77, 1800, True), (2002, 512, 2048, True), (512, 512, 2002, True),
                                          (100, 1000, 8192, True), (257, 130, 4100, True), (16, 6144, 2048, True), (64, 64, 8193, False), (512, 512, 256, False), (64, 256, 512, True),
                                          (70, 100, 449, True), (512, 512, 8192, True), (4096, 4096, 2048, False)])
def test_products_on_clusters_of_k_slices(M, N, K, sliced):
    """Both orders of both operands, remainders in every dimension, a bias and a residual of odd rows, a factor, fp32 results; and
    the rule's lines. Against 64 bits, and the sum of the slices is the same bits on every run."""
    from nabla_b200.native import gemm as G

    assert (G.cluster_slices(M, N, K) > 1) == sliced
    assert G.split_k_factor(M, N, K) in (1, 8) and (G.split_k_factor(M, N, K) == 8) == ((M, N, K) == (512, 512, 8192))
    torch.manual_seed(0)
    mk = lambda r, c: torch.randn(r, c, device="cuda").bfloat16()  # noqa: E731
    orders = [(mk(M, K), mk(K, N)), (mk(K, M).t(), mk(K, N)), (mk(M, K), mk(N, K).t()), (mk(K, M).t(), mk(N, K).t())]
    bias, res, s = torch.randn(N, device="cuda"), mk(M, N), torch.tensor([0.5], device="cuda")
    for a, b in orders if M * N < 1 << 22 else orders[:1]:
        ref = a.double() @ b.double()
        got = G.gemm_bf16(a, b)
        assert _rel2(got, ref) < STORED[torch.bfloat16] and torch.equal(got, G.gemm_bf16(a, b))
        # each MMA of 16 products cuts its fp32 sum by less than one unit in the last place: a slice has fewer of them
        err = _rel2(G.gemm_bf16(a, b, out_dtype=torch.float32), ref)
        assert err < (K / 16 / G.cluster_slices(M, N, K) + 8) * 2.0**-23
        if sliced:
            assert err <= _rel2(G.gemm_bf16(a, b, out_dtype=torch.float32, block_n=64, split_k=1), ref)
        got = G.gemm_bf16(a, b, alpha=s, bias=bias, aux="add", aux_in=res)
        assert _rel2(got, 0.5 * ref + bias.double() + res.double()) < STORED[torch.bfloat16]


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (256, 10, 1568), (33, 31, 32), (32, 32, 33), (65, 10, 4097), (7, 1000, 3), (1, 4000, 500), (3000, 1, 65), (255, 255, 255)])
@pytest.mark.parametrize("ta,tb", [(False, False), (True, False), (False, True), (True, True)])
def test_small_fp32_products(M, N, K, ta, tb):
    """Every order of the operands, tiles and slices with remainders, a bias, an infinite operand beside the padding, and what the
    kernel leaves to the library. 2e-6: the rounding of sums of some hundred terms."""
    from nabla_b200.native import kernels

    torch.manual_seed(K)
    a = torch.randn(K, M, device="cuda").t() if ta else torch.randn(M, K, device="cuda")
    b = torch.randn(N, K, device="cuda").t() if tb else torch.randn(K, N, device="cuda")
    bias = torch.randn(1, N, device="cuda")
    ref = a.double() @ b.double()
    bound = 2e-6 * (a.double().abs() @ b.double().abs() + bias.double().abs())
    assert ((kernels.sgemm(a, b).double() - ref).abs() <= bound).all()
    assert ((kernels.sgemm(a, b, bias).double() - ref - bias.double()).abs() <= bound).all()
    a[0, K - 1] = float("inf")
    got = kernels.sgemm(a, b)
    assert torch.isinf(got[0]).all() and torch.isfinite(got[1:]).all()
    assert kernels.sgemm(a.bfloat16(), b.bfloat16()) is None and kernels.sgemm(a[None], b[None]) is None
    assert kernels.sgemm(a, b, bias.bfloat16()) is None and kernels.sgemm(a[:0], b) is None


def test_rule_of_small_fp32_products():
    """Both sides of the rule's lines, and that both entry points take the same bits from either side's kernel."""
    from nabla_b200.native import kernels
    from nabla_b200.ops import binary, fused

    for args, pays in (((9, 9, 256), True), ((8, 100, 512), False), ((100, 8, 512), False), ((256, 128, 256), True), ((257, 128, 256), False),
                       ((64, 10, 255), False), ((64, 10, 4096), True), ((64, 10, 4097), False)):
        assert kernels.sgemm_pays(*args) == pays
    torch.manual_seed(0)
    x, w, b = torch.randn(64, 300, device="cuda"), torch.randn(300, 10, device="cuda"), torch.randn(10, device="cuda")
    assert torch.equal(binary.MatmulOp().kernel(x, w), kernels.sgemm(x, w))
    assert torch.equal(fused.LinearOp().kernel(x, w, b), kernels.sgemm(x, w, b))
    y, z = fused.LinearOp().kernel(x, w, b, activation="relu")
    assert torch.equal(z, kernels.sgemm(x, w, b)) and torch.equal(y, z.clamp_min(0))


# ---------------------------------------------------------------- embedding gradient
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab,dim,n,hot", [
    (1, 8, 1, 0.0), (50, 33, 700, 0.0), (100, 256, 33, 1.0), (300, 64, 4096, 0.3), (300, 64, 4801, 0.3), (300, 33, 4801, 0.3),
    (4096, 2048, 500, 0.1), (4097, 2048, 500, 0.1), (4080, 2056, 3000, 0.05), (4097, 2056, 3000, 0.05), (50, 40, 801, 1.0),
    (8200, 1032, 9000, 0.5), (9000, 1001, 700, 0.5), (9000, 1040, 1030, 1.0), (9000, 1040, 1060, 1.0), (4097, 2056, 33000, 0.9), (40, 1032, 70000, 0.5)])
def test_embedding_scatter_add(dtype, vocab, dim, n, hot):
    """Both ways of adding (an fp32 table, the bucketed ids), rows of one to thousands of entries (segments of 32, groups
    of 32 segments), ids out of range, rows that are and are not whole 16-byte vectors, with and without a base table."""
    from nabla_b200.native import kernels

    torch.manual_seed(n)
    ids = torch.randint(-2, vocab + 2, (n,), device="cuda")
    ids[torch.rand(n, device="cuda") < hot] = vocab // 2
    upd = torch.randn(n, dim, device="cuda").to(dtype)
    base = torch.randn(vocab, dim, device="cuda").to(dtype)
    ok = (ids >= 0) & (ids < vocab)
    ref = torch.zeros(vocab, dim, dtype=torch.float64, device="cuda").index_add_(0, ids[ok], upd[ok].double())
    assert _rel2(kernels.embedding_scatter_add(base, ids, upd), ref + base.double()) < STORED[dtype]
    got = kernels.embedding_scatter_add(None, ids, upd, vocab, dtype)
    assert got.shape == (vocab, dim) and got.dtype is dtype and _rel2(got, ref) < STORED[dtype]
    empty = kernels.embedding_scatter_add(base, ids[:0], upd[:0])
    assert torch.equal(empty, base)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab,dim", [(40000, 264), (9000, 1048), (9001, 2056), (40000, 517), (1100000, 8)])
def test_embedding_gradient_by_row_counts(dtype, vocab, dim):
    """Rows of 0 to 4 entries (a warp's work), of 5 and more (a block's), at the ends of the segments of 32, spread over the
    table; the rows without an entry are the base's bit for bit."""
    from nabla_b200.native import kernels

    torch.manual_seed(dim)
    counts = [1, 2, 3, 4, 5, 31, 32, 33, 64, 65] * 12 + [1] * 200 + [1100]
    rows = torch.randperm(vocab - 2, device="cuda")[:len(counts)] + 1
    rows[0], rows[1] = 0, vocab - 1
    ids = torch.repeat_interleave(rows, torch.tensor(counts, device="cuda"))
    ids = ids[torch.randperm(ids.numel(), device="cuda")]
    n = ids.numel()
    assert kernels._L().nb_embedding_scatter_work(n, dim, vocab, 1 if dtype == torch.bfloat16 else 0) != vocab * dim
    upd = torch.randn(n, dim, device="cuda").to(dtype)
    base = torch.randn(vocab, dim, device="cuda").to(dtype)
    ref = torch.zeros(vocab, dim, dtype=torch.float64, device="cuda").index_add_(0, ids, upd.double())
    idle = torch.ones(vocab, dtype=torch.bool, device="cuda")
    idle[rows] = False
    got = kernels.embedding_scatter_add(base, ids, upd)
    assert torch.equal(got[idle], base[idle]) and _rel2(got[rows], ref[rows] + base[rows].double()) < STORED[dtype]
    got = kernels.embedding_scatter_add(None, ids, upd, vocab, dtype)
    assert not got[idle].any() and _rel2(got[rows], ref[rows]) < STORED[dtype]


@pytest.mark.parametrize("dtype,vocab,dim,n", [(torch.float32, 9000, 1048, 35999), (torch.float32, 9000, 1048, 36000), (torch.float32, 1300, 1020, 31200), (torch.float32, 1300, 1020, 31199),
                                               (torch.bfloat16, 400, 4096, 9600), (torch.bfloat16, 400, 4096, 9599), (torch.bfloat16, 3, 2048, 60000)])
def test_embedding_gradient_into_crowded_tables(dtype, vocab, dim, n):
    """Both sides of the line from which on only the rows that occur are written over a copy of the base."""
    from nabla_b200.native import kernels

    torch.manual_seed(n)
    assert kernels._L().nb_embedding_scatter_work(n, dim, vocab, 1 if dtype == torch.bfloat16 else 0) != vocab * dim
    ids = (vocab * torch.rand(n, device="cuda") ** 3).long().clamp_(max=vocab - 1)
    ids[ids == 1] = 0                                        # a row without an entry
    ids[3], ids[7] = -1, vocab                               # outside the table
    inside = (ids >= 0) & (ids < vocab)
    upd = torch.randn(n, dim, device="cuda").to(dtype)
    base = torch.randn(vocab, dim, device="cuda").to(dtype)
    ref = torch.zeros(vocab, dim, dtype=torch.float64, device="cuda").index_add_(0, ids[inside], upd[inside].double())
    got = kernels.embedding_scatter_add(base, ids, upd)
    assert torch.equal(got[1], base[1]) and _rel2(got, ref + base.double()) < STORED[dtype]
    got = kernels.embedding_scatter_add(None, ids, upd, vocab, dtype)
    assert not got[1].any() and _rel2(got, ref) < STORED[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("ids,add,fused", [
    ((3, 70), (70, 64), True), ((3, 70), (64,), True), ((3, 70), (1, 70, 64), True), ((3, 70), (1, 1, 64), True), ((7,), (7, 64), True),
    ((3, 70), (3, 70, 64), True), ((3, 70), (3, 70, 33), True), ((3, 70), (3, 1, 64), False), ((3, 70), (70, 1), False), ((2, 3), (4, 2, 3, 64), False)])
def test_embedding_plus_a_tensor_over_trailing_dims(dtype, ids, add, fused):
    """One pass where the added tensor covers trailing dims (the sum is the one of two passes, bit for bit), two elsewhere, also
    where the rows are asked for on their own."""
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    torch.manual_seed(1)
    dim = add[-1] if add[-1] > 1 else 64
    table = torch.randn(50, dim, device="cuda").to(dtype)
    pos = torch.randn(add, device="cuda").to(dtype)
    idx = torch.randint(0, 50, ids, device="cuda")
    ref = (table[idx].float() + pos.float()).to(dtype)
    tt, pt, it = nb.Tensor.from_torch(table), nb.Tensor.from_torch(pos), nb.Tensor.from_torch(idx)
    for order in (lambda a, b: a + b, lambda a, b: b + a):
        f = nb.compile(lambda t, p, i: nb.vjp(lambda a, b: order(F.embedding(i, a), b), t, p, create_graph=False)[0])
        g = nb.compile(lambda t, p, i: (lambda rows: (rows, order(rows, p)))(F.embedding(i, t)))
        for _ in range(2):
            assert torch.equal(f(tt, pt, it).to_torch(), ref)
            rows, out = g(tt, pt, it)
            assert torch.equal(rows.to_torch(), table[idx]) and torch.equal(out.to_torch(), ref)
        assert ("gather_add" in f.dump_plan()) == fused and "gather_add" not in g.dump_plan()


@pytest.mark.parametrize("vocab,dim,n,dtype,atomics", [
    (16, 8, 1000, 1, True), (4096, 2048, 12288, 1, True), (4097, 2048, 100, 1, False), (4096, 2048, 12289, 1, False), (1000, 64, 49152, 0, True),
    (1000, 64, 49153, 0, False), (256, 64, 100000, 0, True), (256, 64, 131073, 0, False), (9000, 1001, 700, 1, True), (32000, 1001, 700, 1, False),
    (32000, 1001, 32001, 1, True), (9000, 1004, 700, 1, True), (9000, 1004, 700, 0, False)])
def test_ways_of_adding_an_embedding_gradient(vocab, dim, n, dtype, atomics):
    """On both sides of the rule's lines: the atomics' scratch is the table in fp32."""
    from nabla_b200.native import kernels

    assert (kernels._L().nb_embedding_scatter_work(n, dim, vocab, dtype) == vocab * dim) == atomics


def test_gradient_of_an_embedding_takes_no_table_of_zeros():
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    torch.manual_seed(0)
    table = torch.randn(500, 64, device="cuda")
    ids = torch.randint(0, 500, (3, 70), device="cuda")
    w = torch.randn(3, 70, 64, device="cuda")
    wt, it, tt = nb.Tensor.from_torch(w), nb.Tensor.from_torch(ids), nb.Tensor.from_torch(table)
    f = nb.compile(lambda t: nb.grad(lambda a: nb.reduce_sum(F.embedding(it, a) * wt), create_graph=False)(t))
    ref = torch.zeros(500, 64, dtype=torch.float64, device="cuda").index_add_(0, ids.reshape(-1), w.double().reshape(-1, 64))
    for _ in range(2):
        assert _rel2(f(tt).to_torch(), ref) < STORED[torch.float32]
    assert "scatter_zeros" in f.dump_plan()


# ---------------------------------------------------------------- reductions
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape,axis", [((1, 40, 8192), 0), ((5, 37, 8192), 0), ((256, 40, 8192), 0), ((257, 40, 8192), 0), ((3, 6, 128, 1024), 1),
                                        ((4, 300, 1001), 0), ((4095, 16), 0), ((4097, 8), 0), ((70001, 24), 0), ((9000, 248), 0)])
def test_reductions_over_leading_axes(dtype, shape, axis):
    """The kernel for few rows and its neighbours (257 rows, columns that are no whole vectors), and the column
    sums of narrow matrices around the row count where they take over."""
    from nabla_b200.native import kernels

    torch.manual_seed(1)
    x = torch.randn(shape, device="cuda").to(dtype)
    for op, ref in (("sum", x.double().sum(axis)), ("mean", x.double().mean(axis))):
        assert _rel2(kernels.reduce(x, axis, op), ref) < STORED[dtype]
    x.view(-1)[::977] = float("-inf")
    x.view(-1)[5::3001] = float("nan")
    for op, fn in (("max", torch.amax), ("min", torch.amin)):
        torch.testing.assert_close(kernels.reduce(x, axis, op), fn(x, axis), rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape,axis", [((1, 40, 8192), 0), ((7, 40, 8192), 0), ((8, 40, 8192), 0), ((33, 40, 8192), 0), ((256, 40, 8192), 0),
                                        ((5000, 21, 64), 1)])
def test_sums_over_few_rows_in_eight_chains(dtype, shape, axis):
    """Row r adds to chain r % 8 and the chains are joined in order, as in the kernel for longer sums: the
    same fp32 additions one by one."""
    from nabla_b200.native import kernels

    torch.manual_seed(14)
    x = torch.randn(shape, device="cuda").to(dtype)
    rows = x.movedim(axis, 0).float()
    chains = torch.zeros(8, *rows.shape[1:], device="cuda")
    for r, row in enumerate(rows):
        chains[r % 8] += row
    ref = chains[0]
    for c in chains[1:]:
        ref = ref + c
    assert torch.equal(kernels.reduce(x, axis, "sum"), ref.to(dtype))
    assert torch.equal(kernels.reduce(x, axis, "mean"), (ref / torch.full_like(ref, rows.shape[0])).to(dtype))


@pytest.mark.parametrize("axes", [(0, 1), (0, 1, 2), (1, 2), (0, 2), (0, 1, 2, 3)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sums_over_neighbouring_axes(axes, dtype):
    import nabla_b200 as nb

    x = torch.randn(6, 7, 50, 16, device="cuda").to(dtype)
    t = nb.Tensor.from_torch(x)
    for keep in (False, True):
        got = nb.reduce_sum(t, axis=axes, keepdims=keep).to_torch()
        ref = x.double().sum(axes, keepdim=keep)
        assert got.shape == ref.shape and _rel2(got, ref) < len(axes) * STORED[dtype]
    f = nb.compile(lambda a: nb.reduce_sum(a, axis=axes))
    f(t)
    assert _rel2(f(t).to_torch(), x.double().sum(axes)) < len(axes) * STORED[dtype]
    assert ("sum_axes" in f.dump_plan()) == (dtype is torch.bfloat16 and axes in ((0, 1), (0, 1, 2), (1, 2)))


@pytest.mark.parametrize("shape,axes,joined", [((20, 15, 14, 32), (0, 1, 2), True), ((16, 16, 4096), (0, 1), False), ((4, 60, 50, 24), (1, 2), False),
                                               ((64, 65, 128), (0, 1), False), ((2, 64, 65, 16), (0, 1, 2), True)])
def test_joined_sums_round_no_more_than_one_sum_per_axis(shape, axes, joined):
    """fp32: one reduction takes over only where its chains of additions are short (see ``kernels.joined_sum``)."""
    import nabla_b200 as nb
    from nabla_b200.native import kernels

    f = nb.compile(lambda a: nb.reduce_sum(a, axis=axes))
    one = each = 0.0
    for seed in range(8):                             # 8 draws: the error of a sum of few results scatters
        torch.manual_seed(seed)
        x = torch.randn(shape, device="cuda")
        f(nb.Tensor.from_torch(x))
        got, ref = f(nb.Tensor.from_torch(x)).to_torch(), x.double().sum(axes)
        y = x
        for axis in reversed(axes):
            y = kernels.reduce(y, axis, "sum")
        one, each = one + _rel2(got, ref) ** 2, each + _rel2(y, ref) ** 2
    assert one <= 1.1 ** 2 * each
    assert ("sum_axes" in f.dump_plan()) == joined


@pytest.mark.parametrize("args,joined", [((1, 200704, 16, torch.float32), True), ((1, 4096, 16, torch.float32), False), ((1, 1 << 20, 256, torch.bfloat16), False),
                                         ((2, 700000, 8, torch.bfloat16), False), ((1, 16384, 2048, torch.bfloat16), True), ((1, 16, 1 << 20, torch.bfloat16), True)])
def test_rule_of_joined_sums(args, joined):
    from nabla_b200.native import kernels

    assert kernels.joined_sum(*args) == joined


# ---------------------------------------------------------------- launches that follow each other
@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("rows,width", [(64, 128), (1001, 512), (4096, 1024)])
def test_launches_that_start_before_the_one_ahead_has_ended(rows, width, captured):
    """A chain in which every kernel reads what the one ahead of it wrote, in memory that the allocator hands out again at once, and a
    fork and join of two streams: equal, bit for bit, to the same calls with a synchronisation after each."""
    from nabla_b200.native import attention, gemm, kernels

    torch.manual_seed(rows)
    x0 = torch.randn(rows, width, device="cuda").bfloat16()
    w = (torch.randn(width, width, device="cuda") * width ** -0.5).bfloat16()
    g, b = (torch.randn(width, device="cuda").bfloat16() for _ in range(2))
    side = torch.cuda.Stream()

    def chain(between, fork):
        x, sums = x0, []
        for _ in range(12):
            y = kernels.layernorm_fwd(x, g, b, 1e-5)[0]
            between()
            main = torch.cuda.current_stream()
            if fork:
                side.wait_stream(main)
                y.record_stream(side)
            with torch.cuda.stream(side if fork else main):
                z = gemm.gemm_bf16(y, w)
            u = gemm.gemm_bf16(y, w.t())
            if fork:
                main.wait_stream(side)
                z.record_stream(main)
            between()
            h = [t.view(1, rows, width // 64, 64).transpose(1, 2) for t in (u, z, y)]
            o, lse = attention.sdpa_fwd(*h, causal=True, scale=0.125)
            between()
            d = attention.sdpa_bwd(o, *h, o, lse, causal=True, scale=0.125)
            between()
            x = gemm.gemm_bf16(d[0].transpose(1, 2).reshape(rows, width) + o.transpose(1, 2).reshape(rows, width), w)
            sums += [kernels.colsum(x), d[1].sum(), d[2].sum()]
            between()
        return [x, *sums]

    want = chain(torch.cuda.synchronize, False)
    if captured:
        graph = torch.cuda.CUDAGraph()
        chain(lambda: None, True)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            got = chain(lambda: None, True)
        for _ in range(3):
            graph.replay()
    else:
        got = chain(lambda: None, True)
    torch.cuda.synchronize()
    for p, q in zip(got, want):
        assert torch.equal(p, q)


# ---------------------------------------------------------------- attention
def _attention64(q, k, v, causal, mask=None):
    s = q.double() @ k.double().transpose(-1, -2) * q.shape[-1] ** -0.5
    if causal:
        s = s.masked_fill(~torch.ones(s.shape[-2:], dtype=torch.bool, device="cuda").tril(s.shape[-1] - s.shape[-2]), float("-inf"))
    return torch.softmax(s if mask is None else s + mask.double(), -1) @ v.double()


def _attention_check(q, k, v, causal, mask=None, grads=True):
    """Products of bf16 operands with bf16 probabilities: each of the two roundings adds up to 2^-9 relative."""
    from nabla_b200.native import attention

    scale = q.shape[-1] ** -0.5
    o, lse = attention.sdpa_fwd(q, k, v, causal=causal, scale=scale, mask=mask)
    a, b, c = (t.double().requires_grad_(True) for t in (q, k, v))
    ref = _attention64(a, b, c, causal, mask)
    assert _rel2(o, ref) < 6e-3
    if grads:
        do = torch.randn_like(q)
        got = attention.sdpa_bwd(do, q, k, v, o, lse, causal=causal, scale=scale, mask=mask)
        for x, y in zip(got, torch.autograd.grad(ref, (a, b, c), do.double())):
            assert _rel2(x, y) < 8e-3


@pytest.mark.parametrize("B,H,S,D", [(5, 14, 1030, 128), (9, 16, 1030, 64), (1, 1, 129, 128), (3, 1, 2100, 64)])
def test_causal_attention_in_tile_order(B, H, S, D):
    """More (batch, head) pairs than one chunk of the launch order holds (and a last chunk that is not full)."""
    torch.manual_seed(0)
    q, k, v = (torch.randn(B, H, S, D, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    _attention_check(q, k, v, True)


@pytest.mark.parametrize("S,D,causal", [(130, 64, False), (257, 128, False), (777, 64, True), (64, 128, False)])
@pytest.mark.parametrize("shape", ["b11k", "bh1k", "11qk"])
def test_attention_with_additive_masks(S, D, causal, shape):
    """One mask row for all queries (shared memory in the kernels) and one per query, hidden keys as -1e9 and as
    -inf."""
    torch.manual_seed(2)
    B, H = 2, 3
    q, k, v = (torch.randn(B, H, S, D, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    mask = torch.randn({"b11k": (B, 1, 1, S), "bh1k": (B, H, 1, S), "11qk": (1, 1, S, S)}[shape], device="cuda")
    hide = torch.rand(mask.shape, device="cuda") < 0.3
    hide[..., 0] = False                              # every row keeps a key, the causal ones too
    _attention_check(q, k, v, causal, mask.masked_fill(hide, -1e9))
    _attention_check(q, k, v, causal, mask.masked_fill(hide, float("-inf")))


@pytest.mark.parametrize("S,D,causal", [(130, 64, False), (257, 128, False), (777, 64, True), (64, 128, False)])
def test_attention_with_a_large_common_offset_in_the_mask(S, D, causal):
    """One mask row for all queries gives what the same mask with a row per query gives, bit for bit: both add it
    to the scores with one rounding. An offset that all keys share leaves the softmax as it is, but it is
    rounded away from the scores in fp32 and any second rounding shows in the probabilities."""
    from nabla_b200.native import attention

    torch.manual_seed(12)
    B, H = 2, 3
    q, k, v, do = (torch.randn(B, H, S, D, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    for offset in (0.0, -1e4, 65504.0):
        mask = torch.randn(B, 1, 1, S, device="cuda") + offset
        got = []
        for m in (mask, mask.expand(B, 1, S, S).contiguous()):
            o, lse = attention.sdpa_fwd(q, k, v, causal=causal, scale=D ** -0.5, mask=m)
            got.append((o, lse, *attention.sdpa_bwd(do, q, k, v, o, lse, causal=causal, scale=D ** -0.5, mask=m)))
        for a, b in zip(*got):
            assert torch.equal(a, b), offset


@pytest.mark.parametrize("S,D,causal", [(700, 64, False), (700, 64, True), (641, 128, False), (700, 128, True), (384, 64, False)])
def test_attention_with_key_masks_that_are_zero_in_most_tiles(S, D, causal):
    """Tiles without a mask value between tiles with some, tiles that are hidden whole, and one hidden key in the last of a tile
    with a remainder: the kernels leave a mask of zeros out tile by tile."""
    torch.manual_seed(S + D)
    B = 4
    m = torch.zeros(B, 1, 1, S, device="cuda")
    m[0, ..., 256:384] = torch.randn(128, device="cuda")
    m[1, ..., 128:256] = -float("inf")
    m[2, ..., 128:384], m[2, ..., -100:] = -1e9, -float("inf")
    m[3, ..., -1], m[3, ..., 300] = -float("inf"), 2.0
    if not causal:
        m[2, ..., :128] = -float("inf")
        m[2, ..., 200] = 0.0
    q, k, v = (torch.randn(B, 3, S, D, device="cuda").bfloat16() for _ in range(3))
    _attention_check(q, k, v, causal, m)


@pytest.mark.parametrize("D,keys", [(64, False), (64, True), (128, False)])
def test_attention_over_key_ranges_that_one_of_two_query_tiles_sees(D, keys):
    """256 queries over 2048 keys in ranges of one key tile: of the last range the first 128 queries see nothing."""
    from nabla_b200.native import attention

    torch.manual_seed(D)
    attention._lib()
    assert attention._splits(1, 2, 256, 2048, D, int(keys)) == 16
    q, k, v = (torch.randn(1, 2, s, D, device="cuda").bfloat16() for s in (256, 2048, 2048))
    m = None
    if keys:
        m = torch.zeros(1, 1, 1, 2048, device="cuda")
        m[..., 700:900], m[..., 2000:] = -float("inf"), 0.5
    _attention_check(q, k, v, True, m)


@pytest.mark.parametrize("D", [64, 128])
def test_attention_gradients_into_rows_on_16_byte_boundaries(D):
    """Results whose rows start on 16- and not on 32-byte boundaries are the bits of aligned ones, and nothing beside them is written."""
    from nabla_b200.native import attention

    torch.manual_seed(0)
    B, H, S = 2, 3, 200
    q, k, v, do = (torch.randn(B, H, S, D, device="cuda").bfloat16() for _ in range(4))
    o, lse = attention.sdpa_fwd(q, k, v, causal=True, scale=0.1)
    want = attention.sdpa_bwd(do, q, k, v, o, lse, causal=True, scale=0.1)
    bufs = [torch.zeros(B * S * H * (D + 8) + 8, device="cuda", dtype=torch.bfloat16)[8:].view(B, S, H, D + 8) for _ in range(3)]
    out = tuple(t[..., :D].permute(0, 2, 1, 3) for t in bufs)
    assert all(t.data_ptr() % 32 == 16 and t.stride(2) % 16 == 8 for t in out)
    attention.sdpa_bwd(do, q, k, v, o, lse, causal=True, scale=0.1, out=out)
    for got, ref, t in zip(out, want, bufs):
        assert torch.equal(got, ref) and not t[..., D:].any()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("S,D", [(130, 64), (300, 128)])
def test_attention_hides_a_masked_key_that_is_not_finite(S, D, value):
    """Causal: rows before a key never see its mask value, whatever it is; with a row per query the same."""
    from nabla_b200.native import attention

    torch.manual_seed(13)
    q, k, v, do = (torch.randn(1, 2, S, D, device="cuda", dtype=torch.bfloat16) for _ in range(4))
    mask = torch.randn(1, 1, 1, S, device="cuda")
    mask[..., S - 20] = value
    got = []
    for m in (mask, mask.expand(1, 1, S, S).contiguous()):
        o, lse = attention.sdpa_fwd(q, k, v, causal=True, scale=D ** -0.5, mask=m)
        dq, _, _ = attention.sdpa_bwd(do, q, k, v, o, lse, causal=True, scale=D ** -0.5, mask=m)
        assert bool(torch.isfinite(o[:, :, :S - 20]).all()) and bool(torch.isfinite(dq[:, :, :S - 20]).all())
        got.append((o, lse, dq))
    for a, b in zip(*got):
        assert torch.equal(a[:, :, :S - 20], b[:, :, :S - 20])


def test_attention_rows_without_a_visible_key_are_zero():
    from nabla_b200.native import attention

    q, k, v = (torch.randn(2, 2, 150, 64, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    mask = torch.zeros(2, 1, 1, 150, device="cuda")
    mask[1] = float("-inf")
    o, lse = attention.sdpa_fwd(q, k, v, causal=False, scale=0.125, mask=mask)
    assert bool((o[1] == 0).all()) and bool((lse[1] == float("-inf")).all()) and bool(torch.isfinite(lse[0]).all())
    for g in attention.sdpa_bwd(torch.randn_like(q), q, k, v, o, lse, causal=False, scale=0.125, mask=mask):
        assert bool(torch.isfinite(g).all()) and bool((g[1] == 0).all())


# ---------------------------------------------------------------- layer norm backward
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,vectors", [(1, 32), (5, 33), (2, 64), (1000, 65), (3, 96), (777, 125), (4, 128), (9, 160), (300, 224), (6, 256), (5000, 256),
                                          (2, 257), (33, 512)])
def test_layer_norm_backward_by_row_width(dtype, rows, vectors):
    """One warp per row, 2 to 16 warps per row with one or several rows per block, last warps that are partly
    idle, fewer rows than a block holds and many times the grid."""
    from nabla_b200.native import kernels

    D = vectors * (8 if dtype is torch.bfloat16 else 4)
    torch.manual_seed(4)
    x, dy = (torch.randn(rows, D, device="cuda").add_(0.5).to(dtype) for _ in range(2))
    for g in (torch.randn(D, device="cuda").to(dtype), None):
        _, mean, rstd = kernels.layernorm_fwd(x, g, None, 1e-5)
        got = kernels.layernorm_bwd(dy, x, g, mean, rstd)
        a, b, c = x.double().requires_grad_(True), (torch.ones(D, device="cuda") if g is None else g).double().requires_grad_(True), \
            torch.zeros(D, dtype=torch.float64, device="cuda").requires_grad_(True)
        ref = torch.autograd.grad(TF.layer_norm(a, (D,), b, c, 1e-5), (a, b, c), dy.double())
        for y, r in zip(got, ref):
            assert _rel2(y, r) < STORED[dtype]


# ---------------------------------------------------------------- copies around a captured step
def test_copy_batch_moves_every_size_alignment_and_type():
    from nabla_b200.native import kernels

    torch.manual_seed(5)
    pool = torch.randint(0, 255, (1 << 20,), dtype=torch.uint8, device="cuda")
    src = [pool[o:o + n] for o in (0, 1, 2, 3, 4, 8, 16) for n in (0, 1, 2, 3, 15, 16, 17, 4095, 32768, 32769, 100001)]
    src += [torch.randn(n, device="cuda") for n in (1, 7, 300)] + [torch.randn(5, 9, device="cuda", dtype=torch.bfloat16).t() for _ in range(70)]
    src += [torch.randn(6, 8, device="cuda")[:, :5], torch.tensor(3.0), torch.arange(4, device="cuda")]
    fixed = [torch.empty_like(t) for t in src]
    assert len(src) > 128
    batch = kernels.CopyBatch(fixed)
    for _ in range(2):
        batch.run(src, into_fixed=True)
        assert all(torch.equal(a, b) for a, b in zip(src, fixed))
        src = [t if t.dtype is not torch.float32 else t + 1 for t in src]
    out = [torch.empty_like(t) for t in fixed]
    batch.run(out, into_fixed=False)
    assert all(torch.equal(a, b) for a, b in zip(out, fixed))


def test_copy_batch_reads_before_it_writes_where_pairs_share_memory():
    from nabla_b200.native import kernels

    a, b = torch.zeros(8, device="cuda"), torch.ones(8, device="cuda")
    kernels.CopyBatch([a, b], shared=True).run([b, a], into_fixed=True)
    assert bool((a == 1).all()) and bool((b == 0).all())
    c = torch.arange(12.0, device="cuda").view(3, 4)
    d = torch.zeros(4, device="cuda")
    kernels.CopyBatch([c, d], shared=True).run([torch.full((3, 4), 5.0, device="cuda"), c[1]], into_fixed=True)   # a view of another pair
    assert bool((c == 5).all()) and d.tolist() == [4.0, 5.0, 6.0, 7.0]


def test_copy_batch_without_native_kernels(monkeypatch):
    from nabla_b200.native import kernels

    monkeypatch.setenv("NABLA_B200_DISABLE_NATIVE", "1")
    fixed, src = [torch.zeros(9, device="cuda") for _ in range(3)], [torch.randn(9, device="cuda") for _ in range(3)]
    n = kernels.launch_count
    kernels.CopyBatch(fixed).run(src, into_fixed=True)
    assert kernels.launch_count == n and all(torch.equal(a, b) for a, b in zip(fixed, src))


@pytest.mark.parametrize("order", [(1, 0, 2), (1, 2, 0), (0, 1, 2)])
def test_captured_function_whose_donated_results_come_back_in_other_places(order):
    import nabla_b200 as nb

    def step(x, y, z):
        return x, y, z, x * 2.0 + y          # the first three live in the donated buffers

    start = [torch.randn(40, device="cuda") for _ in range(3)]
    got = {}
    for graph in (False, True):
        f = nb.compile(step, cuda_graph=graph, donate_argnums=(0, 1, 2))
        state, seen = [nb.Tensor.from_torch(t.clone()) for t in start], []
        for _ in range(5):
            *out, extra = f(*state)
            seen.append(extra.to_torch().clone())
            state = [out[i] for i in order]
        got[graph] = seen + [t.to_torch().clone() for t in state]
    for a, b in zip(got[True], got[False]):
        assert torch.equal(a, b)


def test_captured_function_with_odd_inputs():
    """Views, a CPU scalar, an input returned as it is and one returned twice, and results that stay valid."""
    import nabla_b200 as nb

    f = nb.compile(lambda x, y, s, c: (x @ y, x, nb.relu(y), y + s, y, y, c), cuda_graph=True)
    first = None
    for i in range(4):
        x = torch.randn(33, 40, device="cuda").t()[:, :17]
        y = torch.randn(17, 24, device="cuda")[:, ::2]
        s = torch.randn(12, device="cuda")
        c = torch.tensor(float(i))                     # stays on the CPU
        out = [t.to_torch() for t in f(*(nb.Tensor.from_torch(t) for t in (x, y, s, c)))]
        assert out[6].device.type == "cpu"
        for got, ref in zip(out, (x @ y, x, y.relu(), y + s, y, y, c)):
            torch.testing.assert_close(got, ref, rtol=1e-4, atol=1e-4)
        if first is not None:
            assert torch.equal(first[0], first[1])
        first = (out[1], x)


# ---------------------------------------------------------------- NF4
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,block,offset", [(1, 64, 0), (16, 16, 0), (1000, 64, 0), (4096, 128, 0), (4113, 10, 0), (4096, 64, 3), (70000, 48, 0)])
def test_nf4_codes(dtype, n, block, offset):
    from nabla_b200.native import kernels

    torch.manual_seed(6)
    codes = torch.randint(0, 16, (n + offset,), device="cuda", dtype=torch.uint8)[offset:]
    scales = torch.rand((n + block - 1) // block, device="cuda") + 0.01
    book = torch.linspace(-1, 1, 16, device="cuda")
    got = kernels.nf4_dequant_codes(codes, scales, book, n, block, dtype)
    assert torch.equal(got, (book[codes.long()] * scales.repeat_interleave(block)[:n]).to(dtype))


# ---------------------------------------------------------------- cross-entropy rows
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,D,offset", [(3, 1, 0), (5, 7, 0), (4, 8, 0), (9, 33, 0), (4, 255, 0), (4, 256, 0), (4, 257, 0), (6, 1000, 0), (7, 2051, 0),
                                           (3, 10001, 0), (2, 32000, 0), (6, 1000, 1), (5, 256, 3), (4, 64, 8)])
def test_logsumexp_and_gradient_at_any_row_alignment(dtype, rows, D, offset):
    """Whole aligned vectors, an element per thread, and vectors between edges; logits that start inside a vector."""
    from nabla_b200.native import kernels

    torch.manual_seed(7)
    x = torch.empty(rows * D + offset, device="cuda", dtype=dtype)[offset:].view(rows, D)
    x.copy_(torch.randn(rows, D, device="cuda") * 3)
    x[0, D // 3: D // 3 + 20] = float("-inf")          # masked classes, here and there a whole vector of them
    if D > 1:
        x[0, D - 1] = 1.0
    t = torch.randint(-1, D + 1, (rows,), device="cuda")
    lse, picked = kernels.lse_pick_fwd(x, t)
    torch.testing.assert_close(lse.double(), torch.logsumexp(x.double(), -1), rtol=1e-5, atol=1e-5)
    ok = (t >= 0) & (t < D)
    assert torch.equal(picked, torch.where(ok, x.float().gather(1, t.clamp(0, D - 1)[:, None])[:, 0], torch.zeros((), device="cuda")))
    gl, gp = torch.rand(rows, device="cuda"), torch.randn(rows, device="cuda")
    safe = torch.where(lse == float("-inf"), torch.zeros_like(lse), lse)
    ref = torch.exp(x.double() - safe.double()[:, None]) * gl.double()[:, None]
    ref[ok] = ref[ok].scatter_add(1, t[ok][:, None], gp.double()[ok][:, None])
    assert _rel2(kernels.lse_pick_bwd(x, t, safe, gl, gp), ref) < STORED[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [5, 256, 1001, 4096])
def test_logsumexp_of_rows_at_the_ends_of_the_range(dtype, D):
    """Rows of -inf, of the type's lowest value, of -inf but for the lowest or for one element, with +inf and NaN."""
    from nabla_b200.native import kernels

    low, inf = torch.finfo(dtype).min, float("inf")
    x = torch.full((7, D), -inf, device="cuda", dtype=dtype)
    x[1] = low
    x[2, D // 2] = low
    x[3, D - 1] = -3.0
    x[4] = 1.0
    x[4, D // 3] = inf
    x[5] = 1.0
    x[5, 0] = float("nan")
    x[6] = torch.finfo(dtype).max / 4
    lse, _ = kernels.lse_pick_fwd(x, torch.zeros(7, dtype=torch.int64, device="cuda"))
    ref = torch.logsumexp(x.double(), -1)
    assert lse[0] == -inf and not bool(torch.isfinite(lse[4])) and bool(torch.isnan(lse[5]))
    torch.testing.assert_close(lse[[1, 2, 3, 6]].double(), ref[[1, 2, 3, 6]], rtol=1e-5, atol=1e-5)


# ---------------------------------------------------------------- GEMM rows that are not 16-byte aligned
@pytest.mark.parametrize("M,N,K", [(1, 1, 64), (130, 33, 72), (257, 77, 200), (100, 255, 64), (300, 513, 128), (4097, 1001, 264), (5000, 4999, 64)])
def test_gemm_with_odd_output_rows(M, N, K):
    from nabla_b200.native import gemm

    torch.manual_seed(8)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16) * 0.1
    bias = torch.randn(N, device="cuda", dtype=torch.bfloat16)
    z = a.double() @ b.double() + bias.double()
    assert _rel2(gemm.gemm_bf16(a, b), a.double() @ b.double()) < STORED[torch.bfloat16]
    assert _rel2(gemm.gemm_bf16(a, b, bias=bias, epilogue="relu"), z.relu()) < STORED[torch.bfloat16]
    y, pre = gemm.gemm_bf16(a, b, bias=bias, epilogue="gelu", aux="store_preact")
    assert _rel2(pre, z) < STORED[torch.bfloat16] and _rel2(y, TF.gelu(z)) < STORED[torch.bfloat16]
    three = gemm.gemm_bf16(torch.stack([a, a * 2]), torch.stack([b, b]))
    assert _rel2(three[1], 2 * (a.double() @ b.double())) < STORED[torch.bfloat16]
    guard = torch.full((M, N + 3), 7.0, device="cuda", dtype=torch.bfloat16)      # rows with another stride: nothing beside them
    gemm.gemm_bf16(a, b, out=guard[:, 1:1 + N])
    assert _rel2(guard[:, 1:1 + N], a.double() @ b.double()) < STORED[torch.bfloat16]
    assert bool((guard[:, 0] == 7).all()) and bool((guard[:, 1 + N:] == 7).all())


# ---------------------------------------------------------------- GEMM operands of one row or column
def test_gemm_operands_of_one_row_or_column():
    from nabla_b200.native import gemm

    torch.manual_seed(11)
    for M, N, K in ((512, 1, 256), (1, 300, 77), (1, 1, 9), (300, 40, 1), (256, 1, 513), (1, 2056, 4096)):
        for ta in (False, True):
            for tb in (False, True):
                a = torch.randn(K, M, device="cuda", dtype=torch.bfloat16).t() if ta else torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
                b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16).t() if tb else torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
                assert _rel2(gemm.gemm_bf16(a, b), a.double() @ b.double()) < STORED[torch.bfloat16]


# ---------------------------------------------------------------- AdamW bias corrections
def test_adam_hyper_counts_its_step():
    from nabla_b200.native import kernels

    for t in (0.0, 1.0, 999.0):
        s, h = kernels.adam_hyper(torch.tensor(t, device="cuda"), 1e-3, 0.9, 0.999, plus=torch.tensor(1.0, device="cuda"))
        assert s.item() == t + 1 and torch.equal(h, kernels.adam_hyper(s, 1e-3, 0.9, 0.999))


def test_adam_hyper():
    from nabla_b200.native import kernels

    for t in (1.0, 2.0, 101.0, 12345.0):
        got = kernels.adam_hyper(torch.tensor(t, device="cuda"), 1e-3, 0.9, 0.999).double().tolist()
        for a, b in zip(got, (1e-3, 1 - 0.9 ** t, 1 - 0.999 ** t, 1.0)):
            assert abs(a - b) <= 1e-7 * abs(b)


@pytest.mark.parametrize("p_dtype,g_dtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_small_adamw_updates_in_one_launch(p_dtype, g_dtype):
    """More tensors than a launch holds, sizes around a block's 2048 elements and the eight of a thread: the bits of one launch
    each, in place or not; a misaligned tensor is refused."""
    from nabla_b200.native import kernels

    torch.manual_seed(0)
    sizes = [1, 7, 8, 9, 2047, 2048, 2049, 4096, 65537, 1 << 18] + list(range(11, 56))
    mk = lambda n, dt: torch.randn(n, device="cuda").to(dt)  # noqa: E731
    leaves = [(mk(n, p_dtype), mk(n, g_dtype), mk(n, torch.float32), mk(n, torch.float32).abs()) for n in sizes]
    hyper = kernels.adam_hyper(torch.tensor(7.0, device="cuda"), 1e-3, 0.9, 0.999)
    kw = dict(lr=1e-3, b1=0.9, b2=0.999, eps=1e-8, wd=0.01)
    for extra in ({"hyper": hyper}, {"step": 7}, {}):
        ref = [kernels.adamw(*leaf, **kw, **extra) for leaf in leaves]
        flags = [i % 2 == 0 for i in range(len(sizes))]
        mine = [tuple(t.clone() for t in leaf) for leaf in leaves]
        got = kernels.adamw_group([(*leaf, f) for leaf, f in zip(mine, flags)], **kw, **extra)
        for r, g, leaf, old, f in zip(ref, got, mine, leaves, flags):
            assert all(torch.equal(a, b) for a, b in zip(r, g))
            assert (g[0].data_ptr() == leaf[0].data_ptr()) == f and (f or torch.equal(leaf[0], old[0]))
    odd = mk(17, torch.float32)[1:]
    assert kernels.adamw_group([(mk(16, p_dtype), mk(16, g_dtype), odd, odd.clone(), False)], **kw) is None


@pytest.mark.parametrize("fault", ["alignment", "size"])
def test_a_group_that_is_refused_updates_nothing(fault):
    """The last of 49 tensors, which a second launch would take, is one that the entry point refuses."""
    import ctypes

    from nabla_b200.native import kernels, ptr, stream_ptr

    n = 49
    leaves = [[torch.full((16,), 0.5, device="cuda") for _ in range(4)] for _ in range(n)]
    sizes = [8] * (n - 1) + [(1 << 20) + 1 if fault == "size" else 8]
    cols = [[t[i].data_ptr() for t in leaves] for i in range(4)]
    if fault == "alignment":
        cols[1][-1] += 4
    arr = [(ctypes.c_void_p * n)(*c) for c in cols + [cols[0], cols[2], cols[3]]]
    rc = kernels._L().nb_adamw_group(*arr, (ctypes.c_int * n)(*sizes), n, 0.1, 0.9, 0.99, 1e-8, 0.0, 0.1, 0.01, 1.0, ptr(None), 0, 0, stream_ptr())
    torch.cuda.synchronize()
    assert rc == -2 and all(bool((t == 0.5).all()) for leaf in leaves for t in leaf)


@pytest.mark.parametrize("donate", [False, True])
def test_compiled_step_groups_its_small_updates(donate):
    import nabla_b200 as nb
    from nabla_b200 import nn

    torch.manual_seed(0)
    shapes = {"a": (64, 40), "b": (40,), "big": (600, 512), "c": (3,), "d": (512, 512)}
    wrap = lambda d: {k: nb.Tensor.from_torch(v.clone()) for k, v in d.items()}  # noqa: E731
    p = {k: torch.randn(v, device="cuda") for k, v in shapes.items()}
    g = {k: torch.randn(v, device="cuda") for k, v in shapes.items()}
    z = {k: torch.zeros(v, device="cuda") for k, v in shapes.items()}

    def step(params, state, grads):
        return nn.adamw_update(params, grads, state, lr=1e-2, weight_decay=0.1, realize=False)

    f = nb.compile(step, cuda_graph=True, donate_argnums=(0, 1) if donate else ())
    new, st = wrap(p), {"m": wrap(z), "v": wrap(z), "step": nb.Tensor.from_torch(torch.tensor(0.0, device="cuda"))}
    ref = {k: v.double() for k, v in p.items()}
    m = {k: v.double() for k, v in z.items()}
    v2 = {k: v.double() for k, v in z.items()}
    for t in range(1, 5):
        new, st = f(new, st, wrap(g))
        for k in p:
            m[k] = 0.9 * m[k] + 0.1 * g[k].double()
            v2[k] = 0.999 * v2[k] + 0.001 * g[k].double() ** 2
            ref[k] = ref[k] - 1e-2 * ((m[k] / (1 - 0.9 ** t)) / ((v2[k] / (1 - 0.999 ** t)).sqrt() + 1e-8) + 0.1 * ref[k])
            assert _rel2(new[k].to_torch(), ref[k]) < t * STORED[torch.float32]      # a rounding of p, m and v per step
    assert sum("adamw_group" in line for line in str(f.dump_plan()).splitlines()) == 1


# ---------------------------------------------------------------- means of a difference
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n", [1, 31, 1025, 4096, 4097, 70001, 1 << 18])
def test_mean_of_a_difference_and_of_its_square(dtype, n):
    from nabla_b200.native import kernels

    torch.manual_seed(23)
    a, b = (torch.randn(n, device="cuda").to(dtype) for _ in range(2))
    for square in (False, True):
        for count in (n, torch.tensor(float(n), device="cuda", dtype=dtype)):
            d, m = kernels.mean_diff(a, b, square, count)
            assert torch.equal(d, a - b)
            terms = d.double() ** 2 if square else d.double()
            c = float(count)
            # fp32: the additions of a thread, a warp, a block and a cluster, each rounded to the sum of magnitudes at most
            bound = (n / 1024 / 8 + 20) * 2.0 ** -24 * terms.abs().sum() / c
            assert abs(m.double() - terms.sum() / c) <= bound + abs(terms.sum() / c) * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22)
    x = torch.tensor([1.0, float("nan"), 3.0], device="cuda").to(dtype)
    assert kernels.mean_diff(x, torch.zeros_like(x), True, 3)[1].isnan()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_compiled_losses_in_one_launch(dtype):
    """Squared error and cross-entropy with their gradients: compiled against plain calls, twice, and what the plan made of them."""
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    torch.manual_seed(24)
    x, y = torch.randn(33, 40, device="cuda").to(dtype), torch.randn(33, 40, device="cuda").to(dtype)
    t = torch.randint(0, 40, (33,), device="cuda")
    wrap = nb.Tensor.from_torch
    for loss, other, steps in ((F.mse_loss, y, ("mean_diff", "twice_product")), (F.cross_entropy_loss, t, ("mean_diff",))):
        f = nb.compile(lambda a, b, loss=loss: nb.value_and_grad(loss, create_graph=False)(a, b))
        for k in range(2):
            arg = (x * (k + 1)).contiguous()
            v, g = f(wrap(arg), wrap(other))
            p = arg.double().requires_grad_(True)
            ref = ((p - other.double()) ** 2).mean() if loss is F.mse_loss else TF.cross_entropy(p, other)
            ref.backward()
            assert _rel2(v.to_torch(), ref.detach()) < STORED[dtype] and _rel2(g.to_torch(), p.grad) < 3 * STORED[dtype]
        plan = f.dump_plan()
        assert all(sum(s in line for line in plan.splitlines()) == 1 for s in steps)
        assert " full" not in plan and "broadcast_to" not in plan              # made with the plan
    # a result that would be the constant itself is made on each call
    f = nb.compile(lambda a: (nb.broadcast_to(nb.reshape(nb.full((), 2.0, device=a.device), (1,)), (4,)), a + 1.0))
    for _ in range(2):
        c, _ = f(wrap(x))
        assert c.to_torch().tolist() == [2.0] * 4
        c.to_torch().zero_() if c.to_torch().is_contiguous() else None


# ---------------------------------------------------------------- column sums
def test_column_sums_around_the_slab_counts():
    from nabla_b200.native import kernels

    torch.manual_seed(10)
    for rows, N in ((1, 8), (63, 512), (64, 512), (65, 256), (512, 256), (2002, 1536), (16384, 264), (5000, 8192)):
        for dtype in (torch.bfloat16, torch.float32):
            x = torch.randn(rows, N, device="cuda").to(dtype)
            assert _rel2(kernels.colsum(x), x.double().sum(0)) < STORED[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_column_sums_by_clusters(dtype):
    """Rows around the slots of a cluster (64 and 256) and eight of them, columns around a tile, odd widths and bases; each alone
    and all in one launch."""
    from nabla_b200.native import kernels

    torch.manual_seed(21)
    v = 16 // dtype.itemsize
    xs = []
    for rows, N, off in ((1, v, 0), (255, 8 * v, 0), (257, 8 * v + v, 0), (512, 1, 0), (2047, 10, 0), (2049, 77, 0), (513, 32 * v, 0),
                         (100, 8 * v, 3), (4097, 1000, 0), (8191, 3, 1), (300, 2048 + v, 0)):
        xs.append((torch.randn(rows * N + off, device="cuda").to(dtype))[off:].view(rows, N))
    for wide in (False, True):
        for x, s in zip(xs, kernels.colsum_group(xs, torch.float32, wide)):
            assert _rel2(s, x.double().sum(0)) < STORED[torch.float32]
    for x, s in zip(xs, kernels.colsum_group(xs * 4)[:len(xs)]):          # more than one launch holds
        assert s.dtype == dtype and _rel2(s, x.double().sum(0)) < STORED[dtype]


def test_compiled_bias_gradients_of_a_step_share_a_launch():
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    torch.manual_seed(22)
    x, w1, b1, w2, b2, dy = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((200, 72), (72, 136), (136,), (136, 9), (9,), (200, 9)))

    def step(x, w1, b1, w2, b2, dy):
        y, pull = nb.vjp(lambda *a: F.linear(F.linear(*a[:3], activation="relu"), *a[3:]), x, w1, b1, w2, b2, create_graph=False)
        return (y, *pull(dy))

    f = nb.compile(step)
    got = [[t.to_torch() for t in f(*(nb.Tensor.from_torch(t) for t in (x, w1, b1, w2, b2, dy)))] for _ in range(2)]
    assert sum("bias_grads" in line for line in f.dump_plan().splitlines()) == 1
    plain = [t.to_torch() for t in step(*(nb.Tensor.from_torch(t) for t in (x, w1, b1, w2, b2, dy)))]
    for a, b, c in zip(*got, plain):
        assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("rows,N", [(4096, 8), (4099, 124), (12544, 48), (50176, 32), (200704, 16), (700001, 120)])
def test_narrow_column_sums_are_short_chains(rows, N):
    """The additions one by one: a slab's rows to the slots of a block, the slots in eight sums and in pairs, the slabs to
    8 or 32 warps and in a tree. No chain is longer than a slot's rows or rpp / 8 or 18."""
    from nabla_b200.native import kernels

    torch.manual_seed(16)
    x = torch.randn(rows, N, device="cuda")

    def chain(t):                                     # one after the other over dim 0
        acc = torch.zeros(t.shape[1:], device="cuda")
        for row in t:
            acc = acc + row
        return acc

    def slots(t, n):                                  # (k, ...) -> (steps, n, ...), zeros behind the last
        pad = torch.zeros(-t.shape[0] % n, *t.shape[1:], device="cuda")
        return torch.cat([t, pad]).view(-1, n, *t.shape[1:])

    def sum8(a):
        return ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]))

    parts = kernels._L().nb_colsum_nparts(rows, N, 0)
    per, rpp = -(-rows // parts), 256 // (N // 4)
    slabs = []
    for b in range(parts):
        a = chain(slots(x[b * per:(b + 1) * per], rpp))
        eight = chain(a[:rpp // 8 * 8].view(-1, 8, N)) if rpp >= 8 else torch.zeros(8, N, device="cuda")
        eight[0] = eight[0] + chain(a[rpp // 8 * 8:]) if rpp % 8 else eight[0] + 0.0
        slabs.append(sum8(eight))
    slabs = torch.stack(slabs)
    if parts < 64:
        ref = sum8(chain(slots(slabs, 8)))
    else:
        ref = chain(slots(slabs, 32))
        for o in (16, 8, 4, 2, 1):
            ref = ref + ref[torch.arange(32, device="cuda") ^ o]
        ref = ref[0]
    assert torch.equal(kernels.colsum(x), ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,inner", [(200, 5), (192, 3), (700, 7), (128, 33)])
def test_reductions_in_an_odd_number_of_parts(dtype, rows, inner):
    """An odd number of partial results: their positions, 8 bytes each, lie behind them in the scratch."""
    from nabla_b200.native import kernels

    torch.manual_seed(31)
    x = torch.randn(rows, inner, device="cuda").to(dtype)
    assert _rel2(kernels.reduce(x, 0, "sum"), x.double().sum(0)) < STORED[dtype]
    assert torch.equal(kernels.reduce(x, 0, "max"), x.amax(0)) and torch.equal(kernels.reduce(x, 0, "argmax"), x.argmax(0))


# ---------------------------------------------------------------- pooling
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mode", ["max", "avg"])
@pytest.mark.parametrize("N,H,W,C,k,s,p", [(2, 8, 8, 16, (2, 2), (2, 2), 0), (1, 7, 9, 8, (2, 2), (2, 2), 0), (3, 5, 11, 24, (1, 2), (2, 3), 0), (2, 9, 9, 8, (3, 3), (3, 3), 0),
                                           (1, 2, 2, 8, (2, 2), (5, 4), 0), (2, 6, 6, 12, (2, 2), (2, 2), 0), (2, 6, 6, 5, (2, 2), (2, 2), 0),
                                           (2, 8, 8, 8, (3, 3), (2, 2), 0), (2, 8, 8, 8, (2, 2), (2, 2), 1),
                                           (2, 20, 20, 8, (20, 20), (20, 20), 0), (3, 11, 13, 16, (11, 13), (40, 50), 0), (64, 7, 7, 128, (7, 7), (7, 7), 0),
                                           (16, 9, 14, 256, (4, 7), (4, 7), 0)])
def test_pooling_cells(dtype, mode, N, H, W, C, k, s, p):
    """Windows that do not overlap (whole images and ragged edges, strides wider than the window) and the sizes
    beside the rule; ties go to the first maximum, a window of -inf routes nothing."""
    from nabla_b200.native import kernels

    torch.manual_seed(9)
    x = torch.randint(-3, 4, (N, H, W, C), device="cuda").to(dtype)
    x[0, :k[0], :k[1], 0] = float("-inf") if mode == "max" and p == 0 else 0.0
    y = kernels.pool2d_fwd(x, *k, *s, p, p, mode)
    xr = x.double().permute(0, 3, 1, 2).requires_grad_(True)
    xp = TF.pad(xr, (p, p, p, p), value=float("-inf") if mode == "max" else 0.0)
    ref = TF.max_pool2d(xp, k, s) if mode == "max" else TF.avg_pool2d(xp, k, s)
    torch.testing.assert_close(y.double(), ref.permute(0, 2, 3, 1), rtol=2.0 ** -8, atol=0)
    dy = torch.randn(y.shape, device="cuda").to(dtype)
    if mode == "max" and p == 0:
        dy[0, 0, 0, 0] = 0.0                           # torch routes a window of -inf to its first element
    (g,) = torch.autograd.grad(ref, xr, dy.double().permute(0, 3, 1, 2))
    torch.testing.assert_close(kernels.pool2d_bwd(x, dy, *k, *s, p, p, mode).double(), g.permute(0, 2, 3, 1), rtol=2.0 ** -7, atol=1e-6)


def test_average_pooling_over_few_large_windows_uses_a_thread_per_pixel():
    """The gradient of global average pooling is one load and one store per pixel. Against the gradient of max
    pooling over the same windows, which threads walk whole cells for, it takes a 19th by pixels and a 4th by cells
    (20, 92 and 395 us); the line is between the two."""
    from nabla_b200.native import kernels

    x = torch.randn(8, 56, 56, 64, device="cuda")
    dy = torch.randn(8, 1, 1, 64, device="cuda")

    def fastest(mode):
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(200000)                  # both events and the launch are queued before the first runs
            a.record()
            kernels.pool2d_bwd(x, dy, 56, 56, 56, 56, 0, 0, mode)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert 9 * fastest("avg") < fastest("max")


# ---------------------------------------------------------------- compiled calls
def test_compiled_calls_that_change_between_calls():
    """The path for a call like the one before it: other shapes, types, structures and deterministic mode in
    between, and two threads on one function."""
    import threading

    import nabla_b200 as nb
    from nabla_b200 import config

    f = nb.compile(lambda d, x: {"y": d["w"] * x + d["b"], "n": x})

    def call(n, dtype, extra=False):
        w, b, x = (torch.randn(n, device="cuda").to(dtype) for _ in range(3))
        d = {"w": nb.Tensor.from_torch(w), "b": nb.Tensor.from_torch(b)}
        if extra:
            d["unused"] = nb.Tensor.from_torch(x)
        out = f(d, nb.Tensor.from_torch(x))
        torch.testing.assert_close(out["y"].to_torch().float(), (w * x + b).float(), rtol=2e-2, atol=2e-2)
        assert torch.equal(out["n"].to_torch(), x)

    for args in [(8, torch.float32), (8, torch.float32), (16, torch.float32), (16, torch.bfloat16), (16, torch.bfloat16), (8, torch.float32),
                 (8, torch.float32, True), (8, torch.float32)] * 2:
        call(*args)
    misses = f.stats.misses
    with config.deterministic():
        call(8, torch.float32)
    assert f.stats.misses == misses + 1
    f.clear_cache()
    call(8, torch.float32)
    assert f.stats.misses == misses + 2
    errors = []

    def worker(n):
        try:
            for _ in range(20):
                call(n, torch.float32)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    for n in (8, 16):
        call(n, torch.float32)
    threads = [threading.Thread(target=worker, args=(n,)) for n in (8, 16)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Sq,Skv", [(2, 148, 128, 128), (2, 74, 129, 200), (3, 37, 300, 300), (3, 37, 300, 400), (2, 37, 512, 512), (2, 16, 1030, 1030)])
def test_attention_with_one_and_two_query_tiles_per_block(B, H, Sq, Skv, D):
    """A batch of more tiles than SMs (blocks of two) and each of its items alone (blocks of one) are equal bit for bit."""
    from nabla_b200.native import attention

    torch.manual_seed(Sq)
    q = torch.randn(B, H, Sq, D, device="cuda").bfloat16()
    k, v = (torch.randn(B, H, Skv, D, device="cuda").bfloat16() for _ in range(2))
    keys = torch.randn(B, 1, 1, Skv, device="cuda")
    keys[..., 1::3] = -float("inf")
    for causal in (False, True):
        for m in (None, keys, keys + torch.randn(B, 1, Sq, Skv, device="cuda")):
            o, lse = attention.sdpa_fwd(q, k, v, causal=causal, scale=D ** -0.5, mask=m)
            for b in range(B):
                one = attention.sdpa_fwd(*(t[b:b + 1] for t in (q, k, v)), causal=causal, scale=D ** -0.5, mask=None if m is None else m[b:b + 1])
                assert torch.equal(o[b:b + 1], one[0]) and torch.equal(lse[b:b + 1], one[1])
    _attention_check(q[:, :3], k[:, :3], v[:, :3], True, keys, grads=False)


@pytest.mark.parametrize("D", [64, 128])
def test_attention_over_key_ranges_with_two_query_tiles_per_block(D):
    """Ranges of three key tiles and one: of the last the first 128 queries of a block see nothing."""
    from nabla_b200.native import attention

    attention._lib()
    assert attention._splits(1, 40, 256, 896, D, 0) == 3
    torch.manual_seed(D)
    _attention_check(*(torch.randn(1, 40, s, D, device="cuda").bfloat16() for s in (256, 896, 896)), True, grads=False)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,H,Sq,Skv", [(1, 1, 1, 1), (2, 3, 1, 31), (1, 2, 2, 127), (1, 2, 3, 128), (2, 1, 4, 257), (1, 4, 1, 4001), (3, 5, 4, 700),
                                        (40, 16, 1, 300), (1, 1, 5, 4000), (2, 4, 33, 2500), (1, 2, 130, 1500), (1, 1, 300, 3000)])
def test_attention_of_few_queries_over_a_long_prefix(B, H, Sq, Skv, D):
    """The decode kernel (up to 4 queries), one key range and many, and the split of the tile kernel; keys and
    values as slices of a longer cache."""
    torch.manual_seed(3)
    q = torch.randn(B, H, Sq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, H, Skv + 8, D, device="cuda", dtype=torch.bfloat16)[:, :, 5:5 + Skv] for _ in range(2))
    for causal in ([False, True] if Sq <= Skv else [False]):
        _attention_check(q, k, v, causal, grads=1 < Skv and Sq * Skv < 100000)    # (one key: the score gradients are 0)


@pytest.mark.parametrize("B,H,Sq,Skv,D,decode,splits", [
    (1, 16, 1, 4001, 128, True, 31), (4, 16, 1, 4001, 128, True, 10), (1, 64, 1, 500, 128, True, 3), (1, 64, 1, 300, 64, True, 1),
    (1, 64, 1, 512, 64, True, 4), (1, 128, 3, 1000, 64, False, 1), (1, 128, 3, 128, 64, True, 1), (1, 256, 4, 1000, 64, True, 3), (8, 16, 4, 4096, 128, False, 1),
    (2, 256, 2, 4096, 128, True, 2), (1, 128, 3, 65, 128, False, 1), (1, 16, 4, 64, 128, True, 1), (1, 149, 4, 255, 128, True, 1),
    (1, 149, 4, 256, 128, False, 1), (1, 16, 5, 500, 64, False, 1), (1, 16, 5, 520, 64, False, 5), (1, 64, 33, 4096, 64, False, 2),
    (1, 8, 300, 4000, 128, False, 1)])
def test_kernel_and_key_ranges_of_few_queries(B, H, Sq, Skv, D, decode, splits):
    """On both sides of the rules' lines: the number of ranges, and whether the call is the decode kernel (it keeps
    the probabilities in fp32, the tile kernel rounds them to bf16: 1.65e-3 and 2.1e-3 or more from 64 bits)."""
    from nabla_b200.native import attention

    attention._lib()
    assert attention._splits(B, H, Sq, Skv, D, 0) == splits
    torch.manual_seed(17)
    q = torch.randn(B, H, Sq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, H, Skv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    o, _ = attention.sdpa_fwd(q, k, v, causal=False, scale=D ** -0.5)
    assert (_rel2(o, _attention64(q, k, v, False)) < 1.85e-3) == decode


@pytest.mark.parametrize("kind", ["keys", "rows", "range hidden"])
@pytest.mark.parametrize("B,H,Sq,Skv,D,splits", [(1, 3, 1, 4001, 128, 32), (2, 1, 4, 700, 64, 6), (2, 4, 33, 2500, 64, 10), (1, 2, 130, 1500, 128, 12),
                                                 (3, 16, 256, 2049, 128, 3)])
def test_masked_attention_over_split_keys(B, H, Sq, Skv, D, splits, kind):
    """Masks are indexed by the key tile of a CTA's range, also where one whole range is hidden from all queries;
    a few queries with a mask take the tile kernel."""
    from nabla_b200.native import attention

    attention._lib()
    assert attention._splits(B, H, Sq, Skv, D, 1) == splits
    torch.manual_seed(15)
    q = torch.randn(B, H, Sq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, H, Skv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    mask = torch.randn((1, 1, Sq, Skv) if kind == "rows" else (B, 1, 1, Skv), device="cuda")
    hide = torch.rand(mask.shape, device="cuda") < 0.3
    hide[..., 0] = False
    if kind == "range hidden":
        per = -(-(-(-Skv // 128)) // splits) * 128           # keys of a range
        hide[..., per:2 * per] = True
    for value in (-1e9, float("-inf")):
        for causal in (False, True):
            _attention_check(q, k, v, causal, mask.masked_fill(hide, value), grads=Sq * Skv < 100000)


def test_attention_shows_a_nan_key_in_every_split():
    from nabla_b200.native import attention

    q = torch.randn(1, 2, 1, 128, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(1, 2, 3000, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    k[0, 1, 2500] = float("nan")
    o, lse = attention.sdpa_fwd(q, k, v, causal=True, scale=0.09)
    assert bool(torch.isfinite(o[0, 0]).all()) and bool(torch.isnan(o[0, 1]).all()) and bool(torch.isnan(lse[0, 1]).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [1023, 4097, 8191, 8192, 8197, 9216, 10241, 16383, 16384, 16391, 18432, 20488, 32000])
def test_log_sum_of_rows_around_three_vectors_per_thread(dtype, D):
    """Rows below, at and above the line (8192 and 16384 elements) and multiples of three vectors of 256 threads, whole and ragged;
    infinities of either sign, a NaN, the type's lowest value, and maxima in the first and the last vector. 4e-6: fp32 sums of D terms by 256 threads, rounded
    logarithm and exponentials."""
    from nabla_b200.native import kernels

    torch.manual_seed(D)
    x = torch.randn(9, D, device="cuda").to(dtype)
    x[1, 0], x[2, D - 1], x[3, D // 2] = 40.0, 40.0, -float("inf")
    x[4, :], x[5, 1], x[6, D - 2] = torch.finfo(dtype).min, float("nan"), float("inf")
    x[7, : D - 1] = -float("inf")
    t = torch.randint(0, D, (9,), device="cuda")
    lse, picked = kernels.lse_pick_fwd(x, t)
    ref = torch.logsumexp(x.double(), 1)
    rows = [0, 1, 2, 3, 7, 8]
    assert ((lse.double() - ref)[rows].abs() <= 4e-6 * (1 + ref[rows].abs())).all() and torch.isnan(lse[5])
    assert torch.equal(picked[rows], x[torch.arange(9, device="cuda"), t].float()[rows])
    assert lse[4].item() <= torch.finfo(dtype).min / 2 and not torch.isfinite(lse[6])


@pytest.mark.parametrize("M,N,K", [(1, 8, 16), (130, 264, 64), (129, 200, 512), (300, 77, 128), (2048, 16400, 64)])
def test_gelu_epilogues_against_64_bits(M, N, K):
    """Tiles of each width with ragged ends, one tile per CTA and several, results beyond half of L2; values into both tails, and
    infinities and NaN, which stay with their own element."""
    from nabla_b200.native.gemm import gemm_bf16

    torch.manual_seed(25)
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), (torch.randn(K, N, device="cuda") * 3 * K ** -0.5).to(torch.bfloat16)
    bias, z = torch.randn(N, device="cuda").to(torch.bfloat16), (torch.randn(M, N, device="cuda") * 3).to(torch.bfloat16)
    x = a.double() @ b.double()
    phi = lambda t: 0.5 * torch.erfc(-t / 2 ** 0.5)  # noqa: E731
    y, pre = gemm_bf16(a, b, bias=bias, epilogue="gelu", aux="store_preact")
    t = x + bias.double()
    assert _rel2(pre, t) < STORED[torch.bfloat16] and _rel2(y, t * phi(t)) < STORED[torch.bfloat16]
    assert torch.equal(y, gemm_bf16(a, b, bias=bias, epilogue="gelu"))
    zd = z.double()
    d = phi(zd) + zd * torch.exp(-zd * zd / 2) / (2 * torch.pi) ** 0.5
    assert _rel2(gemm_bf16(a, b, aux="dgelu", aux_in=z), x * d) < STORED[torch.bfloat16]
    assert _rel2(gemm_bf16(a, b, aux="drelu", aux_in=z), x * (zd > 0)) < STORED[torch.bfloat16]
    assert _rel2(gemm_bf16(a, b, bias=bias, aux="add", aux_in=z), t + zd) < STORED[torch.bfloat16]
    odd = torch.tensor([float("nan"), 1.0, float("inf"), -2.0, -3e38, 3e38, 45.0, -45.0], device="cuda").to(torch.bfloat16)
    bias2 = odd.repeat(-(-N // 8))[:N]
    y = gemm_bf16(torch.zeros_like(a), b, bias=bias2, epilogue="gelu", out_dtype=torch.float32)
    want = TF.gelu(bias2.double()).expand(M, N)
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    ok = want.isfinite()
    assert ((y.double() - want).abs()[ok] <= 2e-6 * want.abs()[ok] + 1e-6).all()


def test_inference_writes_no_pre_activations():
    import nabla_b200 as nb
    from nabla_b200.nn import functional as F

    torch.manual_seed(26)
    x, w, b = (torch.randn(s, device="cuda").to(torch.bfloat16) for s in ((3, 50, 64), (64, 200), (200,)))
    for act, ref in (("relu", torch.relu), ("gelu", TF.gelu), ("gelu_tanh", lambda t: TF.gelu(t, approximate="tanh"))):
        for args in ((x, w, b), (x, w)):
            f = nb.compile(lambda *a, act=act: F.linear(*a, activation=act))
            got = [f(*map(nb.Tensor.from_torch, args)).to_torch() for _ in range(3)][-1]
            t = x.double() @ w.double() + (b.double() if len(args) == 3 else 0)
            assert _rel2(got, ref(t)) < STORED[torch.bfloat16] + (2e-3 if act == "gelu_tanh" else 0)
            assert "linear_act" in f.dump_plan()


# ---------------------------------------------------------------- sums of two products
@pytest.mark.parametrize("M,N,K,K2", [(2048, 1536, 512, 16), (2100, 2056, 1032, 8), (16384, 512, 512, 64), (1300, 520, 456, 1), (9500, 136, 72, 200), (640, 8200, 264, 256)])
def test_sums_of_two_products(M, N, K, K2):
    """Lone CTAs of each width and pairs, ragged ends of all four sizes, every order of the operands, with a bias and without."""
    from nabla_b200.native.gemm import dual_takes, gemm_dual

    torch.manual_seed(27)
    assert dual_takes(M, N, K, K2)
    bias = torch.randn(N, device="cuda").to(torch.bfloat16)
    for order in range(16):
        ops = []
        for i, (r, c, std) in enumerate(((M, K, 1.0), (K, N, K ** -0.5), (M, K2, 1.0), (K2, N, K2 ** -0.5))):
            t = (torch.randn(r, c, device="cuda") * std).to(torch.bfloat16)
            ops.append(t.t().contiguous().t() if order >> i & 1 else t)
        a, b, a2, b2 = ops
        ref = a.double() @ b.double() + a2.double() @ b2.double()
        assert _rel2(gemm_dual(a, b, a2, b2), ref) < STORED[torch.bfloat16]
        if order in (0, 15):
            assert _rel2(gemm_dual(a, b, a2, b2, bias), ref + bias.double()) < STORED[torch.bfloat16]


@pytest.mark.parametrize("M,scale", [(1500, 16.0), (1500, 24.0), (100, 16.0), (1500, None)])
def test_compiled_adapters(M, scale):
    """A frozen product with an adapter beside it and all gradients; 100 rows run as slices of K and keep their launches."""
    import nabla_b200 as nb

    torch.manual_seed(28)
    x, w, a, b, dy = ((torch.randn(s, device="cuda") * std).to(torch.bfloat16) for s, std in (
        ((M, 520), 1.0), ((520, 1032), 520 ** -0.5), ((520, 16), 0.05), ((16, 1032), 0.3), ((M, 1032), 1.0)))

    def layer(x, w, a, b):
        h = (x @ a) @ b
        return x @ w + (h if scale is None else h * (scale / 16))

    def step(x, w, a, b, dy):
        y, pull = nb.vjp(lambda x, a, b: layer(x, w, a, b), x, a, b, create_graph=False)
        return (y, *pull(dy))

    f = nb.compile(step)
    got = [[t.to_torch() for t in f(*map(nb.Tensor.from_torch, (x, w, a, b, dy)))] for _ in range(3)][-1]
    d = [t.double().requires_grad_(True) for t in (x, a, b)]
    ref = layer(d[0], w.double(), d[1], d[2])
    for g, r in zip(got, (ref, *torch.autograd.grad(ref, d, dy.double()))):
        assert _rel2(g, r.detach()) < 2 * STORED[torch.bfloat16]
    assert sum("+gemm_residual" in line for line in f.dump_plan().splitlines()) == 2


@pytest.mark.parametrize("B,H,Sq,Skv,D,warps", [(1, 4, 1, 127, 64, 0), (1, 4, 1, 128, 64, 16), (1, 16, 1, 1023, 128, 64), (1, 3, 2, 8001, 64, 128), (2, 32, 1, 4001, 128, 32),
                                                (4, 16, 2, 300, 128, 32), (37, 1, 2, 3300, 64, 0), (50, 3, 1, 700, 64, 16), (100, 3, 1, 513, 128, 8),
                                                (16, 10, 2, 400, 64, 0), (401, 1, 1, 2000, 64, 0), (1, 4, 3, 128, 64, 0)])
def test_few_queries_over_clusters(B, H, Sq, Skv, D, warps):
    """Both sides of the rule's lines and every number of warps; a NaN key shows, an unseen one does not."""
    from nabla_b200.native import attention

    attention._lib()
    assert attention._warps(B, H, Sq, Skv, D, 0) == warps and attention._warps(B, H, Sq, Skv, D, 1) == 0
    torch.manual_seed(29)
    q = torch.randn(B, H, Sq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(B, H, Skv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    for causal in (False, True):
        o, lse = attention.sdpa_fwd(q, k, v, causal=causal, scale=D ** -0.5)
        s = (q.double() @ k.double().transpose(-1, -2)) * D ** -0.5
        if causal:
            s = s.masked_fill(~torch.ones(Sq, Skv, dtype=torch.bool, device="cuda").tril(Skv - Sq), float("-inf"))
        assert _rel2(o, torch.softmax(s, -1) @ v.double()) < 1.85e-3 and _rel2(lse, torch.logsumexp(s, -1)) < 1e-5
    k[0, 0, Skv - 1, 0] = float("nan")
    o, _ = attention.sdpa_fwd(q, k, v, causal=True, scale=D ** -0.5)
    assert o[0, 0, -1].isnan().all() and not o[0, 0, :-1].isnan().any() and not o.reshape(-1, Sq, D)[1:].isnan().any()


@pytest.mark.parametrize("bh,Sq,Skv,D,warps", [(148, 1, 2001, 128, 0), (149, 1, 2001, 128, 16), (128, 1, 901, 64, 16), (129, 1, 901, 64, 16), (96, 1, 999, 64, 16),
                                               (96, 1, 1001, 64, 32), (296, 1, 700, 64, 0), (297, 1, 700, 64, 8), (290, 1, 700, 64, 8), (400, 1, 700, 128, 8), (16, 1, 2999, 128, 64), (16, 1, 3000, 128, 128), (300, 1, 130, 64, 0),
                                               (192, 2, 999, 64, 8), (192, 2, 1000, 64, 0), (24, 2, 8000, 128, 0),
                                               (48, 1, 300, 128, 64), (32, 2, 301, 128, 64), (1, 1, 1500, 64, 128)])
def test_few_queries_by_what_fits_the_chip(bh, Sq, Skv, D, warps):
    """Grids that load ahead and that do not, in clusters (up to 512 blocks) and in ranges (592), one block to either side, against 64 bits."""
    from nabla_b200.native import attention

    attention._lib()
    assert attention._warps(1, bh, Sq, Skv, D, 0) == warps
    torch.manual_seed(31)
    q = torch.randn(1, bh, Sq, D, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn(1, bh, Skv, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    o, lse = attention.sdpa_fwd(q, k, v, causal=True, scale=D ** -0.5)
    for h in range(0, bh, 64):
        w = slice(h, h + 64)
        s = (q[:, w].double() @ k[:, w].double().transpose(-1, -2)) * D ** -0.5
        s = s.masked_fill(~torch.ones(Sq, Skv, dtype=torch.bool, device="cuda").tril(Skv - Sq), float("-inf"))
        assert _rel2(o[:, w], torch.softmax(s, -1) @ v[:, w].double()) < 1.85e-3 and _rel2(lse[:, w], torch.logsumexp(s, -1)) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,H,C,F,k,pool,stride", [(3, 12, 1, 8, 3, 2, 2), (2, 11, 4, 12, 3, 2, 2), (2, 9, 3, 5, 2, 3, 2), (5, 16, 8, 32, 3, 2, 2)])
def test_compiled_convolutions_take_their_relu(dtype, N, H, C, F, k, pool, stride):
    """Convolution, relu, max pooling (windows apart and overlapping) and all gradients, compiled against plain; and NaN as a plain relu has it."""
    import nabla_b200 as nb

    torch.manual_seed(30)
    x, w, b = ((torch.randn(s, device="cuda") * std).to(dtype) for s, std in (((N, H, H, C), 1.0), ((k, k, C, F), 0.3), ((F,), 0.3)))

    def net(x, w, b):
        h = nb.max_pool2d(nb.relu(nb.conv2d(x, w, bias=b, padding=1)), pool, stride)
        return h * 1.5

    def step(x, w, b, dy):
        y, pull = nb.vjp(net, x, w, b, create_graph=False)
        return (y, *pull(dy))

    ts = [nb.Tensor.from_torch(t) for t in (x, w, b)]
    dy = nb.Tensor.from_torch(torch.randn_like(net(*ts).to_torch()))
    f = nb.compile(step)
    got = [[t.to_torch() for t in f(*ts, dy)] for _ in range(3)][-1]
    plan = f.dump_plan()
    assert plan.count("conv_relu") == 1 and plan.count("pool_bwd_relu") == 1
    for a, c in zip(got, step(*ts, dy)):
        assert _rel2(a, c.to_torch()) < 4 * STORED[dtype]
    assert torch.equal(got[0], net(*ts).to_torch())
    x[0, 0, 0, 0] = float("nan")
    g = nb.compile(lambda x, w, b: nb.relu(nb.conv2d(x, w, bias=b, padding=1)))
    for _ in range(2):
        y = g(nb.Tensor.from_torch(x), *ts[1:]).to_torch()
        assert torch.equal(y.isnan(), nb.relu(nb.conv2d(nb.Tensor.from_torch(x), ts[1], bias=ts[2], padding=1)).to_torch().isnan())
    assert "conv_relu" in g.dump_plan()


def test_flipped_filters():
    from nabla_b200.native import kernels

    for shape in ((1, 1, 1, 1), (3, 2, 5, 7), (7, 7, 3, 64)):
        for dtype in (torch.float32, torch.bfloat16):
            w = torch.randn(shape, device="cuda").to(dtype)
            assert torch.equal(kernels.conv_flip(w), w.flip(0, 1).permute(0, 1, 3, 2).contiguous())


def test_captured_leaves_run_beside_the_chain():
    """Weight and bias gradients of a captured step on streams of their own: the same bits as from one chain, over many replays whose
    inputs change while the one before may still run; results of earlier calls stay what they were."""
    import nabla_b200 as nb
    from nabla_b200.models import transformer as T

    cfg = T.TransformerConfig(n_layers=1, d_model=256, n_heads=4, d_ff=1024)
    names = ("ln1_g", "ln1_b", "wqkv", "bqkv", "wo", "bo", "ln2_g", "ln2_b", "w1", "b1", "w2", "b2")
    torch.manual_seed(32)
    d, f = 256, 1024
    shapes = ((d,), (d,), (d, 3 * d), (3 * d,), (d, d), (d,), (d,), (d,), (d, f), (f,), (f, d), (d,))
    p = [(torch.randn(s, device="cuda") * (s[0] ** -0.5 if len(s) == 2 else 0.1)).to(torch.bfloat16) for s in shapes]
    xs = [torch.randn(2, 200, d, device="cuda").to(torch.bfloat16) for _ in range(12)]
    dys = [torch.randn(2, 200, d, device="cuda").to(torch.bfloat16) for _ in range(12)]

    def step(x, dy, *q):
        y, pull = nb.vjp(lambda t, *q: T.block(t, dict(zip(names, q)), cfg), x, *q, create_graph=False)
        return (y, *pull(dy))

    wrap = nb.Tensor.from_torch
    g, plain = nb.compile(step, cuda_graph=True), nb.compile(step)
    want = [[t.to_torch() for t in plain(wrap(x), wrap(dy), *map(wrap, p))] for x, dy in zip(xs, dys)]
    got = [[t.to_torch() for t in g(wrap(x.clone()), wrap(dy.clone()), *map(wrap, p))] for _ in range(4) for x, dy in zip(xs, dys)]
    recs = [r for e in g._cache.values() for r in e.values() if hasattr(r, "branch_steps")]
    assert g.stats.cuda_graphs == 1 and len(recs) == 1 and len(recs[0].branch_steps) >= 5
    for k, outs in enumerate(got):
        for a, b in zip(outs, want[k % 12]):
            assert torch.equal(a, b)
    h = nb.compile(step, cuda_graph=True, donate_argnums=(0,))
    h(wrap(xs[0].clone()), wrap(dys[0]), *map(wrap, p))
    assert not any(r.branch_steps for e in h._cache.values() for r in e.values() if hasattr(r, "branch_steps"))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(1, 512), (100, 4096), (296, 3072), (297, 3072), (700, 1536), (5000, 1536), (2047, 1000), (601, 264)])
@pytest.mark.parametrize("add", [False, True])
def test_layer_norm_backward_of_less_than_a_chipful_of_blocks(rows, D, dtype, add):
    """Grids whose blocks are kept apart by their shared memory and grids that are not, with and without a gradient that joins, twice in a row."""
    from nabla_b200.native import kernels

    if D > (2048 if dtype == torch.float32 else 4096):
        pytest.skip("rows of at most 16 warps")
    g = torch.Generator("cuda").manual_seed(rows + D)
    x, dy, extra = ((torch.randn(rows, D, generator=g, device="cuda") + 0.1).to(dtype) for _ in range(3))
    gamma = torch.randn(D, generator=g, device="cuda").to(dtype)
    _, mean, rstd = kernels.layernorm_fwd(x, gamma, None, 1e-5)
    d = x.double().requires_grad_(True)
    w = gamma.double().requires_grad_(True)
    dx64, dw64 = torch.autograd.grad(TF.layer_norm(d, (D,), w, None, 1e-5), (d, w), dy.double())
    tol = 2.5e-3 if dtype == torch.bfloat16 else 2e-6         # stored to 2^-9 / 2^-24; sums of up to 5000 rows in fp32
    for _ in range(2):
        dx, dw, db = kernels.layernorm_bwd(dy, x, gamma, mean, rstd, add=extra if add else None)
        assert _rel2(dx, dx64 + extra.double() if add else dx64) < tol and _rel2(dw, dw64) < tol and _rel2(db, dy.double().sum(0)) < tol
