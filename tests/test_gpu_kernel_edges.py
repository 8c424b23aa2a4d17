"""Kernels and dispatch rules at the sizes where they can go wrong (tile edges, remainders, the smallest and
largest of a rule's range) against 64-bit torch results. Needs a B200 (sm_100a)."""
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
