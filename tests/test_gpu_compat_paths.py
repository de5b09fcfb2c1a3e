"""The extension stand-ins' own fast paths (niti_b200/compat) at the edges of their tiles, against the oracle: the weight
gradient of batch-innermost operands, thin matrix products and the fp16 form of the pooling backward."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from niti_b200 import ops  # noqa: E402
from niti_b200.compat import cutlassconv_cuda, int8mm_cuda, int8pool_cuda  # noqa: E402
from oracle import niti_oracle as O  # noqa: E402

DEV = "cuda:0"


def rnd8(rng, shape):
    return rng.integers(-127, 128, size=shape).astype(np.int8)


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def off_by_one(t):
    """The same contiguous tensor, starting one element into its buffer."""
    odd = torch.empty(t.numel() + 1, dtype=t.dtype, device=DEV)[1:].view(t.shape)
    return odd.copy_(t)


@pytest.mark.parametrize("N,H,W,C,K", [
    (16, 4, 4, 16, 16), (48, 5, 7, 32, 144), (128, 3, 6, 144, 128), (144, 2, 2, 16, 272), (256, 8, 8, 128, 64)])
def test_weight_gradient_with_the_batch_innermost(N, H, W, C, K):
    rng = np.random.default_rng(N + H + C + K)
    x, err = rnd8(rng, (N, H, W, C)), rnd8(rng, (N, H, W, K))
    got = cutlassconv_cuda.sp_conv_optimized(cu(x.transpose(3, 1, 2, 0)), cu(err.transpose(3, 1, 2, 0)), 1, 1)
    want = O.conv_wgrad(x, err, 3, 3, 1).transpose(3, 1, 2, 0)
    assert np.array_equal(got.cpu().numpy(), want)
    ops.check_status(DEV)


@pytest.mark.parametrize("which", ["input", "filters", "both"])
def test_weight_gradient_of_operands_off_a_16_byte_boundary(which):
    """A view that starts inside a buffer goes through aligned copies, as any operand did."""
    rng = np.random.default_rng(4)
    x, err = rnd8(rng, (16, 4, 6, 32)), rnd8(rng, (16, 4, 6, 16))
    x_t, err_t = cu(x.transpose(3, 1, 2, 0)), cu(err.transpose(3, 1, 2, 0))
    got = cutlassconv_cuda.sp_conv_optimized(x_t if which == "filters" else off_by_one(x_t), err_t if which == "input" else off_by_one(err_t), 1, 1)
    assert np.array_equal(got.cpu().numpy(), O.conv_wgrad(x, err, 3, 3, 1).transpose(3, 1, 2, 0))


@pytest.mark.parametrize("M,K,N", [(1, 256, 4), (128, 1028, 12), (77, 2048, 8), (296, 4096, 16), (299, 260, 12), (1, 259, 12)])
def test_thin_products(M, K, N):
    rng = np.random.default_rng(M + K + N)
    a, b = rnd8(rng, (M, K)), rnd8(rng, (K, N))
    assert np.array_equal(int8mm_cuda.int8_mm(cu(a), cu(b)).cpu().numpy(), O.int8_mm(a, b))
    c, mx = ops.gemm_acc(cu(a), cu(b))
    assert np.array_equal(c.cpu().numpy(), O.int8_mm(a, b)) and int(mx) == int(np.abs(O.int8_mm(a, b)).max())


@pytest.mark.parametrize("N,H,W,C", [(1, 2, 2, 8), (3, 6, 4, 24), (16, 16, 16, 64), (2, 4, 4, 12), (2, 5, 5, 16)])
def test_pool_backward_on_fp16_copies(N, H, W, C):
    """Even maps in channels of 8 are routed on the fp16 words themselves; the last two shapes take the int8 kernels."""
    rng = np.random.default_rng(N + H + C)
    x = rng.integers(-4, 5, size=(N, H, W, C)).astype(np.int8)  # few values: many ties
    y = O.maxpool_fwd(x)
    dy = rnd8(rng, y.shape)
    dx = int8pool_cuda.int8_pool_backward(cu(y).half(), cu(dy).half(), cu(x).half(), 2, 2, 0)
    assert dx.dtype == torch.float16
    assert np.array_equal(dx.cpu().numpy(), O.maxpool_bwd(x, dy).astype(np.float16))


@pytest.mark.parametrize("which", ["input", "error", "both"])
def test_pool_backward_of_fp16_operands_off_a_16_byte_boundary(which):
    """A view that starts inside a buffer is narrowed to int8 on the way, as any operand was."""
    rng = np.random.default_rng(6)
    x = rng.integers(-4, 5, size=(2, 6, 4, 16)).astype(np.int8)
    dy = rnd8(rng, (2, 3, 2, 16))
    xh, dyh = cu(x).half(), cu(dy).half()
    dx = int8pool_cuda.int8_pool_backward(cu(O.maxpool_fwd(x)).half(), dyh if which == "input" else off_by_one(dyh),
                                          xh if which == "error" else off_by_one(xh), 2, 2, 0)
    assert dx.dtype == torch.float16
    assert np.array_equal(dx.cpu().numpy(), O.maxpool_bwd(x, dy).astype(np.float16))
