"""The denoiser's pooling and upsampling kernels at the edges of their grids
(GPU): image rows wider than a block, more image rows than a grid is high, and
the smallest image.

A pixel's sums do not depend on the images beside it, so a large batch of the
same images gives the same bits as a small one.  Against the oracle that rounds
to BF16 wherever the library stores BF16, the bounds are those of an exact
network (3 % of the largest output, 20 % of a layer's gradient): a wrong index
is an error of order one.
"""
import numpy as np
import pytest

from oracle import unet_oracle as U
from pt_gb300.denoise import UNet, init_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _inputs(seed, n, h, w):
    rng = np.random.default_rng(seed)
    x = U.bf16(rng.uniform(-1, 1, (n, h, w, 16)))
    t = rng.uniform(0, 3, (n, h, w, 4)).astype(np.float32)
    return torch.from_numpy(x.astype(np.float32)).cuda(), torch.from_numpy(t).cuda(), x, t


def _forward(n, h, w, x, p):
    net = UNet(n, h, w)
    net.set_params(p)
    net.input_tensor().copy_(x.to(torch.bfloat16))
    net.base_tensor().zero_()
    net.forward()
    torch.cuda.synchronize()
    return net


@pytest.mark.parametrize("n,h,w,copies", [(8, 16, 8, 1024), (2, 8, 520, 3)])
def test_batch_does_not_change_an_image(n, h, w, copies):
    """8192 images of 16 rows are 65536 pooled rows, one more than a grid is high."""
    p = init_params(2)
    x, _, _, _ = _inputs(11, n, h, w)
    small = _forward(n, h, w, x, p)
    ref = small.output_tensor().clone()
    large = _forward(n * copies, h, w, x.repeat(copies, 1, 1, 1), p)
    got = large.output_tensor().view(copies, n, h, w, -1)
    assert torch.equal(got, ref.unsqueeze(0).expand_as(got))


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (1, 8, 1032), (3, 24, 56)])
def test_forward_and_gradients_match_oracle(n, h, w):
    p = init_params(3)
    x, t, xh, th = _inputs(12, n, h, w)
    net = _forward(n, h, w, x, p)
    out = net.output_tensor().cpu().numpy().astype(np.float64)
    loss = net.backward(t.data_ptr())
    g = net.grads().astype(np.float64)
    pw = p.astype(np.float64).copy()
    for wt, _ in U.split_params(pw):
        wt[...] = U.bf16(wt)
    ref_out, cache = U.forward(pw, xh.astype(np.float64), bf16_storage=True, base=np.zeros((n, h, w, 4)))
    ref_loss, ref_g = U.backward(cache, th)
    assert np.abs(out - ref_out).max() <= 0.03 * np.abs(ref_out).max() + 1e-4
    assert abs(loss - ref_loss) <= 0.02 * ref_loss
    offs = np.cumsum([0] + [9 * ci * co + co for ci, co, _ in U.LAYERS])
    for li in range(len(U.LAYERS)):
        a, b = g[offs[li]:offs[li + 1]], ref_g[offs[li]:offs[li + 1]]
        assert np.linalg.norm(a - b) <= 0.20 * np.linalg.norm(b), li
