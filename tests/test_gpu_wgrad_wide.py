"""Weight gradient of layers with 16 output channels and many input channels,
where the tiles that the accumulators leave room for do not fit shared memory
(288 input channels and more at a width above 32): against the FP64 sums over
the same BF16 values, with the tolerance of the other weight gradients
(test_gpu_nn.py: 1e-5 of the value and of the largest; FP32 sums of fewer terms
than there)."""
import numpy as np
import pytest

from oracle import unet_oracle as U
from pt_gb300 import abi

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SHAPES = [  # n, h, w, pitch, c0, cin, cout
    (1, 4, 72, 272, 0, 272, 16),  # the widest that fits as it is
    (1, 4, 72, 288, 0, 288, 16),
    (1, 1, 33, 288, 0, 288, 16),
    (2, 3, 40, 416, 16, 400, 16),  # ten tiles, as many as the accumulators hold
    (1, 5, 65, 512, 0, 512, 16),  # more
    (1, 2, 32, 512, 0, 512, 16),
]


@pytest.mark.parametrize("shape", SHAPES)
def test_wide_layers(shape):
    n, h, w, pitch, c0, cin, cout = shape
    rng = np.random.default_rng(pitch + w)
    x = U.bf16(rng.uniform(-1, 1, (n, h, w, pitch)))
    g = U.bf16(rng.standard_normal((n, h, w, cout)))
    xd = torch.from_numpy(np.asarray(x, np.float32)).to(torch.bfloat16).cuda()
    gd = torch.from_numpy(np.asarray(g, np.float32)).to(torch.bfloat16).cuda()
    dw = torch.zeros((9, cin, cout), dtype=torch.float32, device="cuda")
    rc = abi.lib().pt_nn_conv3x3_wgrad(xd.data_ptr(), n, h, w, pitch, c0, cin, gd.data_ptr(), cout, dw.data_ptr(), None)
    assert rc == abi.PT_OK
    ref = U.conv3x3_wgrad(x[..., c0:c0 + cin].astype(np.float64), g.astype(np.float64))
    got = dw.cpu().numpy().astype(np.float64)
    tol = 1e-5 * np.abs(ref) + 1e-5 * np.abs(ref).max()
    bad = np.abs(got - ref) > tol
    assert not bad.any(), f"{bad.sum()} of {bad.size} outside tolerance; max err {np.abs(got - ref).max():.3g}"
