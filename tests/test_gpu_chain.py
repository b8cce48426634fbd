"""Kernels that are brought up before the one ahead of them ends keep the order
of their stream (GPU): a network called between other work of the same stream, which
writes its input and reads its output, gives the bits of the same calls with a
synchronization around each.  No tolerance: a pixel's sums are in a fixed
order."""
import numpy as np
import pytest

from pt_gb300.denoise import UNet, init_params

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 8, 8), (2, 24, 136), (1, 256, 512)])
def test_back_to_back_forward_keeps_stream_order(n, h, w):
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.uniform(-1, 1, (n, h, w, 16)).astype(np.float32)).cuda().to(torch.bfloat16)
    net = UNet(n, h, w)
    net.set_params(init_params(4))
    net.base_tensor().zero_()
    out, inp = net.output_tensor(), net.input_tensor()
    steps = 12
    ref = []
    for i in range(steps):
        inp.copy_(x.roll(i, 0 if n > 1 else 2) * (1 + i))
        torch.cuda.synchronize()
        net.forward()
        torch.cuda.synchronize()
        ref.append(out.clone())
        torch.cuda.synchronize()
    ref = torch.stack(ref)
    got = torch.empty_like(ref)
    st = torch.cuda.Stream()

    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        for i in range(steps):
            inp.copy_(x.roll(i, 0 if n > 1 else 2) * (1 + i))
            net.forward(stream=st.cuda_stream)
            got[i].copy_(out)
    torch.cuda.synchronize()
    assert torch.equal(got, ref)
