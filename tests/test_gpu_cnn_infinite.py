"""Weight gradients over activations past BF16's range: infinite, of the sign
of the sum of products, and NaN only where the products themselves are.

One pixel of layer 1 overflows in channel 0; everything else is finite and
positive, so the sums have to be infinite wherever a product with that pixel
enters.  Compared with FP64 sums over the operands that the device holds."""
import numpy as np
import pytest
import torch

from gpu_util import need_gpu
from oracle import cnn_oracle as C
from test_gpu_cnn_wgrad_sums import HID, _sums

GRID = (32, 48)


def _params(f_low):
    """Channel 0 of layer 1: 4 ulp of the bias at feature f_low, past the range
    13 above it; the other channels 1."""
    w, ulp = 3e37, 2.0**103
    w1 = np.zeros((3, 3, 2, HID), np.float32)
    w1[1, 1, 0, 0] = C.bf16_round(np.float32(w))
    b1 = np.ones(HID, np.float32)
    b1[0] = -float(w1[1, 1, 0, 0]) * f_low + 4 * ulp
    w2 = np.full((3, 3, HID, HID), 0.1, np.float32)
    w2[:, :, 0, :] = 1e-32
    rest = (np.full(HID, 0.1), np.full((3, 3, HID, 1), 0.1), np.zeros(1))
    return np.concatenate([a.astype(np.float32).ravel() for a in (w1, b1, w2, *rest)])


@pytest.mark.gpu
@pytest.mark.parametrize("pixel", [(15, 31), (5, 10), (20, 47)])
def test_infinite_activation_gives_infinite_sums(pixel):
    need_gpu()
    from fbme_b200.learned import WarmStartNet
    from test_gpu_cnn import _flat_to_dict

    n = GRID[0] * GRID[1]
    bp = np.ones((1, n), np.complex64)
    bp[0, pixel[0] * GRID[1] + pixel[1]] = 1e3
    f = C.bf16_round(C.features(bp, GRID)[0, ..., 0].astype(np.float32))
    net = WarmStartNet(torch.device("cuda", 0), _params(float(f[0, 0])))
    net.features(torch.from_numpy(bp).cuda(), *GRID)
    net.forward(1, *GRID)
    net.backward(torch.zeros(1, n, device="cuda"), 1, *GRID)
    torch.cuda.synchronize()
    buf, ptr, nbytes = net._ws[(1, *GRID)]
    ws = buf[ptr - buf.data_ptr():][:nbytes]
    off = 64 * 1024

    def take(width, dtype):
        nonlocal off
        size = n * width * dtype.itemsize
        a = ws[off:off + size].view(dtype).reshape(1, *GRID, width).double().cpu().numpy()
        off += (size + 255) // 256 * 256
        return a

    x8, h1, h2 = (take(HID, torch.bfloat16) for _ in range(3))
    take(1, torch.float32)
    dout, dh2, dh1 = (take(HID, torch.float32) for _ in range(3))
    assert np.isinf(h1).sum() == 1 and np.isinf(h1[0, pixel[0], pixel[1], 0])
    assert not np.isnan(h2).any() and (h2 > 0).all() and np.isinf(h2).any()
    grad = _flat_to_dict(net.grad.cpu().numpy())
    for x, g, mask, dw, db in ((h2, dout[..., :1], None, grad["W3"], grad["b3"]), (h1, dh2, h2, grad["W2"], grad["b2"]),
                               (x8[..., :2], dh1, h1, grad["W1"], grad["b1"])):
        with np.errstate(invalid="ignore"):
            ref = _sums(x, g, mask)
        for a, b in zip((dw, db), ref):
            assert np.array_equal(np.isnan(a), np.isnan(b))
            assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
    if pixel[1] < GRID[1] - 5:  # away from the border no product is NaN
        assert np.isposinf(grad["W3"]).all() and np.isposinf(grad["W2"]).all()
