"""The warm-start network's weight gradients as sums over their own operands:
the activations, propagated gradients and ReLU masks that the device holds are
read back and contracted in FP64.

Tolerance, relative to the sum of the terms' magnitudes: a run of 16 pixels is
exact to the last bit, and a block adds at most 4 runs a tile, then 8 warps'
sums, in FP32 before the FP64 sum of the blocks.  One tile a block bounds the
worst case by 12 x 2^-24 < 1e-6; over many blocks those roundings are unbiased
and average out to below 1e-7.  A gradient of one or two BF16 parts and a
truncating running sum, formed here in numpy, have to lie outside the bounds."""
import numpy as np
import pytest
import torch

from gpu_util import need_gpu
from oracle import cnn_oracle as C

HID = 8


def _train(batch, grid, make_target, seed=11):
    """One backward pass; the layers' (x, g, mask, dW, db) as FP64 arrays."""
    from fbme_b200.learned import WarmStartNet, init_params
    from test_gpu_cnn import _flat_to_dict

    rng = np.random.default_rng(seed)
    n = grid[0] * grid[1]
    bp = (rng.normal(size=(batch, n)) + 1j * rng.normal(size=(batch, n))).astype(np.complex64)
    net = WarmStartNet(torch.device("cuda", 0), init_params(seed))
    net.features(torch.from_numpy(bp).cuda(), *grid)
    out = net.forward(batch, *grid)
    net.backward(make_target(out, rng), batch, *grid)
    torch.cuda.synchronize()
    buf, ptr, nbytes = net._ws[(batch, *grid)]
    ws = buf[ptr - buf.data_ptr():][:nbytes]
    off = 64 * 1024

    def take(width, dtype):  # the workspace's arrays, each from a 256-byte boundary
        nonlocal off
        size = batch * n * width * dtype.itemsize
        a = ws[off:off + size].view(dtype).reshape(batch, *grid, width).double().cpu().numpy()
        off += (size + 255) // 256 * 256
        return a

    x8, h1, h2 = (take(HID, torch.bfloat16) for _ in range(3))
    take(1, torch.float32)  # the output
    dout, dh2, dh1 = (take(HID, torch.float32) for _ in range(3))
    grad = _flat_to_dict(net.grad.cpu().numpy())
    return [(h2, dout[..., :1], None, grad["W3"], grad["b3"]), (h1, dh2, h2, grad["W2"], grad["b2"]),
            (x8[..., :2], dh1, h1, grad["W1"], grad["b1"])]


def _sums(x, g, mask):
    """(dW, db) of the layer: sums over the pixels."""
    if mask is not None:
        g = np.where(mask > 0, g, 0.0)
    _, h, w, ci = x.shape
    xp = np.pad(x, ((0, 0), (1, 1), (1, 1), (0, 0)))
    flat = g.reshape(-1, g.shape[-1])
    dw = np.stack([np.stack([xp[:, dy:dy + h, dx:dx + w].reshape(-1, ci).T @ flat for dx in range(3)]) for dy in range(3)])
    return dw, flat.sum(0)


def _parts(g, n):
    """g as its first n BF16 parts."""
    s, r = np.zeros_like(g), g
    for _ in range(n):
        p = C.bf16_round(r.astype(np.float32))
        s, r = s + p, r - p
    return s


def _worst(got, ref, scale):
    return max(float(np.max(np.abs(a - b) / np.maximum(c, 1e-300))) for a, b, c in zip(got, ref, scale))


# two parts leave 7e-6 of this gradient out in every pixel, one part 2e-3
ONE_SIGNED = 1.0 + 2.0**-9 + 0.45 * 2.0**-16


@pytest.mark.gpu
@pytest.mark.parametrize("batch,grid", [(1, (8, 16)), (2, (40, 48)), (1, (8, 272))])
def test_sums_hold_the_whole_gradient(batch, grid):
    need_gpu()
    n = batch * grid[0] * grid[1]
    layers = _train(batch, grid, lambda out, rng: out - ONE_SIGNED * n / 2)
    for x, g, mask, dw, db in layers:
        ref, scale = _sums(x, g, mask), _sums(np.abs(x), np.abs(g), mask)
        assert _worst((dw, db), ref, scale) < 1e-6
    x, g, mask, _, _ = layers[0]
    for parts in (1, 2):
        assert _worst(_sums(x, _parts(g, parts), mask), _sums(x, g, mask), _sums(np.abs(x), np.abs(g), mask)) > 1e-6


@pytest.mark.gpu
def test_sums_are_unbiased():
    need_gpu()
    batch, grid = 16, (256, 256)
    n = batch * grid[0] * grid[1]

    def target(out, rng):
        return out - torch.from_numpy(rng.uniform(0.5, 1.5, out.shape).astype(np.float32)).cuda() * (n / 2)

    layers = _train(batch, grid, target)
    for x, g, mask, dw, db in layers:
        assert _worst((dw, db), _sums(x, g, mask), _sums(np.abs(x), np.abs(g), mask)) < 1e-7
    # the runs of a block, summed in FP32 toward zero
    runs = layers[0][1].reshape(-1, 16).sum(1)[: n // 16 // 256 * 256].reshape(-1, 256).astype(np.float32)
    acc = np.zeros(256, np.float32)
    for r in runs[:28]:
        s = acc.astype(np.float64) + r
        up = s.astype(np.float32)
        acc = np.where(up > s, np.nextafter(up, np.float32(0)), up)
    exact = runs[:28].astype(np.float64).sum(0)
    assert float(np.mean(exact - acc) / np.mean(exact)) > 1e-7


@pytest.mark.gpu
def test_infinite_gradient_gives_infinite_sums():
    need_gpu()

    def target(out, rng):
        t = torch.zeros_like(out)
        t[0, 37] = float("inf")
        return t

    for x, g, mask, dw, db in _train(1, (16, 32), target):
        with np.errstate(invalid="ignore"):
            ref = _sums(x, g, mask)
        for a, b in zip((dw, db), ref):
            assert np.array_equal(np.isnan(a), np.isnan(b))
            assert np.array_equal(np.isposinf(a), np.isposinf(b)) and np.array_equal(np.isneginf(a), np.isneginf(b))
