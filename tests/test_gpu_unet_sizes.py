"""The network's convolution kernels at the edges of their tiles (csrc/unet.cu): the smallest grid
(one pixel on the coarsest level), widths that leave each tile shape partly filled, coarse widths that
are not multiples of four, against the float64 oracle with the same BF16 weights.  Inputs, sparse
weights and biases are small integers, so every forward sum (multiples of 1/64 below 2^18) is exact in
FP32: the output equals the oracle's, and no ReLU is decided by rounding.  A weight gradient sums up
to 57,000 products in FP32 partials of at most 1,000: 1e-3 of the maximum is above 1000 2^-24 of the
sum of magnitudes."""
import numpy as np
import pytest

from conftest import load_package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('b,h,w', [(1, 8, 8), (2, 8, 40), (1, 24, 72), (3, 16, 104), (1, 40, 136), (1, 72, 264), (2, 64, 128)])
def test_sizes_match_oracle(b, h, w):
    torch = pytest.importorskip('torch')
    import unet_oracle as uo
    learned = load_package().learned
    wts = learned.UNetWeights(seed=h + w)
    rng = np.random.default_rng(w)
    with torch.no_grad():
        for t, bias in zip(wts.w, wts.b):
            keep = rng.random(tuple(t.shape)) < min(1.0, 4.0 / (9 * t.shape[1]))
            t.copy_(torch.from_numpy(np.where(keep, rng.integers(0, 2, tuple(t.shape)) * 2 - 1, 0)).float())
            bias.copy_(torch.from_numpy(rng.integers(-1, 2, bias.numel())).float())
    wts.refresh()
    x = rng.integers(-3, 4, (b, 2, h, w)).astype(np.float32)
    net = learned.UNet(b, h, w)
    xd = torch.from_numpy(x).cuda()
    y = net.forward(wts, xd)
    ws = [t.to(torch.float32).cpu().numpy().astype(np.float64) for t in wts.w16]
    bs = [t.detach().cpu().numpy().astype(np.float64) for t in wts.b]
    ref, saved = uo.forward(x.astype(np.float64), ws, bs)
    assert np.max(np.abs(ref)) < 2 ** 18 and np.array_equal(y.cpu().numpy(), ref)
    dy = rng.integers(-3, 4, ref.shape).astype(np.float32)
    dw, db = net.backward(wts, torch.from_numpy(dy).cuda())
    dws, dbs = uo.backward(saved, ws, dy.astype(np.float64))
    for k in range(12):
        for g, r in ((dw[k], dws[k]), (db[k], dbs[k])):
            assert np.max(np.abs(g.cpu().numpy() - r)) < 1e-3 * max(np.max(np.abs(r)), 1e-12), k
    net.close()


def test_output_at_an_odd_address():
    """The caller's output may start at any float: no wide stores there then."""
    torch = pytest.importorskip('torch')
    import ctypes as C
    pkg = load_package()
    learned, lib = pkg.learned, pkg._lib.lib
    wts, net = learned.UNetWeights(seed=1), learned.UNet(1, 16, 32)
    x = torch.randn(1, 2, 16, 32, device='cuda')
    want = net.forward(wts, x)
    buf = torch.zeros(16 * 32 + 8, device='cuda')
    assert lib.gm_unet_forward(net._u, wts.wp, wts.bp, C.c_void_p(x.data_ptr()), C.c_void_p(buf[3:].data_ptr()), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(buf[3:3 + 512], want.reshape(-1)) and not buf[:3].any() and not buf[515:].any()
    net.close()
