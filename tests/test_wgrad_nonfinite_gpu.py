"""Weight gradient of the convolution with infinite and NaN activations at the
image's edges: an activation reaches the taps whose output pixel lies in the
image, and no others, also where the kernel's 8x16 pixel tiles overhang it."""
import ctypes as C

import pytest

import voreen_gb300 as v

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("n,h,w", [(1, 9, 17), (2, 5, 15), (1, 8, 15), (1, 15, 16), (1, 3, 31), (1, 8, 16), (1, 1, 1)])
@pytest.mark.parametrize("cin,cout", [(16, 16), (48, 32), (64, 64), (80, 128)])
def test_weight_gradient_of_activations_that_are_not_finite(vrc_lib, n, h, w, cin, cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(h * w + cin)
    x = torch.randn((n, h, w, cin), device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randn((n, h, w, cout), device="cuda", generator=g).to(torch.bfloat16)
    dy[dy == 0] = 1.0
    inf, nan = float("inf"), float("nan")
    x[:, :, w - 1, 0], x[:, h - 1, :, 1], x[n - 1, h - 1, w - 1, 2] = inf, -inf, nan
    x[:, :, 0, 3], x[:, 0, :, 4], x[0, h // 2, w // 2, cin - 1] = nan, inf, inf
    dw = torch.zeros((cout, 9, cin), device="cuda")
    torch.cuda.synchronize()
    assert v.lib().vrc_nn_conv3x3_wgrad(_p(x), _p(dy), n, h, w, cin, cout, _p(dw), None, None) == 0
    torch.cuda.synchronize()
    dw, x64, d64 = dw.double(), x.double(), dy.double()
    for ky in range(3):
        for kx in range(3):
            # output pixels whose input pixel (y + ky - 1, x + kx - 1) lies in the image
            ys, xs = slice(max(1 - ky, 0), min(h + 1 - ky, h)), slice(max(1 - kx, 0), min(w + 1 - kx, w))
            yi, xi = slice(ys.start + ky - 1, ys.stop + ky - 1), slice(xs.start + kx - 1, xs.stop + kx - 1)
            d, a = d64[:, ys, xs].reshape(-1, cout, 1), x64[:, yi, xi].reshape(-1, 1, cin)
            got = dw[:, 3 * ky + kx]
            want = (d * a).sum(0)
            finite = torch.isfinite(want)
            assert torch.equal(torch.isfinite(got), finite), (ky, kx)
            # BF16 products are exact in FP32; the sums of K of them within K * 2^-24 of their magnitudes'
            bound = (d * a).abs().sum(0) * (n * h * w * 2.0 ** -24) + 1e-30
            assert ((got - want).abs()[finite] <= bound[finite]).all(), (ky, kx)

