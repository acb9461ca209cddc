"""The convolution kernels at the edges of their tiles and chunks against
float64: one and many 16-channel chunks, images smaller than a tile and one
pixel past it, runs of one and several tiles, gradients on and off 8 bytes; the
wide and the scalar forms of the pool and the head give the same bits."""
import ctypes as C

import numpy as np
import pytest

import voreen_gb300 as v

pytestmark = pytest.mark.gpu


def _p(t, shift=0):
    return C.c_void_p(t.data_ptr() + shift)


def _taps(x):
    import torch
    h, w = x.shape[1:3]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    return [p[:, ky:ky + h, kx:kx + w] for ky in range(3) for kx in range(3)]


# BF16 products are exact in FP32; the sums of K of them in FP32, in any order,
# are within K * 2^-24 of the sum of their magnitudes, and the BF16 result
# within 2^-8 of its own
@pytest.mark.parametrize("n,h,w,cin,cout", [(1, 1, 1, 16, 16), (1, 16, 16, 16, 32), (2, 17, 33, 32, 32), (1, 8, 15, 48, 64),
                                            (3, 9, 17, 128, 128), (1, 40, 47, 64, 16), (2, 33, 16, 96, 64)])
def test_forward_and_weight_gradient(vrc_lib, n, h, w, cin, cout):
    import torch
    g = torch.Generator(device="cuda").manual_seed(h * w + cin)
    x = torch.randn((n, h, w, cin), device="cuda", generator=g).to(torch.bfloat16)
    dy = torch.randn((n, h, w, cout), device="cuda", generator=g).to(torch.bfloat16)
    wt = (torch.randn((cout, 3, 3, cin), device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda", generator=g)
    y = torch.empty((n, h, w, cout), dtype=torch.bfloat16, device="cuda")
    assert v.lib().vrc_nn_conv3x3_fwd(_p(x), n, h, w, cin, _p(wt), _p(b), cout, 0, _p(y), 0, None) == 0
    w64, x64, d64 = wt.double().reshape(cout, 9, cin), x.double(), dy.double()
    ref = sum(t @ w64[:, k].T for k, t in enumerate(_taps(x64))) + b.double()
    mag = sum(t @ w64[:, k].abs().T for k, t in enumerate(_taps(x64.abs()))) + b.double().abs()
    assert ((y.double() - ref).abs() <= ref.abs() * 2.0 ** -8 + mag * (9 * cin + 1) * 2.0 ** -24).all()
    pixels = n * h * w
    dref = torch.stack([torch.einsum("nhwo,nhwi->oi", d64, t) for t in _taps(x64)], 1)
    dmag = torch.stack([torch.einsum("nhwo,nhwi->oi", d64.abs(), t) for t in _taps(x64.abs())], 1)
    for shift in (0, 4):  # gradients on 8 bytes and off them
        buf = torch.zeros(9 * cin * cout + 4, device="cuda")
        db = torch.zeros(cout, device="cuda")
        torch.cuda.synchronize()
        assert v.lib().vrc_nn_conv3x3_wgrad(_p(x), _p(dy), n, h, w, cin, cout, _p(buf, shift), _p(db), None) == 0
        torch.cuda.synchronize()
        dw = buf[shift // 4:shift // 4 + 9 * cin * cout].reshape(cout, 9, cin).double()
        assert ((dw - dref).abs() <= dmag * pixels * 2.0 ** -24 + 1e-30).all()
        assert ((db.double() - d64.sum((0, 1, 2))).abs() <= d64.abs().sum((0, 1, 2)) * pixels * 2.0 ** -24 + 1e-30).all()
        assert float(buf[: shift // 4].abs().sum()) == 0.0


@pytest.mark.parametrize("n,h,w", [(1, 2, 2), (2, 6, 10), (1, 130, 258)])
def test_wide_pool_and_head_equal_the_scalar_forms(vrc_lib, n, h, w):
    import torch
    g = torch.Generator(device="cuda").manual_seed(h + w)
    for c in (8, 16, 32):
        x = torch.randn(n * h * w * c + 8, device="cuda", generator=g).to(torch.bfloat16)
        outs = []
        for shift in (0, 2):  # on 16 bytes, and one element off them
            src = torch.zeros_like(x)
            src[shift // 2:shift // 2 + n * h * w * c] = x[: n * h * w * c]
            out = torch.zeros((n, h // 2, w // 2, c), dtype=torch.bfloat16, device="cuda")
            torch.cuda.synchronize()
            assert v.lib().vrc_nn_avgpool2(_p(src, shift), n, h, w, c, 1.0, _p(out), None) == 0
            torch.cuda.synchronize()
            outs.append(out.view(torch.int16).cpu().numpy())
        np.testing.assert_array_equal(outs[0], outs[1])
    feat = torch.randn((n, h, w, 16), device="cuda", generator=g)
    base = torch.rand((n, h, w, 4), device="cuda", generator=g)
    ref = torch.nn.functional.interpolate(base.double().permute(0, 3, 1, 2), scale_factor=2, mode="bilinear",
                                          align_corners=False).permute(0, 2, 3, 1)
    ref = ref + feat.double().reshape(n, h, w, 2, 2, 4).permute(0, 1, 3, 2, 4, 5).reshape(n, 2 * h, 2 * w, 4)
    for shift in (0, 1):
        buf = torch.zeros(ref.numel() + 4, device="cuda")
        torch.cuda.synchronize()
        assert v.lib().vrc_nn_head_fwd(_p(feat), _p(base), n, h, w, _p(buf, 4 * shift), None) == 0
        torch.cuda.synchronize()
        out = buf[shift:shift + ref.numel()].reshape(ref.shape).double()
        # a few FP32 roundings of values up to |feature| + 1
        assert ((out - ref).abs() <= 8 * 2.0 ** -24 * (feat.abs().max().double() + 1)).all()


@pytest.mark.parametrize("h,w", [(16, 16), (70, 130), (200, 312)])
def test_chained_launches_see_what_came_before(vrc_lib, h, w):
    """Layers that read what the launch before wrote, into buffers that the
    launch before that read, with weights that another kernel just changed:
    the same bits as with a synchronisation after every call."""
    import torch
    L, c = v.lib(), 64
    seen = []
    for wait in (True, False):
        g = torch.Generator(device="cuda").manual_seed(h + w)
        a = torch.randn((1, h, w, c), device="cuda", generator=g).to(torch.bfloat16)
        b, pooled = torch.zeros_like(a), torch.zeros((1, h // 2, w // 2, c), dtype=torch.bfloat16, device="cuda")
        w0 = (torch.randn((c, 3, 3, c), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
        wt, wtc, bias = w0.clone(), torch.empty_like(w0), torch.randn(c, device="cuda", generator=g) * 0.1
        sums, err = [], torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()

        def call(r):
            assert r == 0
            if wait:
                torch.cuda.synchronize()

        for i in range(12):
            wt.copy_(torch.roll(w0, i, 0))
            call(L.vrc_nn_weights_tc(_p(wt), c, c, 0, 1, _p(wtc), None))
            call(L.vrc_nn_conv3x3_fwd(_p(a), 1, h, w, c, _p(wt), _p(bias), c, 2, _p(b), 0, None))
            call(L.vrc_nn_conv3x3_tc(_p(b), c, None, 0, 1, h, w, _p(wtc), _p(bias), c, 1, 2, _p(a), 0, _p(err), None))
            call(L.vrc_nn_avgpool2(_p(a), 1, h, w, c, C.c_float(1.0), _p(pooled), None))
            call(L.vrc_nn_conv3x3_tc(_p(a), c, None, 0, 1, h, w, _p(wtc), _p(bias), c, 1, 2, _p(b), 0, _p(err), None))
            call(L.vrc_nn_conv3x3_fwd(_p(b), 1, h, w, c, _p(wt), _p(bias), c, 2, _p(a), 0, None))
            sums += [pooled.clone(), b.clone(), a.clone()]
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        seen.append(sums)
    assert all(torch.equal(x, y) for x, y in zip(*seen))
    assert all(bool(torch.isfinite(x.float()).all()) and float(x.float().abs().sum()) > 0 for x in seen[0])
