"""The learned form's chained launches on streams of their own, one and two at a
time: the bits of the same calls with a synchronisation after each."""
import ctypes as C

import pytest

import voreen_gb300 as v

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("h,w", [(70, 130), (200, 312)])
def test_chains_on_streams_of_their_own(vrc_lib, h, w):
    import torch
    L, c = v.lib(), 64

    class Chain:
        """Layers that read what the launch before wrote, into buffers that the
        launch before that read, with weights that another kernel just changed."""

        def __init__(self, seed, stream):
            g = torch.Generator(device="cuda").manual_seed(seed)
            self.stream, self.sums = stream, []
            self.a = torch.randn((1, h, w, c), device="cuda", generator=g).to(torch.bfloat16)
            self.b = torch.zeros_like(self.a)
            self.pooled = torch.zeros((1, h // 2, w // 2, c), dtype=torch.bfloat16, device="cuda")
            self.w0 = (torch.randn((c, 3, 3, c), device="cuda", generator=g) * 0.05).to(torch.bfloat16)
            self.wt, self.wtc = self.w0.clone(), torch.empty_like(self.w0)
            self.bias = torch.randn(c, device="cuda", generator=g) * 0.1
            self.err = torch.zeros(1, dtype=torch.int32, device="cuda")

        def step(self, i, wait):
            s = C.c_void_p(self.stream.cuda_stream)
            a, b, wt, wtc, bias = (_p(t) for t in (self.a, self.b, self.wt, self.wtc, self.bias))

            def call(r):
                assert r == 0
                if wait:
                    torch.cuda.synchronize()

            with torch.cuda.stream(self.stream):
                self.wt.copy_(torch.roll(self.w0, i, 0))
                call(L.vrc_nn_weights_tc(wt, c, c, 0, 1, wtc, s))
                call(L.vrc_nn_conv3x3_fwd(a, 1, h, w, c, wt, bias, c, 2, b, 0, s))
                call(L.vrc_nn_conv3x3_tc(b, c, None, 0, 1, h, w, wtc, bias, c, 1, 2, a, 0, _p(self.err), s))
                call(L.vrc_nn_avgpool2(a, 1, h, w, c, C.c_float(1.0), _p(self.pooled), s))
                call(L.vrc_nn_conv3x3_fwd(a, 1, h, w, c, wt, bias, c, 2, b, 0, s))
                call(L.vrc_nn_conv3x3_tc(b, c, None, 0, 1, h, w, wtc, bias, c, 1, 2, a, 0, _p(self.err), s))
                self.sums += [self.pooled.clone(), self.a.clone(), self.b.clone()]

    seen = []
    for wait in (True, False):
        chains = [Chain(k, torch.cuda.Stream()) for k in range(2)]
        torch.cuda.synchronize()
        for i in range(10):
            for chain in chains:
                chain.step(i, wait)
        torch.cuda.synchronize()
        assert all(int(chain.err.item()) == 0 for chain in chains)
        seen.append([t for chain in chains for t in chain.sums])
    assert all(torch.equal(x, y) for x, y in zip(*seen))
    assert all(bool(torch.isfinite(x.float()).all()) and float(x.float().abs().sum()) > 0 for x in seen[0])
