"""The march's shortcuts around a division and around per-sample steps
(march_core.cuh), restated with exact rationals: the transfer-function
coordinate as a product corrected twice by its residual equals the correctly
rounded quotient, and the closed-form jump over an empty run lands where the
one-at-a-time accumulation does. On the GPU: transfer-function domains on
both sides of the rule that chooses between product and division."""
from fractions import Fraction as F

import numpy as np
import pytest

f32 = np.float32
CAP = 255 * 255


def rn(q: F) -> float:
    """The binary32 value nearest to q (ties to even), q in the normal range or 0."""
    if q == 0:
        return 0.0
    n, d = abs(q.numerator), q.denominator
    e = n.bit_length() - d.bit_length()
    e -= F(n, d) < F(2) ** e
    u = F(2) ** max(e - 23, -149)
    k = abs(q) / u
    m = k.numerator // k.denominator
    r = k - m
    m += r > F(1, 2) or (r == F(1, 2) and m & 1)
    return float(m * u) * (1 if q > 0 else -1)


def coordinate(rw, lo, hi):
    b = float(f32(hi) - f32(lo))
    rcp = float(f32(1) / f32(b))
    a = float(f32(min(max(rw, lo), hi)) - f32(lo))
    q = float(f32(a) * f32(rcp))
    for _ in range(2):
        q = rn(F(rn(F(a) - F(q) * F(b))) * F(rcp) + F(q))
    return q


@pytest.mark.parametrize("width", [2.0 ** -59, 1e-12, 3e-4, 0.06248, 1.0, 1.9999999, 4095.0, 2.0 ** 59])
def test_tf_coordinate_is_the_rounded_quotient(width):
    rng = np.random.default_rng(5)
    for k in range(400):
        lo = float(f32(rng.choice([0.0, 0.25 * width, -0.5 * width, 3.0 * width])))
        hi = float(f32(lo) + f32(width * (1.0 + 0.3 * rng.random())))
        rw = float(f32(lo + (hi - lo) * rng.random() * (1.0 if k % 3 else 2.0 ** -rng.integers(1, 24))))
        rw = min(max(rw, lo), hi)
        b, a = F(float(f32(hi) - f32(lo))), F(float(f32(rw) - f32(lo)))
        assert coordinate(rw, lo, hi) == rn(a / b), (rw, lo, hi)
    assert coordinate(hi, lo, hi) == 1.0 and coordinate(lo, lo, hi) == 0.0


def jump(t, loop, step, lim):
    """march_core.cuh: jump_empty_run; the reciprocal taken one ulp high and low."""
    T = f32(2.0) ** f32(np.floor(np.log2(t)))
    q = f32(f32(T + step) - T)
    if not T > 2.0 ** -90 or step >= T or not q > 0 or abs(f32(step - q)) == f32(T * f32(2.0 ** -24)):
        return [(t, loop)]
    out = []
    r = f32(1) / q
    for rcp in (np.nextafter(r, f32(0)), r, np.nextafter(r, f32(np.inf))):
        x = f32(f32(min(lim, f32(f32(2) * T - q)) - t) * rcp)
        n = min(int(x), CAP - loop)
        out.append((t, loop) if n <= 0 else (f32(t + f32(f32(n) * q)), loop + n))
    return out


def test_jump_lands_on_the_accumulated_parameter():
    rng = np.random.default_rng(2)
    for _ in range(4000):
        step = f32(1.0 / (f32(rng.choice([33, 64, 255, 512, 1000, 2048, 3000, 65536])) *
                          f32(rng.choice([0.5, 1, 1.5, 2, 3, 7.3, 40]))))
        t = max(f32(rng.uniform(0, 1.7)), step)
        lim = f32(t + f32(rng.uniform(0, 0.3)))
        loop = int(rng.choice([0, 10, CAP - 3]))
        for tj, lj in jump(t, loop, step, lim):
            assert lj <= CAP
            te, le = t, loop
            while le < lj:  # every sample jumped over lies in the run
                assert te <= lim
                te, le = f32(te + step), le + 1
            assert te == tj


@pytest.mark.gpu
@pytest.mark.parametrize("width", [1e-25, 2.0 ** -58, 0.5, 2.0 ** 59, 1e25])
@pytest.mark.parametrize("brick", [16, 32])
def test_tf_domain_widths_match_the_oracle(ctx, width, brick):
    """Domains whose width takes the corrected product and the division, and
    compile-time and run-time brick geometry, bit for bit."""
    import voreen_gb300 as v
    from helpers import Case
    rng = np.random.default_rng(9)
    vox = (rng.random((37, 35, 41)) * width).astype(np.float32)
    vox[0, 0, :3] = [np.nan, np.inf, -np.inf]
    keys = [(0.0, (0, 0, 255, 0)), (0.4, (0, 255, 0, 20)), (1.0, (255, 0, 0, 200))]
    p = v.default_params(61, 47)
    p.camera = v.make_camera((80.0, 60.0, 90.0), (20.0, 17.0, 18.0), near=1.0, far=400.0)
    c = Case(ctx, vox, v.TransferFunction.bake(keys, 4096), (0.1 * width, 0.9 * width), p, brick=brick)
    img, st = c.gpu()
    o32, s32, _ = c.oracle(32)
    assert (img[..., 3] > 0).any() and st.samples == s32.sum()
    np.testing.assert_array_equal(img.view(np.uint32), o32.view(np.uint32))
