"""The ways a frame's rays are spread over lanes (several lanes a ray for small
images, one lane and a queue of unfinished rays, one lane): every mode on image
sizes to each side of the rules' lines gives the pixels, sample counts and
auxiliary image of the same rays marched in one call of another size class."""
import ctypes as C

import numpy as np
import pytest

import voreen_gb300 as v
from voreen_gb300 import synth

pytestmark = pytest.mark.gpu


def _setup(ctx, dtype):
    dims = (70, 61, 53)
    vox = synth.synth_volume(synth.SHELLS, dtype, dims, 77)
    scale = {v.U8: 255.0, v.U16: 65535.0, v.F32: 1.0}[dtype]
    keys = synth.tf_keys_trapezoids([0.25, 0.45, 0.65, 0.8], 3, alpha_range=(0.1, 0.5), top=(0.02, 0.04))
    vol = v.Volume(ctx, vox, (0.8, 1.0, 1.1))
    tf = v.TransferFunction(ctx, v.TransferFunction.bake(keys, 1024), (float(vox.min()) / scale, float(vox.max()) / scale))
    pos, focus, near, far = synth.orbit_camera(dims, (0.8, 1.0, 1.1), 30.0, 20.0, 1.1)
    return vol, tf, v.make_camera(pos, focus, near=near, far=far), pos


def _render(ctx, vol, tf, p, region):
    """Image, auxiliary image and stats of a pixel window (vrc_render_aux)."""
    import torch
    img = torch.zeros((p.height, p.width, 4), dtype=torch.float32, device="cuda")
    aux = torch.zeros((p.height, p.width, 2), dtype=torch.float32, device="cuda")
    p.region[:] = list(region)
    torch.cuda.synchronize()
    st = v.RenderStats()
    r = v.lib().vrc_render_aux(ctx.handle, vol.handle, tf.handle, C.byref(p), None, None, C.c_void_p(img.data_ptr()),
                               v.OUT_RGBA32F, C.c_void_p(aux.data_ptr()), C.byref(st))
    assert r == 0
    x, y, w, h = region
    return img[y:y + h, x:x + w].cpu().numpy(), aux[y:y + h, x:x + w].cpu().numpy(), st


# one window of a frame takes one lane count, its quarters and strips others:
# 1920x1080 = 64,800 tiles (queue / one lane), 640x540 = 10,800 (4 lanes),
# 1921 x 270 = 16,388 (queue / 2 lanes), 480x360 and odd rests (8 lanes)
@pytest.mark.parametrize("dtype", [v.U8, v.U16, v.F32])
@pytest.mark.parametrize("comp,shade", [(v.DVR, 1), (v.DVR, 0), (v.ISO, 1), (v.MIP, 0), (v.MOP, 1), (v.MIDA, 1)])
def test_lanes_per_ray_agree(ctx, dtype, comp, shade):
    vol, tf, cam, pos = _setup(ctx, dtype)
    p = v.default_params(1923, 1081)
    p.camera, p.compositing, p.shading = cam, comp, shade
    p.light_position[:] = [*pos, 1.0]
    p.entry_exit_mode, p.iso_value, p.mida_gamma = v.EE_ANALYTIC, 0.3, 0.4
    whole, aux, st = _render(ctx, vol, tf, p, (0, 0, 1923, 1081))
    assert (whole[..., 3] > 0).any()
    got, got_aux = np.empty_like(whole), np.empty_like(aux)
    samples = shaded = 0
    windows = [(0, 0, 1923, 270), (0, 270, 640, 540), (640, 270, 640, 540), (1280, 270, 643, 540)]
    windows += [(x, 810, w, 271) for x, w in ((0, 480), (480, 7), (487, 1), (488, 952), (1440, 483))]
    for x, y, w, h in windows:
        a, b, s = _render(ctx, vol, tf, p, (x, y, w, h))
        got[y:y + h, x:x + w], got_aux[y:y + h, x:x + w] = a, b
        samples += s.samples
        shaded += s.samples_shaded
    np.testing.assert_array_equal(got.view(np.uint32), whole.view(np.uint32))
    np.testing.assert_array_equal(got_aux.view(np.uint32), aux.view(np.uint32))
    assert samples == st.samples and shaded == st.samples_shaded


@pytest.mark.parametrize("size", [(1, 1), (3, 2), (31, 5), (700, 500), (1921, 300)])
@pytest.mark.parametrize("ert", [-1.0, 0.0, 0.3, 2.0])
def test_early_termination_in_a_group(ctx, size, ert):
    """The sample a ray ends at does not depend on its lanes, whatever the threshold."""
    vol, tf, cam, _ = _setup(ctx, v.U16)
    p = v.default_params(*size)
    p.camera, p.ert_threshold, p.entry_exit_mode = cam, ert, v.EE_ANALYTIC
    q = v.default_params(*size)
    C.memmove(C.byref(q), C.byref(p), C.sizeof(p))
    a, sa = v.render(ctx, vol, tf, p, None, None, v.OUT_RGBA32F)
    # pre-integration's sibling path: brick size 16 takes one lane a ray at every size
    vox = synth.synth_volume(synth.SHELLS, v.U16, (70, 61, 53), 77)
    vol16 = v.Volume(ctx, vox, (0.8, 1.0, 1.1), brick_size=16)
    b, sb = v.render(ctx, vol16, tf, q, None, None, v.OUT_RGBA32F)
    np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
    assert sa.samples == sb.samples


@pytest.mark.parametrize("rate", [0.7, 1.0, 2.0, 3.3])  # steps above and below a voxel: without and with the run rule
@pytest.mark.parametrize("shade", [0, 1])
@pytest.mark.parametrize("dtype", [v.U8, v.F32])
def test_preintegration_lanes_agree(ctx, dtype, shade, rate):
    """Pre-integration on several lanes a ray, with the queue and on one lane
    (16^3 bricks): image, auxiliary image, samples, with and without skipping,
    early termination off and on."""
    dims = (70, 61, 53)
    vox = synth.synth_volume(synth.SHELLS, dtype, dims, 77)
    unit = {v.U8: 255.0, v.F32: 1.0}[dtype]
    keys = synth.tf_keys_trapezoids([0.25, 0.45, 0.65, 0.8], 3, alpha_range=(0.1, 0.5), top=(0.02, 0.04))
    vols = [v.Volume(ctx, vox, (0.8, 1.0, 1.1), brick_size=b) for b in (32, 16)]
    tf = v.TransferFunction(ctx, v.TransferFunction.bake(keys, 1024), (float(vox.min()) / unit, float(vox.max()) / unit))
    table = v.PreIntegrationTable(ctx, v.PreIntegrationTable.bake_source(keys, 256), v.sampling_step(vols[0], rate))
    tf.set_preintegration(table)
    pos, focus, near, far = synth.orbit_camera(dims, (0.8, 1.0, 1.1), 30.0, 20.0, 1.1)
    for width, height in ((203, 151), (641, 360), (1403, 320)):  # 8 lanes, 4 lanes, queue
        for skip, ert in ((1, 0.95), (0, 0.95), (1, 1.5), (1, 0.0)):
            got = []
            for vol in vols:
                p = v.default_params(width, height)
                p.camera = v.make_camera(pos, focus, near=near, far=far)
                p.light_position[:] = [*pos, 1.0]
                p.sampling_rate, p.shading, p.ert_threshold = rate, shade, ert
                p.empty_space_skipping, p.entry_exit_mode = skip, v.EE_ANALYTIC
                p.classification = v.CLASSIFY_PREINTEGRATED
                got.append(_render(ctx, vol, tf, p, (0, 0, width, height)))
            (a, ax, sa), (b, bx, sb) = got
            np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
            np.testing.assert_array_equal(ax.view(np.uint32), bx.view(np.uint32))
            assert sa.samples == sb.samples and (ert == 0.0 or (a[..., 3] > 0).any())
    tf.close()
    table.close()
