"""The device memory that a context keeps for its next volume: who may free a
volume and when, and who gets the memory back."""
import gc
import threading

import numpy as np
import pytest

import voreen_gb300 as v
from voreen_gb300 import synth

pytestmark = pytest.mark.gpu
MIB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _voxels(n, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    vox = torch.randint(0, 256, (n, n, n), dtype=torch.uint8, device="cuda", generator=g)
    torch.cuda.synchronize()
    return vox


def _volume(ctx, n=256, seed=1):
    return v.Volume(ctx, _voxels(n, seed))


def _frame(ctx, vol, out=None):
    p = v.default_params(128, 96)
    pos, focus, near, far = synth.orbit_camera(vol.dims, (1.0, 1.0, 1.0), 30.0, 20.0, 1.1)
    p.camera, p.entry_exit_mode = v.make_camera(pos, focus, near=near, far=far), v.EE_ANALYTIC
    tf = v.TransferFunction(ctx, v.TransferFunction.bake([(0.0, (0, 0, 0, 0)), (1.0, (255, 200, 100, 60))], 256), (0.0, 1.0))
    image, _ = v.render(ctx, vol, tf, p, out_format=v.OUT_RGBA32F)
    tf.close()
    return np.array(image)


def test_volume_destroyed_while_another_stream_captures(vrc_lib):
    """A thread frees volumes while another one captures a graph (thread-local
    mode): the capture is not touched, the memory serves the next volume."""
    import torch
    ctx = v.Context(0)
    want = _frame(ctx, _volume(ctx, seed=2))
    vol = _volume(ctx)
    _frame(ctx, vol)
    a = torch.zeros(1024, device="cuda")
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        graph.capture_begin(capture_error_mode="thread_local")
        a.add_(1.0)
        t = threading.Thread(target=vol.close)
        t.start()
        t.join()
        a.add_(1.0)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert bool((a == 2.0).all())
    np.testing.assert_array_equal(_frame(ctx, _volume(ctx, seed=2)), want)
    ctx.close()


def test_volume_destroyed_under_a_frame_on_another_stream(vrc_lib):
    """A frame that vrc_render_noalloc has queued on the caller's stream, behind
    other work, shows the volume it was given, though that was destroyed and
    the next one uploaded meanwhile."""
    import torch
    ctx = v.Context(0)
    p = v.default_params(128, 96)
    tf = v.TransferFunction(ctx, v.TransferFunction.bake([(0.0, (0, 0, 0, 0)), (1.0, (255, 200, 100, 60))], 256), (0.0, 1.0))
    busy, side = torch.ones(1 << 28, device="cuda"), torch.cuda.Stream()
    seen, first, second = [], _voxels(256, 1), _voxels(256, 3)
    for hurry in (False, True):
        vol = v.Volume(ctx, first)
        pos, focus, near, far = synth.orbit_camera(vol.dims, (1.0, 1.0, 1.0), 30.0, 20.0, 1.1)
        p.camera, p.entry_exit_mode = v.make_camera(pos, focus, near=near, far=far), v.EE_ANALYTIC
        out = torch.zeros((96, 128, 4), device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            for _ in range(60):  # some 20 ms
                busy.mul_(1.0)
        v.render_noalloc(vol, tf, p, None, None, out, v.OUT_RGBA32F, side.cuda_stream)
        if not hurry:
            torch.cuda.synchronize()
        vol.close()
        other = v.Volume(ctx, second)
        torch.cuda.synchronize()
        seen.append(out.cpu().numpy())
        other.close()
    assert seen[0].any()
    np.testing.assert_array_equal(seen[0], seen[1])
    tf.close()
    ctx.close()


def test_failing_allocations_give_the_memory_back(vrc_lib, tmp_path):
    """An allocation of the context that finds no memory: what the context keeps
    goes back first (a file of 550 GB of voxels; the volume itself)."""
    import torch
    ctx = v.Context(0)
    raw = tmp_path / "huge.raw"
    raw.write_bytes(b"\0" * 64)
    (tmp_path / "huge.vvd").write_text(
        '<?xml version="1.0" ?><VoreenData version="1"><Volumes><Volume><RawData filename="huge.raw" format="uint8" x="8192" '
        'y="8192" z="8192" /></Volume></Volumes></VoreenData>')
    desc = v.make_desc(v.U8, (8192, 8192, 8192))
    one = torch.zeros(64, dtype=torch.uint8, device="cuda")

    def load():
        v.Volume.load_vvd(ctx, str(tmp_path / "huge.vvd"))

    def upload():
        import ctypes as C
        h = C.c_void_p()
        st = v.lib().vrc_volume_upload(ctx.handle, C.byref(desc), C.c_void_p(one.data_ptr()), 1, 0, C.byref(h))
        if st:
            raise v.VrcError(st, "upload")

    for call in (load, upload, ctx.trim):
        vol, host = _volume(ctx, 512), v.Volume(ctx, np.ones((250, 512, 512), np.uint8))
        torch.cuda.empty_cache()
        for x in (host, vol):
            x.close()
        held = _free()
        if call != ctx.trim:
            with pytest.raises(v.VrcError, match="OUT_OF_MEMORY"):
                call()
        else:
            call()
        # the 512^3 volume's block (214 MB) and the staging of the other (66 MB)
        assert _free() - held >= 260 * MIB, call
    vol = _volume(ctx, 512)  # and no error is left for the next call's launches
    vol.close()
    ctx.close()


def test_captured_frames_keep_what_they_read(vrc_lib):
    """A graph of a frame whose maps it builds, replayed on another stream, behind
    other work: memory given back, and the volume destroyed and the next one
    uploaded meanwhile, do not reach it."""
    import torch
    ctx = v.Context(0)
    first, second = _voxels(256, 1), _voxels(256, 3)
    rgba = v.TransferFunction.bake([(0.0, (0, 0, 0, 0)), (0.5, (0, 0, 0, 0)), (1.0, (255, 200, 100, 60))], 256)
    vol = v.Volume(ctx, first)
    p = v.default_params(128, 96)
    pos, focus, near, far = synth.orbit_camera(vol.dims, (1.0, 1.0, 1.0), 30.0, 20.0, 1.1)
    p.camera, p.entry_exit_mode = v.make_camera(pos, focus, near=near, far=far), v.EE_ANALYTIC
    tfs = [v.TransferFunction(ctx, rgba, (0.0, 1.0)) for _ in range(2)]
    want = np.array(v.render(ctx, vol, tfs[0], p, out_format=v.OUT_RGBA32F)[0])
    v.render(ctx, vol, tfs[1], p, out_format=v.OUT_RGBA32F)  # its alpha table
    v.render(ctx, vol, tfs[0], p, out_format=v.OUT_RGBA32F)  # the maps are of the other one again
    out, busy = torch.zeros((96, 128, 4), device="cuda"), torch.ones(1 << 28, device="cuda")
    torch.cuda.synchronize()
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(ctx.stream)):
        v.render_async(ctx, vol, tfs[1], p, None, None, out)
    ctx.trim()
    spoil = torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda")  # where the scratch would have been
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(60):  # some 20 ms
            busy.mul_(1.0)
        graph.replay()
    vol.close()
    other = v.Volume(ctx, second)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    assert want.any() and bool((spoil == 255).all())
    del graph
    for x in (other, *tfs, ctx):
        x.close()


def test_a_refused_frame_does_not_count_as_one_on_another_stream(vrc_lib):
    """Volumes too large for vrc_render_noalloc's scratch (the learned form's
    probe asks first) leave their memory to the next volume, like others."""
    import torch
    ctx = v.Context(0)
    vol = _volume(ctx, 512)
    p = v.default_params(32, 32)
    p.entry_exit_mode, p.skip_cell_size = v.EE_ANALYTIC, 2
    p.camera = v.make_camera((256, 256, 1500), (256, 256, 256), near=1.0, far=3000.0)
    tf = v.TransferFunction(ctx, v.TransferFunction.bake([(0.0, (0, 0, 0, 0)), (1.0, (255, 255, 255, 255))], 256))
    with pytest.raises(v.VrcError) as ei:
        v.render_noalloc(vol, tf, p, None, None, torch.zeros((32, 32, 4), device="cuda"), v.OUT_RGBA32F, ctx.stream)
    assert ei.value.status == 8
    tf.close()
    before = _free()
    vol.close()
    assert _free() - before < MIB
    ctx.close()


def test_scratch_of_the_maps_is_taken_only_to_build_them(vrc_lib):
    """Frames whose maps are there take no scratch; one that builds them takes it
    again after it was given back: the same image each time."""
    ctx = v.Context(0)
    vol = _volume(ctx, 512)
    p = v.default_params(64, 48)
    pos, focus, near, far = synth.orbit_camera(vol.dims, (1.0, 1.0, 1.0), 30.0, 20.0, 1.1)
    p.camera, p.entry_exit_mode = v.make_camera(pos, focus, near=near, far=far), v.EE_ANALYTIC
    tfs = [v.TransferFunction(ctx, v.TransferFunction.bake([(0.0, (0, 0, 0, 0)), (1.0, (255, 200, 100, 60))], 256), (0.0, 1.0))
           for _ in range(2)]
    first = np.array(v.render(ctx, vol, tfs[0], p, out_format=v.OUT_RGBA32F)[0])
    held = _free()
    ctx.trim()
    trimmed = _free()
    assert trimmed - held >= 30 * MIB  # 2^24 cells
    np.testing.assert_array_equal(v.render(ctx, vol, tfs[0], p, out_format=v.OUT_RGBA32F)[0], first)
    assert _free() >= trimmed - MIB
    np.testing.assert_array_equal(v.render(ctx, vol, tfs[1], p, out_format=v.OUT_RGBA32F)[0], first)
    assert _free() < trimmed - 16 * MIB
    for x in (*tfs, vol, ctx):
        x.close()


def test_memory_returns_with_the_context_whoever_goes_first(vrc_lib):
    """A context closed before its volumes, and one after: nothing stays."""
    import torch
    c = v.Context(0)
    _frame(c, _volume(c, 64))
    c.close()
    gc.collect()
    torch.cuda.empty_cache()
    before = _free()
    for context_first in (True, False):
        ctx = v.Context(0)
        vol, host = _volume(ctx, 512), v.Volume(ctx, np.ones((200, 512, 512), np.uint8))
        _frame(ctx, vol)
        for x in (ctx, vol, host) if context_first else (vol, host, ctx):
            x.close()
        torch.cuda.empty_cache()
        assert _free() >= before - 4 * MIB, context_first
