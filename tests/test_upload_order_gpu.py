"""Host voxels are copied on a stream of their own, through memory that the context
keeps: their place among the work of the context, which is ordered on the
context's stream, and uploads of several threads."""
import threading

import numpy as np
import pytest

import voreen_gb300 as v

pytestmark = pytest.mark.gpu


def _brick_minmax(vox, brick=32):
    Z, Y, X = vox.shape
    parts = [vox[z:z + brick + 1, y:y + brick + 1, x:x + brick + 1]
             for z in range(0, Z, brick) for y in range(0, Y, brick) for x in range(0, X, brick)]
    unit = np.float32(np.iinfo(vox.dtype).max)
    return (np.array([np.float32(p.min()) / unit for p in parts]), np.array([np.float32(p.max()) / unit for p in parts]))


@pytest.mark.parametrize("dims", [(70, 50, 40), (1024, 1024, 150)])  # one slab, and three
def test_upload_waits_for_the_context_stream(ctx, dims):
    """Pinned voxels that work queued on the context's stream is still to write
    are uploaded as that work leaves them, also into memory that the volume
    before left behind."""
    import torch
    vox = np.random.default_rng(dims[0]).integers(1, 256, dims[::-1], dtype=np.uint8)
    want = _brick_minmax(vox)
    stream = torch.cuda.ExternalStream(ctx.stream)
    fresh, busy = torch.from_numpy(vox).cuda(), torch.ones(1 << 28, device="cuda")
    pinned = torch.empty(dims[::-1], dtype=torch.uint8, pin_memory=True)
    torch.cuda.synchronize()
    for _ in range(2):
        pinned.zero_()
        with torch.cuda.stream(stream):
            for _ in range(60):  # some 20 ms
                busy.mul_(1.0)
            pinned.copy_(fresh, non_blocking=True)
        vol = v.Volume(ctx, pinned.numpy())
        lo, hi, _ = vol.brick_minmax()
        vol.close()
        np.testing.assert_array_equal(lo, want[0])
        np.testing.assert_array_equal(hi, want[1])


def test_uploads_of_two_threads_share_a_context(ctx):
    """Each thread's volumes hold its own voxels (three slabs each; the calls
    release the interpreter lock)."""
    voxels = [np.random.default_rng(k).integers(0, 256, (150, 1024, 1024), dtype=np.uint8) for k in range(2)]
    want = [_brick_minmax(vox) for vox in voxels]
    wrong, start = [], threading.Barrier(2)

    def upload(k):
        start.wait(60)
        for _ in range(6):
            vol = v.Volume(ctx, voxels[k])
            lo, hi, _ = vol.brick_minmax()
            vol.close()
            if not (np.array_equal(lo, want[k][0]) and np.array_equal(hi, want[k][1])):
                wrong.append(k)

    threads = [threading.Thread(target=upload, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
