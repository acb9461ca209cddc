"""Upload tables: per-brick min/max (the end of the chain voxels -> 2^3 cells ->
... -> bricks) against numpy over the voxels, for row lengths on both sides of
the wide-load rule, every brick edge and type; and the distance field on grids
whose rows are and are not multiples of four cells, to each side of the cap
and of a word of bits."""
import ctypes as C

import numpy as np
import pytest

import voreen_gb300 as v
from voreen_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 33, 40), (8, 8, 8), (72, 70, 3), (65, 64, 66), (1, 5, 131), (40, 1, 1)])
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
@pytest.mark.parametrize("brick", [8, 16, 32, 64])
def test_brick_minmax_is_the_voxels(ctx, dims, dtype, brick):
    rng = np.random.default_rng(sum(dims) + brick)
    X, Y, Z = dims
    if dtype == np.float32:
        vox = rng.normal(0.0, 3.0, (Z, Y, X)).astype(np.float32)
    else:
        vox = rng.integers(0, np.iinfo(dtype).max + 1, (Z, Y, X)).astype(dtype)
    vol = v.Volume(ctx, vox, brick_size=brick)
    mn, mx, nb = vol.brick_minmax()
    assert nb == tuple((d + brick - 1) // brick for d in dims)
    unit = np.float32(1.0 if dtype == np.float32 else np.iinfo(dtype).max)
    k = 0
    for z in range(0, Z, brick):
        for y in range(0, Y, brick):
            for x in range(0, X, brick):
                part = vox[z:z + brick + 1, y:y + brick + 1, x:x + brick + 1]
                assert mn[k] == np.float32(part.min()) / unit and mx[k] == np.float32(part.max()) / unit, (x, y, z)
                k += 1
    vol.close()


@pytest.mark.parametrize("shape", [(3, 5, 4), (2, 3, 1), (40, 33, 61), (20, 36, 64), (17, 18, 50), (1, 1, 200), (34, 2, 31)])
@pytest.mark.parametrize("share", [0.0, 0.0005, 0.02, 1.0])
def test_distance_field_on_any_row_length(ctx, shape, share):
    import torch
    nz, ny, nx = shape
    rng = np.random.default_rng(nx * 7 + ny)
    occ = rng.random(shape) < share
    if share and not occ.any():
        occ[nz // 2, ny // 2, nx // 2] = True
    flat = np.zeros((occ.size + 31) // 32 * 32, np.uint8)
    flat[: occ.size] = occ.reshape(-1)
    bits = torch.from_numpy(np.packbits(flat, bitorder="little").view(np.int32).copy()).cuda()
    buf = torch.full((occ.size + 16,), 77, dtype=torch.uint8, device="cuda")
    want = np.full(shape, 16, np.int64)
    z, y, x = np.meshgrid(*(np.arange(n) for n in shape), indexing="ij")
    for pz, py, px in np.argwhere(occ) if share < 1.0 else []:
        np.minimum(want, np.maximum(np.maximum(abs(z - pz), abs(y - py)), abs(x - px)), out=want)
    if share == 1.0:
        want[:] = 0
    for shift in (0, 3):  # an output that starts on a word, and one that does not
        buf.fill_(77)
        torch.cuda.synchronize()
        out = buf[shift:]
        assert v.lib().vrc_occupancy_distance(ctx.handle, C.c_void_p(bits.data_ptr()), nx, ny, nz,
                                              C.c_void_p(out.data_ptr())) == 0
        got = buf.cpu().numpy()
        np.testing.assert_array_equal(got[shift:shift + occ.size].reshape(shape), want)
        assert (got[:shift] == 77).all() and (got[shift + occ.size:] == 77).all()


@pytest.mark.parametrize("shape", [(17, 130, 64), (9, 33, 460), (33, 65, 78), (1, 2100, 61), (140, 31, 17), (24, 70, 144)])
@pytest.mark.parametrize("share", [0.0, 2e-5, 0.002, 1.0])
def test_distance_field_by_bit_planes(ctx, shape, share):
    """Maps large enough for the bit planes: rows of whole and partial words,
    outputs that start on 16 bytes and that do not, every distance up to the cap."""
    import torch
    from scipy import ndimage
    nz, ny, nx = shape
    occ = np.random.default_rng(nx + ny).random(shape) < share
    if share == 2e-5:
        occ[-1, -1, -1] = occ[0, ny // 3, 0] = True
    want = np.minimum(ndimage.distance_transform_cdt(~occ, "chessboard"), 16) if occ.any() else np.full(shape, 16)
    flat = np.zeros((occ.size + 31) // 32 * 32, np.uint8)
    flat[: occ.size] = occ.reshape(-1)
    bits = torch.from_numpy(np.packbits(flat, bitorder="little").view(np.int32).copy()).cuda()
    buf = torch.full((occ.size + 16,), 77, dtype=torch.uint8, device="cuda")
    for shift in (0, 4, 3):
        buf.fill_(77)
        torch.cuda.synchronize()
        assert v.lib().vrc_occupancy_distance(ctx.handle, C.c_void_p(bits.data_ptr()), nx, ny, nz,
                                              C.c_void_p(buf[shift:].data_ptr())) == 0
        got = buf.cpu().numpy()
        np.testing.assert_array_equal(got[shift:shift + occ.size].reshape(shape), want)
        assert (got[:shift] == 77).all() and (got[shift + occ.size:] == 77).all()


@pytest.mark.parametrize("dims,dtype,brick", [((2048, 1400, 70), np.uint8, 8), ((1203, 1100, 67), np.uint16, 16),
                                              ((2501, 1999, 99), np.uint8, 32), ((1024, 640, 131), np.float32, 64)])
def test_slabs_of_host_voxels_are_the_device_volume(ctx, dims, dtype, brick):
    """Host voxels come in slabs through a ring of slices, device voxels at
    once: the same tables and the same image, also from memory that another
    volume left behind."""
    import torch
    rng = np.random.default_rng(dims[0])
    vox = rng.integers(0, 251, dims[::-1], dtype=np.uint8)
    vox = {np.uint8: lambda x: x, np.uint16: lambda x: x.astype(np.uint16) * np.uint16(257),
           np.float32: lambda x: x.astype(np.float32) / np.float32(250)}[dtype](vox)
    p = v.default_params(96, 64)
    pos, focus, near, far = synth.orbit_camera(dims, (1.0, 1.0, 1.0), 30.0, 20.0, 1.1)
    p.camera, p.sampling_rate, p.entry_exit_mode = v.make_camera(pos, focus, near=near, far=far), 0.5, v.EE_ANALYTIC
    tf = v.TransferFunction(ctx, v.TransferFunction.bake(synth.tf_keys_trapezoids([0.25, 0.65], 3, alpha_range=(0.1, 0.5),
                                                                                 top=(0.02, 0.04)), 1024), (0.0, 1.0))
    seen = []
    for src in (vox, torch.from_numpy(vox).cuda(), vox):
        vol = v.Volume(ctx, src, brick_size=brick)
        lo, hi, _ = vol.brick_minmax()
        image, _ = v.render(ctx, vol, tf, p, out_format=v.OUT_RGBA32F)
        seen.append((vol.minmax(), np.array(lo), np.array(hi), np.array(image)))
        vol.close()
    for got in seen[1:]:
        assert got[0] == seen[0][0]
        for a, b in zip(got[1:], seen[0][1:]):
            np.testing.assert_array_equal(a, b)
    assert seen[0][3].any()
