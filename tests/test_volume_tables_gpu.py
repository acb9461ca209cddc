"""Upload tables: per-brick min/max (the end of the chain voxels -> 2^3 cells ->
... -> bricks) against numpy over the voxels, for row lengths on both sides of
the wide-load rule, every brick edge and type; and the distance field on grids
whose rows are and are not multiples of four cells, to each side of the cap
and of a word of bits."""
import ctypes as C

import numpy as np
import pytest

import voreen_gb300 as v

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
