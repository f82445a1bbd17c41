"""BEV volume to patient grid, dense and supersampled, against the double-precision
oracle at the sizes where the kernels' tiles, tail loops and culling can go wrong.

Tolerance: a sample's place in the beam frame is a sum of some eight float roundings
of coordinates no larger than the farthest voxel's distance d from the source and
the patient grid's extent, so it is off by at most 8 * 2^-24 * d, in texels that
divided by the smallest texel met; the trilinear sample moves by at most the
largest texel value per texel and axis.  Voxels within rounding of the extent are
left out of the supersampled comparison, and so are voxels near the source plane,
where texels shrink to nothing."""
import ctypes as C

import numpy as np
import pytest

import oracle
from fastdose_b200 import _lib, api
from fastdose_b200.types import BEAM_DTYPE, make_volume

pytestmark = pytest.mark.gpu

VOX = 0.25
# dims, fmap, pixel (x, y), slices, sad, angles
GRIDS = {
    "tile_remainders": ((33, 17, 9), (12, 7), (0.2, 0.31), 40, 100.0, (0.7, 0.4, 0.2)),
    "smaller_than_a_tile": ((3, 5, 1), (9, 9), (0.3, 0.3), 30, 100.0, (2.1, -0.6, 0.3)),
    "whole_tiles": ((64, 40, 32), (16, 16), (0.25, 0.25), 60, 100.0, (1.2, 0.9, -0.3)),
    "one_texel_wide": ((40, 33, 18), (1, 16), (0.5, 0.25), 50, 100.0, (0.2, 0.0, 0.0)),
    "one_slice": ((35, 34, 21), (8, 8), (0.4, 0.4), 1, 100.0, (2.8, 1.1, 0.1)),
    "source_in_the_volume": ((48, 44, 37), (11, 11), (0.4, 0.4), 24, 3.0, (0.9, 0.5, 0.1)),
}


def _case(name):
    dim, fmap, pixel, slices, sad, angles = GRIDS[name]
    vol = make_volume(dim, (VOX,) * 3)
    b = np.zeros((), BEAM_DTYPE)
    b["isocenter"] = [n * VOX / 2 for n in dim]
    b["beamlet_size"] = pixel
    b["fmap_size"] = fmap
    b["sad"] = sad
    b["angles"] = angles
    b["long_spacing"] = 0.25
    b = api.calc_range(b, vol)
    b["long_dim"] = min(int(b["long_dim"]), slices)
    rng = np.random.default_rng(len(name))
    bev = (0.2 + rng.random((int(b["long_dim"]), fmap[1], fmap[0]))).astype(np.float32)
    return vol, b, bev


def _axes(b):
    """Unit vectors of the beam frame, by the oracle's rotation of the patient axes."""
    out = np.zeros((3, 3))
    for i in range(3):
        e, r = (C.c_float * 3)(*np.eye(3)[i]), (C.c_float * 3)()
        oracle.oracle.lib("double").or_rotate_beam_f(e, *(C.c_float(float(a)) for a in b["angles"]), r)
        out[:, i] = list(r)
    return out


def _run(ctx, vol, b, bev, ss, extent, pad):
    """The output rows `pad` floats longer than the grid, all floats -7 before."""
    import torch

    nx, ny, nz = (int(v) for v in vol["dim"])
    dens = api.Density(ctx, np.ones((nz, ny, nx), np.float32), vol)
    out = torch.full((nz, ny, nx + pad), -7.0, device="cuda")
    d_bev = torch.from_numpy(bev).cuda()
    bb = np.array(b, BEAM_DTYPE)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    args = [ctx.h, C.c_void_p(bb.ctypes.data), dens.h, p(d_bev), p(out), (nx + pad) * 4]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if ss:
        _lib.check(ctx.lib.fd2_bev2pvcs_supersampling(*args, ss, extent, st), "ss")
    else:
        _lib.check(ctx.lib.fd2_bev2pvcs(*args, st), "dense")
    torch.cuda.synchronize()
    o = out.cpu().numpy()
    assert np.all(o[:, :, nx:] == -7.0)
    return o[:, :, :nx]


def _frame(vol, b):
    """Beam-frame coordinates (x, depth, z) of the voxel centres."""
    nx, ny, nz = (int(v) for v in vol["dim"])
    z, y, x = np.meshgrid(*((np.arange(n) + 0.5) * VOX for n in (nz, ny, nx)), indexing="ij")
    q = np.stack([x, y, z]).reshape(3, -1) - np.asarray(b["source"], np.float64)[:, None]
    return (_axes(b) @ q).reshape(3, nz, ny, nx)


def _tolerance(vol, b, bev, near):
    v = _frame(vol, b)
    far = max(float(np.sqrt((v ** 2).sum(0)).max()), float((np.asarray(vol["dim"]) * VOX).max()))
    texel = float(np.min(b["beamlet_size"])) * max(near, float(np.abs(v[1]).min())) / float(b["sad"])
    return 3 * 8 * 2.0 ** -24 * far / min(texel, float(b["long_spacing"])) * float(bev.max())


@pytest.mark.parametrize("pad", [0, 5])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_dense(ctx, grid, pad):
    vol, b, bev = _case(grid)
    got = _run(ctx, vol, b, bev, 0, 0.0, pad)
    ref = oracle.bev2pvcs(b, bev, vol)
    near = 0.1 * float(b["sad"]) if grid == "source_in_the_volume" else 0.0
    on = np.abs(_frame(vol, b)[1]) >= near
    assert ref[on].max() > 0 and on.mean() > 0.8
    assert np.abs(got - ref)[on].max() <= _tolerance(vol, b, bev, near)
    assert np.all(got >= 0)  # every voxel written


@pytest.mark.parametrize("extent", [0.6, 2.0, 50.0])
@pytest.mark.parametrize("ss", [1, 2, 3, 4, 5, 6, 16])
@pytest.mark.parametrize("grid", list(GRIDS))
def test_supersampled(ctx, grid, ss, extent):
    vol, b, bev = _case(grid)
    got = _run(ctx, vol, b, bev, ss, extent, 3)
    nx, ny, nz = (int(v) for v in vol["dim"])
    ref = oracle.bev2pvcs_ss(b, bev, vol, ssfactor=ss, extent=extent, out=np.full((nz, ny, nx), -7.0, np.float32))
    v = _frame(vol, b)
    near = 0.1 * float(b["sad"]) + VOX if grid == "source_in_the_volume" else 0.0
    on = (np.abs(np.hypot(v[0], v[2]) - extent) > 1e-3) & (np.abs(v[1]) >= near)
    tol = _tolerance(vol, b, bev, near - VOX if near else 0.0)
    # written where the samples add up to 1e-4 or more: at that line one side may leave a voxel alone
    g, r = np.where(got == -7.0, 0.0, got), np.where(ref == -7.0, 0.0, ref)
    assert (ref != -7.0).any() or (grid, ss, extent) == ("one_slice", 1, 0.6)
    assert np.abs(g - r)[on].max() <= tol + 1e-4 / ss ** 3
    clear = on & (np.abs(r) > tol + 1e-4 / ss ** 3)
    assert np.array_equal((got != -7.0)[clear], (ref != -7.0)[clear])
    assert np.all(got[on & (np.hypot(v[0], v[2]) > extent)] == -7.0)
