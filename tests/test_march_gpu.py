"""The voxel-stationary CCCS march (8x8, 12x12 and 16x16 maps) against the
general per-ray instance, which a call with maps of two sizes takes.

Both take the same discrete steps (the same float comparisons); a voxel's dose
is a sum of at most a few hundred positive deposits in FP32, each a product of a
few rounded factors, so the two agree to 300 * 2^-24 = 2e-5 of the voxel and,
where the path sums nearly cancel against the 1e-4 of the normalisation, to
1e-6 of the maximum."""
import ctypes as C

import numpy as np
import pytest

from fastdose_b200 import _lib, api, phantoms
from fastdose_b200.types import make_bundle

pytestmark = pytest.mark.gpu


def _batch(ctx, ph, side, on, dens, spec, gantry, count=6, beamlet_size=0.5):
    bund = make_bundle(ph.centre(), (gantry, 0.3, 0.1), sad=100.0, fluence_dim=count, beamlet_size=beamlet_size,
                       sub_fluence_dim=side, sub_fluence_on=on, long_spacing=0.25)
    flags = np.zeros(count * count, np.uint8)
    flags[:: max(1, count * count // count)] = 1  # distinct beamlet sizes: distinct ray paths
    b = api.BEVBatch(api.bundle_beamlets(bund, flags, ph.volume))
    api.TermaComputeCollective(ctx, b, api.beamlet_fluence(bund), dens, spec)
    return b


@pytest.mark.parametrize("n_phi", [1, 4, 6, 8])
@pytest.mark.parametrize("side,on", [(8, 2), (12, 4), (16, 4)])
def test_march_matches_the_per_ray_instance(ctx, side, on, n_phi):
    import torch

    ph = phantoms.torso_phantom(seed=side + n_phi, dim=(72, 64, 56))
    dens = api.Density(ctx, ph.density, ph.volume)
    spec = api.Spectrum(ctx, phantoms.synthetic_spectrum())
    kern = api.Kernel(ctx, phantoms.synthetic_kernel(n_phi=n_phi))
    b = _batch(ctx, ph, side, on, dens, spec, 0.7)
    got, ref = _march_and_general(ctx, ph, side, dens, spec, kern, b)
    assert torch.all((got - ref).abs() <= 2e-5 * ref + 1e-6 * ref.max())


def _march_and_general(ctx, ph, side, dens, spec, kern, b):
    """The batch's dose, and that of the same beams beside one of another map size,
    which the general instance marches."""
    import torch

    api.DoseComputeCollective(ctx, b, kern)
    other = _batch(ctx, ph, 10, 2, dens, spec, 1.9, count=1)
    dose = [torch.zeros_like(b.dose), torch.zeros_like(other.dose)]
    beams = torch.cat([b.d_beams, other.d_beams])
    ptrs = {}
    for name in ("terma", "dens"):
        ptrs[name] = torch.cat([b._ptrs[name], other._ptrs[name]])
    off = [dose[0].data_ptr() + 4 * int(o) for o in b.offsets[:-1]] + [dose[1].data_ptr()]
    ptrs["dose"] = torch.from_numpy(np.array(off, np.uint64).view(np.int64)).cuda()
    n = len(b.beams) + 1
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(ctx.lib.fd2_dose_compute(ctx.h, side * side, n, p(beams), p(ptrs["terma"]), p(ptrs["dens"]),
                                        p(ptrs["dose"]), kern.h, C.c_void_p(torch.cuda.current_stream().cuda_stream)),
               "dose_compute")
    torch.cuda.synchronize()
    got, ref = b.dose.double(), dose[0].double()
    assert float(ref.max()) > 0
    assert torch.all((got == 0) == (ref == 0))
    return got, ref


def _reach(kern_src, b):
    """Voxels the widest cone moves sideways in a slice, and over the batch's longest beam."""
    t = np.tan(np.float64(kern_src.theta)).max() * max(np.abs(np.cos(kern_src.phi)).max(), np.abs(np.sin(kern_src.phi)).max())
    per = float((b.beams["long_spacing"] * t / b.beams["beamlet_size"].min(axis=1)).max())
    return per, per * int(b.beams["long_dim"].max())


@pytest.mark.parametrize("n_phi", [1, 4, 6, 8])
@pytest.mark.parametrize("side,on,size", [(8, 2, 0.5), (8, 2, 0.1), (12, 4, 0.5), (12, 4, 0.2), (16, 4, 0.5), (16, 4, 0.2)])
def test_march_of_few_and_of_many_beamlets(ctx, side, on, size, n_phi):
    """Few blocks compute their paths warp by warp, many take them from one warp's
    records; the zenith bins go to blocks of their own up to 4 beamlets an SM and
    to one block above.  The same dose, bit for bit."""
    import torch

    ph = phantoms.torso_phantom(seed=side, dim=(48, 44, 40))
    dens = api.Density(ctx, ph.density, ph.volume)
    spec = api.Spectrum(ctx, phantoms.synthetic_spectrum())
    kern = api.Kernel(ctx, phantoms.synthetic_kernel(n_theta=9, n_phi=n_phi))
    few = _batch(ctx, ph, side, on, dens, spec, 0.7, count=3, beamlet_size=size)
    n, total = len(few.beams), int(few.offsets[-1])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    doses = []
    for copies in (1, 8 * sms // (9 * n) + 1, 4 * sms // n + 1):  # blocks an SM: under 1, 8, and 4 of whole beamlets
        b = api.BEVBatch(np.concatenate([few.beams] * copies))
        b.terma.copy_(few.terma.repeat(copies))
        b.dens.copy_(few.dens.repeat(copies))
        api.DoseComputeCollective(ctx, b, kern)
        doses += [b.dose[:total].clone(), b.dose[-total:].clone()]
    torch.cuda.synchronize()
    assert float(doses[0].max()) > 0
    for d in doses[1:]:
        assert torch.equal(doses[0], d)


# Coordinates of up to C voxels: a segment's lateral offset is the difference of two
# products of that size, each of some three roundings, so a step's length is off by
# 6 C 2^-24 voxels, and steps are half a voxel or longer on average
def _far_bound(reach):
    return 12 * reach * 2.0 ** -24 + 2e-5


@pytest.mark.parametrize("side,on", [(8, 2), (12, 4), (16, 4)])
def test_march_of_slices_with_several_rounds_of_path_records(ctx, side, on):
    """Pixels of 0.05 cm: the widest bin takes more than 40 steps a slice (the
    records of one round), up to some 200."""
    import torch

    ph = phantoms.torso_phantom(seed=side, dim=(40, 36, 32))
    dens = api.Density(ctx, ph.density, ph.volume)
    spec = api.Spectrum(ctx, phantoms.synthetic_spectrum())
    src = phantoms.synthetic_kernel(n_theta=20, n_phi=6)
    kern = api.Kernel(ctx, src)
    b = _batch(ctx, ph, side, on, dens, spec, 0.7, beamlet_size=0.05 * on)
    per, total = _reach(src, b)
    assert per > 100 and per < 500 and total < 15000
    got, ref = _march_and_general(ctx, ph, side, dens, spec, kern, b)
    assert torch.all((got - ref).abs() <= _far_bound(total) * ref + 1e-6 * ref.max())


@pytest.mark.parametrize("side,on", [(8, 2), (16, 4)])
def test_batches_that_reach_too_far_take_the_other_march(ctx, side, on):
    """Rays that move more than 15000 voxels sideways: the half-table instance, as
    the tuned key tells, with the dose of the general one."""
    import torch

    ph = phantoms.torso_phantom(seed=side, dim=(72, 64, 56))
    dens = api.Density(ctx, ph.density, ph.volume)
    spec = api.Spectrum(ctx, phantoms.synthetic_spectrum())
    src = phantoms.synthetic_kernel(n_theta=24, n_phi=6)
    kern = api.Kernel(ctx, src)
    b = _batch(ctx, ph, side, on, dens, spec, 0.7, count=3, beamlet_size=0.025 * on)
    per, total = _reach(src, b)
    assert 15000 < total < 28000, total  # beyond 2^15 voxels the reference's 1e-3 step slack is lost
    got, ref = _march_and_general(ctx, ph, side, dens, spec, kern, b)
    assert torch.all((got - ref).abs() <= _far_bound(total) * ref + 1e-6 * ref.max())
    c2 = api.Context(0)
    api.DoseMatConstruction(c2, [b.beams], np.ones(side * side, np.float32), dens, spec, kern).close()
    assert [k >> 48 for k in c2.tuned_schedules()[0]] == [16]
    c2.close()


@pytest.mark.parametrize("n_phi", [4, 6, 8])
@pytest.mark.parametrize("side", [17, 20, 24, 25, 32])
def test_spread_march_is_the_march_of_a_large_batch(ctx, side, n_phi):
    """One beam of a wide map is spread over clusters of blocks with several
    warps an azimuth; 24 copies of it are not.  The same dose, bit for bit."""
    import torch

    from fastdose_b200.types import BEAM_DTYPE

    ph = phantoms.torso_phantom(seed=side, dim=(64, 56, 48))
    dens = api.Density(ctx, ph.density, ph.volume)
    spec = api.Spectrum(ctx, phantoms.synthetic_spectrum())
    kern = api.Kernel(ctx, phantoms.synthetic_kernel(n_phi=n_phi))
    b = np.zeros((), BEAM_DTYPE)
    b["isocenter"] = ph.centre()
    b["beamlet_size"] = (0.23, 0.31)
    b["fmap_size"] = (side, side)
    b["sad"] = 100.0
    b["angles"] = (1.1, 0.4, 0.2)
    b["long_spacing"] = 0.25
    b = api.calc_range(b, ph.volume)
    fl = torch.rand(side * side, device="cuda", generator=torch.Generator(device="cuda").manual_seed(side))
    doses = []
    for n in (1, 24):
        batch = api.BEVBatch(np.array([b] * n, BEAM_DTYPE))
        api.TermaComputeCollective(ctx, batch, fl, dens, spec)
        api.DoseComputeCollective(ctx, batch, kern)
        doses += [batch.get("dose", 0).clone(), batch.get("dose", n - 1).clone()]
    torch.cuda.synchronize()
    assert float(doses[0].max()) > 0
    for d in doses[1:]:
        assert torch.equal(doses[0], d)
