"""The work that the library's performance is followed on: what it does for its users, through its public entry points.

A planning job builds dose-loading matrices (Terma, cone convolution, columns) for one beam up to a whole 4pi candidate
set, and then optimizes the fluence on the matrices; single fields are computed and resampled on their own.  The listed
cases are those steps at the sizes of the repository's configurations, tests and benchmark; draw() gives more of the
same ranges.  A case is a dict of plain values; `kind` names the step.

    prepare(case, seed) -> state     inputs made from the seed, and the handles and buffers a program keeps
    run(state) -> outputs            one pass through the public entry points
    work(case), tolerance(case), exact(case, seed)
"""
import math

import numpy as np
import torch

from fastdose_b200 import api, optimize, phantoms
from fastdose_b200.types import BEAM_DTYPE, make_bundle, make_volume

_CTX = None


def _ctx():
    """The process's context: a program keeps one per host thread."""
    global _CTX
    if _CTX is None:
        _CTX = api.Context(0)
    return _CTX


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the group prox of one solver step on its own: 400 candidate beams of about 100 beamlets (smallest call)
        dict(name="prox_400_beams", kind="prox", groups=400, low=40, high=160),
        # configuration 1: a single beam of 100 open beamlets on the 64^3 slab phantom
        dict(name="plan_slab_1_beam", kind="plan", phantom="slab", nx=64, ny=64, nz=64, beams=1, fluence=10, map=16,
             on=4, values="f32", phis=6, overlap=True, graph=False),
        # a served request: a few beams on a small phantom, 16-bit values, one stream
        dict(name="plan_request_4_beams", kind="plan", phantom="torso", nx=120, ny=120, nz=96, beams=4, fluence=16,
             map=12, on=4, values="f16", phis=6, overlap=False, graph=True),
        # the batched 4pi plan (benchmark phantom and beamlet grid) on 100 of its candidate beams
        dict(name="plan_4pi_100_beams", kind="plan", phantom="torso", nx=200, ny=200, nz=160, beams=100, fluence=16,
             map=16, on=4, values="f32", phis=6, overlap=True, graph=False),
        # one isocentre of the multi-isocentre head-and-neck plan, its wide BEV grid, 16-bit values
        dict(name="plan_wide_map_24_beams", kind="plan", phantom="torso", nx=160, ny=160, nz=128, beams=24, fluence=13,
             map=20, on=4, values="f16", phis=6, overlap=True, graph=False),
        # plain dose of a few open fields: Terma, convolution and the dense resampling, 1024-pixel maps
        dict(name="field_32x32_4_beams", kind="field", nx=128, ny=128, nz=128, beams=4, map=32, pixel=0.3, phis=8),
        # BEV volume to patient grid, dense and supersampled
        dict(name="resample_200", kind="resample", nx=200, ny=200, nz=160, map=16, slices=186, pixel=0.25, ss=5,
             extent=2.0),
        # A x and A^T y over a VOI matrix of 5e7 nonzeros, 32-bit values and columns
        dict(name="products_f32", kind="products", rows=250_000, cols=10_000, share=0.02, values="f32", index="i32"),
        # the same in the 16-bit form the optimizer is run with
        dict(name="products_f16", kind="products", rows=250_000, cols=10_000, share=0.02, values="f16",
             index="packed16"),
        # objective and gradient of a plan of 100 beams of 64 beamlets
        dict(name="gradient_f32", kind="gradient", rows=120_000, beams=100, fluence=8, share=0.03, values="f32",
             index="packed16"),
        # 20 iterations of the group-sparse solver at the size of the optimizer's parity fixture
        dict(name="solver_20_steps", kind="solver", rows=48_000, beams=24, fluence=9, share=0.03, values="f16",
             index="packed16", iters=20),
        # the beam-orientation loop with two prunes, from the beamlet-major matrix of all candidates
        dict(name="orientation_2_prunes", kind="orientation", rows=48_000, beams=24, fluence=9, share=0.03,
             values="f32", index="i32", iters=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan"] * 8 + ["field", "resample", "products", "products", "gradient", "solver", "prox"])
    if kind == "plan":
        mp = rng.choice([8, 11, 12, 15, 16, 16, 16, 17, 20, 20, 24])
        slab = rng.random() < 0.2
        n = rng.randint(48, 80) if slab else 0
        # fewer beams with the wide maps, so that no draw costs more than the 100-beam plan
        beams = 1 if slab else _log(rng, 1, 40 if mp <= 16 else 16)
        return dict(kind="plan", phantom="slab" if slab else "torso", nx=n or rng.randint(90, 200),
                    ny=n or rng.randint(90, 200), nz=n or rng.randint(70, 160), beams=beams,
                    fluence=rng.randint(6, 16), map=mp, on=2 if mp < 12 else 4, values=rng.choice(["f32", "f16", "bf16"]),
                    phis=rng.choice([4, 6, 6, 8]), overlap=rng.random() < 0.6, graph=rng.random() < 0.3)
    if kind == "field":
        return dict(kind="field", nx=rng.randint(60, 150), ny=rng.randint(60, 150), nz=rng.randint(60, 150),
                    beams=rng.randint(1, 6), map=rng.choice([10, 16, 20, 25, 32]), pixel=round(rng.uniform(0.2, 0.5), 2),
                    phis=rng.choice([6, 8]))
    if kind == "resample":
        return dict(kind="resample", nx=rng.randint(80, 200), ny=rng.randint(80, 200), nz=rng.randint(60, 160),
                    map=rng.choice([12, 16, 21, 32]), slices=rng.randint(80, 200), pixel=round(rng.uniform(0.12, 0.4), 2),
                    ss=rng.choice([3, 5, 5]), extent=rng.choice([0.6, 2.0]))
    if kind == "products":
        values = rng.choice(["f32", "f16", "bf16"])
        return dict(kind="products", rows=_log(rng, 5_000, 300_000), cols=_log(rng, 300, 10_000),
                    share=rng.choice([0.01, 0.02]), values=values,
                    index="packed16" if values != "f32" else rng.choice(["i32", "packed16"]))
    if kind == "prox":
        return dict(kind="prox", groups=_log(rng, 20, 1200), low=20, high=rng.randint(60, 400))
    c = dict(kind=kind, rows=_log(rng, 8_000, 150_000), beams=rng.randint(8, 100), fluence=rng.randint(4, 10),
             share=0.03, values=rng.choice(["f32", "f16"]), index="packed16")
    if kind == "solver":
        c["iters"] = rng.randint(8, 20)
    return c


# ------------------------------------------------------------------ inputs
def _phantom(case, seed):
    """(host density [z][y][x], volume, PTV mask or None, isocentre)."""
    dim = (case["nx"], case["ny"], case["nz"])
    vox = 0.25
    if case.get("phantom") == "slab":
        ph = phantoms.slab_phantom(dim[0], bone=(4.0, 2.0, 1.85), lung=(8.0, 3.0, 0.25))
        # each patient's slab has its own noise
        g = torch.Generator(device="cuda").manual_seed(seed)
        d = torch.from_numpy(ph.density).cuda() * (1 + 0.02 * torch.randn(ph.density.shape, device="cuda", generator=g))
        return d.cpu().numpy(), ph.volume, None, ph.centre()
    # the torso of phantoms.torso_phantom, built on the device
    g = torch.Generator(device="cuda").manual_seed(seed)
    ax = [(torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) * vox for n in dim]
    X, Y, Z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    cx, cy, cz = (n * vox / 2 for n in dim)
    rx, ry, rz = cx * 0.9, cy * 0.62, cz * 0.95
    body = ((X - cx) / rx) ** 2 + ((Y - cy) / ry) ** 2 + ((Z - cz) / rz) ** 2 <= 1.0
    d = torch.where(body, 1.0 + 0.03 * torch.randn(body.shape, device="cuda", generator=g), 0.001)
    for s in (-1, 1):
        lung = (((X - (cx + s * rx * 0.45)) / (rx * 0.3)) ** 2 + ((Y - (cy - ry * 0.1)) / (ry * 0.55)) ** 2
                + ((Z - cz) / (rz * 0.6)) ** 2) <= 1.0
        d = torch.where(lung & body, 0.25, d)
    d = torch.where(((X - cx) ** 2 + (Y - (cy + ry * 0.7)) ** 2 <= 1.2 ** 2) & body, 1.5, d)
    off = _geometry(case).uniform(0.0, 0.1, 3) * rx
    pc = (cx + float(off[0]), cy + float(off[1]) * 0.5, cz + float(off[2]) * 0.5)
    ptv = (((X - pc[0]) ** 2 + (Y - pc[1]) ** 2 + (Z - pc[2]) ** 2) <= _ptv_radius(case) ** 2).to(torch.uint8)
    bx = [int(math.floor(c / vox - r / vox)) for c, r in ((cx, rx), (cy, ry), (cz, rz))]
    start = tuple(max(0, b) for b in bx)
    size = tuple(n - 2 * s for n, s in zip(dim, start))
    return d.cpu().numpy(), make_volume(dim, (vox,) * 3, start, size), ptv.cpu().numpy(), pc


def _ptv_radius(case):
    return 0.05 * min(case["nx"], 1.2 * case["ny"], 1.2 * case["nz"]) * 0.25 + 0.6


def _geometry(case):
    """Where the target, the beams and the groups lie: a case's own.  The seed fills in the patient, the fluence and
    the dose values, so that every seed's outputs have the same shapes."""
    return np.random.default_rng([case.get(k, 0) for k in ("nx", "ny", "nz", "beams", "map", "groups", "high")])


def _angles(case):
    a = phantoms.sphere_beam_angles(max(case["beams"], 40))
    pick = _geometry(case).permutation(len(a))[:case["beams"]]
    return a[np.sort(pick)]


def _prepare_plan(case, seed):
    ctx = _ctx()
    dens, vol, ptv, iso = _phantom(case, seed)
    slab = case["phantom"] == "slab"
    angles = np.zeros((1, 3), np.float32) if slab else _angles(case)
    bundles = np.array([make_bundle(iso, a, sad=100.0, fluence_dim=case["fluence"], beamlet_size=0.5,
                                    sub_fluence_dim=case["map"], sub_fluence_on=case["on"], long_spacing=0.25)
                        for a in angles])
    if slab:
        flags = np.ones((1, case["fluence"] ** 2), np.uint8)
    else:
        flags = api.beamletFlagInit(ctx, bundles, ptv, vol)
    return dict(kind="plan", case=case, beamlets=api.bundles_beamlets(bundles, flags, vol),
                fluence=api.beamlet_fluence(bundles[0]), density=api.Density(ctx, dens, vol),
                spectrum=api.Spectrum(ctx, phantoms.synthetic_spectrum(seed=1)),
                kernel=api.Kernel(ctx, phantoms.synthetic_kernel(seed=2, n_phi=case["phis"])), matrix=None)


def _field_beams(case, vol, iso):
    rng = _geometry(case)
    out = []
    for a in _angles(case):
        b = np.zeros((), BEAM_DTYPE)
        b["isocenter"] = iso
        b["beamlet_size"] = (case["pixel"], case["pixel"])
        b["fmap_size"] = (case["map"], case["map"])
        b["sad"] = 100.0
        b["angles"] = a + rng.uniform(-0.05, 0.05, 3).astype(np.float32)
        b["long_spacing"] = 0.25
        out.append(api.calc_range(b, vol))
    return np.array(out, BEAM_DTYPE)


def _prepare_field(case, seed):
    ctx = _ctx()
    dens, vol, _, iso = _phantom(dict(case, phantom="torso"), seed)
    beams = _field_beams(case, vol, iso)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    fl = torch.rand((len(beams), case["map"] ** 2), device="cuda", generator=g)
    return dict(kind="field", batch=api.BEVBatch(beams), fluence=torch.where(fl < 0.2, 0.0, fl),
                density=api.Density(ctx, dens, vol), host=dens,
                spectrum=api.Spectrum(ctx, phantoms.synthetic_spectrum(seed=1)),
                kernel=api.Kernel(ctx, phantoms.synthetic_kernel(seed=2, n_phi=case["phis"])))


def _prepare_resample(case, seed):
    ctx = _ctx()
    dim = (case["nx"], case["ny"], case["nz"])
    vol = make_volume(dim, (0.25,) * 3)
    iso = tuple(n * 0.125 for n in dim)
    rng = _geometry(case)
    b = np.zeros((), BEAM_DTYPE)
    b["isocenter"] = iso
    b["beamlet_size"] = (case["pixel"], case["pixel"])
    b["fmap_size"] = (case["map"], case["map"])
    b["sad"] = 100.0
    b["angles"] = (rng.uniform(0.2, 2.9), rng.uniform(-1.2, 1.2), rng.uniform(-0.3, 0.3))
    b["long_spacing"] = 0.25
    b = api.calc_range(b, vol)
    b["long_dim"] = min(int(b["long_dim"]), case["slices"])
    # a depth-dose curve times a blurred field, as a BEV dose is
    g = torch.Generator(device="cuda").manual_seed(seed)
    bev = torch.rand((int(b["long_dim"]), case["map"], case["map"]), device="cuda", generator=g)
    bev = torch.nn.functional.avg_pool3d(bev[None, None], 3, 1, 1)[0, 0] + 0.05
    depth = torch.arange(bev.shape[0], device="cuda", dtype=torch.float32) * 0.25
    bev = (bev * torch.exp(-0.05 * depth)[:, None, None]).contiguous()
    density = api.Density(ctx, np.ones((dim[2], dim[1], dim[0]), np.float32), vol)
    return dict(kind="resample", beam=b, bev=bev, density=density, ss=case["ss"], extent=case["extent"])


def _voi_matrix(rows, cols, share, seed):
    """A VOI matrix (rows = voxels, columns = beamlets): every beamlet meets a window of the voxels at random, its
    doses falling off along it.  CSR on the device: (offsets int64, columns int64, values f32)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    win = max(8, min(rows, int(rows * share * 2)))
    start = torch.randint(0, rows - win + 1, (cols,), device="cuda", generator=g)
    parts = []
    step = max(1, (1 << 27) // win)
    for c0 in range(0, cols, step):
        n = min(step, cols - c0)
        c, r = (torch.rand((n, win), device="cuda", generator=g) < 0.5).nonzero(as_tuple=True)
        parts.append((r + start[c + c0]) * cols + (c + c0))
    key = torch.cat(parts).sort().values
    r, c = key // cols, key % cols
    off = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.bincount(r, minlength=rows).cumsum(0)
    depth = (r - start[c]).float() / win
    val = (0.3 + 0.7 * torch.rand(c.numel(), device="cuda", generator=g)) * torch.exp(-1.5 * depth) * (30.0 / cols)
    return off, c, val


def _matrix(case, n_cols, seed):
    off, col, val = _voi_matrix(case["rows"], n_cols, case["share"], seed)
    A = optimize.Matrix.from_csr(_ctx(), off.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy(), n_cols,
                                 case["values"], case["index"])
    return A, A.transpose()


def _doses(case, seed):
    """Prescription of a plan: the first tenth of the rows is the PTV."""
    rng = np.random.default_rng(seed + 7)
    n_ptv = case["rows"] // 10
    n_oar = case["rows"] - n_ptv
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    return n_ptv, n_oar, dict(
        max_dose=f(np.concatenate([np.full(n_ptv, 1.05), rng.uniform(0.3, 0.7, n_oar)])),
        max_weights=f(np.concatenate([np.ones(n_ptv), rng.uniform(0.1, 1.0, n_oar)])), min_dose=f(np.ones(n_ptv)),
        min_weights=f(np.ones(n_ptv)), oar_weights=f(rng.uniform(0.0, 0.1, n_oar)))


def _fluence0(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed + 3)
    return torch.rand(n, device="cuda", generator=g) * 0.2


def _prepare_optimizer(case, seed):
    ctx = _ctx()
    nb, fd = case["beams"], case["fluence"]
    n = nb * fd * fd
    A, AT = _matrix(case, n, seed)
    D = optimize.Matrix.from_csr(ctx, *optimize.block_diag([optimize.fluence_grad(fd, np.ones(fd * fd))] * nb))
    DT = D.transpose()
    n_ptv, n_oar, w = _doses(case, seed)
    st = dict(kind=case["kind"], case=case, A=A, AT=AT, D=D, DT=DT, n_ptv=n_ptv, n_oar=n_oar, w=w,
              x=_fluence0(n, seed), groups=np.arange(0, n + 1, fd * fd, dtype=np.int64))
    if case["kind"] != "orientation":
        st["problem"] = optimize.Problem(ctx, A, AT, D, DT, n_ptv, n_oar, w["max_dose"], w["max_weights"],
                                         w["min_dose"], w["min_weights"], w["oar_weights"], 1.0, 0.1)
        if case["kind"] == "solver":
            st["weights"] = 0.1 * st["problem"].beam_weights_init(st["groups"])
    return st


def _groups(case, seed):
    sizes = _geometry(case).integers(case["low"], case["high"] + 1, case["groups"])
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    tau = np.random.default_rng(seed).uniform(0.01, 1.0, case["groups"]).astype(np.float32)
    return off, tau


def _group_input(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, device="cuda", generator=g) * 0.5


def prepare(case, seed):
    kind = case["kind"]
    if kind == "plan":
        return _prepare_plan(case, seed)
    if kind == "field":
        return _prepare_field(case, seed)
    if kind == "resample":
        return _prepare_resample(case, seed)
    if kind == "products":
        A, AT = _matrix(case, case["cols"], seed)
        return dict(kind=kind, A=A, AT=AT, x=_fluence0(case["cols"], seed), y=_fluence0(case["rows"], seed + 1))
    if kind == "prox":
        off, tau = _groups(case, seed)
        return dict(kind=kind, off=off, tau=torch.from_numpy(tau).cuda(), g0=_group_input(int(off[-1]), seed))
    return _prepare_optimizer(case, seed)


# ------------------------------------------------------------------ one pass
class _DeviceArray:
    """A device array of a matrix handle, for torch.as_tensor; keeps the handle alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None}


def _plan_outputs(m, values):
    inf = m.info()
    ro, col, val, sc = m.device_views()
    t = lambda p, n, s: torch.as_tensor(_DeviceArray(m, p, n, s), device="cuda")  # noqa: E731
    out = dict(offsets=t(ro, inf["n_rows"] + 1, "<i8"), columns=t(col, inf["nnz"], "<i4"))
    if values == "f32":
        out["values"] = t(val, inf["nnz"], "<f4")
    else:
        v = t(val, inf["nnz"], "<i2")
        out["values"] = v.view(torch.float16 if values == "f16" else torch.bfloat16)
        out["scales"] = t(sc, inf["n_rows"], "<f4")
    return out


def run(state):
    kind = state["kind"]
    ctx = _ctx()
    if kind == "plan":
        c = state["case"]
        m = api.DoseMatConstruction(ctx, state["beamlets"], state["fluence"], state["density"], state["spectrum"],
                                    state["kernel"], value_type=c["values"], graph=c["graph"], overlap=c["overlap"])
        state["matrix"] = m  # the plan's matrix replaces the one before
        return _plan_outputs(m, c["values"])
    if kind == "field":
        b = state["batch"]
        b.dose.zero_()
        api.TermaComputeCollective(ctx, b, state["fluence"], state["density"], state["spectrum"])
        api.DoseComputeCollective(ctx, b, state["kernel"])
        vols = [api.BEV2PVCS(ctx, b.beams[i], state["density"], b.get("dose", i)) for i in range(len(b.beams))]
        return dict(terma=b.terma, density=b.dens, dose=b.dose, volumes=vols)
    if kind == "resample":
        a = (ctx, state["beam"], state["density"], state["bev"])
        return dict(dense=api.BEV2PVCS(*a), mean=api.BEV2PVCS(*a, ssfactor=state["ss"], extent=state["extent"]))
    if kind == "products":
        return dict(forward=state["A"].spmv(state["x"]), back=state["AT"].spmv(state["y"]))
    if kind == "prox":
        prox, norms = optimize.prox_l2onehalf(ctx, state["off"], state["g0"], state["tau"])
        return dict(prox=prox, norms=norms)
    if kind == "gradient":
        value, grad = state["problem"].eval_grad(state["x"])
        return dict(value=value, grad=grad)
    c, w = state["case"], state["w"]
    if kind == "solver":
        r = state["problem"].boo(state["groups"], state["weights"], state["x"], step_size=1e-3, iters=c["iters"],
                                 change_trigger=10 ** 6)
        return dict(x=r["x"], v=r["v"], loss=r["loss"], norms=r["nrm"])
    fd = c["fluence"]
    r = optimize.beam_orientation_optimization(
        ctx, state["AT"], state["D"], state["groups"], np.arange(c["beams"] + 1) * 2 * fd * (fd - 1), state["n_ptv"],
        state["n_oar"], w["max_dose"], w["max_weights"], w["min_dose"], w["min_weights"], w["oar_weights"], state["x"],
        beam_weight=0.1, max_iter=c["iters"], change_weights_trigger=10 ** 6, n_beams_want=4,
        prune_trigger=(c["iters"] // 3, 2 * c["iters"] // 3))
    return dict(active=r["active"], norms=r["norms"], x=r["x"], costs=r["costs_full"])


# ------------------------------------------------------------------ work
def _march(case, n_maps, chord_cm, pixel):
    """Ray segments of the convolution of n_maps BEV maps: per slice and cone one, and one per lateral crossing."""
    k = phantoms.synthetic_kernel(seed=2, n_phi=case["phis"])
    seg = sum(1 + math.tan(t) * (abs(math.cos(p)) + abs(math.sin(p))) * 0.25 / pixel for t in k.theta for p in k.phi)
    return n_maps * case["map"] ** 2 * (chord_cm / 0.25) * seg


def work(case):
    kind = case["kind"]
    if kind in ("plan", "field", "resample"):
        vox = case["nx"] * case["ny"] * case["nz"]
        chord = 0.25 * (0.9 * case["nx"] + 0.62 * case["ny"] + 0.95 * case["nz"]) / 3
    if kind == "plan":
        pixel = 0.5 / case["on"]
        if case["phantom"] == "slab":
            maps, chord = case["fluence"] ** 2, case["ny"] * 0.25
        else:
            maps = case["beams"] * min(case["fluence"] ** 2, math.pi * (_ptv_radius(case) / 0.5 + 0.5) ** 2)
        side = min(case["map"] * pixel, 4.0)
        nnz = maps * chord * (side + 0.25) ** 2 / 0.25 ** 3
        seg = _march(case, maps, chord, pixel)
        terma = maps * case["map"] ** 2 * chord / 0.25
        return {"bytes": 4 * vox + 96 * maps + 8 * maps + nnz * (8 if case["values"] == "f32" else 6),
                "flops": 20 * seg + 100 * terma + 125 * 10 * nnz}
    if kind == "field":
        P = case["map"] ** 2
        cells = case["beams"] * P * chord / 0.25
        return {"bytes": 4 * vox + 4 * case["beams"] * (P + vox) + 12 * cells,
                "flops": 20 * _march(case, case["beams"], chord, case["pixel"]) + 250 * cells + 40 * vox * case["beams"]}
    if kind == "resample":
        inside = min(vox, math.pi * case["extent"] ** 2 * case["slices"] * 0.25 / 0.25 ** 3)
        return {"bytes": 8 * vox + 4 * case["map"] ** 2 * case["slices"], "flops": 40 * vox + 40 * case["ss"] ** 3 * inside}
    if kind == "prox":
        n = case["groups"] * (case["low"] + case["high"]) / 2
        return {"bytes": 8 * n + 16 * case["groups"], "flops": 6 * n}
    cols = case["cols"] if kind == "products" else case["beams"] * case["fluence"] ** 2
    nnz = case["rows"] * cols * case["share"]
    entry = (4 if case["values"] == "f32" else 2) + (4 if case["index"] == "i32" else 2)
    products = {"products": 2, "gradient": 2, "solver": 3 * case.get("iters", 0),
                "orientation": 2 * case.get("iters", 0)}[kind]
    vectors = 4 * (cols + case["rows"])
    return {"bytes": products * (nnz * entry + vectors) + 20 * case["rows"], "flops": products * 2 * nnz}


def tolerance(case):
    """Measured on the same path with its sums in another order (schedules, instances, value formats), times about four.
    The march's discrete steps are the same in any correct implementation; only its sums may round differently."""
    kind = case["kind"]
    if kind == "plan":  # f16 and bf16 values may round to the neighbour
        return {"f32": {"rel": 1e-5, "max": 1e-3}, "f16": {"rel": 2e-4, "max": 2e-3},
                "bf16": {"rel": 2e-3, "max": 1.6e-2}}[case["values"]]
    if kind == "field":
        return {"rel": 1e-5, "max": 1e-3}
    if kind == "resample":  # a voxel at the very edge of the extent may be in or out
        return {"rel": 1e-4, "max": 0.9}
    if kind in ("products", "gradient", "prox"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-4, "max": 1e-2}  # solver, orientation: rounding travels through the line searches


# ------------------------------------------------------------------ 64-bit results
def _rotation(angles):
    """BEV -> patient rotation of a beam (gantry, couch, collimator), 3x3 in 64 bits."""
    th, ph, co = (float(a) for a in angles)
    a = -(ph + co)
    c, s = math.cos(a), math.sin(a)
    ry = np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]])
    ux, uz = math.sin(-ph), math.cos(-ph)
    u = np.array([ux, 0.0, uz])
    K = np.array([[0, -uz, 0], [uz, 0, -ux], [0, ux, 0]])
    ra = math.cos(th) * np.eye(3) + math.sin(th) * K + (1 - math.cos(th)) * np.outer(u, u)
    return torch.from_numpy(ra @ ry).cuda()


def _trilinear(vol, u, v, w):
    """vol[w][v][u] in 64 bits, texel centres at i + 0.5, zero outside."""
    nz, ny, nx = vol.shape
    f = [torch.floor(t - 0.5) for t in (u, v, w)]
    a = [t - 0.5 - b for t, b in zip((u, v, w), f)]
    i, j, k = (t.long() for t in f)
    flat = vol.reshape(-1)
    out = torch.zeros_like(u)
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                x, y, z = i + di, j + dj, k + dk
                ok = (x >= 0) & (x < nx) & (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
                q = (z.clamp(0, nz - 1) * ny + y.clamp(0, ny - 1)) * nx + x.clamp(0, nx - 1)
                wt = (a[0] if di else 1 - a[0]) * (a[1] if dj else 1 - a[1]) * (a[2] if dk else 1 - a[2])
                out += torch.where(ok, flat[q] * wt, 0.0)
    return out


def _exact_field(case, seed):
    st = _prepare_field(case, seed)
    dens = torch.from_numpy(st["host"]).cuda().double()
    sp = phantoms.synthetic_spectrum(seed=1)
    terma, rho = [], []
    for b, fl in zip(st["batch"].beams, st["fluence"].double()):
        F, L, sad, ls = case["map"], int(b["long_dim"]), float(b["sad"]), float(b["long_spacing"])
        px = (torch.arange(F, device="cuda", dtype=torch.float64) + 0.5 - F / 2)
        p = torch.stack([(px * float(b["beamlet_size"][0])).repeat(F), torch.full((F * F,), sad, device="cuda").double(),
                         (px * float(b["beamlet_size"][1])).repeat_interleave(F)])
        pc = _rotation(b["angles"]) @ p
        k = ls / (sad * 4)
        t = float(b["lim_min"]) / sad + k * torch.arange(1, 4 * L + 1, device="cuda", dtype=torch.float64)[:, None]
        src = [float(v) for v in b["source"]]
        d = _trilinear(dens, *((src[q] + t * pc[q]) / 0.25 for q in range(3)))
        rpl = torch.cumsum(d * (k * pc.norm(dim=0)), 0)
        tl = torch.zeros_like(d)
        for e in range(sp.n):
            tl += float(sp.fluence[e]) * float(sp.energy[e]) * float(sp.mu[e]) * torch.exp(-float(sp.mu[e]) * rpl)
        terma.append((tl * fl / t ** 2).view(L, 4, -1).mean(1).reshape(-1))
        rho.append(d.view(L, 4, -1).mean(1).reshape(-1))
    # the dose has no 64-bit value of its own: the march's discrete steps are defined by its 32-bit ray coordinates
    return dict(terma=torch.cat(terma), density=torch.cat(rho), dose=None, volumes=[None] * case["beams"])


def _exact_resample(case, seed):
    st = _prepare_resample(case, seed)
    b, bev = st["beam"], st["bev"].double()
    R = _rotation(b["angles"]).T
    src = torch.tensor([float(v) for v in b["source"]], device="cuda", dtype=torch.float64)[:, None]
    h = case["map"] / 2

    def grid(p):
        q = R @ (p - src)
        s = q[1] / float(b["sad"])
        return q, (q[0] / (float(b["beamlet_size"][0]) * s) + h, q[2] / (float(b["beamlet_size"][1]) * s) + h,
                   (q[1] - float(b["lim_min"])) / float(b["long_spacing"]))

    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dense = torch.zeros(nz * ny * nx, device="cuda", dtype=torch.float64)
    mean = torch.zeros_like(dense)
    step = nx * ny * 16
    for v0 in range(0, dense.numel(), step):
        v = torch.arange(v0, min(v0 + step, dense.numel()), device="cuda")
        vox = torch.stack([v % nx, v // nx % ny, v // (nx * ny)]).double()
        q, cn = grid((vox + 0.5) * 0.25)
        dense[v] = _trilinear(bev, *cn)
        on = q[0] ** 2 + q[2] ** 2 <= case["extent"] ** 2
        if not bool(on.any()):
            continue
        vox, at = vox[:, on], v[on]
        acc = torch.zeros(vox.shape[1], device="cuda", dtype=torch.float64)
        for s in range(case["ss"] ** 3):
            sub = torch.tensor([s % case["ss"], s // case["ss"] % case["ss"], s // case["ss"] ** 2], device="cuda")
            acc += _trilinear(bev, *grid((vox + ((sub + 0.5) / case["ss"])[:, None]) * 0.25)[1])
        mean[at] = torch.where(acc >= 1e-4, acc / case["ss"] ** 3, 0.0)
    return dict(dense=dense.view(nz, ny, nx), mean=mean.view(nz, ny, nx))


class _Sparse:
    """The stored matrix (16-bit values rounded under their beamlet's scale) in 64 bits."""

    def __init__(self, case, n_cols, seed):
        off, col, val = _voi_matrix(case["rows"], n_cols, case["share"], seed)
        if case["values"] != "f32":
            half = torch.float16 if case["values"] == "f16" else torch.bfloat16
            top = torch.zeros(n_cols, device="cuda").scatter_reduce(0, col, val.abs(), "amax")
            top = torch.where(top > 0, top, 1.0)
            val = (val / top[col]).to(half).double() * top[col].double()
        self.row = torch.repeat_interleave(torch.arange(case["rows"], device="cuda"), off.diff())
        self.col, self.val, self.shape = col, val.double(), (case["rows"], n_cols)

    def mul(self, x):
        return torch.zeros(self.shape[0], device="cuda", dtype=torch.float64).index_add_(0, self.row, self.val * x[self.col])

    def back(self, y):
        return torch.zeros(self.shape[1], device="cuda", dtype=torch.float64).index_add_(0, self.col, self.val * y[self.row])

    def columns(self, keep):
        """These columns, renumbered in the order given."""
        new = torch.full((self.shape[1],), -1, device="cuda", dtype=torch.int64)
        new[keep] = torch.arange(keep.numel(), device="cuda")
        c = new[self.col]
        m = _Sparse.__new__(_Sparse)
        m.row, m.col, m.val, m.shape = self.row[c >= 0], c[c >= 0], self.val[c >= 0], (self.shape[0], keep.numel())
        return m


class _Objective:
    def __init__(self, case, A, seed):
        self.A, self.fd = A, case["fluence"]
        self.n_ptv, _, w = _doses(case, seed)
        self.w = {k: torch.from_numpy(v).cuda().double() for k, v in w.items()}
        self.eta, self.gamma = float(np.float32(0.1)), 1.0

    def value(self, x, grad=False):
        w, p = self.w, self.n_ptv
        ax = self.A.mul(x)
        low, high, oar = (ax[:p] - w["min_dose"]).clamp(max=0), (ax - w["max_dose"]).clamp(min=0), ax[p:]
        m = x.view(-1, self.fd, self.fd)
        dx, dy = m[:, :, 1:] - m[:, :, :-1], m[:, 1:] - m[:, :-1]
        shrink = lambda t: torch.sign(t) * (t.abs() - self.gamma).clamp(min=0)  # noqa: E731
        tv = sum(shrink(t).abs().sum() + 0.5 / self.gamma * (shrink(t) - t).square().sum() for t in (dx, dy))
        g = 0.5 * ((w["min_weights"] * low ** 2).sum() + (w["max_weights"] * high ** 2).sum()
                   + (w["oar_weights"] * oar ** 2).sum()) + self.eta * tv
        if not grad:
            return float(g)
        back = self.A.back(torch.cat([w["min_weights"] * low, w["oar_weights"] * oar]) + w["max_weights"] * high).view_as(m)
        ex, ey = (self.eta / self.gamma * (t - shrink(t)) for t in (dx, dy))
        back[:, :, 1:] += ex
        back[:, :, :-1] -= ex
        back[:, 1:] += ey
        back[:, :-1] -= ey
        return float(g), back.reshape(-1)


def _prox(v, tau):
    """Half-norm prox of each row of v: (scaled rows, their norms)."""
    n2 = v.square().sum(1)
    alpha = tau * torch.where(n2 > 1e-4, n2.clamp(min=1e-30) ** -0.75, 1008611.0)
    s = torch.sin((torch.acos((alpha * (0.75 * math.sqrt(3))).clamp(max=1.0)) + math.pi / 2) / 3) * (2 / math.sqrt(3))
    th = torch.where(alpha > 2 * math.sqrt(6) / 9, 0.0, s * s)
    out = th[:, None] * v
    return out, out.norm(dim=1)


def _solve(obj, weights, st, end, limit, loss, want):
    """The accelerated group-sparse steps from state st = (k, theta, t, x, v) to iteration `end`."""
    k, theta, t, x, v = st
    tk = t
    norms, stop = None, False
    while k < end:
        if k < 50 or k % 5 == 0:
            t *= 2
        while True:
            th, y = 1.0, x
            if k > 1:
                bb = t * theta * theta
                th = (-bb + math.sqrt(bb * bb + 4 * tk * bb)) / (2 * tk)
                y = (1 - th) * x + th * v
            gy, g = obj.value(y, True)
            nx, norms = _prox((y - t * g).clamp(min=0).view(len(weights), -1), weights * t)
            nx = nx.reshape(-1)
            gx = obj.value(nx)
            d = nx - y
            if gx <= gy + float(g @ d) + 0.5 / t * float(d @ d):
                break
            t *= 0.5
        x, v = nx, nx / th + (1 - 1 / th) * x
        theta, tk = th, t
        loss[k] = float((weights * norms.sqrt()).sum()) + gx
        if int((norms > 1e-4).sum()) - 1e-4 <= want:
            stop = True
            break
        k += 1
    return (k, theta, t, x, v), norms, stop or k == limit


def _weights(A, case, n_ptv):
    s = torch.zeros(A.shape[1], device="cuda", dtype=torch.float64).index_add_(0, A.col, torch.where(A.row < n_ptv, A.val, 0.0))
    w = (s.view(case["beams"], -1).mean(1) / n_ptv).sqrt()
    return (w / w.max()).clamp(min=0.1) * float(np.float32(0.1))


def _exact_optimizer(case, seed):
    fd2 = case["fluence"] ** 2
    A = _Sparse(case, case["beams"] * fd2, seed)
    obj = _Objective(case, A, seed)
    x = _fluence0(A.shape[1], seed).double()
    if case["kind"] == "gradient":
        value, grad = obj.value(x, True)
        return dict(value=value, grad=grad)
    w = _weights(A, case, obj.n_ptv)
    loss = torch.zeros(case["iters"], dtype=torch.float64)
    st = (0, 0.0, float(np.float32(1e-3)), x, x)
    if case["kind"] == "solver":
        st, norms, _ = _solve(obj, w, st, case["iters"], case["iters"], loss, 0)
        return dict(x=st[3], v=st[4], loss=loss, norms=norms)
    active, stop = torch.arange(case["beams"], device="cuda"), False
    ends = [case["iters"] // 3, 2 * case["iters"] // 3, case["iters"]]
    while not stop and active.numel():
        end = min(e for e in ends if e > st[0])
        sub = A.columns((active[:, None] * fd2 + torch.arange(fd2, device="cuda")).reshape(-1))
        st, norms, stop = _solve(_Objective(case, sub, seed), w, st, end, case["iters"], loss, 4)
        rank = torch.sort(norms, descending=True, stable=True).indices[:int((norms > 1e-4).sum())]
        active, w, norms = active[rank], w[rank], norms[rank]
        st = st[:3] + tuple(q.view(-1, fd2)[rank].reshape(-1) for q in st[3:])
    return dict(active=active.int(), norms=norms, x=st[3], costs=loss)


def exact(case, seed):
    kind = case["kind"]
    if kind == "plan":
        # no value of its own: the steps of the march and the samples of the columns are defined by 32-bit coordinates
        return None
    if kind == "field":
        return _exact_field(case, seed)
    if kind == "resample":
        return _exact_resample(case, seed)
    if kind == "products":
        A = _Sparse(case, case["cols"], seed)
        return dict(forward=A.mul(_fluence0(case["cols"], seed).double()), back=A.back(_fluence0(case["rows"], seed + 1).double()))
    if kind == "prox":
        off, tau = _groups(case, seed)
        g0 = _group_input(int(off[-1]), seed).double()
        parts = [_prox(g0[a:b][None], torch.tensor([float(t)], device="cuda").double())
                 for a, b, t in zip(off[:-1], off[1:], tau)]
        return dict(prox=torch.cat([p[0][0] for p in parts]), norms=torch.cat([p[1] for p in parts]))
    return _exact_optimizer(case, seed)
