"""The calls that users of the dose engine make, as measurable cases.

Each case is one pass through a public entry point of ``endtoend_gb300.engine``
at a size of real use: the smallest beam dose, one beam of a plan, a candidate
set replayed from a captured plan, the optimiser's loss gradient and its angle
proposals, a server's request mix, the measured-kernel (table) dose, the
supersampled dose, a ragged adjoint, and the sparse beamlet columns.

``exact`` evaluates the same chain in 64 bits with plain torch (or numpy for
the rotations): ray trace, crop box, rotated line convolution, resample back,
and its transpose by automatic differentiation.
"""
import functools
import math

import numpy as np
import torch

from endtoend_gb300 import engine, inputs


# ------------------------------------------------------------------ the list --
def listed():
    hn = {"phantom": "headneck", "nx": 200, "ny": 200, "nz": 160, "voxel": 0.2, "spacing": 0.2}
    return [
        # dosecalc-beam on its smallest plan: one square field on a slab
        # phantom, host buffers in and out; latency and launches count
        dict(name="dose_slab64_host", call="dose_host", phantom="slab", nx=64, ny=64, nz=64, voxel=0.25,
             spacing=0.25, beams=1, nmin=16, nmax=16, beamlet=0.5, disc=False),
        # the adjoint alone on a small ragged volume: calc bbox inside the
        # volume, non-square maps, a REV spacing finer than the voxels
        dict(name="adjoint_ragged_3", call="adjoint", phantom="headneck", nx=97, ny=131, nz=73, voxel=0.3,
             spacing=0.25, beams=3, nmin=7, nmax=23, beamlet=0.37, disc=False, inset=5, ragged=True),
        # one candidate beam per call, forward + adjoint, device buffers
        dict(hn, name="beam_hn_1", call="dose_adjoint", beams=1, nmin=24, nmax=24, beamlet=0.25, disc=True),
        # TERMA supersampling 3, the preprocessing default of dosecalc-beam
        dict(hn, name="dose_hn_ss3_4", call="dose", ss=3, beams=4, nmin=12, nmax=32, beamlet=0.25, disc=True),
        # the table kernel (the reference's own discretisation), forward + adjoint
        dict(hn, name="table_hn_2", call="dose_adjoint", mode="table", beams=2, nmin=12, nmax=32, beamlet=0.25,
             disc=True),
        # a small forward + adjoint batch through the direct call
        dict(hn, name="batch_hn_6", call="dose_adjoint", beams=6, nmin=8, nmax=40, beamlet=0.25, disc=True),
        # forward doses of a candidate set, summed
        dict(hn, name="dose_hn_96", call="dose", beams=96, nmin=8, nmax=40, beamlet=0.25, disc=True),
        # the batched candidate workload: forward + adjoint replayed from a plan
        dict(hn, name="plan_hn_64", call="plan", beams=64, nmin=8, nmax=40, beamlet=0.25, disc=True),
        # one gradient of the fluence optimiser: 20 beams of 128^2 pixels
        dict(hn, name="loss_hn_20", call="loss", beams=20, nmin=128, nmax=128, beamlet=0.078, disc=False,
             eta=1e-3, sigma=1.5),
        # a batch of the annealer's angle proposals
        dict(hn, name="proposals_hn_6x20", call="proposals", proposals=6, beams=20, nmin=128, nmax=128,
             beamlet=0.078, disc=False),
        # mixed requests of the serving loop, from submit to results
        dict(name="server_mix_8", call="server", phantom="headneck", nx=96, ny=96, nz=96, nx2=160, ny2=160, nz2=160,
             voxel=0.2, spacing=0.2, requests=8, beams=8, nmin=16, nmax=64, beamlet=0.25, disc=True),
        # dosecalc-beamlet: every column of one beam, sparse
        dict(hn, name="columns_hn_40x40", call="columns", beams=1, nmin=40, nmax=40, beamlet=0.25, disc=False,
             thresh=1e-4),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges: sizes over their logarithm, odd ones among them."""
    call = rng.choice(["dose_host", "adjoint", "dose", "dose", "dose_adjoint", "dose_adjoint", "plan", "loss",
                       "proposals", "server", "columns"])
    voxel = round(rng.uniform(0.18, 0.3), 3)
    # the largest volumes at the coarse end stay within the listed extents
    nx, ny, nz = (int(_log(rng, 60, 200)) | rng.randint(0, 1) for _ in range(3))
    c = dict(call=call, phantom="headneck", nx=nx, ny=ny, nz=min(nz, 160), voxel=voxel,
             spacing=round(voxel * rng.choice([1.0, 1.0, 1.25]), 4), beams=int(_log(rng, 1, 40)),
             nmin=rng.randint(5, 16), beamlet=round(rng.uniform(0.2, 0.3), 3), disc=rng.random() < 0.6,
             pick=rng.randint(0, 9999))
    c["nmax"] = c["nmin"] + rng.randint(1, 24)
    if call in ("dose", "adjoint") and rng.random() < 0.4:
        c.update(inset=rng.randint(1, 7), ragged=True)
    if call == "dose_host":
        c["beams"] = rng.randint(1, 4)
    if call in ("dose", "dose_adjoint"):
        option = rng.choice(["", "", "ss", "table"])
        if option == "ss":
            c.update(ss=rng.choice([2, 3]), beams=rng.randint(1, 4))
        elif option == "table":
            c.update(mode="table", beams=rng.randint(1, 2), nmax=min(c["nmax"], 24))
    if call == "loss":
        c.update(nmin=rng.randint(31, 128), beamlet=0.078, beams=rng.randint(2, 20), eta=1e-3,
                 sigma=rng.choice([0.0, 1.5]), disc=False)
        c["nmax"] = c["nmin"]
    if call == "proposals":
        c.update(nmin=rng.randint(31, 128), beamlet=0.078, beams=rng.randint(2, 20), proposals=rng.randint(2, 6),
                 disc=False)
        c["nmax"] = c["nmin"]
    if call == "server":
        c.update(nx2=rng.randint(90, 160), ny2=rng.randint(90, 160), nz2=rng.randint(90, 160),
                 requests=rng.randint(2, 8), beams=rng.randint(2, 8))
    if call == "columns":
        # the beamlet path's own convolution grid is the volume's spacing
        c.update(beams=1, nmin=rng.randint(4, 24), beamlet=0.25, disc=False, thresh=rng.choice([1e-4, 1e-3]),
                 spacing=voxel)
        c["nmax"] = c["nmin"]
    return c


# --------------------------------------------------------------------- inputs --
@functools.lru_cache(maxsize=8)
def _phantom(kind, nx, ny, nz, voxel):
    if kind == "slab":
        return inputs.slab_phantom(nx, voxel)
    return inputs.head_neck_phantom(shape=(nx, ny, nz), voxel_cm=voxel, with_oars=True)


def _volume(case, seed, second=False):
    """The phantom with the noise of a CT: one per cent of each voxel's density."""
    key = ("nx2", "ny2", "nz2") if second else ("nx", "ny", "nz")
    base = _phantom(case["phantom"], *(case[k] for k in key), case["voxel"])
    rng = np.random.default_rng([seed, 1])
    noise = rng.standard_normal(base.density.shape, dtype=np.float32)
    inset = case.get("inset", 0)
    return inputs.Volume(density=base.density * np.maximum(1 + 0.01 * noise, 0), voxel=base.voxel, start=base.start,
                         bbox_start=base.bbox_start + inset, bbox_size=base.bbox_size - 2 * inset, masks=base.masks)


def _physics(case):
    return inputs.make_physics(seed=0, spacing_cm=case["spacing"])


def _beams(case, seed, n=None, which=0):
    """n beams of the 4-pi grid; angles and map sizes are the plan's, the
    fluence is the seed's (U(0,1), inside a disc where the case says so)."""
    n = n or case["beams"]
    plan = np.random.default_rng([case.get("pick", 0), which])
    rng = np.random.default_rng([seed, 2, which])
    if case["phantom"] == "slab":
        angles = [(0.0, 0.0)] * n
    else:
        angles = inputs.four_pi_angles(n, seed=int(plan.integers(1 << 30)))
    out = []
    for gantry, couch in angles:
        nx = ny = int(plan.integers(case["nmin"], case["nmax"] + 1))
        coll = 0.0
        if case.get("ragged"):
            ny = int(plan.integers(case["nmin"], case["nmax"] + 1))
            coll = float(plan.uniform(0, 90))
        b = inputs.single_beam(fmap=(nx, ny), beamlet_cm=case["beamlet"], gantry_deg=float(gantry),
                               couch_deg=float(couch), coll_deg=coll)
        b.fluence = rng.uniform(0.05, 1.0, (ny, nx)).astype(np.float32)
        if case["disc"]:
            yy, xx = np.mgrid[0:ny, 0:nx]
            b.fluence[((xx + 0.5) * 2 / nx - 1) ** 2 + ((yy + 0.5) * 2 / ny - 1) ** 2 > 1] = 0
        if case["call"] == "columns":
            b.fluence = np.ones((ny, nx), np.float32)
        out.append(b)
    return out


def _dose_grad(case, seed, vol, which=0):
    """A dose gradient as an optimiser has it: of the size of the dose, over the body."""
    rng = np.random.default_rng([seed, 3, which])
    return rng.standard_normal(vol.density.shape, dtype=np.float32) * (vol.density > 0)


def _objective(vol, seed):
    """PTV and OAR weights and targets of the loss, [nz, ny, nx] float32."""
    rng = np.random.default_rng([seed, 4])
    ptv = vol.masks["PTV"].astype(np.float32)
    ow, ot = np.zeros_like(ptv), np.zeros_like(ptv)
    for k in range(3):
        m = vol.masks["OAR%d" % k]
        ow[m] += rng.uniform(0.1, 0.5)
        ot[m] = rng.uniform(0.3, 0.6)
    return {"ptv_w": ptv, "ptv_t": ptv.copy(), "oar_w": ow, "oar_t": ot}


def _moved(beams, case, seed):
    """Whole-set proposals: every angle moved by N(0, 5 degrees)."""
    plan = np.random.default_rng([case.get("pick", 0), 77])
    sets = []
    for _ in range(case["proposals"]):
        moved = []
        for b in beams:
            c = inputs.Beam(**b.__dict__)
            c.azimuth = b.azimuth + float(plan.normal(0, math.radians(5)))
            c.zenith = b.zenith + float(plan.normal(0, math.radians(5)))
            moved.append(c)
        sets.append(moved)
    return sets


def _requests(case, seed, vols):
    """(volume, beams, dose gradient or None) of each request of the mix."""
    plan = np.random.default_rng([case.get("pick", 0), 88])
    out = []
    for k in range(case["requests"]):
        v = int(plan.integers(2))
        beams = _beams(case, seed, n=int(plan.integers(1, case["beams"] + 1)), which=10 + k)
        out.append((v, beams, _dose_grad(case, seed, vols[v], which=k) if plan.integers(2) else None))
    return out


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32).ravel()).cuda()


def prepare(case, seed):
    call, phys = case["call"], _physics(case)
    vol = _volume(case, seed)
    s = {"case": case, "vol": vol}
    if call == "server":
        vols = [vol, _volume(case, seed, second=True)]
        s["server"] = engine.Server(0, slots=2)
        s["server"].set_physics(phys, mode="exp")
        ids = [s["server"].add_volume(v) for v in vols]
        s["requests"] = [(ids[v], b, g) for v, b, g in _requests(case, seed, vols)]
        return s
    eng = s["engine"] = engine.Engine(0)
    eng.set_volume(vol)
    eng.set_physics(phys, mode=case.get("mode", "exp"))
    if case.get("ss", 1) > 1:
        eng.set_terma_supersampling(case["ss"])
    beams = s["beams"] = _beams(case, seed)
    if call == "dose_host":
        return s
    if call == "columns":
        # buffers that hold any such beam's columns, as a program that collects them keeps
        n = case["nmin"]
        size = {"beamlet": n * n, "col_ptr": n * n + 1, "row": _column_capacity(case, n)}
        size["value"] = size["row"]
        kinds = {"beamlet": torch.int32, "col_ptr": torch.int64, "row": torch.int32, "value": torch.float32}
        s.update({k: torch.zeros(size[k], dtype=kinds[k], device="cuda") for k in size})
        return s
    s["fluence"] = _cuda(engine.concat_fluence(beams))
    s["dose"] = torch.zeros(vol.nvoxels, device="cuda")
    if call in ("adjoint", "dose_adjoint", "plan", "loss"):
        s["fgrad"] = torch.zeros_like(s["fluence"])
    if call in ("adjoint", "dose_adjoint", "plan"):
        s["grad"] = _cuda(_dose_grad(case, seed, vol))
    if call == "plan":
        s["plan"] = eng.plan(beams, s["fluence"].data_ptr(), s["dose"].data_ptr(), s["grad"].data_ptr(),
                             s["fgrad"].data_ptr())
    if call in ("loss", "proposals"):
        o = s["objective"] = {k: _cuda(v) for k, v in _objective(vol, seed).items()}
        s["ptv"] = (o["ptv_w"].data_ptr(), o["ptv_t"].data_ptr())
        s["oar"] = (o["oar_w"].data_ptr(), o["oar_t"].data_ptr())
    if call == "proposals":
        s["loss"] = eng.make_loss(ptv=s["ptv"], oar=s["oar"])
        s["sets"] = _moved(beams, case, seed)
    return s


class _DeviceArray:
    """A device array of the engine as the CUDA array interface describes it."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": (n,), "typestr": typestr, "version": 3}


def _take(into, ptr, n, typestr):
    """Copies n values the engine owns (its next call, or its end, reuses them) to the front of `into`."""
    if n:
        into[:n].copy_(torch.as_tensor(_DeviceArray(ptr, n, typestr), device="cuda"))


def _column_capacity(case, n):
    """Entries kept for n^2 columns: a column's pillar is the kernel's extent (2 cm) about the beamlet axis."""
    extent = max(case["nx"], case["ny"], case["nz"]) * case["voxel"]
    return int(n * n * (1.3 * case["beamlet"] + 4.0) ** 2 * extent / case["voxel"] ** 3)


def run(s):
    call = s["case"]["call"]
    if call == "server":
        tickets = [s["server"].submit(v, b, g) for v, b, g in s["requests"]]
        out = []
        for t in tickets:
            dose, grads = s["server"].wait(t)
            out.append([dose] if grads is None else [dose, np.concatenate([g.ravel() for g in grads])])
        return out
    eng, beams = s["engine"], s["beams"]
    if call == "dose_host":
        return {"dose": eng.beam_dose(beams)}
    if call == "columns":
        d = eng.beamlet_columns_device(beams[0], s["case"]["thresh"])
        _take(s["beamlet"], d.beamlet_index, d.nbeamlets, "<i4")
        _take(s["col_ptr"], d.col_ptr, d.nbeamlets + 1, "<i8")
        _take(s["row"], d.row_index, d.nnz, "<i4")
        _take(s["value"], d.value, d.nnz, "<f4")
        return {k: s[k] for k in ("beamlet", "col_ptr", "row", "value")}
    x, dose = s["fluence"].data_ptr(), s["dose"].data_ptr()
    if call == "dose":
        eng.beam_dose_device(beams, x, dose)
        return {"dose": s["dose"]}
    if call == "adjoint":
        eng.beam_dose_adjoint_device(beams, x, s["grad"].data_ptr(), s["fgrad"].data_ptr())
        return {"fgrad": s["fgrad"]}
    if call == "dose_adjoint":
        eng.dose_and_adjoint_device(beams, x, dose, s["grad"].data_ptr(), s["fgrad"].data_ptr())
        return {"dose": s["dose"], "fgrad": s["fgrad"]}
    if call == "plan":
        s["plan"].launch()
        return {"dose": s["dose"], "fgrad": s["fgrad"]}
    if call == "loss":
        terms = eng.loss_and_grad_device(beams, x, dose, s["fgrad"].data_ptr(), ptv=s["ptv"], oar=s["oar"],
                                         eta=s["case"]["eta"], spread_sigma=s["case"]["sigma"])
        return {"terms": terms, "dose": s["dose"], "fgrad": s["fgrad"]}
    return {"losses": eng.evaluate_proposals(s["sets"], x, s["loss"]).tolist()}


# ----------------------------------------------------------------------- work --
# Arithmetic that one crop-box voxel costs per collapsed cone: the rotated
# coordinates (18), one density and one TERMA sample (2 x 14), both walks of
# the two exponentials (2 x 2 x 9), and the resample back (14 + 18); the
# transpose has the same parts.
_CONE_FLOPS = 114


def _crop_voxels(case, n, second=False):
    """Voxels of the crop box of a beam with an n x n map: the field at the
    far side of the volume plus the penumbra, along the mean extent."""
    key = ("nx2", "ny2", "nz2") if second else ("nx", "ny", "nz")
    extent = sum(case[k] for k in key) / 3 * case["voxel"]
    side = min(n * case["beamlet"] * (1 + extent / 200) + 2.0, extent)
    return side * side * extent / case["spacing"] ** 3


def work(case):
    """Each input once and each output once; the chain's arithmetic on the
    crop boxes (24 cone directions)."""
    call, nvox = case["call"], case["nx"] * case["ny"] * case["nz"]
    n = 0.5 * (case["nmin"] + case["nmax"])
    beams = case["beams"]
    directions = 2 if call in ("dose_adjoint", "plan", "loss") else 1
    if call == "server":
        total = case["requests"] * (case["beams"] + 1) / 2
        big = case["nx2"] * case["ny2"] * case["nz2"]
        voxels = total * 0.5 * (_crop_voxels(case, n) + _crop_voxels(case, n, second=True))
        return {"bytes": 4.0 * (nvox + big + case["requests"] * 0.75 * (nvox + big) + 1.5 * total * n * n),
                "flops": 1.5 * 24 * _CONE_FLOPS * voxels}
    if call == "columns":
        # a column is a pillar of the kernel's extent (2 cm) about the beamlet
        # axis; about 35 kB of it pass the threshold per cm of depth
        extent = (case["nx"] + case["ny"] + case["nz"]) / 3 * case["voxel"]
        pillar = (case["beamlet"] + 4.0) ** 2 * extent / case["spacing"] ** 3
        return {"bytes": 4.0 * nvox + 8.0 * n * n * 0.3 * pillar, "flops": 24 * 50.0 * n * n * pillar}
    if call == "proposals":
        beams *= case["proposals"]
    sub = case.get("ss", 1) ** 3
    # the ray traces: about one density sample (14 flops) per voxel of path
    field = (n * case["beamlet"]) ** 2 * (case["nx"] + case["ny"] + case["nz"]) / 3 * case["voxel"] / case["voxel"] ** 3
    rays = beams * sub * field * 14 * (case["nx"] + case["ny"] + case["nz"]) / 6
    volumes = {"dose_host": 2, "dose": 2, "adjoint": 2, "dose_adjoint": 3, "plan": 3, "loss": 6, "proposals": 5}[call]
    cone = _CONE_FLOPS if case.get("mode", "exp") == "exp" else 2 * 23 * 8 + _CONE_FLOPS
    return {"bytes": 4.0 * (volumes * nvox + (2 if directions == 2 else 1) * beams * n * n),
            "flops": directions * beams * 24 * cone * _crop_voxels(case, n) + rays}


# ---------------------------------------------------------------------- exact --
# The chain in 64 bits.  Coordinates of a beam: patient voxel index -> BEV
# (beam's eye view, crop-box relative) -> REV of each cone (i along the line,
# then the two lateral axes).
def _rot(axis, t):
    """Rodrigues matrix of a rotation about a unit axis."""
    x, y, z = axis
    k = np.array([[0, -z, y], [z, 0, -x], [-y, x, 0]], np.float64)
    return np.eye(3) * math.cos(t) + math.sin(t) * k + (1 - math.cos(t)) * np.outer(axis, axis)


def _beam_matrix(az, zen, coll):
    return _rot((0.0, 1.0, 0.0), zen + coll) @ _rot((math.sin(-zen), 0.0, math.cos(-zen)), -az)


def _cone_matrix(th, ph):
    return _rot((0.0, 1.0, 0.0), -ph) @ _rot((math.cos(ph), 0.0, -math.sin(ph)), -th)


def _f(v):
    return np.asarray(v, np.float32).astype(np.float64)


def _snap_ceil(v):
    r = np.rint(v)
    return np.where(np.abs(v - r) <= 1e-3, r, np.ceil(v))


def _bordered(v):
    """v[z, y, x] with a border of zeros, for _trilinear."""
    return torch.nn.functional.pad(v, (1, 2) * 3)


def _trilinear(p, x, y, z):
    """The volume of _bordered() between its points, 0 outside: coordinates are the volume's indices."""
    nz, ny, nx = p.shape
    x, y, z = x.clamp(-1, nx - 3), y.clamp(-1, ny - 3), z.clamp(-1, nz - 3)
    i, j, k = torch.floor(x), torch.floor(y), torch.floor(z)
    a, b, c = x - i, y - j, z - k
    at = ((k + 1) * ny + (j + 1)).mul_(nx).add_(i + 1).long()
    flat = p.reshape(-1)
    row = lambda o: torch.lerp(flat[at + o], flat[at + (o + 1)], a)  # noqa: E731
    plane = lambda o: torch.lerp(row(o), row(o + nx), b)  # noqa: E731
    return torch.lerp(plane(0), plane(nx * ny), c)


class _Chain:
    def __init__(self, vol, phys, dev):
        t = lambda a: torch.as_tensor(_f(a), device=dev)  # noqa: E731
        self.dev, self.phys = dev, phys
        self.dens = _bordered(t(vol.density))
        self.voxel, self.start = _f(vol.voxel), _f(vol.start)
        self.size = np.array(vol.density.shape[::-1], np.float64)
        self.bb0, self.bbs = np.asarray(vol.bbox_start, np.int64), np.asarray(vol.bbox_size, np.int64)
        w = np.asarray(phys.fluence, np.float32).astype(np.float64)
        self.spec = [(float(a), float(b), float(c)) for a, b, c in zip(_f(w / w.sum()), _f(phys.energy), _f(phys.mu))]
        self.lat, self.lng = float(_f(phys.rev_latspacing)), float(_f(phys.rev_longspacing))
        self.pen = float(_f(phys.penumbra))
        # voxels of the calc bbox, [nz, ny, nx] flattened
        g = [torch.arange(int(n), device=dev, dtype=torch.float64) for n in self.bbs]
        z, y, x = torch.meshgrid(g[2], g[1], g[0], indexing="ij")
        self.rel = torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)])

    def t(self, a):
        return torch.as_tensor(np.asarray(a, np.float64), device=self.dev)

    def beamlets(self, B, p):
        """Fluence-map index of points p [3, n] (RCS cm), -1 outside the field."""
        diff = p - self.t(B["src"])[:, None]
        along = (diff * self.t(B["dir"])[:, None]).sum(0)
        rej = diff - along * self.t(B["dir"])[:, None]
        pb = self.t(B["MB"]) @ (rej * (B["isodist"] / along.abs()))
        fx = pb[0] / B["beamlet"][0] + B["fmap"][0] * 0.5
        fz = pb[2] / B["beamlet"][1] + B["fmap"][1] * 0.5
        ok = (fx >= 0) & (fx < B["fmap"][0]) & (fz >= 0) & (fz < B["fmap"][1]) & (rej.square().sum(0) > 0)
        return torch.where(ok, torch.floor(fx).long() + B["fmap"][0] * torch.floor(fz).long(), -1)

    def path(self, p, src):
        """Radiological path src -> p [3, n]: plane crossings advanced from a
        common first parameter, midpoint densities, short segments dropped."""
        src, start, voxel = self.t(src)[:, None], self.t(self.start)[:, None], self.t(self.voxel)[:, None]
        d = p - src
        first = (start - src - 0.5 * voxel) / d
        last = (start + self.t(self.size)[:, None] * voxel - src + 0.5 * voxel) / d
        lo = torch.minimum(first, last).amax(0).clamp(min=0)
        hi = torch.maximum(first, last).amin(0).clamp(max=1)
        step = (voxel / d).abs()
        length = d.norm(dim=0)
        total = torch.zeros_like(lo)
        origin = src - start
        at = torch.nonzero(lo < hi).reshape(-1)
        d, step, length, hi, alpha = d[:, at], step[:, at], length[at], hi[at], lo[at]
        a = alpha.expand(3, -1).clone()
        acc, nxt = torch.zeros_like(alpha), torch.zeros_like(alpha)
        ax, ay, az = a
        sx, sy, sz = step
        for n in range(5000):
            live = (alpha < hi) & (torch.minimum(torch.minimum(ax, ay), az) < 1)
            if n % 16 == 0 and not bool(live.all()):
                total[at[~live]] = acc[~live]
                keep = torch.nonzero(live).reshape(-1)
                if not keep.numel():
                    return total
                d, at = d[:, keep], at[keep]
                ax, ay, az, sx, sy, sz, length, hi, alpha, acc, nxt, live = (
                    v[keep] for v in (ax, ay, az, sx, sy, sz, length, hi, alpha, acc, nxt, live))
            # a crossing still inside is below 1, so the tests between two
            # axes need no more than their order
            hit = live & (ax < 1) & (ax <= ay) & (ax <= az)
            vy, vz = live & (ay < 1), live & (az < 1)
            nxt, ax = torch.where(hit, ax, nxt), torch.where(hit, ax + sx, ax)
            hit = vy & (ay <= ax) & (ay <= az)
            nxt, ay = torch.where(hit, ay, nxt), torch.where(hit, ay + sy, ay)
            hit = vz & (az <= ax) & (az <= ay)
            nxt, az = torch.where(hit, az, nxt), torch.where(hit, az + sz, az)
            seg = (length * (nxt - alpha)).abs()
            q = torch.addcmul(origin, d, (0.5 * (nxt + alpha))[None]) / voxel - 0.5
            use = live & (seg >= 0.001)
            acc = torch.where(use, acc + seg * _trilinear(self.dens, q[0], q[1], q[2]), acc)
            alpha = torch.where(live, nxt, alpha)
        total[at] = acc
        return total

    def beam(self, b, ss, table, grad, fluence=None):
        """(dose on the bbox, fluence gradient or None) of one beam; grad: on
        the bbox, flat; fluence: the map in 64 bits, the beam's own by default."""
        B = {}
        az, zen = math.fmod(float(_f(b.azimuth)), 2 * math.pi), math.fmod(float(_f(b.zenith)), 2 * math.pi)
        if abs(zen) > 1e-6 and (abs(az) <= 1e-6 or abs(az - math.pi) <= 1e-6):
            zen = 0.0
        coll, iso, sad = float(_f(b.coll)), _f(b.isocenter), float(_f(b.sad))
        B["MB"] = _beam_matrix(az, zen, coll)
        B["src"] = iso + _beam_matrix(az, zen, 0.0).T @ np.array([0.0, -sad, 0.0])
        B["isodist"] = float(np.linalg.norm(iso - B["src"]))
        B["dir"] = (iso - B["src"]) / B["isodist"]
        B["fmap"], B["beamlet"] = tuple(int(v) for v in b.fmap_size), _f(b.beamlet_size)
        fluence = self.t(_f(b.fluence).ravel()) if fluence is None else fluence

        # TERMA: the mean over ss^3 points of each voxel
        voxel, start = self.t(self.voxel)[:, None], self.t(self.start)[:, None]
        centre = start + (self.rel + self.t(self.bb0)[:, None]) * voxel
        n = self.rel.shape[1]
        terma = torch.zeros(n, dtype=torch.float64, device=self.dev)
        points, lists = [], []
        for k in range(ss ** 3):
            off = np.array([k % ss, (k // ss) % ss, k // (ss * ss)], np.float64)
            p = centre + (self.t((off + 0.5) / ss - 0.5)[:, None]) * voxel
            bl = self.beamlets(B, p)
            at = torch.nonzero(bl >= 0).reshape(-1)
            points.append(p[:, at])
            lists.append((at, bl[at]))
        p, owner, bl = torch.cat(points, 1), torch.cat([v[0] for v in lists]), torch.cat([v[1] for v in lists])
        rpl = self.path(p, B["src"])
        unit = sum(w * e * m * torch.exp(-m * rpl) for w, e, m in self.spec)
        unit = unit * sad ** 2 / (p - self.t(B["src"])[:, None]).square().sum(0) / ss ** 3
        terma.index_add_(0, owner, unit * fluence[bl].clamp(min=0))

        # crop box of the voxels with TERMA, the penumbra around it
        MB, MBi = B["MB"], B["MB"].T
        bev = (self.t(MB) @ self.rel)[:, terma != 0]
        pad = np.array([self.pen / self.lat, self.pen / self.lng, self.pen / self.lat])
        mn = bev.amin(1).cpu().numpy() - pad
        mx = np.maximum(bev.amax(1).cpu().numpy(), 1.17549435e-38) + pad
        box = _snap_ceil(np.abs(mx - mn))
        off = MBi @ mn + self.bb0  # crop-box origin, patient index

        bi = self.t(MB) @ (self.rel + self.t(self.bb0 - off)[:, None])
        sees = ((bi >= -2) & (bi <= self.t(box + 2)[:, None])).all(0)
        seen = torch.nonzero(sees).reshape(-1)
        bi = bi[:, seen]
        terma = terma.reshape(*(int(v) for v in self.bbs[::-1])).requires_grad_(grad is not None)
        dose = torch.zeros(n, dtype=torch.float64, device=self.dev)
        cm = box * np.array([self.lat, self.lng, self.lat])
        corners = np.array([[cm[0] * (c & 1), cm[1] * (c >> 1 & 1), cm[2] * (c >> 2)] for c in range(8)]).T
        for th, ph, row in zip(np.radians(_f(self.phys.theta_deg)), np.radians(_f(self.phys.phi_deg)),
                               np.arange(self.phys.nrays) % (self.phys.ntheta // 2)):
            MK = _cone_matrix(th, ph)
            o = MK @ corners
            lo, hi = o.min(1), np.maximum(o.max(1), 1.17549435e-38)
            size = _snap_ceil(np.abs(hi - lo) / np.array([self.lat, self.lng, self.lat])).astype(int)
            q0 = lo / np.array([self.lat, self.lng, self.lat])
            L, n1, n2 = int(size[1]), int(size[2]), int(size[0])  # along the line, then tY, tZ
            i, y, z = (torch.arange(m, device=self.dev, dtype=torch.float64) for m in (L, n1, n2))
            i, y, z = (v.reshape(-1) for v in torch.meshgrid(i, y, z, indexing="ij"))
            bev = self.t(MK.T) @ (torch.stack([z, i, y]) + self.t(q0)[:, None])
            pt = self.t(MBi) @ bev + self.t(off)[:, None]
            b0, b1 = self.t(self.bb0)[:, None], self.t(self.bb0 + self.bbs)[:, None]
            ok = ((bev >= 0) & (bev < self.t(box)[:, None]) & (pt >= b0) & (pt < b1)).all(0)
            del bev
            use = torch.nonzero(ok).reshape(-1)
            pt = pt[:, use]
            rho = torch.zeros(L * n1 * n2, dtype=torch.float64, device=self.dev)
            rho[use] = _trilinear(self.dens, pt[0], pt[1], pt[2])
            pt = pt - b0
            T = torch.zeros_like(rho).index_put((use,), _trilinear(_bordered(terma), pt[0], pt[1], pt[2]))
            del pt
            # without TERMA a line has no dose, but its samples have a gradient
            some = ok if grad is not None else T != 0
            lines = torch.nonzero(some.reshape(L, -1).any(0)).reshape(-1)
            r, t, v = (w.reshape(L, -1)[:, lines] for w in (rho, T, ok))
            if table:
                D = self.table(r, t, row) + self.table(r.flip(0), t.flip(0), self.phys.ntheta - 1 - row).flip(0)
            else:
                D = self.recur(r, t, row)
            D = torch.where(v, D, torch.zeros_like(D)) / self.phys.nphi
            full = torch.zeros(L, n1 * n2, dtype=torch.float64, device=self.dev).index_copy(1, lines, D)
            full = full.reshape(L, n1, n2).permute(2, 1, 0).contiguous()  # [tZ, tY, i]
            q = self.t(MK) @ bi - self.t(q0)[:, None]
            fits = (q >= 0).all(0) & (q[1] < L) & (q[2] < n1) & (q[0] < n2)
            at = torch.nonzero(fits).reshape(-1)
            part = _trilinear(_bordered(full), q[1, at], q[2, at], q[0, at])
            dose.index_add_(0, seen[at], part.detach())
            if grad is not None:
                (part * grad[seen[at]]).sum().backward()
        if grad is None:
            return dose, None
        tg = terma.grad.reshape(-1)
        return dose, torch.zeros_like(fluence).index_add_(0, bl, unit * tg[owner])

    def recur(self, r, t, row):
        """Both walks of the double-exponential kernel on [L, lines]: the two
        exponentials of either walk side by side."""
        par = _f(self.phys.exp_params)[[row, self.phys.ntheta - 1 - row]].reshape(4, 2)  # (amplitude, rate)
        rate, amp = self.t(par[:, 1])[None, :, None], self.t(par[:, 0] / par[:, 1])[None, :, None]
        both = lambda v: torch.stack([v, v, v.flip(0), v.flip(0)], 1)  # noqa: E731  [L, 4, lines]
        h, t4 = torch.exp(-0.5 * self.lng * rate * both(r)), both(t)
        hm = torch.cat([torch.ones_like(h[:1]), h[:-1]])
        tm = torch.cat([torch.zeros_like(t4[:1]), t4[:-1]])
        gain, add = h * h, tm * h * (1 - hm * h)
        Y, rows = torch.zeros_like(h[0]), []
        for i in range(r.shape[0]):
            rows.append(Y)
            Y = torch.addcmul(add[i], gain[i], Y)
        D = amp * (torch.stack(rows) + tm * (1 - hm))
        return D[:, 0] + D[:, 1] + (D[:, 2] + D[:, 3]).flip(0)

    def table(self, r, t, row):
        """One walk of the cumulative table: receiver w gets T_k (K(c_k) - K(c_k+1)) of the sources k < w."""
        R = self.t(np.concatenate([[0.0], _f(self.phys.radii)]))
        K = self.t(np.concatenate([[0.0], _f(self.phys.cumkern)[row]]))
        L, out = r.shape[0], []
        for at in range(0, r.shape[1], 512):
            p = self.lng * r[:, at:at + 512].T
            P = torch.cumsum(p, 1) - p
            c = P[:, :, None] - (P + 0.5 * p)[:, None, :]  # [line, receiver, source]
            below = torch.tril(torch.ones(L, L, dtype=torch.bool, device=self.dev), -1)
            c = torch.where(below, c, torch.zeros_like(c))
            seg = (torch.bucketize(c, R) - 1).clamp(0, len(R) - 2)
            k = K[seg] + (c - R[seg]) / (R[seg + 1] - R[seg]) * (K[seg + 1] - K[seg])
            nearer = torch.cat([c[:, :, 1:], torch.zeros_like(c[:, :, :1])], 2)
            w = k - torch.cat([k[:, :, 1:], torch.zeros_like(k[:, :, :1])], 2)
            reach = below & ((c <= R[-2]) | ((nearer <= R[-2]) & (c <= R[-1])))
            w = torch.where(reach, w, torch.zeros_like(w))
            out.append((w @ t[:, at:at + 512].T[:, :, None])[:, :, 0].T)
        return torch.cat(out, 1) if out else torch.zeros_like(t)


    def dose(self, beams, ss=1, table=False, grad=None, fluences=None):
        """(summed dose on the bbox, the beams' fluence gradients or None)."""
        got = [self.beam(b, ss, table, grad, f) for b, f in zip(beams, fluences or [None] * len(beams))]
        return sum(d for d, _ in got), None if grad is None else torch.cat([f for _, f in got])


def _terms(dose, o):
    """PTV and OAR terms of the loss and their gradient by the dose."""
    e, h = dose - o["ptv_t"], (dose - o["oar_t"]).clamp(min=0)
    return (o["ptv_w"] * e * e).sum(), (o["oar_w"] * h * h).sum(), 2 * o["ptv_w"] * e + 2 * o["oar_w"] * h


def _spread(x, sigma):
    """Normalised Gaussian spread of a map [fy, fx], zeros beyond its edge."""
    if not sigma:
        return x
    r = math.ceil(3 * sigma)
    w = np.exp(-0.5 * (np.arange(-r, r + 1) / sigma) ** 2)
    w = torch.as_tensor(w / w.sum(), device=x.device)
    grid = [torch.arange(n, device=x.device) for n in x.shape]
    band = [torch.where((g[:, None] - g).abs() <= r, w[(g[:, None] - g + r).clamp(0, 2 * r)], 0.0) for g in grid]
    return band[0] @ x @ band[1]


def _exact_loss(case, seed, chain, vol, beams):
    o = {k: chain.t(v).ravel() for k, v in _objective(vol, seed).items()}
    maps = [chain.t(_f(b.fluence)) for b in beams]
    seen = [_spread(x, case["sigma"]).ravel() for x in maps]
    dose, _ = chain.dose(beams, fluences=seen)
    ptv, oar, grad = _terms(dose, o)
    _, fgrad = chain.dose(beams, grad=grad, fluences=seen)
    out, smooth, at = [], 0.0, 0
    for x in maps:
        g = _spread(fgrad[at:at + x.numel()].reshape(x.shape), case["sigma"])
        at += x.numel()
        for axis in (0, 1):
            d = torch.diff(x, dim=axis)
            smooth += case["eta"] * float(d.abs().sum())
            edge = torch.zeros_like(x.narrow(axis, 0, 1))
            g = g - case["eta"] * torch.diff(torch.cat([edge, d.sign(), edge], axis), dim=axis)
        out.append(g.ravel())
    return {"terms": [float(ptv), float(oar), smooth], "dose": dose, "fgrad": torch.cat(out)}


def _exact_seconds(case, requests):
    """About what exact() takes on a GPU: most of it is the launches of the line walks."""
    call = case["call"]
    vols = case["nx"] * case["ny"] * case["nz"] / 6.4e6 + 0.4
    if call == "server":
        return sum(len(b) for _, b, _ in requests) * 1.0
    one = {"loss": 2.2, "proposals": 0.8 * case.get("proposals", 1)}.get(call, 1.3)
    return case["beams"] * vols * (7 if case.get("mode") == "table" else one)


def exact(case, seed):
    call = case["call"]
    if call == "columns":
        # the columns keep the entries that pass a threshold on FP32 values
        # sampled through 8-bit filter weights: no list in 64 bits has their layout
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    vol, phys = _volume(case, seed), _physics(case)
    vols = [vol] + ([_volume(case, seed, second=True)] if call == "server" else [])
    requests = _requests(case, seed, vols) if call == "server" else []
    if _exact_seconds(case, requests) > 20:
        return None
    chains = [_Chain(v, phys, dev) for v in vols]
    if call == "server":
        out = []
        for v, beams, g in requests:
            dose, fgrad = chains[v].dose(beams, grad=None if g is None else chains[v].t(_f(g)).ravel())
            dose = dose.reshape(vols[v].density.shape).cpu().numpy()
            out.append([dose] if g is None else [dose, fgrad.cpu().numpy()])
        return out
    chain, beams = chains[0], _beams(case, seed)
    if call == "loss":
        return _exact_loss(case, seed, chain, vol, beams)
    if call == "proposals":
        o = {k: chain.t(v).ravel() for k, v in _objective(vol, seed).items()}
        return {"losses": [float(sum(_terms(chain.dose(b)[0], o)[:2])) for b in _moved(beams, case, seed)]}
    (x0, y0, z0), (bx, by, bz) = (tuple(int(v) for v in w) for w in (vol.bbox_start, vol.bbox_size))
    box = (slice(z0, z0 + bz), slice(y0, y0 + by), slice(x0, x0 + bx))
    grad = None
    if call in ("adjoint", "dose_adjoint", "plan"):
        grad = chain.t(_f(_dose_grad(case, seed, vol))[box].ravel())
    got, fgrad = chain.dose(beams, case.get("ss", 1), case.get("mode", "exp") == "table", grad)
    dose = torch.zeros(vol.density.shape, dtype=torch.float64, device=dev)
    dose[box] = got.reshape(bz, by, bx)
    if call == "dose_host":
        return {"dose": dose.cpu().numpy()}
    out = {"dose": dose.ravel(), "fgrad": fgrad}
    return {k: out[k] for k in {"dose": ["dose"], "adjoint": ["fgrad"]}.get(call, ["dose", "fgrad"])}
