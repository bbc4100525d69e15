"""The measured work of the photon-transport framework, through its public entry points.

Kinds of case:

* ``job``: one transport job on a resident world and table, as a server or a
  planning loop submits it: ``Job`` -> ``result_async`` into page-locked
  buffers -> ``result_wait``.  The world, the table, the local-majorant grid
  and the source tables are what such a program keeps.
* ``call``: ``Transport()(world, source)``, the drop-in call: world upload,
  table, local-majorant grid, transport and results from host arrays to host
  arrays.
* ``batch``: many jobs of uneven size in one ``Batch``, each with its results.
* ``paths``: radiological paths of straight rays (``DeviceWorld.radiological_path``),
  host rays in, host results out.

Beams and phantoms are those of the repository's workloads (pencil beam in a
water cube, projection radiography on grids with ellipsoid inclusions, CT
spiral on a body phantom) and the CTDI phantom of the dose calibration, built
here from the seed with torch so that a new phantom takes milliseconds.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import dxmclib_gb300 as dx
from dxmclib_gb300 import _capi as A
from dxmclib_gb300 import api, workloads
from dxmclib_gb300.calibration import CTDIPhantom

_CTX = None


def _context():
    """The process's context: a program makes one and keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = dx.GpuContext(device=0)
    return _CTX


def _job(name, beam, nx, ny, nz, histories, model=1, layout="palette", result="f32", mode="ev", precision=32, kind="job"):
    return dict(name=name, kind=kind, beam=beam, nx=nx, ny=ny, nz=nz, histories=histories, model=model, layout=layout,
                result=result, mode=mode, precision=precision)


def listed():
    return [
        # the smallest request: a quick look at a pencil beam in the 64^3 water cube, where latency counts
        _job("pencil 64^3, 1e5", "pencil", 64, 64, 64, 100_000, result="f64"),
        # the plain method's own example through the drop-in call: 1e6 histories of a 60 keV pencil beam
        _job("call, pencil 64^3, 1e6", "pencil", 64, 64, 64, 1_000_000, result="f64", kind="call"),
        # one ordinary radiography request on a resident phantom
        _job("DX 160^3, 5e6", "dx", 160, 160, 160, 5_000_000),
        # the impulse-approximation model, which samples the Compton profile, on an odd grid
        _job("DX 127^3, 4e6, IA", "dx", 127, 127, 127, 4_000_000, model=2),
        # the headline: a CT spiral over a body of 512 x 512 x 200 voxels
        _job("CT 512x512x200, 1e8", "ct", 512, 512, 200, 100_003_500),
        # a CT volume with a density of its own in every voxel (8-byte voxels), as a patient scan converts to
        _job("CT 512x512x100, 3e7, wide", "ct", 512, 512, 100, 30_000_000, layout="wide"),
        # the drop-in call with a new ragged CT volume: upload, majorant grid, transport and dose in one call
        _job("call, CT 333x287x77, 2e7", "ct", 333, 287, 77, 20_000_000, result="f64", mode="dose", kind="call"),
        # the dose calibration's run: forced scoring in the holes of the CTDI phantom
        _job("CTDI 323x323x60, 1e7", "ctdi", 323, 323, 60, 10_000_000, result="f64", mode="dose"),
        # double precision throughout, the check of a single-precision result
        _job("DX 96^3, 1e6, FP64", "dx", 96, 96, 96, 1_000_000, precision=64, result="f64"),
        # a worklist of uneven radiography jobs submitted at once
        dict(name="batch of 16 DX", kind="batch", n=16, small=64, large=192, histories=3_000_000, mode="concurrent"),
        # many small jobs in one launch of the persistent multi-job kernel
        dict(name="batch of 20 small DX", kind="batch", n=20, small=48, large=96, histories=400_000, mode="persistent"),
        # primary transmission: one ray per detector pixel of a 1024 x 1024 projection of the CT body
        dict(name="paths, 2^20 rays, CT", kind="paths", nx=512, ny=512, nz=200, rays=1 << 20, layout="palette"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["job", "job", "job", "job", "call", "batch", "paths"])
    if kind == "batch":
        mode = rng.choice(["concurrent", "persistent"])
        small = rng.randint(40, 72)
        return dict(kind="batch", n=rng.randint(3, 16), small=small, large=small + rng.randint(8, 88), mode=mode,
                    histories=_log(rng, 100_000, 2_000_000))
    if kind == "paths":
        return dict(kind="paths", nx=_log(rng, 40, 512), ny=_log(rng, 40, 512), nz=_log(rng, 20, 200),
                    rays=_log(rng, 1_000, 1 << 20), layout=rng.choice(["palette", "palette", "wide"]))
    beam = rng.choice(["pencil", "dx", "dx", "ct", "ct", "ctdi"])
    if beam == "ctdi":
        n = rng.randint(60, 160) * 2 + 3
        return _drawn(rng, kind, beam, n, n, 60, _log(rng, 1_000_000, 20_000_000), "palette")
    if beam == "pencil":
        n = rng.randint(30, 100)
        return _drawn(rng, kind, beam, n, n, n, _log(rng, 50_000, 10_000_000), "palette")
    if beam == "dx":
        n = rng.randint(50, 256)
        return _drawn(rng, kind, beam, n, n, n, _log(rng, 200_000, 30_000_000), rng.choice(["palette", "palette", "wide"]))
    return _drawn(rng, kind, beam, rng.randint(100, 512), rng.randint(100, 512), rng.randint(30, 200),
                  _log(rng, 1_000_000, 60_000_000), rng.choice(["palette", "palette", "wide"]))


def _drawn(rng, kind, beam, nx, ny, nz, histories, layout):
    model = rng.choice([1, 1, 1, 0, 2])
    precision = 32
    if kind == "job" and rng.random() < 0.1:
        precision, histories = 64, min(histories, 2_000_000)
    result = "f64" if kind == "call" else rng.choice(["f32", "f64"])
    c = _job("", beam, nx, ny, nz, histories, model, layout, result, rng.choice(["ev", "ev", "dose"]), precision, kind)
    del c["name"]
    return c


# ---- phantoms ---------------------------------------------------------------------------
def _grid(nx, ny, nz, spacing):
    """Voxel centre coordinates (mm) along each axis, broadcastable to (nz, ny, nx)."""
    ax = []
    for n, s in zip((nx, ny, nz), spacing):
        ax.append((torch.arange(n, device="cuda", dtype=torch.float32) - (n - 1) / 2) * s)
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _arrays(case, seed):
    """(dims, spacing, material, density) of the case's phantom, on the GPU."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    beam = case.get("beam", "ct")
    if beam == "pencil":
        sp = (128.0 / nx,) * 3
        mat = torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda")
        dens = torch.ones((nz, ny, nx), dtype=torch.float32, device="cuda")
    elif beam == "dx":
        # soft tissue with 3-8 ellipsoid inclusions of three materials, densities 0.2-2.0
        sp = (300.0 / nx,) * 3
        x, y, z = _grid(nx, ny, nz, sp)
        mat = torch.zeros((nz, ny, nx), dtype=torch.uint8, device="cuda")
        dens = torch.ones((nz, ny, nx), dtype=torch.float32, device="cuda")
        for _ in range(int(rng.integers(3, 9))):
            c, a = rng.uniform(-90.0, 90.0, 3), rng.uniform(15.0, 75.0, 3)
            inside = ((x - c[0]) / a[0]) ** 2 + ((y - c[1]) / a[1]) ** 2 + ((z - c[2]) / a[2]) ** 2 <= 1
            mat[inside] = int(rng.integers(0, 3))
            dens[inside] = float(np.float32(rng.uniform(0.2, 2.0)))
    else:
        # the CT body: elliptic soft tissue in air, two lungs, 30 bone spheres
        sp = (409.6 / nx, 409.6 / ny, 2.5)
        x, y, z = _grid(nx, ny, nz, sp)
        half = nz * sp[2] / 2
        body = (x / 160.0) ** 2 + (y / 120.0) ** 2 <= 1
        mat = torch.where(body.expand(nz, ny, nx), workloads.SOFT, workloads.AIR).to(torch.uint8)
        for cx in (-75.0, 75.0):
            t = ((x - cx) / 55.0) ** 2 + ((y + 5.0) / 70.0) ** 2 + (z / (0.84 * half)) ** 2
            mat[(t <= 1) & body] = workloads.LUNG
        for _ in range(30):
            phi, r = rng.uniform(0.0, 2 * math.pi), math.sqrt(rng.uniform(0.0, 0.8))
            c = (160.0 * r * math.cos(phi), 120.0 * r * math.sin(phi), rng.uniform(-half, half))
            t = (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2
            mat[(t <= rng.uniform(5.0, 20.0) ** 2) & body] = workloads.BONE
        of = torch.tensor([d for _, d in workloads.CT_MATERIALS], dtype=torch.float32, device="cuda")
        dens = of[mat.long()]
    if case.get("layout") == "wide":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        dens = dens * (0.95 + 0.1 * torch.rand(dens.shape, generator=gen, device="cuda"))
    return (nx, ny, nz), sp, mat, dens


def _world(case, seed):
    beam = case.get("beam", "ct")
    if beam == "ctdi":
        return CTDIPhantom(case["nx"] - 3)
    dims, sp, mat, dens = _arrays(case, seed)
    w = dx.World()
    w.setDimensions(dims)
    w.setSpacing(sp)
    w.setDensityArray(dens.reshape(-1).cpu().numpy())
    w.setMaterialIndexArray(mat.reshape(-1).cpu().numpy())
    if beam == "pencil":
        w.addMaterialToMap(dx.Material("Water, Liquid"))
    elif beam == "dx":
        for name in workloads.DX_MATERIALS:
            w.addMaterialToMap(dx.Material(name))
    else:
        for name, d in workloads.CT_MATERIALS:
            w.addMaterialToMap(dx.Material(name, density=d))
    return w


def _source(case, world, seed):
    beam, histories = case["beam"], case["histories"]
    if beam == "pencil":
        src = api.PencilSource()
        src.setPosition((0, 0, -128.0))
        src.setDirectionCosines((1, 0, 0, 0, 1, 0))
        src.setPhotonEnergy(60.0)
        src.setTotalExposures(10)
        src.setHistoriesPerExposure(max(histories // 10, 1))
    elif beam == "dx":
        src = workloads.dx_source(np.random.default_rng(seed + 1), histories, kvp=80.0)
    elif beam == "ctdi":
        src = api.CTAxialSource()
        src.tube().setVoltage(120.0)
        src.setCollimation(40.0)
        src.setScanLenght(0)
        src.setExposureAngleStepDeg(5.0)
        src.setHistoriesPerExposure(max(histories // src.totalExposures(), 1))
    else:
        src = workloads.ct_source(world, histories)
    src.updateFromWorld(world)
    src.validate()
    return src


def _resident(world, source, layout="palette"):
    """What a program keeps of a phantom: the world and the table on the device, with the majorant grid built."""
    ctx = _context()
    dworld = dx.DeviceWorld(ctx, world, layout=1 if layout == "wide" else 0)
    energy = 150.0 if source is None else source.maxPhotonEnergyProduced()
    blob = api.LutBlob.cached(world.materialMap(), dworld.max_density(), energy)
    dlut = dx.DeviceLut(ctx, blob)
    return dworld, dlut, blob


def _buffers(n, result):
    kind = torch.float32 if result == "f32" else torch.float64
    return [torch.empty(n, dtype=kind, pin_memory=True).numpy() for _ in range(2)] + [
        torch.empty(n, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)]


class _Kept:
    """A state whose device objects are given back when it goes."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for o in getattr(self, "owned", []):
            o.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "paths":
        world = _world(case, seed)
        dworld, dlut, blob = _resident(world, None, case["layout"])
        return _Kept(case=case, dworld=dworld, dlut=dlut, rays=_rays(case, seed), owned=[dlut, dworld])
    if kind == "batch":
        return _prepare_batch(case, seed)
    world = _world(case, seed)
    source = _source(case, world, seed)
    if kind == "call":
        tr = dx.Transport(_context())
        tr.setLowEnergyCorrectionModel(case["model"])
        tr.setOutputMode(dx.Transport.DOSE if case["mode"] == "dose" else dx.Transport.EV_PER_HISTORY)
        tr.setSeed(seed)
        world.isValid()
        return _Kept(case=case, transport=tr, world=world, source=source)
    dworld, dlut, _ = _resident(world, source, case["layout"])
    dworld.prepare(dlut)
    beam = source.beams(world.directionCosines())[0]
    return _Kept(case=case, dworld=dworld, dlut=dlut, beam=beam, seed=seed, out=_buffers(world.size(), case["result"]),
                 owned=[dlut, dworld])


def _prepare_batch(case, seed):
    ctx = _context()
    entries, outs, owned = [], [], []
    for k in range(case["n"]):
        # uneven jobs: grids spread over the stated sizes, a third to three times the stated histories
        n = case["small"] + int((case["large"] - case["small"] + 1) * ((0.618 * k + 0.5) % 1.0))
        h = int(case["histories"] * math.exp(2.2 * ((0.414 * k + 0.9) % 1.0) - 1.1))
        c = dict(beam="dx", nx=n, ny=n, nz=n, histories=h)
        world = _world(c, seed + 100 * k)
        source = _source(c, world, seed + 100 * k)
        dworld, dlut, _ = _resident(world, source)
        dworld.prepare(dlut)
        beam = source.beams(world.directionCosines())[0]
        entries.append(api.BatchEntry(dworld, dlut, beam.exposures, beam.spectrum, beam.heel, beam.bowtie, seed + k))
        outs.append(_buffers(world.size(), "f32"))
        owned += [dlut, dworld]
    mode = api.Batch.CONCURRENT if case["mode"] == "concurrent" else api.Batch.PERSISTENT
    return _Kept(case=case, ctx=ctx, entries=entries, outs=outs, mode=mode, owned=owned)


def _rays(case, seed):
    """Rays of a cone from a point source 600 mm from the centre to a flat detector, at energies of 30-120 keV."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    side = max(int(math.ceil(math.sqrt(n))), 1)
    i = np.arange(n)
    u = ((i % side) + 0.5) / side * 500.0 - 250.0
    v = ((i // side) + 0.5) / side * 500.0 - 250.0
    a = rng.uniform(0.0, 2 * math.pi)
    src = np.array([600.0 * math.cos(a), 600.0 * math.sin(a), 0.0])
    end = np.stack([-500.0 * math.cos(a) - u * math.sin(a), -500.0 * math.sin(a) + u * math.cos(a), v], axis=1)
    rays = np.empty((n, 7), np.float32)
    rays[:, 0:3] = src
    rays[:, 3:6] = end - src
    rays[:, 6] = rng.uniform(30.0, 120.0, n)
    return rays


# ---- one pass -----------------------------------------------------------------------------
def run(state):
    case = state.case
    if case["kind"] == "call":
        r = state.transport(state.world, state.source, useSourceDoseCalibration=False)
        return {"dose": r.dose, "variance": r.variance, "events": _whole(r.nEvents)}
    if case["kind"] == "paths":
        return state.dworld.radiological_path(state.dlut, state.rays)
    if case["kind"] == "batch":
        batch = api.Batch(state.ctx, state.entries, mode=state.mode)
        for job, out in zip(batch.jobs, state.outs):
            job.result_async(out=out, dtype=np.float32)
        got = [job.result_wait()[:3] for job in batch.jobs]
        batch.close()
        return [[d, v, _whole(n)] for d, v, n in got]
    job = api.Job(_context(), state.dworld, state.dlut, state.beam.exposures, state.beam.spectrum, state.beam.heel,
                  state.beam.bowtie, state.seed, case["model"],
                  precision=A.PRECISION_FP64 if case["precision"] == 64 else A.PRECISION_FP32)
    dose, var, events, _ = _finish(job, case, state.out)
    job.close()
    return {"dose": dose, "variance": var, "events": _whole(events)}


def _finish(job, case, out):
    mode = A.OUTPUT_DOSE if case["mode"] == "dose" else A.OUTPUT_EV_PER_HISTORY
    job.result_async(mode, out=out, dtype=np.float32 if case["result"] == "f32" else np.float64)
    return job.result_wait()


def _whole(events):
    return events.view(np.int32)


# ---- what a pass cannot do without ----------------------------------------------------------
#: Arithmetic of one history: about six flights of 60 operations, a source sample of 250 and one or two
#: interactions of 150.
OPS_PER_HISTORY = 900


def work(case):
    kind = case["kind"]
    if kind == "paths":
        voxels = case["nx"] * case["ny"] * case["nz"]
        crossed = 0.6 * (case["nx"] + case["ny"])  # voxels on an ordinary ray
        return {"bytes": voxels * (1 if case["layout"] == "palette" else 8) + case["rays"] * 36,
                "flops": case["rays"] * crossed * 10.0}
    if kind == "batch":
        voxels = case["n"] * ((case["small"] + case["large"]) / 2) ** 3
        histories = case["n"] * case["histories"] * 1.2
        return {"bytes": voxels * 13, "flops": histories * OPS_PER_HISTORY}
    voxels = case["nx"] * case["ny"] * case["nz"]
    read = 5 if kind == "call" else (8 if case["layout"] == "wide" else 1)
    written = 12 if case["result"] == "f32" else 20
    return {"bytes": voxels * (read + written), "flops": case["histories"] * OPS_PER_HISTORY}


# ---- in 64 bits ------------------------------------------------------------------------------
def exact(case, seed):
    """The radiological paths in double precision from the table that the kernel reads; the transport's
    outputs are sums over random tracks, which have no closed value."""
    if case["kind"] != "paths":
        return None
    (nx, ny, nz), sp, mat, dens = _arrays(case, seed)
    world = _world(case, seed)
    state = prepare(case, seed)
    blob = api.LutBlob.cached(world.materialMap(), state.dworld.max_density(), 150.0)
    info = blob.info()
    rays = torch.from_numpy(state.rays).cuda().double()
    x = torch.from_numpy(info["x"]).cuda()
    coef = torch.from_numpy(info["coef"]).cuda().reshape(-1, info["n_energy"], 3, 2)
    mat, dens = mat.reshape(-1).long(), dens.reshape(-1).double()
    dims = (nx, ny, nz)
    out = torch.zeros(len(rays), dtype=torch.float64, device="cuda")
    for at in range(0, len(rays), 1 << 15):
        r = rays[at:at + (1 << 15)]
        o, d, energy = r[:, 0:3], r[:, 3:6], r[:, 6]
        d = d / d.norm(dim=1, keepdim=True)
        le = energy.log10()
        linear = ((le - info["linear_energy"]) / info["linear_step"]).floor().long() + info["linear_index"]
        seg = torch.where(le > info["linear_energy"], linear, torch.searchsorted(x, le, right=True))
        seg = seg.clamp(max=info["n_energy"] - 1)
        mu = (10.0 ** (coef[:, seg, :, 0] + coef[:, seg, :, 1] * le[None, :, None])).sum(-1)  # (materials, rays)
        cuts, near, far = [], torch.zeros_like(le), torch.full_like(le, math.inf)
        for k in range(3):
            planes = (torch.arange(dims[k] + 1, device="cuda", dtype=torch.float64) - dims[k] / 2) * sp[k]
            t = (planes[None, :] - o[:, k:k + 1]) / d[:, k:k + 1]
            near, far = torch.maximum(near, t.amin(1)), torch.minimum(far, t.amax(1))
            cuts.append(t)
        t = torch.cat(cuts, 1)
        t = torch.minimum(torch.maximum(t, near[:, None]), torch.maximum(near, far)[:, None]).sort(1).values
        length, mid = t[:, 1:] - t[:, :-1], (t[:, 1:] + t[:, :-1]) / 2
        index, stride = 0, 1
        for k in range(3):
            p = (o[:, k:k + 1] + d[:, k:k + 1] * mid) / sp[k] + dims[k] / 2
            index = index + p.floor().long().clamp(0, dims[k] - 1) * stride
            stride *= dims[k]
        out[at:at + (1 << 15)] = 0.1 * (length * dens[index] * mu.gather(0, mat[index].T.contiguous()).T).sum(1)
    return out
