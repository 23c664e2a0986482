"""The work that users of this framework have it do, as timed cases.

Four families, all through the public entry points of lbmb200:

kernel  a row of the kernel table on a full-array lattice: kd->Kernel over a
        number of time steps, which leaves the PDFs in the host mirror
        (Instance.run), as the benchmark driver calls it
list    a fluid-node list row that keeps its state on the device between
        calls, as the permeability solver and the precision runs use it
        (Instance.step_device; with "sums" the solver's conservation sums)
batch   many porous domains advanced together for one check interval with
        their FP64 sums read back, as the serving loop does it; with "admit" a
        domain joins before the interval and leaves after it
solve   one whole permeability solve to its stopping rule (porous.solve_fp64)

Geometries and sizes are those of the tests and the benchmark: channels,
boxes and block lattices for the full-array rows, seeded sphere packings for
the lists, cubic porous domains of edge 32 to 192 for the batches.
"""
import concurrent.futures
import ctypes
import functools
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "lbm-benchmark-kernels_b200"))

import lbmb200  # noqa: E402
from lbmb200 import porous  # noqa: E402

Q = 19
LAMBDA = 3.0 / 16.0
_CX = [0, 0, 1, -1, 1, 1, -1, -1, 0, 0, 1, -1, 0, 0, 0, 0, -1, 1, 0]
_CY = [1, -1, 0, 0, 1, -1, 1, -1, 0, 1, 0, 0, -1, 0, -1, 1, 0, 0, 0]
_CZ = [0, 0, 0, 0, 0, 0, 0, 0, 1, 1, 1, 1, 1, -1, -1, -1, -1, -1, 0]
_INV = [1, 0, 3, 2, 7, 6, 5, 4, 13, 14, 16, 17, 15, 8, 9, 12, 10, 11, 18]
_W = [1 / 3 if not (_CX[d] or _CY[d] or _CZ[d]) else (1 / 18 if abs(_CX[d]) + abs(_CY[d]) + abs(_CZ[d]) == 1 else 1 / 36)
      for d in range(Q)]
_HALF_SCALE = [2.0 ** (15 if w > 0.3 else (18 if w > 0.05 else 19)) for w in _W]  # FP16 storage: delta * 2^k


def _kernel(name, row, geo, dims, periodic, steps, omega=1.0, xforce=1e-5):
    return {"name": name, "family": "kernel", "row": row, "geo": geo, "nx": dims[0], "ny": dims[1], "nz": dims[2],
            "periodic": periodic, "steps": steps, "omega": omega, "xforce": xforce}


def _list(name, row, dims, steps, precision="fp64", porosity=0.4, rmin=6.0, rmax=12.0, packing=1, sums=False,
          omega=1.0):
    return {"name": name, "family": "list", "row": row, "nx": dims[0], "ny": dims[1], "nz": dims[2], "steps": steps,
            "precision": precision, "porosity": porosity, "rmin": rmin, "rmax": rmax, "packing": packing,
            "sums": sums, "omega": omega, "xforce": 1e-5}


def _batch(name, precision, domains, emin, emax, steps, packing=1, admit=0):
    return {"name": name, "family": "batch", "precision": precision, "domains": domains, "emin": emin, "emax": emax,
            "steps": steps, "packing": packing, "admit": admit}


def listed():
    return [
        # the smallest call: a short verification-sized run on an odd lattice (launches and copies)
        _kernel("aa_box_small", "cuda-aa-soa", "box", (21, 18, 13), "xy", 20),
        # the plain method: 64^3 channel, periodic in x, force for u_max about 0.05, 1000 iterations
        _kernel("aa_channel_64", "cuda-aa-soa", "channel", (64, 64, 64), "x", 1000, xforce=1.734e-5),
        # the same far beyond the caches, ragged rows
        _kernel("aa_channel_large", "cuda-aa-soa", "channel", (203, 190, 197), "x", 200),
        # the two-grid full-array row on a lattice with solid blocks
        _kernel("push_blocks", "cuda-push-soa", "blocks-8", (128, 112, 120), "xyz", 100, omega=1.3),
        # the indirect-addressing workload: 256^3 packing, porosity 0.40, radii 6 to 12
        _list("list_aa_fp64_256", "cuda-list-aa-pv-soa", (256, 256, 256), 100),
        # a solver's check interval on an ordinary, ragged domain: 100 steps and the conservation sums
        _list("list_aa_fp64_solver", "cuda-list-aa-pv-soa", (97, 83, 101), 100, porosity=0.45, rmin=3.0, rmax=8.0,
              packing=2, sums=True, omega=1.2),
        # the two-grid pull kernel of the same workload
        _list("list_pull_fp64_160", "cuda-list-pull-split-nt-1s-soa", (160, 160, 160), 50, packing=3),
        # reduced storage on the full packing: PDFs as FP32 and as FP16 deviations
        _list("list_aa_fp32_256", "cuda-list-aa-pv-soa", (256, 256, 256), 100, precision="fp32"),
        _list("list_aa_fp16_256", "cuda-list-aa-pv-soa", (256, 256, 256), 100, precision="fp16"),
        # a serving check interval over many uneven domains
        _batch("batch_fp32_48", "fp32", 48, 32, 128, 100),
        # a lightly loaded server: a domain joins a few small ones for one interval and leaves
        _batch("batch_admit_small", "fp32", 5, 32, 56, 100, packing=2, admit=64),
        # one request served by the plain FP64 kernel, start to stop
        {"name": "solve_fp64_48", "family": "solve", "edge": 48, "porosity": 0.45, "packing": 4, "tol": 1e-6,
         "cap": 20000},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["kernel", "kernel", "list", "list", "list", "batch", "batch", "solve"])
    if kind == "kernel":
        edge = size(14, 200)
        dims = [max(7, int(edge * rng.uniform(0.75, 1.25))) for _ in range(3)]
        row, geo, per = rng.choice([("cuda-aa-soa", "channel", "x"), ("cuda-aa-soa", "box", "xy"),
                                    ("cuda-aa-soa", "fluid", "xyz"), ("cuda-aa-soa", "blocks-5", "xyz"),
                                    ("cuda-push-soa", "channel", "x"), ("cuda-pull-soa", "fluid", "xyz")])
        steps = 2 * max(5, min(200, int(4e8 / (dims[0] * dims[1] * dims[2])) // 2))
        c = _kernel("", row, geo, dims, per, steps, omega=round(rng.uniform(0.8, 1.6), 3))
    elif kind == "list":
        row = rng.choice(["cuda-list-aa-pv-soa"] * 3 + ["cuda-list-pull-soa", "cuda-list-push-soa"])
        edge = size(24, 240)
        dims = [max(20, int(edge * rng.uniform(0.8, 1.2))) for _ in range(3)]
        small = edge < 100 or rng.random() < 0.3
        c = _list("", row, dims, 2 * max(10, min(50, int(4e8 / (dims[0] * dims[1] * dims[2])))),
                  precision=rng.choice(["fp64", "fp32", "fp16"]) if "aa" in row else "fp64",
                  porosity=round(rng.uniform(0.3, 0.6), 3), rmin=3.0 if small else 6.0, rmax=8.0 if small else 12.0,
                  packing=rng.randrange(1, 1 << 20), sums=rng.random() < 0.4, omega=round(rng.uniform(0.8, 1.6), 3))
    elif kind == "batch":
        n = size(1, 40)
        emin = rng.randrange(32, 65)
        c = _batch("", rng.choice(["fp32", "fp32", "fp16"]), n, emin, emin + rng.randrange(8, 64), 100,
                   packing=rng.randrange(1, 1 << 20), admit=rng.choice([0, 0, rng.randrange(32, 100)]))
    else:
        c = {"name": "", "family": "solve", "edge": size(32, 64), "porosity": round(rng.uniform(0.35, 0.6), 3),
             "packing": rng.randrange(1, 1 << 20), "tol": 1e-6, "cap": 20000}
    del c["name"]
    return c


# --- lattices (built once per process; the geometry is the case's, the PDFs are the seed's) ---------------------

@functools.lru_cache(maxsize=256)
def _packing(nx, ny, nz, seed, porosity, rmin, rmax):
    return lbmb200.spheres((nx, ny, nz), seed, porosity, rmin, rmax)[0]


def _periodic(text):
    return tuple(int(a in text) for a in "xyz")


@functools.lru_cache(maxsize=32)
def _geometry(geo, nx, ny, nz, periodic):
    return lbmb200.geometry(geo, (nx, ny, nz), _periodic(periodic))


def _lattice(case):
    if case["family"] == "kernel":
        return _geometry(case["geo"], case["nx"], case["ny"], case["nz"], case["periodic"])
    if case["family"] == "solve":
        e = case["edge"]
        return _packing(e, e, e, case["packing"], case["porosity"], 3.0, 8.0)
    return _packing(case["nx"], case["ny"], case["nz"], case["packing"], case["porosity"], case["rmin"], case["rmax"])


def _domains(case, seed):
    """(lattices, omegas, forces) of a batch: residents, then the one that joins."""
    rng = random.Random(case["packing"])
    specs = [(rng.randint(case["emin"], case["emax"]), rng.randrange(1 << 30), rng.uniform(0.3, 0.6))
             for _ in range(case["domains"])]
    if case["admit"]:
        specs.append((case["admit"], rng.randrange(1 << 30), rng.uniform(0.3, 0.6)))
    with concurrent.futures.ThreadPoolExecutor(max(1, min(16, os.cpu_count() or 1))) as pool:
        lats = list(pool.map(lambda s: _packing(s[0], s[0], s[0], s[1], s[2], 3.0, 8.0), specs))
    r = random.Random(seed)
    return lats, [r.uniform(0.8, 1.6) for _ in lats], [1e-5 * r.uniform(0.5, 2.0) for _ in lats]


def _solid_free(lat):
    """Fluid cells as a (nX, nY, nZ) boolean array."""
    nx, ny, nz = lat.dims
    return np.ascontiguousarray((lat.mask.reshape(nz, ny, nx) != 0).transpose(2, 1, 0))


# --- inputs ------------------------------------------------------------------------------------------------------

def _start(n, seed):
    """PDFs of n nodes near a random equilibrium: (19, n), FP64, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def noise(a):
        return a * torch.randn(n, generator=g, device="cuda", dtype=torch.float64).clamp_(-3, 3)

    rho, ux, uy, uz = 1.0 + noise(0.005), 0.02 + noise(0.01), noise(0.01), noise(0.01)
    usq = 1.5 * (ux * ux + uy * uy + uz * uz)
    f = torch.empty((Q, n), device="cuda", dtype=torch.float64)
    for d in range(Q):
        cu = _CX[d] * ux + _CY[d] * uy + _CZ[d] * uz
        f[d] = _W[d] * (rho + 3.0 * cu + 4.5 * cu * cu - usq) * (1.0 + noise(1e-3))
    return f


def _stored(f, precision):
    """PDFs in a storage format: as they are, or deviations from the weights."""
    if precision == "fp64":
        return f
    w = torch.tensor(_W, device=f.device, dtype=torch.float64)[:, None]
    if precision == "fp32":
        return (f - w).float()
    return ((f - w) * torch.tensor(_HALF_SCALE, device=f.device, dtype=torch.float64)[:, None]).half()


def _restored(raw, precision):
    if precision == "fp64":
        return raw.double()
    w = torch.tensor(_W, device=raw.device, dtype=torch.float64)[:, None]
    if precision == "fp32":
        return raw.double() + w
    return raw.double() / torch.tensor(_HALF_SCALE, device=raw.device, dtype=torch.float64)[:, None] + w


class _Instance:
    """A kernel instance that lives as long as anything that refers to its memory."""

    def __init__(self, row, lat, args):
        self.inst = lbmb200.kernel(row).init(lat, args)

    def __del__(self):
        self.inst.deinit()


class _DeviceArray:
    """Device memory of an instance, for torch.as_tensor."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 2}


class _HostArray:
    """Host memory of an instance, for numpy.asarray."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 3}


class _Domains:
    """A batch that closes with its last reference."""

    def __init__(self, precision, n):
        self.batch = lbmb200.Batch(precision, budget_gb=20.0, max_domains=n)

    def __del__(self):
        self.batch.close()


class _State:
    pass


def _device_view(owner, precision):
    """The list instance's PDFs on the device, (19, nFluid), without a copy."""
    p, nc, nf, st = ctypes.c_void_p(), ctypes.c_longlong(), ctypes.c_int(), ctypes.c_void_p()
    if lbmb200.lib().lbm_b200_device_state(owner.inst.kdp, ctypes.byref(p), ctypes.byref(nc), ctypes.byref(nf),
                                           ctypes.byref(st)):
        raise RuntimeError("no device state")
    kind = {"fp64": "<f8", "fp32": "<f4", "fp16": "<f2"}[precision]
    return torch.as_tensor(_DeviceArray(owner, p.value, (Q, nc.value), kind), device="cuda")[:, : nf.value]


def _mirror_views(owner, row):
    """Per direction, the (nX, nY, nZ) logical PDFs in the host mirror of a full-array row."""
    kd = owner.inst.kd
    nx, ny, nz = (kd.Dims[i] for i in range(3))
    gx, gy = nx + 2, ny + 2
    z0 = 4  # first interior z of a row
    pitch = (nz + z0 + 1 + 3) // 4 * 4
    m = np.asarray(_HostArray(owner, ctypes.cast(kd.Pdfs[0], ctypes.c_void_p).value, (Q, gx, gy, pitch)))
    out = []
    for d in range(Q):
        sx, sy, sz = (_CX[d], _CY[d], _CZ[d]) if row == "cuda-pull-soa" else (0, 0, 0)
        out.append(m[d, 1 - sx: 1 - sx + nx, 1 - sy: 1 - sy + ny, z0 - sz: z0 - sz + nz])
    return out


def prepare(case, seed):
    s = _State()
    s.case = case
    fam = case["family"]
    if fam == "batch":
        s.lats, s.omegas, s.forces = _domains(case, seed)
        s.owner = _Domains(case["precision"], case["domains"] + 1)
        for k in range(case["domains"]):
            s.owner.batch.add(s.lats[k], omega=s.omegas[k], lam=LAMBDA, xforce=s.forces[k])
        return s
    if fam == "solve":
        s.lat = _lattice(case)
        s.omega = 0.8 + 0.8 * random.Random(seed).random()
        return s
    lat = _lattice(case)
    s.cd = lbmb200.case(omega=case["omega"], xforce=case["xforce"], iterations=case["steps"])
    if fam == "list":
        s.owner = _Instance(case["row"], lat, ["-lambda", "3/16"] + (
            [] if case["precision"] == "fp64" else ["-precision", case["precision"]]))
        _device_view(s.owner, case["precision"]).copy_(_stored(_start(lat.n_fluid, seed), case["precision"]))
        torch.cuda.synchronize()  # the instance steps on a stream of its own
        return s
    s.owner = _Instance(case["row"], lat, ["-lambda", "3/16"])
    s.views = _mirror_views(s.owner, case["row"])
    f = _start(lat.mask.size, seed).reshape(Q, *lat.dims)
    f *= torch.from_numpy(_solid_free(lat)).to(f.device)
    f = f.cpu().numpy()
    for d in range(Q):
        s.views[d][...] = f[d]
    lbmb200.lib().lbm_b200_mark_mirror_dirty(s.owner.inst.kdp)
    return s


def run(s):
    case = s.case
    fam = case["family"]
    if fam == "kernel":
        s.owner.inst.run(s.cd)
        return s.views
    if fam == "list":
        s.owner.inst.step_device(s.cd, case["steps"])
        out = {"pdfs": _device_view(s.owner, case["precision"])}
        if case["sums"]:
            out["sums"] = list(s.owner.inst.moments())
        return out
    if fam == "batch":
        b, slot = s.owner.batch, None
        if case["admit"]:
            slot = b.add(s.lats[-1], omega=s.omegas[-1], lam=LAMBDA, xforce=s.forces[-1])
        b.step(case["steps"], graph=True)
        out = {"sums": b.moments()}
        if slot is not None:
            out["left"] = b.remove(slot)
        else:
            out["field"] = b.get_field(0)
        return out
    r = porous.solve_fp64(s.lat, omega=s.omega, lam=LAMBDA, tol=case["tol"], cap=case["cap"])
    return {"k": r["k"], "u": r["u"], "steps": r["steps"]}


# --- what a pass cannot do without -------------------------------------------------------------------------------

_FLOPS = 225  # one relaxation with its body force, adds and multiplies


def work(case):
    """Each pass reads its PDFs once and writes them once; the links of a list once."""
    fam = case["family"]
    if fam == "batch":
        n = sum(lat.n_fluid for lat in _domains(case, 0)[0])
        per = {"fp32": 4, "fp16": 2}[case["precision"]]
        return {"bytes": 2 * Q * per * n, "flops": _FLOPS * n * case["steps"]}
    n = _lattice(case).n_fluid
    if fam == "solve":
        return {"bytes": 2 * Q * 8 * n, "flops": _FLOPS * n * 1000}
    per = {"fp64": 8, "fp32": 4, "fp16": 2}[case.get("precision", "fp64")]
    return {"bytes": 2 * Q * per * n, "flops": _FLOPS * n * case["steps"]}


# --- the same in plain torch, 64 bits ----------------------------------------------------------------------------

def _relax(f, omega):
    """TRT relaxation of (19, ...) PDFs."""
    odd = 1.0 / (0.5 + LAMBDA / (1.0 / omega - 0.5))
    rho = f.sum(0)
    ux = sum(_CX[d] * f[d] for d in range(Q) if _CX[d])
    uy = sum(_CY[d] * f[d] for d in range(Q) if _CY[d])
    uz = sum(_CZ[d] * f[d] for d in range(Q) if _CZ[d])
    dit = rho - 1.5 * (ux * ux + uy * uy + uz * uz)
    out = torch.empty_like(f)
    out[18] = f[18] - omega * (f[18] - _W[18] * dit)
    for d in range(18):
        j = _INV[d]
        if j < d:
            continue
        cu = _CX[d] * ux + _CY[d] * uy + _CZ[d] * uz
        even = omega * (0.5 * (f[d] + f[j]) - _W[d] * (4.5 * cu * cu + dit))
        anti = odd * (0.5 * (f[d] - f[j]) - 3.0 * _W[d] * cu)
        out[d] = f[d] - even - anti
        out[j] = f[j] - even + anti
    return out


class _Links:
    """Streaming with bounce back on a lattice whose open faces are periodic or solid."""

    def __init__(self, lat):
        self.fluid = torch.from_numpy(_solid_free(lat)).cuda()
        self.wall = [~torch.roll(self.fluid, (_CX[d], _CY[d], _CZ[d]), (0, 1, 2)) for d in range(18)]

    def stream(self, post, xforce):
        """Incoming PDFs: direction d from x - c_d, or what the node itself sent against a wall there."""
        out = torch.empty_like(post)
        for d in range(18):
            moved = torch.roll(post[d], (_CX[d], _CY[d], _CZ[d]), (0, 1, 2))
            out[d] = torch.where(self.wall[d], post[_INV[d]], moved) + 3.0 * _W[d] * _CX[d] * xforce
        out[18] = post[18]
        return out * self.fluid


def _steps(f, links, omega, xforce, n):
    for _ in range(n):
        f = links.stream(_relax(f, omega), xforce)
    return f


def _pull_steps(f, links, omega, xforce, n):
    """The state of a two-grid pull row: a node's own outgoing PDFs, body force included."""
    force = torch.tensor([3.0 * _W[d] * _CX[d] * xforce for d in range(Q)], device=f.device,
                         dtype=torch.float64)[:, None, None, None]
    for _ in range(n):
        f = (_relax(links.stream(f, 0.0), omega) + force) * links.fluid
    return f


def _sums(f):
    jx = sum(_CX[d] * f[d].sum() for d in range(Q))
    jy = sum(_CY[d] * f[d].sum() for d in range(Q))
    jz = sum(_CZ[d] * f[d].sum() for d in range(Q))
    return [float(f.sum()), float(jx), float(jy), float(jz)]


def _rest(links):
    w = torch.tensor(_W, device="cuda", dtype=torch.float64)[:, None, None, None]
    return w * links.fluid


def _exact_batch(case, seed):
    lats, omegas, forces = _domains(case, seed)
    sums = np.zeros((case["domains"] + 1, 4))
    field = None
    for k, lat in enumerate(lats):
        links = _Links(lat)
        f = _steps(_rest(links), links, omegas[k], forces[k], case["steps"])
        sums[k] = _sums(f)
        if k == 0 and not case["admit"]:
            a = f.permute(3, 2, 1, 0).reshape(-1, Q).cpu().numpy()
            field = np.where((lat.mask != 0)[:, None], a, np.nan)
    return {"sums": sums, "left": None} if case["admit"] else {"sums": sums, "field": field}


def _exact_solve(case, seed):
    lat = _lattice(case)
    links, omega, x = _Links(lat), 0.8 + 0.8 * random.Random(seed).random(), 1e-5
    f, prev, steps = _rest(links), None, 0
    while True:
        f = _steps(f, links, omega, x, 100)
        steps += 100
        jx = _sums(f)[1]
        u = porous.mean_ux(jx, lat.n_fluid, x)
        if porous.stop_status(u, prev, steps, case["tol"], case["cap"]):
            return {"k": porous.permeability(jx, lat.n_fluid, lat.mask.size, omega, x), "u": u, "steps": None}
        prev = u


def exact(case, seed):
    fam = case["family"]
    if fam == "batch":
        return _exact_batch(case, seed)
    if fam == "solve":
        return _exact_solve(case, seed)
    lat = _lattice(case)
    links = _Links(lat)
    if fam == "kernel":
        f = _start(lat.mask.size, seed).reshape(Q, *lat.dims) * links.fluid
        f = _steps(f, links, case["omega"], case["xforce"], case["steps"])
        return [f[d] for d in range(Q)]
    f = torch.zeros((Q, *lat.dims), device="cuda", dtype=torch.float64)
    f[:, links.fluid] = _restored(_stored(_start(lat.n_fluid, seed), case["precision"]), case["precision"])
    walk = _pull_steps if "pull" in case["row"] else _steps
    f = walk(f, links, case["omega"], case["xforce"], case["steps"])[:, links.fluid]
    if case["precision"] == "fp64":
        out = {"pdfs": f}
    else:
        w = torch.tensor(_W, device="cuda", dtype=torch.float64)[:, None]
        sc = torch.tensor(_HALF_SCALE if case["precision"] == "fp16" else [1.0] * Q, device="cuda",
                          dtype=torch.float64)[:, None]
        out = {"pdfs": (f - w) * sc}
    if case["sums"]:
        out["sums"] = _sums(f)
    return out
