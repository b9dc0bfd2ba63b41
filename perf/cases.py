"""Performance cases of the FDM stepper: what users have it do, through its public entry points.

A case is a dict of plain values.  Its "kind" says which entry points a pass calls:

  run      upload a state, take "steps" steps of the plan's integrator, read the state back.
           "stats" = "each" calls step() for every step and keeps the last statistics (the
           runner's loop); "last" calls step_n() once (a time window without a host round trip).
  batch    "steps" Heun steps of an ensemble of uneven problems, all states read back.
  adjoint  upload, a Heun trajectory with checkpoints, its pull-back: all gradients.
  field    upload, refresh the observables, read H_eff (the multilayer host's call).
  demag    the allocation-free demag entry point on device arrays.

Common fields: nx, ny, nz; "dtype" f64 or f32 (the FP32-mixed form); "material" uniform, mask
(a disk with a hole), ms_map (per-cell Ms), mask_ms (both) or regions (two exchange regions);
"integrator" heun, rk4, rk23 or dp45; dt.  The adaptive integrators run with dt_max = dt, a
window of equal steps well inside their error bound.  States are random unit vectors, as the
planner's "random" initial magnetisation.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from fullmag_b200 import native_fdm as nf

MS, AEX, GAMMA = 8.0e5, 1.3e-11, 2.211e5
MAX_ERROR = 1e-5
INTEGRATORS = {"heun": nf.HEUN, "rk4": nf.RK4, "rk23": nf.RK23, "dp45": nf.DP45}
EVALS = {"heun": 2, "rk4": 4, "rk23": 3, "dp45": 6}
ENERGIES = ("exchange_energy_joules", "demag_energy_joules", "external_energy_joules", "total_energy_joules")
AMPLITUDES = ("max_effective_field_amplitude", "max_demag_field_amplitude", "max_rhs_amplitude")


def listed():
    return [
        # the smallest film (3.125 nm cells), one call per step with its statistics: launches and latency
        dict(name="film_64x16_f64", kind="run", nx=64, ny=16, nz=1, dtype="f64", integrator="heun", material="uniform",
             cell=3.125e-9, alpha=0.02, dt=1e-13, steps=40, stats="each"),
        # a film whose sides are not powers of two, RK4, a window of steps
        dict(name="film_250x100_f64_rk4", kind="run", nx=250, ny=100, nz=1, dtype="f64", integrator="rk4",
             material="uniform", cell=2.5e-9, alpha=0.02, dt=5e-14, steps=20, stats="last"),
        # an ordinary extended film in FP32-mixed
        dict(name="film_512x512_f32", kind="run", nx=512, ny=512, nz=1, dtype="f32", integrator="heun",
             material="uniform", cell=4e-9, alpha=0.1, dt=5e-14, steps=40, stats="last"),
        # the headline grid in both precisions: a window between two outputs of the state
        dict(name="slab_512x512x8_f32", kind="run", nx=512, ny=512, nz=8, dtype="f32", integrator="heun",
             material="uniform", cell=2e-9, alpha=0.5, dt=5e-14, steps=20, stats="last"),
        dict(name="slab_512x512x8_f64", kind="run", nx=512, ny=512, nz=8, dtype="f64", integrator="heun",
             material="uniform", cell=2e-9, alpha=0.5, dt=5e-14, steps=10, stats="each"),
        # the largest: a thick masked disk (a band of the 1024 x 1024 x 16 one), adaptive DP45
        dict(name="disk_1024x512x16_f32_dp45", kind="run", nx=1024, ny=512, nz=16, dtype="f32", integrator="dp45",
             material="mask", cell=2e-9, alpha=0.1, dt=1e-14, steps=4, stats="each"),
        # odd grids in three dimensions, as they come from a geometry and a cell size
        dict(name="slab_300x180x5_f32_mask_ms", kind="run", nx=300, ny=180, nz=5, dtype="f32", integrator="dp45",
             material="mask_ms", cell=2.5e-9, alpha=0.05, dt=1e-14, steps=6, stats="each"),
        dict(name="slab_240x150x6_f64_regions", kind="run", nx=240, ny=150, nz=6, dtype="f64", integrator="heun",
             material="regions", cell=2e-9, alpha=0.1, dt=5e-14, steps=15, stats="last"),
        # an ensemble of uneven problems, as a parameter study draws them
        dict(name="batch_48_f32", kind="batch", count=48, ensemble=45, dtype="f32", dt=5e-14, steps=30),
        # gradients of a film with respect to its Ms map and fields
        dict(name="adjoint_256x256_f64", kind="adjoint", nx=256, ny=256, nz=1, dtype="f64", material="ms_map",
             cell=4e-9, alpha=0.05, dt=1e-13, steps=32),
        # one layer's fields for a host that couples several layers
        dict(name="field_128x64x4_f64", kind="field", nx=128, ny=64, nz=4, dtype="f64", material="uniform",
             cell=2.5e-9, alpha=0.1),
        # the demag field alone, inside a host framework that owns the device memory
        dict(name="demag_128x128x8_f64", kind="demag", nx=128, ny=128, nz=8, dtype="f64", cell=2e-9),
    ]


# padded lengths 2n with prime factors up to 7: the grids the entry points take
_SMOOTH = [n for n in range(8, 1025) if math.prod(p ** e for p in (2, 3, 5, 7)
                                                  for e in [next(k for k in range(12) if n % p ** (k + 1))]) == n]
_POW2 = [n for n in _SMOOTH if n & (n - 1) == 0]


def _nearest(v, of):
    return min(of, key=lambda n: abs(math.log(n / v)))


def draw(rng):
    kind = rng.choices(("run", "batch", "adjoint", "field", "demag"), (8, 1, 1.5, 1, 1))[0]
    cell = rng.uniform(2e-9, 4e-9)
    alpha = rng.choice((0.02, 0.05, 0.1, 0.5))
    dtype = rng.choice(("f64", "f32"))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(8, 64), ensemble=rng.randint(0, 10 ** 6), dtype=dtype, dt=5e-14, steps=rng.randint(8, 30))
    if kind == "demag":
        while True:
            nx, ny, nz = (2 ** rng.randint(4, 8), 2 ** rng.randint(4, 8), 2 ** rng.randint(0, 3))
            if 3 * nz * (nx + 1) * (ny if nz == 1 else 3 * ny) * 16 < 30 << 20:
                return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype="f64", cell=cell)
    most = {"run": 2.1e6, "adjoint": 2.5e5, "field": 1e6}[kind]
    least = {"run": 512.0, "adjoint": 4096.0, "field": 2048.0}[kind]
    cells = math.exp(rng.uniform(math.log(least), math.log(most)))
    nz = 1 if kind == "adjoint" or rng.random() < 0.4 else rng.choice((2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 15, 16))
    nz = min(nz, max(1, int(cells / 512)))
    nz = nz if nz not in (11, 13) else nz - 1
    of = _POW2 if rng.random() < 0.4 else _SMOOTH
    ratio = math.exp(rng.uniform(-math.log(4), math.log(4)))
    nx = _nearest(min(1024.0, math.sqrt(cells / nz * ratio)), of)
    ny = _nearest(min(1024.0, cells / nz / nx), of)
    case = dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype, cell=cell, alpha=alpha)
    if kind == "adjoint":
        return case | dict(material=rng.choice(("uniform", "ms_map")), dt=1e-13, steps=rng.randint(8, 32))
    case["material"] = rng.choice(("uniform", "uniform", "mask", "ms_map", "mask_ms", "regions"))
    if kind == "field":
        return case
    integrator = rng.choice(("heun", "heun", "rk4", "rk23", "dp45"))
    steps = max(3, min(40, int(8e6 / (nx * ny * nz)))) * 2 // EVALS[integrator]
    return case | dict(integrator=integrator, dt=rng.choice((1e-14, 2e-14)) if integrator in ("rk23", "dp45") else 5e-14,
                       steps=max(2, steps), stats=rng.choice(("each", "last")))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _numpy_dtype(case):
    return np.float64 if case["dtype"] == "f64" else np.float32


def _precision(case):
    return nf.PRECISION_DOUBLE if case["dtype"] == "f64" else nf.PRECISION_SINGLE


def _unit_vectors(seed, n, dtype):
    """(n, 3) random unit vectors as the case's state type holds them, in float64."""
    g = torch.Generator().manual_seed(seed)
    v = torch.rand((n, 3), generator=g, dtype=torch.float64) * 2.0 - 1.0
    v /= v.norm(dim=1, keepdim=True).clamp_min(1e-12)
    return v.numpy().astype(dtype).astype(np.float64)


def _material(case, seed):
    """The plan's material fields: active_mask, ms_map, region_mask and exchange_lut."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind, out = case.get("material", "uniform"), {}
    x, y = np.arange(nx) + 0.5 - nx / 2, np.arange(ny) + 0.5 - ny / 2
    r2 = (x[None, :] / (nx / 2)) ** 2 + (y[:, None] / (ny / 2)) ** 2
    if kind in ("mask", "mask_ms"):
        disk = (r2 <= 1.0) & (r2 > 0.15 ** 2)
        out["active_mask"] = np.repeat(disk[None], nz, axis=0).astype(np.uint8).reshape(-1)
    if kind in ("ms_map", "mask_ms"):
        out["ms_map"] = np.random.default_rng(seed + 1).uniform(6e5, 1e6, nx * ny * nz)
    if kind == "regions":
        lut = np.zeros((nf.MAX_EXCHANGE_REGIONS, nf.MAX_EXCHANGE_REGIONS))
        lut[0, 0], lut[1, 1], lut[0, 1], lut[1, 0] = AEX, 0.6 * AEX, 0.75 * AEX, 0.75 * AEX
        out["region_mask"] = np.repeat((r2 <= 0.5)[None], nz, axis=0).astype(np.uint32).reshape(-1)
        out["exchange_lut"] = lut.reshape(-1)
    return out


def _h_ext():
    return (10e-3 / nf.MU0, 5e-3 / nf.MU0, -2e-3 / nf.MU0)


def _plan(case, seed, m0):
    kw = _material(case, seed)
    if case.get("integrator") in ("rk23", "dp45"):
        kw["adaptive"] = (MAX_ERROR, 1e-18, case["dt"], 0.8)
    if case["kind"] == "adjoint":
        kw.update(ac_field=(20e-3 / nf.MU0, 0.0, 0.0), ac_frequency_hz=5e9)
    return nf.FdmPlan(cells=(case["nx"], case["ny"], case["nz"]), cell_size=(case["cell"],) * 3,
                      initial_magnetization=m0, saturation_magnetisation=MS, exchange_stiffness=AEX,
                      damping=case["alpha"], gyromagnetic_ratio=GAMMA, precision=_precision(case),
                      integrator=INTEGRATORS[case.get("integrator", "heun")], external_field=_h_ext(),
                      demag_source=nf.DEMAG_NEWELL, **kw)


def _batch_problems(case, seed=None):
    """Grids 32x32x1 to 256x128x4, Ms, A, alpha and in-plane field drawn per problem of the
    ensemble; the states (left out without a seed) come from the seed."""
    rng = np.random.default_rng(case["ensemble"])
    out = []
    for i in range(case["count"]):
        nx, ny, nz = int(rng.integers(32, 257)), int(rng.integers(32, 129)), int(rng.integers(1, 5))
        d, ang, b = rng.uniform(2e-9, 4e-9), rng.uniform(0, 2 * np.pi), rng.uniform(0, 50e-3) / nf.MU0
        out.append(dict(cells=(nx, ny, nz), cell_size=(d, d, d), ms=rng.uniform(6e5, 1.2e6),
                        aex=rng.uniform(1e-11, 2e-11), alpha=rng.uniform(0.01, 0.5),
                        h_ext=(b * np.cos(ang), b * np.sin(ang), 0.0), gamma=GAMMA))
        if seed is not None:
            out[-1]["m0"] = _unit_vectors(seed * 1009 + i, nx * ny * nz, _numpy_dtype(case)).reshape(-1)
    return out


def _loss_gradient(case, seed):
    """dL/dm of a weighted mean over the central quarter of the film (AoS)."""
    nx, ny = case["nx"], case["ny"]
    w = np.zeros((ny, nx, 3))
    rng = np.random.default_rng(seed + 2)
    part = w[ny // 4: ny - ny // 4, nx // 4: nx - nx // 4]
    part[...] = rng.uniform(0.5, 1.0, part.shape)
    return w.reshape(-1)


def _octant(spectra, nx, ny, nz):
    """[6][KZ][nx+1][ny+1] of the interleaved spectra (KZ = 1 for a film)."""
    Lz, KZ = (1, 1) if nz == 1 else (2 * nz, nz + 1)
    return np.ascontiguousarray(np.stack([
        s[0::2].reshape(Lz, 2 * ny, 2 * nx)[:KZ, :ny + 1, :nx + 1].transpose(0, 2, 1) for s in spectra]))


def _noalloc_entry():
    fn = nf.load_library().fullmag_fdm_demag_field_f64_noalloc
    fn.restype = C.c_int
    fn.argtypes = [C.c_uint32, C.c_uint32, C.c_uint32, C.c_int, C.c_void_p, C.c_void_p, C.c_double, C.c_void_p,
                   C.c_void_p, C.c_char_p, C.c_uint64]
    return fn


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return dict(case=case, batch=nf.NativeFdmBatch(_batch_problems(case, seed), _precision(case)))
    n = case["nx"] * case["ny"] * case["nz"]
    m0 = _unit_vectors(seed, n, _numpy_dtype(case))
    if kind == "demag":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        spectra = nf.newell_spectra(nx, ny, nz, *(case["cell"],) * 3, thin_film_2d=nz == 1)
        return dict(case=case, fn=_noalloc_entry(), octant=torch.from_numpy(_octant(spectra, nx, ny, nz)).cuda(),
                    m=torch.from_numpy(np.ascontiguousarray(m0.T)).cuda(), h=torch.empty(3 * n, dtype=torch.float64, device="cuda"),
                    err=C.create_string_buffer(512))
    # page-locked host arrays, as a program that moves states every window keeps them
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    host_in = torch.from_numpy(m0.reshape(-1)).to(dtype).pin_memory()
    host_out = torch.empty(3 * n, dtype=dtype, pin_memory=True)
    state = dict(case=case, be=nf.NativeFdmBackend(_plan(case, seed, m0.reshape(-1))), m0=host_in.numpy(),
                 out=host_out.numpy(), keep=(host_in, host_out))
    if kind == "adjoint":
        state["g"] = _loss_gradient(case, seed)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind, dtype = case["kind"], _numpy_dtype(case)
    if kind == "demag":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        rc = state["fn"](nx, ny, nz, int(nz == 1), state["octant"].data_ptr(), state["m"].data_ptr(), MS,
                         state["h"].data_ptr(), torch.cuda.current_stream().cuda_stream, state["err"], 512)
        if rc != nf.OK:
            raise nf.RunError(state["err"].value.decode())
        return state["h"]
    if kind == "batch":
        b = state["batch"]
        b.step_n(case["dt"], case["steps"])
        return np.concatenate([b.copy_m(i).astype(dtype) for i in range(case["count"])])
    be = state["be"]
    be.upload_m(state["m0"])
    if kind == "field":
        be.refresh_observables()
        return be.copy_field(nf.OBS_H_EFF, dtype=dtype, out=state["out"])
    if kind == "adjoint":
        be.adjoint_forward(case["dt"], case["steps"])
        g = be.adjoint_backward(state["g"])
        return {"m": be.copy_field(nf.OBS_M, dtype=dtype, out=state["out"]),
                **{k: g[k].astype(dtype) for k in ("dl_dms", "dl_dh_ext", "dl_dh_ac", "dl_dm0")}}
    if case["stats"] == "each":
        for _ in range(case["steps"]):
            st = be.step(case["dt"])
    else:
        st = be.step_n(case["dt"], case["steps"])
    return {"m": be.copy_field(nf.OBS_M, dtype=dtype, out=state["out"]),
            "energies": np.array([st[k] for k in ENERGIES], dtype), "amplitudes": np.array([st[k] for k in AMPLITUDES], dtype)}


# ---------------------------------------------------------------------------
# work: per field evaluation the state and the field's tensor (the real octant of
# its spectrum) read once and a state or slope written once; flops of the pruned
# real transforms (x of the rows, y of the half spectrum, z of its columns, both
# ways), the tensor product and the pointwise model
# ---------------------------------------------------------------------------
def _eval_work(nx, ny, nz, scalar):
    lg = lambda n: math.log2(max(2, n))  # noqa: E731
    n, kx = nx * ny * nz, nx + 1
    flops = 3 * nz * ny * 2.5 * 2 * nx * lg(2 * nx) + 3 * nz * kx * 5 * 2 * ny * lg(2 * ny)
    if nz > 1:
        flops += 3 * kx * 2 * ny * 5 * 2 * nz * lg(2 * nz)
    flops = 2 * flops + 36 * kx * 2 * ny * max(1, 2 * nz if nz > 1 else 1) + 120 * n
    tensor = (4 if nz == 1 else 6) * kx * (ny + 1) * (1 if nz == 1 else nz + 1) * scalar
    return 6 * n * scalar + tensor, flops


def work(case):
    s = 8 if case["dtype"] == "f64" else 4
    if case["kind"] == "batch":
        per = [_eval_work(*p["cells"], s) for p in _batch_problems(case)]
        evals = 2 * case["steps"]
        return {"bytes": float(evals * sum(b for b, _ in per)), "flops": float(evals * sum(f for _, f in per))}
    b, f = _eval_work(case["nx"], case["ny"], case["nz"], s)
    evals = {"run": lambda: EVALS[case["integrator"]] * case["steps"], "adjoint": lambda: 6 * case["steps"],
             "field": lambda: 1, "demag": lambda: 1}[case["kind"]]()
    return {"bytes": float(evals * b), "flops": float(evals * f)}


# ---------------------------------------------------------------------------
# the same model in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _newell_f(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    r = torch.sqrt(x2 + y2 + z2)
    out = (2 * x2 - y2 - z2) * r / 6

    def part(c, a2, b2, num):
        d = a2 + b2
        return torch.where(d > 0, num * torch.log1p(2 * c * (c + r) / torch.where(d > 0, d, torch.ones_like(d))), 0 * d)
    out = out + part(y, x2, z2, y * (z2 - x2) / 4) + part(z, x2, y2, z * (y2 - x2) / 4)
    xr = x * r
    return out - torch.where(xr != 0, x * y * z * torch.atan(y * z / torch.where(xr != 0, xr, torch.ones_like(xr))), 0 * xr)


def _newell_g(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    r = torch.sqrt(x2 + y2 + z2)
    out = -x * y * r / 3

    def part(c, a2, b2, num):
        d = a2 + b2
        return torch.where(d > 0, num * torch.log1p(2 * c * (c + r) / torch.where(d > 0, d, torch.ones_like(d))), 0 * d)

    def angle(c, a, b, num):
        d = c * r
        return torch.where(d != 0, num * torch.atan(a * b / torch.where(d != 0, d, torch.ones_like(d))), 0 * d)
    out = out + part(z, x2, y2, x * y * z / 2) + part(x, y2, z2, y * (3 * z2 - y2) / 12) + part(y, x2, z2, x * (3 * z2 - x2) / 12)
    return out - angle(z, x, y, z2 * z / 6) - angle(y, x, z, y2 * z / 2) - angle(x, y, z, x2 * z / 2)


def _tensor(nx, ny, nz, d, device):
    """The demag tensor xx, yy, zz, xy, xz, yz at the offsets [0, n): (nz, ny, nx) each;
    Newell's second differences up to 40 cells, the point dipole beyond."""
    ax = lambda n, lo: torch.arange(lo, n, dtype=torch.float64, device=device)  # noqa: E731
    far_from = 40
    near = [min(n, far_from) for n in (nx, ny, nz)]
    gx, gy, gz = (ax(near[i] + 1, -1) for i in range(3))
    Z, Y, X = torch.meshgrid(gz, gy, gx, indexing="ij")
    pots = (_newell_f(X, Y, Z), _newell_f(Y, X, Z), _newell_f(Z, Y, X),
            _newell_g(X, Y, Z), _newell_g(X, Z, Y), _newell_g(Y, Z, X))
    zz, yy, xx = torch.meshgrid(ax(nz, 0), ax(ny, 0), ax(nx, 0), indexing="ij")
    r2 = xx * xx + yy * yy + zz * zz
    rr = torch.sqrt(torch.where(r2 > 0, r2, torch.ones_like(r2)))
    r3 = rr ** 3
    dip = (lambda a: (1 / r3 - 3 * a * a / (r3 * rr * rr)) / (4 * math.pi),
           lambda a, b: -3 * a * b / (4 * math.pi * r3 * rr * rr))
    far = (dip[0](xx), dip[0](yy), dip[0](zz), dip[1](xx, yy), dip[1](xx, zz), dip[1](yy, zz))
    out = []
    for pot, asym in zip(pots, far):
        for dim in range(3):
            c = pot.shape[dim]
            pot = 2 * pot.narrow(dim, 1, c - 2) - pot.narrow(dim, 0, c - 2) - pot.narrow(dim, 2, c - 2)
        val = asym.clone()
        val[:near[2], :near[1], :near[0]] = pot / (4 * math.pi)
        out.append(torch.where(r2 >= far_from ** 2, asym, val))
    return out


class _Model:
    """Exchange, demag, Zeeman and LLG on (3, nz, ny, nx) fields in 64 bits."""

    def __init__(self, cells, d, device, *, ms=MS, aex=AEX, alpha=0.1, h_ext=(0.0, 0.0, 0.0), mask=None, ms_map=None,
                 region=None, lut=None, h_ac=(0.0, 0.0, 0.0), frequency=0.0):
        self.nx, self.ny, self.nz = nx, ny, nz = cells
        self.d, self.aex, self.alpha = d, aex, alpha
        f = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=device)  # noqa: E731
        self.ms = f(ms_map).reshape(nz, ny, nx) if ms_map is not None else torch.full((nz, ny, nx), ms, dtype=torch.float64, device=device)
        self.on = f(mask).reshape(nz, ny, nx) if mask is not None else torch.ones((nz, ny, nx), dtype=torch.float64, device=device)
        self.region = torch.as_tensor(region.astype(np.int64), device=device).reshape(nz, ny, nx) if region is not None else None
        self.lut = f(lut).reshape(nf.MAX_EXCHANGE_REGIONS, -1) if lut is not None else None
        self.h_ext, self.h_ac, self.frequency = f(h_ext), f(h_ac), frequency
        odd = ((), (), (), (2, 1), (2, 0), (1, 0))  # odd axes (dims of (z, y, x)) of each component
        L = (2 * nz if nz > 1 else 1, 2 * ny, 2 * nx)
        self.L, self.spec = L, []
        for comp, axes in zip(_tensor(nx, ny, nz, d, device), odd):
            for dim, n in ((0, nz), (1, ny), (2, nx)):
                if L[dim] == 1:
                    continue
                back = comp.narrow(dim, 1, n - 1).flip(dim) if n > 1 else comp.narrow(dim, 0, 0)
                gap = torch.zeros_like(comp.narrow(dim, 0, 1))
                comp = torch.cat((comp, gap, -back if dim in axes else back), dim)
            if nz == 1 and 0 in axes:
                comp = torch.zeros_like(comp)
            self.spec.append(torch.fft.rfftn(comp))

    def demag(self, m):
        mk = torch.fft.rfftn(m * (self.ms * self.on), s=self.L, dim=(1, 2, 3))
        xx, yy, zz, xy, xz, yz = self.spec
        out = []
        for row in ((xx, xy, xz), (xy, yy, yz), (xz, yz, zz)):
            h = torch.fft.irfftn(row[0] * mk[0] + row[1] * mk[1] + row[2] * mk[2], s=self.L)
            out.append(-h[:self.nz, :self.ny, :self.nx] * self.on)
        return torch.stack(out)

    def _pairs(self, dim):
        """(low, high, weight) of the neighbouring pairs along a dim: both active, with A."""
        n = self.on.shape[dim]
        lo, hi = (lambda a, k=0: a.narrow(a.dim() - 3 + dim, 0, n - 1)), (lambda a: a.narrow(a.dim() - 3 + dim, 1, n - 1))
        w = lo(self.on) * hi(self.on)
        w = w * (self.lut[lo(self.region), hi(self.region)] if self.region is not None else self.aex)
        return lo, hi, w

    def exchange(self, m):
        acc = torch.zeros_like(m)
        for dim in range(3):
            if self.on.shape[dim] == 1:
                continue
            lo, hi, w = self._pairs(dim)
            flow = w * (hi(m) - lo(m))
            pad = torch.zeros_like(m.narrow(1 + dim, 0, 1))
            acc = acc + torch.cat((flow, pad), 1 + dim) - torch.cat((pad, flow), 1 + dim)
        return acc * (2.0 / (nf.MU0 * self.ms * self.d * self.d))

    def zeeman(self, t):
        return (self.h_ext + self.h_ac * math.sin(2 * math.pi * self.frequency * t)).reshape(3, 1, 1, 1)

    def fields(self, m, t):
        ex, hd = self.exchange(m), self.demag(m)
        return ex, hd, (ex + hd + self.zeeman(t)) * self.on

    def rhs(self, m, t):
        return self._torque(m, self.fields(m, t)[2])

    def _torque(self, m, h):
        p = torch.linalg.cross(m, h, dim=0)
        q = torch.linalg.cross(m, p, dim=0)
        return -(GAMMA / (1 + self.alpha ** 2)) * (p + self.alpha * q) * self.on

    def unit(self, v):
        n = torch.sqrt((v * v).sum(0))
        return v / torch.where(n > 0, n, torch.ones_like(n))

    def step(self, m, t, dt, integrator):
        k = [self.rhs(m, t)]
        if integrator == "heun":
            k2 = self.rhs(self.unit(m + dt * k[0]), t + dt)
            return self.unit(m + (k[0] + k2) * (0.5 * dt)) * self.on
        rows = {"rk4": ((0.5,), (0, 0.5), (0, 0, 1.0)), "rk23": ((0.5,), (0, 0.75)),
                "dp45": ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
                         (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
                         (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656))}[integrator]
        last = {"rk4": (1 / 6, 1 / 3, 1 / 3, 1 / 6), "rk23": (2 / 9, 1 / 3, 4 / 9),
                "dp45": (35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84)}[integrator]
        at = {"rk4": (0.5, 0.5, 1), "rk23": (0.5, 0.75), "dp45": (0.2, 0.3, 0.8, 8 / 9, 1)}[integrator]
        for row, c in zip(rows, at):
            k.append(self.rhs(self.unit(m + dt * sum(a * x for a, x in zip(row, k) if a)), t + c * dt))
        return self.unit(m + dt * sum(a * x for a, x in zip(last, k) if a))

    def stats(self, m, t):
        vol = self.d ** 3
        ex, hd, he = self.fields(m, t)
        e_ex = 0.0
        for dim in range(3):
            if self.on.shape[dim] > 1:
                lo, hi, w = self._pairs(dim)
                e_ex += float((w * (hi(m) - lo(m)) ** 2).sum()) * vol / self.d ** 2
        moment = nf.MU0 * vol * self.ms * self.on
        e_d = -0.5 * float((moment * m * hd).sum())
        e_z = -float((moment * m * self.zeeman(t)).sum())
        top = lambda v: math.sqrt(float((v * v).sum(0).max()))  # noqa: E731
        return [e_ex, e_d, e_z, e_ex + e_d + e_z], [top(he), top(hd), top(self._torque(m, he))]


def _aos(v):
    return v.reshape(3, -1).T.reshape(-1)


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    soa = lambda m, cells: torch.from_numpy(np.ascontiguousarray(m.reshape(-1, 3).T)).to(device).reshape(3, *cells[::-1])  # noqa: E731
    kind = case["kind"]
    if kind == "batch":
        out = []
        for p in _batch_problems(case, seed):
            model = _Model(p["cells"], p["cell_size"][0], device, ms=p["ms"], aex=p["aex"], alpha=p["alpha"], h_ext=p["h_ext"])
            m = soa(p["m0"], p["cells"])
            for i in range(case["steps"]):
                m = model.step(m, i * case["dt"], case["dt"], "heun")
            out.append(_aos(m).cpu().numpy())
        return np.concatenate(out)
    cells = (case["nx"], case["ny"], case["nz"])
    m = soa(_unit_vectors(seed, math.prod(cells), _numpy_dtype(case)), cells)
    if kind == "demag":
        return (_Model(cells, case["cell"], device).demag(m)).reshape(-1).cpu().numpy()
    mat = _material(case, seed)
    ac = dict(h_ac=(20e-3 / nf.MU0, 0.0, 0.0), frequency=5e9) if kind == "adjoint" else {}
    model = _Model(cells, case["cell"], device, alpha=case["alpha"], h_ext=_h_ext(), mask=mat.get("active_mask"),
                   ms_map=mat.get("ms_map"), region=mat.get("region_mask"), lut=mat.get("exchange_lut"), **ac)
    m = m * model.on
    if kind == "field":
        return _aos(model.fields(m, 0.0)[2]).cpu().numpy()
    if kind == "adjoint":
        leaves = [m.clone(), model.ms, model.h_ext, model.h_ac]
        for v in leaves:
            v.requires_grad_(True)
        m = leaves[0]
        for i in range(case["steps"]):
            m = model.step(m, i * case["dt"], case["dt"], "heun")
        g = torch.autograd.grad((m * soa(_loss_gradient(case, seed), cells)).sum(), leaves)
        return {"m": _aos(m.detach()).cpu().numpy(), "dl_dms": g[1].reshape(-1).cpu().numpy(),
                "dl_dh_ext": g[2].cpu().numpy(), "dl_dh_ac": g[3].cpu().numpy(), "dl_dm0": _aos(g[0]).cpu().numpy()}
    for i in range(case["steps"]):
        m = model.step(m, i * case["dt"], case["dt"], case["integrator"])
    energies, amplitudes = model.stats(m, case["steps"] * case["dt"])
    return {"m": _aos(m).cpu().numpy(), "energies": np.array(energies), "amplitudes": np.array(amplitudes)}
