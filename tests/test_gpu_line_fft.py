"""The line-FFT demag passes, the fused stage combinations and the step graphs.

- Fields at every padded in-plane length the passes have (grids of 2n just below, at and
  just above a length, odd row counts, both spectra sources) against the FP64 oracle, at
  the field tolerances of the other parity tests: 1e-13 (FP64) and 2e-6 (FP32-mixed) of
  each field's own maximum.
- The switches of the z and fused passes on grids padded beyond 2n (the fused y-z pass,
  which has no padding of its own, must leave them to the split kernels): fields as above,
  m after 5 Heun steps at 1e-12 and 1e-6.
- Supplied spectra with more than rounding at a frequency where a Newell tensor is zero:
  the field of numpy's FFT with every entry, at the FP64 field tolerance.
- Which grids are padded where the z pass is the shared-memory FFT, and their fields
  against those at 2n (bit for bit where 2n is kept).
- A Runge-Kutta step on either side of the cell count up to which the FP32 group kernels
  form the next stage state themselves, FP32-mixed against FP64 at 1e-5 (the tolerance
  of the FP32-mixed trajectories).
- Steps replayed as CUDA graphs (counted) against the same launches issued one by one
  (per-kernel timing on), bit for bit, through dt changes; no replay where the rule has none.
- A film's tensor with all six components (random octants) against numpy's FFT at the
  FP64 field tolerance.
- Handles created where the device memory is short (the rest held by torch), against the
  same steps with memory enough, at 1e-12.
- A handle with small blocks created after one with large blocks leaves its launches valid.
"""
import ctypes as C

import numpy as np
import pytest

from fullmag_b200 import native_fdm as nf
from gpu_helpers import make_pair, max_abs

pytestmark = pytest.mark.gpu

D = (2e-9, 2.5e-9, 3e-9)
H = (1e4, -2e4, 3e3)


# (nx, ny, nz): 2n -> 16, 32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072 along x or y
_CELLS = [(5, 7, 1), (9, 15, 3), (20, 36, 1), (48, 36, 2), (49, 64, 1), (70, 96, 2), (100, 7, 3),
          (128, 25, 1), (135, 192, 1), (200, 245, 1), (3, 300, 2), (384, 9, 1), (10, 490, 1), (525, 4, 2),
          (6, 625, 1), (800, 5, 1), (4, 1000, 2), (1050, 5, 1), (3, 1280, 1), (7, 1125, 2), (1536, 2, 2),
          # the z tables' layouts: k_zdw's windows and elements, the fused plane pass's slots, the z FFT
          (20, 150, 9), (18, 36, 10), (70, 128, 3), (32, 100, 4), (49, 25, 12)]


@pytest.mark.parametrize("prec", [nf.PRECISION_DOUBLE, nf.PRECISION_SINGLE])
@pytest.mark.parametrize("cells", _CELLS)
def test_padded_lengths_match_oracle(cells, prec):
    nx, ny, nz = cells
    rng = np.random.default_rng(nx + ny)
    kw = dict(mask=(rng.random(nx * ny * nz) > 0.2).astype(np.uint8)) if ny % 2 else {}
    source = "oracle" if nx % 2 else "newell"
    be, sim, _ = make_pair(cells, D, h_ext=H, precision=prec, symmetric_kernel=True, seed=nx + 3, spectra=source, **kw)
    be.refresh_observables()
    obs = sim.observe()
    tol = 1e-13 if prec == nf.PRECISION_DOUBLE else 2e-6
    for o, key in ((nf.OBS_H_DEMAG, "h_demag"), (nf.OBS_H_EFF, "h_eff")):
        assert max_abs(be.copy_field(o), obs[key]) <= tol * np.abs(obs[key]).max(), key
    be.close()


@pytest.mark.parametrize("env", [("YZ", "fused"), ("ZCONV", "fft"), ("YZY", "off"), ("ROW", "on"), ("FFT", "stockham")])
@pytest.mark.parametrize("cells,prec", [((64, 50, 4), nf.PRECISION_DOUBLE), ((64, 50, 8), nf.PRECISION_SINGLE),
                                        ((50, 32, 2), nf.PRECISION_SINGLE), ((64, 96, 4), nf.PRECISION_SINGLE)])
def test_switched_passes_on_padded_lengths(monkeypatch, env, cells, prec):
    for k in ("YZ", "ZCONV", "YZY", "ROW", "FFT", "YZ_P"):
        monkeypatch.delenv("FULLMAG_FDM_" + k, raising=False)
    monkeypatch.setenv("FULLMAG_FDM_" + env[0], env[1])
    be, sim, _ = make_pair(cells, D, alpha=0.3, h_ext=H, precision=prec, symmetric_kernel=True, seed=11, spectra="newell")
    be.set_profiling(True)
    be.refresh_observables()
    names = set(be.profile())
    be.set_profiling(False)
    assert "demag_yz" not in names  # none of these has both lengths 2n
    obs = sim.observe()
    tol = 1e-13 if prec == nf.PRECISION_DOUBLE else 2e-6
    for o, key in ((nf.OBS_H_DEMAG, "h_demag"), (nf.OBS_H_EFF, "h_eff")):
        assert max_abs(be.copy_field(o), obs[key]) <= tol * np.abs(obs[key]).max(), key
    for _ in range(5):
        be.step(2e-14)
        sim.step(2e-14)
    assert max_abs(be.copy_m(), sim.m) <= (1e-12 if prec == nf.PRECISION_DOUBLE else 1e-6)
    be.close()


@pytest.mark.parametrize("noise", [0.0, 4e-9])
@pytest.mark.parametrize("cells", [(9, 15, 1), (18, 10, 1), (10, 9, 2)])
def test_supplied_spectra_keep_every_entry(cells, noise):
    """What a supplied tensor holds where a Newell tensor is zero counts (noise of single
    precision, within what a plan may carry): xy at the Nyquist frequency along y."""
    nx, ny, nz = cells
    L = (1 if nz == 1 else 2 * nz, 2 * ny, 2 * nx)
    spec = [s.copy() for s in nf.newell_spectra(nx, ny, nz, *D, thin_film_2d=nz == 1)]
    xx, yy, zz, xy, xz, yz = (s.reshape(L + (2,))[..., 0] for s in spec)
    xy[:, ny, :] += noise * max(np.abs(a).max() for a in (xx, yy, zz))
    m = nf.random_unit_vectors(3, nx * ny * nz)
    M = np.fft.fftn(8e5 * m.reshape(nz, ny, nx, 3), L, axes=(0, 1, 2))
    H = -np.stack([(a * M).sum(-1) for a in (np.stack(r, -1) for r in ((xx, xy, xz), (xy, yy, yz), (xz, yz, zz)))], -1)
    want = np.fft.ifftn(H, axes=(0, 1, 2)).real[:nz, :ny, :nx].reshape(-1)
    plan = nf.FdmPlan(cells=cells, cell_size=D, initial_magnetization=m, saturation_magnetisation=8e5,
                      precision=nf.PRECISION_DOUBLE, integrator=nf.HEUN, demag_spectra=spec)
    with nf.NativeFdmBackend(plan) as be:
        assert (be.memory_info()[1][:2] == (2 * nx, 2 * ny)) == (noise > 0.0)
        be.refresh_observables()
        assert max_abs(np.asarray(be.copy_field(nf.OBS_H_DEMAG)).reshape(-1), want) <= 1e-13 * np.abs(want).max()


@pytest.mark.parametrize("prec", [nf.PRECISION_DOUBLE, nf.PRECISION_SINGLE])
@pytest.mark.parametrize("cells,padded", [((70, 70, 32), False), ((70, 70, 24), True), ((135, 135, 8), True), ((63, 63, 40), True)])
def test_padding_only_where_the_z_fft_can_bear_it(monkeypatch, cells, padded, prec):
    """Above 2^17 cells a grid with the shared-memory z FFT and over 1.7 times the columns keeps 2n."""
    kw = dict(cells=cells, cell_size=D, precision=prec, integrator=nf.HEUN, demag_source=nf.DEMAG_NEWELL, damping=0.1,
              initial_magnetization=nf.random_unit_vectors(5, cells[0] * cells[1] * cells[2]))
    fields = []
    for fft in ("line", "stockham"):
        monkeypatch.setenv("FULLMAG_FDM_FFT", fft)
        with nf.NativeFdmBackend(nf.FdmPlan(**kw)) as be:
            assert (be.memory_info()[1][0] > 2 * cells[0]) == (padded and fft == "line")
            fields.append(np.asarray(be.copy_field(nf.OBS_H_DEMAG), dtype=np.float64))
    tol = 1e-13 if prec == nf.PRECISION_DOUBLE else 2e-6
    assert max_abs(*fields) <= (tol * np.abs(fields[1]).max() if padded else 0.0)


def _plan(cells, prec, integrator, seed=5, **kw):
    n = cells[0] * cells[1] * cells[2]
    m0 = nf.random_unit_vectors(seed, n).astype(np.float32).astype(np.float64)
    if integrator in (nf.DP45, nf.RK23):
        kw["adaptive"] = (1e-5, 1e-18, 2e-14, 0.8)
    return nf.FdmPlan(cells=cells, cell_size=D, initial_magnetization=m0, damping=0.1, external_field=H,
                      precision=prec, integrator=integrator, demag_source=nf.DEMAG_NEWELL, **kw)


@pytest.mark.parametrize("integrator", [nf.RK4, nf.RK23, nf.DP45])
@pytest.mark.parametrize("cells,masked", [((512, 512, 1), False), ((540, 512, 1), False), ((64, 48, 3), True), ((25, 18, 2), True)])
def test_fused_combination_fp32_matches_fp64(cells, masked, integrator):
    kw = {}
    if masked:
        kw["active_mask"] = (np.random.default_rng(3).random(cells[0] * cells[1] * cells[2]) > 0.2).astype(np.uint8)
    out = []
    for prec in (nf.PRECISION_SINGLE, nf.PRECISION_DOUBLE):
        with nf.NativeFdmBackend(_plan(cells, prec, integrator, **kw)) as be:
            for _ in range(3):
                be.step(2e-14)
            out.append(be.copy_m())
    assert max_abs(out[0], out[1]) <= 1e-5


@pytest.mark.parametrize("integrator", [nf.HEUN, nf.RK4, nf.RK23, nf.DP45, nf.ABM3])
@pytest.mark.parametrize("cells,prec", [((40, 24, 1), nf.PRECISION_DOUBLE), ((36, 20, 3), nf.PRECISION_SINGLE)])
def test_step_graphs_equal_single_launches(cells, prec, integrator):
    dts = [1e-14] * 5 + [2e-14] * 4 + [1e-14] * 3
    with nf.NativeFdmBackend(_plan(cells, prec, integrator)) as a, nf.NativeFdmBackend(_plan(cells, prec, integrator)) as b:
        b.set_profiling(True)  # times each launch: no graphs
        for i, dt in enumerate(dts):
            sa, sb = a.step(dt), b.step(dt)
            sa.pop("wall_time_ns"), sb.pop("wall_time_ns")
            assert sa == sb, i
        a.step_n(1e-14, 6)
        b.step_n(1e-14, 6)
        for o in (nf.OBS_M, nf.OBS_H_DEMAG, nf.OBS_H_EFF):
            assert np.array_equal(a.copy_field(o), b.copy_field(o)), o
        # 18 steps of two step sizes: of each, one issued as it is, one captured, the rest
        # replays (the accepted states of the adaptive integrators alternate between two
        # sets of buffers); ABM3 has graphs in its Heun start-up only
        assert a.graph_launches() >= (1 if integrator == nf.ABM3 else 6) and b.graph_launches() == 0


@pytest.mark.parametrize("kw", [dict(cells=(540, 512, 1)), dict(cells=(64, 16, 1), ac_field=(1e3, 0.0, 0.0), ac_frequency_hz=1e9)])
def test_no_graphs_for_large_grids_and_time_dependent_fields(kw):
    with nf.NativeFdmBackend(_plan(prec=nf.PRECISION_SINGLE, integrator=nf.HEUN, **kw)) as be:
        for _ in range(6):
            be.step(1e-14)
        assert be.graph_launches() == 0


@pytest.mark.parametrize("cells,integrator", [((525, 270, 4), nf.HEUN), ((525, 270, 4), nf.RK4),
                                              ((512, 512, 8), nf.RK4), ((512, 512, 8), nf.DP45), ((512, 512, 8), nf.RK23)])
def test_handle_that_fits_only_without_padding(monkeypatch, cells, integrator):
    """Where the device lacks the memory of padded lengths and a second stage state, a handle
    is created without them and takes the same steps."""
    import torch

    def run():
        with nf.NativeFdmBackend(_plan(cells, nf.PRECISION_DOUBLE, integrator)) as be:
            for _ in range(2):
                be.step(2e-14)
            return be.copy_m(), *be.memory_info()

    monkeypatch.setenv("FULLMAG_FDM_FFT", "stockham")
    least = run()[1]
    if integrator != nf.HEUN:
        least -= 3 * 8 * cells[0] * cells[1] * cells[2]
    monkeypatch.delenv("FULLMAG_FDM_FFT")
    want, most, _ = run()
    assert least < most
    room, held = (least + most) // 2, []
    torch.cuda.empty_cache()
    while (free := torch.cuda.mem_get_info()[0] - room) > (1 << 21):
        held.append(torch.empty(min(free, 8 << 30) >> 21 << 21, dtype=torch.uint8, device="cuda"))
    try:
        got, nbytes, dims = run()
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert nbytes < room and dims[:2] == (2 * cells[0], 2 * cells[1])
    assert max_abs(got, want) <= 1e-12


def test_small_handle_does_not_limit_a_large_one():
    for prec in (nf.PRECISION_DOUBLE, nf.PRECISION_SINGLE):
        with nf.NativeFdmBackend(_plan((512, 512, 4), prec, nf.HEUN)) as big:
            with nf.NativeFdmBackend(_plan((512, 2, 1), prec, nf.HEUN)) as small, \
                    nf.NativeFdmBackend(_plan((2, 512, 2), prec, nf.HEUN)) as tall:
                for be in (big, small, tall, big):
                    assert np.isfinite(be.step(1e-14)["total_energy_joules"])


@pytest.mark.parametrize("nx,ny", [(16, 16), (64, 32), (8, 128)])
def test_film_octant_with_all_six_components(nx, ny):
    """The allocation-free film call takes any real octant: xz and yz count where they are not zero."""
    import torch
    from test_zz_no_alloc import _entry

    rng = np.random.default_rng(nx)
    oct6, m, ms = rng.standard_normal((6, nx + 1, ny + 1)), rng.standard_normal((3, ny, nx)), 2.0
    k = np.arange(2 * ny)
    ky = np.where(k > ny, 2 * ny - k, k)
    N = oct6[:, :, ky]                                     # [6][kx][ky], xy and yz odd in ky
    N[[3, 5]] *= np.where(k > ny, -1.0, 1.0)
    M = np.fft.fft(np.fft.rfft(ms * m, 2 * nx, axis=2), 2 * ny, axis=1).transpose(0, 2, 1)
    xx, yy, zz, xy, xz, yz = N
    H = -np.stack([xx * M[0] + xy * M[1] + xz * M[2], xy * M[0] + yy * M[1] + yz * M[2], xz * M[0] + yz * M[1] + zz * M[2]])
    want = np.fft.irfft(np.fft.ifft(H, axis=2).transpose(0, 2, 1), 2 * nx, axis=2)[:, :ny, :nx]

    dev = torch.device("cuda", 0)
    o, mm = torch.from_numpy(oct6.copy()).to(dev), torch.from_numpy(np.ascontiguousarray(m)).to(dev)
    h, err = torch.empty(3 * nx * ny, dtype=torch.float64, device=dev), C.create_string_buffer(512)
    rc = _entry()(nx, ny, 1, 1, o.data_ptr(), mm.data_ptr(), ms, h.data_ptr(), torch.cuda.current_stream().cuda_stream, err, len(err))
    assert rc == nf.OK, err.value.decode()
    torch.cuda.synchronize()
    assert np.abs(h.cpu().numpy().reshape(want.shape) - want).max() <= 1e-13 * np.abs(want).max()
