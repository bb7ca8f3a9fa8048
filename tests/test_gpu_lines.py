"""Transforms and steps at the edges of the line kernels' ranges: the shortest and longest
lines of every axis, lengths with a factor 3, planes whose columns end inside a column tile.

The transforms are compared with numpy / scipy in FP64; an FFT of n points of unit-variance
data loses about eps * log2(n) in relative L2 norm, so the bounds are 4 eps log2(points).
The steps are compared with the FP64 oracle from states with energy in every mode, so that a
lost or wrongly dealiased row shows.  The time step is such that a step moves the state by at
most CHANGE = 5 %: its error is the rounding of the stored state (half an ulp in FP32, where one
fma chain ends it; three roundings in FP64) plus CHANGE times that of the transforms (step_tol)."""
import gc
import math

import numpy as np
import pytest

from capture import captured
from oracle import tarang_ref as R

pytestmark = pytest.mark.gpu

EPS = {"f32": 2.0 ** -23, "f64": 2.0 ** -52}
CHANGE = 0.05


def step_tol(prec, N):
    return EPS[prec] * ({"f32": 0.5, "f64": 1.5}[prec] + CHANGE * math.log2(np.prod(N)))


def lively(g, seed):
    """A solenoidal field: the benchmark's spectrum plus noise of the same energy in every mode."""
    rng = np.random.default_rng(seed)
    F = np.stack([R.reality_fix(g, R.forward(g, 0.3 * rng.standard_normal(g.rshape))) for _ in range(3)])
    return R.init_energy_spectrum(g, R.spectrum_k4_gauss(g.n_shells(), 4.0), seed, 0.5) - R.project_rhs(g, F)


def small_dt(N):
    """CHANGE / (largest wavenumber times largest speed, 5)"""
    return CHANGE / (5 * max(N) / 2)


def rel(a, b):
    return float(np.linalg.norm((np.asarray(a) - b).ravel()) / np.linalg.norm(np.asarray(b).ravel()))


TRANSFORMS = [("FFF", "FFF", N) for N in ((16, 16, 16), (1024, 16, 16), (16, 1024, 32), (32, 16, 1024), (512, 32, 16),
                                          (16, 512, 64), (32, 16, 512))]
TRANSFORMS += [("SFF", p, N) for p in ("SFF", "CFF") for N in ((16, 48, 16), (96, 16, 32), (512, 16, 16), (48, 96, 64))]
TRANSFORMS += [("SSF", p, N) for p in ("SCF", "CSF") for N in ((16, 512, 16), (48, 96, 32), (256, 16, 128))]
TRANSFORMS += [("SSS", p, N) for p in ("SCC", "CSS") for N in ((16, 16, 16), (96, 48, 1024), (512, 16, 32))]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("basis,parity,N", TRANSFORMS)
def test_transforms_at_line_edges(cuda, basis, parity, N, prec):
    import torch
    import tarang_b200 as tb
    g = R.Grid(N, (1.0, 1.0, 1.0), basis)
    plan = tb.Plan(N, basis=basis, precision=prec)
    rt = torch.float32 if prec == "f32" else torch.float64
    rng = np.random.default_rng(7)
    u = rng.standard_normal((2,) + N)
    par = {"FFF": "F", "SFF": parity[0]}.get(basis, parity)
    want = np.stack([R.forward(g, u[i], par) for i in range(2)])
    real = torch.zeros((2,) + N[:2] + (N[2] + 2,), dtype=rt, device=cuda)
    real[..., : N[2]] = torch.from_numpy(u).to(rt)
    real[..., N[2]:] = float("nan")  # the padding is not read
    spec = torch.empty((2,) + plan.spec_shape, dtype=plan.torch_dtype(), device=cuda)
    plan.forward(real, spec, parity)
    got = spec.cpu().numpy()
    if basis == "SSS":
        got = got.view(got.real.dtype)
        assert np.all(got[..., N[2]:] == 0)
        got = got[..., : N[2]]
    tol = 4 * EPS[prec] * math.log2(np.prod(N))
    assert rel(got, want) < tol
    back = torch.full_like(real, float("nan"))
    plan.inverse(spec, back, parity)
    out = back.cpu().numpy()
    assert np.all(out[..., N[2]:] == 0)
    u0 = np.stack([R.inverse(g, want[i], par) for i in range(2)])
    assert rel(out[..., : N[2]], u0) < 2 * tol


STEPS = [("rotational", "two_thirds", N) for N in ((16, 16, 16), (1024, 16, 32), (16, 1024, 16), (16, 32, 1024),
                                                   (512, 16, 16), (32, 16, 512), (128, 32, 16), (256, 16, 32))]
STEPS += [("conservative", "reference", N) for N in ((16, 16, 16), (1024, 16, 16), (16, 512, 32), (16, 16, 1024), (64, 32, 256),
                                                     (128, 16, 16), (256, 16, 16))]
# 32 and 64 points along x: the pipelined forward x pass on small fields, the split one above (FP64
# 64 x 128 x 64: 4.3 MB a component)
STEPS += [(f, d, N) for f, d in (("rotational", "two_thirds"), ("conservative", "reference"))
          for N in ((32, 16, 16), (32, 64, 32), (64, 16, 16), (64, 128, 64))]


# more column tiles than blocks of the persistent pipelined kernel (148, or 296 at 32 and 64 points; no
# field of its size has more at 64): a block's buffers are used again
STEPS += [("conservative", "reference", (32, 128, 128)), ("rotational", "two_thirds", (128, 64, 256)),
          ("conservative", "two_thirds", (128, 64, 128)), ("rotational", "reference", (256, 64, 128)),
          ("conservative", "reference", (256, 64, 128))]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("form,dealias,N", STEPS)
def test_forced_step_at_line_edges(cuda, form, dealias, N, prec):
    import torch
    import tarang_b200 as tb
    g = R.Grid(N)
    es = np.zeros(g.n_shells())
    es[3] = 0.1
    V, dt = lively(g, 0), small_dt(N)
    mode = {"reference": 1, "two_thirds": 2}[dealias]
    plan = tb.Plan(N, precision=prec, nlin_form=form, dealias=dealias, nu=0.01, dt=dt, forcing=tb.Forcing(2.0, 3.0, es))
    u = torch.from_numpy(V).to(plan.torch_dtype()).to(cuda)
    V = u.cpu().numpy().astype(np.complex128)
    want = R.rk4_step(R.FluidConfig(g, 0.01, dt, mode, form, True, R.CaratiForcing(2.0, 3.0, es)), V)
    plan.rk4_step(u, 1)
    assert rel(u.cpu().numpy(), want) < step_tol(prec, N)


MORE = [(N, d) for N in ((16, 16, 16), (1024, 16, 16), (16, 1024, 16), (16, 32, 1024), (512, 16, 32), (16, 512, 64), (32, 16, 512),
                         (128, 64, 64), (256, 16, 128)) for d in ("reference", "two_thirds")]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("kind", ["scalar", "mhd"])
@pytest.mark.parametrize("N,dealias", MORE)
def test_scalar_and_mhd_step_at_line_edges(cuda, N, dealias, kind, prec):
    import torch
    import tarang_b200 as tb
    g = R.Grid(N)
    dt, mode = small_dt(N), {"reference": 1, "two_thirds": 2}[dealias]
    U, B = lively(g, 0), lively(g, 1)
    if kind == "scalar":
        B = B[:1]
    plan = tb.Plan(N, precision=prec, dealias=dealias, nu=0.01, kappa=0.02, dt=dt)
    u, b = (torch.from_numpy(a).to(plan.torch_dtype()).to(cuda) for a in (U, B))
    U, B = (x.cpu().numpy().astype(np.complex128) for x in (u, b))
    if kind == "scalar":
        wu, wb = R.rbc_rk4_step(R.ScalarConfig(g, nu=0.01, kappa=0.02, dt=dt, dealias_mode=mode), U, B[0])
        plan.rk4_step_scalar(u, b, 1)
        wb = wb[None]
    else:
        wu, wb = R.mhd_rk4_step(R.MHDConfig(g, nu=0.01, eta=0.02, dt=dt, dealias_mode=mode), U, B)
        plan.rk4_step_mhd(u, b, 1)
    assert rel(u.cpu().numpy(), wu) < step_tol(prec, N)
    assert rel(b.cpu().numpy(), wb) < step_tol(prec, N)


@pytest.mark.parametrize("N", [(128, 64, 64), (128, 16, 256), (256, 16, 32), (64, 32, 128)])
def test_adjoint_step_at_line_edges(cuda, N):
    """FP64, the bound of the oracle comparisons of the adjoint; 128 x 64 x 64 has more column tiles
    than the pipelined kernel has blocks."""
    import torch
    import tarang_b200 as tb
    g, dt = R.Grid(N), small_dt(N)
    V = lively(g, 0)
    rng = np.random.default_rng(5)
    Lam = rng.standard_normal((3,) + g.shape) + 1j * rng.standard_normal((3,) + g.shape)
    plan = tb.Plan(N, precision="f64", nlin_form="rotational", dealias="two_thirds", nu=0.01, dt=dt)
    u = torch.from_numpy(V).to(cuda)
    lam = torch.from_numpy(Lam.copy()).to(cuda)
    work = torch.empty(plan.adjoint_work_bytes(1), dtype=torch.uint8, device=cuda)
    plan.adjoint_window(u, 1, lam, work)
    cfg = R.FluidConfig(g, nu=0.01, dt=dt, dealias_mode=2, nlin_form="rotational", reality_fix=True)
    assert rel(lam.cpu().numpy(), R.rk4_step_adjoint(cfg, V, Lam)) < 1e-11


RBC = [("SFF", (16, 16, 48)), ("SFF", (96, 48, 16)), ("SFF", (16, 1, 96)), ("SFF", (512, 16, 16)), ("SSF", (48, 96, 16)),
       ("SSF", (16, 16, 96)), ("SSF", (512, 16, 16)), ("SSS", (16, 96, 16)), ("SSS", (96, 16, 512)), ("SSS", (16, 16, 1024))]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dealias", ["reference", "two_thirds"])
@pytest.mark.parametrize("basis,N", RBC)
def test_convection_step_at_line_edges(cuda, basis, N, dealias, prec):
    import torch
    import tarang_b200 as tb
    kf = (math.pi, 2 * math.pi, 2 * math.pi) if basis == "SFF" else (math.pi,) * 3
    g = R.Grid(N, kf, basis)
    rng = np.random.default_rng(3)
    par = {"SFF": ("S", "C", "C", "S"), "SSF": ("SCF", "CSF", "CCF", "SCF"), "SSS": ("SCC", "CSC", "CCS", "SCC")}[basis]
    # random fields with energy in every mode but the Nyquist planes, U solenoidal
    F = np.stack([R.reality_fix(g, R.forward(g, 0.3 * rng.standard_normal(N), p)) for p in par])
    if basis == "SFF" and N[1] > 1:
        F[:, :, N[1] // 2] = 0
    if basis != "SSS":
        F[..., N[2] // 2] = 0
    U, T = -R.project_rhs(g, F[:3]), F[3]
    kmax = max(f * n / (1 if b == "S" else 2) for f, n, b in zip(kf, N, basis))
    dt = CHANGE / (2 * kmax)  # speeds stay below 2
    cfg = R.RBCConfig(grid=g, Ra=1e4, Pr=1.0, dt=dt, dealias_mode={"reference": 1, "two_thirds": 2}[dealias])
    plan = tb.Plan(N, basis=basis, precision=prec, kfactor=kf, dealias=dealias, nu=cfg.nu, kappa=cfg.kappa, Ra=1e4,
                   Pr=1.0, dt=dt)

    def pack(a):
        if basis == "SSS":
            p = np.zeros(a.shape[:-1] + (a.shape[-1] + 2,))
            p[..., : a.shape[-1]] = a
            a = p.view(np.complex128)
        return torch.from_numpy(np.ascontiguousarray(a)).to(plan.torch_dtype()).to(cuda)

    def unpack(x):
        x = x.cpu().numpy().astype(np.complex128)
        return x.view(np.float64)[..., : N[2]] if basis == "SSS" else x

    u, t = pack(U), pack(T[None])
    wu, wt = R.rbc_rk4_step(cfg, unpack(u), unpack(t)[0])
    plan.rk4_step_rbc(u, t, 1)
    assert rel(unpack(u), wu) < step_tol(prec, N)
    assert rel(unpack(t)[0], wt) < step_tol(prec, N)


def in_place():
    """A tuning whose y passes take a blocks-per-SM count: the inverse-transformed fields then keep
    their lines of Nz / 2 + 1 and the products go over them."""
    return {"variant": [0] * 5, "blocks_per_sm": [0, 1, 0, 1, 0]}


COMPACT = [((16, 16, 128), "rotational"), ((32, 16, 128), "conservative"), ((128, 16, 256), "conservative"),
           ((256, 32, 128), "rotational"), ((16, 64, 512), "rotational"), ((512, 16, 256), "conservative"),
           ((32, 16, 512), "mhd"), ((256, 16, 128), "mhd"), ((128, 32, 128), "adjoint"), ((64, 32, 64), "rotational")]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("N,kind", COMPACT)
def test_compact_inverse_lines_match_in_place(cuda, N, kind, prec):
    """Two-thirds dealiased right-hand sides on compact inverse-transformed lines (FP32, 128 points
    along z and more) against the same steps in place.  The arithmetic of a mode is the same but
    for the order of the y butterflies' rounding, so the two agree to a few roundings of the state.
    The layout shows in the y inverse's grid: tiles of 16 columns over whole compact lines."""
    import torch
    import tarang_b200 as tb
    g = R.Grid(N)
    V = R.init_energy_spectrum(g, R.spectrum_k4_gauss(g.n_shells(), 4.0), 0, 0.5)
    B = R.init_energy_spectrum(g, R.spectrum_k4_gauss(g.n_shells(), 3.0), 1, 0.3)
    form = {"adjoint": "rotational", "mhd": "conservative"}.get(kind, kind)
    got = []
    for tuning in (None, in_place()):
        plan = tb.Plan(N, precision=prec, nlin_form=form, dealias="two_thirds", nu=0.01, kappa=0.02, dt=1e-2)
        if tuning:
            plan.set_tuning(tuning)
        u, b = (torch.from_numpy(a).to(plan.torch_dtype()).to(cuda) for a in (V, B))
        if kind == "mhd":
            call = lambda: plan.rk4_step_mhd(u, b, 2)
        elif kind == "adjoint":
            work = torch.empty(plan.adjoint_work_bytes(2), dtype=torch.uint8, device=cuda)
            call = lambda: plan.adjoint_window(u, 2, b, work)
        else:
            call = lambda: plan.rk4_step(u, 2)
        call()
        plan.status()
        got.append((u.cpu().numpy(), b.cpu().numpy()))
        pitch = (N[2] // 3 + 1 + 15) // 16 * 16
        tiles = (3 if kind == "conservative" else 6) * N[0] * pitch // 16
        assert (tiles in captured(plan, call)[0]) == (prec == "f32" and N[2] >= 128 and not tuning)
    tol = 16 * math.log2(np.prod(N)) * EPS[prec]
    for x, y in zip(*got):
        assert rel(x, y) < tol


@pytest.mark.parametrize("kind,spare", [("fluid", 140 << 20), ("mhd", 200 << 20)])
def test_compact_lines_leave_a_full_device_its_memory(cuda, kind, spare):
    """With little memory free a plan keeps the work fields of the in-place step and takes that step;
    results as with the compact lines."""
    import torch
    import tarang_b200 as tb
    N = (128, 64, 128)  # 4.3 MB a component
    V, dt = lively(R.Grid(N), 0), small_dt(N)
    got, took = [], []
    for full in (False, True):
        gc.collect()
        torch.cuda.empty_cache()
        hog = torch.empty(max(0, torch.cuda.mem_get_info()[0] - spare) if full else 0, dtype=torch.uint8, device=cuda)
        before = torch.cuda.mem_get_info()[0]
        u = torch.from_numpy(V).to(torch.complex64).to(cuda)
        b = u.flip(0).contiguous()
        plan = tb.Plan(N, precision="f32", nlin_form="conservative", dealias="two_thirds", nu=0.01, kappa=0.02, dt=dt)
        call = (lambda: plan.rk4_step_mhd(u, b, 1)) if kind == "mhd" else (lambda: plan.rk4_step(u, 1))
        call()
        plan.status()
        got.append((u.cpu().numpy(), b.cpu().numpy()))
        took.append(before - torch.cuda.mem_get_info()[0])
        tiles = (6 if kind == "mhd" else 3) * N[0] * 48 // 16
        compact = tiles in captured(plan, call)[0]
        del hog, plan, call, u, b
        torch.cuda.empty_cache()  # the library allocates beside torch's cache
        assert compact == (not full)
    assert took[1] < took[0]
    for x, y in zip(*got):
        assert rel(x, y) < 16 * math.log2(np.prod(N)) * EPS["f32"]


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_a_step_that_finds_no_memory_leaves_the_plan_usable(cuda, prec):
    """MHD needs larger stage, accumulator and work fields than the plan has; on a full device it
    says so, and the plan's fluid step, transform and flux run as before."""
    import torch
    import tarang_b200 as tb
    N = (64, 64, 64)
    V, dt = lively(R.Grid(N), 0), small_dt(N)
    plan = tb.Plan(N, precision=prec, dealias="two_thirds", nu=0.01, kappa=0.02, dt=dt)
    u = torch.from_numpy(V).to(plan.torch_dtype()).to(cuda)
    w = u.clone()
    plan.rk4_step(w, 1)
    want, flux = w.clone(), plan.flux(u, [2.0, 5.0])
    x, b = u.clone(), u.clone()
    gc.collect()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (4 << 20), dtype=torch.uint8, device=cuda)
    try:
        for _ in range(2):
            with pytest.raises(tb.TsError) as e:
                plan.rk4_step_mhd(x, b, 1)
            assert e.value.status == 6  # TS_ERR_NOMEM
        w.copy_(u)
        plan.rk4_step(w, 1)
        plan.status()
        again = plan.flux(u, [2.0, 5.0])
    finally:
        del hog
        torch.cuda.empty_cache()
    assert torch.equal(w, want) and np.array_equal(again, flux)
    plan.rk4_step_mhd(x, b, 1)
    plan.status()


@pytest.mark.parametrize("prec,tol", [("f64", 1e-12), ("f32", 2e-6)])
@pytest.mark.parametrize("N", [(16, 16, 16), (1024, 16, 16), (512, 16, 32), (64, 32, 16), (256, 16, 16), (128, 16, 64)])
def test_flux_at_line_edges(cuda, N, prec, tol):
    """The per-sphere flux at the edges of its x lines, and the same bits twice."""
    import torch
    import tarang_b200 as tb
    g = R.Grid(N)
    V = R.init_energy_spectrum(g, R.spectrum_k4_gauss(g.n_shells(), 6.0), 3, 0.5)
    radii = [0.0, 2.0, 5.0, 5.0, 1e9]
    ref = R.flux_per_sphere(g, V, radii, 1)
    plan = tb.Plan(N, precision=prec, dealias="reference")
    u = torch.from_numpy(V).to(plan.torch_dtype()).to(cuda)
    Pi = plan.flux(u, radii)
    assert np.max(np.abs(Pi - ref)) < tol * np.max(np.abs(ref))
    assert np.array_equal(Pi, plan.flux(u, radii))


@pytest.mark.parametrize("prec,tol", [("f64", 1e-12), ("f32", 2e-6)])
@pytest.mark.parametrize("dealias", ["none", "reference", "two_thirds"])
def test_flux_takes_every_radius(cuda, dealias, prec, tol):
    """Radii that do not ascend (the per-sphere form on every dealias mode), among them the sphere
    that holds no mode, the one that holds all and one whose square overflows."""
    import torch
    import tarang_b200 as tb
    N = (32, 16, 16)
    g = R.Grid(N)
    V = R.init_energy_spectrum(g, R.spectrum_k4_gauss(g.n_shells(), 6.0), 3, 0.5)
    radii = [3.0, math.inf, -1.0, 1e200, 0.0, -math.inf]
    ref = R.flux_per_sphere(g, V, radii, {"none": 0, "reference": 1, "two_thirds": 2}[dealias])
    plan = tb.Plan(N, precision=prec, dealias=dealias)
    Pi = plan.flux(torch.from_numpy(V).to(plan.torch_dtype()).to(cuda), radii)
    assert np.max(np.abs(Pi - ref)) < tol * np.max(np.abs(ref))
    assert np.all(Pi[[1, 2, 3, 5]] == 0)


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("basis,parity", [("FFF", "FFF"), ("SFF", "CFF"), ("SSF", "SCF"), ("SSS", "SCC")])
def test_inverse_takes_inputs_aligned_to_a_real(cuda, basis, parity, prec):
    """A spectrum that starts between two complex values (a C program's pointer into its own
    buffer): the same bits as from an aligned one, and the input untouched."""
    import ctypes
    import torch
    import tarang_b200 as tb
    N = (32, 16, 64)
    plan = tb.Plan(N, basis=basis, precision=prec)
    rt = torch.float32 if prec == "f32" else torch.float64
    spec = torch.randn((2,) + plan.spec_shape, dtype=plan.torch_dtype(), device=cuda)
    want = torch.zeros((2,) + N[:2] + (N[2] + 2,), dtype=rt, device=cuda)
    plan.inverse(spec, want, parity)
    flat = torch.view_as_real(spec).reshape(-1)
    buf = torch.zeros(flat.numel() + 1, dtype=rt, device=cuda)
    buf[1:] = flat
    got = torch.zeros_like(want)
    rc = plan.lib.ts_fft_inverse(plan.h, parity.encode(), ctypes.c_void_p(buf[1:].data_ptr()),
                                 ctypes.c_void_p(got.data_ptr()), 2)
    torch.cuda.synchronize()
    assert rc == 0 and torch.equal(got, want) and torch.equal(buf[1:], flat)
