"""Parallel flows: one velocity component, along an axis on which it does not depend, with a mean wind.
The nonlinear term of such a flow is zero (u_i u_j vanishes or is constant along the axis it is
differentiated on), so the other components, a passive scalar, a temperature or a magnetic field
that start at zero stay at zero, and the flow decays by exp(-nu K^2 t): two roundings of the stored
state a step.

Along z they stay exactly zero.  Along x the projection has to cancel the gradient of the u1u1 that a
step takes off the product tensor, and along y the neighbouring z lines that ride in one complex
transform differ by its rounding; what is left is a derivative of the rounding of u_i u_i, whose
norm is at most max |u| times that of u, and which a transform of n points loses eps log2(n) of
(four times that, as for the transforms)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"f32": 2.0 ** -23, "f64": 2.0 ** -52}
STEPS, NU = 2, 0.01
LONG = 800


def flow(basis, N, axis, rng):
    """coefficients of the component along `axis`: random values of a mean wind of 10 plus a unit
    field, zero where the wavenumber along the axis is not"""
    Nx, Ny, Nz = N
    shape = [Nx, Ny, Nz]
    shape[axis] = 1
    w = 10 + rng.standard_normal(shape)
    if basis == "FFF":
        A = np.fft.rfftn(np.broadcast_to(w, N), norm="forward")
    else:
        # sin/cos axes: a cosine series' coefficients are as good as its values
        A = w / math.sqrt(w.size)
        for ax in range(3):
            if basis[ax] == "F":
                n = N[ax] if ax != 2 else Nz // 2 + 1
                A = np.fft.fft(A, axis=ax, norm="forward") if ax != 2 else A
                if ax == axis:
                    pad = [(0, 0)] * 3
                    pad[ax] = (0, n - 1)
                    A = np.pad(A, pad)
                elif ax == 2:
                    A = np.fft.rfft(A, axis=2, norm="forward") if not np.iscomplexobj(A) else A[:, :, :n]
    A = np.array(np.broadcast_to(A, (Nx, Ny, Nz // 2 + 1)), dtype=np.complex128)
    idx = [slice(None)] * 3
    idx[axis] = slice(1, None)
    A[tuple(idx)] = 0
    A[:, :, Nz // 2] = 0
    return A


def decay(basis, N, kf, time):
    ks = [np.arange(N[ax]) if basis[ax] == "S" else np.fft.fftfreq(N[ax], 1 / N[ax]) for ax in range(3)]
    ks[2] = np.arange(N[2] // 2 + 1)
    K = np.meshgrid(*[k * f for k, f in zip(ks, kf)], indexing="ij")
    return np.exp(-NU * time * sum(k ** 2 for k in K))


CASES = [("FFF", kind, axis, N) for kind in ("fluid", "scalar", "mhd") for axis in range(3)
         for N in ((32, 16, 32), (128, 16, 16), (512, 16, 16))]
CASES += [("FFF", "fluid", axis, N) for axis in range(3) for N in ((256, 32, 16), (16, 32, 1024), (64, 128, 64))]
CASES += [("SFF", "rbc", axis, N) for axis in (1, 2) for N in ((32, 16, 16), (96, 16, 48))]
CASES += [("SSF", kind, 2, N) for kind in ("fluid", "rbc") for N in ((32, 16, 16), (96, 48, 16))]


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("basis,kind,axis,N", CASES)
def test_parallel_flows_only_decay(cuda, basis, kind, axis, N, prec):
    import torch
    import tarang_b200 as tb
    kf = {"FFF": (1.0,) * 3, "SFF": (math.pi, 2 * math.pi, 2 * math.pi), "SSF": (math.pi,) * 3}[basis]
    kmax = max(f * n / (1 if b == "S" else 2) for f, n, b in zip(kf, N, basis))
    dt = 0.5 / (20 * kmax)  # the wind stays below 20: noise is carried, not amplified
    plan = tb.Plan(N, basis=basis, precision=prec, kfactor=kf, dealias="reference", nu=NU, kappa=NU, dt=dt, Ra=1e4, Pr=1.0)
    u, other = plan.field(3), plan.field(3 if kind == "mhd" else 1)
    u[axis] = torch.from_numpy(flow(basis, N, axis, np.random.default_rng(2))).to(plan.torch_dtype())
    start = u[axis].cpu().numpy().astype(np.complex128)
    if kind == "fluid":
        plan.rk4_step(u, STEPS)
    else:
        {"scalar": plan.rk4_step_scalar, "rbc": plan.rk4_step_rbc, "mhd": plan.rk4_step_mhd}[kind](u, other, STEPS)
    plan.status()
    zero = [u[i] for i in range(3) if i != axis] + [other]
    noise = max(torch.linalg.vector_norm(f).item() for f in zero)
    if axis == 2:
        assert noise == 0
    else:
        assert noise < 4 * EPS[prec] * math.log2(np.prod(N)) * STEPS * dt * kmax * 20 * np.linalg.norm(start)
    want = start * decay(basis, N, kf, STEPS * dt)
    err = np.linalg.norm(u[axis].cpu().numpy() - want) / np.linalg.norm(want)
    assert err < 2 * STEPS * EPS[prec]


@pytest.mark.parametrize("basis,kind,N", [("FFF", k, N) for k in ("fluid", "scalar", "mhd")
                                          for N in ((32, 16, 32), (128, 16, 16), (256, 16, 16), (512, 16, 16))]
                         + [("SFF", "rbc", (32, 16, 16)), ("SSF", "fluid", (32, 16, 16)), ("SSF", "rbc", (96, 48, 16))])
def test_integrating_factors_have_no_bias(cuda, basis, kind, N):
    """A flow along z in FP32 over LONG steps: every step is one rounding of u0 exp(-nu K^2 dt), so the
    state stays within a rounding of the same product rounded in numpy.  A factor rounded to FP32
    leaves it by 1e-5."""
    import torch
    import tarang_b200 as tb
    kf = {"FFF": (1.0,) * 3, "SFF": (math.pi, 2 * math.pi, 2 * math.pi), "SSF": (math.pi,) * 3}[basis]
    K2max = sum((f * n / (1 if b == "S" else 2)) ** 2 for f, n, b in zip(kf, N, basis))
    dt = 1.0 / (LONG * NU * K2max)  # the smallest scales lose a factor e
    plan = tb.Plan(N, basis=basis, precision="f32", kfactor=kf, dealias="reference", nu=NU, kappa=NU, dt=dt, Ra=1e4, Pr=1.0)
    u, other = plan.field(3), plan.field(3 if kind == "mhd" else 1)
    u[2] = torch.from_numpy(flow(basis, N, 2, np.random.default_rng(2))).to(plan.torch_dtype())
    u[2, 0, 0, 0] = 0
    want = u[2].cpu().numpy()
    for _ in range(LONG):
        want = (want.astype(np.complex128) * decay(basis, N, kf, dt)).astype(np.complex64)
    if kind == "fluid":
        plan.rk4_step(u, LONG)
    else:
        {"scalar": plan.rk4_step_scalar, "rbc": plan.rk4_step_rbc, "mhd": plan.rk4_step_mhd}[kind](u, other, LONG)
    plan.status()
    err = np.linalg.norm(u[2].cpu().numpy() - want) / np.linalg.norm(want)
    assert err < 2.0 ** -24
