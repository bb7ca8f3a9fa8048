"""The workloads whose speed this repository follows: one dict per workload, the inputs a
program holds before the call, one pass through the public Python entry points, and a
plain torch restatement in 64 bits of what the pass returns.

kinds: "fluid" (Plan.rk4_step), "rbc" (rk4_step_rbc), "mhd" (rk4_step_mhd), "adjoint"
(rk4_evolve and its gradient), "ensemble" (Ensemble.run), "transform" (inverse + forward),
"diagnostics" (shell_spectrum + flux).  Plans keep their default launch rules (no autotuning).
"""
import math

import numpy as np
import torch

import tarang_b200 as tb
from tarang_b200.adjoint import energy_norm_loss, rk4_evolve

PI = math.pi
# SFF / SSF / SSS boxes of the convection runs (x bounded, aspect ratio 1)
KF_RBC = (PI, 2 * PI, 2 * PI)
KF_BOX = (PI, PI, PI)


def _case(name, kind, N, basis="FFF", prec="f32", form="conservative", dealias="reference", steps=1, **more):
    c = {"name": name, "kind": kind, "nx": N[0], "ny": N[1], "nz": N[2], "basis": basis, "prec": prec, "form": form,
         "dealias": dealias, "steps": steps, "forced": False, "members": 0, "window": 0, "radii": 0}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a 32^3 run of the reference's defaults, all launch latency
        _case("fluid_32_f32", "fluid", (32, 32, 32)),
        # the plain FP64 method at its usual size (64^3, two-thirds dealiasing)
        _case("fluid_64_f64", "fluid", (64, 64, 64), prec="f64", dealias="two_thirds"),
        # forced isotropic turbulence, the benchmark's headline
        _case("forced_256_f32", "fluid", (256, 256, 256), form="rotational", dealias="two_thirds", forced=True),
        # decaying turbulence at scale: 1024-point lines, a field far larger than any cache
        _case("decay_1024x512x512_f32", "fluid", (1024, 512, 512), form="rotational", dealias="two_thirds"),
        # transforms on their own (output to and input from real space, three components)
        _case("transform_256_f32", "transform", (256, 256, 256)),
        # one convection run in a wide box
        _case("rbc_sff_128x256x256_f32", "rbc", (128, 256, 256), basis="SFF"),
        # many convection runs of uneven sizes (32^3 .. 128^3) advanced together
        _case("ensemble_32_f32", "ensemble", (0, 0, 0), basis="SFF", members=32, steps=8),
        # sensitivities in FP64: forward steps, and the gradient with recomputed windows
        _case("adjoint_128_f64", "adjoint", (128, 128, 128), prec="f64", form="rotational", dealias="two_thirds",
              steps=4, window=2),
        # convection between walls on three axes, and on two axes with 96-point lines (a factor 3)
        _case("rbc_sss_128_f32", "rbc", (128, 128, 128), basis="SSS"),
        _case("rbc_ssf_96_f32", "rbc", (96, 96, 96), basis="SSF"),
        # magnetohydrodynamics
        _case("mhd_256_f32", "mhd", (256, 256, 256), dealias="two_thirds"),
        # E(k) and the energy flux through 18 spheres, as a run writes them every few steps
        _case("diagnostics_128_f32", "diagnostics", (128, 128, 128), radii=18),
    ]


# the largest listed case bounds a drawn one: grid points of one FP32 rotational step
_MAX_POINTS = 1024 * 512 * 512
# rough cost of one step of a kind, in FP32 FFF fluid steps of the same grid
_COST = {"fluid": 1.0, "rbc": 1.6, "mhd": 2.2, "adjoint": 9.0, "transform": 0.2, "diagnostics": 9.0}


def draw(rng):
    kind = rng.choice(["fluid", "fluid", "fluid", "rbc", "rbc", "rbc", "mhd", "adjoint", "ensemble", "transform", "diagnostics"])
    if kind == "ensemble":
        return _drawn(kind, (0, 0, 0), basis="SFF", prec=rng.choice(["f32", "f32", "f64"]), steps=rng.choice([1, 3, 8]),
                      members=rng.randint(2, 14))
    basis = "FFF"
    if kind == "rbc":
        basis = rng.choice(["SFF", "SFF", "SSF", "SSS"])
    elif kind == "transform":
        basis = rng.choice(["FFF", "FFF", "SFF", "SSF", "SSS"])
    elif kind == "fluid":
        basis = rng.choice(["FFF", "FFF", "FFF", "FFF", "SSF", "SSS"])
    prec = rng.choice(["f32", "f32", "f64"])
    form = rng.choice(["rotational", "conservative"]) if basis == "FFF" and kind == "fluid" else "conservative"
    if kind == "adjoint":
        form = "rotational"
    steps = rng.randint(1, 3) if kind == "adjoint" else 1
    cost = _COST[kind] * (2.5 if prec == "f64" else 1.0) * steps
    low = 6.0 if kind == "diagnostics" else 5.0
    high = {"adjoint": 7.0, "diagnostics": 7.0}.get(kind, 8.3 if basis == "FFF" else 7.7)
    while True:
        # three axis lengths around one size, spread over its logarithm
        size = 2 ** rng.uniform(low, high)
        N = []
        for ax in range(3):
            sizes = [16, 32, 64, 128, 256, 512]
            if basis == "FFF":
                sizes = sizes + [1024]
            elif ax < 2 or (basis != "SSS" and kind != "transform"):
                sizes = sizes + [48, 96]  # not offered along z by SSS plans and by the transforms
            s = size * 2 ** rng.uniform(-1, 1)
            N.append(min(sizes, key=lambda n: abs(math.log(n / s))))
        if basis == "SFF" and kind == "rbc" and rng.random() < 0.1:
            N[1] = 1  # a two-dimensional run in the x-z plane
        points = N[0] * N[1] * N[2]
        if points * cost <= _MAX_POINTS / 4:
            break
    return _drawn(kind, N, basis=basis, prec=prec, form=form, dealias=rng.choice(["reference", "two_thirds"]), steps=steps,
                  forced=kind == "fluid" and basis == "FFF" and rng.random() < 0.3, window=rng.randint(1, 2) if kind == "adjoint" else 0,
                  radii=rng.randint(4, 20) if kind == "diagnostics" else 0)


def _drawn(kind, N, **kw):
    c = _case("", kind, N, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# parameters of a case
# ---------------------------------------------------------------------------
def _N(c):
    return (c["nx"], c["ny"], c["nz"])


def _kf(c):
    if c["basis"] == "FFF":
        return (1.0, 1.0, 1.0)
    return KF_RBC if c["basis"] == "SFF" else KF_BOX


def _physics(c):
    """nu, kappa, dt of a case."""
    if c["kind"] in ("rbc", "ensemble"):
        return math.sqrt(1.0 / 1e6), 1.0 / math.sqrt(1e6), 1e-4
    if c["kind"] == "adjoint":
        return 5e-3, 1e-3, 1e-3
    small = max(_N(c)) <= 64
    return (0.01 if small else 1e-3), (0.01 if small else 1e-3), (1e-3 if small else 2e-4)


def _members(c):
    """(N, Ra, Pr) of the ensemble's runs."""
    return tb.ensemble_members(c["members"])


def _plan_args(c):
    nu, kappa, dt = _physics(c)
    kw = dict(basis=c["basis"], precision=c["prec"], nlin_form=c["form"], dealias=c["dealias"], nu=nu, kappa=kappa, dt=dt,
              kfactor=_kf(c))
    if c["kind"] == "rbc":
        kw.update(Ra=1e6, Pr=1.0)
    return kw


# energy supply 0.1 on the shell 2 < |K| <= 3
_FORCE = (2.0, 3.0, 0.1)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _rdtype(c):
    return torch.float32 if c["prec"] == "f32" else torch.float64


def _axes(N, basis, kf, dev="cuda"):
    """Kx, Ky, Kz broadcastable over a spectral component (real coefficients along z on SSS)."""
    f64 = dict(dtype=torch.float64, device=dev)
    out = []
    for ax in range(3):
        if basis[ax] == "S":
            k = torch.arange(N[ax], **f64)
        elif ax == 2:
            k = torch.arange(N[ax] // 2 + 1, **f64)
        else:
            k = torch.arange(N[ax], **f64)
            k = torch.where(k <= N[ax] // 2, k, k - N[ax])
        shape = [1, 1, 1]
        shape[ax] = -1
        out.append((k * kf[ax]).reshape(shape))
    return out


def _deriv(A, K, letter):
    """Derivative along an axis: Fourier i K, sine series +K, cosine series -K."""
    return A * (1j * K) if letter == "F" else A * (K if letter == "S" else -K)


def _letters(basis, i):
    """Series of velocity component i (the temperature has those of component 0): a sine series along its own walls."""
    return "".join(("S" if ax == i else "C") if b == "S" else "F" for ax, b in enumerate(basis))


def _mul(p, q):
    return "".join("F" if a == "F" else ("C" if a == b else "S") for a, b in zip(p, q))


def _noise(N, basis, gen):
    """A random real field's coefficients along the Fourier axes (Hermitian), its values along the others."""
    a = torch.randn(N, generator=gen, device="cuda", dtype=torch.float32)
    if basis[2] == "F":
        a = torch.fft.rfft(a, dim=2, norm="ortho")
    for ax in (0, 1):
        if basis[ax] == "F":
            a = torch.fft.fft(a, dim=ax, norm="ortho")
    return a


def _random_fields(c, N, seed, ncomp, energy):
    """ncomp spectral components, the first three solenoidal, with the spectrum of developed
    turbulence (rising to k0, k^-5/3, an exponential roll-off), zero on the Nyquist modes."""
    basis = c["basis"]
    K = _axes(N, basis, _kf(c))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 17)
    K2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    k = torch.sqrt(K2)
    kmax = max(2.0, min(_kf(c)[ax] * N[ax] / (1 if basis[ax] == "S" else 2) for ax in range(3) if N[ax] > 1))
    k0 = 4.0 * min(_kf(c))
    env = (k / k0) ** 2 / (1 + (k / k0) ** 2) ** (17.0 / 12.0) * torch.exp(-2.0 * k / kmax) / torch.clamp(k, min=1e-3)
    for ax in range(3):
        if basis[ax] == "F" and N[ax] > 1:
            env.narrow(ax, N[ax] // 2, 1).zero_()
    env = env.to(torch.float32)
    F = []
    for i in range(ncomp):
        a = _noise(N, basis, gen) * env
        for ax in range(3):
            if _letters(basis, i if i < 3 else 0)[ax] == "S":
                a.narrow(ax, 0, 1).zero_()
        F.append(a)
    K32 = [x.to(torch.float32) for x in K]
    inv = torch.where(K2 > 0, 1.0 / torch.clamp(K2, min=1e-30), torch.zeros_like(K2)).to(torch.float32)
    for o in range(0, ncomp - 2, 3):
        div = sum(_deriv(F[o + i], K32[i], _letters(basis, i)[i]) for i in range(3)) * inv
        for i in range(3):
            F[o + i] = F[o + i] + _deriv(div, K32[i], "C" if basis[i] == "S" else "F")
        del div
    w = torch.stack([(a.abs() ** 2).sum(dtype=torch.float64) for a in F]).sum()
    s = torch.sqrt(energy / w).to(torch.float32)
    return [(a * s).to(torch.complex64 if a.is_complex() else torch.float32) for a in F]


def _store(c, F):
    """Components in the library's layout (Nx, Ny, Nz/2+1) complex; real SSS coefficients pairwise, padded."""
    out = []
    for a in F:
        if not a.is_complex():
            p = torch.zeros(a.shape[:2] + (a.shape[2] + 2,), dtype=a.dtype, device=a.device)
            p[..., : a.shape[2]] = a
            a = torch.view_as_complex(p.reshape(p.shape[:2] + (-1, 2)))
        out.append(a)
    return torch.stack(out).to(torch.complex64 if c["prec"] == "f32" else torch.complex128).contiguous()


def _fields(c, seed):
    """The fields of a case before the pass."""
    kind, N = c["kind"], _N(c)
    if kind == "rbc":
        f = _store(c, _random_fields(c, N, seed, 4, 0.02))
        return {"u": f[:3].clone(), "T": f[3:].clone()}
    if kind == "mhd":
        f = _store(c, _random_fields(c, N, seed, 6, 1.0))
        return {"u": f[:3].clone(), "b": f[3:].clone()}
    if kind == "adjoint":
        return {"u": _store(c, _random_fields(c, N, seed, 3, 0.5)), "target": _store(c, _random_fields(c, N, seed + 1000, 3, 0.5))}
    if kind == "ensemble":
        out = {}
        for m, (n, _, _) in enumerate(_members(c)):
            n = (n, n, n) if isinstance(n, int) else n
            f = _store(c, _random_fields(c, n, seed * 64 + m, 4, 0.02))
            out["u%d" % m], out["T%d" % m] = f[:3].clone(), f[3:].clone()
        return out
    return {"u": _store(c, _random_fields(c, N, seed, 3, 0.5))}


def _radii(c):
    """Sphere radii spread geometrically from 2 to two thirds of the smallest axis' Nyquist wavenumber."""
    top = max(3.0, min(_N(c)) / 3.0)
    return np.array([2.0 * (top / 2.0) ** (i / max(1, c["radii"] - 1)) for i in range(c["radii"])])


class _MemberField:
    """One field of an ensemble member where it lies; the tensor made of it keeps the ensemble alive."""

    def __init__(self, ens, m, which):
        self.ens, v = ens, ens.view(m, which)
        self.__cuda_array_interface__ = {"shape": tuple(v.shape), "typestr": "<c8" if v.dtype == torch.complex64 else "<c16",
                                         "data": (v.data_ptr(), False), "version": 3}


def prepare(case, seed):
    c = case
    s = {"case": c}
    f = _fields(c, seed)
    if c["kind"] == "ensemble":
        s["ens"] = tb.Ensemble(_members(c), dt=_physics(c)[2], precision=c["prec"], dealias=c["dealias"])
        s["views"] = []
        for m in range(c["members"]):
            u, T = (torch.as_tensor(_MemberField(s["ens"], m, which), device="cuda") for which in "UT")
            u.copy_(f["u%d" % m])
            T.copy_(f["T%d" % m])
            s["views"] += [u, T]
        torch.cuda.synchronize()
        return s
    kw = _plan_args(c)
    if c["forced"]:
        es = np.zeros(int(_FORCE[1]) + 1)
        es[int(_FORCE[1])] = _FORCE[2]
        kw["forcing"] = tb.Forcing(_FORCE[0], _FORCE[1], es)
    s["plan"] = tb.Plan(_N(c), **kw)
    s.update(f)
    if c["kind"] == "transform":
        Nx, Ny, Nz = _N(c)
        s["real"] = torch.zeros((3, Nx, Ny, Nz + 2), dtype=_rdtype(c), device="cuda")
        s["spec"] = torch.zeros_like(s["u"])
    if c["kind"] == "diagnostics":
        s["radii"] = _radii(c)
    if c["kind"] == "adjoint":
        s["u"].requires_grad_(True)
    return s


def run(state):
    s = state
    c = s["case"]
    kind = c["kind"]
    if kind == "fluid":
        s["plan"].rk4_step(s["u"], c["steps"])
        return s["u"]
    if kind == "rbc":
        s["plan"].rk4_step_rbc(s["u"], s["T"], c["steps"])
        return [s["u"], s["T"]]
    if kind == "mhd":
        s["plan"].rk4_step_mhd(s["u"], s["b"], c["steps"])
        return [s["u"], s["b"]]
    if kind == "ensemble":
        s["ens"].run(c["steps"])
        s["ens"].synchronize()  # the steps run on the ensemble's own stream; a program waits before it reads the states
        return s["views"]
    if kind == "adjoint":
        u = rk4_evolve(s["u"], s["plan"], c["steps"], c["window"])
        J = energy_norm_loss(u, s["target"])
        return [u.detach(), torch.autograd.grad(J, s["u"])[0]]
    if kind == "transform":
        par = _transform_parity(c["basis"])
        s["plan"].inverse(s["u"], s["real"], par)
        s["plan"].forward(s["real"], s["spec"], par)
        return [s["real"], s["spec"]]
    return [s["plan"].shell_spectrum(s["u"]), s["plan"].flux(s["u"], s["radii"])]


def _transform_parity(basis):
    return {"FFF": "FFF", "SFF": "CFF", "SSF": "SCF", "SSS": "SCC"}[basis]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _one(N, basis):
    """(complex elements of a component, real operations of one transform of it)."""
    S = N[0] * N[1] * (N[2] // 2 + 1)
    pts = N[0] * N[1] * N[2]
    return S, 2.5 * pts * math.log2(max(2, pts))


def work(case):
    c = case
    cb = 8 if c["prec"] == "f32" else 16
    kind, N, basis = c["kind"], _N(c), c["basis"]
    if kind == "ensemble":
        b = f = 0.0
        for n, _, _ in _members(c):
            n = (n, n, n) if isinstance(n, int) else n
            S, t = _one(n, basis)
            b += 8 * S * cb
            f += c["steps"] * 4 * (13 * t + 60 * S)
        return {"bytes": b, "flops": f}
    S, t = _one(N, basis)
    if kind == "transform":
        return {"bytes": 2 * 3 * 2 * S * cb, "flops": 2 * 3 * t}
    if kind == "diagnostics":
        return {"bytes": 3 * S * cb, "flops": c["radii"] * (15 * t + 60 * S)}
    if kind == "rbc":
        return {"bytes": 8 * S * cb, "flops": c["steps"] * 4 * (13 * t + 60 * S)}
    if kind == "mhd":
        return {"bytes": 12 * S * cb, "flops": c["steps"] * 4 * (15 * t + 90 * S)}
    if kind == "adjoint":
        return {"bytes": 9 * S * cb, "flops": c["steps"] * 4 * ((9 + 15) * t + 120 * S)}
    return {"bytes": 6 * S * cb, "flops": c["steps"] * 4 * (9 * t + 60 * S)}


def tolerance(case):
    """Relative differences of two correct implementations at the same precision, about four times the error of one of
    them against exact(): a step moves the state by a few per mille, so what is left is the rounding of the stored state
    (2.5e-8 for one step, 9e-8 for eight); transforms 2.6e-7, energy fluxes 4e-7, gradients 1.2e-7; FP64 2e-16 to
    1.1e-15 of the same."""
    f64 = case["prec"] == "f64"
    rel = {"transform": (1e-6, 4e-15), "diagnostics": (2e-6, 2e-14), "adjoint": (6e-7, 6e-15), "ensemble": (4e-7, 2e-15)}
    return {"rel": rel.get(case["kind"], (1.5e-7, 1e-15))[1 if f64 else 0]}


# ---------------------------------------------------------------------------
# the same passes in 64 bits
# ---------------------------------------------------------------------------
class _Ref:
    """Spectral operators of one basis in complex128 (float64 on SSS), sin/cos axes by dense matrices."""

    def __init__(self, c, N):
        self.N, self.basis, self.dealias = N, c["basis"], c["dealias"]
        self.K = _axes(N, self.basis, _kf(c))
        self.K2 = self.K[0] ** 2 + self.K[1] ** 2 + self.K[2] ** 2
        self.iK2 = torch.where(self.K2 > 0, 1.0 / torch.clamp(self.K2, min=1e-300), torch.zeros_like(self.K2))
        self.mat = {}
        for ax in range(3):
            if self.basis[ax] == "S":
                n = torch.arange(N[ax], dtype=torch.float64, device="cuda")
                arg = PI * (2 * n[:, None] + 1) * n[None, :] / (2 * N[ax])
                C, S = 2 * torch.cos(arg), 2 * torch.sin(arg)
                C[:, 0], S[:, 0] = 1.0, 0.0
                Cf, Sf = torch.cos(arg).T / N[ax], torch.sin(arg).T / N[ax]
                self.mat[ax] = {("C", 1): C, ("S", 1): S, ("C", -1): Cf.contiguous(), ("S", -1): Sf.contiguous()}
        self.keep = self._keep()

    def _keep(self):
        """1 where dealiasing keeps a mode."""
        m = []
        for ax in range(3):
            n = self.N[ax]
            l = torch.arange(self.K[ax].numel(), device="cuda")
            if self.dealias == "reference":
                if self.basis[ax] == "S":
                    z = l >= (n // 3 if ax == 2 else 2 * n // 3 + 1)
                else:
                    z = (l >= n // 3 + 1) & (l <= (n // 2 if ax == 2 else 2 * n // 3 - 1))
            else:
                z = 3 * l > 2 * n if self.basis[ax] == "S" else 3 * torch.minimum(l, n - l) > n
            shape = [1, 1, 1]
            shape[ax] = -1
            m.append(z.reshape(shape))
        zero = (m[0] & m[1] & m[2]) if self.dealias == "reference" else (m[0] | m[1] | m[2])
        return (~zero).to(torch.float64)

    def _apply(self, A, ax, M):
        shape, z = A.shape, A.is_complex()
        A = torch.view_as_real(A).flatten(-2) if z else A
        if ax == 0:
            A = (M @ A.reshape(shape[0], -1)).reshape(A.shape)
        elif ax == 1:
            A = M @ A
        else:
            A = A @ M.T
        return torch.view_as_complex(A.reshape(shape + (2,))) if z else A

    def inverse(self, A, par):
        if par == "FFF":
            return torch.fft.irfftn(A, s=self.N, norm="forward")
        for ax in (0, 1):
            A = self._apply(A, ax, self.mat[ax][par[ax], 1]) if par[ax] != "F" else torch.fft.ifft(A, dim=ax, norm="forward")
        return self._apply(A, 2, self.mat[2][par[2], 1]) if par[2] != "F" else torch.fft.irfft(A, n=self.N[2], dim=2, norm="forward")

    def forward(self, u, par):
        if par == "FFF":
            return torch.fft.rfftn(u, norm="forward")
        A = self._apply(u, 2, self.mat[2][par[2], -1]) if par[2] != "F" else torch.fft.rfft(u, dim=2, norm="forward")
        for ax in (1, 0):
            A = self._apply(A, ax, self.mat[ax][par[ax], -1]) if par[ax] != "F" else torch.fft.fft(A, dim=ax, norm="forward")
        return A

    def deriv(self, A, ax, par):
        return _deriv(A, self.K[ax], par[ax])

    def reality(self, A):
        """A(kx, ky, 0) = conj A(-kx, -ky, 0) on the copied half of the kz = 0 plane, and kz = Nz/2 cleared."""
        if self.basis in ("SSF", "SSS"):
            return A
        Nx, Ny, Nz = self.N
        lx = torch.arange(Nx, device="cuda")[:, None]
        ly = torch.arange(Ny, device="cuda")[None, :]
        iy = (-torch.arange(Ny, device="cuda")) % Ny
        p = A[:, :, 0]
        neg = ly > Ny // 2
        if self.basis == "FFF":
            q = p[(-torch.arange(Nx, device="cuda")) % Nx][:, iy].conj()
            sel = ((lx > Nx // 2) & (ly != Ny // 2)) | ((lx == 0) & neg)
        else:
            q = p[:, iy].conj()
            sel = (neg | (ly == 0)).expand(Nx, Ny)
        plane = torch.where(sel, q, p)
        return torch.cat([plane[..., None], A[:, :, 1 : Nz // 2], torch.zeros_like(plane)[..., None]], dim=2)

    def project(self, Nl):
        """-(N - grad (div N) / lap)"""
        L = [_letters(self.basis, i) for i in range(3)]
        p = sum(self.deriv(Nl[i], i, L[i]) for i in range(3)) * self.iK2
        cos = "".join("C" if b == "S" else "F" for b in self.basis)
        return [-(Nl[i] + self.deriv(p, i, cos)) for i in range(3)]

    def products(self, u, v, i, lu, lv):
        """sum_j D_j F[u_j v_i] (v_i of series lv)"""
        out = 0
        for j in range(3):
            par = _mul(lu[j], lv)
            out = out + self.deriv(self.forward(u[j] * v[i], par), j, par)
        return out

    def fluid_nlin(self, U, form):
        L = [_letters(self.basis, i) for i in range(3)]
        u = [self.inverse(U[i], L[i]) for i in range(3)]
        if form == "conservative":
            return u, [self.products(u, u, i, L, L[i]) for i in range(3)]
        D = lambda f, ax: self.deriv(U[f], ax, "FFF")
        w = [self.inverse(x, "FFF") for x in (D(2, 1) - D(1, 2), D(0, 2) - D(2, 0), D(1, 0) - D(0, 1))]
        return u, [self.forward(u[(i + 2) % 3] * w[(i + 1) % 3] - u[(i + 1) % 3] * w[(i + 2) % 3], "FFF") for i in range(3)]

    def carati(self, U):
        """Constant energy supply on the band: alpha U + beta (curl U), then the reality condition."""
        lo, hi, eps = _FORCE
        k = torch.sqrt(self.K2)
        n = int(hi) + 1
        r = torch.arange(-n, n + 1, dtype=torch.float64)
        kk = torch.sqrt(r[:, None, None] ** 2 + r[None, :, None] ** 2 + r[None, None, :] ** 2)
        modes = float((torch.ceil(kk) == int(hi)).sum())
        band = (k > lo) & (k <= hi)
        e = sum(a.real ** 2 + a.imag ** 2 for a in U) / 2
        re, im = [a.real for a in U], [a.imag for a in U]
        h = sum(self.K[i] * (re[(i + 1) % 3] * im[(i + 2) % 3] - re[(i + 2) % 3] * im[(i + 1) % 3]) for i in range(3))
        den = 2 * ((k * e) ** 2 - h ** 2)
        on = band & (e > 1e-15) & (den.abs() > 1e-15)
        den = torch.where(on, den, torch.ones_like(den))
        al = torch.where(on, self.K2 * (eps / modes) * e / den, torch.zeros_like(den))
        be = torch.where(on, -(eps / modes) * h / den, torch.zeros_like(den))
        D = lambda f, ax: self.deriv(U[f], ax, "FFF")
        w = [D(2, 1) - D(1, 2), D(0, 2) - D(2, 0), D(1, 0) - D(0, 1)]
        return [self.reality(al * U[i] + be * w[i]) for i in range(3)]

    def step(self, rhs, F0, diss, dt, fix=True):
        """One integrating-factor RK4 step of the fields F0 with diffusivities diss; the first stage starts from the
        dealiased fields."""
        E = [torch.exp(-d * 0.5 * dt * self.K2) for d in diss]
        n = range(len(F0))
        R = rhs(F0)
        F = [(F0[i] * self.keep + 0.5 * dt * R[i]) * E[i] for i in n]
        tot = [(dt / 6) * R[i] * E[i] ** 2 for i in n]
        R = rhs(F)
        F = [F0[i] * E[i] + 0.5 * dt * R[i] for i in n]
        tot = [tot[i] + (dt / 3) * R[i] * E[i] for i in n]
        R = rhs(F)
        F = [(F0[i] * E[i] + dt * R[i]) * E[i] for i in n]
        tot = [tot[i] + (dt / 3) * R[i] * E[i] for i in n]
        R = rhs(F)
        out = [F0[i] * E[i] ** 2 + tot[i] + (dt / 6) * R[i] for i in n]
        return [self.reality(a) for a in out] if fix else out


def _load(c, f):
    """Library layout -> 64-bit components."""
    out = []
    for a in f:
        a = a.detach().to(torch.complex128)
        if c["basis"] == "SSS":
            a = torch.view_as_real(a).flatten(-2)[..., : 2 * (a.shape[-1] - 1)].contiguous()
        out.append(a)
    return out


def _back(c, F):
    out = []
    for a in F:
        if not a.is_complex():
            p = torch.zeros(a.shape[:2] + (a.shape[2] + 2,), dtype=a.dtype, device=a.device)
            p[..., : a.shape[2]] = a
            a = torch.view_as_complex(p.reshape(p.shape[:2] + (-1, 2)))
        out.append(a)
    return torch.stack(out)


def _rbc_steps(c, N, f, steps, nu, kappa, dt):
    r = _Ref(c, N)
    L = [_letters(c["basis"], i) for i in range(3)]

    def rhs(F):
        d = [a * r.keep for a in F]
        u, Nl = r.fluid_nlin(d[:3], "conservative")
        T = r.inverse(d[3], L[0])
        NT = r.products(u, [T], 0, L, L[0])
        Nl[0] = Nl[0] - F[3]
        return r.project(Nl) + [-(NT - F[0])]

    for _ in range(steps):
        f = r.step(rhs, f, [nu] * 3 + [kappa], dt)
    return f


def exact(case, seed):
    c = case
    kind, N = c["kind"], _N(c)
    nu, kappa, dt = _physics(c)
    f = _fields(c, seed)
    if kind == "ensemble":
        out = []
        for m, (n, Ra, Pr) in enumerate(_members(c)):
            n = (n, n, n) if isinstance(n, int) else n
            F = _rbc_steps(c, n, _load(c, f["u%d" % m]) + _load(c, f["T%d" % m]), c["steps"], math.sqrt(Pr / Ra),
                           1.0 / math.sqrt(Pr * Ra), dt)
            out += [_back(c, F[:3]), _back(c, F[3:])]
        return out
    if kind == "rbc":
        F = _rbc_steps(c, N, _load(c, f["u"]) + _load(c, f["T"]), c["steps"], nu, kappa, dt)
        return [_back(c, F[:3]), _back(c, F[3:])]
    r = _Ref(c, N)
    U = _load(c, f["u"])
    if kind == "transform":
        par = _transform_parity(c["basis"])
        u = [r.inverse(a, par) for a in U]
        pad = torch.zeros((3, N[0], N[1], N[2] + 2), dtype=torch.float64, device="cuda")
        for i in range(3):
            pad[i, :, :, : N[2]] = u[i]
        return [pad, _back(c, [r.forward(a, par) for a in u])]
    if kind == "diagnostics":
        return _exact_diagnostics(c, r, U)
    if kind == "mhd":
        B = _load(c, f["b"])

        def rhs(F):
            d = [r.inverse(a * r.keep, "FFF") for a in F]
            zp, zm = [d[i] + d[3 + i] for i in range(3)], [d[i] - d[3 + i] for i in range(3)]
            Np = [r.products(zm, zp, i, ["FFF"] * 3, "FFF") for i in range(3)]
            Nm = [r.products(zp, zm, i, ["FFF"] * 3, "FFF") for i in range(3)]
            return r.project([(Np[i] + Nm[i]) / 2 for i in range(3)]) + [-(Np[i] - Nm[i]) / 2 for i in range(3)]

        F = U + B
        for _ in range(c["steps"]):
            F = r.step(rhs, F, [nu] * 3 + [kappa] * 3, dt)
        return [_back(c, F[:3]), _back(c, F[3:])]

    def rhs(F):
        Nl = r.fluid_nlin([a * r.keep for a in F], c["form"])[1]
        if c["forced"]:
            Fo = r.carati(F)
            Nl = [Nl[i] - Fo[i] for i in range(3)]
        return r.project(Nl)

    if kind == "adjoint":
        u0 = torch.stack(U).requires_grad_(True)
        F = list(u0)
        for _ in range(c["steps"]):
            F = r.step(rhs, F, [nu] * 3, dt)
        u = torch.stack(F)
        d = u - f["target"].to(torch.complex128)
        w = torch.ones(d.shape[-1], dtype=torch.float64, device="cuda")
        w[0] = 0.5
        J = ((d.real ** 2 + d.imag ** 2) * w).sum()
        return [u.detach(), torch.autograd.grad(J, u0)[0]]
    for _ in range(c["steps"]):
        U = r.step(rhs, U, [nu] * 3, dt)
    return _back(c, U)


def _exact_diagnostics(c, r, U):
    Nx, Ny, Nz = _N(c)
    k = torch.sqrt(r.K2)
    mult = torch.ones_like(k)
    mult[:, :, 0] = 0.5
    mult[Nx // 2, :, :] *= 2
    mult[:, Ny // 2, :] *= 2
    mult[Nx // 2, Ny // 2, :] /= 2
    n = int(math.ceil(math.sqrt((Nx // 2) ** 2 + (Ny // 2) ** 2 + (Nz // 2) ** 2))) + 1
    idx = torch.ceil(k).long().flatten()
    zero = torch.zeros(n, dtype=torch.float64, device="cuda")
    cnt = zero.index_add(0, idx, 2 * mult.flatten())
    e = (sum(a.real ** 2 + a.imag ** 2 for a in U) * mult * r.K2).flatten()
    S = zero.index_add(0, idx, e)
    Ek = torch.where(cnt > 0, S * 4 * PI / torch.clamp(cnt, min=1e-30), zero)
    D = [a * r.keep for a in U]
    u = [r.inverse(a, "FFF") for a in D]
    Pi = []
    for R in _radii(c):
        g = [r.inverse(a * (k <= R), "FFF") for a in D]
        Nl = [r.products(u, g, i, ["FFF"] * 3, "FFF") for i in range(3)]
        t = sum((Nl[i] * D[i].conj()).real for i in range(3)) * 2 * mult * (k > R)
        Pi.append(-float(t.sum()))
    return [Ek.cpu().numpy(), np.array(Pi)]
