"""The work a program has this framework do, as cases that can be timed and checked.

Six kinds of pass, each through the public entry points:

* ``dns``     coupled time steps: ``Flow.step(droplets)`` then ``Partlib.particle_step()``
              (interpolation, drag, cell lists, collisions; with ``hdi`` hydrodynamic
              interaction and overlap removal; with ``grow`` coalescence), then the
              statistics and the droplet state read back as a driver does at an output step;
* ``flow``    the carrier flow alone (spin-up of a forced field, decaying turbulence);
* ``update``  droplets advanced in a field that an outside solver hands over;
* ``calls``   the separate subroutines in the order of the Fortran main loop, the field
              handed over component by component;
* ``adjoint`` loss and gradients of a droplet statistic through many substeps (autograd);
* ``diag``    the growth diagnostics of an output step: dissipation field, its
              interpolation to the droplets, Stokes averages and size distribution.

Sizes, physical constants and droplet populations are those of the repository's benchmark
configurations (64^3 / 20,000, 128^3 / 100,000 and 200,000, 256^3 / 1M, 512^3 / 5M) and of
grids and counts between them.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from mpi_2d_domain_decomp_turb_particles_b200 import ParticleParams, Partlib
from mpi_2d_domain_decomp_turb_particles_b200.adjoint import AdjointParams, DropletAdjoint, droplet_loss
from mpi_2d_domain_decomp_turb_particles_b200.flow import Flow

PI2 = 2.0 * math.pi
SETS_UM = [10.0, 20.0, 30.0, 40.0]


def listed():
    return [
        # smallest call: one time step of a 64^3 / 20,000 droplet run by the separate
        # subroutines; latency and launches
        dict(name="calls-64-fp64", kind="calls", n=64, npart=20_000, precision="fp64", steps=1),
        # the CPU-runnable configuration: deterministic forcing, collisions, FP64
        dict(name="dns-64-fp64", kind="dns", n=64, npart=20_000, precision="fp64", hdi=False, grow=False,
             forcing=1, steps=5),
        # 128^3 with stochastic forcing, two radii, mixed precision, an odd droplet count
        dict(name="dns-128-mixed", kind="dns", n=128, npart=99_991, precision="mixed", hdi=False, grow=False,
             forcing=2, steps=5),
        # hydrodynamic interaction in FP64 (the accuracy reference of the mixed path)
        dict(name="dns-128-hdi-fp64", kind="dns", n=128, npart=100_000, precision="fp64", hdi=True, grow=False,
             forcing=1, steps=5),
        # the production run: 256^3, a million droplets, hydrodynamic interaction, mixed
        dict(name="dns-256-hdi-mixed", kind="dns", n=256, npart=1_000_000, precision="mixed", hdi=True, grow=False,
             forcing=1, steps=5),
        # the largest: 512^3, five million lognormal droplets that coalesce
        dict(name="dns-512-grow-mixed", kind="dns", n=512, npart=5_000_000, precision="mixed", hdi=True, grow=True,
             forcing=1, steps=5),
        # droplets in a field handed over by another solver, both precisions
        dict(name="update-256-mixed", kind="update", n=256, npart=1_000_000, precision="mixed", steps=16),
        dict(name="update-256-fp64", kind="update", n=256, npart=1_000_000, precision="fp64", steps=16),
        # the flow alone: spin-up at the production size, and a decaying field on a grid
        # that is not a power of two
        dict(name="flow-256", kind="flow", n=256, forcing=1, steps=5),
        dict(name="flow-192", kind="flow", n=192, forcing=0, steps=5),
        # gradients through 100 substeps
        dict(name="adjoint-128-mixed", kind="adjoint", n=128, npart=200_000, precision="mixed", steps=100),
        # diagnostics of an output step of a growth run
        dict(name="diag-256", kind="diag", n=256, npart=1_000_000, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dns", "dns", "dns", "flow", "flow", "update", "update", "calls", "adjoint", "diag"])
    # grids: powers of two (what the reference runs on), otherwise any even size
    n = rng.choice([32, 64, 128, 128, 256, 256]) if rng.random() < 0.6 else 2 * _log(rng, 16, 160)
    npart = min(_log(rng, 500, 40 * n * n), 1_500_000, n ** 3 // 12)   # up to the listed densities
    precision = rng.choice(["fp64", "mixed"])
    if kind == "flow":
        if rng.random() < 0.2:
            n = 512
        return dict(kind=kind, n=n, forcing=rng.choice([0, 1, 2]), steps=rng.choice([2, 3, 5]))
    if kind == "dns":
        hdi = rng.random() < 0.5
        return dict(kind=kind, n=n, npart=npart, precision=precision, hdi=hdi, grow=hdi and rng.random() < 0.3,
                    forcing=rng.choice([0, 1, 2]), steps=5)
    if kind == "update":
        return dict(kind=kind, n=n, npart=npart, precision=precision, steps=rng.choice([8, 16, 20]))
    if kind == "calls":
        return dict(kind=kind, n=n, npart=npart, precision=precision, steps=rng.choice([1, 2]))
    if kind == "adjoint":
        return dict(kind=kind, n=min(n, 128), npart=min(npart, 150_000), precision=precision,
                    steps=rng.choice([25, 40, 60]))
    return dict(kind=kind, n=n, npart=npart, precision=precision)


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
def _constants(case):
    """dt, viscosity, Kolmogorov scales and cloud constants of the benchmark configuration
    whose grid is nearest; the stochastic forcing has its own set (its amplitude needs a
    larger viscosity and a smaller step)."""
    n = case["n"]
    if case.get("forcing") == 2:
        if n <= 160:
            return dict(dt=1e-4, rnu=0.09449408, etk_dns=0.02189, tauk_dns=0.005072)
        return dict(dt=4.1e-5, rnu=0.0375, etk_dns=0.0118, tauk_dns=0.0037)
    if n <= 96:
        return dict(dt=1e-3, rnu=0.0025, etk_dns=0.0282, tauk_dns=0.318, ediss_cloud=1554.0, gravity=771.0)
    if n <= 384:
        return dict(dt=5e-4, rnu=8e-4, etk_dns=0.0079, tauk_dns=0.078)
    return dict(dt=2.5e-4, rnu=3e-4, etk_dns=0.00484, tauk_dns=0.078)


def _radii(case):
    """The set radii (um) of the population."""
    if case.get("grow"):
        return [10.0, 25.0, 60.0]
    if case["kind"] == "dns" and not case["hdi"]:
        return [20.0] if case["n"] <= 96 else [20.0, 30.0]
    return SETS_UM


def _field(n, seed, pad=0):
    """Periodic solenoidal velocity (3, n, n, n + pad), x fastest, random phases, spectrum
    k^4 exp(-2 (k/4)^2), u' = 1 per component: what the repository's configurations start
    from."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    kr = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
    kv = (kr[None, None, :], k[None, :, None], k[:, None, None])
    k2 = kv[0] ** 2 + kv[1] ** 2 + kv[2] ** 2
    amp = k2.sqrt() * torch.exp(-k2 / 16.0)
    a = [torch.view_as_complex(torch.randn(*k2.shape, 2, generator=gen, device="cuda", dtype=torch.float64)) * amp
         for _ in range(3)]
    k2[0, 0, 0] = 1.0
    div = (kv[0] * a[0] + kv[1] * a[1] + kv[2] * a[2]) / k2
    out = torch.zeros((3, n, n, n + pad), device="cuda", dtype=torch.float64)
    for c in range(3):
        u = torch.fft.irfftn(a[c] - kv[c] * div, s=(n, n, n))
        out[c, :, :, :n] = u / u.square().mean().sqrt()
    return out


def _scales(case):
    """Unit scalings of the particle path: radius in DNS units per um, 2/9 rho-ratio drag
    constant (tau_p = tau2 a^2) and settling constant (W = sv a^2)."""
    c = dict(dict(ediss_cloud=400.0, gravity=980.0), **_constants(case))
    visc, rho = 0.17, 1000.0
    etk = (visc ** 3 / c["ediss_cloud"]) ** 0.25
    tauk = (visc / c["ediss_cloud"]) ** 0.5
    vk_ratio = (etk / tauk) / (c["etk_dns"] / c["tauk_dns"])
    tau1 = 2.0 * rho * (etk / c["etk_dns"]) ** 2 / (9.0 * visc)
    return c["etk_dns"] / etk / 1e4, tau1 / (tauk / c["tauk_dns"]), tau1 * c["gravity"] / vk_ratio


def _droplets(case, seed):
    """yp rows (npart, 8): uniform positions, the population's radii, id."""
    rng = np.random.default_rng(seed)
    npart, um = case["npart"], _radii(case)
    yp = np.zeros((npart, 8))
    yp[:, :3] = rng.uniform(0.0, PI2, size=(npart, 3))
    if case.get("grow"):
        a = np.clip(rng.lognormal(math.log(25.0) - 0.045, 0.3, npart), 10.0, 60.0)
    elif um is SETS_UM:
        a = rng.uniform(10.0, 40.0, npart)
    else:
        a = np.asarray(um)[np.arange(npart) * len(um) // npart]
    yp[:, 6] = a * _scales(case)[0]
    yp[:, 7] = np.arange(1, npart + 1)
    return yp


def _partlib(case, seed):
    hdi = bool(case.get("hdi"))
    p = ParticleParams(nx=case["n"], npart=case["npart"], radius_um=_radii(case), precision=case["precision"],
                       hdi_included=hdi, nonoverlap=hdi, msize=case["npart"], mevent=case["npart"],
                       **_constants(case))
    g = Partlib(p)
    g.part_init()
    g.set_particles(_droplets(case, seed))
    return g


class _State:
    """What the program keeps between passes; the droplet arrays live in pinned host memory."""

    def __init__(self, case):
        self.case = case
        if "npart" in case and case["kind"] != "adjoint":
            self.yp = torch.zeros((case["npart"], 8), dtype=torch.float64, pin_memory=True)
            self.vp = torch.zeros((case["npart"], 3), dtype=torch.float64, pin_memory=True)

    def read_droplets(self):
        """yp and vp in reference order through the C boundary (a driver's own arrays)."""
        g, n = self.g, C.c_int(0)
        ptr = [C.cast(C.c_void_p(t.data_ptr()), C.POINTER(C.c_double)) for t in (self.yp, self.vp)]
        g._chk(g.lib.dl_get_particles(g.h, C.byref(n), ptr[0], None, None, ptr[1], None))
        if n.value < self.case["npart"]:   # droplets lost to coalescence
            self.yp[n.value:] = 0.0
            self.vp[n.value:] = 0.0
        return {"pos": self.yp[:, 0:3], "vel": self.yp[:, 3:6], "radius": self.yp[:, 6], "id": self.yp[:, 7],
                "vp": self.vp}


def _flow(case, u0):
    c = _constants(case)
    fl = Flow(case["n"], c["rnu"], c["dt"], forcing=case["forcing"], force=(0.01, 0.1))
    fl.set_velocity(u0)
    return fl


def prepare(case, seed):
    s = _State(case)
    kind, n = case["kind"], case["n"]
    if kind == "adjoint":
        s.u = _field(n, seed, pad=2).requires_grad_()
        yp = torch.from_numpy(_droplets(case, seed)).cuda()
        _, tau2, sv = _scales(case)
        s.x0 = yp[:, :3].contiguous().requires_grad_()
        s.radius = yp[:, 6].contiguous()
        s.tau = (tau2 * s.radius ** 2).requires_grad_()
        s.problem = DropletAdjoint(AdjointParams(n=n, nsteps=case["steps"], dt=_constants(case)["dt"],
                                                 gravity=sv / tau2, precision=case["precision"]), case["npart"])
        return s
    if kind in ("flow", "dns"):
        s.fl = _flow(case, _field(n, seed))
    if kind == "diag":
        s.fl = _flow(dict(case, forcing=1), _field(n, seed))
    if kind in ("update", "calls"):
        f = _field(n, seed, pad=2)
        s.field = [f[c] for c in range(3)]
    if kind != "flow":
        s.g = _partlib(case, seed)
        if case.get("hdi"):
            if case["grow"]:
                s.g.set_step(40_000)   # past the step at which collided droplets coalesce
            s.g.overlap_det()
    return s


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def _velocity(s):
    """The flow's velocity buffers; the views keep the flow alive."""
    u = s.fl.velocity_tensors()
    for t in u:
        t.owner = s
    return u


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "adjoint":
        loss = droplet_loss(s.u, s.x0, s.tau, s.radius, s.problem)
        du, dx0, dtau = torch.autograd.grad(loss, (s.u, s.x0, s.tau))
        return {"loss": loss.detach(), "du": du, "dx0": dx0, "dtau": dtau}
    if kind == "flow":
        for _ in range(case["steps"]):
            s.fl.step()
        return {"u": _velocity(s)}
    if kind == "dns":
        for _ in range(case["steps"]):
            s.fl.step(s.g)
            rep, _ = s.g.particle_step()
        out = s.read_droplets()
        h = s.g.histograms(written=True)
        counts = [*rep.icc, rep.ncoll, rep.ntotpair, rep.ncontact]
        out["counts"] = np.concatenate([np.asarray(counts, np.int32), h.pop("nirbin").ravel()])
        out["sums"] = np.stack([h[k] for k in sorted(h)])
        out["mean_vel"] = s.g.mean_vel()
        out["u"] = _velocity(s)
        return out
    if kind == "update":
        s.g.set_fields(*s.field)
        for _ in range(case["steps"]):
            s.g.update_step()
        return s.read_droplets()
    if kind == "calls":
        for _ in range(case["steps"]):
            s.g.prepare_interp()
            for c in range(3):
                s.g.interpolate(s.field[c], c + 1)
            s.g.part_history_fvp()
            s.g.part_history_fdp()
            s.g.part_advance()
            s.g.update_part_position()
            s.g.periodic()
        return s.read_droplets()
    e = s.fl.dissipation_tensor()
    e.owner = s
    s.g.interp_scalar(e, 2)
    sizes, mass = s.g.size_dist_log()
    return {"dissipation": e, "disp_p": s.g.scalar(2), "stokes": np.array(s.g.local_st_avg()), "sizes": sizes,
            "mass": mass, "size": np.array(s.g.size_avg())}


# ---------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------
def work(case):
    """Per flow step: the spectral velocity and the previous nonlinear term read and
    written, the physical velocity written, 9 transforms of 2.5 n^3 log2(n^3) operations.
    Per droplet step: the field read once, the droplet's position, velocity and histories
    (188 bytes mixed, 324 FP64), 216 points x 3 components x 2 operations and the drag.
    With hydrodynamic interaction: the neighbour solve reads and writes its vectors and
    about one neighbour per droplet a few times."""
    n, kind, steps = case["n"], case["kind"], case.get("steps", 1)
    n3, np_ = n ** 3, case.get("npart", 0)
    e = 4 if case.get("precision") == "mixed" else 8
    spec, fft = 16 * n * n * (n // 2 + 1), 2.5 * n3 * math.log2(n3)
    b = f = 0.0
    if kind in ("flow", "dns"):
        b += steps * (4 * 3 * spec + 3 * 8 * n3)
        f += steps * (9 * fft + 60 * n3)
    if kind in ("update", "dns", "calls"):
        b += steps * (3 * n3 * e + np_ * (188 if e == 4 else 324))
        f += steps * np_ * (1296 + 300)
        b += np_ * 11 * 8
    if kind in ("update", "calls"):
        b += 3 * n3 * 8 * (steps if kind == "calls" else 1)
    if kind == "dns":
        b += steps * np_ * (13 * 8 + 48)           # collision detection: state and cell keys
        if case["hdi"]:
            b += steps * np_ * (2 * 48 + 10 * (6 * e + 28))
            f += steps * np_ * 10 * 40
    if kind == "adjoint":
        # forward, recomputation and reverse sweep each gather the stencils; the gradient scatters once
        b += 2 * 3 * n3 * 8 + 3 * steps * np_ * 188
        f += 3 * steps * np_ * 1600 + 2 * steps * np_ * 1300
    if kind == "diag":
        b += 3 * spec + 8 * n3 + 8 * n3 + np_ * (24 + 8 + 8)
        f += 6 * fft + 20 * n3 + np_ * 700
    return {"bytes": b, "flops": f}


def tolerance(case):
    """FP64 paths differ by the rounding of transforms and sums (1e-15 here, a few steps
    long).  The mixed path holds FP32 velocities: 1e-6 at most between it and FP64, counts
    equal.  The adjoint's loss averages the relative velocity of a few close pairs, a small
    difference of FP32 velocities: 4e-4 from FP64, its gradients 1.4e-4."""
    kind = case["kind"]
    if kind == "adjoint":
        return {"rel": 1.5e-3, "max": 0.1} if case["precision"] == "mixed" else {"rel": 1e-10}
    if case.get("precision") == "mixed" and kind != "diag":
        return {"rel": 4e-6, "max": 4e-5, "differ": 0.003}
    return {"rel": 1e-8 if case.get("hdi") else 1e-11, "differ": 0.002}


# ---------------------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------
class _Ran:
    """Minimal standard generator with Bays-Durham shuffle (the stochastic forcing's)."""

    def __init__(self, seed):
        self.s = max(seed, 1)
        self.v = [0] * 32
        for j in range(40, 0, -1):
            self.s = self.s * 16807 % 2147483647
            if j <= 32:
                self.v[j - 1] = self.s
        self.y = self.v[0]

    def __call__(self):
        self.s = self.s * 16807 % 2147483647
        j = self.y // (1 + 2147483646 // 32)
        self.y, self.v[j] = self.v[j], self.s
        return min(self.y / 2147483647, 1.0 - 1.2e-7)


class _ExactFlow:
    """Pseudo-spectral step: u x omega, spherical dealiasing, Crank-Nicolson + AB2, forcing of
    the large scales, projection, conjugate symmetry of kx = 0."""

    def __init__(self, case, u0):
        c, n = _constants(case), case["n"]
        self.n, self.nu, self.dt, self.forcing = n, c["rnu"], c["dt"], case["forcing"]
        k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
        kr = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
        self.k = (kr[None, None, :], k[None, :, None], k[:, None, None])
        k2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        self.shell = torch.floor(k2.sqrt() + 0.5)
        self.keep = self.shell <= int(n / 2 - 1.5)
        k2[0, 0, 0] = 1e-5
        self.k2 = k2
        self.b, self.ran = np.zeros((3, 5, 5, 6)), _Ran(232300)
        self.uh = self.finish(self.project([self.fwd(u0[c]) for c in range(3)]))
        self.old = [a.clone() for a in self.uh]

    def fwd(self, a):
        return torch.fft.rfftn(a, norm="forward")

    def inv(self, a):
        return torch.fft.irfftn(a, s=(self.n,) * 3, norm="forward")

    def project(self, v):
        t = (self.k[0] * v[0] + self.k[1] * v[1] + self.k[2] * v[2]) / self.k2
        return [v[c] - self.k[c] * t for c in range(3)]

    def finish(self, v):
        h, out = self.n // 2, []
        for a in v:
            a = torch.where(self.keep, a, 0.0)
            a[0, 0, 0] = 0.0
            a[:, :, h] = 0.0
            a[:, h, :] = 0.0
            a[h, :, :] = 0.0
            p = a[:, :, 0]
            a[:, :, 0] = 0.5 * (p + torch.roll(torch.flip(p, (0, 1)), (1, 1), (0, 1)).conj())
            out.append(a)
        return out

    def amplitudes(self):
        """Ornstein-Uhlenbeck forcing of the modes kx <= 2, |ky|, |kz| <= 2, solenoidal."""
        var, tf, dt, kw = 447.31, 0.038, self.dt, (0, 1, 2, -2, -1)
        fr = np.zeros((3, 5, 5, 6))
        for q in range(3 * 25 * 3):
            r = math.sqrt(-4.0 * var * dt * math.log(max(self.ran(), 1e-6)) / tf)
            ph = 8.0 * math.atan(1.0) * self.ran()
            fr.reshape(-1, 2)[q] = r * math.cos(ph), r * math.sin(ph)

        def mirror(v):
            for k in range(5):
                for j in (1, 2):
                    v[-k % 5, 5 - j, 0:2] = v[k, j, 0], -v[k, j, 1]
            for k in (1, 2):
                v[5 - k, 0, 0:2] = v[k, 0, 0], -v[k, 0, 1]

        for c in range(3):
            mirror(fr[c])
            fr[c, 0, 0, 0:2] = 0.0
        a = np.zeros_like(fr)
        for k in range(5):
            for j in range(5):
                for i in range(6):
                    kk = np.array([i // 2, kw[j], kw[k]], float)
                    rad = math.sqrt(kk @ kk)
                    if rad < math.sqrt(8.0):
                        self.b[:, k, j, i] = self.b[:, k, j, i] * (1.0 - dt / tf) + fr[:, k, j, i]
                        b = self.b[:, k, j, i]
                        a[:, k, j, i] = b - kk * ((kk @ b) / rad ** 2 if rad else 0.0)
        for c in range(3):
            a[c, 0, 0, 0:2] = 0.0
            mirror(a[c])
        return a

    def step(self):
        k, dth = self.k, 0.5 * self.dt
        u = [self.inv(a) for a in self.uh]
        rot = [self.inv(1j * (k[(c + 1) % 3] * self.uh[(c + 2) % 3] - k[(c + 2) % 3] * self.uh[(c + 1) % 3]))
               for c in range(3)]
        new = [torch.where(self.keep, self.fwd(u[(c + 1) % 3] * rot[(c + 2) % 3] - u[(c + 2) % 3] * rot[(c + 1) % 3]),
                           0.0) for c in range(3)]
        lin = 1.0 - self.nu * dth * self.k2
        v = [self.uh[c] * lin + 1.5 * self.dt * new[c] - dth * self.old[c] for c in range(3)]
        if self.forcing == 2:
            a, at = self.amplitudes(), (0, 1, 2, self.n - 2, self.n - 1)
            for c in range(3):
                f = torch.from_numpy(a[c, :, :, 0::2] + 1j * a[c, :, :, 1::2]).cuda()
                for q in range(5):
                    for j in range(5):
                        v[c][at[q], at[j], 0:3] += self.dt * f[q, j]
        v = [a / (1.0 + self.nu * dth * self.k2) for a in self.project(v)]
        if self.forcing == 1:
            for s, f in ((1.0, 0.01), (2.0, 0.1)):
                w = torch.where(self.shell == s, 1.0, 0.0).to(torch.float64)
                w[:, :, 0] *= 0.5
                e = sum((w * (a.real ** 2 + a.imag ** 2)).sum() for a in v)
                v = [torch.where(self.shell == s, a * torch.sqrt(f / e), a) for a in v]
        self.uh, self.old = self.finish(v), new
        return u

    def dissipation(self):
        k, v, e = self.k, self.uh, 0.0
        for i in range(3):
            for j in range(i, 3):
                t = self.inv(0.5j * (k[j] * v[i] + k[i] * v[j]))
                e = e + (1.0 if i == j else 2.0) * t * t
        return 2.0 * self.nu * e


def _weights(z):
    """Lagrange weights of the nodes -2..3 at fraction z, as products over the other nodes."""
    out = []
    for a in range(-2, 4):
        w = torch.ones_like(z)
        for m in range(-2, 4):
            if m != a:
                w = w * ((z - m) / (a - m))
        out.append(w)
    return torch.stack(out, -1)


def _interp(fields, x, n):
    """Six-point Lagrange interpolation of each (n, n, >= n) field at x (np, 3)."""
    dx = PI2 / n
    node = torch.floor(x.detach() / dx)
    z = x / dx - node
    w = [_weights(z[:, d]) for d in range(3)]
    i = [(node[:, d, None].long() + torch.arange(-2, 4, device=x.device)) % n for d in range(3)]
    py, pz = fields[0].stride(1), fields[0].stride(0)
    at = (i[2][:, :, None, None] * pz + i[1][:, None, :, None] * py + i[0][:, None, None, :]).reshape(len(x), -1)
    ww = (w[2][:, :, None, None] * w[1][:, None, :, None] * w[0][:, None, None, :]).reshape(len(x), -1)
    return torch.stack([(f.reshape(-1)[at] * ww).sum(1) for f in fields], -1)


def _interp_all(fields, x, n):
    return torch.cat([_interp(fields, c, n) for c in x.split(1 << 16)])


def _reorder(y, z):
    """Order of the droplets after PERIODIC on one rank: a droplet that leaves through y or z
    is replaced by the last one still in the list; the departed are appended by neighbour."""
    hi, lo = y > PI2, y < 0.0
    up, dn = z > PI2, z < 0.0
    nid = np.select([hi & up, hi & dn, hi, lo & up, lo & dn, lo, up, dn], [2, 8, 1, 4, 6, 5, 3, 7], 0)
    order, n, gone = np.arange(len(y)), len(y), [[] for _ in range(9)]
    out = 0
    for at in np.flatnonzero(nid):
        while at < n - out and nid[order[at]]:
            gone[nid[order[at]]].append(order[at])
            out += 1
            order[at] = order[n - out]
    return np.concatenate([order[:n - out]] + [np.asarray(q, order.dtype) for q in gone[1:]])


class _ExactDroplets:
    """Interpolation, implicit multistep drag and gravity, wrap and reorder (no HDI)."""

    def __init__(self, case, seed):
        yp = torch.from_numpy(_droplets(case, seed)).cuda()
        _, self.tau2, self.sv = _scales(case)
        self.n, self.dt = case["n"], _constants(case)["dt"]
        self.x, self.r, self.id = yp[:, :3].clone(), yp[:, 6].clone(), yp[:, 7].clone()
        self.v = None

    def step(self, u):
        dt, vp = self.dt, _interp_all(u, self.x, self.n)
        if self.v is None:
            self.v = torch.zeros_like(self.x)
            self.v[:, 0] = self.sv * self.r ** 2
            self.fv, self.fd = [self.v, self.v], [vp, vp, vp]
        tau = (self.tau2 * self.r ** 2)[:, None]
        g = torch.zeros_like(self.x)
        g[:, 0] = self.sv / self.tau2
        d = dt / (24.0 * tau)
        tv = 19.0 * self.v - 5.0 * self.fv[0] + self.fv[1]
        td = 55.0 * vp - 59.0 * self.fd[0] + 37.0 * self.fd[1] - 9.0 * self.fd[2]
        new = (self.v + dt * g - d * tv + d * td) / (1.0 + 9.0 * d)
        self.x = self.x + dt / 24.0 * (9.0 * new + tv)
        self.fv, self.fd, self.v, self.vp = [self.v, self.fv[0]], [vp, self.fd[0], self.fd[1]], new, vp
        yz = self.x[:, 1:].cpu().numpy()
        o = torch.from_numpy(_reorder(yz[:, 0], yz[:, 1])).cuda()
        self.x, self.r, self.id, self.v = self.x[o], self.r[o], self.id[o], self.v[o]
        self.fv, self.fd = [a[o] for a in self.fv], [a[o] for a in self.fd]
        self.x = torch.where(self.x >= PI2, self.x - PI2, self.x)
        self.x = torch.where(self.x < 0.0, self.x + PI2, self.x)

    def out(self, vp):
        return {"pos": self.x, "vel": self.v, "radius": self.r, "id": self.id, "vp": vp}


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint
    n, np_, dt = case["n"], case["npart"], _constants(case)["dt"]
    _, tau2, sv = _scales(case)
    u = _field(n, seed, pad=2).requires_grad_()
    yp = torch.from_numpy(_droplets(case, seed)).cuda()
    x0, rad = yp[:, :3].contiguous().requires_grad_(), yp[:, 6].contiguous()
    tau = (tau2 * rad ** 2).requires_grad_()
    grav = torch.tensor([sv / tau2, 0.0, 0.0], device="cuda", dtype=torch.float64)

    def step(u, x, v, f1, f2, u1, u2, u3, tau, first):
        u0 = _interp(list(u), x, n)
        u1, u2, u3 = (u0, u0, u0) if first else (u1, u2, u3)
        d = dt / (24.0 * tau[:, None])
        tv = 19.0 * v - 5.0 * f1 + f2
        td = 55.0 * u0 - 59.0 * u1 + 37.0 * u2 - 9.0 * u3
        new = (v + dt * grav - d * tv + d * td) / (1.0 + 9.0 * d)
        return x + dt / 24.0 * (9.0 * new + tv), new, u0, u1, u2

    x, v = x0, grav * tau[:, None]
    f1 = f2 = v
    h = [torch.zeros_like(x0)] * 3
    for q in range(case["steps"]):
        x, new, *h = checkpoint(step, u, x, v, f1, f2, *h, tau, q == 0, use_reentrant=False)
        v, f1, f2 = new, v, f1
    loss = ((x - x0) ** 2).sum() / np_
    xd, pairs = x.detach(), []
    for lo in range(0, np_, 4096):
        r2 = 0.0
        for c in range(3):
            r = xd[lo:lo + 4096, c, None] - xd[None, :, c]
            r2 = r2 + (r - PI2 * torch.floor(r / PI2 + 0.5)) ** 2
        i, j = torch.nonzero(r2 < (2.0 * (rad[lo:lo + 4096, None] + rad[None, :])) ** 2, as_tuple=True)
        pairs.append(torch.stack([i + lo, j])[:, i + lo < j])
    i, j = torch.cat(pairs, 1)
    if len(i):
        r = x[i] - x[j]
        r = r - PI2 * torch.floor(r.detach() / PI2 + 0.5)
        loss = loss + (((v[i] - v[j]) * r).sum(1) / r.norm(dim=1)).mean()
    du, dx0, dtau = torch.autograd.grad(loss, (u, x0, tau))
    return {"loss": loss.detach(), "du": du, "dx0": dx0, "dtau": dtau}


def exact(case, seed):
    """None for what has no closed 64-bit counterpart here: the state after hydrodynamic
    interaction (an iterative solve), counts and histogram sums."""
    kind, n = case["kind"], case["n"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if kind in ("update", "calls"):
        f = _field(n, seed, pad=2)
        d = _ExactDroplets(case, seed)
        for _ in range(case["steps"]):
            d.step(list(f))
        return d.out(None)
    fl = _ExactFlow(dict(dict(forcing=1), **case), _field(n, seed))
    if kind == "flow":
        for _ in range(case["steps"]):
            u = fl.step()
        return {"u": u}
    if kind == "dns":
        d = None if case["hdi"] else _ExactDroplets(case, seed)
        for _ in range(case["steps"]):
            u = fl.step()
            if d is not None:
                d.step(u)
        out = dict.fromkeys(("pos", "vel", "radius", "id", "vp")) if d is None else d.out(None)
        return dict(out, counts=None, sums=None, mean_vel=None, u=u)
    e = fl.dissipation()
    yp = torch.from_numpy(_droplets(case, seed)).cuda()
    scale, tau2, _ = _scales(case)
    c, r, a0 = _constants(case), yp[:, 6], _radii(case)[0] * scale
    at = _interp_all([e], yp[:, :3], n)[:, 0]
    at = torch.where(at < 0.0, 1e-5, at)
    st = tau2 * r ** 2 * torch.sqrt(at / c["rnu"])
    st1 = tau2 * a0 ** 2 / c["tauk_dns"]
    ir = torch.clamp(torch.log((r / a0) ** 3) / (math.log(2.0) / 32.0) + 1.5, 1.0, 360.0).long() - 1
    mass = torch.zeros(360, device="cuda", dtype=torch.float64).index_add_(0, ir, 4.0 / 3.0 * math.pi * r ** 3)
    return {"dissipation": e, "disp_p": at, "stokes": torch.stack([st.mean(), st[r.argmax()]]) / st1,
            "sizes": torch.bincount(ir, minlength=360).int(), "mass": mass * 96.0 / math.log(2.0),
            "size": torch.stack([(r ** 3).mean() ** (1.0 / 3.0), r.max()]) / a0}
