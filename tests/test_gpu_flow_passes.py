"""The flow step's own transform passes (grids 2^a and 3 * 2^a, csrc/dl_flow_passes.cuh)
against the numpy restatement, at every supported size class: two-stage and three-stage
lines, radix 12 and 6 butterflies, partly filled stages, and the library path beside them.

Tolerance: one step's transforms round at a few 1e-16 relative to the field's norm (the
error of an FFT grows like log n), the nonlinear term is a product of two of them; 2e-14
leaves a factor of about 20.
"""
import numpy as np
import pytest
import torch

from cases import dense_params
from flow_oracle import FlowOracle
from test_flow_oracle import random_velocity
from mpi_2d_domain_decomp_turb_particles_b200 import Partlib
from mpi_2d_domain_decomp_turb_particles_b200.flow import Flow

pytestmark = pytest.mark.gpu
TOL = 2e-14


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n,forcing,steps", [(32, 1, 3), (40, 1, 2), (48, 2, 3), (64, 0, 2), (64, 1, 2), (96, 2, 2),
                                             (128, 1, 2), (192, 1, 1), (256, 1, 1)])
def test_steps_match_restatement(n, forcing, steps):
    kw = dict(forcing=forcing, force=(0.3, 0.2), iseedf=232300)
    o = FlowOracle(n, 0.02, 0.001, workers=8, **kw)
    g = Flow(n, 0.02, 0.001, **kw)
    u0 = random_velocity(n)
    o.set_velocity(u0)
    g.set_velocity(u0)
    for _ in range(steps):
        uo = o.step()
        g.step()
    uh, nold = g.spectral()
    assert rel(g.velocity(), uo) < TOL
    assert rel(uh, o.uh) < TOL and rel(nold, o.nold) < TOL
    assert rel(g.dissipation(), o.dissipation()) < TOL
    # the transform of the diagnostics leaves the next step as it was
    uo = o.step()
    g.step()
    assert rel(g.velocity(), uo) < TOL
    g.close()


@pytest.mark.parametrize("n", [384, 512])
def test_three_stage_lines(n):
    """Velocity and nonlinear term of the largest grids against torch's transforms."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    kv = (torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)[None, None, :], k[None, :, None], k[:, None, None])
    g = Flow(n, 1e-3, 1e-4)
    g.set_velocity(torch.randn((3, n, n, n), generator=gen, device="cuda", dtype=torch.float64))
    uh = torch.from_numpy(g.spectral()[0]).cuda()
    g.step()
    nold = torch.from_numpy(g.spectral()[1]).cuda()
    inv = lambda a: torch.fft.irfftn(a, s=(n,) * 3, norm="forward")   # noqa: E731
    u = [inv(uh[c]) for c in range(3)]
    for c, t in enumerate(g.velocity_tensors()):
        assert float((t - u[c]).norm() / u[c].norm()) < TOL
    w = [inv(1j * (kv[(c + 1) % 3] * uh[(c + 2) % 3] - kv[(c + 2) % 3] * uh[(c + 1) % 3])) for c in range(3)]
    keep = torch.floor((kv[0] ** 2 + kv[1] ** 2 + kv[2] ** 2).sqrt() + 0.5) <= int(n / 2 - 1.5)
    for c in range(3):
        a, b = (c + 1) % 3, (c + 2) % 3
        ref = torch.where(keep, torch.fft.rfftn(u[a] * w[b] - u[b] * w[a], norm="forward"), 0.0)
        assert float((nold[c] - ref).norm() / ref.norm()) < TOL
    g.close()


@pytest.mark.parametrize("n", [48, 64])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_emitted_field_equals_the_converted_one(n, precision):
    """The droplet field the x pass writes (with its periodic halo) interpolates to the same
    bits as the step's velocity handed over through dl_set_field."""
    g = Flow(n, 0.02, 0.001)
    g.set_velocity(random_velocity(n))
    d = [Partlib(dense_params(n=n, npart=4000, precision=precision)) for _ in range(2)]
    for p in d:
        p.part_init()
    g.step(d[0])
    d[1].set_fields(*g.velocity_tensors())
    for p in d:
        p.update_step()
    a, b = (p.get_particles() for p in d)
    assert all(np.array_equal(a[k], b[k]) for k in a)
    for p in d:
        p.close()
    g.close()


def test_n_old_outside_the_sphere_is_dropped():
    """A state set with N_old in the dealiased modes: kept as given until the step, zero after."""
    n = 32
    o, g = FlowOracle(n, 0.02, 0.001), Flow(n, 0.02, 0.001)
    rng = np.random.default_rng(3)
    o.set_velocity(random_velocity(n))
    o.nold = rng.standard_normal(o.nold.shape) + 1j * rng.standard_normal(o.nold.shape)
    g.set_spectral(o.uh, o.nold)
    uh, nold = g.spectral()
    assert np.array_equal(nold, o.nold) and rel(uh, o.uh) < 1e-15
    o.step()
    g.step()
    uh, nold = g.spectral()
    assert rel(uh, o.uh) < TOL and rel(nold, o.nold) < TOL
    assert not nold[:, o.ik2 > o.nek].any() and not uh[:, o.ik2 > o.nek].any()
    g.close()


def spectral_state(n, scale, seed):
    """Spectra of three real random fields of the given magnitudes, dealiased, on the device."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k, keep = wavenumbers(n)
    uh = [torch.fft.rfftn(torch.randn((n, n, n), generator=gen, device="cuda", dtype=torch.float64), norm="forward")
          for _ in range(3)]
    return torch.stack([torch.where(keep, s * a, 0.0) for s, a in zip(uh, scale)])


def wavenumbers(n):
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=torch.float64)
    kv = (torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)[None, None, :], k[None, :, None], k[:, None, None])
    return kv, torch.floor((kv[0] ** 2 + kv[1] ** 2 + kv[2] ** 2).sqrt() + 0.5) <= int(n / 2 - 1.5)


@pytest.mark.parametrize("n,c", [(32, 0), (48, 1), (64, 2), (96, 0), (128, 1), (192, 2), (256, 0), (384, 1)])
def test_components_keep_their_own_accuracy(n, c):
    """Component c a million times the others: every component of the velocity and of N is as
    accurate, against its own norm, as it is where all three are of one magnitude."""
    kv, keep = wavenumbers(n)
    g = Flow(n, 1e-3, 1e-4)
    g.set_spectral(spectral_state(n, [1e6 if q == c else 1.0 for q in range(3)], n).cpu().numpy())
    uh = torch.from_numpy(g.spectral()[0]).cuda()
    g.step()
    nold = torch.from_numpy(g.spectral()[1]).cuda()
    inv = lambda a: torch.fft.irfftn(a, s=(n,) * 3, norm="forward")   # noqa: E731
    u = [inv(uh[q]) for q in range(3)]
    for q, t in enumerate(g.velocity_tensors()):
        assert float((t - u[q]).norm() / u[q].norm()) < TOL
    w = [inv(1j * (kv[(q + 1) % 3] * uh[(q + 2) % 3] - kv[(q + 2) % 3] * uh[(q + 1) % 3])) for q in range(3)]
    for q in range(3):
        a, b = (q + 1) % 3, (q + 2) % 3
        ref = torch.where(keep, torch.fft.rfftn(u[a] * w[b] - u[b] * w[a], norm="forward"), 0.0)
        assert float((nold[q] - ref).norm() / ref.norm()) < TOL
    g.close()


@pytest.mark.parametrize("n", [32, 48, 96, 128, 256])
@pytest.mark.parametrize("c", [0, 1, 2])
def test_plane_flow_stays_plane(n, c):
    """A flow without component c that does not vary along c: exactly so along x and z; along y
    the two rows of a pair round differently."""
    kv, keep = wavenumbers(n)
    a, b = (c + 1) % 3, (c + 2) % 3
    psi = torch.where(kv[c] == 0, spectral_state(n, (1.0, 1.0, 1.0), c)[0], 0.0)
    uh = torch.zeros((3, *psi.shape), dtype=torch.complex128, device="cuda")
    uh[a], uh[b] = 1j * kv[b] * psi, -1j * kv[a] * psi
    g = Flow(n, 1e-2, 1e-4)
    g.set_spectral(uh.cpu().numpy())
    for _ in range(3):
        g.step()
    u = g.velocity_tensors()
    s, nold = (torch.from_numpy(v).cuda() for v in g.spectral())
    mean = u[a].select(2 - c, 0).unsqueeze(2 - c)
    parts = [(u[c], u[a]), (u[a] - mean, u[a]), (s[c], s), (nold[c], nold), (torch.where(kv[c] == 0, 0.0, s), s)]
    for zero, whole in parts:
        assert float(zero.norm() / whole.norm()) <= (TOL if c == 1 else 0.0)
    g.close()


@pytest.mark.parametrize("n", [32, 96, 128, 192, 256, 384, 512])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_emission_of_every_plan(n, precision):
    """As above for every plan and barrier form of the x pass, with droplets at the faces."""
    gen = torch.Generator(device="cuda").manual_seed(n)
    g = Flow(n, 1e-3, 1e-4)
    g.set_velocity(torch.randn((3, n, n, n), generator=gen, device="cuda", dtype=torch.float64))
    d = [Partlib(dense_params(n=n, npart=4000, precision=precision)) for _ in range(2)]
    rng = np.random.default_rng(n)
    faces = rng.choice([0.0, 1e-9, 2 * np.pi - 1e-9], (1000, 3))
    for p in d:
        p.part_init()
        yp = p.get_particles()["yp"]
        yp[:1000, :3] = faces
        p.set_particles(yp)
    g.step(d[0])
    d[1].set_fields(*g.velocity_tensors())
    for p in d:
        p.update_step()
    a, b = (p.get_particles() for p in d)
    assert a["fdp"].any() and all(np.array_equal(a[k], b[k]) for k in a)
    for p in d:
        p.close()
    g.close()


@pytest.mark.parametrize("n", [384, 512])
def test_dissipation_and_forced_step_of_the_largest_grids(n):
    """DISSIP and the update with the deterministic forcing against torch."""
    nu, dt, force = 1e-2, 1e-3, (0.3, 0.2)
    gen = torch.Generator(device="cuda").manual_seed(6)
    kv, _ = wavenumbers(n)
    g = Flow(n, nu, dt, forcing=1, force=force)
    g.set_velocity(torch.randn((3, n, n, n), generator=gen, device="cuda", dtype=torch.float64))
    uh = torch.from_numpy(g.spectral()[0]).cuda()
    diss = torch.zeros((n, n, n), dtype=torch.float64, device="cuda")
    for a in range(3):
        for b in range(a + 1):
            s = torch.fft.irfftn(0.5j * (kv[a] * uh[b] + kv[b] * uh[a]), s=(n,) * 3, norm="forward")
            diss += 2 * nu * (1 if a == b else 2) * s * s
    t = g.dissipation_tensor()
    assert float((t - diss).norm() / diss.norm()) < TOL
    del diss, s
    g.step()
    new, nold = (torch.from_numpy(v).cuda() for v in g.spectral())
    k2 = kv[0] ** 2 + kv[1] ** 2 + kv[2] ** 2
    shell = (k2 > 0).int() * ((k2 <= 2).int() + ((k2 > 2) & (k2 <= 6)).int() * 2)
    k2[0, 0, 0] = 1e-5
    # N_old of the first step is the state itself
    v = uh * (1 - 0.5 * nu * dt * k2) + dt * (1.5 * nold - 0.5 * uh)
    div = (kv[0] * v[0] + kv[1] * v[1] + kv[2] * v[2]) / k2
    v = torch.stack([v[c] - kv[c] * div for c in range(3)]) / (1 + 0.5 * nu * dt * k2)
    e = (v.abs() ** 2).sum(0)
    e[:, :, 0] *= 0.5
    for q in (1, 2):
        v = torch.where(shell == q, v * (force[q - 1] / e[shell == q].sum()).sqrt(), v)
    v[:, 0, 0, 0] = 0.0
    assert float((new - v).norm() / v.norm()) < TOL
    assert float((torch.where(shell > 0, new - v, 0.0)).norm() / torch.where(shell > 0, v, 0.0).norm()) < TOL
    g.close()
