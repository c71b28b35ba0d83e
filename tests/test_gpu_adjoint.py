"""GPU droplet adjoint (dl_adj_*) against the FP64 adjoint reference in the oracle and
against central finite differences.

Bars: FP64 forward bit-identical to the reference (final positions and velocities); FP64
gradients within 1e-12 of the largest entry (only the order of atomic sums differs);
mixed-precision gradients within 1e-4; checkpoint interval invisible; central
differences (h = 1e-6) of the GPU's own FP64 loss within 1e-6; torch.autograd.Function
gradients equal to the direct calls.
"""
import numpy as np
import pytest

import oracle as orc
from test_oracle_adjoint import clustered_case
from mpi_2d_domain_decomp_turb_particles_b200._lib import DropletError
from mpi_2d_domain_decomp_turb_particles_b200.adjoint import AdjointParams, DropletAdjoint, droplet_loss

pytestmark = pytest.mark.gpu

KW = dict(n=16, nsteps=40, dt=0.01, gravity=1.0, pair_factor=3.0)


def gpu_problem(precision, init_velocity=0, checkpoint_every=20, u=None, x0=None, tau=None, rad=None):
    p = AdjointParams(precision=precision, init_velocity=init_velocity, checkpoint_every=checkpoint_every, **KW)
    a = DropletAdjoint(p, len(x0))
    a.set_field(u)
    a.set_droplets(x0, tau, rad)
    return a


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("init_velocity", [0, 1])
def test_fp64_adjoint_matches_reference(init_velocity):
    u, x0, tau, rad = clustered_case()
    ref = orc.AdjointOracle(init_velocity=init_velocity, **KW)
    loss_o, npairs_o, xN_o, vN_o = ref.forward(u, x0, tau, rad)
    _, dx0_o, dtau_o, du_o = ref.gradient(u, x0, tau, rad)
    a = gpu_problem("fp64", init_velocity, u=u, x0=x0, tau=tau, rad=rad)
    loss, npairs = a.forward()
    xN, vN = a.final_state()
    assert npairs == npairs_o >= 10
    assert np.array_equal(xN, xN_o) and np.array_equal(vN, vN_o)
    assert abs(loss - loss_o) <= 1e-14 * abs(loss_o)
    dx0, dtau, du = a.backward()
    assert rel(dx0, dx0_o) < 1e-12
    assert rel(dtau, dtau_o) < 1e-12
    assert rel(du, du_o) < 1e-12
    a.close()


def test_mixed_adjoint_within_1e4_of_fp64_reference():
    u, x0, tau, rad = clustered_case()
    ref = orc.AdjointOracle(**KW)
    _, dx0_o, dtau_o, du_o = ref.gradient(u, x0, tau, rad)
    a = gpu_problem("mixed", u=u, x0=x0, tau=tau, rad=rad)
    a.forward()
    dx0, dtau, du = a.backward()
    assert rel(dx0, dx0_o) < 1e-4
    assert rel(dtau, dtau_o) < 1e-4
    assert rel(du, du_o) < 1e-4
    a.close()


def test_checkpoint_interval_is_invisible():
    u, x0, tau, rad = clustered_case()
    outs = []
    for k in (7, 40):
        a = gpu_problem("fp64", checkpoint_every=k, u=u, x0=x0, tau=tau, rad=rad)
        loss, _ = a.forward()
        outs.append((loss,) + a.backward())
        a.close()
    assert outs[0][0] == outs[1][0]
    assert np.array_equal(outs[0][1], outs[1][1]) and np.array_equal(outs[0][2], outs[1][2])
    assert rel(outs[0][3], outs[1][3]) < 1e-13


def test_fp64_gpu_gradient_matches_central_differences():
    u, x0, tau, rad = clustered_case()
    a = gpu_problem("fp64", u=u, x0=x0, tau=tau, rad=rad)
    a.forward()
    dx0, dtau, du = a.backward()
    h = 1e-6

    def loss_at(u_, x_, t_):
        a.set_field(u_)
        a.set_droplets(x_, t_, rad)
        return a.forward()[0]

    scale = max(np.abs(dx0).max(), np.abs(dtau).max(), np.abs(du).max())
    for i, c in ((0, 0), (17, 1), (33, 2), (50, 0)):
        xp, xm = x0.copy(), x0.copy()
        xp[i, c] += h; xm[i, c] -= h
        fd = (loss_at(u, xp, tau) - loss_at(u, xm, tau)) / (2 * h)
        assert abs(fd - dx0[i, c]) <= 1e-6 * scale
    for i in (3, 41):
        tp_, tm = tau.copy(), tau.copy()
        tp_[i] += h; tm[i] -= h
        fd = (loss_at(u, x0, tp_) - loss_at(u, x0, tm)) / (2 * h)
        assert abs(fd - dtau[i]) <= 1e-6 * scale
    for q in np.argsort(np.abs(du).ravel())[-3:]:
        idx = np.unravel_index(q, du.shape)
        up, um = u.copy(), u.copy()
        up[idx] += h; um[idx] -= h
        fd = (loss_at(up, x0, tau) - loss_at(um, x0, tau)) / (2 * h)
        assert abs(fd - du[idx]) <= 1e-6 * scale
    a.close()


def test_torch_autograd_function():
    import torch
    u, x0, tau, rad = clustered_case()
    a = gpu_problem("fp64", u=u, x0=x0, tau=tau, rad=rad)
    a.forward()
    dx0, dtau, du = a.backward()
    tu = torch.tensor(u, device="cuda", requires_grad=True)
    tx = torch.tensor(x0, device="cuda", requires_grad=True)
    tt = torch.tensor(tau, device="cuda", requires_grad=True)
    tr = torch.tensor(rad, device="cuda")
    loss = droplet_loss(tu, tx, tt, tr, a)
    loss.backward()
    assert np.array_equal(tx.grad.cpu().numpy(), dx0)
    assert np.array_equal(tt.grad.cpu().numpy(), dtau)
    assert rel(tu.grad.cpu().numpy(), du) < 1e-13
    a.close()


@pytest.mark.parametrize("n,np_", [(8, 1), (20, 255), (64, 700), (130, 1025)])
def test_internal_order_is_invisible(n, np_):
    """The device sort of the droplets (2 to 3 digit passes, one to five blocks): host and device
    inputs give the same bits, and droplets handed over in another order give the same final
    states and per-droplet gradients in that order (FP64: every droplet's own arithmetic)."""
    import torch
    from mpi_2d_domain_decomp_turb_particles_b200.adjoint import AdjointParams, DropletAdjoint
    rng = np.random.default_rng(n)
    u = rng.standard_normal((3, n, n, n))
    x0 = rng.uniform(-7.0, 14.0, (np_, 3))
    x0[np_ // 2:] = x0[:np_ - np_ // 2] + 1e-9   # equal keys
    tau, rad = rng.uniform(0.5, 2.0, np_), np.full(np_, 1e-6)
    p = AdjointParams(n=n, nsteps=3, dt=1e-3, gravity=1.0, precision="fp64", pair_factor=0.0)
    perm = rng.permutation(np_)
    res = []
    for order, dev in ((np.arange(np_), False), (np.arange(np_), True), (perm, False)):
        a = DropletAdjoint(p, np_)
        a.set_field(u)
        args = [np.ascontiguousarray(v[order]) for v in (x0, tau, rad)]
        a.set_droplets(*[torch.from_numpy(v).cuda() for v in args] if dev else args)
        a.forward()
        x, v = a.final_state()
        dx0, dtau, _ = a.backward()
        out = [np.empty_like(q) for q in (x, v, dx0, dtau)]
        for o, q in zip(out, (x, v, dx0, dtau)):
            o[order] = q
        res.append(out)
        a.close()
    for r in res[1:]:
        assert all(np.array_equal(p_, q) for p_, q in zip(res[0], r))


@pytest.mark.parametrize("np_", [1, 7, 9, 33])
def test_mixed_gather_at_partial_warps(np_):
    """FP32 gathers eight droplets per warp: counts around a multiple of eight, against FP64.
    One step's interpolant and Jacobian are sums of 216 FP32 terms, a few 1e-7 of the
    field; 2e-5 covers the 10 steps and the division by the small displacement."""
    rng = np.random.default_rng(np_)
    n = 12
    u = rng.standard_normal((3, n, n, n))
    x0, tau = rng.uniform(-3.0, 9.0, (np_, 3)), rng.uniform(0.5, 2.0, np_)
    out = {}
    for prec in ("fp64", "mixed"):
        a = DropletAdjoint(AdjointParams(n=n, nsteps=10, dt=0.01, gravity=1.0, precision=prec, checkpoint_every=4,
                                         pair_factor=0.0), np_)
        a.set_field(u)
        a.set_droplets(x0, tau, np.full(np_, 1e-6))
        loss, _ = a.forward()
        out[prec] = (np.array([loss]), *a.final_state(), *a.backward())
        a.close()
    for p, q in zip(out["mixed"], out["fp64"]):
        assert rel(p, q) < 2e-5


@pytest.mark.parametrize("np_", [1, 8, 33])
def test_recomputation_repeats_the_forward_pass(np_):
    """Mixed: the reverse sweep runs along the trajectory that the forward pass took, bit for
    bit.  All droplets sit half-way between two x planes whose six neighbours' weighted values
    cancel, so the velocity they see is rounding alone (1e-7 of the field) and another order
    of the sum gives another velocity.  One step from rest without gravity gives V = 24 d U /
    (1 + 9 d), d = dt / 24 tau, and a displacement s = 9 dt V / 24; the gradient of the mean
    of s^2 by tau is then -2 s^2 / (np tau (1 + 9 d)) with the s of the forward pass, if both
    passes had the same U.  About 20 FP32 roundings lie between: 1e-5."""
    n, m, dt = 16, 5, 0.1
    rng = np.random.default_rng(np_)
    w = np.array([3.0, -25.0, 150.0, 150.0, -25.0, 3.0]) / 256.0   # 6-point weights at 1/2
    line = np.zeros(n)
    line[m - 2:m + 4] = rng.uniform(0.5, 1.5, 6)
    line[m + 3] = -(w[:5] @ line[m - 2:m + 3]) / w[5]
    u = 1e4 * rng.uniform(0.5, 1.5, (3, n, n, 1)) * line
    dx = 2 * np.pi / n
    x0 = np.stack([np.full(np_, (m + 0.5) * dx), *rng.uniform(0.0, 2 * np.pi, (2, np_))], axis=1)
    tau = rng.uniform(0.05, 0.2, np_)
    a = DropletAdjoint(AdjointParams(n=n, nsteps=1, dt=dt, gravity=0.0, precision="mixed", pair_factor=0.0), np_)
    a.set_field(u)
    a.set_droplets(x0, tau, np.full(np_, 1e-6))
    a.forward()
    s2 = ((a.final_state()[0] - x0) ** 2).sum(axis=1)
    dtau = a.backward()[1]
    assert (s2 > 0.0).all()
    assert np.allclose(dtau, -2.0 * s2 / (np_ * tau * (1.0 + 9.0 * dt / (24.0 * tau))), rtol=1e-5, atol=0.0)
    a.close()


def test_droplets_partly_on_the_host_are_refused():
    """Device positions with host drag times: an error, and the droplets set before stay."""
    import torch
    u, x0, tau, rad = clustered_case()
    a = gpu_problem("fp64", u=u, x0=x0, tau=tau, rad=rad)
    loss, _ = a.forward()
    for q in (1, 2):
        args = [torch.from_numpy(x0 + 0.5).cuda(), torch.from_numpy(tau).cuda(), torch.from_numpy(rad).cuda()]
        args[q] = (x0, tau, rad)[q]
        with pytest.raises(DropletError):
            a.set_droplets(*args)
    assert a.forward()[0] == loss
    a.close()


@pytest.mark.parametrize("seed", [0, 1])
def test_mixed_velocity_takes_no_rounding_per_step(seed):
    """Mixed: the droplet velocity after 100 steps of slow drag is as far from FP64 as one
    interpolation and one stored FP32 value round, about 1e-7, and not as 100 updates in FP32
    do (1e-6 and more here); 3e-7 lies between."""
    rng = np.random.default_rng(seed)
    n, np_ = 16, 300
    x = np.arange(n) * (2 * np.pi / n)
    Z, Y, X = np.meshgrid(x, x, x, indexing="ij")
    u = np.stack([sum(rng.standard_normal() * np.cos(k[0] * X + k[1] * Y + k[2] * Z + rng.uniform(0, 6.28))
                      for k in rng.integers(-3, 4, (8, 3))) for _ in range(3)])
    x0, tau = rng.uniform(0, 2 * np.pi, (np_, 3)), rng.uniform(1.0, 3.0, np_)
    v = {}
    for prec in ("fp64", "mixed"):
        a = DropletAdjoint(AdjointParams(n=n, nsteps=100, dt=0.01, gravity=1.0, precision=prec,
                                         checkpoint_every=100, pair_factor=0.0), np_)
        a.set_field(u)
        a.set_droplets(x0, tau, np.full(np_, 1e-6))
        a.forward()
        v[prec] = a.final_state()[1]
        a.close()
    assert np.linalg.norm(v["mixed"] - v["fp64"]) < 3e-7 * np.linalg.norm(v["fp64"])
