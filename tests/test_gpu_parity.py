"""GPU parity: libdroplet.so (sm_100a) against the FP64 CPU oracle on identical seeded
inputs, through the C ABI.

Bars: the FP64 path is bit-identical to the oracle for positions, velocities, histories
and interpolated velocities (same operations, same order, no FMA contraction); pair
lists, removal lists and integer histogram counts are bit-exact in both precisions on
identical inputs; floating-point histogram sums (accumulated with device atomics in a
different order) agree to 1e-10 relative in FP64; the mixed path's interpolated velocity
has relative L2 error < 1e-5 against FP64.
"""
import numpy as np
import pytest

import oracle as orc
from cases import config0_params, dense_params, random_field, smooth_field
from mpi_2d_domain_decomp_turb_particles_b200 import Partlib

pytestmark = pytest.mark.gpu

HIST_NAMES = ("wrbin", "wxbin", "wybin", "wzbin", "urbin", "thetabin", "wrtanbin")


def make(p):
    g = Partlib(p)
    g.part_init()
    o = orc.Oracle(**p.oracle_kwargs())
    o.part_init()
    return g, o


def live_state(yp, fvp, fdp):
    """Positions/velocities and the history levels that are live between steps."""
    return np.concatenate([yp[:, :8], fvp[:, 1:3].reshape(len(yp), -1), fdp[:, 1:4].reshape(len(yp), -1)], 1)


def oracle_state(o):
    n = o.nps
    return live_state(o.yp[:n], o.fvp[:n], o.fdp[:n])


def gpu_state(g):
    s = g.get_particles()
    return live_state(s["yp"], s["fvp"], s["fdp"])


def pair_set(rows, ncol_type):
    return sorted(tuple(int(v) for v in r) for r in rows[:, list(ncol_type)])


def gpu_step_separate(g, dist, nonoverlap):
    """turb.f90:553-610 through the separate C-ABI entry points."""
    g.prepare_interp()
    for k in (1, 2, 3):
        g.interpolate(None, k)
    g.part_history_fvp()
    g.headlist(dist)
    g.part_history_fdp()
    g.part_advance()
    g.complete_ypn()
    rep = g.collision_det()
    g.update_part_position()
    if nonoverlap and rep.ncoll > 0:
        g.relocate()
    g.periodic()
    if nonoverlap:
        g.overlap_det()
    return rep


# ------------------------------------------------------------------------------------
def test_part_init_positions_and_scalars_match():
    for prec in ("fp64", "mixed"):
        g, o = make(dense_params(npart=3000, precision=prec))
        s = g.scalars()
        assert s.radmax == o.getd("radmax") and s.d_coll == o.getd("d_coll")
        assert s.sv_const == o.getd("sv_const") and s.tau_cloud_const2 == o.getd("tau_cloud_const2")
        yp = g.get_particles()["yp"]
        assert np.array_equal(yp[:, [0, 1, 2, 6, 7]], o.yp[:o.nps][:, [0, 1, 2, 6, 7]])
        g.close()


def test_prepare_interp_weights_bitexact():
    g, o = make(dense_params(npart=4000))
    g.prepare_interp()
    o.prepare_interp()
    lh, bg = g.interp_weights()
    n = o.nps
    assert np.array_equal(lh.T, o.lhnode[:, :n])
    assert np.array_equal(bg.transpose(1, 2, 0), o.bg[:, :, :n])


@pytest.mark.parametrize("field", ["smooth", "random"])
def test_interpolate_fp64_bitexact(field):
    n = 32
    g, o = make(dense_params(n=n, npart=5000))
    f = smooth_field(n) if field == "smooth" else random_field(n)
    o.prepare_interp()
    g.prepare_interp()
    for k in range(3):
        o.interpolate(f[k], k + 1)
        g.interpolate(f[k], k + 1)
    vp = g.get_particles()["vp"]
    assert np.array_equal(vp, o.vp[:o.nps])


def test_interpolate_mixed_relative_error():
    n = 64
    g, o = make(config0_params(precision="mixed"))
    f = smooth_field(n)
    o.prepare_interp()
    g.prepare_interp()
    for k in range(3):
        o.interpolate(f[k], k + 1)
        g.interpolate(f[k], k + 1)
    vp = g.get_particles()["vp"]
    ref = o.vp[:o.nps]
    rel = np.linalg.norm(vp - ref) / np.linalg.norm(ref)
    assert rel < 1e-5, rel


def test_fused_update_step_fp64_bitexact_over_steps():
    n = 32
    g, o = make(dense_params(n=n, npart=5000))
    f = smooth_field(n)
    g.set_fields(*f)
    for step in range(12):
        g.update_step()
        o.update_step(*f)
        o.periodic()
    assert g.nps == o.nps
    assert np.array_equal(gpu_state(g), oracle_state(o))


def _compare_collision(g, o, rep, exact_sums):
    assert rep.icc[:] == o.arr("icc", np.int32).tolist()
    assert rep.ncoll == o.geti("ncoll")
    assert np.array_equal(g.removal_list(), o.removepart())
    gp = g.pairs()                                  # (ih1, src2, jid2, type)
    op = o.pairs()                                  # (ih1, ih2, src2, jid2, type)
    assert pair_set(gp, (0, 1, 2, 3)) == pair_set(op, (0, 2, 3, 4))
    # collist in the reference's detection order
    cl = g.collist()
    ocl = o.arr("collist").reshape(-1, 20)[:o.geti("ntotpair")]
    assert np.array_equal(cl[:, [8, 18]], ocl[:, [8, 18]])
    ct, nir = g.collision_counts()
    nset = o.geti("nset")
    assert np.array_equal(ct.T.ravel(), o.arr("colltype", np.int32))
    assert np.array_equal(nir.T.ravel(), o.arr("nir", np.int32))
    # contact-shell records in the reference's detection order (the Vp*.dat line order)
    ids, rec = g.contacts()
    oc = o.contacts()
    assert ids.tolist() == [[c[0], c[1], c[2]] for c in oc]
    orec = np.array([c[3] for c in oc]).reshape(-1, 12)
    if exact_sums:
        assert np.array_equal(rec, orec)
    else:
        assert np.array_equal(rec[:, :2], orec[:, :2])


def test_particle_steps_separate_calls_fp64_match_oracle():
    n = 32
    p = dense_params(n=n, npart=6000)
    g, o = make(p)
    f = smooth_field(n)
    g.set_fields(*f)
    d = g.scalars().d_coll
    total_pairs = 0
    for step in range(1, 11):
        g.set_step(step, 0.0)
        rep = gpu_step_separate(g, d, False)
        o_out = o.particle_step(*f)
        total_pairs += len(o_out["pairs"])
        _compare_collision(g, o, rep, True)
        assert np.array_equal(gpu_state(g), oracle_state(o)), f"step {step}"
        if step % 5 == 4:
            h = g.histograms(written=True)
            assert np.array_equal(h["nirbin"], o.hist("out_nirbin"))
            for nm in HIST_NAMES:
                assert np.allclose(h[nm], o.hist("out_" + nm), rtol=1e-10, atol=1e-12), nm
    assert total_pairs > 0


def test_fused_particle_step_fp64_match_oracle():
    n = 32
    p = dense_params(n=n, npart=6000)
    g, o = make(p)
    f = smooth_field(n)
    g.set_fields(*f)
    for step in range(1, 11):
        rep, _ = g.particle_step()
        o.particle_step(*f)
        _compare_collision(g, o, rep, True)
        assert np.array_equal(gpu_state(g), oracle_state(o)), f"step {step}"


def test_nonoverlap_relocation_and_overlap_det_match_oracle():
    n = 32
    p = dense_params(n=n, npart=6000, nonoverlap=True)
    g, o = make(p)
    f = smooth_field(n)
    g.set_fields(*f)
    # PART_INIT is followed by PERIODIC and OVERLAP_DET (turb.f90:426-429)
    g.periodic(); g.overlap_det()
    o.periodic(); o.overlap_det()
    assert np.array_equal(gpu_state(g), oracle_state(o))
    relocated = 0
    for step in range(1, 9):
        rep, _ = g.particle_step()
        oo = o.particle_step(*f)
        relocated += rep.ncoll
        _compare_collision(g, o, rep, True)
        assert np.array_equal(gpu_state(g), oracle_state(o)), f"step {step}"
    assert relocated > 0


def test_mixed_pairs_bitexact_on_identical_inputs():
    """Mixed-precision state after PART_ADVANCE, fed to the FP64 oracle: same pairs."""
    n = 32
    p = dense_params(n=n, npart=6000, precision="mixed")
    g, o = make(p)
    f = smooth_field(n)
    g.set_fields(*f)
    d = g.scalars().d_coll
    for step in range(1, 7):
        g.set_step(step, 0.0)
        g.prepare_interp()
        for k in (1, 2, 3):
            g.interpolate(None, k)
        g.part_history_fvp()
        g.headlist(d)
        g.part_history_fdp()
        g.part_advance()
        g.complete_ypn()
        rep = g.collision_det()
        s = g.get_particles()
        # load the identical snapshot into the oracle and detect there
        m = s["yp"].shape[0]
        o.nps = m
        o.yp[:m] = s["yp"]
        o.fvp[:m] = s["fvp"]
        o.dmove[:m] = s["dmove"]
        o.vp[:m] = s["vp"]
        o.seti("istep", step)
        o.headlist(d)
        o.complete_ypn()
        o.collision_det()
        _compare_collision(g, o, rep, False)
        assert np.array_equal(g.histograms(written=False)["nirbin"], o.hist("nirbin"))
        g.update_part_position()
        g.periodic()


def test_mixed_trajectories_close_to_fp64():
    n = 64
    g, o = make(config0_params(precision="mixed"))
    f = smooth_field(n)
    g.set_fields(*f)
    for _ in range(10):
        g.update_step()
        o.update_step(*f)
        o.periodic()
    s = g.get_particles()
    m = o.nps
    ref = o.yp[:m]
    vrel = np.linalg.norm(s["yp"][:, 3:6] - ref[:, 3:6]) / np.linalg.norm(ref[:, 3:6])
    assert vrel < 1e-5, vrel
    # FP32 velocities: ~1e-7 relative per step on displacements of ~1e-3
    assert np.abs(s["yp"][:, :3] - ref[:, :3]).max() < 1e-7


@pytest.mark.parametrize("radii", [[20.0, 30.0], [10.0, 15.0, 20.0, 25.0, 30.0, 35.0, 40.0]])
def test_mean_vel_matches_oracle(radii):
    """Two sets (one pass of the per-set sums) and seven sets (two passes)."""
    n = 32
    g, o = make(dense_params(n=n, npart=4000, radius_um=radii))
    f = smooth_field(n)
    g.set_fields(*f)
    for _ in range(3):
        g.update_step()
        o.update_step(*f)
        o.periodic()
    assert np.allclose(g.mean_vel(), o.mean_vel(), rtol=1e-12, atol=1e-14)
    for _ in range(2):   # repeated calls: the same sums, bit for bit
        assert np.array_equal(g.mean_vel(), g.mean_vel())


def test_device_resort_is_invisible():
    n = 32
    f = smooth_field(n)
    states = []
    for interval in (1, 1000):
        p = dense_params(n=n, npart=5000, resort_interval=interval)
        g = Partlib(p)
        g.part_init()
        g.set_fields(*f)
        for _ in range(6):
            g.particle_step()
        states.append(gpu_state(g))
        g.close()
    assert np.array_equal(states[0], states[1])


def test_periodic_reorder_matches_oracle():
    n = 32
    p = dense_params(n=n, npart=2000)
    g, o = make(p)
    rng = np.random.default_rng(11)
    yp = o.yp[:o.nps].copy()
    pi2 = o.getd("pi2")
    k = rng.choice(o.nps, 300, replace=False)
    yp[k, 1] += rng.choice([-1.0, 1.0], 300) * pi2 * 0.51 * rng.integers(0, 2, 300)
    yp[k, 2] += rng.choice([-1.0, 1.0], 300) * pi2 * 0.51 * rng.integers(0, 2, 300)
    o.yp[:o.nps] = yp
    g.set_particles(yp)
    o.periodic()
    g.periodic()
    assert np.array_equal(g.get_particles()["yp"], o.yp[:o.nps])


def test_coalescence_growth_mode_matches_oracle():
    """Past nstep_grow (turb.f90:588-590) collided pairs merge (COALESCE) instead of being
    relocated: FP64 state, droplet count and merged radii identical to the oracle."""
    n = 32
    p = dense_params(n=n, npart=6000, nonoverlap=True)
    g, o = make(p)
    f = smooth_field(n)
    g.set_fields(*f)
    g.periodic(); g.overlap_det()
    o.periodic(); o.overlap_det()
    g.set_step(39998, 0.0)
    o.seti("istep", 39998)
    merged = 0
    mass0 = np.sum(g.get_particles()["yp"][:, 6] ** 3)
    for step in range(8):
        n0 = g.nps
        rep, _ = g.particle_step()
        o.particle_step(*f)
        merged += n0 - g.nps
        assert g.nps == o.nps, f"step {step}"
        assert np.array_equal(gpu_state(g), oracle_state(o)), f"step {step}"
    assert merged > 0
    # COALESCE conserves droplet mass: a^3 = a1^3 + a2^3 (partlib.f90:3684)
    assert abs(np.sum(g.get_particles()["yp"][:, 6] ** 3) - mass0) <= 1e-12 * mass0


@pytest.mark.parametrize("n,pad", [(13, 2), (32, 0), (37, 5), (70, 2), (130, 1), (260, 2)])
def test_field_conversion_at_ragged_sizes(n, pad):
    """The padded copy of a field (rows shorter and longer than a block's threads, odd row
    pitches, periodic images in x, y and z): INTERPOLATE equals the oracle bit for bit for
    droplets all over the box and at its faces."""
    p = dense_params(n=n, npart=400)
    g, o = Partlib(p), orc.Oracle(**p.oracle_kwargs())
    g.part_init()
    o.part_init()
    rng = np.random.default_rng(n)
    yp = g.get_particles()["yp"]
    yp[:200, :3] = rng.choice([0.0, 1e-9, 2 * np.pi - 1e-9], (200, 3))
    g.set_particles(yp)
    o.yp[:400] = yp
    g.prepare_interp()
    o.prepare_interp()
    for k in range(3):
        v = rng.standard_normal((n, n, n + pad))
        g.interpolate(v, k + 1)
        o.interpolate(v, k + 1)
    assert np.array_equal(g.get_particles()["vp"], o.vp[:400])
    g.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8])
def test_field_conversion_on_grids_narrower_than_the_halo(n, precision):
    """Below n = 8 a column has periodic images on both sides of the padded row, and at n = 3,
    the smallest grid PART_INIT takes, some planes are two periods away.  FP64 bit for bit; mixed within 1e-5 of the largest field value: about 30 FP32 roundings (6e-8) of the
    field, the three weights and the sums, times the weights' absolute sum, at most 1.4 per
    direction and 2.7 for the three."""
    p = dense_params(n=n, npart=400, precision=precision)
    g, o = Partlib(p), orc.Oracle(**p.oracle_kwargs())
    g.part_init()
    o.part_init()
    rng = np.random.default_rng(n)
    yp = g.get_particles()["yp"]
    yp[:200, :3] = rng.choice([0.0, 1e-9, 2 * np.pi - 1e-9], (200, 3))
    g.set_particles(yp)
    o.yp[:400] = yp
    g.prepare_interp()
    o.prepare_interp()
    for k in range(3):
        v = rng.standard_normal((n, n, n + 2))
        g.interpolate(v, k + 1)
        o.interpolate(v, k + 1)
        err = np.abs(g.get_particles()["vp"][:, k] - o.vp[:400, k]).max()
        assert err == 0.0 if precision == "fp64" else err < 1e-5 * np.abs(v).max()
    g.close()
