"""Both sides of the size rules of the mixed walk, the FP64 adjoint and the
rollout's buffers, against direct summation or a fresh simulation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 39999, 40000])
def test_mixed_walk_split(nbb_mod, n):
    """Four warps to a target group below 40000 particles, one above.  With
    theta = 0 the list holds every particle; an FP32 sum of at most 96 terms,
    each with a relative error of at most 16 roundings, is within (96 + 16)
    2^-24 of the terms' magnitudes."""
    from nbb import ics

    p = ics.plummer(n, seed=4)
    soft = 0.02
    sim = nbb_mod.Simulation(p, nbb_mod.SimulationConfig(1e-3, 0.0, soft, 1.0, group_size=32,
                                                         precision=nbb_mod.PRECISION_MIXED))
    sim.initialize()
    acc = np.stack(sim.accelerations())
    sim.close()
    x = np.stack([p.x, p.y, p.z])
    for i in np.random.default_rng(1).choice(n, min(n, 128), replace=False):
        d = x - x[:, i:i + 1]
        term = p.mass * (np.sum(d * d, axis=0) + soft * soft) ** -1.5 * d
        assert np.all(np.abs(acc[:, i] - term.sum(axis=1)) <= 112 * 2.0 ** -24 * np.abs(term).sum(axis=1).max())


@pytest.mark.parametrize("n", [7, 32767, 32768])
def test_fp64_adjoint_targets(nbb_mod, n):
    """Eight targets to a warp below 32768 particles, 32 above: theta = 0
    against the direct-summation adjoint; the two add n terms in different
    orders (n 2^-52 of the largest, with a factor of 16)."""
    from nbb import ics

    p = ics.plummer(n, seed=6)
    gp = np.random.default_rng(2).standard_normal((3, n)) / n
    cfg = nbb_mod.SimulationConfig(1e-3, 0.0, 0.05, 1.0)
    sim = nbb_mod.Simulation(p, cfg)
    sim.initialize()
    sim.rollout(1, 1)
    got = sim.backward(gp, gp)
    sim.close()
    ref = nbb_mod.direct_rollout_adjoint(p, cfg, 1, gp, gp)[1:]
    for a, b in zip(got, ref):
        assert np.max(np.abs(a - b)) <= 16 * n * 2.0 ** -52 * np.max(np.abs(b)) + 1e-18


@pytest.mark.parametrize("lengths", [(3, 7), (7, 3), (4, 4)])
def test_rollout_buffers(nbb_mod, lengths):
    """A second rollout, shorter, longer or alike, in the first one's buffers
    gives what it gives in new ones (the adjoint's atomics may add in another
    order)."""
    from nbb import ics

    n = 3000
    p = ics.plummer(n, seed=7)
    gp = np.random.default_rng(3).standard_normal((3, n)) / n
    cfg = nbb_mod.SimulationConfig(1e-3, 0.5, 0.05, 1.0)
    used, fresh = nbb_mod.Simulation(p, cfg), nbb_mod.Simulation(p, cfg)
    used.initialize()
    fresh.initialize()
    used.rollout(lengths[0], 2)
    used.backward(gp, gp)
    fresh.run(lengths[0])
    for sim in (used, fresh):
        sim.rollout(lengths[1], 2)
    got, ref = used.backward(gp, gp), fresh.backward(gp, gp)
    used.close()
    fresh.close()
    for a, b in zip(got, ref):
        assert np.max(np.abs(a - b)) <= 16 * n * 2.0 ** -52 * np.max(np.abs(b))


@pytest.mark.parametrize("n", [2, 7, 8, 9, 31, 33, 65])
@pytest.mark.parametrize("soft", [0.0, 0.05])
def test_mixed_adjoint_blocks(nbb_mod, n, soft):
    """Lists that end inside a block of eight entries, without softening and
    with zero masses: theta = 0 against the direct-summation adjoint in FP64.
    64 roundings of FP32 in each of n terms; a lost or doubled entry is of the
    order of the gradient itself."""
    from nbb import ics

    p = ics.plummer(n, seed=8)
    p.mass[n // 2:n // 2 + n // 5] = 0.0
    gp = np.random.default_rng(5).standard_normal((3, n)) / n
    cfg = nbb_mod.SimulationConfig(1e-3, 0.0, soft, 1.0, precision=nbb_mod.PRECISION_MIXED, group_size=32)
    sim = nbb_mod.Simulation(p, cfg)
    sim.initialize()
    sim.rollout(1, 1)
    got = sim.backward(gp, gp)
    sim.close()
    ref = nbb_mod.direct_rollout_adjoint(p, nbb_mod.SimulationConfig(1e-3, 0.0, soft, 1.0), 1, gp, gp)[1:]
    heavy = p.mass > 0.0
    for a, b in zip(got, ref):
        a, b = a[..., heavy], b[..., heavy]
        assert np.max(np.abs(a - b)) <= 64 * n * 2.0 ** -24 * np.max(np.abs(b))


@pytest.mark.parametrize("n,total", [(2, 1.0), (33, 1.0), (33, 33.0), (65, 1.0), (1000, 1.0), (1000, 1000.0), (40001, 1.0)])
@pytest.mark.parametrize("soft", [1e-9, 2e-8])
def test_mixed_adjoint_small_softening(nbb_mod, n, total, soft):
    """A softening whose m eps^-5 overflows in FP32 and target groups with idle
    lanes: finite gradients, and those of the direct-summation adjoint as in the
    test above, each term with at most 64 roundings (a batch's sum and the
    offset's, which weighs by the group's extent over the pair's distance, up
    to 128 here)."""
    from nbb import ics

    p = ics.plummer(n, seed=8, total_mass=total)
    gp = np.random.default_rng(5).standard_normal((3, n)) / n
    cfg = nbb_mod.SimulationConfig(1e-3, 0.0, soft, 1.0, precision=nbb_mod.PRECISION_MIXED, group_size=32)
    sim = nbb_mod.Simulation(p, cfg)
    sim.initialize()
    sim.rollout(1, 1)
    got = sim.backward(gp, gp)
    sim.close()
    ref = nbb_mod.direct_rollout_adjoint(p, nbb_mod.SimulationConfig(1e-3, 0.0, soft, 1.0), 1, gp, gp)[1:]
    for a, b in zip(got, ref):
        assert np.all(np.isfinite(a))
        assert np.max(np.abs(a - b)) <= 64 * min(n, 128) * 2.0 ** -24 * np.max(np.abs(b))


@pytest.mark.parametrize("extra,group", [(0, 32), (40000, 32), (0, 64), (0, 128)])
def test_mixed_batch_sum(nbb_mod, extra, group):
    """Plain FP32 sums run over 64 entries in two chains before they are added
    with compensation.  One heavy source and then 95 whose terms are 0.49 ulp
    of its own: at most the 31 later terms of its chain are lost, and one from
    adding the two chains (a batch of 96 entries loses 47)."""
    from nbb import ics

    k = 96
    n = k + 1 + extra
    rng = np.random.default_rng(12)
    x = np.full((3, n), -1.0)  # the sources: one leaf, in this order
    x[0, k] = -0.25            # the target
    x[:, k + 1:] = rng.uniform(0.2, 1.0, (3, extra))  # without mass, in cells of their own

    def accel(m):
        mass = np.zeros(n)
        mass[0], mass[1:k] = 1.0, m
        z = np.zeros(n)
        p = ics.ParticleData(mass, x[0].copy(), x[1].copy(), x[2].copy(), z, z, z)
        sim = nbb_mod.Simulation(p, nbb_mod.SimulationConfig(1e-3, 0.5, 0.01, 1.0, group_size=group,
                                                             precision=nbb_mod.PRECISION_MIXED))
        sim.initialize()
        a = np.stack(sim.accelerations())[0, k]
        sim.close()
        return a

    one = accel(0.0)
    m = 0.49 * float(np.spacing(np.float32(abs(one)))) / abs(one)
    kept = (accel(m) - one) / (m * one)
    assert 95 - 32 - 1 <= kept <= 95 + 1


@pytest.mark.parametrize("n", [50, 1000, 45001])
@pytest.mark.parametrize("group", [0, 32, 64, 128])
def test_mixed_no_softening(nbb_mod, n, group):
    """Groups that fill only some of a lane's target slots, without softening:
    theta = 0 against direct summation (as in test_mixed_walk_split; a close
    pair's offset weighs by the group's extent over the distance, up to 64
    here), and a pair in one place is still singular."""
    from nbb import ics

    p = ics.plummer(n, seed=10)
    cfg = nbb_mod.SimulationConfig(1e-3, 0.0, 0.0, 1.0, group_size=group, precision=nbb_mod.PRECISION_MIXED)
    sim = nbb_mod.Simulation(p, cfg)
    sim.initialize()
    acc = np.stack(sim.accelerations())
    sim.close()
    x = np.stack([p.x, p.y, p.z])
    for i in np.random.default_rng(1).choice(n, min(n, 128), replace=False):
        d = x - x[:, i:i + 1]
        r2 = np.sum(d * d, axis=0)
        r2[i] = 1.0
        term = p.mass * r2 ** -1.5 * d
        assert np.all(np.abs(acc[:, i] - term.sum(axis=1)) <= 64 * 80 * 2.0 ** -24 * np.abs(term).sum(axis=1).max())
    for a in (p.x, p.y, p.z):
        a[n - 1] = a[0]
    sim = nbb_mod.Simulation(p, cfg)
    with pytest.raises(nbb_mod.DeviceError, match="Singular"):
        sim.initialize()
    sim.close()


@pytest.mark.parametrize("systems", [12, 13])
def test_mixed_ensemble_split(nbb_mod, systems):
    """Up to 12 systems four warps take a target group, above it one: forces and
    gradients of an ensemble (theta = 0) against each system's direct sums, as
    in the tests of single systems above."""
    from nbb import ics

    size = 70
    n = size * systems
    parts = [ics.plummer(size, seed=30 + k) for k in range(systems)]
    p = ics.ParticleData(*(np.concatenate(a) for a in zip(*[q.arrays() for q in parts])))
    ens = ics.Ensemble(p, np.arange(systems + 1, dtype=np.int64) * size, np.full(systems, 0.02))
    cfg = nbb_mod.SimulationConfig(1e-3, 0.0, 0.02, 1.0, precision=nbb_mod.PRECISION_MIXED, group_size=32)
    gp = np.random.default_rng(5).standard_normal((3, n)) / size
    sim = nbb_mod.EnsembleSimulation(ens, cfg)
    sim.initialize()
    acc = np.stack(sim.accelerations())
    sim.rollout(1, 1)
    got = sim.backward(gp, gp)
    sim.close()
    one = nbb_mod.SimulationConfig(1e-3, 0.0, 0.02, 1.0)
    for k, q in enumerate(parts):
        at = slice(k * size, (k + 1) * size)
        ref = np.stack(nbb_mod.compute_accelerations(q, 0.0, 0.02, 1.0))
        assert np.max(np.abs(acc[:, at] - ref)) <= 64 * size * 2.0 ** -24 * np.max(np.abs(ref))
        grads = nbb_mod.direct_rollout_adjoint(q, one, 1, gp[:, at], gp[:, at])[1:]
        for a, b in zip(got, grads):
            assert np.max(np.abs(a[..., at] - b)) <= 64 * size * 2.0 ** -24 * np.max(np.abs(b))
