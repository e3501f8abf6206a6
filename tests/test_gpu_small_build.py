"""The one-block sort (up to 4096 particles) and numbering (up to 2048) of
small systems, around their limits and with partly filled warps: FP64 forces
and node counts bit for bit against the oracle, ensembles against their systems
on their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _particles(shape, n):
    from nbb import ics

    p = ics.plummer(n, seed=9)
    if shape == "one point":  # one leaf
        for a in (p.x, p.y, p.z):
            a[:] = 0.5
    elif shape == "pairs":  # chains of cells with one child, leaves of many particles
        for a in (p.x, p.y, p.z):
            a[: n // 2] = a[0]
            a[n // 2:] = a[0] + 1e-3
        p.x[0] += 50.0
    return p


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097])
@pytest.mark.parametrize("shape", ["plummer", "one point", "pairs"])
def test_small_build(nbb_mod, oracle, shape, n):
    p = _particles(shape, n)
    ax, ay, az, st = nbb_mod.compute_accelerations(p, 0.6, 0.05, 1.0, stats=True)
    ref = oracle.pipeline(p.mass, p.x, p.y, p.z, theta=0.6, soft=0.05, g=1.0)
    assert st.interactions == ref["interactions"]
    for a, k in ((ax, "ax"), (ay, "ay"), (az, "az")):
        assert np.array_equal(a, ref[k]), (k, float(np.max(np.abs(a - ref[k]))))


@pytest.mark.parametrize("sizes", [(1, 2, 40, 980, 1), (700, 1348), (1000, 1049), (5, 1500, 2591), (3, 4094)])
def test_small_ensemble(nbb_mod, sizes):
    from nbb import ics

    parts = [ics.plummer(k, seed=20 + i) for i, k in enumerate(sizes)]
    ens = ics.Ensemble(ics.ParticleData(*[np.concatenate(a) for a in zip(*[q.arrays() for q in parts])]),
                       np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64), np.full(len(sizes), 0.03))
    for prec in (nbb_mod.PRECISION_FP64, nbb_mod.PRECISION_MIXED):
        cfg = nbb_mod.SimulationConfig(1e-3, 0.5, 0.03, 1.0, precision=prec, group_size=32 if prec else 0)
        sim = nbb_mod.EnsembleSimulation(ens, cfg)
        sim.initialize()
        acc = np.stack(sim.accelerations())
        sim.close()
        at = 0
        for q in parts:
            one = nbb_mod.Simulation(q, cfg)
            one.initialize()
            ref = np.stack(one.accelerations())
            one.close()
            got = acc[:, at: at + len(q)]
            at += len(q)
            if prec == nbb_mod.PRECISION_FP64:
                assert np.array_equal(got, ref)
            else:  # the same interactions, batched from other list positions: FP32 sums of at most 96 terms
                assert np.max(np.abs(got - ref)) <= 96 * 2.0 ** -24 * np.max(np.linalg.norm(ref, axis=0))


@pytest.mark.parametrize("sizes", [(33,), (40,) * 40, (32, 33) * 20, (400, 1, 3, 50, 399, 4, 5, 6, 200, 2), (1000, 31, 500, 260, 130, 70, 35, 9, 1),
                                   (100,) * 40, (1500,) + (40,) * 31, (3000, 1500, 700, 90, 45, 33, 32) + (8,) * 30, (1000,) * 33])
def test_large_leaves(nbb_mod, oracle, sizes):
    """Leaves of many particles, summed by a thread each or by their warp: one
    large leaf, many alike and mixed ones, below and above the one-block build."""
    from nbb import ics

    rng = np.random.default_rng(13)
    x = np.repeat(rng.uniform(-1.0, 1.0, (3, len(sizes))), sizes, axis=1) + rng.uniform(-1e-9, 1e-9, (3, sum(sizes)))
    z = np.zeros(x.shape[1])
    p = ics.ParticleData(rng.uniform(0.5, 1.0, x.shape[1]), *[np.ascontiguousarray(a) for a in x], z, z, z)
    ax, ay, az, st = nbb_mod.compute_accelerations(p, 0.8, 0.05, 1.0, stats=True)
    ref = oracle.pipeline(p.mass, p.x, p.y, p.z, theta=0.8, soft=0.05, g=1.0)
    assert st.interactions == ref["interactions"]
    for a, k in ((ax, "ax"), (ay, "ay"), (az, "az")):
        assert np.array_equal(a, ref[k]), (k, float(np.max(np.abs(a - ref[k]))))
