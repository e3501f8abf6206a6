"""The plain FP64 walk on its ordered interaction lists, at the sizes and
shapes where a list can go wrong, bit for bit against the oracle (which
evaluates every target on its own in the reference's order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _particles(shape, n):
    from nbb import ics

    p = ics.plummer(n, seed=5)
    if shape == "coincident":  # one leaf of many particles, listed in parts
        k = n // 3
        for a in (p.x, p.y, p.z):
            a[:k] = a[0]
        p.x[:k] += 1e-9 * np.arange(k)
    elif shape == "two clusters":  # a warp's targets far apart
        p.x[n // 2:] += 1000.0
    elif shape == "zero masses":
        p.mass[::3] = 0.0
        p.mass[n // 4: n // 2] = 0.0
    elif shape == "line":
        p.y[:] = 0.0
        p.z[:] = 0.0
    return p


def _check(nbb, oracle, p, theta, soft, g=1.0):
    ax, ay, az, st = nbb.compute_accelerations(p, theta, soft, g, stats=True)
    ref = oracle.pipeline(p.mass, p.x, p.y, p.z, theta=theta, soft=soft, g=g)
    if np.all(p.mass > 0.0):  # the library does not count a zero-mass particle, the oracle does
        assert st.interactions == ref["interactions"]
    for a, k in ((ax, "ax"), (ay, "ay"), (az, "az")):
        assert np.array_equal(a, ref[k]), (k, float(np.max(np.abs(a - ref[k]))))


# one target to a set below 5000 particles, 32 above; two warps to a set below
# 65536; target groups of up to 32 below 131072, of up to 128 cut into 32 above
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 97, 1025, 4999, 5000, 8191, 8192, 65535, 65536, 131071, 131072])
def test_sizes(nbb_mod, oracle, n):
    _check(nbb_mod, oracle, _particles("plummer", n), 0.5, 0.01)


@pytest.mark.parametrize("n", [900, 9001])
@pytest.mark.parametrize("shape", ["coincident", "two clusters", "zero masses", "line"])
@pytest.mark.parametrize("theta", [0.0, 0.7, 3.0])
def test_shapes(nbb_mod, oracle, shape, n, theta):
    _check(nbb_mod, oracle, _particles(shape, n), theta, 0.02)


@pytest.mark.parametrize("n", [900, 9001])
@pytest.mark.parametrize("unit", [1e-90, 1e-30, 1e21, 1e90])  # past 1e-100 the force itself overflows
def test_units_of_length(nbb_mod, oracle, n, unit):
    """The box tests run in FP32 in units of the bounding box; the terms'
    short square root covers part of the range of FP64."""
    p = _particles("plummer", n)
    for a in (p.x, p.y, p.z):
        a *= unit
    _check(nbb_mod, oracle, p, 0.6, 0.01 * unit)


def test_rounding_exception(nbb_mod, oracle):
    """d^2 + eps^2 = 4 - 2^-51: the one significand whose reciprocal square
    root the short sequence would round the wrong way."""
    from nbb import ics

    h = 2.0 ** -26
    z = np.zeros(2)
    p = ics.ParticleData(np.array([1.0, 3.0]), np.array([0.0, h]), np.array([0.0, h]), z, z, z, z)
    soft = 2.0 - 2.0 ** -52
    x = np.float64(2.0 ** -51 + soft * soft)
    assert x == 4.0 - 2.0 ** -51
    _check(nbb_mod, oracle, p, 0.5, soft)
    inv = 1.0 / np.sqrt(x)
    assert nbb_mod.compute_accelerations(p, 0.5, soft, 1.0)[0][1] == -((inv * inv) * inv) * h


@pytest.mark.parametrize("n", [900, 9001, 65537])
@pytest.mark.parametrize("shape", ["plummer", "coincident", "zero masses"])
def test_no_softening(nbb_mod, oracle, shape, n):
    """Without softening every term's range is looked at on its own."""
    _check(nbb_mod, oracle, _particles(shape, n), 0.6, 0.0)


@pytest.mark.parametrize("n", [900, 9001, 65537])
def test_singular_pair(nbb_mod, n):
    p = _particles("plummer", n)
    for a in (p.x, p.y, p.z):
        a[n - 1] = a[0]
    with pytest.raises(nbb_mod.DeviceError, match="Singular"):
        nbb_mod.compute_accelerations(p, 0.6, 0.0, 1.0)


# both significands whose root is 2 - 2^-52, in each form of the walk
@pytest.mark.parametrize("n", [2, 5000, 65537])
@pytest.mark.parametrize("extent", [2.0 ** -28, 2.0 ** -25])
def test_rounding_exceptions(nbb_mod, oracle, n, extent):
    """eps^2 = 4 - 2^-50 and distances that round it to 4 - 2^-50 (the smaller
    extent: d^2 < 2^-52) or to values from there to 4."""
    from nbb import ics

    rng = np.random.default_rng(11)
    z = np.zeros(n)
    x = rng.uniform(0.0, extent, (3, n))
    p = ics.ParticleData(rng.uniform(0.5, 1.0, n), x[0].copy(), x[1].copy(), x[2].copy(), z, z, z)
    soft = 2.0 - 2.0 ** -52
    assert soft * soft == 4.0 - 2.0 ** -50
    _check(nbb_mod, oracle, p, 0.5, soft)
