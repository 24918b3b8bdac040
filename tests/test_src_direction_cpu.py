"""A source's direction from one octant angle, on the CPU: phi is the one of
cart2sph bit for bit, every RING pixel it decides is the double one (random
positions, positions next to pixel edges, the axes and the poles), and few
are left open; the neighbour of a float by its bits is nextafter's."""
import numpy as np
import pytest


def _positions(g, ns, n):
    v = g.normal(size=(n, 3)) * 10.0 ** g.uniform(-2, 4, (n, 1))
    k = n // 4
    # next to the equatorial edge lines and the lines phi = k pi/2
    z = g.uniform(-2 / 3, 2 / 3, k)
    t = (g.integers(0, 4 * ns + 2, k) / ns - 0.5 + 0.75 * z) % 4 + g.normal(0, 1e-7, k)
    s = np.sqrt(1 - z * z)
    v[:k] = 1000 * np.stack([s * np.cos(t * np.pi / 2), s * np.sin(t * np.pi / 2), z], 1)
    t = g.integers(0, 4, k) + g.normal(0, 1e-7, k)
    z = g.uniform(-1, 1, k)
    s = np.sqrt(1 - z * z)
    v[k:2 * k] = 1000 * np.stack([s * np.cos(t * np.pi / 2), s * np.sin(t * np.pi / 2), z], 1)
    axes = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, 1, 1],
                     [1, -1, -1], [-0.0, -0.0, 1], [1e-20, 0, 1], [3, -0.0, 2], [-3, -0.0, 2]])
    return np.concatenate([v, axes * 7.0]).astype(np.float32)


@pytest.mark.parametrize("ns", [1, 2, 64, 512, 8192])
def test_direction_and_pixels(built, ns):
    import oracle as orc
    v = _positions(np.random.default_rng(ns), ns, 400000)
    ph, ref, pix = orc.dir_phi(ns, v)
    assert np.array_equal(ph.view(np.uint32), ref.view(np.uint32))
    ok = pix >= 0
    want = orc.pix64(ns, v.astype(np.float64))
    assert np.array_equal(pix[ok], want[ok])
    assert ok[len(v) // 2:].mean() > 1 - 1e-5 * (ns + 30), "random positions left open"


def test_next_float(built):
    import oracle as orc
    g = np.random.default_rng(1)
    f = np.concatenate([g.normal(size=20000) * 10.0 ** g.uniform(-38, 37, 20000),
                        [0.0, -0.0, 1.0, -1.0, 2.0, -2.0, 1.17549435e-38, -1.17549435e-38, 1e-45, -1e-45]])
    f = f.astype(np.float32)
    for up in (0, 1):
        got = orc.next_float(f, np.full(len(f), up))
        want = np.nextafter(f, np.float32(np.inf if up else -np.inf))
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
