"""The first tier of the Poisson counts on the CPU: lambda from the
per-segment tables lies within its bound of the double lambda for every bias
model and table shape, over the whole box (observer's corner, table nodes,
the radius limit) and density range (-1, next to -1, 0, large), and every
count it settles is the double one."""
import numpy as np
import pytest

NA = 5001


def _tables(shape, r, rmax):
    x = r / rmax
    nz = {"gauss": np.exp(-0.5 * ((x - 0.5) / 0.12) ** 2),
          "flat": 0.5 * (np.tanh((x - 0.2) / 0.004) - np.tanh((x - 0.7) / 0.004)) - 1e-9,
          "steep": 1.0 / (1e-3 + x * x),
          "ringing": np.sin(60 * x) * np.exp(-3 * x)}[shape]
    return 2e-3 * nz, 1.0 + 2.0 * x, 1.0 + 0.2 * np.cos(9 * x)


@pytest.mark.parametrize("model", [1, 2, 3])
@pytest.mark.parametrize("shape", ["gauss", "flat", "steep", "ringing"])
def test_lambda_bound_and_counts(built, model, shape):
    import oracle as orc
    g = np.random.default_rng(model * 10 + len(shape))
    ng, l_box = 256, 2600.0
    dx = l_box / ng
    idr = (NA - 1) / (0.95 * l_box)
    r = np.arange(NA) / idr
    nz, bz, norm = _tables(shape, r, 0.5 * l_box)
    n = 400000
    cell = g.integers(0, ng, (n, 3))
    cell[:2000] = ng // 2 + g.integers(-2, 3, (2000, 3))  # around the observer
    d = np.exp(g.normal(0, 1.2, n)) - 1
    d[2000:4000] = -1
    d[4000:6000] = -1 + 2.0 ** -g.integers(1, 25, 2000)
    d[6000:8000] = g.uniform(0, 300, 2000)
    d[8000:10000] = 0
    bits = g.integers(0, 2 ** 24, n)
    lam, elam, lam64, got, ref = orc.count_seg(r, nz, bz, norm, idr, dx, [0.5 * l_box] * 3, dx ** 3, 0.5 * l_box + 20,
                                               model, cell, d, bits)
    rc = dx * np.sqrt(((cell - ng // 2) ** 2).sum(1))
    inside = (rc > 0) & (rc < 0.5 * l_box + 19.9)
    # the reference draws nothing where n(r) <= 0; the tier's value is then at most its bound
    certain = inside & (lam64 > 0)
    assert np.all(np.abs(lam[certain] - lam64[certain]) <= elam[certain])
    none = inside & (lam64 == 0)
    assert np.all(lam[none] <= elam[none])
    settled = got >= 0
    small = settled & (ref >= 0)
    assert np.array_equal(got[small], ref[small])
    assert not np.any(settled & (ref < 0)), "counts with lambda >= 10 are not this tier's"
    assert settled[inside & (lam64 < 9)].mean() > 0.99
    assert got[(rc > 0.5 * l_box + 20.1)].max(initial=0) == 0
