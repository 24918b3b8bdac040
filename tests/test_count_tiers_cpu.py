"""The first tier's decisions that the counting kernel takes, over densities from
nothing to hundreds of sources a cell: a cell without a source has none in
double, one for inversion has the double count where the margins keep it, one
left to PTRS has a double lambda of 10 or more, and few cells stay open."""
import numpy as np
import pytest

NA = 5001


@pytest.mark.parametrize("model", [1, 2, 3])
@pytest.mark.parametrize("scale", [1e-12, 1e-3, 0.1, 3.0])
def test_decisions(built, model, scale):
    import oracle as orc
    g = np.random.default_rng(int(1000 * scale) + model)
    ng, l_box = 128, 1300.0
    dx = l_box / ng
    idr = (NA - 1) / (0.9 * l_box)
    r = np.arange(NA) / idr
    nz = scale * (0.2 + np.exp(-0.5 * ((r / l_box - 0.3) / 0.1) ** 2)) / dx ** 3 * 10
    n = 200000
    cell = g.integers(0, ng, (n, 3))
    cell[:1000] = ng // 2 + g.integers(-1, 2, (1000, 3))
    d = np.exp(g.normal(0, 1.0, n)) - 1
    bits = g.integers(0, 2 ** 24, n)
    bits[:2000] = 2 ** 24 - 1
    lam, elam, lam64, got, ref = orc.count_seg(r, nz, 1 + r / l_box, 1 + 0.1 * np.cos(r / 100), idr, dx,
                                               [0.5 * l_box] * 3, dx ** 3, 0.5 * l_box + 20, model, cell, d, bits)
    none = (got == 0) & (ref >= 0)
    assert np.array_equal(ref[none], got[none])
    assert np.all(lam64[got == 0] < 17)  # -ln 2^-24: no uniform leaves a denser cell empty
    inv = got > 0
    assert np.array_equal(ref[inv], got[inv])
    ptrs = got == -2
    assert np.all(lam64[ptrs] >= 10)
    sure = (lam64 > 10.1) & (np.sqrt(((cell - ng // 2) ** 2).sum(1)) * dx < 0.5 * l_box + 19.9)
    sure &= np.any(cell != ng // 2, 1)
    if sure.any():
        assert ptrs[sure].mean() > 0.99
    assert (got == -1).mean() < (0.02 if scale > 0.05 else 0.01)
