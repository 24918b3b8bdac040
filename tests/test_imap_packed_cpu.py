"""A bound on the samples of one pixel of an intensity map, below which the
counts are held as floats without losing any: no pixel lies farther from its
centre than the radius the bound takes, and over maps of few and of many
pixels, thin and thick shells, down to the observer, with and without radial
shifts, every pixel's samples stay below it.  Full-size maps stay a factor of
thirty below a float's whole numbers."""
import numpy as np
import pytest

RADIUS = 1.25  # CG_PIX_RADIUS


@pytest.mark.parametrize("nside", [1, 2, 4, 16, 128, 1024])
def test_pixel_radius(built, nside):
    import oracle as orc
    g = np.random.default_rng(nside)
    n = 400000
    v = g.normal(size=(n, 3))
    v[: n // 2, 2] = np.hypot(v[: n // 2, 0], v[: n // 2, 1]) * g.uniform(0.7, 1.1, n // 2)  # where pixels are longest
    v[-1000:, :2] *= 1e-3 / nside
    v /= np.linalg.norm(v, axis=1)[:, None]
    ring = orc.pix64(nside, v.astype(np.float32))
    nest = np.arange(12 * nside * nside)
    u, inv = np.unique(ring, return_inverse=True)
    by_ring = np.empty(12 * nside * nside, np.int64)
    by_ring[orc.nest2ring(nside, nest)] = nest
    c = orc.pix2vec_nest(nside, by_ring[u])[inv].astype(float)
    ang = 2 * np.arcsin(np.minimum(0.5 * np.linalg.norm(v - c / np.linalg.norm(c, axis=1)[:, None], axis=1), 1))
    assert ang.max() * nside < 0.9 * RADIUS
    assert ang.max() * nside > 0.6


CASES = {  # grid, z_max, z range, bands, nside, spread of the potential
    "few pixels": (96, 0.6, (0.06, 0.59), 1, 1, 0.0),
    "few pixels, thin": (64, 0.6, (0.1, 0.55), 40, 2, 1e-3),
    "coarse": (64, 0.6, (0.1, 0.55), 5, 8, 0.0),
    "fine": (64, 0.6, (0.2, 0.5), 12, 64, 1e-3),
    "to the observer": (32, 0.3, (0.004, 0.29), 4, 8, 0.0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_samples_per_pixel(built, tmp_path, name):
    import oracle as orc
    from colore_gb300 import inputs
    n, zmax, zr, nb, nside, amp = CASES[name]
    cfg = orc.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.001, z_max=zmax, r_smooth=2.0, seed=3, dens_type=0, bias_model=2,
        imap=[dict(tz=0.1, bias=("const", 1.0), z_range=zr, nbands=nb, nside=nside)]))).config
    phi = amp * np.random.default_rng(5).normal(size=(n, n, n))
    _, nadd = orc.imap64(cfg, 0, np.zeros((n, n, n)), phi, np.ones(5001), (1.0, 1.0))
    most, bound = nadd.sum(0).max(), orc.imap_pixel_max(cfg, 0)
    print(name, most, bound)
    assert 0 < most <= bound
    assert bound < 60 * most + 200


def test_full_size_maps_are_packed(built, tmp_path):
    import oracle as orc
    from colore_gb300 import inputs
    for cfg, n in (("c4", 1024), ("c4", 512), ("c4", 256)):
        spec = inputs.scaled(cfg, n)
        assert orc.imap_pixel_max(orc.Params(inputs.write_inputs(str(tmp_path), spec)).config, 0) < 2 ** 24 / 30
