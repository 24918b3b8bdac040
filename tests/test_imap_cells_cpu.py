"""Intensity-map cells and samples on the CPU.  Samples by per-cell constants:
for cells all over the box (next to the observer, the axes' planes, the
diagonals, |cos theta| = 2/3 and the poles) every sample the constants decide
has the double arithmetic's pixel and shell; most cells qualify and most
samples are decided.  Cells listed from per-segment tables: everything they
settle is as in double, and few cells stay open."""
import numpy as np
import pytest


def _cells(g, ng, n):
    c = g.integers(0, ng, (n, 3))
    h, k = ng // 2, n // 8
    c[:k] = h + g.integers(-12, 12, (k, 3))                              # near the observer
    c[k:2 * k, 1] = h + g.integers(-2, 2, k)                             # y = 0
    c[2 * k:3 * k, 0] = h + g.integers(-2, 2, k)                         # x = 0
    c[3 * k:4 * k, 1] = c[3 * k:4 * k, 0] + g.integers(-2, 3, k)         # the diagonal
    rho = np.hypot(c[4 * k:5 * k, 0] - h, c[4 * k:5 * k, 1] - h)
    c[4 * k:5 * k, 2] = h + np.rint(rho * 0.8944 * g.choice([-1, 1], k)) + g.integers(-2, 3, k)  # |cos theta| = 2/3
    c[5 * k:6 * k, :2] = h + g.integers(-6, 6, (k, 2))                   # towards the poles
    return np.clip(c, 0, ng - 1)


@pytest.mark.parametrize("nside", [1, 2, 32, 512, 4096])
def test_samples_of_cells_match_double(built, nside):
    import oracle as orc
    g = np.random.default_rng(nside)
    ng, l_box = 1024, 6121.33
    dx = float(np.float32(l_box)) / ng
    pos = [0.5 * float(np.float32(l_box))] * 3
    n = 16000
    cell = _cells(g, ng, n)
    nsub = g.choice([1, 2, 3, 4, 5, 8], n)
    r = dx * np.sqrt(((cell - ng // 2 + 0.5) ** 2).sum(1))
    drr64 = g.normal(0, 4.0, n)
    edrr = 1e-4
    drr = (drr64 + g.uniform(-0.9, 0.9, n) * edrr).astype(np.float32)
    edge = np.where(g.random(n) < 0.5, np.maximum(r + drr64 + g.uniform(-0.5, 0.5, n) * dx, 1.0), -1.0)
    fast, eq, samples, decided, wrong = orc.imap_fast(nside, ng, dx, pos, cell, nsub, edge, drr, drr64, edrr)
    assert wrong == 0
    assert fast > 0.4 * n and 0.3 * fast < eq < 0.95 * fast
    # a sample stays open with the margins' share of a pixel: three decisions
    # of some 1e-6 nside each, and the edge's 2e-4 of a cell
    assert decided > (1 - 2e-5 * nside - 1e-3) * samples
    far = r > 60 * dx
    f2 = orc.imap_fast(nside, ng, dx, pos, cell[far][-n // 4:], nsub[far][-n // 4:], edge[far][-n // 4:],
                       drr[far][-n // 4:], drr64[far][-n // 4:], edrr)
    assert f2[0] > 0.9 * (n // 4) and f2[4] == 0


SPECS = {
    "coarse": dict(n_grid=64, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=41, dens_type=0, bias_model=2,
                   imap=[dict(tz=0.1, bias=("const", 1.0), z_range=(0.05, 0.5), nbands=12, nside=64)]),
    "thin": dict(n_grid=64, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=43, dens_type=0, bias_model=1,
                 imap=[dict(tz=0.1, bias=("1+z",), z_range=(0.2, 0.55), nbands=60, nside=256)]),
    "to the origin": dict(n_grid=32, z_min=0.001, z_max=0.3, r_smooth=1.0, seed=47, dens_type=0, bias_model=2,
                          imap=[dict(tz=0.1, bias=("1+z",), z_range=(0.002, 0.29), nbands=5, nside=16)]),
}


@pytest.mark.parametrize("name", list(SPECS))
def test_cells_from_segments_match_double(built, tmp_path, name):
    import oracle as orc
    from colore_gb300 import inputs
    cfg = orc.Params(inputs.write_inputs(str(tmp_path), SPECS[name])).config
    n = cfg.n_grid
    d64, p64, st = orc.field64(cfg)
    d32 = orc.density64(cfg, d64, st[3]).astype(np.float32)
    tabs, e0f, _ = orc.norm_tables64(cfg, d32.astype(np.float64))
    pad = lambda a: np.ascontiguousarray(np.pad(a, ((0, 0), (0, 0), (0, 2 * (n // 2 + 1) - n))))
    t64, e64 = tabs[0], np.asarray(e0f[0], np.float64)
    settled, listed, still_open, *faults = orc.imap_cells(
        cfg, 0, pad(d32), pad(p64.astype(np.float32)), t64.astype(np.float32), e64.astype(np.float32), t64, e64)
    assert faults == [0] * 5
    assert settled + still_open == n ** 3 and listed > 0.05 * n ** 3
    # open: the segments where the brightness begins or ends, and the corners
    # within 5e-7 r of an edge
    assert still_open < 2e-3 * n ** 3
