"""Room for the listed cells of an intensity map: thick shells, shells thinner
than a cell, shells thinner than the redshift-space shift (whose cells span
several, which no per-cell loop paints), overlapping and gapped shells, down to
the observer.  However the cells divide into general and fast ones, each
shell's equatorial and polar rooms hold all of them; rooms in all take little
more than the cells they can be asked to hold."""
import numpy as np
import pytest

CASES = {  # grid, z_max, z range, bands, shift amplitude, whether most cells are general
    "thick": (96, 0.6, (0.1, 0.55), 4, 1.0, False),
    "thin": (64, 0.6, (0.2, 0.55), 80, 1.0, None),
    "shift across shells": (96, 0.3, (0.1, 0.28), 30, 60.0, True),
    "to the observer": (48, 0.3, (0.002, 0.29), 5, 1.0, None),
    "one shell": (64, 0.4, (0.02, 0.39), 1, 1.0, False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_rooms_hold_the_cells(built, tmp_path, name):
    import oracle as orc
    from colore_gb300 import inputs
    n, zmax, zr, nb, amp, general = CASES[name]
    cfg = orc.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.001, z_max=zmax, r_smooth=2.0, seed=53, dens_type=0, bias_model=2,
        imap=[dict(tz=0.1, bias=("const", 1.0), z_range=zr, nbands=nb, nside=64)]))).config
    d64, p64, st = orc.field64(cfg)
    d32 = orc.density64(cfg, d64, st[3]).astype(np.float32)
    tabs, e0f, _ = orc.norm_tables64(cfg, d32.astype(np.float64))
    pad = lambda a: np.ascontiguousarray(np.pad(a, ((0, 0), (0, 0), (0, 2 * (n // 2 + 1) - n))))
    t64, e64 = tabs[0], np.asarray(e0f[0], np.float64)
    cells, room, part = orc.imap_rooms(cfg, 0, pad(d32), pad((amp * p64).astype(np.float32)), t64.astype(np.float32),
                                        e64.astype(np.float32), t64, e64)
    used = cells.sum(2)
    print(name, "cells", used.sum(), "general", cells[:, :, 0].sum(), "rooms", room.sum(), "fill %.2f" % (used / room).max())
    assert used.sum() > 0.05 * n ** 3
    assert np.all(used <= room)
    assert np.all((part > 0) & (part <= 0.5))
    if general is not None:
        assert (cells[:, :, 0].sum() > 0.5 * used.sum()) == general
    # what the shells' volumes hold, a half cell's layer on either side and the
    # layers about the cones
    dx = cfg.l_box / n
    r0 = np.sort([cfg.imap_r0[0][i] for i in range(nb)])
    rf = np.sort([cfg.imap_rf[0][i] for i in range(nb)])
    vol = 4 / 3 * np.pi * ((rf + 0.9 * dx) ** 3 - np.maximum(r0 - 0.9 * dx, 0) ** 3) / dx ** 3
    ir = np.minimum(dx / np.maximum(r0 - 0.9 * dx, dx), 1)
    assert np.all(room[1:-1].sum(1) <= vol * (1 + 2 * ir) + 130)
