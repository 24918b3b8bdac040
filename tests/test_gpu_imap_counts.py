"""Intensity maps whose samples per pixel exceed a float's whole numbers on
paper (12 pixels for all cells: the counts are kept as integers), thin shells
(every cell walks the edges), and shells down to the observer: hit counts equal
the double restatement's, brightness within the float sum's own bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = {
    "few pixels": (96, 2.0, 0.05, 0.6, dict(tz=0.1, bias=("const", 1.0), z_range=(0.06, 0.59), nbands=1, nside=1)),
    "thin shells": (64, 2.0, 0.05, 0.6, dict(tz=0.1, bias=("1+z",), z_range=(0.2, 0.55), nbands=80, nside=64)),
    "to the observer": (64, 1.0, 0.001, 0.3, dict(tz=0.1, bias=("1+z",), z_range=(0.002, 0.29), nbands=3, nside=16)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_hits_equal_double(built, tmp_path, name):
    import colore_gb300 as cg
    import oracle as orc
    from colore_gb300 import inputs
    n, smooth, z0, z1, imap = CASES[name]
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=z0, z_max=z1, r_smooth=smooth, seed=29, dens_type=0, bias_model=2, imap=[imap])))
    m = cg.Mock(prm)
    m.run()
    got, hits = m.imap(0, with_nadd=True)
    dens, phi = m.grid(0)[:, :, :n].astype(np.float64), m.grid(1)[:, :, :n].astype(np.float64)
    t64, e64 = m.norm_table64(1, 0)
    data, nadd = orc.imap64(prm.config, 0, dens, phi, t64, e64)
    m.close()
    assert nadd.sum() > 10 ** 4
    assert np.array_equal(hits, nadd), int((hits != nadd).sum())
    # a pixel's sum rounds once per addition, at most once per sample
    want = np.where(nadd > 0, data / np.maximum(nadd, 1), 0)
    assert np.all(np.abs(got - want) <= (nadd * 2.0 ** -24 + 2e-5) * np.abs(want))
