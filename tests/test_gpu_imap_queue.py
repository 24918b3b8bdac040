"""The painting's stages of samples left to double, filled past their room:
with every decision forced into double a warp stages each of its samples, from
a few to a thousand per unit, and flushes groups of every fill.  The hit counts
are those of the margins, and every sample drawn is decided."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nside,z0,z1,nb,zmax", [  # 2, 3, 7, 14 and 47 sub-cells per axis
    (128, 64, 0.3, 0.5, 4, 0.52), (64, 64, 0.44, 0.5, 5, 0.52), (96, 256, 0.34, 0.4, 5, 0.42),
    (64, 256, 0.1, 0.108, 1, 0.16), (64, 32, 0.01, 0.012, 1, 0.52)])
def test_forced_double_stages(built, tmp_path, n, nside, z0, z1, nb, zmax):
    import colore_gb300 as cg
    from colore_gb300 import inputs
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.005, z_max=zmax, r_smooth=2.0, seed=31, dens_type=0, bias_model=2,
        imap=[dict(tz=0.1, bias=("const", 1.0), z_range=(z0, z1), nbands=nb, nside=nside)])))
    out = []
    for double in (False, True):
        m = cg.Mock(prm)
        m.set_decisions_in_double(double)
        m.run()
        out.append((m.imap(0, with_nadd=True)[1].copy(), m.imap_samples(0), m.exact_stats()["imap_samples"]))
        m.close()
    (a, na, _), (b, nb, doubles) = out
    assert na == nb and na > 10 ** 4 and doubles == nb
    assert np.array_equal(a, b), int((a != b).sum())
