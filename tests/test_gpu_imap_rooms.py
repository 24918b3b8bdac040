"""Intensity maps whose cells span several shells (shells thinner than the
redshift-space shift), listed in full and with the list cut so that both ends
of the rooms overflow: the hit counts are those of double decisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cells_across_shells(built, tmp_path):
    import colore_gb300 as cg
    from colore_gb300 import inputs
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=128, z_min=0.002, z_max=0.06, r_smooth=1.0, seed=37, dens_type=0, bias_model=2,
        imap=[dict(tz=0.1, bias=("const", 1.0), z_range=(0.01, 0.055), nbands=48, nside=64)])))
    m = cg.Mock(prm)
    m.run()
    want = m.imap(0, with_nadd=True)[1].copy()
    for cap in (400000, 50000, 1000, 1):
        m.set_imap_list_cap(cap)
        m.imap_set_cartesian()
        assert np.array_equal(m.imap(0, with_nadd=True)[1], want), cap
    m.set_imap_list_cap(0)
    m.set_decisions_in_double(True)
    m.run()
    assert want.sum() > 10 ** 5
    assert np.array_equal(m.imap(0, with_nadd=True)[1], want)
    m.close()
