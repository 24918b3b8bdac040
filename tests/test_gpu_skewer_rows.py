"""Skewers of rows that are not a whole number of warps (48 and 96 steps), of a
few sources and of more than one pass of the launch, density and Gaussian: the
single-precision restatement's bits, zeros past each source."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,density,gauss", [(96, 0.01, False), (96, 0.5, True), (192, 0.6, False)])
def test_rows_match_oracle(built, tmp_path, n, density, gauss):
    import colore_gb300 as cg
    import oracle as orc
    from colore_gb300 import inputs
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=53, dens_type=0, bias_model=2,
        srcs=[dict(nz=("gauss", 0.3, 0.1), density=density, bias=("const", 1.5), nside_count=0, skewers=True,
                   gaussian_skewers=gauss)])))
    m = cg.Mock(prm)
    m.create_cartesian_fields()
    s2 = m.sigma2()[0]
    m.compute_physical_density_field()
    m.compute_density_normalization()
    m.srcs_set_cartesian()
    m.get_beam_properties()
    pos = m.catalog(0, pos=True, ipix=False, src=False)["pos"]
    d, v = m.skewers(0)
    dens, phi = m.grid(0), m.grid(1)
    m.close()
    assert len(pos) > 50 and d.shape == (len(pos), n // 2)
    d32, v32 = orc.skw32(prm.config, dens, phi, gauss, np.float32(s2), pos)
    assert np.array_equal(d32.view(np.uint32), d.view(np.uint32))
    assert np.array_equal(v32.view(np.uint32), v.view(np.uint32))
