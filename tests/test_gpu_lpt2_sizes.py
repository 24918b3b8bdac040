"""2LPT displacements at grid sizes whose plans differ (two and three stages,
partial tiles): the nine fields of one fill, the source formed with its
transform, and the second order against the FP64 restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [96, 128, 192])
def test_displacements_match_double(built, tmp_path, n):
    import colore_gb300 as cg
    import oracle as orc
    from colore_gb300 import inputs
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=61, dens_type=2, bias_model=2,
        srcs=[dict(nz=("gauss", 0.3, 0.1), density=0.01, bias=("const", 1.5), nside_count=0)])))
    m = cg.Mock(prm)
    m.create_cartesian_fields()
    m.compute_physical_density_field()
    got = [m.grid(2 + a)[:, :, :n].astype(np.float64) for a in range(6)]
    m.close()
    d64, _, _ = orc.field64(prm.config)
    _, d1, d2 = orc.lpt2_64(prm.config, d64)
    # the bounds of single precision: 2e-5 of the first order, 1e-4 of the
    # second, whose source is made of products of derivatives
    for a in range(3):
        assert np.sqrt(np.mean((got[a] - d1[a]) ** 2)) < 2e-5 * np.sqrt(np.mean(d1[a] ** 2)), a
        assert np.sqrt(np.mean((got[3 + a] - d2[a]) ** 2)) < 1e-4 * np.sqrt(np.mean(d2[a] ** 2)), a
