"""Particles displaced by many cells: deposits that leave their block's box, and
boxes that reach over the ends of the grid, in a box so small that the
displacements exceed the halo.  NGP, CIC and TSC, 1LPT and 2LPT, against the
FP64 restatement of the same scheme."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dens_type,interp", [(1, 0), (1, 1), (1, 2), (2, 1)])
def test_far_particles_match_double(built, tmp_path, dens_type, interp):
    import colore_gb300 as cg
    import oracle as orc
    from colore_gb300 import inputs
    n = 64
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.001, z_max=0.02, r_smooth=0.5, seed=31, dens_type=dens_type, lpt_interp_type=interp, bias_model=2,
        srcs=[dict(nz=("gauss", 0.01, 0.005), density=0.01, bias=("const", 1.0), nside_count=0)])))
    m = cg.Mock(prm)
    m.create_cartesian_fields()
    m.compute_physical_density_field()
    got = m.grid(0)[:, :, :n].astype(np.float64)
    disp = np.array([m.grid(2 + a)[:, :, :n] for a in range(3)])
    m.close()
    cells = np.abs(disp) * n / prm.config.l_box
    assert cells.max() > 4, cells.max()
    d64, _, _ = orc.field64(prm.config)
    out = (orc.lpt2_64 if dens_type == 2 else orc.lpt64)(prm.config, d64)[0]
    assert abs(np.mean(got + 1.0) - 1.0) < 1e-6
    # positions to the displacements' relative error (2e-5, second order 1e-4)
    # times their size in cells, on each of three axes; a weight's slope is 1
    err = (1e-4 if dens_type == 2 else 2e-5) * np.sqrt(np.mean(cells ** 2)) * 4 + 1e-5
    if interp == 0:
        # whole particles: one within err of a cell's edge may fall either side, out of one cell into another
        assert (np.abs(got - out) > 1e-3).mean() < 4 * err
    else:
        assert np.sqrt(np.mean((got - out) ** 2)) < err * np.sqrt(np.mean((out + 1.0) ** 2)) + 1e-4
