"""The bins pass carries up to eight tracers per launch: populations with one
and the same bias give, each of them and whatever their number, the
normalisation table of a single population bit for bit (the sums of a value
do not depend on its place among the values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tables(tmp_path, n, model, dens_type):
    import colore_gb300 as cg
    from colore_gb300 import inputs
    spec = dict(n_grid=64, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=17, dens_type=dens_type, bias_model=model,
                srcs=[dict(nz=("gauss", 0.3, 0.1), density=1.0, bias=("1+z",), nside_count=0) for _ in range(n)])
    m = cg.Mock(cg.Params(inputs.write_inputs(str(tmp_path / ("n%d" % n)), spec)))
    m.create_cartesian_fields()
    m.compute_physical_density_field()
    m.compute_density_normalization()
    out = [m.norm_table64(0, i) for i in range(n)]
    m.close()
    return out


@pytest.mark.parametrize("model,dens_type", [(1, 0), (2, 1), (3, 3)])
def test_tables_do_not_depend_on_the_number_of_tracers(built, tmp_path, model, dens_type):
    one, = _tables(tmp_path, 1, model, dens_type)
    assert np.all(np.isfinite(one[0])) and one[0].std() > 0
    for n in range(2, 9):
        for t, e in _tables(tmp_path, n, model, dens_type):
            assert np.array_equal(t, one[0]) and np.array_equal(e, one[1]), n
