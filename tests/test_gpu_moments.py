"""The Gaussian field's mean and variance from the x pass's partial sums, below
and above the number of partial sums at which they are added in two launches
(256^3: 4096, 384^3: 9216), against the field's own moments in double."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [256, 384])
def test_moments_equal_the_fields(built, tmp_path, n):
    import colore_gb300 as cg
    from colore_gb300 import inputs
    m = cg.Mock(cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=71, dens_type=0, bias_model=2,
        srcs=[dict(nz=("gauss", 0.3, 0.1), density=0.01, bias=("const", 1.5), nside_count=0)]))))
    for _ in range(2):  # the sums start from the pass's own each time
        m.create_cartesian_fields()
        s2, mean = m.sigma2()
        d = m.grid(0)[:, :, :n].astype(np.float64)
        # the pass adds a thread's few values and a warp's in single precision:
        # 2^-24 of each sum per addition, sixteen deep
        assert abs(s2 - d.var()) < 1e-6 * d.var()
        assert abs(mean - d.mean()) < 1e-6 * d.std()
    m.close()
