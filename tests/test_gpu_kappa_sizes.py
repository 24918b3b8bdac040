"""Convergence maps of both block sizes and both index widths against the
single-precision oracle, bit for bit: a small and a large map on 64^3 (32-bit
byte offsets, rays up to the box faces) and a small map on 1024^3, whose
potential needs 64-bit offsets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nside", [(64, 8), (64, 256), (1024, 4)])
def test_kappa_matches_oracle(built, tmp_path, n, nside):
    import colore_gb300 as cg
    import oracle as orc
    from colore_gb300 import inputs
    spec = dict(n_grid=n, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=23, dens_type=0, bias_model=2,
                srcs=[dict(nz=("gauss", 0.3, 0.1), density=0.01, bias=("const", 1.0), nside_count=0)],
                kappa=dict(z_out=[0.2, 0.4, 0.6], nside=nside))
    prm = cg.Params(inputs.write_inputs(str(tmp_path), spec))
    m = cg.Mock(prm)
    m.run()
    got = m.kappa()
    phi = m.grid(1)
    m.close()
    want = orc.kappa32(prm.config, phi)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
