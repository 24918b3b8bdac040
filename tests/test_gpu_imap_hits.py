"""The hit counts alone: no device memory is taken and a captured sequence keeps
its graph; maps of more pixels than one piece of the download come whole."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _hits(cg, m, shape):
    a = np.full(shape, -1, np.int32)
    assert cg.lib().cg_download_imap(m._c, 0, None, C.c_void_p(a.ctypes.data)) == 0
    return a


@pytest.mark.parametrize("nside,nbands", [(16, 3), (512, 3)])  # 9216 and 9.4e6 pixels: one piece and three
def test_hits_alone(built, tmp_path, nside, nbands):
    import torch
    import colore_gb300 as cg
    from colore_gb300 import inputs
    m = cg.Mock(cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=64, z_min=0.05, z_max=0.6, r_smooth=2.0, seed=11, dens_type=0, bias_model=2,
        imap=[dict(tz=0.1, bias=("const", 1.0), z_range=(0.4, 0.55), nbands=nbands, nside=nside)]))))
    try:
        m.run()
        m.graph_capture()
        m.graph_launch()
        m.sync()
        free = torch.cuda.mem_get_info()[0]
        got = _hits(cg, m, (nbands, 12 * nside * nside))
        assert torch.cuda.mem_get_info()[0] == free
        m.graph_launch()  # refused if the graph had been dropped
        m.sync()
        assert np.array_equal(_hits(cg, m, got.shape), got)
        assert got.min() >= 0 and got.sum() > 10 ** 4
        assert np.array_equal(m.imap(0, with_nadd=True)[1], got)
    finally:
        m.close()
