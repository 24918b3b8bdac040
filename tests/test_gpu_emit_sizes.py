"""The emission at either side of its rule (records written directly where 2048
cells hold few sources, staged where they hold many), from a handful of sources
in all to thousands per block of cells: catalogues and count maps equal the CPU
restatement bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("density,lo,hi", [(0.0005, 0, 1), (0.05, 5, 40), (0.3, 60, 128), (0.6, 144, 300), (20.0, 4000, 9000)])
def test_catalogue_bits(built, tmp_path, density, lo, hi):
    import colore_gb300 as cg
    import oracle as orc
    from colore_gb300 import inputs
    n = 64
    prm = cg.Params(inputs.write_inputs(str(tmp_path), dict(
        n_grid=n, z_min=0.05, z_max=0.4, r_smooth=2.0, seed=19, dens_type=0, bias_model=2,
        srcs=[dict(nz=("flat", 0.06, 0.39), density=density, bias=("const", 1.5), nside_count=32)])))
    m = cg.Mock(prm)
    try:
        m.run()
        g = m.catalog(0)
        total = m.num_sources(0)
        assert lo <= total / (n ** 3 / 2048) <= hi and total > 5
        tab, e = m.norm_table(0, 0)
        t64, e64 = m.norm_table64(0, 0)
        ref = orc.emit32(prm.config, 0, m.grid(0), m.grid(1), tab, e, t64, e64, cap=total + 100)
        assert len(ref["pos"]) == total
        for k in ("pos", "src"):
            assert np.array_equal(ref[k].view(np.uint32), g[k].view(np.uint32)), k
        assert np.array_equal(ref["ipix"], g["ipix"])
        assert np.array_equal(ref["cmap"], m.count_map(0))
    finally:
        m.close()
