"""Forced tile widths reach the passes they name: the Gaussian potential's x
pass (a launch of its own) and the nine-grid fill of 2LPT, with the same bits
for every width; the tuner times what a run uses and nothing else."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spec(n, dens_type):
    return dict(n_grid=n, z_min=0.05, z_max=0.4, r_smooth=2.0, seed=73, dens_type=dens_type, bias_model=2,
                srcs=[dict(nz=("gauss", 0.2, 0.05), density=10.0, bias=("const", 1.0))])


@pytest.mark.parametrize("n", [64, 96, 256])
def test_forced_widths(built, tmp_path, n):
    import colore_gb300 as cg
    from colore_gb300 import inputs
    m = cg.Mock(cg.Params(inputs.write_inputs(str(tmp_path), _spec(n, 2))))
    try:
        def grids():
            k = m.launches()
            m.create_cartesian_fields()
            k = m.launches() - k
            out = [m.grid(0).copy(), m.grid(1).copy()]
            m.compute_physical_density_field()
            return k, out + [m.grid(w).copy() for w in range(2, 8)]
        for p in m.PASSES:
            m.set_field_variant(p, 0)
        k0, ref = grids()
        forced = {"x": 0, "fill3": 0}
        for p in forced:
            for v in (1, 2):
                try:
                    m.set_field_variant(p, v)
                except cg.CGError:
                    continue  # not a valid width at this size
                k, got = grids()
                for a, b in zip(got, ref):
                    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (p, v)
                assert k == k0 + (p == "x")
                forced[p] += 1
            m.set_field_variant(p, 0)
        assert all(forced.values())
        for p in m.PASSES:
            m.set_field_variant(p, -1)
        grids()
        plan = m.field_plan()
        assert plan["fill3"]["timed"] or not plan["tuned"]
    finally:
        m.close()


def test_potential_pass_above_512(built, tmp_path):
    import torch
    import colore_gb300 as cg
    from colore_gb300 import inputs
    m = cg.Mock(cg.Params(inputs.write_inputs(str(tmp_path), _spec(1024, 0))))
    try:
        ref, got = (torch.empty(cg.grid_shape(1024), dtype=torch.float32, device="cuda") for _ in range(2))
        m.set_field_variant("x", 0)
        m.create_cartesian_fields()
        m.grid(1, out=ref)
        for v in (1, 2):
            m.set_field_variant("x", v)
            m.create_cartesian_fields()
            m.grid(1, out=got)
            # the two floats past each row are scratch
            assert torch.equal(got[:, :, :1024].view(torch.int32), ref[:, :, :1024].view(torch.int32)), v
    finally:
        m.close()


def test_tuner_times_what_runs(built, tmp_path):
    from colore_gb300 import inputs
    prog = ("import sys, colore_gb300 as cg\n"
            "out = []\n"
            "for f in sys.argv[1:]:\n"
            "    m = cg.Mock(cg.Params(f))\n"
            "    m.create_cartesian_fields()\n"
            "    m.compute_physical_density_field()\n"
            "    p = m.field_plan()\n"
            "    out.append([p['tuned']] + [p[k]['timed'] for k in ('fill2', 'fill3', 'y', 'x')])\n"
            "    m.close()\n"
            "print(out)\n")
    files = []
    for t in (0, 2, 1):
        d = tmp_path / str(t)
        d.mkdir()
        files.append(inputs.write_inputs(str(d), _spec(64, t)))
    env = dict(os.environ, COLORE_GB300_TUNE="1")
    r = subprocess.run([sys.executable, "-c", prog] + files, capture_output=True, text=True, env=env,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr
    lognormal, lpt2, lpt = eval(r.stdout.strip().splitlines()[-1])
    assert lognormal == [True, True, False, True, False]
    assert lpt2 == [True] * 5
    assert lpt == [True] * 5
