"""The Maxwell update on grids at the edges of its tiles (32 columns by 8
threads of several rows): one cell, one column, one row, a tile and its
neighbours, and a grid long enough for several rows per thread, against the
oracle's restatement.  Operations and their order are the oracle's, up to
FMA contraction: within 1e-12 of each vector's largest magnitude, the bound
the field test derives for sums of differences of nearby values."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nz,substeps", [(1, 1, 1), (1, 9, 2), (9, 1, 2), (2, 2, 1), (31, 7, 2), (32, 8, 1),
                                            (33, 9, 3), (64, 17, 2), (130, 3001, 2)])
def test_field_step_at_tile_edges(nr, nz, substeps):
    from oracle import oracle
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu
    build.build()
    oracle.load_tables(TABLES)
    rng = np.random.default_rng(100 * nr + nz)
    dr, dz, dt = 0.8, 0.9, 5.0e-10
    ctx = gpu.RreaGpuContext(gpu.default_config(r_hi=nr * dr, z_lo=0.0, z_hi=nz * dz, nr=nr, nz=nz), 16)
    er = rng.normal(0.0, 2.0e3, (nz, nr + 1))
    er[:, 0] = 0.0
    bt = rng.normal(0.0, 1.0e-5, (nz + 1, nr + 1))
    bt[:, 0] = 0.0
    ez = rng.normal(0.0, 2.0e3, nr * (nz + 1))
    ctx.set_field(er.ravel(), ez, bt.ravel(), np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1)))
    ctx.reset_current()
    before = ctx.field()
    ctx.advance_field(dt, substeps)
    c = ctx.config
    ref = oracle.advance_maxwell(nr, nz, (c.r_hi - c.r_lo) / nr, (c.z_hi - c.z_lo) / nz, dt, substeps, *before,
                                 np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1)))
    for name, g, o in zip(("er", "ez", "bt"), ctx.field(), ref):
        np.testing.assert_allclose(g, o, rtol=0, atol=1e-12 * max(np.abs(o).max(), 1e-300), err_msg=name)
    ctx.close()
