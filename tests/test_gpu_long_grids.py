"""Grids with more rows than one launch dimension of the field kernels holds
(65,535 blocks of 8 threads with up to 4 rows each where the cell averages are
formed, with up to 8 in the Maxwell update), and the largest below:

  * the electron phase over the whole length against the oracle, by the phase
    tests' rule (the cell averages are what it gathers);
  * the Maxwell update against the oracle's, within the bound of
    test_gpu_field_tiles.py."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu

PREP_ROWS = 65535 * 8 * 4
MAXWELL_ROWS = 65535 * 8 * 8


@pytest.fixture(scope="module")
def mods():
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu, workloads
    from oracle import compare, oracle
    build.build()
    oracle.load_tables(TABLES)
    return gpu, workloads, oracle, compare


def _fields(rng, nr, nz):
    er = rng.normal(0.0, 2.0e3, (nz, nr + 1))
    er[:, 0] = 0.0
    bt = rng.normal(0.0, 1.0e-6, (nz + 1, nr + 1))
    bt[:, 0] = 0.0
    return dict(er=er.ravel(), ez=rng.normal(0.0, 2.0e3, nr * (nz + 1)), bt=bt.ravel(),
                amb_er=np.zeros((nr + 1) * nz), amb_ez=np.full(nr * (nz + 1), -2.0e5))


@pytest.mark.parametrize("nz", [PREP_ROWS, PREP_ROWS + 1])
def test_electrons_along_a_long_grid_match_oracle(mods, nz):
    gpu, workloads, oracle, compare = mods
    nr, n = 1, 500
    cfg = workloads.make_config(gpu, "scaleup_c1")
    cfg.nr, cfg.nz, cfg.z_lo, cfg.z_hi = nr, nz, 0.0, float(nz)
    rng = np.random.default_rng(nz)
    field = _fields(rng, nr, nz)
    arr = workloads.make_electrons("scaleup_c1", n, seed=3)
    arr["z"][:] = rng.uniform(0.0, 1.0, n) * nz
    arr["z"][: n // 4] = nz - rng.uniform(0.2, 30.0, n // 4)
    workloads.capture_prev(arr)
    ctx = gpu.RreaGpuContext(cfg, 4096)
    ctx.load_tables(TABLES)
    ctx.set_field(**field)
    g, o = compare.run_pair(ctx, cfg, field, arr, 3, 5.0e-10)
    problems = compare.compare(cfg, g, o, max(cfg.r_hi, cfg.z_hi))
    ctx.close()
    assert not problems, "; ".join(problems)


@pytest.mark.parametrize("nr,nz", [(1, MAXWELL_ROWS - 1), (1, MAXWELL_ROWS), (2, MAXWELL_ROWS + 77)])
def test_field_update_on_a_long_grid_matches_oracle(mods, nr, nz):
    gpu, _, oracle, _ = mods
    dr, dz, dt = 0.8, 0.9, 5.0e-10
    f = _fields(np.random.default_rng(nz), nr, nz)
    ctx = gpu.RreaGpuContext(gpu.default_config(r_hi=nr * dr, z_lo=0.0, z_hi=nz * dz, nr=nr, nz=nz), 16)
    ctx.set_field(**f)
    ctx.reset_current()
    before = ctx.field()
    ctx.advance_field(dt, 2)
    c = ctx.config
    ref = oracle.advance_maxwell(nr, nz, (c.r_hi - c.r_lo) / nr, (c.z_hi - c.z_lo) / nz, dt, 2, *before,
                                 np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1)))
    for name, g, o in zip(("er", "ez", "bt"), ctx.field(), ref):
        np.testing.assert_allclose(g, o, rtol=0, atol=1e-12 * np.abs(o).max(), err_msg=name)
    ctx.close()
