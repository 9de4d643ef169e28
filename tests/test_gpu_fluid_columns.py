"""The coupled fluid and field step on grids whose edges do not fill the
32 x 8 column blocks of the fluid kernels, against the oracle: fewer cells
than one block, one column short of, at and past a block's 32, one row past
its 8, and more rows than the launch has threads for.  Tolerances as in the
coupled step of test_gpu_fluid.py."""
import os

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CLOSURE = os.path.join(ROOT, "data", "closure", "dry_air_swarm_hybrid_v3.csv")
QE = 1.602176634e-19


@pytest.mark.parametrize("nr,nz", [(5, 7), (31, 9), (32, 8), (33, 65), (65, 2051)])
def test_odd_grids_match_oracle(nr, nz):
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu
    from oracle import fluid as ofl
    build.build()
    ofl.load_closure(CLOSURE)
    rng = np.random.default_rng(1000 * nr + nz)
    n, dr, dz, dt = nr * nz, 2.0, 10.0, 5.0e-10
    er = rng.normal(0, 2e3, (nr + 1) * nz)
    er.reshape(nz, nr + 1)[:, 0] = 0.0
    ez, bt = rng.normal(0, 2e3, nr * (nz + 1)), rng.normal(0, 1e-6, (nr + 1) * (nz + 1))
    amb_er, amb_ez = np.zeros((nr + 1) * nz), np.full(nr * (nz + 1), -4.0e5)
    peak = 1.0e12
    state = dict(ne=peak * rng.uniform(0.5, 1.5, n), np=peak * rng.uniform(0.5, 1.5, n),
                 nn=0.3 * peak * rng.uniform(0.5, 1.5, n), se=1.0e20 * rng.uniform(0, 1, n),
                 sp=1.0e20 * rng.uniform(0, 1, n), sn=1.0e18 * rng.uniform(0, 1, n))
    state["rho"] = QE * (state["np"] - state["nn"] - state["ne"])
    fcfg = ofl.default_config(ion_drift_enable=1, transport_density_ratio=0.948,
                              electron_ion_recombination_coefficient_m3_per_s=2.0e-13,
                              ion_ion_recombination_coefficient_m3_per_s=2.0e-12)
    fcfg.electron_mobility_model = ofl.MOBILITY_EN_TABLE_FLUX
    fcfg.attachment_model = ofl.ATTACHMENT_EN_TABLE
    ctx = gpu.RreaGpuContext(gpu.default_config(r_hi=nr * dr, z_lo=0.0, z_hi=nz * dz, nr=nr, nz=nz), 1024)
    ctx.set_field(er=er, ez=ez, bt=bt, amb_er=amb_er, amb_ez=amb_ez)
    ctx.fluid_configure(gpu.RreaFluidConfig.from_buffer_copy(bytes(fcfg)))
    ctx.fluid_load_closure(CLOSURE)
    ctx.fluid_set_state(n_pos=state["np"], n_neg=state["nn"], n_e=state["ne"], rho=state["rho"])
    ctx.fluid_set_source_rates(state["se"], state["sp"], state["sn"])
    ctx.reset_current()
    gd = ctx.advance_field_coupled(dt)
    f, st, od = ofl.coupled_step(fcfg, nr, nz, 0.0, dr, dz, dt, (er, ez, bt), (amb_er, amb_ez),
                                 (np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1))), dict(state))
    assert gd["substeps"] == od["substeps"]
    for name, g, o in zip(("er", "ez", "bt"), ctx.field(), f):
        np.testing.assert_allclose(g, o, rtol=0, atol=1e-12 * np.abs(o).max(), err_msg=name)
    gs = ctx.fluid_state()
    for key, okey in (("n_e", "ne"), ("n_pos", "np"), ("n_neg", "nn")):
        np.testing.assert_allclose(gs[key], st[okey], rtol=1e-12, atol=1e-12 * st[okey].max(), err_msg=key)
    np.testing.assert_allclose(gs["rho"], st["rho"], rtol=0, atol=1e-12 * QE * st["ne"].max())
    np.testing.assert_allclose(gs["sigma"], st["sigma"], rtol=1e-12, atol=1e-12 * st["sigma"].max())
    ctx.close()
