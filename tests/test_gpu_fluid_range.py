"""The closure's cell fields and the diffusion tensor's check at field
magnitudes and tensor entries whose squares leave the range of doubles, where
|E| is hypot's and the direction E / |E|: subnormal fields up to 1e307 V/m,
against the oracle (the reference's hypot and divisions) cell by cell.
Tolerances as in test_gpu_fluid.py: 1e-13 relative, the tensor's 1e-13 of its
largest entry (in range, all entries are of one size), counts exact."""
import os

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CLOSURE = os.path.join(ROOT, "data", "closure", "dry_air_swarm_hybrid_v3.csv")


@pytest.mark.parametrize("log10_lo,log10_hi", [(-320, -290), (-200, -140), (-80, 2), (3, 4.5), (140, 200), (290, 307)])
def test_closure_fields_over_the_range_of_doubles(log10_lo, log10_hi):
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu
    from oracle import fluid as ofl
    build.build()
    ofl.load_closure(CLOSURE)
    rng = np.random.default_rng(int(log10_hi) + 400)
    nr, nz, dr, dz = 33, 9, 2.0, 3.0
    n = nr * nz
    phi = rng.uniform(-np.pi, np.pi, n)
    mag = 10.0 ** rng.uniform(log10_lo, log10_hi, n)
    er, ez = mag * np.cos(phi), mag * np.sin(phi)
    er[:3], ez[:3] = [mag[0], 0.0, -mag[2]], [0.0, -mag[1], 0.0]
    if log10_hi == 2:
        er[3] = ez[3] = 0.0
    ne, src = 1.0e12 * rng.uniform(0.5, 1.5, n), 1.0e20 * rng.uniform(0.0, 1.0, n)
    ctx = gpu.RreaGpuContext(gpu.default_config(r_hi=nr * dr, z_lo=0.0, z_hi=nz * dz, nr=nr, nz=nz), 1024)
    ctx.fluid_configure(electron_mobility_model=gpu.MOBILITY_EN_TABLE_FLUX, attachment_model=gpu.ATTACHMENT_EN_TABLE)
    ctx.fluid_load_closure(CLOSURE)
    ctx.fluid_set_state(n_e=ne)
    ctx.fluid_set_source_rates(s_e=src)
    d = ctx.fluid_evaluate_closure(er, ez)
    mu, nu, d3 = ctx.fluid_closure_fields()
    ctx.close()
    w_mu, w_nu, w_d3, diag = ofl.closure_fields(nr, nz, 0.0, 0.0, dr, dz, er, ez, ne=ne, src=src)
    np.testing.assert_allclose(mu, w_mu, rtol=1e-13, atol=0)
    np.testing.assert_allclose(nu, w_nu, rtol=1e-13, atol=0)
    np.testing.assert_allclose(d3, w_d3, rtol=1e-13, atol=1e-13 * np.abs(w_d3).max())
    assert (d["held_below"], d["above_range"], d["invalid"]) == tuple(diag[2:5])
    assert d["min_en_td"] == pytest.approx(diag[0], rel=4e-15)
    assert d["max_en_td"] == pytest.approx(diag[1], rel=4e-15)


@pytest.mark.parametrize("scale", [1.0e-290, 1.0e-170, 1.0, 1.0e160])
def test_diffusion_number_over_the_range_of_doubles(scale):
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu
    from oracle import fluid as ofl
    build.build()
    rng = np.random.default_rng(5)
    nr, nz, dr, dz, dt = 33, 9, 2.0, 3.0, 1.0e-9
    n, zero = nr * nz, np.zeros(nr * nz)
    rr, zz = rng.uniform(0.5, 1.0, (2, n)) * scale
    d3 = np.stack([rr, 0.4 * scale * rng.uniform(-1.0, 1.0, n), zz])
    ctx = gpu.RreaGpuContext(gpu.default_config(r_hi=nr * dr, z_lo=0.0, z_hi=nz * dz, nr=nr, nz=nz), 1024)
    fcfg = ofl.default_config()
    fcfg.electron_mobility_model = ofl.MOBILITY_EN_TABLE_FLUX
    ctx.fluid_configure(gpu.RreaFluidConfig.from_buffer_copy(bytes(fcfg)))
    ctx.fluid_load_closure(CLOSURE)
    ctx.fluid_set_state(n_pos=zero, n_neg=zero, n_e=zero, rho=zero)
    ctx.fluid_set_closure_fields(mu=zero, diffusion=d3)
    faces = np.zeros((nr + 1) * nz), np.zeros(nr * (nz + 1))
    if scale > 1.0e100:   # far past the explicit update's bound
        with pytest.raises(gpu.RreaGpuError):
            ctx.fluid_transport(dt, *faces)
        ctx.close()
        return
    got = ctx.fluid_transport(dt, *faces)[2]
    ctx.close()
    want = ofl.transport(fcfg, (nr, nz, 0.0, 0.0, dr, dz, 0), dt, zero, zero, zero, zero, *faces, mu=zero,
                         diffusion=d3)["diag"]["max_diffusion_number"]
    assert want > 0.0
    assert got["max_diffusion_number"] == pytest.approx(want, rel=4e-15)
