"""A photon's resident flight without an interaction against extended
precision: the straight push from (r, theta, z) and the end point's radius
and angle.  Angles on the 256 steps of the sine table, half way between two,
at 0, +-pi/2 and +-pi and many turns on; flights along, across and through the
axis, and from it.

The start's sine and cosine are within 2^-52, the products and the push round
three more times: the end point is within 4 x 2^-52 x (r + path) of the exact
one, its radius within that and two roundings, its angle within that over the
radius and two ulps of pi (beyond a turn the angle's own argument is exact)."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu

C = 299792458.0


@pytest.mark.parametrize("kind", ["random", "steps", "axis", "turns"])
def test_flight_matches_extended_precision(kind):
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu, workloads
    build.build()
    rng = np.random.default_rng(7)
    n, dt = 20_011, 5.0e-10
    cfg = workloads.make_config(gpu, "scaleup_c1")
    tile = workloads.make_photons("scaleup_c1", n, dt, seed=3, e_lo=2.0e5, e_hi=1.0e7)
    r = rng.uniform(0.0, 0.9, n) ** 2 * cfg.r_hi
    th = rng.uniform(-np.pi, np.pi, n)
    phi = rng.uniform(-np.pi, np.pi, n)
    if kind == "steps":
        th = (rng.integers(-256, 257, n) / 256.0 * np.pi) + np.where(rng.uniform(size=n) < 0.5, 0.0, 1e-15)
        th[:6] = [0.0, -0.0, np.pi / 2, -np.pi / 2, np.pi, -np.pi]
    elif kind == "axis":
        r[::2] = rng.uniform(0.0, 0.2, n)[::2]
        r[::16] = 0.0
        phi = np.where(rng.uniform(size=n) < 0.5, th + np.pi, th)
    elif kind == "turns":
        th = th + 2.0 * np.pi * rng.integers(-400, 401, n)
    z = cfg.z_lo + rng.uniform(0.05, 0.95, n) * (cfg.z_hi - cfg.z_lo)
    mu = rng.uniform(-1.0, 1.0, n)
    e = np.exp(rng.uniform(np.log(2.0e5), np.log(1.0e7), n))
    st = np.sqrt(1.0 - mu * mu)
    ux, uy, uz = e * st * np.cos(phi), e * st * np.sin(phi), e * mu
    for name, v in (("r", r), ("theta", th), ("z", z), ("ux", ux), ("uy", uy), ("uz", uz)):
        tile[name][:] = v
        tile["prev_" + name][:] = v
    ctx = gpu.RreaGpuContext(cfg, 1 << 15)
    ctx.load_tables(TABLES)
    ctx.set_field(**workloads.make_field("scaleup_c1"))
    ctx.stage_photons(tile)
    ctx.step_photons_resident(1, dt)
    out = {k: np.zeros_like(v) for k, v in tile.items()}
    ctx.fetch_photons(out)
    ctx.close()
    L = np.longdouble
    u = np.sqrt(L(ux) ** 2 + L(uy) ** 2 + L(uz) ** 2)
    path = L(C) * L(dt)
    x = L(r) * np.cos(L(th)) + path * L(ux) / u
    y = L(r) * np.sin(L(th)) + path * L(uy) / u
    zz = L(z) + path * L(uz) / u
    keep = (out["id"] > 0) & (out["ux"] == ux) & (out["uy"] == uy)   # no interaction on the way
    assert keep.sum() > 0.9 * n
    eps = 2.0 ** -52
    near = 4.0 * eps * (r + float(path))
    rr = np.hypot(x, y).astype(np.longdouble)
    assert (np.abs(out["r"] - rr)[keep] <= (near + 2.0 * eps * rr)[keep]).all()
    assert (np.abs(out["z"] - zz)[keep] <= (4.0 * eps * (np.abs(z) + float(path)))[keep]).all()
    dth = np.abs(out["theta"] - np.arctan2(y, x))
    dth = np.minimum(dth, np.abs(dth - 2.0 * L(np.pi)))
    far = keep & (rr > 0.0)
    assert (dth[far] <= (near / np.maximum(rr, 1e-300) + 2.0 * eps * np.pi)[far]).all()
    assert (np.abs(out["theta"])[keep] <= np.pi).all()
