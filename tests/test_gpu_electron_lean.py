"""Large electron tiles run the common-history loop and then the full loop
over the electrons it recorded.  At tile sizes from the switch (98304) on,
with ragged last warps:

  * the scale-up population against the oracle, by the phase tests' rule
    (discrete outcomes equal, FP64 state within 1e-12 relative,
    oracle/compare.py);
  * a population that makes every kind of record (events, the cutoff, the
    faces of the domain, energies at the hard-Moller threshold, ended
    particles), with and without a bound density profile, against the same
    electrons in two tiles below the switch, which take the full loop alone:
    outcomes, substeps, draws and secondaries equal, states within 1e-12
    (both loops run the same formulas, a few roundings apart), the sums of the
    deposits within 1e-12 of the largest cell."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods():
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu, workloads
    from oracle import compare, oracle
    build.build()
    oracle.load_tables(TABLES)
    return gpu, workloads, oracle, compare


def _mixed(workloads, cfg, n, seed):
    """Scale-up electrons, a third of them replaced: slow ones around the
    tracking cut and the 50 keV threshold, ones near the domain's faces on
    their way out, and ended ones."""
    rng = np.random.default_rng(seed)
    t = workloads.make_electrons("scaleup_c1", n, seed=seed)
    k = workloads.kinetic_energy(t["ux"], t["uy"], t["uz"])
    kind = rng.integers(0, 12, n)
    k = np.where(kind == 0, rng.uniform(1.0e4, 1.2e5, n), k)
    k = np.where(kind == 1, np.exp(rng.uniform(np.log(1.0001e4), np.log(1.0e6), n)), k)
    scale = workloads.proper_velocity(k) / np.sqrt(t["ux"] ** 2 + t["uy"] ** 2 + t["uz"] ** 2)
    for f in ("ux", "uy", "uz"):
        t[f][:] = t[f] * scale
    out = kind == 2
    t["r"][out] = cfg.r_hi * (1.0 - 10.0 ** rng.uniform(-10, -3, out.sum()))
    top = kind == 3
    t["z"][top] = cfg.z_hi * (1.0 - 10.0 ** rng.uniform(-10, -4, top.sum()))
    t["id"][rng.uniform(size=n) < 0.01] *= -1
    t["w"][:] = rng.uniform(0.5, 2.0, n)
    workloads.capture_prev(t)
    return t


def _setup(gpu, workloads, n):
    cfg = workloads.make_config(gpu, "scaleup_c1")
    ctx = gpu.RreaGpuContext(cfg, n)
    ctx.load_tables(TABLES)
    field = workloads.make_field("scaleup_c1")
    rng = np.random.default_rng(n)
    field["ez"] = rng.normal(0.0, 1.0e3, field["ez"].shape)
    field["bt"] = rng.normal(0.0, 1.0e-6, field["bt"].shape)
    field["bt"].reshape(cfg.nz + 1, cfg.nr + 1)[:, 0] = 0.0
    ctx.set_field(**field)
    return cfg, ctx, field


@pytest.mark.parametrize("n", [3 << 15, (3 << 15) + 33])
def test_large_tile_matches_oracle(mods, n):
    gpu, workloads, oracle, compare = mods
    cfg, ctx, field = _setup(gpu, workloads, n)
    arr = workloads.make_electrons("scaleup_c1", n, seed=6)
    g, o = compare.run_pair(ctx, cfg, field, arr, 3, 5.0e-10)
    problems = compare.compare(cfg, g, o, max(cfg.r_hi, cfg.z_hi))
    ctx.close()
    assert not problems, "; ".join(problems)


@pytest.mark.parametrize("n,profile", [(3 << 15, False), ((3 << 15) + 1, True), (190_003, False)])
def test_large_tile_matches_the_full_loop(mods, n, profile):
    gpu, workloads, oracle, compare = mods
    cfg, ctx, _ = _setup(gpu, workloads, n)
    if profile:
        alt = np.arange(-100.0, 2200.0, 50.0)
        ctx.set_density_profile(alt, 1.225 * np.exp(-alt / 7200.0), 0.0, workloads.TABLE_DENSITY)
    arr = _mixed(workloads, cfg, n, 5)
    runs = []
    for parts in ((slice(0, n),), (slice(0, n // 2), slice(n // 2, n))):
        tiles, secs, diags = [], [], []
        ctx.reset_sources()
        ctx.reset_current()
        for part in parts:
            t = {f: a[part].copy() for f, a in arr.items()}
            sec = ctx.apply_electrons(t, 3, 5.0e-10)
            sec["parent_index"] += part.start
            diags.append(ctx.diagnostics(part.stop - part.start))
            tiles.append(t)
            secs.append(sec)
        runs.append(({f: np.concatenate([t[f] for t in tiles]) for f in arr}, np.concatenate(secs),
                     [np.concatenate(d) for d in zip(*diags)], ctx.sources(), ctx.current()))
    ctx.close()
    (a, sa, da, ca, ja), (b, sb, db, cb, jb) = runs
    np.testing.assert_array_equal(a["id"], b["id"])
    for x, y, name in zip(da, db, ("substeps", "draws", "disposition")):
        np.testing.assert_array_equal(x, y, err_msg=name)
    # every kind of outcome occurs: survival, escape, demotion
    assert all((da[2] == d).sum() > 100 for d in (0, 1, 2))
    assert len(sa) == len(sb) > 1000
    for f in ("species", "process", "parent_index", "root_key", "lineage", "root_species", "weight"):
        np.testing.assert_array_equal(sa[f], sb[f], err_msg=f)
    scale = 1.0e-12 * max(cfg.r_hi, cfg.z_hi)
    for f in ("x", "y", "z"):
        np.testing.assert_allclose(sa[f], sb[f], rtol=0, atol=scale, err_msg=f)
    for f in ("dir_x", "dir_y", "dir_z", "birth_fraction"):
        np.testing.assert_allclose(sa[f], sb[f], rtol=0, atol=1.0e-12, err_msg=f)
    np.testing.assert_allclose(sa["energy_eV"], sb["energy_eV"], rtol=1.0e-12, atol=0)
    for f in ("r", "z"):
        np.testing.assert_allclose(a[f], b[f], rtol=0, atol=scale, err_msg=f)
    u = np.sqrt(b["ux"] ** 2 + b["uy"] ** 2 + b["uz"] ** 2)
    for f in ("ux", "uy", "uz"):
        assert np.all(np.abs(a[f] - b[f]) <= 1.0e-12 * u), f
    for x, y in [(ca[k], cb[k]) for k in range(5)] + [(ja[k], jb[k]) for k in range(2)]:
        assert np.abs(x - y).max() <= 1.0e-12 * max(np.abs(y).max(), 1e-300)
