"""The hand-over from the common-history loop to the full one, beyond
test_gpu_electron_lean.py: the mixed population there as positrons (events of
all three channels, annihilation at rest at the cutoff, escapes, ended
particles, varied weights), with and without a bound density profile, and as
electrons at every register variant and block size of the launch, each
against the same particles in two tiles below the switch, which take the full
loop alone.

Outcomes, substeps, draws and secondaries' keys equal; states within 1e-12; a
secondary's energy within 1e-12 of it or of its parent's energy, its direction
within 1e-12 times the parent's energy over its own momentum (the phase tests'
rule for differences of parent-scale quantities, oracle/compare.py); the sums
of the deposits within 1e-12 of the largest cell."""
import numpy as np
import pytest

from test_gpu_electron_lean import _mixed, _setup, mods  # noqa: F401

pytestmark = pytest.mark.gpu

ME_C2 = 510998.95


def _compare_with_full_loop(workloads, ctx, cfg, arr, species, launch=(128, 16)):
    n = len(arr["id"])
    apply = ctx.apply_positrons if species == "positron" else ctx.apply_electrons
    parent = workloads.kinetic_energy(arr["ux"], arr["uy"], arr["uz"]) + (2.0 * ME_C2 if species == "positron" else 0.0)
    runs = []
    for parts in ((slice(0, n),), (slice(0, n // 2), slice(n // 2, n))):
        ctx.set_launch(*launch)
        tiles, secs, diags = [], [], []
        ctx.reset_sources()
        ctx.reset_current()
        for part in parts:
            t = {f: a[part].copy() for f, a in arr.items()}
            sec = apply(t, 3, 5.0e-10)
            sec["parent_index"] += part.start
            diags.append(ctx.diagnostics(part.stop - part.start))
            tiles.append(t)
            secs.append(sec)
        runs.append(({f: np.concatenate([t[f] for t in tiles]) for f in arr}, np.concatenate(secs),
                     [np.concatenate(d) for d in zip(*diags)], ctx.sources(), ctx.current()))
        launch = (128, 16)
    (a, sa, da, ca, ja), (b, sb, db, cb, jb) = runs
    np.testing.assert_array_equal(a["id"], b["id"])
    for x, y, name in zip(da, db, ("substeps", "draws", "disposition")):
        np.testing.assert_array_equal(x, y, err_msg=name)
    # every kind of outcome occurs: survival, escape, the end at the cutoff
    assert all((da[2] == d).sum() > 100 for d in (0, 1, 2))
    assert len(sa) == len(sb) > 1000
    for f in ("species", "process", "parent_index", "root_key", "lineage", "root_species", "weight"):
        np.testing.assert_array_equal(sa[f], sb[f], err_msg=f)
    scale = 1.0e-12 * max(cfg.r_hi, cfg.z_hi)
    for f in ("x", "y", "z"):
        np.testing.assert_allclose(sa[f], sb[f], rtol=0, atol=scale, err_msg=f)
    np.testing.assert_allclose(sa["birth_fraction"], sb["birth_fraction"], rtol=0, atol=1.0e-12)
    e = sb["energy_eV"]
    pe = np.maximum(parent[sb["parent_index"]], e)
    assert (np.abs(sa["energy_eV"] - e) <= 1.0e-12 * pe).all()
    p = np.where(sb["species"] == 2, e, np.sqrt(e * (e + 2.0 * ME_C2)))
    for f in ("dir_x", "dir_y", "dir_z"):
        assert (np.abs(sa[f] - sb[f]) <= 1.0e-12 * np.maximum(1.0, pe / p)).all(), f
    for f in ("r", "z"):
        np.testing.assert_allclose(a[f], b[f], rtol=0, atol=scale, err_msg=f)
    u = np.sqrt(b["ux"] ** 2 + b["uy"] ** 2 + b["uz"] ** 2)
    for f in ("ux", "uy", "uz"):
        assert np.all(np.abs(a[f] - b[f]) <= 1.0e-12 * u), f
    for x, y in [(ca[k], cb[k]) for k in range(5)] + [(ja[k], jb[k]) for k in range(2)]:
        assert np.abs(x - y).max() <= 1.0e-12 * max(np.abs(y).max(), 1e-300)
    return sa


@pytest.mark.parametrize("n,profile", [(3 << 15, False), ((3 << 15) + 1, True), (190_003, False)])
def test_mixed_positrons_match_the_full_loop(mods, n, profile):  # noqa: F811
    gpu, workloads, oracle, compare = mods
    cfg, ctx, _ = _setup(gpu, workloads, n)
    if profile:
        alt = np.arange(-100.0, 2200.0, 50.0)
        ctx.set_density_profile(alt, 1.225 * np.exp(-alt / 7200.0), 0.0, workloads.TABLE_DENSITY)
    sec = _compare_with_full_loop(workloads, ctx, cfg, _mixed(workloads, cfg, n, 7), "positron")
    ctx.close()
    # Bhabha electrons, bremsstrahlung and annihilation photons
    assert len(np.unique(sec["process"])) >= 3


@pytest.mark.parametrize("launch", [(128, 2), (128, 4), (128, 8), (128, 12), (64, 32), (32, 32)])
def test_launch_shapes_match_the_full_loop(mods, launch):  # noqa: F811
    gpu, workloads, oracle, compare = mods
    n = (3 << 15) + 33
    cfg, ctx, _ = _setup(gpu, workloads, n)
    _compare_with_full_loop(workloads, ctx, cfg, _mixed(workloads, cfg, n, 9), "electron", launch)
    ctx.close()
