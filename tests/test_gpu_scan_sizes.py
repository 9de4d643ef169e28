"""Ranks by the one-block scan and by the three-pass scan around the length
where they meet (8192 counts) and around a block's 1024: the commit of drain
survivors ranks three rows of n records as one row of 3 n, the compaction
ranks n rows.  Both only copy and count, so everything is equal."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu


def _ctx(capacity):
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu, workloads
    build.build()
    ctx = gpu.RreaGpuContext(workloads.make_config(gpu, "uniform_c0"), capacity)
    ctx.load_tables(TABLES)
    ctx.set_field(**workloads.make_field("uniform_c0"))
    return gpu, workloads, ctx


def _fetch(workloads, ctx, fetch, n):
    out = {k: np.zeros(n, v.dtype) for k, v in workloads.make_electrons("uniform_c0", 1, seed=1).items()}
    fetch(out)
    return out


@pytest.mark.parametrize("n", [1, 341, 342, 2730, 2731, 20_001])
def test_commit_keeps_record_order(n):
    gpu, workloads, ctx = _ctx(1 << 15)
    rng = np.random.default_rng(n)
    rec = np.zeros(n, dtype=gpu.SECONDARY_DTYPE)
    rec["species"] = rng.integers(0, 3, n)
    rec["root_key"], rec["lineage"] = rng.integers(1, 1 << 30, n), np.arange(n) % 4096
    cfg = ctx.config
    rec["x"], rec["z"] = rng.uniform(0.1, 0.9, n) * cfg.r_hi, cfg.z_lo + rng.uniform(0.1, 0.9, n) * (cfg.z_hi - cfg.z_lo)
    rec["dir_z"], rec["energy_eV"], rec["birth_fraction"] = 1.0, rng.uniform(2.0e5, 2.0e6, n), 1.0
    rec["weight"] = 1.0 + np.arange(n)
    surv = ctx.drain_secondaries(rec, 1, 5.0e-10)
    np.testing.assert_array_equal(surv["weight"], rec["weight"])
    added = ctx.commit_survivors_resident()
    for species, fetch in enumerate((ctx.fetch_electrons, ctx.fetch_positrons, ctx.fetch_photons)):
        want = rec[rec["species"] == species]
        assert added[species] == len(want)
        if len(want) == 0:
            continue
        got = _fetch(workloads, ctx, fetch, len(want))
        for key, w in (("w", want["weight"]), ("z", want["z"]), ("r", want["x"])):
            np.testing.assert_array_equal(got[key], w, err_msg=f"{species} {key}")
        np.testing.assert_array_equal(np.diff(got["id"]), np.ones(len(want) - 1, dtype=np.int64))
    ctx.close()


@pytest.mark.parametrize("n", [1, 1023, 1025, 8192, 8193, 33_000])
def test_compaction_keeps_row_order(n):
    gpu, workloads, ctx = _ctx(1 << 16)
    e = workloads.make_electrons("uniform_c0", n, seed=n)
    dead = np.random.default_rng(n).uniform(size=n) < 0.4
    e["id"] = np.where(dead, -np.abs(e["id"]), np.abs(e["id"]))
    ctx.stage_electrons(e)
    live = ctx.compact_resident(0)
    assert live == int((~dead).sum())
    if live:
        got = _fetch(workloads, ctx, ctx.fetch_electrons, int(live))
        for key in ("r", "z", "theta", "ux", "uy", "uz", "id"):
            np.testing.assert_array_equal(got[key], e[key][~dead], err_msg=key)
    ctx.close()
