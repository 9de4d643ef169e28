"""Large positron tiles run the common-history loop and then the full loop over
the positrons it recorded: the scale-up distribution as positrons against the
oracle from the switch on, with a ragged last warp, by the phase tests' rule."""
import pytest

from test_gpu_electron_lean import _setup, mods  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3 << 15, (3 << 15) + 33])
def test_large_positron_tile_matches_oracle(mods, n):  # noqa: F811
    gpu, workloads, oracle, compare = mods
    cfg, ctx, field = _setup(gpu, workloads, n)
    arr = workloads.make_electrons("scaleup_c1", n, seed=8)
    g, o = compare.run_pair(ctx, cfg, field, arr, 3, 5.0e-10, species="positron")
    e0 = workloads.kinetic_energy(arr["ux"], arr["uy"], arr["uz"])
    problems = compare.compare(cfg, g, o, max(cfg.r_hi, cfg.z_hi), parent_energy=e0 + 1.022e6)
    ctx.close()
    assert not problems, "; ".join(problems)
