"""The newborn kernels at the queue lengths where the items per warp change
(one per warp up to 4 per SM, then doubling) and past the last doubling,
where warps loop: the drain of that many records against the oracle's.
Tolerances as in test_gpu_newborn.py."""
import numpy as np
import pytest

from test_gpu_newborn import _compare_cells, _compare_survivors, _pending, _setup, mods  # noqa: F401

pytestmark = pytest.mark.gpu

SMS = 152


@pytest.mark.parametrize("n", [1, 31, 4 * SMS, 4 * SMS + 1, 8 * SMS + 1, 128 * SMS + 33, 32 * SMS, 32 * SMS + 1, 64 * SMS + 1, 1024 * SMS + 33])
def test_drain_lengths_match_oracle(mods, n):  # noqa: F811
    gpu, workloads, oracle, compare = mods
    cfg, ctx, field = _setup(gpu, workloads, "scaleup_c1", 1 << 18)
    step, dt_s = 3, 2.0e-9
    pending = np.resize(_pending(workloads, oracle, cfg, field, "scaleup_c1", 4096, step, dt_s), n)
    ctx.reset_sources()
    got = ctx.drain_secondaries(pending, step, dt_s)
    o = oracle.drain(cfg, field, step, dt_s, pending)
    _compare_survivors(compare, cfg, got, o["survivors"])
    _compare_cells(compare, ctx.sources(), o["cells"])
    ctx.close()
