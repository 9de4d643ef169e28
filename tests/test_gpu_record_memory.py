"""Device memory of a context that cannot run the common-history loop: its
records (88 bytes a slot) are not allocated in a periodic domain (which has no
net-chord segments either, 64 bytes a slot), nor below the tile size from
which the loop runs."""
import pytest

pytestmark = pytest.mark.gpu

RECORD, SEGMENT = 88, 64


def _bytes_held(gpu, capacity, periodic):
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    ctx = gpu.RreaGpuContext(gpu.default_config(periodic_z=periodic), capacity)
    held = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    return held


def test_records_only_where_the_loop_runs():
    from rrea_feedback_warpx_amrex_geant4_gb300 import build, gpu
    build.build()
    _bytes_held(gpu, 1 << 16, 0)   # the module and its first-use allocations
    n = 1 << 22
    assert _bytes_held(gpu, n, 0) - _bytes_held(gpu, n, 1) >= (RECORD + SEGMENT) * n - (1 << 22)
    small = 3 << 15
    # one slot more than the switch's predecessor brings the whole record array
    assert _bytes_held(gpu, small, 0) - _bytes_held(gpu, small - 1, 0) >= RECORD * small - (1 << 22)
