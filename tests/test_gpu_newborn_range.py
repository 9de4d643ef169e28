"""A newborn whose residual step ends above the tables' highest charged energy
is refused as out of range, like one that passes it on the way, whichever of
its substeps it is: positrons and electrons born just below 10 GeV in a field
that carries them over.  The same birth a little lower survives."""
import numpy as np
import pytest

from test_gpu_newborn import _pending, mods  # noqa: F401
from conftest import TABLES

pytestmark = pytest.mark.gpu

TOP_EV = 1.0e10


@pytest.mark.parametrize("species", [0, 1])
def test_leaving_the_certified_range_is_refused(mods, species):  # noqa: F811
    gpu, workloads, oracle, compare = mods
    cfg = workloads.make_config(gpu, "scaleup_c1")
    field = workloads.make_field("scaleup_c1")
    field["amb_ez"] = np.full_like(field["amb_ez"], 1.0e7 if species == 1 else -1.0e7)
    ctx = gpu.RreaGpuContext(cfg, 4096)
    ctx.load_tables(TABLES)
    ctx.set_field(**field)
    dt_s = 2.0e-9
    rec = _pending(workloads, oracle, cfg, workloads.make_field("scaleup_c1"), "scaleup_c1", 64, 3, dt_s)[:1].copy()
    rec["species"], rec["energy_eV"], rec["birth_fraction"] = species, 0.0, 0.5
    rec["x"], rec["y"], rec["z"] = 0.0, 0.0, 1.0
    rec["dir_x"], rec["dir_y"], rec["dir_z"] = 0.0, 0.0, 1.0
    refused = survived = 0
    for lack in np.linspace(1.0e5, 4.0e6, 40):   # the residual's work is 3 MeV
        rec["energy_eV"] = TOP_EV - lack
        try:
            oracle.drain(cfg, field, 3, dt_s, rec)
        except oracle.OracleFailure as e:
            with pytest.raises(gpu.RreaGpuError) as info:
                ctx.drain_secondaries(rec, 3, dt_s)
            assert info.value.status == e.code, lack
            refused += 1
        else:
            ctx.drain_secondaries(rec, 3, dt_s)
            survived += 1
    ctx.close()
    assert refused > 10 and survived > 5
