"""The reverse pass where the tape that the forward pass leaves holds only the
last segments (it is limited to 8 GiB): one segment kept, two, and all but
one, each with a short last segment.  In turn: twice on the forward's nodes
(the second time the kept tape has been overwritten), then on other nodes and
back, each against the gradient computed from the checkpoints alone; tolerance
as in test_gpu_adjoint_tape.py."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu

ENTRY = 13 * 8   # bytes of one particle's tape entry
LIMIT = 8 << 30


@pytest.mark.parametrize("n,steps,kept", [(420_001, 70, 1), (300_007, 100, 2), (120_003, 180, 5)])
def test_partly_kept_tape(n, steps, kept):
    import torch
    from rrea_feedback_warpx_amrex_geant4_gb300 import adjoint, build
    build.build()
    every, substeps = 32, 4
    segments = -(-steps // every)
    assert min(segments, LIMIT // (n * ENTRY * every * substeps)) == kept < segments and steps % every
    rng = np.random.default_rng(steps)
    mu = rng.uniform(0.6, 1.0, n)
    s, phi = np.sqrt(1.0 - mu * mu), rng.uniform(0.0, 2.0 * np.pi, n)
    seeds = dict(z=rng.uniform(0.0, 5.0, n), dir=np.stack([s * np.cos(phi), s * np.sin(phi), mu], 1),
                 k=np.exp(rng.uniform(np.log(3.0e5), np.log(2.0e7), n)), w=rng.uniform(0.5, 2.0, n),
                 id=np.arange(1, n + 1, dtype=np.uint64))
    cfg = adjoint.default_config(steps=steps, substeps=substeps, checkpoint_every=every, k_threshold_eV=8.0e6,
                                 k_width_eV=1.0e6, z_plane_m=8.0)
    prob = adjoint.PushAdjoint(cfg, seeds, tables=TABLES)
    e1 = torch.tensor(adjoint.adjoint_field_profile(), dtype=torch.float64, device="cuda")
    e2 = e1 * 1.0001

    def recomputed(nodes):
        prob.forward(e1)
        prob.forward(e1, frozen=True)   # leaves no tape
        return prob.backward(nodes)

    want1, want2 = recomputed(e1), recomputed(e2)
    prob.forward(e1)
    got = [prob.backward(e1), prob.backward(e1), prob.backward(e2), prob.backward(e1)]
    prob.forward(e1)
    got += [prob.backward(e2), prob.backward(e1)]
    assert float(want1.abs().max()) > 0.0
    for g, w in zip(got, (want1, want1, want2, want1, want2, want1)):
        np.testing.assert_allclose(g.cpu(), w.cpu(), rtol=0, atol=1e-12 * float(w.abs().max()))
    prob.close()
