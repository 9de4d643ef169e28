"""The reverse pass from the tape that the forward pass left against the one
that computes its segments again from the checkpoints: one segment and
several, a last one cut short, one step per segment; twice in a row; and with
other nodes than the forward pass had, where the tape must not be used.

The two run the same arithmetic on the same states; the compiler may contract
it differently in the two kernels, so the states differ by a few roundings a
substep, some hundred over a run: 1e-12 of the largest gradient."""
import numpy as np
import pytest

from conftest import TABLES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps,every,n", [(10, 4, 2003), (7, 32, 65), (9, 1, 700), (12, 6, 1)])
def test_taped_and_recomputed_gradients_agree(steps, every, n):
    import torch
    from rrea_feedback_warpx_amrex_geant4_gb300 import adjoint, build
    build.build()
    rng = np.random.default_rng(steps)
    mu = rng.uniform(0.6, 1.0, n)
    mu[::10] *= -1.0
    s = np.sqrt(1.0 - mu * mu)
    phi = rng.uniform(0.0, 2.0 * np.pi, n)
    seeds = dict(z=rng.uniform(0.0, 5.0, n), dir=np.stack([s * np.cos(phi), s * np.sin(phi), mu], 1),
                 k=np.exp(rng.uniform(np.log(3.0e5), np.log(2.0e7), n)), w=rng.uniform(0.5, 2.0, n),
                 id=np.arange(1, n + 1, dtype=np.uint64))
    cfg = adjoint.default_config(steps=steps, substeps=3, checkpoint_every=every, k_threshold_eV=8.0e6,
                                 k_width_eV=1.0e6, z_plane_m=3.0)
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
    assert float(want1.abs().max()) > 0.0
    for g, w in zip(got, (want1, want1, want2, want1)):
        np.testing.assert_allclose(g.cpu(), w.cpu(), rtol=0, atol=1e-12 * float(w.abs().max()))
    prob.close()
