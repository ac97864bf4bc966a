"""The FP32 path's filters by pair of atoms against its evaluation by
directed edge (what the parameter gradients need): atoms without edges, one
pair, odd batches, periodic boxes.

Tolerance: the forward pass is the same arithmetic (equal energies); the
reverse pass adds the two directions of a pair before the filter's GEMMs
instead of after, sums of up to 384 terms of FP32: 384^0.5 * 6e-8 = 1.2e-6 of
the forces' 2-norm per layer, 1e-5 asked for three."""
import numpy as np
import pytest
import torch

from test_gpu_table_path import batch_of, model, rel, system

pytestmark = pytest.mark.gpu


def cluster(n, spread):
    from mlff_gb300 import systems
    rng = np.random.default_rng(n)
    pos = spread * np.stack([np.arange(n), rng.random(n), rng.random(n)], 1)
    return systems.System(np.full(n, 6), pos, np.array([0, n]), np.zeros((1, 3)), np.zeros(1, bool))


@pytest.mark.parametrize("name", ["one", "apart", "pair", "isolated", "molecules1", "molecules7", "water64", "box1503"])
def test_pairs_match_directed_edges(weights_bias, name):
    from mlff_gb300 import _lib
    from mlff_gb300.training import param_grads
    s = {"one": lambda: cluster(1, 1.0), "apart": lambda: cluster(2, 20.0), "pair": lambda: cluster(2, 1.1)}.get(
        name, lambda: system(name))()
    b, m = batch_of(s), model(weights_bias, "fp32")
    E, F, _ = m.engine().energy_forces(b, _lib.PATH_PLAIN_FP32, graph=False)
    E0, _, F0 = param_grads(m, b, torch.ones(s.n_mol), forces=True)
    assert torch.equal(E, E0)
    assert float(F0.norm()) == 0.0 or rel(F, F0) < 1e-5
    assert (float(F.norm()) == 0.0) == (float(F0.norm()) == 0.0)


@pytest.mark.parametrize("name", ["one", "apart", "pair", "isolated", "molecules1", "molecules7", "water64", "box1503"])
def test_training_forward_keeps_the_fused_fp32_bits(weights_bias, name):
    """The forward pass of a training step on pairs against the fused FP32
    kernels' (equal energies); forces with the tables' 2e-5."""
    from mlff_gb300 import _lib
    s = {"one": lambda: cluster(1, 1.0), "apart": lambda: cluster(2, 20.0), "pair": lambda: cluster(2, 1.1)}.get(
        name, lambda: system(name))()
    b, eng = batch_of(s), model(weights_bias, "tuned_fp32").engine()
    E, F, _ = eng.energy_forces(b, _lib.PATH_TRAIN_TABLE, graph=False)
    E0, F0, _ = eng.energy_forces(b, _lib.PATH_TUNED_FP32, graph=False)
    assert torch.equal(E, E0)
    assert float((F - F0).norm()) <= 2e-5 * float(F0.norm())
