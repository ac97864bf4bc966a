"""Weights packed anew between calls that hold a captured graph: filters
sharper than the tables resolve (accuracy class 0) move a captured table path
back to the network kernels."""
import numpy as np
import pytest
import torch

from test_gpu_table_path import batch_of, model

pytestmark = pytest.mark.gpu


def sharpen(m):
    """Filters of accuracy class 0."""
    with torch.no_grad():
        for blk in m.interactions:
            blk.message.rbf_to_scalar[0].weight.mul_(20.0)
    assert m.engine().table_class == 0


@pytest.mark.parametrize("precision", ["fp16x3", "tuned_fp32"])
def test_md_goes_on_with_weights_the_tables_do_not_serve(weights_bias, precision):
    """Replayed blocks of steps give the eager steps' bits before and after."""
    from mlff_gb300 import _lib, systems
    from mlff_gb300.md import VelocityVerletGPU
    s = systems.molecule_batch(3, 20, 40, seed=6)
    m = model(weights_bias, precision)
    assert m.engine().table_class == 2
    runs = [VelocityVerletGPU(m, s.Z, s.pos, s.mol_ptr, timestep_fs=0.05) for _ in range(2)]
    assert runs[0].path in (_lib.PATH_TABLE, _lib.PATH_TABLE_FP32)
    first = [d.run(10, graph=g, block=5) for d, g in zip(runs, (True, False))]
    sharpen(m)
    second = [d.run(10, graph=g, block=5) for d, g in zip(runs, (True, False))]
    for a, b in (first, second):
        np.testing.assert_array_equal(a["potential_energy"], b["potential_energy"])
    np.testing.assert_array_equal(runs[0].positions(), runs[1].positions())
    assert not np.array_equal(first[0]["potential_energy"][-1], second[0]["potential_energy"][0])


@pytest.mark.parametrize("precision", ["fp16x3", "tuned_fp32"])
def test_captured_call_follows_the_weights(weights_bias, precision):
    """Engine.capture's replay refreshes the same two tensors with the
    results of the weights packed last."""
    from mlff_gb300 import _lib, systems
    s = systems.molecule_batch(3, 20, 40, seed=6)
    b = batch_of(s)
    m = model(weights_bias, precision)
    eng = m.engine()
    path, network = ((_lib.PATH_TABLE, _lib.PATH_TUNED_TC) if precision == "fp16x3" else
                     (_lib.PATH_TABLE_FP32, _lib.PATH_TUNED_FP32))
    assert m.path == path
    replay, E, F = eng.capture(b, path)
    old = {k: v.clone() for k, v in m.state_dict().items()}
    for change, now in ((None, path), (sharpen, network), (lambda m: m.load_state_dict(old), path)):
        if change is not None:
            change(m)
            m.engine()
        replay()
        replay()
        E0, F0, _ = eng.energy_forces(b, now, graph=False)
        assert torch.equal(E, E0) and torch.equal(F, F0)
