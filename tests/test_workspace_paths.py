"""Workspace of the plain-FP32 paths: every path that evaluates filters by
pair of atoms has the pair arrays (base [N + 1], edge -> pair [cap], pair ->
edge [cap / 2 + 1]), also the one laid out for the force-loss gradients
(path 4), whose energies and forces run as path 0."""
import ctypes

import pytest
import torch

from mlff_gb300 import _lib


def bytes_per_edge(path):
    """Workspace growth per edge slot at a fixed number of atoms (steps that
    keep every array a multiple of the 256-byte alignment)."""
    from mlff_gb300.engine import dims_of
    lib = _lib.load()
    d = dims_of(128, 20, 3, 119, 5.0)
    a, b = (lib.mlff_workspace_size(ctypes.byref(d), 1024, 4, cap, path) for cap in (1 << 17, 1 << 18))
    assert 0 < a < b and (b - a) % (1 << 17) == 0
    return (b - a) >> 17


def test_pair_arrays_are_laid_out():
    common = bytes_per_edge(_lib.PATH_TUNED_FP32)          # neighbour list and edge sums
    assert common == 3 * 4 + 16
    # geometry, basis and its derivative; z and f of three layers, h, dE/df
    arrays = 16 + 2 * 32 * 4 + 3 * (128 + 384) * 4 + (128 + 384) * 4
    pairs = 4 + 4 // 2
    assert bytes_per_edge(_lib.PATH_PLAIN_FP32) == common + arrays + pairs
    assert bytes_per_edge(_lib.PATH_TRAIN) == common + arrays + pairs
    # (value, tangent) in the float arrays
    assert bytes_per_edge(_lib.PATH_TRAIN_FORCES) == common + 2 * arrays + pairs


@pytest.mark.gpu
@pytest.mark.parametrize("path", [_lib.PATH_TRAIN, _lib.PATH_TRAIN_FORCES])
@pytest.mark.parametrize("name", ["isolated", "molecules7", "water64"])
def test_training_layouts_evaluate_as_the_plain_path(weights_bias, name, path):
    """The same kernels on the same arguments in another layout: the same
    bits."""
    from test_gpu_table_path import batch_of, model, system
    s = system(name)
    b, eng = batch_of(s), model(weights_bias, "fp32").engine()
    want = eng.energy_forces(b, _lib.PATH_PLAIN_FP32, virial=True, graph=False)
    got = eng.energy_forces(b, path, virial=True, graph=False)
    for x, y in zip(got, want):
        assert torch.equal(x, y)
