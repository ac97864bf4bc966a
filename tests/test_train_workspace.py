"""Workspace of a training-mode forward pass: the gradient passes' one for
small systems, one of its own for large ones, the network kernels' where that
does not fit; energies and forces are the same bits in the first two, the
energies in all three."""
import ctypes

import numpy as np
import pytest
import torch

from mlff_gb300 import _lib

STEP, ALONE, NETWORK = _lib.PATH_TRAIN_TABLE, _lib.PATH_TRAIN_TABLE_FORWARD, _lib.PATH_TUNED_FP32


def sizes(n_atoms, cap, paths=(NETWORK, ALONE, STEP)):
    from mlff_gb300.engine import dims_of
    d = dims_of(128, 20, 3, 119, 5.0)
    return [_lib.load().mlff_workspace_size(ctypes.byref(d), n_atoms, 1, cap, p) for p in paths]


def test_sizes():
    network, alone, step = sizes(100_000, 6_400_000)
    assert network < 2.7e9 and alone < 10.5e9 < 19e9 < step


@pytest.fixture
def engine():
    """An engine without a device that records the paths of its calls."""
    from mlff_gb300.engine import Engine, dims_of
    eng = Engine.__new__(Engine)
    eng.lib, eng.dims = _lib.load(), dims_of(128, 20, 3, 119, 5.0)
    eng.edge_capacity, eng.table_class, eng.short = {}, 2, False
    eng.calls = []

    def energy_forces(batch, path):
        eng.calls.append(path)
        if eng.short and path != NETWORK:
            raise torch.OutOfMemoryError("no room")
        return path

    eng.energy_forces = energy_forces
    return eng


def batch(n):
    from mlff_gb300.engine import make_batch
    return make_batch(np.ones(n), np.zeros((n, 3)), [0, n], device="cpu")


def test_path_of_a_training_step(engine):
    assert engine.train_energy_forces(batch(100)) == STEP
    assert engine.train_energy_forces(batch(20_000)) == STEP
    assert engine.train_energy_forces(batch(24_000)) == ALONE
    engine.edge_capacity[ALONE] = 200 * 20_000          # denser than the default capacity
    assert engine.train_energy_forces(batch(20_000)) == ALONE
    engine.table_class = 1
    assert engine.train_energy_forces(batch(24_000)) == NETWORK
    engine.table_class, engine.short, engine.calls = 2, True, []
    assert engine.train_energy_forces(batch(24_000)) == NETWORK
    assert engine.calls == [ALONE, NETWORK]


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["isolated", "molecules1", "molecules30", "box1503", "box4097"])
def test_layouts_give_the_same_bits(weights_bias, name):
    from test_gpu_table_path import batch_of, model, system
    s = system(name)
    b, eng = batch_of(s), model(weights_bias, "tuned_fp32").engine()
    want = eng.energy_forces(b, STEP, virial=True, graph=False)
    got = eng.energy_forces(b, ALONE, virial=True, graph=False)
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    assert torch.equal(got[0], eng.energy_forces(b, NETWORK, graph=False)[0])


@pytest.mark.gpu
def test_forward_only_call_of_a_large_system(weights_bias):
    from test_gpu_table_path import model
    from mlff_gb300 import systems
    s = systems.large_box(24_000, seed=4)
    m = model(weights_bias, "tuned_fp32").train()
    pos = torch.tensor(s.pos.astype(np.float32), device="cuda")
    m(torch.tensor(s.Z, device="cuda"), pos, cell=torch.tensor(np.diag(s.box[0])), pbc=torch.tensor([True] * 3))
    eng = m.engine()
    assert eng.workspace.numel() == sizes(24_000, eng.capacity(24_000, ALONE), (ALONE,))[0] < 3e9


def test_fp32_call_whose_records_do_not_fit(engine):
    """The table path's workspace is larger than the network kernels'; where
    only theirs fits they run, other paths' shortage is the caller's."""
    del engine.energy_forces
    engine.use_graphs, engine.short = False, True
    table = _lib.PATH_TABLE_FP32
    calls = []

    def eager(b, path, *args):
        calls.append(path)
        if engine.short and path != NETWORK:
            raise torch.OutOfMemoryError("no room")
        return path

    engine._eager_call = eager
    assert engine.energy_forces(batch(5), table) == NETWORK and calls == [table, NETWORK]
    with pytest.raises(torch.OutOfMemoryError):
        engine.energy_forces(batch(5), _lib.PATH_TABLE)
    engine.short = False
    assert engine.energy_forces(batch(5), table) == table
    network, records = sizes(100_000, 6_400_000, (NETWORK, table))
    assert 0 < records - network < 101 * 6_400_000
