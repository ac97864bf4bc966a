"""Shape cache of the tensor-core paths on the host: the table form of path 1
(path 5) takes path 1's shape unless it has one of its own."""
import ctypes

import pytest

from mlff_gb300 import _lib

TC, TABLE = _lib.PATH_TUNED_TC, _lib.PATH_TABLE


@pytest.fixture
def lib():
    lib = _lib.load()
    lib.mlff_autotune_reset()
    yield lib
    lib.mlff_autotune_reset()


def shape(lib, path, n_atoms=3000, n_mol=1):
    f, ut = ctypes.c_int32(), ctypes.c_int32()
    assert lib.mlff_autotune_query_shape(path, n_atoms, n_mol, ctypes.byref(f), ctypes.byref(ut)) == _lib.OK
    return f.value, ut.value


def test_table_path_takes_the_shape_set_for_path_1(lib):
    assert shape(lib, TABLE) == (1, 64)
    assert lib.mlff_autotune_set_shape(TC, 3000, 1, 2, 32) == _lib.OK
    assert shape(lib, TC) == shape(lib, TABLE) == (2, 32)
    assert shape(lib, TABLE, 2048) == (1, 64)                                  # another bucket
    assert lib.mlff_autotune_set_shape(TABLE, 3000, 1, 4, 64) == _lib.OK      # its own entry goes first
    assert shape(lib, TC) == (2, 32) and shape(lib, TABLE) == (4, 64)
    assert lib.mlff_autotune_set(TABLE, 3000, 1, 0) == _lib.OK                # removed
    assert shape(lib, TABLE) == (2, 32)
    assert lib.mlff_autotune_set(TABLE, 3000, 1, 4) == _lib.OK                # a factor alone keeps the tile
    assert shape(lib, TABLE) == (4, 32) and shape(lib, TC) == (2, 32)
    assert lib.mlff_autotune_set(TC, 3000, 1, 0) == _lib.OK
    assert shape(lib, TC) == (1, 64) and shape(lib, TABLE) == (4, 32)
    assert lib.mlff_autotune_reset() == _lib.OK
    assert shape(lib, TABLE) == (1, 64)


@pytest.mark.gpu
def test_pinned_shape_reaches_the_model_call(lib, weights_bias):
    """Tuned by the program, then pinned: the model's calls, which the tables
    serve, do not tune over it; the results are the same bits."""
    import torch
    from mlff_gb300 import systems
    from test_gpu_table_path import batch_of, model
    s = systems.molecule_batch(11, 20, 40, seed=6)
    b, m = batch_of(s), model(weights_bias)
    eng = m.engine()
    assert m.path == TABLE
    E0, F0, _ = eng.energy_forces(b, TABLE, graph=False)
    eng.autotune(b, repeats=1)
    assert lib.mlff_autotune_set_shape(TC, b.n_atoms, b.n_mol, 4, 32) == _lib.OK
    for _ in range(2):   # captured, then replayed
        E, F, _ = eng.energy_forces(b, TABLE)
        assert torch.equal(E, E0) and torch.equal(F, F0)
    assert shape(lib, TABLE, b.n_atoms, b.n_mol) == (4, 32)
