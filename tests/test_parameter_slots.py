"""The model's parameter slots on the CPU: the names and order of
named_parameters, a replaced submodule, and no cycle that would keep a model
(and its GPU workspace) alive."""
import gc
import weakref

from torch import nn


def test_slots():
    from mlff_gb300.student_model import StudentForceField, _trainable
    m = StudentForceField()
    m.embedding.weight.requires_grad_(False)
    names = [n for n, p in m.named_parameters() if p.requires_grad]
    assert [n for n, _ in _trainable(m, True)] == names
    m.energy_head[0] = nn.Linear(128, 64)
    now = {n: p for n, p in _trainable(m, True)}
    assert now["energy_head.0.weight"] is m.energy_head[0].weight
    gc.collect()
    gc.disable()
    try:
        ref = weakref.ref(m)
        del m, now
        assert ref() is None
    finally:
        gc.enable()
