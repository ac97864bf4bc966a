"""What the engine is given to pack, on the CPU (the engine replaced by a
recorder): the weights that the model holds at the call, also after a
submodule was replaced in eval mode.  On the GPU: the energies follow."""
import numpy as np
import pytest
import torch
from torch import nn


class OnCuda(nn.Parameter):
    """A host parameter that reports a CUDA device."""
    @property
    def device(self):
        return torch.device("cuda", 0)


class Recorder:
    def __init__(self, dims, device):
        self.device, self.packs = device, []

    def pack(self, sd):
        self.packs.append({k: v.detach().clone() for k, v in sd.items()})


@pytest.fixture
def model(monkeypatch):
    from mlff_gb300 import student_model
    monkeypatch.setattr(student_model, "Engine", Recorder)
    torch.manual_seed(3)
    m = student_model.StudentForceField().eval()
    m.embedding.weight = OnCuda(m.embedding.weight.data)
    return m


def assert_packed(m, n_packs):
    packs = m.engine().packs
    assert len(packs) == n_packs
    for k, v in m.state_dict().items():
        assert torch.equal(packs[-1][k], v), k
    m.engine()
    assert len(packs) == n_packs      # nothing changed since


def test_replaced_submodule_is_packed(model):
    assert_packed(model, 1)
    model.energy_head[0] = nn.Linear(128, 64)
    assert_packed(model, 2)
    ckpt = {k: v + 0.25 for k, v in model.state_dict().items()}
    model.load_state_dict(ckpt)
    assert_packed(model, 3)
    model.interactions[1].update.update_mlp = type(model)(num_interactions=1).interactions[0].update.update_mlp
    assert_packed(model, 4)
    model.rbf = type(model)(learnable_rbf=True).rbf
    with torch.no_grad():
        model.rbf.centers.add_(0.125)
    assert_packed(model, 5)


def energies(m):
    from mlff_gb300 import systems
    s = systems.lattice_molecule(30, seed=7)
    with torch.no_grad():
        return m(torch.tensor(s.Z, device="cuda"), torch.tensor(s.pos.astype(np.float32), device="cuda"))


@pytest.mark.gpu
def test_energies_follow_a_replaced_submodule():
    from mlff_gb300.student_model import StudentForceField
    torch.manual_seed(3)
    m = StudentForceField().cuda().eval()
    e = energies(m)
    m.energy_head[0] = nn.Linear(128, 64).cuda()
    other = StudentForceField().cuda().eval()
    other.load_state_dict(m.state_dict())
    got = energies(m)
    assert not torch.equal(got, e) and torch.equal(got, energies(other))


def test_shared_blocks_are_packed_under_both_names(model):
    model.interactions[1] = model.interactions[0]
    assert_packed(model, 1)
    with torch.no_grad():
        model.interactions[1].update.mixing_matrix.add_(1.0)
    assert_packed(model, 2)


def test_shared_blocks_train_once():
    """named_parameters() lists a shared parameter once."""
    from mlff_gb300.student_model import StudentForceField, _trainable
    m = StudentForceField()
    m.interactions[2] = m.interactions[0]
    assert [(n, id(p)) for n, p in _trainable(m, True)] == [(n, id(p)) for n, p in m.named_parameters()]


@pytest.mark.gpu
def test_shared_blocks_evaluate_as_equal_blocks():
    from mlff_gb300.student_model import StudentForceField
    torch.manual_seed(3)
    m = StudentForceField().cuda().eval()
    other = StudentForceField().cuda().eval()
    m.interactions[1] = m.interactions[0]
    other.load_state_dict(m.state_dict())
    assert torch.equal(energies(m), energies(other))
