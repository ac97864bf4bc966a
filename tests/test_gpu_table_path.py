"""Tabulated edge filters (GPU): the table path against the float64 oracle
and the network evaluation at sizes on both sides of its receiver groups
(1 and 2 receivers; table read from memory or staged in shared memory),
for open and periodic batches, atoms without neighbours and ragged last
groups; the accuracy class of tables of sharp and of many-basis filters; and
the fallback when the table does not serve the weights.

Tolerances: the FP32 paths' own against float64 (2e-5 eV per atom, 1e-3
eV/A in tests/test_gpu_parity.py, which runs the split-FP16 path too);
between two FP32 evaluations twice the
measured FP32 error of the forces (5e-6 relative, 2-norm) plus the table's
(5e-7): 1.1e-5, asked 2e-5.  The split-FP16 path keeps its tensor-core
forward pass (equal energies); its reverse pass differs by the split-FP16
filter derivatives' 1e-5."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def model(weights=None, precision="fp16x3", **kw):
    from mlff_gb300.student_model import StudentForceField
    torch.manual_seed(5)
    m = StudentForceField(precision=precision, **kw)
    if weights is not None:
        m.load_state_dict({k: torch.tensor(v) for k, v in weights.items()})
    return m.to("cuda").eval()


def batch_of(s):
    from mlff_gb300.engine import make_batch
    per = bool(s.pbc.any())
    return make_batch(s.Z, s.pos.astype(np.float32), s.mol_ptr, s.box if per else None, s.pbc if per else None)


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def system(name):
    from mlff_gb300 import systems
    if name.startswith("molecules"):
        return systems.molecule_batch(int(name[9:]), 3, 90, seed=31)
    if name.startswith("water"):
        n = int(name[5:])
        return systems.water_box(n, L=31.0 * (n / 1000.0) ** (1.0 / 3.0), seed=32)
    if name.startswith("box"):
        return systems.large_box(int(name[3:]), seed=33)
    s = systems.lattice_molecule(60, seed=34)      # plus far atoms: rows without edges
    far = systems.System(np.array([1, 8, 6]), np.array([[50.0, 0, 0], [90.0, 0, 0], [93.0, 0, 0]]),
                         np.array([0, 3]), np.zeros((1, 3)), np.zeros(1, bool))
    return systems.concat([far, s, far])


# group shapes change at 1,500 atoms, staging at 400 (training) and 750
SIZES = ["isolated", "molecules1", "molecules7", "molecules30", "water64", "box1499", "box1500", "box1503",
         "box4095", "box4097", "molecules120"]


@pytest.mark.parametrize("precision", ["fp16x3", "tuned_fp32"])
@pytest.mark.parametrize("name", SIZES)
def test_table_path_matches_network_evaluation(weights_bias, name, precision):
    from mlff_gb300 import _lib
    s = system(name)
    b = batch_of(s)
    m = model(weights_bias, precision)
    eng = m.engine()
    assert eng.table_class == 2 and m.path in (_lib.PATH_TABLE, _lib.PATH_TABLE_FP32)
    E, F, V = eng.energy_forces(b, m.path, virial=True, graph=False)
    network = _lib.PATH_TUNED_TC if precision == "fp16x3" else _lib.PATH_TUNED_FP32
    E0, F0, V0 = eng.energy_forces(b, network, virial=True, graph=False)
    assert rel(F, F0) < 2e-5 and rel(V, V0) < 2e-5
    if precision == "fp16x3":      # the same forward pass
        assert torch.equal(E, E0)
    else:
        assert np.abs((E - E0).cpu().numpy() / np.diff(s.mol_ptr)).max() < 2e-5
    E1, F1, _ = eng.energy_forces(b, m.path, virial=True, graph=False)
    assert torch.equal(E, E1) and torch.equal(F, F1)


def test_fp32_table_path_vs_float64_oracle(weights_bias):
    from oracle import painn
    s = system("molecules30")
    m = model(weights_bias, "tuned_fp32")
    E, F, _ = m.engine().energy_forces(batch_of(s), m.path, graph=False)
    pos = s.pos.astype(np.float32).astype(np.float64)
    E0, F0 = painn.energy_forces(weights_bias, s.Z, pos, s.mol_ptr)
    assert np.abs((E.cpu().numpy() - E0.numpy()) / np.diff(s.mol_ptr)).max() < 2e-5
    assert np.abs(F.cpu().numpy() - F0.numpy()).max() < 1e-3


def test_structure_results_do_not_depend_on_the_batch(weights_bias):
    """A structure alone (groups of 1 receiver) and in a batch of 4-receiver
    groups gives the same bits: a row's edges keep their order."""
    from mlff_gb300 import systems
    s = systems.molecule_batch(120, 3, 90, seed=31)
    m = model(weights_bias, "tuned_fp32")
    eng = m.engine()
    E, F, _ = eng.energy_forces(batch_of(s), m.path, graph=False)
    for k in (0, 57, 119):
        one = s.molecule(k)
        E1, F1, _ = eng.energy_forces(batch_of(one), m.path, graph=False)
        a, b = int(s.mol_ptr[k]), int(s.mol_ptr[k + 1])
        assert torch.equal(F[a:b], F1) and torch.equal(E[k:k + 1], E1)


def test_accuracy_class_and_fallback(weights_bias):
    from mlff_gb300 import _lib, systems
    s = system("molecules7")
    assert model().engine().table_class == 2
    assert model(num_rbf=7).engine().table_class == 2
    assert model(num_rbf=32).engine().table_class == 0     # functions of width cutoff / 32
    m = model(weights_bias)
    b = batch_of(s)
    path = (m.engine(), m.path)[1]
    assert path == _lib.PATH_TABLE
    with torch.no_grad():                                   # much sharper filters
        for blk in m.interactions:
            blk.message.rbf_to_scalar[0].weight.mul_(20.0)
    eng = m.engine()
    assert eng.table_class == 0 and m.path == _lib.PATH_TUNED_TC
    E, F, _ = eng.energy_forces(b, path, graph=False)       # a path chosen for the earlier weights
    E0, F0, _ = eng.energy_forces(b, _lib.PATH_TUNED_TC, graph=False)
    np.testing.assert_array_equal(E.cpu().numpy(), E0.cpu().numpy())
    np.testing.assert_array_equal(F.cpu().numpy(), F0.cpu().numpy())


@pytest.mark.parametrize("name", ["isolated", "molecules1", "molecules7", "box1499", "box1503", "box4097"])
def test_table_gradients_match_the_plain_path(weights_bias, name):
    """Energy and force / stress gradient terms through the tables against
    the plain FP32 path.  Both are FP32: against float64 the plain path's
    energy term is off by up to 2e-6 and its force term by up to 2e-5
    (2-norm per tensor); asked of the two together 1e-5 and 5e-5."""
    from mlff_gb300.training import force_term_grads, param_grads
    s = system(name)
    m = model(weights_bias, "tuned_fp32")
    b = batch_of(s)
    g = torch.Generator(device="cuda").manual_seed(8)
    w = torch.randn(b.n_mol, device="cuda", generator=g, dtype=torch.float64)
    G = torch.randn(b.n_atoms, 3, device="cuda", generator=g)
    S = torch.randn(b.n_mol, 3, 3, device="cuda", generator=g, dtype=torch.float64) if b.box is not None else None
    eng = m.engine()
    got = [param_grads(m, b, w)[:2], (None, force_term_grads(m, b, G, S))]
    again = force_term_grads(m, b, G, S)
    assert all(torch.equal(again[k], v) for k, v in got[1][1].items())
    cls, eng.table_class = eng.table_class, 0
    try:
        want = [param_grads(m, b, w)[:2], (None, force_term_grads(m, b, G, S))]
    finally:
        eng.table_class = cls
    assert float(((got[0][0] - want[0][0]).abs().cpu() / torch.tensor(np.diff(s.mol_ptr))).max()) < 2e-5
    for (_, a), (_, e), tol in zip(got, want, (1e-5, 5e-5)):
        for k in e:
            n = float(e[k].double().norm())
            d = float((a[k].double() - e[k].double()).norm())
            # a tensor whose gradient cancels is held to the scale of the others
            floor = 1e-3 * max(float(x.double().norm()) for x in e.values())
            assert d <= tol * max(n, floor), (k, d, n)
