"""Edges of the table path that ordinary structures do not reach (GPU):
receiver groups of more than 256 edges, whose record sort recomputes the
geometry instead of keeping it in registers, and weights of accuracy class 1,
which the split-FP16 path's reverse pass alone takes from the tables.

Tolerances: tests/test_gpu_table_path.py asks 2e-5 of the forces for two FP32
evaluations, twice the measured 5e-6 plus the table's 5e-7, at about 50
neighbours per atom.  Rounding errors of sums grow with the root of their
length: up to 420 neighbours, a factor of 2.9, 2 (2.9 x 5.5e-6) = 3.2e-5, 4e-5
asked; the energy term's gradients' 1e-5 become 2.9e-5.  Atomic energies of
two FP32 evaluations: sums of 420 terms (1.2e-6) in three layers, 1e-5.  The
crystals' vector features cancel, and the force term's gradients divide by
them: FP32 is off from float64 by 1e-2 there whichever way it is evaluated, so
those are held to the plain path's own error.  Their sums also leave the range
of FP16, so the split-FP16 path runs on the molecule alone."""
import numpy as np
import pytest
import torch

from test_gpu_table_path import batch_of, model, rel

pytestmark = pytest.mark.gpu


def dense(name):
    """(structure, receivers per group): a compact 1,500-atom molecule, groups
    of two receivers; crystals of 1 A spacing, groups of one, the table read
    from memory or staged (training: from 400 atoms)."""
    from mlff_gb300 import systems
    if name == "molecule1500":
        return systems.lattice_molecule(1500, seed=3), 2
    k = int(name[7:])
    rng = np.random.default_rng(k)
    pos = np.stack(np.meshgrid(*[np.arange(k)] * 3), -1).reshape(-1, 3) + rng.normal(0.0, 0.05, (k ** 3, 3))
    Z = rng.choice([1, 6, 7, 8], k ** 3, p=[0.5, 0.3, 0.1, 0.1])
    return systems.System(Z, pos, np.array([0, k ** 3]), np.zeros((1, 3)), np.zeros(1, bool)), 1


DENSE = ["molecule1500", "crystal7", "crystal8"]


def largest_group(eng, b, g):
    row_ptr = eng.neighbors(b)[0].cpu().numpy()
    return int(np.diff(np.append(row_ptr[:-1:g], row_ptr[-1])).max())


@pytest.mark.parametrize("name, precision", [("molecule1500", "fp16x3")] + [(n, "tuned_fp32") for n in DENSE])
def test_dense_rows_match_network_evaluation(weights_bias, name, precision):
    from mlff_gb300 import _lib
    s, g = dense(name)
    b, m = batch_of(s), model(weights_bias, precision)
    eng = m.engine()
    assert largest_group(eng, b, g) > 256
    path, network = ((_lib.PATH_TABLE, _lib.PATH_TUNED_TC) if precision == "fp16x3" else
                     (_lib.PATH_TABLE_FP32, _lib.PATH_TUNED_FP32))
    assert m.path == path
    _, F, V, A = eng.energy_forces(b, path, virial=True, atom_energy=True, graph=False)
    _, F0, V0, A0 = eng.energy_forces(b, network, virial=True, atom_energy=True, graph=False)
    assert rel(F, F0) < 4e-5 and rel(V, V0) < 4e-5
    assert torch.equal(A, A0) if precision == "fp16x3" else rel(A, A0) < 1e-5


@pytest.mark.parametrize("precision", ["fp16x3", "tuned_fp32"])
def test_rows_keep_their_order_in_either_branch(weights_bias, precision):
    """A molecule alone (groups of one receiver, geometry in registers) and
    beside 200 far atoms (groups of two, up to 300 edges): the same bits."""
    from mlff_gb300 import systems
    s = systems.lattice_molecule(1400, seed=3)
    far = systems.System(np.full(200, 6), np.arange(600.0).reshape(200, 3) * 40.0, np.arange(201),
                         np.zeros((200, 3)), np.zeros(200, bool))
    b, both = batch_of(s), batch_of(systems.concat([s, far]))
    m = model(weights_bias, precision)
    eng = m.engine()
    assert largest_group(eng, b, 1) <= 256 < largest_group(eng, both, 2)
    E, F, V = eng.energy_forces(b, m.path, virial=True, graph=False)
    E1, F1, V1 = eng.energy_forces(both, m.path, virial=True, graph=False)
    assert torch.equal(E, E1[:1]) and torch.equal(F, F1[:1400]) and torch.equal(V, V1[:1])


@pytest.mark.parametrize("name", DENSE[1:])
def test_dense_rows_gradients_against_float64(weights_bias, name):
    """Off from float64 by no more than the plain path and the sums' bound."""
    from mlff_gb300.training import force_term_grads, param_grads
    from oracle import painn
    s, g = dense(name)
    b, m = batch_of(s), model(weights_bias, "tuned_fp32")
    eng = m.engine()
    assert largest_group(eng, b, g) > 256
    G = torch.randn(b.n_atoms, 3, device="cuda", generator=torch.Generator(device="cuda").manual_seed(8))
    w = torch.ones(1, dtype=torch.float64)
    got = [param_grads(m, b, w)[1], force_term_grads(m, b, G)]
    cls, eng.table_class = eng.table_class, 0
    try:
        plain = [param_grads(m, b, w)[1], force_term_grads(m, b, G)]
    finally:
        eng.table_class = cls
    pos = s.pos.astype(np.float32).astype(np.float64)
    exact = [painn.param_grads(weights_bias, s.Z, pos, s.mol_ptr, w.numpy())[1],
             painn.param_grads_forces(weights_bias, s.Z, pos, s.mol_ptr, np.zeros(1), G.double().cpu().numpy())[2]]
    for a, p, e, tol in zip(got, plain, exact, (2.9e-5, 1.45e-4)):
        floor = 1e-3 * max(float(x.norm()) for x in e.values())
        for k, x in e.items():
            x = x.to("cuda")
            err, err_plain = float((a[k].double() - x).norm()), float((p[k].double() - x).norm())
            assert err <= 1.25 * err_plain + tol * max(float(x.norm()), floor), k


@pytest.mark.parametrize("scale", [3.0, 8.0])
def test_class_1_weights(weights_bias, scale):
    """Filters sharp enough to miss the FP32 class: split FP16 keeps the table
    reverse pass, whose forces are off from float64 by no more than the
    network kernels' and the class's bound on the derivative (1.2e-5, and FP32
    sums: 2e-5); the FP32 paths go back to the network."""
    from mlff_gb300 import _lib, systems
    from oracle import painn
    s = systems.molecule_batch(7, 3, 90, seed=31)
    w = {k: (v * np.float32(scale) if k.endswith("rbf_to_scalar.0.weight") else v) for k, v in weights_bias.items()}
    b, m = batch_of(s), model(w)
    eng = m.engine()
    assert eng.table_class == 1 and m.path == _lib.PATH_TABLE
    E, F, _ = eng.energy_forces(b, m.path, graph=False)
    E0, F0, _ = eng.energy_forces(b, _lib.PATH_TUNED_TC, graph=False)
    _, F64 = painn.energy_forces(w, s.Z, s.pos.astype(np.float32).astype(np.float64), s.mol_ptr)
    F64 = F64.to("cuda")
    assert torch.equal(E, E0) and rel(F, F64) <= rel(F0, F64) + 2e-5
    m.precision = "tuned_fp32"
    assert m.path == _lib.PATH_TUNED_FP32
    F1 = eng.energy_forces(b, _lib.PATH_TABLE_FP32, graph=False)[1]      # a path chosen for earlier weights
    assert torch.equal(F1, eng.energy_forces(b, _lib.PATH_TUNED_FP32, graph=False)[1])
    with pytest.raises(_lib.MLFFError):
        eng.energy_forces(b, _lib.PATH_TRAIN_TABLE, graph=False)
