"""Performance cases of mlff_gb300: what a user of the force field has it do,
each through a public entry point.

``listed()`` is the fixed set, ``draw(rng)`` gives further cases of the same
ranges, ``prepare`` makes what a program holds before the call, ``run`` is
one call, ``work`` the bytes and operations the call cannot do without and
``exact`` the same call's results in float64, in plain torch.

The kinds of case:

* ``single``  -- energy and forces of one structure on the device
  (``StudentForceField.predict_energy_and_forces``): relaxations and MD steps
  of a molecule, a water box or a large periodic box.
* ``batch``   -- energies and forces of many molecules at once
  (``forward_with_analytical_forces``): screening, batched inference.
* ``energy``  -- energies only of many molecules (``forward`` without
  gradients): ranking of conformers.
* ``train``   -- one optimisation step of the reference's training loop:
  energies, forces with ``create_graph=True``, ``ForceFieldLoss``,
  ``loss.backward()``, gradient clipping, optimiser step.
* ``message`` / ``update`` -- one block of the network on its own, forward
  and backward, as a program that builds its own model from the blocks uses
  it.

Weights are the module's own seeded initialisation with normal(0, 0.1)
biases added (an untrained model has zero biases, a trained one does not);
structures come from the package's seeded generators.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "mlff-distiller_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

from mlff_gb300 import systems  # noqa: E402
from mlff_gb300.student_model import PaiNNMessage, PaiNNUpdate, StudentForceField  # noqa: E402
from mlff_gb300.training import ForceFieldLoss  # noqa: E402

CUTOFF = 5.0
GRAD_CLIP = 1.0          # the reference's gradient-norm clip
LEARNING_RATE = 1e-4


# ------------------------------------------------------------------- cases
def listed():
    return [
        # one H/C/N/O molecule, the call an interactive relaxation makes: latency
        {"name": "molecule60", "kind": "single", "system": "molecule", "atoms": 60, "precision": "fp16x3"},
        # 256 molecules of 10 to 120 atoms: the headline batch
        {"name": "batch256", "kind": "batch", "n_mol": 256, "n_min": 10, "n_max": 120, "precision": "fp16x3"},
        # 1,000 water molecules in a periodic box
        {"name": "water3000", "kind": "single", "system": "water", "atoms": 3000, "precision": "fp16x3"},
        # 100,000 atoms in a periodic box: the largest system
        {"name": "box100k", "kind": "single", "system": "box", "atoms": 100000, "precision": "fp16x3"},
        # energies only of 200 small molecules (the sizes the reference quotes: 3 to 32 atoms)
        {"name": "energies200", "kind": "energy", "n_mol": 200, "n_min": 3, "n_max": 32, "precision": "fp16x3"},
        # the FP32 options of ``precision``
        {"name": "batch64_tuned_fp32", "kind": "batch", "n_mol": 64, "n_min": 10, "n_max": 120,
         "precision": "tuned_fp32"},
        {"name": "batch37_fp32", "kind": "batch", "n_mol": 37, "n_min": 10, "n_max": 120, "precision": "fp32"},
        # training on energies and forces: a small batch and the benchmark's 64 structures
        {"name": "train8", "kind": "train", "n_mol": 8, "n_min": 10, "n_max": 120, "forces": True},
        {"name": "train64", "kind": "train", "n_mol": 64, "n_min": 10, "n_max": 120, "forces": True},
        # training on energies alone
        {"name": "train_energy100", "kind": "train", "n_mol": 100, "n_min": 3, "n_max": 64, "forces": False},
        # the blocks on their own, forward and backward: the model's width and the unit tests' 64
        {"name": "message128", "kind": "message", "hidden": 128, "n_mol": 32, "n_min": 10, "n_max": 120},
        {"name": "update64", "kind": "update", "hidden": 64, "atoms": 5001},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "batch", "batch", "energy", "train", "train", "message", "update"])
    precision = rng.choice(["fp16x3", "fp16x3", "fp16x3", "tuned_fp32", "fp32"])
    n_min = rng.randint(3, 20)
    n_max = n_min + rng.randint(1, 110)
    if kind == "single":
        system = rng.choice(["molecule", "water", "box"])
        if system == "molecule":
            atoms = _log_int(rng, 5, 1500)
        elif system == "water":
            atoms = 3 * _log_int(rng, 64, 1000)
        else:
            atoms = _log_int(rng, 1500, 100000 if precision == "fp16x3" else 6000)
        return {"kind": kind, "system": system, "atoms": atoms, "precision": precision}
    if kind == "batch":
        n_mol = _log_int(rng, 2, 300 if precision == "fp16x3" else 80)
        return {"kind": kind, "n_mol": n_mol, "n_min": n_min, "n_max": n_max, "precision": precision}
    if kind == "energy":
        return {"kind": kind, "n_mol": _log_int(rng, 2, 400), "n_min": n_min, "n_max": n_max,
                "precision": precision}
    if kind == "train":
        return {"kind": kind, "n_mol": _log_int(rng, 2, 48), "n_min": n_min, "n_max": n_max,
                "forces": rng.random() < 0.7}
    hidden = rng.choice([32, 64, 96, 128])
    if kind == "message":
        return {"kind": kind, "hidden": hidden, "n_mol": _log_int(rng, 1, 28), "n_min": n_min, "n_max": n_max}
    return {"kind": kind, "hidden": hidden, "atoms": _log_int(rng, 50, 20000)}


# ------------------------------------------------------------------ inputs
def _system(case, seed):
    """The case's structures.  A batch's molecule sizes (uniform in n_min ..
    n_max) belong to the case, positions and elements to the seed."""
    if case["kind"] != "single":
        lo, hi = case["n_min"], case["n_max"]
        sizes = np.random.default_rng([case["n_mol"], lo, hi]).integers(lo, hi + 1, size=case["n_mol"])
        rng = np.random.default_rng(seed)
        return systems.concat([systems.lattice_molecule(int(n), rng=rng) for n in sizes])
    n = case["atoms"]
    if case["system"] == "molecule":
        return systems.lattice_molecule(n, seed=seed)
    if case["system"] == "water":
        n_water = n // 3
        return systems.water_box(n_water, L=31.0 * (n_water / 1000.0) ** (1.0 / 3.0), seed=seed)
    return systems.large_box(n, seed=seed)


def _model(case, seed, device="cuda"):
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        model = StudentForceField(precision=case.get("precision", "fp16x3"))
        with torch.no_grad():
            for name, p in model.named_parameters():
                if name.endswith(".bias"):
                    p.add_(torch.randn(p.shape) * 0.1)
    return model.to(device)


def _tensors(case, seed, device="cuda"):
    s = _system(case, seed)
    t = {"Z": torch.tensor(s.Z, device=device), "pos": torch.tensor(s.pos, dtype=torch.float32, device=device),
         "batch": torch.tensor(np.repeat(np.arange(s.n_mol), np.diff(s.mol_ptr)), device=device), "n_mol": s.n_mol,
         "cell": None, "pbc": None}
    if bool(s.pbc.any()):
        t["cell"] = torch.tensor(np.diag(s.box[0]), dtype=torch.float32)
        t["pbc"] = torch.tensor([True, True, True])
    return t


def _targets(case, seed, n_atoms, device="cuda"):
    g = torch.Generator().manual_seed(seed + 77)
    return {"energy": (torch.randn(case["n_mol"], generator=g) * 5.0).to(device),
            "forces": torch.randn(n_atoms, 3, generator=g).to(device)}


def _block_inputs(case, seed, device="cuda"):
    """Features, graph and cotangents of one block: unit-variance features
    from the seed on the edges and radial basis of the case's molecules."""
    H = case["hidden"]
    g = torch.Generator(device=device).manual_seed(seed)
    rnd = lambda *shape: torch.randn(*shape, generator=g, device=device)  # noqa: E731
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        block = PaiNNMessage(H, 20) if case["kind"] == "message" else PaiNNUpdate(H)
        with torch.no_grad():
            for name, p in block.named_parameters():
                if name.endswith(".bias"):
                    p.normal_(0.0, 0.1)
    block = block.to(device)
    t = {"block": block}
    if case["kind"] == "message":
        m = _tensors(case, 0, device)
        src, dst, vec = _graph(m["pos"], m["batch"], None)
        d = vec.norm(dim=1)
        centers = torch.linspace(0, CUTOFF, 20, device=device)
        t["edge_index"] = torch.stack([src, dst])
        t["rbf"] = (torch.exp(-((d.unsqueeze(1) - centers) * (20 / CUTOFF)) ** 2)
                    * (0.5 * (torch.cos(math.pi * d / CUTOFF) + 1.0)).unsqueeze(1)).float().requires_grad_(True)
        t["unit"] = (vec / d.unsqueeze(1)).float().requires_grad_(True)
        n = m["pos"].shape[0]
    else:
        n = case["atoms"]
    t["s"] = rnd(n, H).requires_grad_(True)
    t["v"] = rnd(n, 3, H).requires_grad_(True)
    t["gs"], t["gv"] = rnd(n, H), rnd(n, 3, H)
    return t


def prepare(case, seed):
    if case["kind"] in ("message", "update"):
        return dict(_block_inputs(case, seed), case=case)
    model = _model(case, seed)
    st = dict(_tensors(case, seed), case=case, model=model)
    if case["kind"] == "train":
        model.train()
        st["target"] = _targets(case, seed, st["Z"].shape[0])
        st["loss"] = ForceFieldLoss(force_weight=100.0 if case["forces"] else 0.0,
                                    angular_weight=10.0 if case["forces"] else 0.0)
        st["opt"] = torch.optim.SGD(model.parameters(), lr=LEARNING_RATE)
    else:
        model.eval()
    return st


# --------------------------------------------------------------------- run
def _run_block(st):
    block = st["block"]
    if st["case"]["kind"] == "message":
        ins = [st["s"], st["v"], st["rbf"], st["unit"]] + list(block.parameters())
        s, v = block(st["s"], st["v"], st["edge_index"], st["rbf"], st["unit"])
    else:
        ins = [st["s"], st["v"]] + list(block.parameters())
        s, v = block(st["s"], st["v"])
    grads = torch.autograd.grad([s, v], ins, [st["gs"], st["gv"]])
    return {"s": s.detach(), "v": v.detach(), "grads": list(grads)}


def _run_train(st):
    model, tgt = st["model"], st["target"]
    st["opt"].zero_grad(set_to_none=True)
    pos = st["pos"].detach().requires_grad_(st["case"]["forces"])
    E = model(st["Z"], pos, batch=st["batch"])
    pred = {"energy": E}
    if st["case"]["forces"]:
        pred["forces"] = -torch.autograd.grad(E, pos, torch.ones_like(E), create_graph=True)[0]
    loss = st["loss"](pred, tgt)["total"]
    loss.backward()
    torch.nn.utils.clip_grad_norm_(model.parameters(), GRAD_CLIP)
    st["opt"].step()
    out = {"energy": E.detach(), "loss": loss.detach(),
           "grads": {n: p.grad for n, p in model.named_parameters()}}
    if "forces" in pred:
        out["forces"] = pred["forces"].detach()
    return out


def run(st):
    kind = st["case"]["kind"]
    if kind in ("message", "update"):
        return _run_block(st)
    if kind == "train":
        return _run_train(st)
    model = st["model"]
    if kind == "single":
        E, F = model.predict_energy_and_forces(st["Z"], st["pos"], cell=st["cell"], pbc=st["pbc"])
    elif kind == "batch":
        E, F = model.forward_with_analytical_forces(st["Z"], st["pos"], batch=st["batch"])
    else:
        with torch.no_grad():
            return {"energy": model(st["Z"], st["pos"], batch=st["batch"])}
    return {"energy": E, "forces": F}


# -------------------------------------------------------------------- work
def work(case):
    """Positions, numbers and weights read once, results written once; the
    filter network once per pair, the messages per directed edge, the update
    and readout networks per atom; a reverse pass costs two forwards, the
    gradients of a force loss twice an energy loss's pass."""
    if case["kind"] == "update":
        n, H = case["atoms"], case["hidden"]
        return {"bytes": 4.0 * n * 4 * H * 4, "flops": 3.0 * n * 2 * 5 * H * H}
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t = _tensors(case, 0, dev)
    n, pairs = t["Z"].shape[0], _count_pairs(t["pos"], t["batch"], t["cell"])
    if case["kind"] == "message":
        H = case["hidden"]
        flops = 3.0 * (2 * pairs * 2 * (20 * H + 3 * H * H) + 2 * pairs * 14 * H)
        return {"bytes": 4.0 * (n * 4 * H * 4 + 2 * pairs * 2 * 23) + 16.0 * 2 * pairs, "flops": flops}
    H, L = 128, 3
    forward = L * (pairs * 2.0 * (20 * H + 3 * H * H) + 2 * pairs * 14 * H + n * 2.0 * 5 * H * H) + n * 2.0 * (
        H * H // 2 + H * H // 8)
    weights = 4.0 * 3 * (20 * H + 3 * H * H + 5 * H * H)
    passes = {"energy": 1, "single": 3, "batch": 3}.get(case["kind"])
    if case["kind"] == "train":
        passes = 9 if case["forces"] else 3
        weights *= 3
    return {"bytes": n * (12.0 + 8 + 8 + 12) + weights, "flops": forward * passes}


# ------------------------------------------------------------------- exact
def _pair_blocks(pos, batch, cell, rows):
    """(i, j) of pairs within the cutoff, decided in float32 as the radius
    graph is defined: x*x rounded, two fused multiply-adds, square root,
    minimum image by the rounded reciprocal of the box edge."""
    n = pos.shape[0]
    L = None if cell is None else torch.diagonal(cell).to(pos.device, torch.float32)
    for a in range(0, n, rows):
        b = min(n, a + rows)
        # atoms are grouped by structure: only the columns of the rows' structures
        lo = int(torch.searchsorted(batch, batch[a]))
        hi = int(torch.searchsorted(batch, batch[b - 1], right=True))
        comp = []
        for k in range(3):
            x = pos[a:b, k].unsqueeze(1) - pos[lo:hi, k].unsqueeze(0)
            if L is not None:
                w = torch.round(x * (1.0 / L[k]))
                x = (x.double() - w.double() * L[k].double()).float()
            comp.append(x)
        r2 = (comp[1].double() ** 2 + (comp[0] * comp[0]).double()).float()
        r2 = (comp[2].double() ** 2 + r2.double()).float()
        ok = (torch.sqrt(r2) <= CUTOFF) & (batch[a:b].unsqueeze(1) == batch[lo:hi].unsqueeze(0))
        i, j = torch.nonzero(ok, as_tuple=True)
        keep = (i + a) != (j + lo)
        yield i[keep] + a, j[keep] + lo


def _rows(pos, batch):
    return 256 if pos.shape[0] > 20000 else 1024


def _count_pairs(pos, batch, cell):
    return sum(int(i.shape[0]) for i, _ in _pair_blocks(pos, batch, cell, _rows(pos, batch))) // 2


def _graph(pos, batch, cell):
    """(src, dst, float64 edge vectors pos[src] - pos[dst]), source-major."""
    parts = list(_pair_blocks(pos, batch, cell, _rows(pos, batch)))
    src, dst = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
    return src, dst, _vectors(pos.double(), src, dst, cell)


def _vectors(pos, src, dst, cell):
    vec = pos[src] - pos[dst]
    if cell is not None:
        L = torch.diagonal(cell).to(pos.device, pos.dtype)
        vec = vec - L * torch.round(vec.detach() / L)
    return vec


def _silu(x):
    return x * torch.sigmoid(x)


def _norm3(v):
    """|v| over axis 1 with derivative 0 where v = 0, twice differentiable elsewhere."""
    n2 = (v * v).sum(1)
    ok = n2 > 0
    return torch.where(ok, torch.sqrt(torch.where(ok, n2, torch.ones_like(n2))), torch.zeros_like(n2))


def _message(s, v, e, u, src, dst, w1, b1, w2, b2):
    H = s.shape[1]
    f = _silu(e @ w1.T + b1) @ w2.T + b2
    ds = torch.zeros_like(s).index_add(0, dst, s[src] * f[:, :H])
    dv = torch.zeros_like(v).index_add(0, dst, v[src] * f[:, H:2 * H].unsqueeze(1)
                                       + u.unsqueeze(2) * f[:, 2 * H:].unsqueeze(1))
    return ds, dv


def _update(s, v, w1, b1, w2, b2, mix):
    a = _silu(torch.cat([s, _norm3(v)], 1) @ w1.T + b1) @ w2.T + b2
    H = s.shape[1]
    s = s + a[:, :H]
    v = v * a[:, H:2 * H].unsqueeze(1) + torch.einsum("ij,njk->nik", mix, v) * a[:, 2 * H:].unsqueeze(1)
    return s, v


def _energies(p, t, pos, chunk=400000):
    from torch.utils.checkpoint import checkpoint
    src, dst, _ = _graph(t["pos"], t["batch"], t["cell"])
    vec = _vectors(pos, src, dst, t["cell"])
    d = torch.sqrt((vec * vec).sum(1))
    u = vec / (d.unsqueeze(1) + 1e-8)
    rbf = torch.exp(-((d.unsqueeze(1) - p["rbf.centers"]) / p["rbf.widths"]) ** 2)
    e = rbf * (0.5 * (torch.cos(math.pi * d / CUTOFF) + 1.0) * (d < CUTOFF)).unsqueeze(1)
    s = p["embedding.weight"][t["Z"]]
    v = torch.zeros(s.shape[0], 3, s.shape[1], dtype=s.dtype, device=s.device)
    for l in range(3):
        f = "interactions.%d.message.rbf_to_scalar." % l
        w = [p[f + k] for k in ("0.weight", "0.bias", "2.weight", "2.bias")]
        if src.shape[0] <= 2 * chunk:
            ds, dv = _message(s, v, e, u, src, dst, *w)
        else:
            ds, dv = torch.zeros_like(s), torch.zeros_like(v)
            for c in range(0, src.shape[0], chunk):
                c = slice(c, c + chunk)
                x = checkpoint(_message, s, v, e[c], u[c], src[c], dst[c], *w, use_reentrant=False)
                ds, dv = ds + x[0], dv + x[1]
        g = "interactions.%d.update." % l
        s, v = _update(s + ds, v + dv, *[p[g + k] for k in ("update_mlp.0.weight", "update_mlp.0.bias",
                                                            "update_mlp.2.weight", "update_mlp.2.bias",
                                                            "mixing_matrix")])
    for k in ("0", "2"):
        s = _silu(s @ p["energy_head.%s.weight" % k].T + p["energy_head.%s.bias" % k])
    a = (s @ p["energy_head.4.weight"].T + p["energy_head.4.bias"])[:, 0]
    return torch.zeros(t["n_mol"], dtype=a.dtype, device=a.device).index_add(0, t["batch"], a)


def _exact_block(case, seed):
    t = _block_inputs(case, seed)
    par = [p.detach().double().requires_grad_(True) for p in t["block"].parameters()]
    x = {k: t[k].detach().double().requires_grad_(True) for k in ("s", "v", "rbf", "unit") if k in t}
    if case["kind"] == "message":
        src, dst = t["edge_index"]
        ds, dv = _message(x["s"], x["v"], x["rbf"], x["unit"], src, dst, *par)
        s, v = x["s"] + ds, x["v"] + dv
    else:
        mix, w = par[0], par[1:]
        s, v = _update(x["s"], x["v"], *w, mix)
    grads = torch.autograd.grad([s, v], list(x.values()) + par, [t["gs"].double(), t["gv"].double()])
    return {"s": s.detach(), "v": v.detach(), "grads": list(grads)}


def _exact_train(case, p, t, target, names):
    pos = t["pos"].double().requires_grad_(True)
    E = _energies(p, t, pos, chunk=1 << 40)
    loss = ((E - target["energy"].double()) ** 2).mean()
    out = {"energy": E.detach()}
    if case["forces"]:
        F = -torch.autograd.grad(E.sum(), pos, create_graph=True)[0]
        ref = target["forces"].double()
        norm = lambda x: torch.sqrt((x * x).sum(1, keepdim=True)).clamp(min=1e-8)  # noqa: E731
        cos = (F / norm(F) * (ref / norm(ref))).sum(1)
        loss = loss + 100.0 * ((F - ref) ** 2).mean() + 10.0 * (1.0 - cos).mean()
        out["forces"] = F.detach()
    grads = torch.autograd.grad(loss, [p[n] for n in names], allow_unused=True)
    grads = [torch.zeros_like(p[n]) if g is None else g for n, g in zip(names, grads)]
    total = torch.sqrt(sum((g * g).sum() for g in grads))
    scale = torch.clamp(GRAD_CLIP / (total + 1e-6), max=1.0)
    return dict(out, loss=loss.detach(), grads={n: g * scale for n, g in zip(names, grads)})


def exact(case, seed):
    if case["kind"] in ("message", "update"):
        return _exact_block(case, seed)
    model = _model(case, seed)
    t = _tensors(case, seed)
    p = {k: v.detach().double() for k, v in model.state_dict().items()}
    names = [n for n, _ in model.named_parameters()]
    if case["kind"] == "train":
        for n in names:
            p[n].requires_grad_(True)
        return _exact_train(case, p, t, _targets(case, seed, t["Z"].shape[0]), names)
    if case["kind"] == "energy":
        with torch.no_grad():
            E = _energies(p, t, t["pos"].double())
        return {"energy": E}
    pos = t["pos"].double().requires_grad_(True)
    E = _energies(p, t, pos)
    F = -torch.autograd.grad(E.sum(), pos)[0]
    return {"energy": E[0].detach() if case["kind"] == "single" else E.detach(), "forces": F}
