"""PaiNNMessage and PaiNNUpdate forward and backward against float64
autograd at widths, basis sizes and row counts on both sides of the GEMM
tiles (32, 64, 128), the row splits of the weight gradients and the 16-byte
row rule.

Tolerance: outputs are at most three chained FP32 sums of up to a few
thousand terms of random sign (row splits of the weight gradients included),
error about 3 * eps * sqrt(4000) = 1.1e-5 of the 2-norm; 2e-5 is asked."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 2e-5


def ref_message(s, v, ei, rbf, evec, w1, b1, w2, b2):
    H = s.shape[1]
    f = torch.nn.functional.silu(rbf @ w1.T + b1) @ w2.T + b2
    src, dst = ei
    so = s.index_add(0, dst, s[src] * f[:, :H])
    return so, v.index_add(0, dst, v[src] * f[:, None, H:2 * H] + evec[:, :, None] * f[:, None, 2 * H:])


def ref_update(s, v, mix, w1, b1, w2, b2):
    H = s.shape[1]
    a = torch.nn.functional.silu(torch.cat([s, v.norm(dim=1)], 1) @ w1.T + b1) @ w2.T + b2
    mixed = torch.einsum("ij,njk->nik", mix, v)
    return s + a[:, :H], v * a[:, None, H:2 * H] + mixed * a[:, None, 2 * H:]


def close(got, want):
    for g, w in zip(got, want):
        d = (g.double() - w).norm()
        assert float(d) <= TOL * max(float(w.norm()), 1e-30), (tuple(w.shape), float(d), float(w.norm()))


def compare(block, ins, extra, ref):
    g = torch.Generator(device=DEV).manual_seed(9)
    par = list(block.parameters())
    out = block(*[x for x in ins[:2]], *extra[:1], *ins[2:])
    cot = [torch.randn(o.shape, device=DEV, generator=g) for o in out]
    got = torch.autograd.grad(out, ins + par, cot)
    d = [x.detach().double().requires_grad_(True) for x in ins + par]
    want_out = ref(d[:len(ins)], d[len(ins):])
    want = torch.autograd.grad(want_out, d, [c.double() for c in cot])
    close(list(out) + list(got), list(want_out) + list(want))


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "odd_base"])
@pytest.mark.parametrize("H,R,N,E", [(1, 1, 2, 1), (5, 3, 7, 63), (33, 20, 40, 65), (64, 20, 50, 1000),
                                     (128, 20, 300, 4097), (130, 32, 60, 515), (128, 7, 1, 31)])
def test_message_block(H, R, N, E, offset):
    from mlff_gb300.student_model import PaiNNMessage
    torch.manual_seed(H + E)
    g = torch.Generator(device=DEV).manual_seed(E)

    def rnd(*shape):   # contiguous, its first element `offset` floats behind a 16-byte boundary
        n = 1
        for k in shape:
            n *= k
        return torch.randn(n + 4, device=DEV, generator=g)[offset:offset + n].view(*shape).requires_grad_(True)

    block = PaiNNMessage(H, R).to(DEV)
    ei = torch.randint(0, N, (2, E), device=DEV, generator=g)
    ins = [rnd(N, H), rnd(N, 3, H), rnd(E, R), rnd(E, 3)]
    compare(block, ins, [ei], lambda x, p: ref_message(x[0], x[1], ei, x[2], x[3], *p))


@pytest.mark.parametrize("H,N", [(1, 1), (5, 63), (33, 65), (64, 129), (128, 1000), (130, 257), (96, 20000)])
def test_update_block(H, N):
    from mlff_gb300.student_model import PaiNNUpdate
    torch.manual_seed(H + N)
    g = torch.Generator(device=DEV).manual_seed(N)
    block = PaiNNUpdate(H).to(DEV)
    ins = [torch.randn(*s, device=DEV, generator=g).requires_grad_(True) for s in ((N, H), (N, 3, H))]
    compare(block, ins, [], lambda x, p: ref_update(x[0], x[1], *p))


@pytest.mark.parametrize("H,R,N,E", [(128, 20, 300, 9999), (132, 24, 200, 7041), (68, 36, 100, 19457)])
def test_message_block_wide_tiles(H, R, N, E):
    """Enough rows for the 64 x 128 tiles, with remainders in every direction."""
    test_message_block(H, R, N, E, 0)
