"""Linears of more than 8 tokens on the GPU, at the sizes where their cut into row panels, row tiles, chunks and parts of k can go wrong: fewer rows
than workers, rows that are no multiple of four, a last chunk that is not whole, panels shared by several workers, several tasks a worker."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernel(tokens):
    import mirage_b200 as mi
    params = mi.PersistentKernel.get_default_init_parameters()
    params.update(test_mode=True, num_workers=0, max_num_batched_tokens=tokens, max_num_batched_requests=tokens)
    return mi.PersistentKernel(**params)


def _close(got, want):
    """bf16 of sums in fp32: half a unit of the last place (8 bits: up to 2^-8 of the value), and K <= 12288 terms of unit size added in fp32, whose errors stay below
    2^-12 of the largest sum."""
    want = want.float()
    bound = want.abs() * 2 ** -8 + 2 ** -12 * want.abs().max()
    assert bool(((got.float() - want).abs() <= bound).all()), float(((got.float() - want).abs() - bound).max())


@pytest.mark.parametrize("tokens", [9, 16, 33, 64])
@pytest.mark.parametrize("rows,k", [(8, 64), (148, 704), (449, 192), (1187, 1024), (4096, 4096), (2048, 12288), (40004, 128)])
def test_linear_with_residual(tokens, rows, k):
    g = torch.Generator(device="cuda").manual_seed(rows + k + tokens)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, res = rnd(tokens, k), rnd(rows, k), rnd(tokens, rows)
    pk = _kernel(tokens)
    plain, summed = torch.zeros_like(res), torch.zeros_like(res)
    tx, tw = pk.attach_input(x, "x"), pk.attach_input(w, "w")
    grid = dict(grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    pk.linear_layer(input=tx, weight=tw, output=pk.attach_input(plain, "plain"), **grid)
    pk.linear_with_residual_layer(input=tx, weight=tw, residual=pk.attach_input(res, "res"), output=pk.attach_input(summed, "summed"), **grid)
    pk.compile()
    want = x.double() @ w.double().T
    for _ in range(2):   # a second launch finds the rings, tickets and parts as the first one left them
        plain.zero_()
        summed.zero_()
        pk.run_test_mode()
        _close(plain, want)
        _close(summed, want + res.double())
    first = summed.clone()
    pk.run_test_mode()
    assert torch.equal(first, summed)


@pytest.mark.parametrize("tokens,rows,k", [(9, 64, 4096), (16, 2367, 4096), (16, 2368, 4096), (64, 256, 1024), (64, 4096, 1024)])
def test_norm_in_front(tokens, rows, k):
    """Whole normed rows in the linear's tile (few rows a worker) and the norm as a task group of its own."""
    g = torch.Generator(device="cuda").manual_seed(rows + tokens)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, gamma, w = rnd(tokens, k), rnd(k), rnd(rows, k)
    pk = _kernel(tokens)
    out = torch.zeros(tokens, rows, dtype=torch.bfloat16, device="cuda")
    normed = pk.new_tensor((tokens, k), name="normed")
    grid = dict(grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    pk.rmsnorm_layer(input=pk.attach_input(x, "x"), weight=pk.attach_input(gamma, "gamma"), output=normed, **grid)
    pk.linear_layer(input=normed, weight=pk.attach_input(w, "w"), output=pk.attach_input(out, "out"), **grid)
    pk.compile()
    xd = x.double()
    y = (xd / torch.sqrt((xd * xd).mean(-1, keepdim=True) + 1e-6) * gamma.double()).bfloat16().double()
    pk.run_test_mode()
    # (the operand is bf16: a value next to the middle of two goes either way, 2^-8 of a term of the sum, so sqrt(k) of them at random)
    want = y @ w.double().T
    assert float((out.double() - want).norm() / want.norm()) <= 4e-3
