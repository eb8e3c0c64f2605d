"""The allocation-free attention at the edges of its batches of positions, with every grouping of kv heads, caches on 8- and 16-byte boundaries, and another
number of chunks from call to call (the tickets are left at zero)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("offset", [0, 4])
def test_noalloc_attention_sizes(group, offset):
    import mirage_b200 as mi
    kv, page, lengths = 3, 5, [1, 15, 16, 17, 31, 64, 65, 127, 129, 300]
    n = len(lengths)
    g = torch.Generator(device="cuda").manual_seed(group + offset)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    need = [-(-l // page) for l in lengths]
    pool = torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)).tolist()
    starts = [sum(need[:r]) for r in range(n + 1)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    shape = (sum(need), page, kv, 128)
    size = shape[0] * page * kv * 128
    k, v = (rnd(size + 8)[offset:offset + size].view(shape) for _ in range(2))
    qkv, out = rnd(n, kv * (group + 2) * 128), torch.zeros(n, kv * group * 128, dtype=torch.bfloat16, device="cuda")
    x = qkv.double().view(n, kv, group + 2, 128)
    want = []
    for r, l in enumerate(lengths):
        rows = torch.tensor(pool[starts[r]:starts[r + 1]], device="cuda")
        kk, vv = k[rows].flatten(0, 1)[:l].double(), v[rows].flatten(0, 1)[:l].double()
        kk[-1], vv[-1] = x[r, :, -2], x[r, :, -1]
        p = torch.softmax(torch.einsum("hgd,nhd->hgn", x[r, :, :-2], kk) * 128 ** -0.5, -1)
        want.append(torch.einsum("hgn,nhd->hgd", p, vv).flatten())
    want = torch.stack(want)
    for chunks in (8, 3, 1, 8):
        out.zero_()
        mi.paged_decode_attention_noalloc(qkv, k, v, out, i32(starts), i32(pool), i32([(l - 1) % page + 1 for l in lengths]), kv * group, kv, num_chunks=chunks)
        # the output's rounding (at most 2^-8 of a value); scores, weights and sums in fp32
        assert bool(((out.double() - want).abs() <= want.abs() * 2 ** -8 + want.abs().amax(-1, keepdim=True) * 2 ** -14).all()), chunks
