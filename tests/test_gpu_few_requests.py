"""Attention of graphs of up to 8 tokens on the general instantiation (seven and more requests, or more tasks than workers) against 64 bits: its softmax
weights are no coarser than the batch-1 form's, which holds them in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv", [(8, 8), (16, 8), (32, 8), (32, 4), (6, 6)])
@pytest.mark.parametrize("lengths", [(1, 9, 700), (1500, 1, 8, 16, 300), (5, 64, 65, 200, 129, 7, 1000, 33)])
def test_attention_of_few_requests(heads, kv, lengths):
    import mirage_b200 as mi
    n, page = len(lengths), 16
    g = torch.Generator(device="cuda").manual_seed(heads + n)
    need = [-(-l // page) for l in lengths]
    pool = torch.randperm(sum(need) + 2, generator=torch.Generator().manual_seed(3)).tolist()
    starts = [sum(need[:r]) for r in range(n + 1)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    meta = {"qo_indptr_buffer": i32(list(range(n + 1))), "paged_kv_indptr_buffer": i32(starts), "paged_kv_indices_buffer": i32(pool[:starts[-1]]),
            "paged_kv_last_page_len_buffer": i32([(l - 1) % page + 1 for l in lengths])}
    params = mi.PersistentKernel.get_default_init_parameters()
    params.update(test_mode=True, num_workers=0, max_num_batched_tokens=n, max_num_batched_requests=n, max_num_pages=len(pool), page_size=page,
                  max_seq_length=-(-max(lengths) // page) * page, meta_tensors=meta)
    pk = mi.PersistentKernel(**params)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    qkv, kc, vc = rnd(n, (heads + 2 * kv) * 128), rnd(len(pool), page, kv, 128), rnd(len(pool), page, kv, 128)
    k0, v0 = kc.clone(), vc.clone()
    out = torch.zeros(n, heads * 128, dtype=torch.bfloat16, device="cuda")
    pk.paged_attention_layer(input=pk.attach_input(qkv, "qkv"), k_cache=pk.attach_input(kc, "k"), v_cache=pk.attach_input(vc, "v"), q_norm=None, k_norm=None,
                             cos_pos_embed=None, sin_pos_embed=None, output=pk.attach_input(out, "out"), grid_dim=(n, kv, 1), block_dim=(128, 1, 1))
    pk.compile()
    x = qkv.double().view(n, kv, heads // kv + 2, 128)
    want = []
    for r, l in enumerate(lengths):
        rows = torch.tensor(pool[starts[r]:starts[r + 1]], device="cuda")
        k, v = k0[rows].flatten(0, 1)[:l].double(), v0[rows].flatten(0, 1)[:l].double()
        k[-1], v[-1] = x[r, :, -2], x[r, :, -1]
        q = x[r, :, :-2].reshape(heads, 128)
        p = torch.softmax(torch.einsum("hd,nhd->hn", q, k.repeat_interleave(heads // kv, 1)) * 128 ** -0.5, -1)
        want.append(torch.einsum("hn,nhd->hd", p, v.repeat_interleave(heads // kv, 1)).flatten())
    want = torch.stack(want)
    for _ in range(2):
        out.zero_()
        pk.run_test_mode()
        # the output's rounding (2^-8 of a value at most) and scores, weights and sums in fp32 and 2^-17: below 2^-12 of the largest value
        assert bool(((out.double() - want).abs() <= want.abs() * 2 ** -8 + want.abs().amax(-1, keepdim=True) * 2 ** -12).all())
