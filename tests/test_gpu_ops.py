"""GPU parity of single task bodies, run through PersistentKernel test mode (one launch of the task
graph), against the CPU oracle and the golden fixtures.  Tolerances: bf16 outputs within max relative
error 2e-2."""
import os

import pytest
import torch

from oracle import mpk_ops as ops
from gpu_util import rel_err, make_test_kernel

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.fixture(scope="module")
def mi():
    import mirage_b200
    return mirage_b200


def _bf16(*shape, seed, scale=1.0, shift=0.0):
    g = torch.Generator().manual_seed(seed)
    return (shift + scale * torch.randn(*shape, generator=g)).to(torch.bfloat16)


def test_rmsnorm_linear_baseline_config1(mi):
    """x[8,4096] ~ N(0,1), g = 1 + N(0,0.02), W[6144,4096] ~ N(0,0.02), eps 1e-6, seed 0."""
    torch.manual_seed(0)
    x = torch.randn(8, 4096).to(torch.bfloat16)
    g = (1 + 0.02 * torch.randn(4096)).to(torch.bfloat16)
    w = (0.02 * torch.randn(6144, 4096)).to(torch.bfloat16)
    ref = ops.rmsnorm_linear(x, g, w, 1e-6)
    pk = make_test_kernel(mi, 8)
    out = torch.zeros(8, 6144, dtype=torch.bfloat16, device="cuda")
    tx, tg = pk.attach_input(x.cuda(), "x"), pk.attach_input(g.cuda(), "g")
    tw, to = pk.attach_input(w.cuda(), "w"), pk.attach_input(out, "out")
    pk.rmsnorm_linear_layer(input=tx, weight_norm=tg, weight_linear=tw, output=to, grid_dim=(96, 1, 1),
                            block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert rel_err(out.cpu(), ref) <= TOL
    # a second launch gives bit-identical results (monotonic counters, no state left behind)
    first = out.clone()
    pk.run_test_mode()
    assert torch.equal(first, out)


def test_rmsnorm_linear_golden_fixture(mi, golden_dir):
    f = torch.load(os.path.join(golden_dir, "ref_norm_linear.pt"), weights_only=False)
    x, g, w = f["x"], f["g"].reshape(-1), f["w"]
    pk = make_test_kernel(mi, x.shape[0])
    out = torch.zeros(x.shape[0], w.shape[0], dtype=torch.bfloat16, device="cuda")
    pk.rmsnorm_linear_layer(input=pk.attach_input(x.cuda(), "x"), weight_norm=pk.attach_input(g.cuda(), "g"),
                            weight_linear=pk.attach_input(w.cuda(), "w"), output=pk.attach_input(out, "o"),
                            grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert rel_err(out.cpu(), f["out_f32"]) <= TOL


@pytest.mark.parametrize("B,N,K", [(1, 4096, 4096), (1, 4096, 12288), (2, 1000, 512), (3, 6144, 4096),
                                   (4, 520, 1536), (8, 777, 2048), (1, 37, 64), (5, 300, 6144),
                                   (16, 520, 4096), (33, 300, 1536), (64, 256, 12288), (64, 777, 512),
                                   (9, 96, 256)])
def test_linear_with_residual_shapes(mi, B, N, K):
    x = _bf16(B, K, seed=1)
    w = _bf16(N, K, seed=2, scale=0.02)
    r = _bf16(B, N, seed=3)
    ref = ops.linear(x, w, r)
    ref_plain = ops.linear(x, w)
    pk = make_test_kernel(mi, B)
    o1 = torch.zeros(B, N, dtype=torch.bfloat16, device="cuda")
    o2 = torch.zeros(B, N, dtype=torch.bfloat16, device="cuda")
    o3 = r.clone().cuda()
    tx, tw = pk.attach_input(x.cuda(), "x"), pk.attach_input(w.cuda(), "w")
    pk.linear_with_residual_layer(input=tx, weight=tw, residual=pk.attach_input(r.cuda(), "r"),
                                  output=pk.attach_input(o1, "o1"), grid_dim=(64, 1, 1), block_dim=(128, 1, 1))
    pk.linear_layer(input=tx, weight=tw, output=pk.attach_input(o2, "o2"), grid_dim=(64, 1, 1), block_dim=(128, 1, 1))
    pk.splitk_linear_layer(input=tx, weight=tw, output=pk.attach_input(o3, "o3"), grid_dim=(32, 4, 1),
                           block_dim=(256, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert rel_err(o1.cpu(), ref) <= TOL
    assert rel_err(o2.cpu(), ref_plain) <= TOL
    assert rel_err(o3.cpu(), ref) <= TOL      # split-K semantics: output += x W^T


@pytest.mark.parametrize("B", [16, 40, 64])
def test_rmsnorm_linear_large_batches(mi, B):
    """More than one tile of 8 tokens: token tiles are spread over the compute warps; at 64 tokens the norm can
    no longer be folded (the activation tile does not hold whole rows) and runs as its own task."""
    x = _bf16(B, 4096, seed=21)
    g = _bf16(4096, seed=22, scale=0.02, shift=1.0)
    w = _bf16(640, 4096, seed=23, scale=0.02)
    ref = ops.rmsnorm_linear(x, g, w, 1e-6)
    pk = make_test_kernel(mi, B)
    out = torch.zeros(B, 640, dtype=torch.bfloat16, device="cuda")
    normed = pk.new_tensor((B, 4096), name="normed")
    tx, tg, tw = pk.attach_input(x.cuda(), "x"), pk.attach_input(g.cuda(), "g"), pk.attach_input(w.cuda(), "w")
    pk.rmsnorm_layer(input=tx, weight=tg, output=normed, grid_dim=(B, 1, 1), block_dim=(128, 1, 1))
    pk.linear_layer(input=normed, weight=tw, output=pk.attach_input(out, "out"), grid_dim=(10, 1, 1),
                    block_dim=(128, 1, 1))
    pk.compile()
    assert pk.graph_info()["num_folded"] == (1 if B <= 16 else 0)
    pk.run_test_mode()
    assert rel_err(out.cpu(), ref) <= TOL


def test_mlp_pipeline_golden_fixture(mi, golden_dir):
    """gate_up (interleaved) -> silu_mul -> down + residual, the graph of the reference's
    test_qwen3_mlp_testmode.py, against the fixture its reference code produced."""
    f = torch.load(os.path.join(golden_dir, "ref_mlp.pt"), weights_only=False)
    x, res = f["x"], f["residual"]
    B, H = x.shape
    I = f["w_gate"].shape[0]
    groups = 4
    for fold in (True, False):
        pk = make_test_kernel(mi, B)
        tx = pk.attach_input(x.cuda(), "x")
        wg, wu = pk.attach_input(f["w_gate"].cuda(), "wg"), pk.attach_input(f["w_up"].cuda(), "wu")
        wgu = pk.shuffle_tensors([wg, wu], 0, groups, name="wgu")
        if fold:
            mid = pk.new_tensor((B, 2 * I), name="mid")
            act = pk.new_tensor((B, I), name="act")
        else:   # caller-visible intermediates stay materialised and are produced by stand-alone tasks
            mid_t = torch.zeros(B, 2 * I, dtype=torch.bfloat16, device="cuda")
            act_t = torch.zeros(B, I, dtype=torch.bfloat16, device="cuda")
            mid, act = pk.attach_input(mid_t, "mid"), pk.attach_input(act_t, "act")
        out = torch.zeros(B, H, dtype=torch.bfloat16, device="cuda")
        pk.linear_layer(input=tx, weight=wgu, output=mid, grid_dim=(2 * groups, 1, 1), block_dim=(128, 1, 1))
        pk.silu_mul_layer(input=mid, output=act, grid_dim=(groups, 1, 1), block_dim=(128, 1, 1))
        pk.linear_with_residual_layer(input=act, weight=pk.attach_input(f["w_down"].cuda(), "wd"),
                                      residual=pk.attach_input(res.cuda(), "res"), output=pk.attach_input(out, "out"),
                                      grid_dim=(H // 64, 1, 1), block_dim=(128, 1, 1))
        pk.compile()
        assert pk.graph_info()["num_folded"] == (1 if fold else 0)
        pk.run_test_mode()
        assert rel_err(out.cpu(), f["out"]) <= TOL
        if not fold:
            mid_ref = ops.linear(x, ops.shuffle_rows([f["w_gate"], f["w_up"]], groups))
            assert rel_err(mid_t.cpu(), mid_ref) <= TOL
            assert rel_err(act_t.cpu(), ops.silu_mul(mid_ref, groups)) <= TOL


def test_rmsnorm_layer_golden_fixture(mi, golden_dir):
    f = torch.load(os.path.join(golden_dir, "ref_rmsnorm.pt"), weights_only=False)
    x, w = f["x"], f["w"]
    pk = make_test_kernel(mi, x.shape[0])
    out = torch.zeros_like(x, device="cuda")
    pk.rmsnorm_layer(input=pk.attach_input(x.cuda(), "x"), weight=pk.attach_input(w.cuda(), "w"),
                     output=pk.attach_input(out, "o"), grid_dim=(x.shape[0], 1, 1), block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert rel_err(out.cpu(), f["out"]) <= TOL
    assert rel_err(out.cpu(), ops.rmsnorm(x, w, 1e-6)) <= 1e-2


def test_embedding_and_argmax(mi):
    V, H, B = 1000, 256, 4
    tab = _bf16(V, H, seed=5)
    ids = torch.tensor([[3], [999], [-1], [0]], dtype=torch.int64)
    logits = _bf16(B, V, seed=6)
    logits[1, 10] = logits[1, 700] = 9.0      # tie: lowest index must win
    pk = make_test_kernel(mi, B)
    out = torch.zeros(B, H, dtype=torch.bfloat16, device="cuda")
    tok = torch.zeros(B, 1, dtype=torch.int64, device="cuda")
    pk.embed_layer(input=pk.attach_input(ids.cuda(), "ids"), weight=pk.attach_input(tab.cuda(), "tab"),
                   output=pk.attach_input(out, "out"), grid_dim=(1, 1, 1), block_dim=(128, 1, 1), input_source=1)
    nparts = 7
    pv = pk.new_tensor((B, nparts), name="pv")
    pi = pk.new_tensor((B, nparts), dtype=mi.int64, name="pi")
    pk.argmax_partial_layer(input=pk.attach_input(logits.cuda(), "logits"), output=(pv, pi),
                            grid_dim=(nparts, 1, 1), block_dim=(128, 1, 1))
    pk.argmax_reduce_layer(input=(pv, pi), output=pk.attach_input(tok, "tok"), grid_dim=(1, 1, 1),
                           block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert torch.equal(out.cpu(), ops.embedding(ids, tab))
    assert tok.cpu().reshape(-1).tolist() == ops.argmax(logits).tolist()
    assert tok[1, 0].item() == 10


@pytest.mark.parametrize("token_budget", [0, 16])
@pytest.mark.parametrize("n_new,prefix,pages", [(3, 40, [2]), (1, 200, [1, 3, 0, 2]), (1, 63, [0]), (4, 124, [3, 1])])
def test_paged_attention(mi, golden_dir, n_new, prefix, pages, token_budget):
    """Fused QK-norm + RoPE + KV append + split-KV attention for one request; the (3, 40, [2]) case is
    the reference fixture (torch_multitoken_paged_attention).  A token budget of 16 selects the instantiation of
    the megakernel that serves many requests, whose attention tasks stream the cached rows through shared memory."""
    D, G, P = 128, 4, 64
    if (n_new, prefix) == (3, 40):
        f = torch.load(os.path.join(golden_dir, "ref_paged_attention.pt"), weights_only=False)
        qkv, kc, vc = f["qkv"], f["k_cache"].clone().unsqueeze(2), f["v_cache"].clone().unsqueeze(2)
        cos, sin, qn, kn = f["cos"], f["sin"], f["q_norm"].reshape(-1), f["k_norm"].reshape(-1)
    else:
        f = None
        qkv = _bf16(n_new, (G + 2) * D, seed=11)
        kc, vc = _bf16(4, P, 1, D, seed=12), _bf16(4, P, 1, D, seed=13)
        cos, sin = ops.rope_tables(D, 512, 1e6)
        qn, kn = _bf16(D, seed=14, scale=0.1, shift=1.0), _bf16(D, seed=15, scale=0.1, shift=1.0)
    seq_len = prefix + n_new
    assert len(pages) == (seq_len + P - 1) // P
    kc_ref, vc_ref = kc.clone(), vc.clone()
    ref = ops.paged_attention_request(qkv, kc_ref, vc_ref, pages, seq_len, G, 1, qn, kn, cos, sin, 1e-6)
    dev = "cuda"
    meta = {
        "qo_indptr_buffer": torch.tensor([0, n_new], dtype=torch.int32, device=dev),
        "paged_kv_indptr_buffer": torch.tensor([0, len(pages)], dtype=torch.int32, device=dev),
        "paged_kv_indices_buffer": torch.tensor(pages + [0] * (4 - len(pages)), dtype=torch.int32, device=dev),
        "paged_kv_last_page_len_buffer": torch.tensor([(seq_len - 1) % P + 1], dtype=torch.int32, device=dev),
    }
    pk = make_test_kernel(mi, max(n_new, token_budget), max_num_batched_requests=1, max_num_pages=4, page_size=P,
                          max_seq_length=256, meta_tensors=meta)
    kc_d, vc_d = kc.cuda(), vc.cuda()
    out = torch.zeros(n_new, G * D, dtype=torch.bfloat16, device=dev)
    pk.paged_attention_layer(
        input=pk.attach_input(qkv.cuda(), "qkv"), k_cache=pk.attach_input(kc_d, "kc"), v_cache=pk.attach_input(vc_d, "vc"),
        q_norm=pk.attach_input(qn.cuda(), "qn"), k_norm=pk.attach_input(kn.cuda(), "kn"),
        cos_pos_embed=pk.attach_input(cos.cuda(), "cos"), sin_pos_embed=pk.attach_input(sin.cuda(), "sin"),
        output=pk.attach_input(out, "out"), grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert rel_err(out.cpu(), ref) <= TOL
    assert rel_err(kc_d.cpu(), kc_ref) <= 1e-2 and torch.equal(vc_d.cpu(), vc_ref)
    if f is not None:
        assert rel_err(out.cpu().reshape(n_new * G, D), f["out"]) <= TOL


@pytest.mark.parametrize("token_budget", [0, 16])
@pytest.mark.parametrize("lens,new,hkv,max_seq", [([3000, 257], [1, 2], 2, 4096), ([4096], [1], 8, 4096),
                                                  ([700, 64, 1, 2049, 65], [1, 3, 1, 2, 1], 1, 4096)])
def test_paged_attention_long_context(mi, lens, new, hkv, max_seq, token_budget):
    """Long sequences: chunks are longer than the rows a task fetches ahead of its dependency, so the per-row loop,
    many pages per request and the merge of the maximum number of chunks are exercised; two requests of very
    different lengths share the launch in the first case."""
    D, G, P = 128, 4, 64
    R, mbt = len(lens), sum(new)
    total_pages = sum((n + P - 1) // P for n in lens) + 3
    g = torch.Generator().manual_seed(sum(lens))
    qkv = (torch.randn(mbt, hkv * (G + 2) * D, generator=g)).to(torch.bfloat16)
    kc = torch.randn(total_pages, P, hkv, D, generator=g).to(torch.bfloat16)
    vc = torch.randn(total_pages, P, hkv, D, generator=g).to(torch.bfloat16)
    cos, sin = ops.rope_tables(D, max_seq, 1e6)
    qn, kn = _bf16(D, seed=14, scale=0.1, shift=1.0), _bf16(D, seed=15, scale=0.1, shift=1.0)
    perm = torch.randperm(total_pages, generator=g).tolist()
    indptr, indices, last, qo = [0], [], [], [0]
    for n, nn in zip(lens, new):
        k = (n + P - 1) // P
        indices += perm[indptr[-1]:indptr[-1] + k]
        indptr.append(indptr[-1] + k)
        last.append((n - 1) % P + 1)
        qo.append(qo[-1] + nn)
    kc_ref, vc_ref = kc.clone(), vc.clone()
    ref = torch.cat([ops.paged_attention_request(qkv[qo[r]:qo[r + 1]], kc_ref, vc_ref, indices[indptr[r]:indptr[r + 1]],
                                                 lens[r], hkv * G, hkv, qn, kn, cos, sin, 1e-6) for r in range(R)])
    dev = "cuda"
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    meta = {"qo_indptr_buffer": i32(qo), "paged_kv_indptr_buffer": i32(indptr),
            "paged_kv_indices_buffer": i32(indices + [0] * (total_pages - len(indices))),
            "paged_kv_last_page_len_buffer": i32(last)}
    pk = make_test_kernel(mi, max(mbt, token_budget), max_num_batched_requests=R, max_num_pages=total_pages, page_size=P,
                          max_seq_length=max_seq, meta_tensors=meta)
    kc_d, vc_d = kc.cuda(), vc.cuda()
    out = torch.zeros(mbt, hkv * G * D, dtype=torch.bfloat16, device=dev)
    pk.paged_attention_layer(
        input=pk.attach_input(qkv.cuda(), "qkv"), k_cache=pk.attach_input(kc_d, "kc"), v_cache=pk.attach_input(vc_d, "vc"),
        q_norm=pk.attach_input(qn.cuda(), "qn"), k_norm=pk.attach_input(kn.cuda(), "kn"),
        cos_pos_embed=pk.attach_input(cos.cuda(), "cos"), sin_pos_embed=pk.attach_input(sin.cuda(), "sin"),
        output=pk.attach_input(out, "out"), grid_dim=(R, hkv, 1), block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    first = out.clone()
    assert rel_err(out.cpu(), ref) <= TOL
    assert rel_err(kc_d.cpu(), kc_ref) <= 1e-2 and torch.equal(vc_d.cpu(), vc_ref)
    # a second launch appends the same rows again and must reproduce the output bit for bit
    pk.run_test_mode()
    assert torch.equal(first, out)


class _Ranges:
    """One paged attention layer over requests of `lens` positions, the last new[r] of them appended by the launch."""

    def __init__(self, mi, hkv, G, page, lens, new, shift=0, **kw):
        self.hkv, self.G, self.page, self.lens, self.new = hkv, G, page, lens, new
        D, R, T = 128, len(lens), sum(new)
        g = torch.Generator().manual_seed(sum(lens))
        need = [(n + page - 1) // page for n in lens]
        total = sum(need) + 2
        self.perm = perm = torch.randperm(total, generator=g).tolist()
        self.indptr, self.qo = [0], [0]
        for n, k in zip(new, need):
            self.indptr.append(self.indptr[-1] + k)
            self.qo.append(self.qo[-1] + n)
        self.qkv = torch.randn(T, hkv * (G + 2) * D, generator=g).to(torch.bfloat16)
        kc, vc = (torch.randn(total, page, hkv, D, generator=g).to(torch.bfloat16) for _ in range(2))
        self.kc_ref, self.vc_ref = kc.clone(), vc.clone()
        for r, n in enumerate(lens):      # what lies behind a request's cached rows is never used
            for pos in range(n - new[r], need[r] * page):
                kc[self.row(r, pos)] = vc[self.row(r, pos)] = float("nan")
        self.tables = ops.rope_tables(D, max(lens) + 1, 1e6)
        self.qn, self.kn = _bf16(D, seed=14, scale=0.1, shift=1.0), _bf16(D, seed=15, scale=0.1, shift=1.0)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
        meta = {"qo_indptr_buffer": i32(self.qo), "paged_kv_indptr_buffer": i32(self.indptr), "paged_kv_indices_buffer": i32(perm),
                "paged_kv_last_page_len_buffer": i32([(n - 1) % page + 1 for n in lens])}
        self.params = dict(max_num_batched_requests=R, max_num_pages=total, page_size=page, max_seq_length=max(need) * page, meta_tensors=meta, **kw)
        self.kernel = lambda **params: make_test_kernel(mi, max(T, 16), **params)
        self.qkv_d, self.kc, self.vc = self.qkv.cuda(), kc.cuda(), vc.cuda()
        self.buffer = torch.full((T * hkv * G * D + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
        self.out = self.buffer[shift:shift + T * hkv * G * D].view(T, -1)
        self.pk = self.kernel(**self.params)
        self.layer(self.pk)
        self.pk.compile()

    def layer(self, pk, name=""):
        att = lambda t, what: pk.attach_input(t, what + name)
        pk.paged_attention_layer(
            input=att(self.qkv_d, "qkv"), k_cache=att(self.kc, "kc"), v_cache=att(self.vc, "vc"), q_norm=att(self.qn.cuda(), "qn"),
            k_norm=att(self.kn.cuda(), "kn"), cos_pos_embed=att(self.tables[0].cuda(), "cos"), sin_pos_embed=att(self.tables[1].cuda(), "sin"),
            output=att(self.out, "out"), grid_dim=(len(self.lens), self.hkv, 1), block_dim=(128, 1, 1))

    def row(self, r, pos):
        return self.perm[self.indptr[r] + pos // self.page], pos % self.page

    def launch(self):
        self.pk.run_test_mode()
        return self.out.clone()

    def reference(self):
        return torch.cat([ops.paged_attention_request(self.qkv[self.qo[r]:self.qo[r + 1]], self.kc_ref, self.vc_ref, self.perm[self.indptr[r]:self.indptr[r + 1]],
                                                      n, self.hkv * self.G, self.hkv, self.qn, self.kn, *self.tables, 1e-6)
                          for r, n in enumerate(self.lens) if self.new[r]])

    def check(self):
        ref, first = self.reference(), self.launch()
        assert rel_err(first.cpu(), ref) <= TOL
        kc, vc = self.kc.cpu(), self.vc.cpu()
        for r, n in enumerate(self.lens):
            for pos in range(n):
                at = self.row(r, pos)
                assert rel_err(kc[at], self.kc_ref[at]) <= 1e-2 and torch.equal(vc[at], self.vc_ref[at])
        assert torch.equal(first, self.launch())


# query tiles of 16 rows with one, some and all of them in use; requests shorter than a step, idle slots (on 148 workers all but the
# fifth share tiles)
@pytest.mark.parametrize("hkv,G,page,lens,new", [
    (1, 8, 8, [8, 1, 129, 17], [1, 1, 9, 3]),
    (3, 2, 24, [65, 200, 7], [16, 30, 7]),
    (16, 1, 64, [300, 40, 64], [17, 1, 1]),
    (2, 4, 16, [(i * 97) % 611 + 1 for i in range(40)], [0 if i % 7 == 3 else 1 for i in range(40)]),
    (8, 4, 64, [1500, 64], [60, 4]),
    (4, 1, 32, [2100, 31, 33], [12, 31, 2]),
])
def test_paged_attention_ranges(mi, hkv, G, page, lens, new):
    _Ranges(mi, hkv, G, page, lens, new).check()


def _form(hkv, G, lens, new, workers):
    """How the layer's steps are shared out: steps of a range (0: the warps of a worker share tiles), parts per tile, tiles and parts in all."""
    hh, workers = min(hkv & -hkv, 8), workers or torch.cuda.get_device_properties(0).multi_processor_count
    live = [(hkv * -(-t * G // 16), -(-n // 8)) for n, t in zip(lens, new) if t]
    steps, ranges = sum(nt // hh * S for nt, S in live), workers * (8 // hh)
    if steps >= ranges * 16:
        return -(-steps // ranges), [], 0
    parts = [max(1, min(S * workers // (steps * hh), 16 + S // 96, 64)) for _, S in live]
    if hkv * len(live) <= workers:      # a limit of steps instead of whole shares
        longest = max(-(-S // p) for (_, S), p in zip(live, parts))
        for k in range(8, 40):
            limit = -(-(-(-steps * hh // workers)) * k // 8)
            cut = [min(-(-S // limit), 16 + S // 96, 64) for _, S in live]
            if sum(nt * p for (nt, _), p in zip(live, cut)) <= workers and max(-(-S // p) for (_, S), p in zip(live, cut)) < longest:
                parts = cut
                break
    return 0, parts, sum(nt * p for (nt, _), p in zip(live, parts))


# ranges of steps: one, two, four and eight kv heads side by side (with fewer than eight a worker has several ranges), one and several
# groups of them; pages of one, three and eight steps; decoding batches, prompts, idle slots, requests shorter than a step
@pytest.mark.parametrize("workers,hkv,G,page,lens,new", [
    (2, 1, 8, 8, [600, 1, 700, 999, 64], [1, 1, 4, 0, 1]),
    (1, 3, 4, 24, [200, 65, 7, 300], [16, 30, 7, 1]),
    (3, 2, 1, 64, [(i * 97) % 211 + 1 for i in range(40)], [0 if i % 7 == 3 else 1 for i in range(40)]),
    (2, 6, 2, 8, [400, 33, 90], [9, 1, 24]),
    (4, 4, 4, 16, [1500, 3, 250, 31], [1, 1, 1, 1]),
    (3, 16, 1, 64, [300, 40, 64, 9], [17, 1, 1, 0]),
    (5, 24, 2, 24, [240, 100], [1, 40]),
])
def test_paged_attention_equal_ranges(mi, workers, hkv, G, page, lens, new):
    assert _form(hkv, G, lens, new, workers)[0] >= 16
    _Ranges(mi, hkv, G, page, lens, new, num_workers=workers).check()


# contiguous caches, one token a slot: steps that end behind a slot read its neighbour's first rows, the last slot's end behind the cache
@pytest.mark.parametrize("workers,seq", [(1, 100), (0, 100), (1, 96), (0, 13)])
def test_contiguous_attention_of_many_slots(mi, workers, seq):
    hkv, G, D, R = 2, 2, 128, 12
    lens = [(i * 41) % seq + 1 for i in range(R - 2)] + [seq - 1, seq]
    assert (_form(hkv, G, lens, [1] * R, workers)[0] > 0) == (workers == 1)
    qkv, kc, vc = _bf16(R, hkv * (G + 2) * D, seed=3), _bf16(R, seq, hkv, D, seed=4), _bf16(R, seq, hkv, D, seed=5)
    qn, kn, tables = _bf16(D, seed=14, scale=0.1, shift=1.0), _bf16(D, seed=15, scale=0.1, shift=1.0), ops.rope_tables(D, seq, 1e6)
    kc_ref, vc_ref = kc.clone(), vc.clone()
    ref = torch.cat([ops.paged_attention_request(qkv[r:r + 1], kc_ref, vc_ref, [r], n, hkv * G, hkv, qn, kn, *tables, 1e-6) for r, n in enumerate(lens)])
    for r, n in enumerate(lens):
        kc[r, n - 1:] = vc[r, n - 1:] = float("nan")
    pk = make_test_kernel(mi, R, num_workers=workers, meta_tensors={"step": torch.tensor([n - 1 for n in lens], dtype=torch.int32, device="cuda")})
    kc_d, vc_d, out = kc.cuda(), vc.cuda(), torch.zeros(R, hkv * G * D, dtype=torch.bfloat16, device="cuda")
    att = lambda t, name: pk.attach_input(t, name)
    pk.attention_layer(input=att(qkv.cuda(), "qkv"), k_cache=att(kc_d, "kc"), v_cache=att(vc_d, "vc"), q_norm=att(qn.cuda(), "qn"), k_norm=att(kn.cuda(), "kn"),
                       cos_pos_embed=att(tables[0].cuda(), "cos"), sin_pos_embed=att(tables[1].cuda(), "sin"), output=att(out, "out"),
                       grid_dim=(R, hkv, 1), block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    assert rel_err(out.cpu(), ref) <= TOL
    for r, n in enumerate(lens):
        assert rel_err(kc_d[r, :n].cpu(), kc_ref[r, :n]) <= 1e-2 and torch.equal(vc_d[r, :n].cpu(), vc_ref[r, :n])


# one long request among short ones: tiles of several parts beside whole ones, and more of them than workers
@pytest.mark.parametrize("workers,hkv,G,page,lens,new", [
    (8, 2, 4, 16, [20] * 9 + [700] + [23] * 11, [1] * 4 + [0, 3] + [1] * 15),
    (0, 8, 4, 64, [3000] + [40] * 18, [1] * 19),
    (0, 4, 8, 8, [1200] + [9, 30] * 20, [3] + [1, 2] * 20),
    (16, 3, 1, 24, [3, 500, 3, 1, 3, 17, 9], [3, 20, 1, 1, 2, 17, 0]),
])
def test_paged_attention_unequal_requests(mi, workers, hkv, G, page, lens, new):
    a = _Ranges(mi, hkv, G, page, lens, new, num_workers=workers)
    per, parts, items = _form(hkv, G, lens, new, workers)
    assert per == 0 and max(parts) > 1 and min(parts) == 1 and items > (workers or 148)
    a.check()


# few tiles of unlike lengths: cut by a limit of steps, every part at once
@pytest.mark.parametrize("workers,hkv,G,page,lens,new,parts", [
    (148, 8, 2, 64, [700, 1400, 870, 950, 1100, 1010, 1290, 780], [1] * 8, [2, 3, 2, 2, 2, 2, 3, 2]),   # (whole shares: 1 3 1 2 2 2 2 1)
    (148, 2, 4, 8, [90, 170, 120, 9] * 6, [1, 2, 1, 1] * 6, [3, 5, 3, 1] * 6),                          # (2 5 3 1 ..)
    (32, 4, 1, 16, [300, 170, 450], [1, 16, 3], [2, 2, 3]),                                             # (2 1 3)
])
def test_paged_attention_limited_parts(mi, workers, hkv, G, page, lens, new, parts):
    assert _form(hkv, G, lens, new, workers)[1] == parts
    _Ranges(mi, hkv, G, page, lens, new, num_workers=workers).check()


# more requests than the request table holds at once: two workers take ranges, all of them share tiles
@pytest.mark.parametrize("workers", [2, 0])
def test_paged_attention_many_requests(mi, workers):
    lens = [(i * 37) % 23 + 1 for i in range(1100)]
    lens[700] = 400
    a = _Ranges(mi, 2, 2, 8, lens, [0 if i % 11 == 5 else 1 for i in range(1100)], num_workers=workers)
    a.check()


# an output that starts on any element; one worker: whole tiles, two: merged ones as well, all of them: shared tiles
@pytest.mark.parametrize("workers", [1, 2, 0])
@pytest.mark.parametrize("shift", [1, 2])
def test_paged_attention_output_without_alignment(mi, workers, shift):
    lens, new = [300, 40, 90], [21, 1, 2]
    aligned, a = (_Ranges(mi, 2, 2, 16, lens, new, shift=k, num_workers=workers) for k in (0, shift))
    aligned.check()
    assert torch.equal(a.launch(), aligned.launch())
    edge = torch.cat([a.buffer[:shift], a.buffer[shift + a.out.numel():]])
    assert edge.numel() == 8 and bool((edge == 7.0).all())


# layers of different head counts that do not depend on one another: the request table is built again, and neither meets the other's records
@pytest.mark.parametrize("workers", [2, 0])
def test_paged_attention_layers_side_by_side(mi, workers):
    lens, new = [700, 40, 90, 1100], [1, 1, 2, 9]
    pair = [_Ranges(mi, hkv, G, 16, lens, new, num_workers=workers) for hkv, G in ((4, 2), (1, 8))]
    want = [a.launch() for a in pair]
    pk = pair[0].kernel(**pair[0].params)
    for i, a in enumerate(pair):
        a.out.zero_()
        a.layer(pk, str(i))
    pk.compile()
    for _ in range(20):
        pk.run_test_mode()
        for a, w in zip(pair, want):
            assert torch.equal(a.out, w)
            a.out.zero_()


# one worker: ranges of steps; all of them: the warps of a worker share a tile
@pytest.mark.parametrize("workers", [1, 0])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_paged_attention_value_rows_that_are_not_finite(mi, workers, bad):
    """A value row reaches the tokens that see its position and no others, bit for bit."""
    hkv, G, lens, new = 2, 1, [300, 40], [21, 5]
    a = _Ranges(mi, hkv, G, 16, lens, new, num_workers=workers)
    clean = a.launch()
    values = a.qkv_d.view(-1, hkv, G + 2, 128)[:, :, G + 1]
    for token, head, column in ((6, 0, 3), (13, 1, 127), (20, 0, 64), (22, 1, 0)):
        values[token, head, column] = bad
    out, sees = a.launch().view(-1, hkv, 128), clean.view(-1, hkv, 128).clone()
    for first, last, head, column in ((6, 21, 0, 3), (13, 21, 1, 127), (20, 21, 0, 64), (22, 26, 1, 0)):
        assert not out[first:last, head, column].isfinite().any()
        sees[first:last, head, column] = out[first:last, head, column]
    assert torch.equal(out.nan_to_num(7.0, 8.0), sees.nan_to_num(7.0, 8.0))


# (1 worker: tiles that lie in one range and tiles that are merged)
@pytest.mark.parametrize("workers", [1, 0])
def test_paged_attention_key_row_that_is_nan(mi, workers):
    """Rows of tokens that see a NaN score are zero, whichever way the positions are shared out; the others keep their bits."""
    a = _Ranges(mi, 2, 1, 16, [300, 40, 90], [21, 5, 2], num_workers=workers)
    clean = a.launch().view(-1, 2, 128)
    keys = a.qkv_d.view(-1, 2, 3, 128)[:, :, 1]
    for token, head in ((6, 0), (22, 1), (26, 0)):
        keys[token, head] = float("nan")
    for first, last, head in ((6, 21, 0), (22, 26, 1), (26, 28, 0)):
        clean[first:last, head] = 0
    assert torch.equal(a.launch().view(-1, 2, 128), clean)


# columns that start on no 16-byte boundary, fewer columns than a vector, fewer tokens than warps; equal maxima: the lowest column wins
@pytest.mark.parametrize("T,V,parts", [(1, 37, 5), (3, 1000, 7), (9, 4099, 148), (64, 777, 3)])
def test_argmax_partial_edges(mi, T, V, parts):
    g = torch.Generator().manual_seed(V)
    x = (torch.randint(-3, 4, (T, V), generator=g)).to(torch.bfloat16)
    x[0] = float("-inf")
    pk = make_test_kernel(mi, T)
    pv, pi = pk.new_tensor((T, parts), name="pv"), pk.new_tensor((T, parts), dtype=mi.int64, name="pi")
    out = torch.full((T, 1), -1, dtype=torch.int64, device="cuda")
    pk.argmax_partial_layer(input=pk.attach_input(x.cuda(), "x"), output=(pv, pi), grid_dim=(parts, 1, 1), block_dim=(128, 1, 1))
    pk.argmax_reduce_layer(input=(pv, pi), output=pk.attach_input(out, "out"), grid_dim=(1, 1, 1), block_dim=(128, 1, 1))
    pk.compile()
    pk.run_test_mode()
    want = torch.stack([(row == row.max()).nonzero()[0, 0] for row in x.float()])
    assert torch.equal(out[:, 0].cpu(), want)
