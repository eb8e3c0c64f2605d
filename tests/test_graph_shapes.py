"""Dependency structure of multi-branch graphs (dry run, no CUDA call): who waits for whom after folding and
transitive reduction, and that the host simulation of the event protocol runs every task exactly once."""
import json

import pytest
import torch

import mirage_b200 as mi
from graph_shapes import KINDS, build


def _compile(kind, B=8, H=512):
    params = mi.PersistentKernel.get_default_init_parameters()
    params.update(test_mode=True, num_workers=0, max_num_batched_tokens=B, max_num_batched_requests=B, dry_run=True)
    pk = mi.PersistentKernel(**params)
    build(pk, kind, B, H, "meta")
    pk.compile()                       # includes simulate_task_graph: a deadlock or a miscounted event is an error
    g = json.loads(pk.dump_task_graph())
    by_out = {e["out"]: e for e in g["events"]}
    deps = {e["out"]: sorted(g["events"][d[0]]["out"] for d in e["deps"]) for e in g["events"]}
    return g, by_out, deps


def test_fork_two_consumers_wait_for_one_producer():
    g, ev, deps = _compile("fork")
    assert deps["xa"] == [] and deps["xb"] == ["xa"] and deps["xc"] == ["xa"]
    # every task of the producer must have finished: the consumers need all its arrivals
    a = ev["xa"]
    assert all(d[1] == a["tasks"] for e in (ev["xb"], ev["xc"]) for d in e["deps"])


def test_join_consumer_waits_for_both_producers():
    g, ev, deps = _compile("join")
    assert deps["xc"] == ["xa", "xb"]


def test_diamond():
    g, ev, deps = _compile("diamond")
    # xa is only read by the two linears, but it is a caller-visible buffer: the norm is not folded away
    assert deps["xb"] == ["xa"] and deps["xc"] == ["xa"] and deps["xd"] == ["xb", "xc"]


def test_residual_shortcut_is_covered_by_the_longer_path():
    g, ev, deps = _compile("residual_shortcut")
    # C reads xa (residual) and xb; xb's producer already waited for xa: transitive reduction leaves one edge
    assert deps["xc"] == ["xb"]


@pytest.mark.parametrize("kind", ["join_and_fork_consumer", "fork_and_join_producer"])
def test_role_combinations_the_reference_refuses_are_plain_graphs_here(kind):
    g, ev, deps = _compile(kind)
    if kind == "join_and_fork_consumer":
        assert deps["xb"] == ["xa", "xe"] and deps["xc"] == ["xa"]
    else:
        assert deps["xc"] == ["xa"] and deps["xd"] == ["xa", "xe"]


@pytest.mark.parametrize("B,H", [(4, 4096), (8, 4096), (16, 4096), (8, 2048)])
def test_fork_over_batch_and_width_sweep(B, H):
    g, ev, deps = _compile("fork", B, H)
    assert ev["xa"]["tasks"] == min(B, 148) and deps["xb"] == ["xa"] and deps["xc"] == ["xa"]


def test_more_than_three_independent_producers_is_refused_with_a_message():
    """The limit of this runtime's task record (three dependency slots) is reported at compile time with a message:
    a linear whose input, residual and WEIGHT come from three different layers and whose output buffer was written by
    a fourth needs four waits."""
    import torch
    params = mi.PersistentKernel.get_default_init_parameters()
    params.update(test_mode=True, num_workers=0, max_num_batched_tokens=4, max_num_batched_requests=4, dry_run=True)
    mk = lambda *s: torch.empty(*s, dtype=torch.bfloat16, device="meta")

    def graph(with_fourth):
        pk = mi.PersistentKernel(**params)
        x, w = pk.attach_input(mk(4, 256), "x"), pk.attach_input(mk(256), "w")
        w0, w1, wl = pk.attach_input(mk(256, 256), "w0"), pk.attach_input(mk(256, 256), "w1"), pk.attach_input(mk(256, 256), "wl")
        a, b, out = pk.attach_input(mk(4, 256), "a"), pk.attach_input(mk(4, 256), "b"), pk.attach_input(mk(4, 256), "out")
        pk.rmsnorm_layer(input=x, weight=w, output=a, grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
        pk.rmsnorm_layer(input=x, weight=w, output=b, grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
        pk.elementwise_add_layer(input_a=w0, input_b=w1, output=wl, grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
        if with_fourth:
            pk.rmsnorm_layer(input=x, weight=w, output=out, grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
        pk.linear_with_residual_layer(input=a, weight=wl, residual=b, output=out, grid_dim=(4, 1, 1), block_dim=(128, 1, 1))
        return pk

    graph(False).compile()
    with pytest.raises(mi.MpkError) as e:
        graph(True).compile()
    assert "more than 3" in str(e.value)


def test_overlapping_views_of_one_allocation_are_ordered():
    """Two attached tensors that alias without sharing a base pointer (a row-offset view of a buffer) must share a
    storage: the layer that reads the view waits for the layer that wrote the buffer."""
    import ctypes as C
    from mirage_b200 import _native as N
    cfg = N.MpkConfig()
    cfg.test_mode, cfg.dry_run, cfg.world_size, cfg.num_workers = 1, 1, 1, 8
    cfg.max_num_batched_tokens = cfg.max_num_batched_requests = 4
    h = C.c_void_p()
    N.check(h, N.lib.mpk_create(C.byref(cfg), C.byref(h)))

    def attach(name, ptr, rows, cols):
        dims = (C.c_int64 * 2)(rows, cols)
        return N.check(h, N.lib.mpk_attach_tensor(h, name.encode(), C.c_void_p(ptr), N.BF16, 2, dims, None))

    base = 0x10000000
    x = attach("x", base + 0x100000, 4, 256)
    w = attach("w", base + 0x200000, 1, 256)
    buf = attach("buf", base, 8, 256)                       # rows 0..7
    view = attach("view", base + 4 * 256 * 2, 4, 256)       # rows 4..7 of the same memory
    out = attach("out", base + 0x300000, 4, 256)
    grid = (C.c_int * 3)(4, 1, 1)
    ids = lambda *v: (C.c_int * len(v))(*v)
    N.check(h, N.lib.mpk_add_layer(h, N.OP_RMSNORM, ids(x, w, buf), 3, grid, None, 0))       # writes rows 0..3 of buf
    N.check(h, N.lib.mpk_add_layer(h, N.OP_RMSNORM, ids(view, w, out), 3, grid, None, 0))    # reads the overlapping view
    N.check(h, N.lib.mpk_compile(h))
    n = N.lib.mpk_dump_task_graph(h, None, 0)
    b = C.create_string_buffer(int(n))
    N.lib.mpk_dump_task_graph(h, b, n)
    ev = json.loads(b.value.decode())["events"]
    assert [d[0] for d in ev[1]["deps"]] == [0]
    N.lib.mpk_destroy(h)


def test_expert_projection_refuses_misaligned_scale_tensors():
    """The FP8 expert projection copies scales and rows 16 bytes at a time: tensors that do not start on a 16-byte
    boundary are refused when the graph is compiled (an error return, not a device fault)."""
    import ctypes as C
    from mirage_b200 import _native as N
    E, topk, n, k, b = 4, 2, 256, 512, 4

    def build(scale_offset):
        cfg = N.MpkConfig()
        cfg.test_mode, cfg.dry_run, cfg.world_size, cfg.num_workers = 1, 1, 1, 4
        cfg.max_num_batched_tokens = cfg.max_num_batched_requests = b
        h = C.c_void_p()
        N.check(h, N.lib.mpk_create(C.byref(cfg), C.byref(h)))

        def attach(name, ptr, dtype, *shape):
            dims = (C.c_int64 * len(shape))(*shape)
            return N.check(h, N.lib.mpk_attach_tensor(h, name.encode(), C.c_void_p(ptr), dtype, len(shape), dims, None))

        base = 0x20000000
        t = [attach("xq", base, N.F8E4M3, b, k), attach("xs", base + 0x100000, N.F32, b, k // 128),
             attach("w", base + 0x200000, N.F8E4M3, E, n, k), attach("ws", base + 0x400000 + scale_offset, N.F32, E, n, k // 128),
             attach("idx", base + 0x500000, N.I32, E, b), attach("mask", base + 0x600000, N.I32, E + 1),
             attach("out", base + 0x700000, N.BF16, b, topk, n)]
        grid = (C.c_int * 3)(4, 1, 1)
        N.check(h, N.lib.mpk_add_layer(h, N.OP_MOE_W13_FP8, (C.c_int * 7)(*t), 7, grid, None, 0))
        try:
            N.check(h, N.lib.mpk_compile(h))
        finally:
            N.lib.mpk_destroy(h)

    build(0)
    with pytest.raises(N.MpkError, match="16-byte"):
        build(4)


def _attention_and_fp8_linear(tokens, requests, heads, kv, K):
    meta = lambda dtype, *s: torch.empty(*s, dtype=dtype, device="meta")
    i32 = lambda n: meta(torch.int32, n)
    params = mi.PersistentKernel.get_default_init_parameters()
    params.update(test_mode=True, num_workers=148, max_num_batched_tokens=tokens, max_num_batched_requests=requests, dry_run=True, page_size=64,
                  max_num_pages=requests, max_seq_length=64,
                  meta_tensors={"qo_indptr_buffer": i32(requests + 1), "paged_kv_indptr_buffer": i32(requests + 1), "paged_kv_indices_buffer": i32(requests),
                                "paged_kv_last_page_len_buffer": i32(requests)})
    pk = mi.PersistentKernel(**params)
    att = lambda name, dtype, *s: pk.attach_input(meta(dtype, *s), name)
    bf = torch.bfloat16
    grid = dict(grid_dim=(requests, kv, 1), block_dim=(128, 1, 1))
    caches = [att(n, bf, requests, 64, kv, 128) for n in ("k", "v")]
    out = att("attention", bf, tokens, heads * 128)
    pk.paged_attention_layer(input=att("qkv", bf, tokens, (heads + 2 * kv) * 128), k_cache=caches[0], v_cache=caches[1], q_norm=att("qn", bf, 128), k_norm=att("kn", bf, 128),
                             cos_pos_embed=att("cos", bf, 64, 128), sin_pos_embed=att("sin", bf, 64, 128), output=out, **grid)
    if K:
        xq, xs = att("xq", torch.float8_e4m3fn, tokens, K), pk.new_tensor((tokens, K // 512), dtype=mi.uint32, name="xs")
        pk.quantize_fp8_layer(input=att("x", bf, tokens, K), output_fp8=xq, output_scale=xs, **grid)
        pk.linear_fp8_layer(input_fp8=xq, input_scale=xs, weight_fp8=att("w", torch.float8_e4m3fn, 512, K), weight_scale=att("ws", torch.uint32, 512, K // 512),
                            output=att("y", bf, tokens, 512), **grid)
    pk.compile()
    return json.loads(pk.dump_task_graph())


@pytest.mark.parametrize("tokens,heads,kv", [(1, 32, 8), (8, 32, 8), (8, 8, 1), (4, 4, 4)])
def test_few_token_graphs_with_attention_keep_four_weight_stages(tokens, heads, kv):
    g = _attention_and_fp8_linear(tokens, tokens, heads, kv, 4096)
    assert g["num_stages"] == 4 and g["stage_bytes"] == 33024
    # two copy stages and a query tile for each of eight warps, from a 1 KB boundary behind the weight stages
    pad = -g["num_stages"] * g["stage_bytes"] % 1024
    assert g["x_tile_bytes"] + 8192 >= pad + 8 * 3 * 4096


@pytest.mark.parametrize("requests", [512, 513, 1400, 8000])
def test_attention_of_any_number_of_requests_fits_shared_memory(requests):
    assert _attention_and_fp8_linear(requests, requests, 8, 2, 0)["num_stages"] >= 2


@pytest.mark.parametrize("depends", [False, True])
def test_attention_layers_share_scratch_only_in_a_chain(depends):
    """The second layer of a chain starts after the first one's merges; layers that are free to overlap have records of their own."""
    meta = lambda dtype, *s: torch.empty(*s, dtype=dtype, device="meta")
    bf, requests, heads, kv = torch.bfloat16, 16, 8, 2
    one = _attention_and_fp8_linear(requests, requests, heads, kv, 0)
    params = mi.PersistentKernel.get_default_init_parameters()
    i32 = lambda n: meta(torch.int32, n)
    params.update(test_mode=True, num_workers=148, max_num_batched_tokens=requests, max_num_batched_requests=requests, dry_run=True, page_size=64,
                  max_num_pages=requests, max_seq_length=64,
                  meta_tensors={"qo_indptr_buffer": i32(requests + 1), "paged_kv_indptr_buffer": i32(requests + 1), "paged_kv_indices_buffer": i32(requests),
                                "paged_kv_last_page_len_buffer": i32(requests)})
    pk = mi.PersistentKernel(**params)
    att = lambda name, *s: pk.attach_input(meta(bf, *s), name)
    norms = dict(q_norm=att("qn", 128), k_norm=att("kn", 128), cos_pos_embed=att("cos", 64, 128), sin_pos_embed=att("sin", 64, 128),
                 grid_dim=(requests, kv, 1), block_dim=(128, 1, 1))
    qkv = att("qkv", requests, (heads + 2 * kv) * 128)
    for i in range(2):
        out = att(f"out{i}", requests, heads * 128)
        pk.paged_attention_layer(input=qkv, k_cache=att(f"k{i}", requests, 64, kv, 128), v_cache=att(f"v{i}", requests, 64, kv, 128), output=out, **norms)
        if depends:
            qkv = att("next", requests, (heads + 2 * kv) * 128)
            pk.linear_layer(input=out, weight=att(f"w{i}", (heads + 2 * kv) * 128, heads * 128), output=qkv, grid_dim=(64, 1, 1), block_dim=(128, 1, 1))
    pk.compile()
    both = json.loads(pk.dump_task_graph())
    assert one["attn_scratch_floats"] > 0 and both["attn_scratch_floats"] == (1 if depends else 2) * one["attn_scratch_floats"]


def test_attention_names_a_misaligned_cache():
    """The general kernel copies cached rows by tensor maps: a cache that starts on no 16-byte boundary is refused by its name."""
    import ctypes as C
    from mirage_b200 import _native as N
    tokens, hkv, G, seq = 16, 2, 2, 64

    def build(offset):
        cfg = N.MpkConfig()
        cfg.test_mode, cfg.dry_run, cfg.world_size, cfg.num_workers = 1, 1, 1, 4
        cfg.max_num_batched_tokens = cfg.max_num_batched_requests = tokens
        h = C.c_void_p()
        N.check(h, N.lib.mpk_create(C.byref(cfg), C.byref(h)))

        def attach(name, ptr, *shape):
            return N.check(h, N.lib.mpk_attach_tensor(h, name.encode(), C.c_void_p(ptr), N.BF16, len(shape), (C.c_int64 * len(shape))(*shape), None))

        base = 0x20000000
        t = [attach("qkv", base, tokens, hkv * (G + 2) * 128), attach("keys", base + 0x1000000, tokens, seq, hkv, 128),
             attach("values", base + 0x2000000 + offset, tokens, seq, hkv, 128), -1, -1, -1, -1, attach("out", base + 0x3000000, tokens, hkv * G * 128)]
        N.check(h, N.lib.mpk_add_layer(h, N.OP_ATTENTION, (C.c_int * 8)(*t), 8, (C.c_int * 3)(tokens, hkv, 1), (C.c_int64 * 4)(hkv * G, hkv, 0, 0), 4))
        try:
            N.check(h, N.lib.mpk_compile(h))
        finally:
            N.lib.mpk_destroy(h)

    build(0)
    with pytest.raises(N.MpkError, match="kv cache starts on a 16-byte boundary: values"):
        build(8)
