"""Launches that do not wait for the launch before them: replayed many times between the kernels that write what they read and
the ones that read what they write, they leave the bits of launches that run one after the other."""
import pytest
import torch

from test_kernels_gpu import DEV, _ctx_for, _paged_case, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


def _replayed(ops, run, outs, fresh):
    """``run`` captured and replayed on changing inputs against the same launches without programmatic dependent launch."""
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        run()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            run()
        for i in range(12):
            fresh(i)
            graph.replay()
            stream.synchronize()
            got = [o.clone() for o in outs]
            ops.set_pdl(False)
            try:
                run()
                stream.synchronize()
            finally:
                ops.set_pdl(True)
            for g, o in zip(got, outs):
                assert torch.equal(g, o), i
    ops.check_device_errors()


def _beside_portions(ops, dtype, seqs, dh, window=None, num_pages=1200):
    """A projection that writes the cache, the portions' attention with the single tokens' beside it and an output product,
    replayed; returns which attention kernels were launched."""
    from mini_llm_b200.engine.context import ATTN_TILE_WIDE, attention_tiles, single_runs
    H = Hkv = 12
    page, D = 16, 12 * dh
    case = _paged_case(dtype, seqs, H, Hkv, dh, page, num_pages=num_pages, seed=5)
    ctx = _ctx_for(case)
    q_lens, starts = [n for _, n in seqs], [c - n for c, n in seqs]
    T = sum(q_lens)
    ctx.decode_only = False
    for name, rows in (("", 64), ("_wide", ATTN_TILE_WIDE)):
        tiles = attention_tiles(q_lens, starts, rows, singles_last=True)
        setattr(ctx, "attn_tiles" + name, torch.tensor(tiles, dtype=torch.int32, device=DEV))
        setattr(ctx, "n_tiles" + name, len(tiles) // 3)
    ctx.single_runs = single_runs(q_lens)
    ctx.max_single_ctx_len = max(c for c, n in seqs if n == 1)
    slots = torch.tensor([int(case["bt"][s, p // page]) * page + p % page
                          for s, p in zip(case["token_seq"], case["positions"])], dtype=torch.int32, device=DEV)
    kp, vp, bt = case["k_pages"].to(dtype).to(DEV), case["v_pages"].to(dtype).to(DEV), case["bt"].to(DEV)
    w_in, w_out = rnd(3 * D, D, seed=1, scale=D ** -0.5, dtype=dtype), rnd(D, D, seed=2, scale=D ** -0.5, dtype=dtype)
    x, q, att = (torch.empty(T, D, dtype=dtype, device=DEV) for _ in range(3))
    y = torch.empty(T, D, device=DEV)

    def run():
        with ops.stream_scope(ctx.ws):
            queries = ops.linear_qkv_cache(x, w_in, None, q, kp, vp, slots, ctx.ws)
            ops.paged_attention(queries, kp, vp, bt, ctx, att, num_heads=H, num_kv_heads=Hkv, head_dim=dh, scale=dh ** -0.5,
                                window=window)
            ops.linear(att, w_out, None, out=y)

    x.copy_(rnd(T, D, seed=3, dtype=dtype))
    before = dict(ops.attention_launches)
    _replayed(ops, run, [att, y], lambda i: x.copy_(rnd(T, D, seed=10 + i, dtype=dtype)))
    return {k for k, n in ops.attention_launches.items() if n > before.get(k, 0)}


# (context, new tokens): one run of single tokens, several, many behind a portion whose tiles fill the GPU, runs that share scratch
@pytest.mark.parametrize("seqs", [[(500, 200), (300, 1), (90, 1)], [(700, 1), (260, 130), (33, 1), (150, 1)],
                                  [(640, 640)] + [(37 * i + 5, 1) for i in range(20)],
                                  [(1100, 1), (200, 200), (1200, 1), (70, 1)]])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_single_tokens_beside_portions(ops, dtype, seqs):  # noqa: F811
    assert "decode" in _beside_portions(ops, dtype, seqs, 64)


# every kernel that portions may take, with heads that decode attention stages and heads that it does not, with and without a window
@pytest.mark.parametrize("dtype,dh,window,seqs,portions", [
    (torch.float32, 32, None, [(700, 400), (300, 1), (90, 1)], "tiled_wide"),
    (torch.float32, 16, 100, [(400, 400), (33, 1), (260, 1)], "tiled_wide"),
    (torch.float32, 128, None, [(300, 60), (90, 1), (500, 1)], "tiled"),
    (torch.float32, 64, 130, [(640, 300), (400, 1), (131, 1)], "split_f32"),
    (torch.bfloat16, 128, 50, [(300, 300), (90, 1), (500, 1)], "flash"),
    (torch.bfloat16, 16, None, [(200, 60), (300, 1), (33, 1)], "flash"),
    (torch.bfloat16, 64, 200, [(900, 512), (700, 1), (201, 1)], "flash_tc")])
def test_single_tokens_beside_every_kernel_of_portions(ops, dtype, dh, window, seqs, portions):  # noqa: F811
    assert _beside_portions(ops, dtype, seqs, dh, window, num_pages=160) == {portions, "decode"}


# several layers: every layer's projection lies at the same addresses, and SMs that run nothing between two layers keep what the
# last one left in their L1
@pytest.mark.parametrize("layers", [1, 4])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("seqs", [[(300, 1), (513, 1), (7, 1)], [(200, 200), (90, 30), (64, 1)], [(5, 1)]])
def test_recurrence_beside_biased_attention(ops, dtype, seqs, layers):  # noqa: F811
    from mini_llm_b200.engine.context import attention_tiles
    H, Hkv, dh, R, ek, ev, page, D = 12, 4, 64, 3, 32, 128, 16, 768
    case = _paged_case(dtype, seqs, H, Hkv, dh, page, num_pages=120, seed=6)
    ctx = _ctx_for(case)
    q_lens, starts = [n for _, n in seqs], [c - n for c, n in seqs]
    T, S, qs, rs = sum(q_lens), len(seqs), H * dh, R * ek
    ctx.S, ctx.decode_only, ctx.n_tiles = S, max(q_lens) == 1, 0
    if not ctx.decode_only:
        tiles = attention_tiles(q_lens, starts)
        ctx.attn_tiles, ctx.n_tiles = torch.tensor(tiles, dtype=torch.int32, device=DEV), len(tiles) // 3
    ctx.cu_q = torch.tensor([sum(q_lens[:i]) for i in range(S + 1)], dtype=torch.int32, device=DEV)
    ctx.state_slots = torch.arange(S, dtype=torch.int32, device=DEV)
    kp, vp, bt = case["k_pages"].to(dtype).to(DEV), case["v_pages"].to(dtype).to(DEV), case["bt"].to(DEV)
    w_in = rnd(qs + 2 * rs + R * ev, D, seed=1, scale=D ** -0.5, dtype=dtype)
    w_out = rnd(D, qs + R * ev, seed=2, scale=D ** -0.5, dtype=dtype)
    f_bias, lower, norm = rnd(rs, seed=3), torch.full((rs,), 0.2, device=DEV), rnd(ev, seed=4) + 1.0
    bias = -0.3 * torch.log1p(torch.arange(600, device=DEV).float()).expand(H, -1).contiguous()
    state0 = rnd(layers, S, R, ek, ev, seed=7)
    state, x, x2 = state0.clone(), torch.empty(T, D, dtype=dtype, device=DEV), torch.empty(T, D, dtype=dtype, device=DEV)
    proj = torch.empty(T, w_in.shape[0], dtype=dtype, device=DEV)
    mid = torch.empty(T, w_out.shape[1], dtype=dtype, device=DEV)

    def run():
        state.copy_(state0)
        with ops.stream_scope(ctx.ws):
            for i in range(layers):
                ops.linear(x2 if i else x, w_in, None, out=proj)
                r = proj[:, qs:]
                ops.biased_attention(
                    proj[:, :qs], kp, vp, bt, ctx, mid[:, :qs], num_heads=H, num_kv_heads=Hkv, scale=0.125, dist_bias=bias,
                    company=lambda: ops.gated_recurrence(r[:, :rs], r[:, rs:2 * rs], r[:, 2 * rs:], f_bias, lower, norm, 1e-5,
                                                         state[i], ctx, mid[:, qs:], heads=R, beside=True))
                ops.linear(mid, w_out, None, out=x2)

    x.copy_(rnd(T, D, seed=3, dtype=dtype))
    _replayed(ops, run, [mid, x2, state], lambda i: x.copy_(rnd(T, D, seed=10 + i, dtype=dtype)))
