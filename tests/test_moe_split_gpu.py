"""The float32 products of routed experts over many pairs on tensor cores (csrc/moe_split_f32.cu)."""
import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


# pairs per expert: full and ragged tiles, an empty expert, one that has them all; columns that end inside a tile, K inside a block
# of both products, rows of the second's result that are not 16-byte aligned; products that stay on CUDA cores (short or odd K)
@pytest.mark.parametrize("counts", [[64], [128, 0, 1, 129, 70], [7] * 40, [0, 300]])
@pytest.mark.parametrize("F,D,top,act", [(512, 768, 2, "silu"), (33, 132, 1, "swiglu_clamp"), (100, 260, 2, "relu_sq"), (132, 772, 2, "silu"),
                                         (260, 302, 1, "relu_sq"), (129 * 4, 300, 2, "swiglu_clamp")])
def test_routed_experts_in_float32(ops, monkeypatch, counts, F, D, top, act):  # noqa: F811
    E, pairs = len(counts), sum(counts)
    pairs -= pairs % top
    counts = list(counts)
    counts[counts.index(max(counts))] -= sum(counts) - pairs
    order = torch.randperm(pairs, generator=torch.Generator().manual_seed(1)).to(torch.int32).to(DEV)
    offsets = torch.tensor([sum(counts[:e]) for e in range(E + 1)], dtype=torch.int32, device=DEV)
    gated = act != "relu_sq"
    h = rnd(pairs // top, D, seed=2)
    w1, w2 = rnd(E, F * (2 if gated else 1), D, seed=3, scale=D ** -0.5), rnd(E, D, F, seed=4, scale=F ** -0.5)
    mid, out = torch.full((pairs, F), 7.0, device=DEV), torch.full((pairs, D), 7.0, device=DEV)
    limit = 3.0 if act == "swiglu_clamp" else 0.0

    names, call = [], ops._call
    monkeypatch.setattr(ops, "_call", lambda name, *args: (names.append(name), call(name, *args))[1])

    def run(split):
        ops.use_moe_split_f32 = split
        try:
            ops.moe_grouped(h, w1, mid, offsets, order, top=top, first=True, act=act, limit=limit, alpha=1.7)
            first = mid.clone()
            ops.moe_grouped(mid, w2, out, offsets, order, top=top, first=False)
        finally:
            ops.use_moe_split_f32 = True
        return first, out.clone()

    expert = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).to(DEV)
    x = h.double()[order.long() // top]
    y = torch.stack([w1[e].double() @ r for e, r in zip(expert.tolist(), x)])
    if act == "relu_sq":
        want = torch.relu(y) ** 2
    else:
        g, u = y[:, :F], y[:, F:]
        if act == "silu":
            want = torch.nn.functional.silu(g) * u
        else:
            g, u = g.clamp(max=limit), u.clamp(-limit, limit)
            want = g * torch.sigmoid(1.7 * g) * (u + 1.0)
    got = run(True)
    assert names == ["mllm_moe_split_f32" if k % 4 == 0 and k >= 128 else "mllm_moe_grouped" for k in (D, F)]
    plain = run(False)
    assert names[2:] == ["mllm_moe_grouped"] * 2
    assert (got[0] - want).abs().max() < 2e-5 * max(1.0, want.abs().max().item())
    assert (got[0] - want).norm() <= 1.1 * (plain[0] - want).norm()
    want2 = torch.empty(pairs, D, dtype=torch.float64, device=DEV)
    want2[order.long()] = torch.stack([w2[e].double() @ r for e, r in zip(expert.tolist(), got[0].double())])
    assert (got[1] - want2).abs().max() < 2e-5 * max(1.0, want2.abs().max().item())
    # infinities and NaN where the chains of fmaf have them
    h[1, 3], w1[E - 1, 0, 5] = float("inf"), float("nan")
    got, plain = run(True), run(False)
    for a, b in zip(got, plain):
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf())
        assert torch.equal(a.sign()[a.isinf()], b.sign()[b.isinf()])
    ops.check_device_errors()


# more experts than the routing kernels take, with weights or identity ones: the CUDA-core, mma.sync and few-pairs kernels
@pytest.mark.parametrize("E,identity", [(1100, 0), (512, 0), (300, 300)])
@pytest.mark.parametrize("pairs", [20, 300])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_experts_beyond_the_routing_kernels_number(ops, dtype, pairs, E, identity):  # noqa: F811
    F, D = 24, 136
    g = torch.Generator().manual_seed(pairs + E)
    expert = torch.randint(0, E + identity, (pairs,), generator=g)
    expert[0], expert[1] = 0, E + identity - 1
    order = torch.argsort(expert, stable=True)
    offsets = torch.searchsorted(expert[order].contiguous(), torch.arange(E + identity + 1)).to(torch.int32).to(DEV)
    h = rnd(pairs, D, seed=2, dtype=dtype)
    w1 = rnd(E, 2 * F, D, seed=3, scale=D ** -0.5, dtype=dtype)
    w2 = rnd(E, D, F, seed=4, scale=F ** -0.5, dtype=dtype)
    mid, out = torch.zeros(pairs, F, dtype=dtype, device=DEV), torch.full((pairs, D), 7.0, device=DEV)
    perm = order.to(torch.int32).to(DEV)
    ops.moe_grouped(h, w1, mid, offsets, perm, top=1, first=True, identity=identity)
    ops.moe_grouped(mid, w2, out, offsets, perm, top=1, first=False, identity=identity, self_rows=h if identity else None)
    eps = 2e-5 if dtype == torch.float32 else 1e-2
    for i, (p, e) in enumerate(zip(order.tolist(), expert[order].tolist())):
        x = h[p].double()
        if e >= E:
            assert torch.equal(out[p], h[p].float())
            continue
        y = w1[e].double() @ x
        y = torch.nn.functional.silu(y[:F]) * y[F:]
        assert (mid[i].double() - y).abs().max() <= eps * max(1.0, y.abs().max().item())
        want = w2[e].double() @ mid[i].double()
        assert (out[p].double() - want).abs().max() <= 2e-5 * max(1.0, want.abs().max().item())
    ops.check_device_errors()


# two or eight columns a warp, by the waves of either: the same bits as every pair alone
@pytest.mark.parametrize("pairs,E,F,D", [(24, 8, 512, 768), (32, 8, 500, 1028), (9, 40, 1030, 130), (17, 3, 2048, 516)])
def test_few_pairs_have_the_bits_of_every_pair_alone(ops, pairs, E, F, D):  # noqa: F811
    expert = torch.randint(0, E, (pairs,), generator=torch.Generator().manual_seed(pairs)).sort().values
    h, w1, w2 = rnd(pairs, D, seed=2), rnd(E, 2 * F, D, seed=3, scale=D ** -0.5), rnd(E, D, F, seed=4, scale=F ** -0.5)

    def run(rows):
        n = rows.stop - rows.start
        order = torch.arange(n, dtype=torch.int32, device=DEV)
        offsets = torch.searchsorted(expert[rows].contiguous(), torch.arange(E + 1)).to(torch.int32).to(DEV)
        mid, out = torch.full((n, F), 7.0, device=DEV), torch.full((n, D), 7.0, device=DEV)
        ops.moe_grouped(h[rows], w1, mid, offsets, order, top=1, first=True)
        ops.moe_grouped(mid, w2, out, offsets, order, top=1, first=False)
        return mid, out

    mid, out = run(slice(0, pairs))
    for i in range(pairs):
        y = w1[expert[i]].double() @ h[i].double()
        y = torch.nn.functional.silu(y[:F]) * y[F:]
        assert (mid[i] - y).abs().max() < 2e-5 * max(1.0, y.abs().max().item())
        want = w2[expert[i]].double() @ mid[i].double()
        assert (out[i] - want).abs().max() < 2e-5 * max(1.0, want.abs().max().item())
        alone = run(slice(i, i + 1))
        assert torch.equal(alone[0][0], mid[i]) and torch.equal(alone[1][0], out[i])
    ops.check_device_errors()
