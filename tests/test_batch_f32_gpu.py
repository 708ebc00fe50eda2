"""The float32 product of 17 to 64 rows on tensor cores (csrc/linear_batch_f32.cu), through the entry that picks it."""
import pytest
import torch

from test_kernels_gpu import DEV, ops, rnd  # noqa: F401

pytestmark = pytest.mark.gpu


def _on_tensor_cores(ops, M, N, K):  # noqa: F811
    return bool(ops.library().mllm_linear_stream_f32_on_tensor_cores(M, N, K))


# one column, one ragged tile, a column over, slices of unequal length, rows of K that end inside a block, CTAs that walk several
# tiles; both widths of the row side at their edges.  The last five stay off the tensor cores at all or some row counts: rows
# under 768, and long rows of few columns up to 40 rows
@pytest.mark.parametrize("M", [17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(1, 768), (127, 772), (129, 1604), (300, 1604), (2304, 768), (19001, 2052), (50257, 768), (2500, 3076),
                                 (1, 128), (127, 132), (129, 520), (19001, 260), (640, 3076)])
def test_float32_product_of_a_batch(ops, M, N, K):  # noqa: F811
    assert _on_tensor_cores(ops, M, N, K) == (K >= 768 and (N != 640 or M > 40))
    x, w, b = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5), rnd(N, seed=3)
    ref = x.double() @ w.double().t()
    # four full-size additions of a block drop at most 2^-23 each, blocks, slices and bias add 2^-24 apiece
    bound = (K / 64 + 12) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t() + b.double().abs())
    full, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.linear(x, w, None, out=full)
    ops.linear(x, w, None, out=plain, impl="simt")
    assert torch.all((full - ref).abs() <= bound)
    # no further off than the chain of fmaf, but for what a single column's few results leave to chance
    assert (full - ref).norm() <= (1.02 if N > 1 else 2.0) * (plain - ref).norm() + 2.0 ** -24 * ref.norm() * (N == 1)
    big = torch.full((M + 1, N + 3), 7.0, device=DEV)
    big[:M, :N] = 1.5
    ops.linear(x, w, b, out=big[:M, :N], act="gelu_tanh", accumulate=True)
    want = torch.nn.functional.gelu(ref + b.double(), approximate="tanh") + 1.5
    assert torch.all((big[:M, :N] - want).abs() <= 1.2 * bound + 4e-7 * want.abs())
    assert torch.all(big[M] == 7.0) and torch.all(big[:, N:] == 7.0)
    wide = torch.zeros(M, K + 8, device=DEV)
    wide[:, 4:4 + K] = x
    part = torch.empty(17, N, device=DEV)
    ops.linear(wide[M - 17:, 4:4 + K], w, None, out=part)
    if ops.library().mllm_linear_stream_f32_kernel_of(17, N, K) == ops.library().mllm_linear_stream_f32_kernel_of(M, N, K):
        assert torch.equal(part, full[M - 17:])
    x[3, 5], x[9, 1], x[16, 0], w[0, 7], w[N // 2, 0] = float("inf"), float("nan"), 3.4e38, -float("inf"), 2.0
    ops.linear(x, w, None, out=full)
    ops.linear(x, w, None, out=plain, impl="simt")
    assert torch.equal(full.isnan(), plain.isnan()) and torch.equal(full.isinf(), plain.isinf())
    assert plain.isinf().any() and torch.equal(full.sign()[full.isinf()], plain.sign()[plain.isinf()])
    ops.check_device_errors()


# a vocabulary's few rows stay with the weights in registers while one pass of eight takes them
@pytest.mark.parametrize("K", [764, 768, 1600])
def test_float32_vocabulary_of_few_rows(ops, K):  # noqa: F811
    N = 38000
    w, x = rnd(N, K, seed=2, scale=K ** -0.5), rnd(16, K, seed=1)
    ref, mass = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
    for M in (1, 8, 9, 16):
        assert _on_tensor_cores(ops, M, N, K) == (K >= 768 and M > 8)
        out = torch.empty(M, N, device=DEV)
        ops.linear(x[:M], w, None, out=out)
        assert torch.all((out - ref[:M]).abs() <= (K / 64 + 12) * 2.0 ** -24 * mass[:M])
    ops.check_device_errors()


# rows that overlap, and one row for all
@pytest.mark.parametrize("stride", [0, 4, 760])
@pytest.mark.parametrize("M", [17, 64])
def test_float32_product_of_overlapping_rows(ops, M, stride):  # noqa: F811
    N, K = 300, 772
    x = rnd(stride * M + K, seed=1).as_strided((M, K), (stride, 1))
    w, out, want = rnd(N, K, seed=2, scale=K ** -0.5), torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    ops.linear(x, w, None, out=out)
    ops.linear(x.contiguous(), w, None, out=want)
    assert torch.equal(out, want)
    ops.check_device_errors()


def test_float32_projection_of_a_batch_writes_the_cache(ops):  # noqa: F811
    from mini_llm_b200.engine.context import Workspace
    M, H, Hkv, dh, page, K = 37, 5, 3, 48, 4, 804
    N, kv = (H + 2 * Hkv) * dh, Hkv * dh
    x, w, b = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5), rnd(N, seed=3)
    qkv = torch.empty(M, N, device=DEV)
    ops.linear(x, w, b, out=qkv)
    slots = torch.randperm(40 * page, generator=torch.Generator().manual_seed(4))[:M].to(torch.int32).to(DEV)
    wk, wv, gk, gv = (torch.full((40, Hkv, page, dh), 9.0, device=DEV) for _ in range(4))
    ops.kv_write(qkv[1:, H * dh:H * dh + kv], qkv[1:, H * dh + kv:], wk, wv, slots[1:])
    slots[0] = -1
    q = ops.linear_qkv_cache(x, w, b, torch.empty(M, H * dh, device=DEV), gk, gv, slots, Workspace(torch.device(DEV), 64))
    assert torch.equal(q, qkv[:, :H * dh]) and torch.equal(gk, wk) and torch.equal(gv, wv)
    ops.check_device_errors()
