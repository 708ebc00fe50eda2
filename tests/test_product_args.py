"""What the products' entry points check and choose on the host, without a GPU: the functions of ops run on CPU tensors with
the launch itself replaced by a recorder, so nothing is computed and no address is used."""
import pytest
import torch


@pytest.fixture
def ops(monkeypatch):
    from mini_llm_b200 import ops

    def named(name, t, dtype=None, contiguous=True):
        if dtype is not None and t.dtype != dtype:
            raise ops.KernelError(f"{name} must be {dtype}, got {t.dtype}")
        if contiguous and not t.is_contiguous():
            raise ops.KernelError(f"{name} must be contiguous")
        return t

    ops.calls = []
    monkeypatch.setattr(ops, "_cuda", named)
    monkeypatch.setattr(ops, "_call", lambda name, *args: ops.calls.append((name, args)))
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    yield ops
    del ops.calls


def _projection(M, H, dh, K, dtype):
    N = 3 * H * dh
    pages = torch.zeros(-(-M // 16), H, 16, dh, dtype=dtype)
    return dict(x=torch.zeros(M, K, dtype=dtype), weight=torch.zeros(N, K, dtype=dtype), bias=torch.zeros(N),
                q_out=torch.zeros(M, H * dh, dtype=dtype), k_pages=pages, v_pages=pages.clone(),
                slot_mapping=torch.arange(M, dtype=torch.int32), ws=None)


# rows of every kernel behind the entry: weight-streaming, tensor cores in pieces, cluster slices, the product and the copy
@pytest.mark.parametrize("M,dh,dtype", [(8, 32, torch.float32), (100, 32, torch.float32), (100, 24, torch.float32),
                                        (300, 32, torch.bfloat16), (100, 24, torch.bfloat16),
                                        (24, 24, torch.bfloat16)])
@pytest.mark.parametrize("what", ["short bias", "long rows of x", "weight in columns"])
def test_cache_writing_projection_refuses_what_does_not_fit(ops, M, dh, dtype, what):
    a = _projection(M, 4, dh, 768, dtype)
    if what == "short bias":
        a["bias"] = a["bias"][:-1]
    elif what == "long rows of x":
        a["x"] = torch.zeros(M, 776, dtype=dtype)
    else:
        a["weight"] = torch.zeros(768, a["weight"].shape[0], dtype=dtype).t()
    from mini_llm_b200.engine.context import Workspace
    a["ws"] = Workspace(torch.device("cpu"), 512)
    with pytest.raises(ops.KernelError):
        ops.linear_qkv_cache(**a)
    assert not ops.calls


def test_slices_of_a_product_are_summed_in_the_callers_own_scratch(ops, monkeypatch):
    """The float32 product in K slices: every workspace brings its own buffer (two runners on two streams may be between
    the product and the sum of its slices at the same time), the same one for every call; without a workspace a call
    allocates for itself."""
    from types import SimpleNamespace
    from mini_llm_b200.engine.context import Workspace
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: SimpleNamespace(cuda_stream=0))
    monkeypatch.setattr(torch.cuda, "stream", lambda s: __import__("contextlib").nullcontext())
    x, w = torch.zeros(100, 768), torch.zeros(768, 768)
    assert ops.library().mllm_linear_split_f32_slices(768, 768) > 1

    def scratch(ws, rows=100):
        with ops.stream_scope(ws):
            ops.linear(x[:rows], w, None, out=torch.zeros(rows, 768))
        name, args = ops.calls[-1]
        assert name == "mllm_linear_split_f32"
        pointer, floats = args[-3:-1]
        assert floats >= 3 * 128 * 768
        return pointer

    a, b = Workspace(torch.device("cpu"), 128), Workspace(torch.device("cpu"), 128)
    assert scratch(a) == scratch(a, 70) != scratch(b) == scratch(b)
    assert scratch(None) not in (scratch(a), scratch(b))
    version = a.version
    x = torch.zeros(1000, 768)
    assert scratch(a, 1000) and a.version > version          # a larger buffer is seen by whoever keeps its address


def test_sizes_that_go_to_the_cluster_kernel(ops, monkeypatch):
    """bfloat16 products of few rows: narrow results of long rows are cut over a cluster, at every count of rows, and wide ones
    are not, whose sums would cost more to exchange than the idle SMs do."""
    monkeypatch.setattr(ops, "sm_count", lambda: 148)
    for M, N, K in ((128, 768, 3072), (65, 1600, 6400), (64, 1024, 1024), (33, 1024, 4096), (24, 4800, 1600), (24, 1600, 6400),
                    (8, 1600, 6400), (3, 50257, 768), (16, 50257, 768)):
        assert ops._cluster_wins(M, N, K), (M, N, K)
    for M, N, K in ((65, 6144, 2048), (128, 2048, 2048), (96, 8192, 2048), (128, 11008, 4096), (48, 11008, 4096), (64, 6144, 2048),
                    (24, 2048, 1024), (24, 11008, 4096), (64, 768, 768), (17, 50257, 768), (129, 768, 3072), (64, 768, 448)):
        assert not ops._cluster_wins(M, N, K), (M, N, K)


def _pieces(x, rounded):
    """The cut of csrc/split_f32.cuh: to nearest, or (what it must not do) by dropping the lower bits."""
    import numpy as np

    def bf16(v):
        u = v.view(np.uint32)
        if rounded:
            u = (u.astype(np.uint64) + 0x7fff + ((u >> 16) & 1)).astype(np.uint32)
        return (u & np.uint32(0xffff0000)).view(np.float32)

    h = bf16(x)
    m = bf16(x - h)
    low = x - h - m
    assert np.array_equal(bf16(low), low)
    return [p.astype(np.float64) for p in (h, m, low)]


def test_dropped_products_of_pieces():
    """Of the nine products of pieces six are formed.  Cut to nearest, all pieces are exact, the three dropped products are
    below 2^-24 of the whole and have either sign; with bits dropped they reach 2^-21 and never change sign."""
    import numpy as np
    rng = np.random.default_rng(1)
    for lo, hi in ((0x3f800000, 0x40000000), (0x3f80f000, 0x3f810000)):
        x, y = (rng.integers(lo, hi, 1 << 20).astype(np.uint32).view(np.float32) for _ in range(2))
        lost = {}
        for rounded in (True, False):
            a, b = _pieces(x, rounded), _pieces(y, rounded)
            assert np.array_equal(a[0] + a[1] + a[2], x.astype(np.float64))
            lost[rounded] = (a[1] * b[2] + a[2] * b[1] + a[2] * b[2]) / (x.astype(np.float64) * y)
        assert np.abs(lost[True]).max() < 2 ** -24 and abs(lost[True].mean()) < 2 ** -34
        assert lost[False].min() >= 0 and lost[False].mean() > 2 ** -25
