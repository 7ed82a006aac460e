"""Each CUDA kernel alone against its plain float64 reference, at sizes other than the engine's."""
import math

import pytest
import torch

from helpers import TOL, batch_index, paged_cache, rel_error
from plain import ops_plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from aegean_tge_b200 import ops as module
    module.core()
    return module


# ---------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab,hidden,tokens", [(97, 72, 13), (331, 200, 1)])
def test_embedding(ops, dtype, vocab, hidden, tokens):
    gen = torch.Generator().manual_seed(1)
    table = torch.randn(vocab, hidden, generator=gen).to(dtype)
    ids = torch.randint(0, vocab, (tokens,), generator=gen, dtype=torch.int32)
    out = ops.embedding(table.to(DEV), ids.to(DEV))
    assert out.dtype == torch.float32
    assert torch.equal(out.cpu(), table[ids.long()].float())
    ops.check_status()


def test_embedding_bad_token_is_reported_not_read(ops):
    table = torch.randn(10, 8).to(DEV)
    out = ops.embedding(table, torch.tensor([3, 10, -1], dtype=torch.int32, device=DEV))
    assert torch.equal(out[1:].cpu(), torch.zeros(2, 8))
    with pytest.raises(ops.DeviceStatusError):
        ops.check_status()
    ops.check_status()      # the word was cleared


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,hidden,eps", [(5, 72, 1e-6), (3, 200, 1e-5), (2, 3000, 3e-6), (1, 5120, 1e-6),
                                             (3, 70, 1e-6), (2, 9004, 1e-6), (300, 3584, 1e-6)])
def test_rmsnorm(ops, out_dtype, rows, hidden, eps):
    gen = torch.Generator().manual_seed(2)
    x = torch.randn(rows, hidden, generator=gen) * 3.0
    w = 1.0 + (torch.rand(hidden, generator=gen) * 0.2 - 0.1)
    out = ops.rmsnorm(x.to(DEV), w.to(DEV), eps, out_dtype)
    assert rel_error(out, ops_plain.rmsnorm(x, w, eps)) < TOL[out_dtype]
    picked = torch.tensor([rows - 1, 0], dtype=torch.int32)
    out = ops.rmsnorm(x.to(DEV), w.to(DEV), eps, out_dtype, rows=picked.to(DEV))
    assert rel_error(out, ops_plain.rmsnorm(x[picked.long()], w, eps)) < TOL[out_dtype]
    ops.check_status()


def test_rmsnorm_eps_matters(ops):
    """Tiny inputs make eps dominate: a wrong or ignored eps shows at once."""
    x = torch.full((1, 64), 1e-4)
    w = torch.ones(64)
    for eps in (1e-6, 1e-5):
        out = ops.rmsnorm(x.to(DEV), w.to(DEV), eps, torch.float32)
        assert rel_error(out, ops_plain.rmsnorm(x, w, eps)) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_add_to_stream(ops, dtype):
    gen = torch.Generator().manual_seed(3)
    x = torch.randn(7, 130, generator=gen)
    y = torch.randn(7, 130, generator=gen).to(dtype)
    dx = x.to(DEV)
    ops.add_to_stream(dx, y.to(DEV))
    assert torch.equal(dx.cpu(), x + y.float())


# ---------------------------------------------------------------------------
# products
# ---------------------------------------------------------------------------
SIMT_SHAPES = [(1, 64, 64), (7, 130, 72), (33, 200, 176), (65, 97, 50), (128, 256, 255)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K", SIMT_SHAPES)
def test_gemm_simt_epilogues(ops, dtype, M, N, K):
    gen = torch.Generator().manual_seed(M * 1000 + N)
    x = torch.randn(M, K, generator=gen).to(dtype)
    w = (torch.randn(N, K, generator=gen) * 0.1).to(dtype)
    b = torch.randn(N, generator=gen)
    ref = ops_plain.linear(x, w, b)
    out = ops.linear(x.to(DEV), w.to(DEV), b.to(DEV), ops.GEMM_STORE, force_simt=True)
    assert out.dtype == dtype and rel_error(out, ref) < TOL[dtype]
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_STORE_F32, force_simt=True)
    assert out.dtype == torch.float32 and rel_error(out, ops_plain.linear(x, w, None)) < 2e-5
    stream = torch.randn(M, N, generator=gen)
    d = stream.to(DEV)
    ops.linear(x.to(DEV), w.to(DEV), b.to(DEV), ops.GEMM_ADD_F32, out=d, force_simt=True)
    assert rel_error(d, stream.double() + ref) < 2e-5
    if N % 2 == 0:
        out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_SWIGLU, force_simt=True)
        assert out.shape == (M, N // 2) and rel_error(out, ops_plain.swiglu_interleaved(x, w)) < TOL[dtype]


def test_gemm_simt_value_does_not_depend_on_the_batch(ops):
    """A row's float32 product is bit-identical alone and inside a larger batch."""
    gen = torch.Generator().manual_seed(5)
    x = torch.randn(70, 200, generator=gen).to(DEV)
    w = torch.randn(150, 200, generator=gen).to(DEV)
    whole = ops.linear(x, w, None, ops.GEMM_STORE_F32, force_simt=True)
    for row in (0, 33, 69):
        alone = ops.linear(x[row:row + 1], w, None, ops.GEMM_STORE_F32, force_simt=True)
        assert torch.equal(alone[0], whole[row])


@pytest.mark.parametrize("N,K", [(33, 4), (31, 64), (130, 68), (96, 256), (64, 700)])
def test_gemm_float32_few_tokens_have_the_bits_of_many(ops, N, K):
    """The kernel for few float32 tokens against the one for many, whose small tiles no longer fit the chip: the same
    chain of FMAs per element, at the edges of its 16 x 32 tiles and k-blocks of 64, in every epilogue."""
    gen = torch.Generator().manual_seed(N + K)
    many = 600 * 16 + 1
    x, w, b = torch.randn(many, K, generator=gen).to(DEV), torch.randn(N, K, generator=gen).to(DEV), torch.randn(N, generator=gen).to(DEV)
    for epilogue in (ops.GEMM_STORE, ops.GEMM_STORE_F32, ops.GEMM_ADD_F32, ops.GEMM_GELU, ops.GEMM_GELU_TANH) + (
            (ops.GEMM_SWIGLU, ops.GEMM_GLU_CLAMPED) if N % 2 == 0 else ()):
        def run(rows):
            out = torch.ones(rows.shape[0], N, device=DEV) if epilogue == ops.GEMM_ADD_F32 else None
            return ops.linear(rows, w, b, epilogue, out=out, force_simt=True, alpha=0.75, act_from=7)
        whole = run(x)
        for first, count in ((0, 1), (17, 16), (100, 19), (many - 64, 64)):
            assert torch.equal(run(x[first:first + count]), whole[first:first + count]), (epilogue, first, count)


@pytest.mark.parametrize("M,N,K", [(1, 512, 512), (8, 1000, 516), (16, 512, 3584), (17, 4608, 1536), (33, 640, 700), (65, 520, 640),
                                   (129, 3584, 512), (300, 514, 4100), (513, 2048, 516)])
def test_gemm_float32_on_the_tensor_cores(ops, M, N, K):
    """Every token tile and ragged edge, products cut along k and whole, panels of tokens; epilogues; a row alone to the same
    bits; an error against float64 no larger than that of one FMA chain along k."""
    gen = torch.Generator().manual_seed(M + N + K)
    x, w, b = (torch.randn(M, K, generator=gen).to(DEV), (torch.randn(N, K, generator=gen) * 0.1).to(DEV),
               torch.randn(N, generator=gen).to(DEV))
    assert ops.core().tge_gemm_f32_tcgen05_scratch_floats(w.data_ptr(), K, M, N, K) > 0
    ref = x.double() @ w.double().T
    out = ops.linear(x, w, None, ops.GEMM_STORE_F32)
    chain = ops.linear(x, w, None, ops.GEMM_STORE_F32, force_simt=True)
    rms = lambda t: float((t.double() - ref).norm() / ref.norm())
    assert rms(out) <= rms(chain)
    for row in (0, M // 2, M - 1):
        assert torch.equal(ops.linear(x[row:row + 1], w, None, ops.GEMM_STORE_F32)[0], out[row])
    # bounds: a sum's error here is below 4e-7 of its root mean square, the largest of a million five times that
    stream = torch.randn(M, N, generator=gen).to(DEV)
    added = stream.clone()
    ops.linear(x, w, b, ops.GEMM_ADD_F32, out=added, alpha=0.5)
    assert rel_error(added, stream.double() + 0.5 * (ref + b.double())) < 2e-6
    wide = torch.zeros(M, N + 3, device=DEV)
    ops.linear(x, w, b, ops.GEMM_GELU, out=wide[:, :N], act_from=100)
    full = ref + b.double()
    act = torch.cat([full[:, :100], torch.nn.functional.gelu(full[:, 100:])], dim=1)
    assert rel_error(wide[:, :N], act) < 2e-6 and float(wide[:, N:].abs().max()) == 0
    g, u = full[:, 0::2], full[:, 1::2]
    assert rel_error(ops.linear(x, w, b, ops.GEMM_SWIGLU), torch.nn.functional.silu(g) * u) < 5e-6    # two sums' errors
    ops.check_status()


def test_gemm_float32_on_the_tensor_cores_keeps_what_is_not_finite(ops):
    gen = torch.Generator().manual_seed(1)
    x, w = torch.randn(20, 600, generator=gen).to(DEV), torch.randn(700, 600, generator=gen).to(DEV)
    x[3, 5], x[4, 599], w[8, 6], w[9, 0] = math.inf, -math.inf, math.nan, 3.4e38
    x[5] = 2e38                                    # parts and sums beyond the range
    for epilogue in (ops.GEMM_STORE_F32, ops.GEMM_SWIGLU):
        out, chain = (ops.linear(x, w, None, epilogue, force_simt=simt) for simt in (False, True))
        odd = ~torch.isfinite(chain)
        assert odd.any() and torch.equal(torch.isfinite(out), ~odd)
        assert torch.equal(torch.nan_to_num(out[odd], nan=7.0), torch.nan_to_num(chain[odd], nan=7.0))
    # tiny numbers keep what a sum of three parts holds of them
    out = ops.linear(x[6:9] * 1e-30, w[10:], None, ops.GEMM_STORE_F32)
    assert rel_error(out * 1e30, x[6:9].double() @ w[10:].double().T) < 1e-6


@pytest.mark.parametrize("N,K,M", [(640, 1024, 8), (2304, 512, 600), (96, 256, 4)])
def test_gemm_float32_weights_and_bias_may_be_the_last_kernels_result(ops, N, K, M):
    """Weights and bias that the kernels just before have written (here by products themselves, long ones, into memory that held
    others) are read after they are there, on the tensor cores (cut along k and whole) and by the kernel for few tokens."""
    gen = torch.Generator().manual_seed(N)
    x = torch.randn(M, K, generator=gen).to(DEV)
    a, b = torch.randn(12, N, 900, generator=gen).to(DEV), torch.randn(K, 900, generator=gen).to(DEV)
    ones = torch.randn(12, N, 3000, generator=gen).to(DEV)
    w, bias = torch.zeros(N, K, device=DEV), torch.zeros(N, device=DEV)
    got, want = [], []
    for i in range(12):
        ops.linear(a[i], b, None, ops.GEMM_STORE_F32, out=w)
        ops.linear(ones[i, :1], ones[i], None, ops.GEMM_STORE_F32, out=bias.view(1, N))
        got.append(ops.linear(x, w, bias, ops.GEMM_STORE_F32))
    for i in range(12):
        ops.linear(a[i], b, None, ops.GEMM_STORE_F32, out=w)
        torch.cuda.synchronize()
        got.append(ops.linear(x, w, None, ops.GEMM_STORE_F32))          # ... the weights alone
        ops.linear(a[i], b, None, ops.GEMM_STORE_F32, out=w)
        want.append(ops.linear(x, w, None, ops.GEMM_STORE_F32))
        ops.linear(ones[i, :1], ones[i], None, ops.GEMM_STORE_F32, out=bias.view(1, N))
        torch.cuda.synchronize()
        assert torch.equal(got[i], ops.linear(x, w, bias, ops.GEMM_STORE_F32))
    assert all(torch.equal(g, h) for g, h in zip(got[12:], want))
    ops.check_status()


@pytest.mark.parametrize("N,K", [(700, 600), (4736, 2048)])
def test_gemm_float32_on_the_tensor_cores_keeps_tiny_numbers(ops, N, K):
    """Rows around and below 1e-33, where three bfloat16 parts no longer hold a float32 number: no more error than one FMA chain's
    (cut along k and whole), and the rows beside them as they are without them.  Zeros stay zeros."""
    gen = torch.Generator().manual_seed(N)
    x, w = torch.randn(12, K, generator=gen).to(DEV), torch.randn(N, K, generator=gen).to(DEV)
    plain = ops.linear(x, w, None, ops.GEMM_STORE_F32)
    for row, scale in ((1, 1e-28), (3, 1e-31), (5, 1e-33), (7, 1e-35), (9, 3e-38), (11, 0.0)):
        x[row] *= scale
    out, chain = (ops.linear(x, w, None, ops.GEMM_STORE_F32, force_simt=simt) for simt in (False, True))
    ref = x.double() @ w.double().T
    assert torch.equal(out[0::2], plain[0::2]) and not out[11].any()
    for row in (1, 3, 5, 7, 9):
        error = lambda got: float((got[row].double() - ref[row]).norm() / ref[row].norm())
        assert error(out) <= 1.05 * error(chain), row
    ops.check_status()


def test_float32_calls_on_two_streams_share_no_memory(ops, monkeypatch):
    """Products and attention in float32 keep what passes between their launches in memory of the call: nothing comes out of the
    device's scratch buffer, and calls on two streams at once have the results they have alone."""
    gen = torch.Generator().manual_seed(2)
    w = torch.randn(640, 2048, generator=gen).to(DEV)
    lengths, heads, kv_heads = [700, 900], 7, 1
    k_pages, v_pages, table, _k, _v = paged_cache(lengths, kv_heads, 128, 16, torch.float32, DEV, seed=8)
    positions, seq_of_token, q_start, start_pos = batch_index([1, 1], [n - 1 for n in lengths], DEV)
    assert ops.core().tge_attention_f32_scratch_floats(2, 2, 1, 900, heads, kv_heads, 128) > 0

    def calls(x, q):
        return (ops.linear(x, w, None, ops.GEMM_STORE_F32), ops.attention(q, k_pages, v_pages, table, q_start, start_pos, positions, seq_of_token,
                                                                          2, 1, 900, heads, kv_heads, 128, 0.1))
    inputs = [(torch.randn(300, 2048, generator=gen).to(DEV), torch.randn(2, heads * 128, generator=gen).to(DEV)) for _ in range(2)]
    monkeypatch.setattr(ops, "_scratch", {})
    alone = [calls(*pair) for pair in inputs]
    assert not ops._scratch
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in inputs]
    together = [[], []]
    for _ in range(20):
        for i, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                together[i].append(calls(*inputs[i]))
    torch.cuda.synchronize()
    for i in range(2):
        for product, attended in together[i]:
            assert torch.equal(product, alone[i][0]) and torch.equal(attended, alone[i][1])
    ops.check_status()


def test_gemm_float32_without_room_for_scratch_is_one_chain(ops, monkeypatch):
    """Where the device has no room for the call's memory the product runs as the FMA chain, as it always did.  A captured
    product finds it in the graph's pool."""
    gen = torch.Generator().manual_seed(2)
    x, w = torch.randn(5, 600, generator=gen).to(DEV), torch.randn(640, 600, generator=gen).to(DEV)
    chain = ops.linear(x, w, None, ops.GEMM_STORE_F32, force_simt=True)
    roomy = ops.linear(x, w, None, ops.GEMM_STORE_F32)
    out = torch.zeros(5, 640, device=DEV)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ops.linear(x, w, None, ops.GEMM_STORE_F32, out=out)
    graph.replay()
    assert torch.equal(out, roomy) and not torch.equal(out, chain)
    monkeypatch.setattr(ops, "call_floats", lambda count: None)
    assert torch.equal(ops.linear(x, w, None, ops.GEMM_STORE_F32), chain)


def test_attention_float32_without_room_for_scratch_has_the_same_bits(ops, monkeypatch):
    case = lambda: _attention_case(ops, torch.float32, 7, 1, 128, [1, 1, 3], [1000, 63, 254])[1]
    roomy = case()
    monkeypatch.setattr(ops, "call_floats", lambda count: None)
    assert torch.equal(case(), roomy)


def test_scratch_memory_that_cannot_grow_stays_as_it_was(ops, monkeypatch):
    """A buffer too large for the device raises, time and again, without filing the one in use among the outgrown."""
    def no_room(*_args, **_kw):
        raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(ops, "_scratch", {})
    monkeypatch.setattr(ops, "_outgrown", {})
    held = ops.scratch_floats(10)
    with monkeypatch.context() as patch:
        patch.setattr(torch, "empty", no_room)
        for _ in range(3):
            with pytest.raises(torch.OutOfMemoryError):
                ops.scratch_floats(held.numel() + 1)
        assert ops.scratch_floats(held.numel()) is held and not ops._outgrown
    grown = ops.scratch_floats(held.numel() + 1)
    assert grown.numel() >= 2 * held.numel() and [t is held for kept in ops._outgrown.values() for t in kept] == [True]


TC_SHAPES = [(1, 128, 64), (8, 384, 176), (16, 200, 256), (33, 130, 72), (64, 512, 1024), (100, 300, 512),
             (200, 640, 320), (300, 1024, 512), (520, 256, 192)]


@pytest.mark.parametrize("M,N,K", TC_SHAPES)
def test_gemm_tcgen05_exact_on_small_integers(ops, M, N, K):
    """Integer-valued operands make every product and sum exact in float32, so any misplaced
    row, column, k-block or swizzle shows as an outright mismatch."""
    gen = torch.Generator().manual_seed(M + N + K)
    x = torch.randint(-2, 3, (M, K), generator=gen).to(torch.bfloat16)
    w = torch.randint(-3, 4, (N, K), generator=gen).to(torch.bfloat16)
    ref = (x.double() @ w.double().T).float()
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_STORE_F32)
    ops.check_status()
    assert torch.equal(out.cpu(), ref)


@pytest.mark.parametrize("M,N,K,bn,splits", [
    (5, 256, 512, 16, 1), (5, 256, 512, 16, 4), (40, 384, 1024, 64, 3), (130, 200, 576, 128, 2),
    (260, 512, 256, 256, 1), (260, 512, 1024, 256, 2), (70, 130, 176, 32, 1), (24, 3584, 512, 32, 1),
    (500, 384, 640, 208, 1), (300, 256, 320, 144, 2), (100, 200, 256, 48, 1), (470, 130, 192, 240, 1)])
def test_gemm_tcgen05_tiles_and_splits(ops, M, N, K, bn, splits):
    gen = torch.Generator().manual_seed(bn + splits + M)
    x = torch.randint(-2, 3, (M, K), generator=gen).to(torch.bfloat16)
    w = torch.randint(-3, 4, (N, K), generator=gen).to(torch.bfloat16)
    ref = (x.double() @ w.double().T).float()
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_STORE_F32, force_bn=bn, force_splits=splits)
    ops.check_status()
    assert torch.equal(out.cpu(), ref)


@pytest.mark.parametrize("M,N,K,splits", [(9, 260, 328, 1), (9, 260, 328, 3), (150, 384, 704, 1), (2048, 512, 256, 1),
                                          (2048, 3584, 128, 1), (1100, 640, 192, 1)])
def test_gemm_tcgen05_epilogues(ops, M, N, K, splits):
    gen = torch.Generator().manual_seed(7 * M + splits)
    x = torch.randn(M, K, generator=gen).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=gen) * 0.1).to(torch.bfloat16)
    b = torch.randn(N, generator=gen)
    ref = ops_plain.linear(x, w, b)
    kw = dict(force_splits=splits)
    out = ops.linear(x.to(DEV), w.to(DEV), b.to(DEV), ops.GEMM_STORE, **kw)
    assert out.dtype == torch.bfloat16 and rel_error(out, ref) < TOL[torch.bfloat16]
    out = ops.linear(x.to(DEV), w.to(DEV), b.to(DEV), ops.GEMM_STORE_F32, **kw)
    assert rel_error(out, ref) < 2e-5
    stream = torch.randn(M, N, generator=gen)
    d = stream.to(DEV)
    ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_ADD_F32, out=d, **kw)
    assert rel_error(d, stream.double() + ops_plain.linear(x, w, None)) < 2e-5
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_SWIGLU, **kw)
    assert out.shape == (M, N // 2) and rel_error(out, ops_plain.swiglu_interleaved(x, w)) < TOL[torch.bfloat16]
    ops.check_status()


@pytest.mark.parametrize("M,N,K,splits", [(1, 4, 512, 2), (3, 260, 512, 4), (7, 516, 704, 5), (193, 1024, 1024, 9)])
def test_gemm_tcgen05_sums_of_splits_by_quads_and_one_by_one(ops, M, N, K, splits):
    """The kernel that adds a product's cuts four columns at a time against the one that takes them singly (an output whose rows
    start on odd elements goes there), to the same bits in every epilogue."""
    gen = torch.Generator().manual_seed(N + splits)
    x, w = torch.randn(M, K, generator=gen).to(torch.bfloat16).to(DEV), (torch.randn(N, K, generator=gen) * 0.1).to(torch.bfloat16).to(DEV)
    b = torch.randn(N, generator=gen).to(DEV)
    for epilogue in (ops.GEMM_STORE, ops.GEMM_STORE_F32, ops.GEMM_ADD_F32, ops.GEMM_SWIGLU, ops.GEMM_GELU, ops.GEMM_GELU_TANH, ops.GEMM_GLU_CLAMPED):
        gated = epilogue in (ops.GEMM_SWIGLU, ops.GEMM_GLU_CLAMPED)
        dtype = torch.float32 if epilogue in (ops.GEMM_STORE_F32, ops.GEMM_ADD_F32) else torch.bfloat16
        columns = N // 2 if gated else N
        quads = torch.ones(M, columns, dtype=dtype, device=DEV)
        wide = torch.ones(M, columns + 5, dtype=dtype, device=DEV)
        for bias in (b, None):
            for out in (quads, wide[:, 3:3 + columns]):
                out.fill_(1.0)
                ops.linear(x, w, bias, epilogue, out=out, force_splits=splits, alpha=0.75, act_from=5)
            assert torch.equal(quads, wide[:, 3:3 + columns]), (epilogue, bias is None)
        assert bool((wide[:, :3] == 1).all()) and bool((wide[:, 3 + columns:] == 1).all())


@pytest.fixture
def pair_everywhere(ops):
    """Every bfloat16 product that the two-SM kernel can run goes to it, also shapes it would not be chosen for."""
    ops.set_pair_gemm(2)
    yield
    ops.set_pair_gemm(1)


@pytest.mark.parametrize("M,N,K", TC_SHAPES + [(2048, 768, 192), (257, 130, 136), (140, 3584, 64), (1000, 520, 1032)])
def test_gemm_pair_exact_on_small_integers(ops, pair_everywhere, M, N, K):
    """The kernel that pairs two SMs on a tile of 256 weight rows: rows of either block, token halves of
    either block, ragged edges in both directions, more k-blocks than stages."""
    gen = torch.Generator().manual_seed(M + N + K)
    x = torch.randint(-2, 3, (M, K), generator=gen).to(torch.bfloat16)
    w = torch.randint(-3, 4, (N, K), generator=gen).to(torch.bfloat16)
    ref = (x.double() @ w.double().T).float()
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_STORE_F32)
    ops.check_status()
    assert torch.equal(out.cpu(), ref)


@pytest.mark.parametrize("M,N,K", [(9, 260, 328), (150, 384, 704), (2048, 512, 256), (1100, 640, 192)])
def test_gemm_pair_epilogues(ops, pair_everywhere, M, N, K):
    gen = torch.Generator().manual_seed(7 * M)
    x = torch.randn(M, K, generator=gen).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=gen) * 0.1).to(torch.bfloat16)
    b = torch.randn(N, generator=gen)
    ref = ops_plain.linear(x, w, b)
    out = ops.linear(x.to(DEV), w.to(DEV), b.to(DEV), ops.GEMM_STORE)
    assert out.dtype == torch.bfloat16 and rel_error(out, ref) < TOL[torch.bfloat16]
    out = ops.linear(x.to(DEV), w.to(DEV), b.to(DEV), ops.GEMM_STORE_F32)
    assert rel_error(out, ref) < 2e-5
    stream = torch.randn(M, N, generator=gen)
    d = stream.to(DEV)
    ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_ADD_F32, out=d)
    assert rel_error(d, stream.double() + ops_plain.linear(x, w, None)) < 2e-5
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_SWIGLU)
    assert out.shape == (M, N // 2) and rel_error(out, ops_plain.swiglu_interleaved(x, w)) < TOL[torch.bfloat16]
    ops.check_status()


@pytest.mark.parametrize("pair", [0, 2])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (15, 260, 128), (17, 132, 64), (145, 130, 192), (193, 388, 320), (257, 131, 64), (500, 640, 128)])
def test_gemm_tcgen05_stores_of_any_width_hold_the_same(ops, pair, M, N, K):
    """Outputs whose rows allow 8-byte stores, 4-byte stores or single ones only, over tokens and weight rows that end inside a tile: the
    same bits in every epilogue, and nothing beside them touched."""
    gen = torch.Generator().manual_seed(N + M)
    x, w = torch.randn(M, K, generator=gen).to(torch.bfloat16).to(DEV), (torch.randn(N, K, generator=gen) * 0.1).to(torch.bfloat16).to(DEV)
    b = torch.randn(N, generator=gen).to(DEV)
    plain_rows = ops_plain.linear(x.cpu(), w.cpu(), b.cpu())
    ops.set_pair_gemm(pair)
    try:
        for epilogue in (ops.GEMM_STORE, ops.GEMM_STORE_F32, ops.GEMM_ADD_F32, ops.GEMM_SWIGLU, ops.GEMM_GELU, ops.GEMM_GELU_TANH, ops.GEMM_GLU_CLAMPED):
            gated = epilogue in (ops.GEMM_SWIGLU, ops.GEMM_GLU_CLAMPED)
            if gated and N % 2:
                continue
            dtype = torch.float32 if epilogue in (ops.GEMM_STORE_F32, ops.GEMM_ADD_F32) else torch.bfloat16
            columns, results = N // 2 if gated else N, []
            for before, width in ((0, -(-columns // 8) * 8), (4, -(-columns // 8) * 8 + 8), (2, -(-columns // 2) * 2 + 4), (3, columns + 5)):
                out = torch.ones(M, width, dtype=dtype, device=DEV)
                view = out[:, before:before + columns]
                ops.linear(x, w, b, epilogue, out=view, alpha=0.75, act_from=5)
                results.append(view.clone())
                assert bool((out[:, :before] == 1).all()) and bool((out[:, before + columns:] == 1).all())
            ops.check_status()
            assert all(torch.equal(results[0], other) for other in results[1:]), epilogue
            if epilogue == ops.GEMM_STORE:
                assert rel_error(results[0], 0.75 * plain_rows) < TOL[torch.bfloat16]
            if epilogue == ops.GEMM_ADD_F32:
                assert rel_error(results[0], 1.0 + 0.75 * plain_rows) < 2e-5
    finally:
        ops.set_pair_gemm(1)


@pytest.mark.parametrize("pair,M", [(0, 3), (2, 150)])
def test_gated_epilogue_over_the_whole_range_of_gates(ops, pair, M):
    """g / (1 + exp(-g)) u where the product is zero and the bias holds g and u: gates from -1e4 to 1e4, where exp(-g) overflows and where a
    quotient's divisor does, infinities and NaN.  2^-8: the rounding to bfloat16; 89 * 3 / 2^126, the largest |g u| over the smallest such
    divisor: CUDA's fast division gives zero for divisors above 2^126, which |g| <= 89 reaches."""
    edges = [0.0, -0.0, 1e-30, -1e-30, -87.0, -87.5, -88.0, -88.5, -88.8, -89.0, -103.0, -1e4, 88.0, 1e4, 3e38, -3e38, float("inf"), float("-inf"),
             float("nan")]
    gates = torch.cat([torch.tensor(edges), torch.linspace(-110.0, 110.0, 4001), torch.linspace(-4.0, 4.0, 1000)])
    gates = torch.cat([gates, torch.zeros(-gates.numel() % 64)])
    up = torch.where(torch.arange(gates.numel()) % 2 == 0, 1.0, -3.0)
    bias = torch.stack([gates, up], 1).reshape(-1).to(DEV)
    x = torch.zeros(M, 64, dtype=torch.bfloat16, device=DEV)
    w = torch.randn(bias.numel(), 64, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).to(DEV)
    ops.set_pair_gemm(pair)
    try:
        got = ops.linear(x, w, bias, ops.GEMM_SWIGLU).double().cpu()
    finally:
        ops.set_pair_gemm(1)
    ops.check_status()
    exact = (gates.double() / (1.0 + torch.exp(-gates.double())) * up.double())[None].expand(M, -1)
    special = ~torch.isfinite(exact) | (exact.abs() > 3e38)
    assert torch.equal(torch.isnan(got), torch.isnan(exact))
    off = ((got - exact).abs() > 2.0 ** -8 * exact.abs() + 89 * 3 * 2.0 ** -126) & ~special
    assert not bool(off.any()), gates[off[0]].tolist()
    infinite = torch.isinf(exact)
    assert torch.equal(got[infinite], exact[infinite])


@pytest.mark.parametrize("M,N,K", [(150, 256, 64), (193, 3584, 704), (300, 4608, 512), (2048, 768, 1024)])
def test_gemm_pair_settled_weights_change_no_bit(ops, pair_everywhere, M, N, K):
    """Weights asked for ahead of the kernel in front (fewer k-blocks than stages, cuts along k, several tiles to a pair), each product
    reading what the one before it has written."""
    gen = torch.Generator().manual_seed(N)
    x, w = torch.randn(M, K, generator=gen).to(torch.bfloat16).to(DEV), (torch.randn(N, K, generator=gen) * 0.1).to(torch.bfloat16).to(DEV)
    back = (torch.randn(K, N, generator=gen) * 0.05).to(torch.bfloat16).to(DEV)
    results = []
    for settled in (False, True):
        rows = x
        for _ in range(6):
            rows = ops.linear(ops.linear(rows, w, None, ops.GEMM_STORE, settled=settled), back, None, ops.GEMM_STORE, settled=settled)
        results.append(rows)
    ops.check_status()
    assert torch.equal(results[0], results[1]) and bool(torch.isfinite(results[0]).all())


@pytest.mark.parametrize("pair", [0, 2])
@pytest.mark.parametrize("M", [4, 100, 200])
def test_products_wait_for_weights_that_the_kernel_in_front_has_just_written(ops, pair, M):
    """Weights and biases that come out of the kernel right in front, other ones in every turn: without ``settled`` a product on one SM or on
    pairs, the kernel that adds its cuts, and the fused forms see them.  Expected: the same calls, everything waited for."""
    gen = torch.Generator().manual_seed(M)
    N, K, turns = 1536, 2048, 4
    seeds = [(torch.randn(N, 256, generator=gen) * 0.1).to(torch.bfloat16).to(DEV) for _ in range(turns)]
    basis = (torch.randn(K, 256, generator=gen) * 0.1).to(torch.bfloat16).to(DEV)
    row = [torch.randn(1, 512, generator=gen).to(torch.bfloat16).to(DEV) for _ in range(turns)]
    maker = (torch.randn(N, 512, generator=gen) * 0.1).to(torch.bfloat16).to(DEV)
    x = torch.randn(M, K, generator=gen).to(torch.bfloat16).to(DEV)
    w, bias = torch.zeros(N, K, dtype=torch.bfloat16, device=DEV), torch.zeros(1, N, device=DEV)
    norm = 1.0 + 0.1 * torch.randn(N, generator=gen).to(DEV)

    def turn(i, between):
        results, stream = [], torch.ones(M, N, device=DEV)
        ops.linear(row[i], maker, None, ops.GEMM_STORE_F32, out=bias)
        between()
        ops.linear(seeds[i], basis, None, ops.GEMM_STORE, out=w)
        between()
        results.append(ops.linear(x, w, bias[0], ops.GEMM_STORE_F32, force_splits=3))
        between()
        ops.linear(seeds[i - 1], basis, None, ops.GEMM_STORE, out=w)
        between()
        results.append(ops.linear(x, w, None, ops.GEMM_STORE))
        between()
        ops.linear(seeds[i], basis, None, ops.GEMM_STORE, out=w)
        ops.linear(row[i - 1], maker, None, ops.GEMM_STORE_F32, out=bias)
        between()
        results.append(ops.linear(x, w, bias[0], ops.GEMM_STORE_F32))
        between()
        ops.linear(seeds[i - 1], basis, None, ops.GEMM_STORE, out=w)
        between()
        results += [ops.linear_add_norm(x, w, bias[0], stream, norm, 1e-5, torch.bfloat16), stream]
        between()
        return results

    ops.set_pair_gemm(pair)
    try:
        wanted = [turn(i, torch.cuda.synchronize) for i in range(turns)]
        for _ in range(6):
            got = [turn(i, lambda: None) for i in range(turns)]
            for i in range(turns):
                assert all(torch.equal(a, b) for a, b in zip(got[i], wanted[i])), i
        ops.check_status()
    finally:
        ops.set_pair_gemm(1)
    assert rel_error(wanted[0][0], ops_plain.linear(x.cpu(), ops_plain.linear(seeds[0].cpu(), basis.cpu(), None).to(torch.bfloat16),
                                                    ops_plain.linear(row[0].cpu(), maker.cpu(), None)[0])) < TOL[torch.bfloat16]


@pytest.mark.parametrize("M,N,K", [(1, 256, 128), (8, 3584, 512), (33, 520, 264), (128, 1024, 320), (140, 384, 192), (150, 384, 192)])
@pytest.mark.parametrize("defer", [False, True])
def test_linear_add_norm_and_rows_without_their_factor(ops, M, N, K, defer):
    """stream += x . w^T; the next product's input = RMSNorm(stream) * weight, either complete or (up to 128
    rows, if asked) without the norm's factor, which the product that takes the rows then applies: with a bias,
    with the gated epilogue, cut along k or not, and completed on their own."""
    gen = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=gen).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=gen) * 0.1).to(torch.bfloat16)
    stream = torch.randn(M, N, generator=gen) * 3.0
    gain = 1.0 + 0.2 * torch.randn(N, generator=gen)
    eps = 1e-5
    new_stream = stream.double() + ops_plain.linear(x, w, None)
    normed = ops_plain.rmsnorm(new_stream, gain, eps)
    d_stream = stream.to(DEV)
    rows = ops.linear_add_norm(x.to(DEV), w.to(DEV), None, d_stream, gain.to(DEV), eps, torch.bfloat16, defer=defer)
    assert rel_error(d_stream, new_stream) < 2e-5
    assert isinstance(rows, ops.DeferredRows) == (defer and M <= 128)
    if isinstance(rows, ops.DeferredRows):
        assert rel_error(rows.complete(), normed) < 2 * TOL[torch.bfloat16]
    else:
        assert rel_error(rows, normed) < TOL[torch.bfloat16]
    # takers: a plain product with a bias (few weight rows and a long k: cut along k) and a gated one
    for rows_out, k_cut in ((40, True), (768, False)):
        w2 = (torch.randn(rows_out, N, generator=gen) * 0.05).to(torch.bfloat16)
        b2 = torch.randn(rows_out, generator=gen)
        want = ops_plain.linear(normed, w2, b2)
        got = ops.linear(rows, w2.to(DEV), b2.to(DEV), ops.GEMM_STORE_F32)
        assert rel_error(got, want) < TOL[torch.bfloat16], (rows_out, k_cut)
        got = ops.linear(rows, w2.to(DEV), None, ops.GEMM_SWIGLU)
        assert rel_error(got, ops_plain.swiglu_interleaved(normed, w2)) < 2 * TOL[torch.bfloat16]
    ops.check_status()


def test_gemm_tcgen05_refuses_what_tma_cannot_address(ops):
    """K that is no multiple of 8 cannot be a TMA row pitch: the product still comes out right (CUDA cores)."""
    gen = torch.Generator().manual_seed(11)
    x = torch.randn(5, 50, generator=gen).to(torch.bfloat16)
    w = torch.randn(24, 50, generator=gen).to(torch.bfloat16)
    out = ops.linear(x.to(DEV), w.to(DEV), None, ops.GEMM_STORE_F32)
    assert rel_error(out, ops_plain.linear(x, w, None)) < 2e-5


# ---------------------------------------------------------------------------
# rotation + cache store
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,head_dim,rotary", [(6, 2, 48, 48), (5, 1, 64, 32), (4, 4, 16, 16), (3, 1, 80, 0),
                                                          (2, 1, 20, 12), (28, 4, 128, 128), (3, 2, 36, 36)])
def test_rope_kv_store(ops, dtype, heads, kv_heads, head_dim, rotary):
    from aegean_tge_b200.parts.rope import rotary_tables
    page_size = 16
    q_lens, starts = [5, 1, 20], [30, 47, 0]          # portions crossing page edges at odd offsets
    positions, seq_of_token, _, _ = batch_index(q_lens, starts, DEV)
    T = sum(q_lens)
    width = (heads + 2 * kv_heads) * head_dim
    gen = torch.Generator().manual_seed(heads * 10 + head_dim)
    qkv = torch.randn(T, width, generator=gen).to(dtype)
    lengths = [s + n for s, n in zip(starts, q_lens)]
    k_pages, v_pages, table, _, _ = paged_cache(lengths, kv_heads, head_dim, page_size, dtype, DEV, seed=4)
    before_k = k_pages.clone()
    cos = sin = None
    if rotary:
        cos, sin = rotary_tables(12345.0, rotary, 64)
    dq = qkv.to(DEV)
    ops.rope_kv_store(dq, None if cos is None else cos.to(DEV), None if sin is None else sin.to(DEV), rotary,
                      positions, seq_of_token, table, k_pages, v_pages, heads, kv_heads, head_dim)
    ops.check_status()
    pos = positions.cpu().long()
    q = qkv[:, :heads * head_dim].view(T, heads, head_dim)
    k = qkv[:, heads * head_dim:(heads + kv_heads) * head_dim].view(T, kv_heads, head_dim)
    v = qkv[:, (heads + kv_heads) * head_dim:].view(T, kv_heads, head_dim)
    c = cos[pos] if rotary else None
    s = sin[pos] if rotary else None
    q_ref = ops_plain.rotate_half(q, c, s, rotary)
    k_ref = ops_plain.rotate_half(k, c, s, rotary)
    assert rel_error(dq[:, :heads * head_dim].reshape(T, heads, head_dim), q_ref) < TOL[dtype]
    touched = torch.zeros_like(before_k, dtype=torch.bool)
    for t in range(T):
        page = int(table[int(seq_of_token[t]), int(pos[t]) // page_size])
        slot = int(pos[t]) % page_size
        assert rel_error(k_pages[page, :, slot], k_ref[t]) < TOL[dtype]
        assert torch.equal(v_pages[page, :, slot].cpu(), v[t])
        touched[page, :, slot] = True
    assert torch.equal(k_pages[~touched], before_k[~touched]), "a slot outside the step's positions was written"


@pytest.mark.parametrize("heads,kv_heads,head_dim,rotary,hidden", [(7, 1, 128, 128, 512), (4, 2, 128, 0, 256), (6, 2, 64, 64, 384),
                                                                 (5, 1, 64, 32, 320)])
@pytest.mark.parametrize("q_lens,starts", [([1, 1, 1], [30, 47, 0]), ([5, 1, 20], [30, 47, 0]), ([70, 58], [3, 16]), ([80, 62], [3, 16]), ([90, 70], [3, 6])])
@pytest.mark.parametrize("deferred", [False, True])
def test_linear_qkv_rope_store(ops, heads, kv_heads, head_dim, rotary, hidden, q_lens, starts, deferred):
    """The q/k/v product fused with bias, rotation and the cache store, for small batches (one kernel adds the
    product's partial sums, rotates and stores) and larger ones (separate kernels), with rows that still lack
    their norm factor and with complete ones, at two head sizes, with a full, a partial and no rotation."""
    from aegean_tge_b200.parts.rope import rotary_tables
    page_size = 16
    positions, seq_of_token, _, _ = batch_index(q_lens, starts, DEV)
    T = sum(q_lens)
    width = (heads + 2 * kv_heads) * head_dim
    gen = torch.Generator().manual_seed(heads * 10 + head_dim + T)
    x = torch.randn(T, hidden, generator=gen).to(torch.bfloat16)
    w = (torch.randn(width, hidden, generator=gen) * 0.1).to(torch.bfloat16)
    bias = torch.randn(width, generator=gen)
    lengths = [s + n for s, n in zip(starts, q_lens)]
    cos = sin = None
    if rotary:
        cos, sin = rotary_tables(12345.0, rotary, 96)
    taken = x
    normed = x.double()
    if deferred and T <= 128:
        # rows = stream * gain in bfloat16 plus the sums of squares of the stream in slices: what linear_add_norm hands on
        stream = torch.randn(T, hidden, generator=gen) * 2.0
        gain = 1.0 + 0.2 * torch.randn(hidden, generator=gen)
        rows = (stream * gain).to(torch.bfloat16)
        slices = -(-hidden // 96)
        sums = torch.stack([(stream[:, i * 96:(i + 1) * 96].double() ** 2).sum(1) for i in range(slices)]).float()
        taken = ops.DeferredRows(rows.to(DEV), sums.to(DEV).contiguous(), hidden, 1e-5)
        normed = rows.double() / torch.sqrt((stream.double() ** 2).mean(1, keepdim=True) + 1e-5)
    qkv_ref = ops_plain.linear(normed, w, bias)
    pos = positions.cpu().long()
    q = qkv_ref[:, :heads * head_dim].view(T, heads, head_dim)
    k = qkv_ref[:, heads * head_dim:(heads + kv_heads) * head_dim].view(T, kv_heads, head_dim)
    v = qkv_ref[:, (heads + kv_heads) * head_dim:].view(T, kv_heads, head_dim)
    c = cos[pos] if rotary else None
    s = sin[pos] if rotary else None
    q_ref, k_ref = ops_plain.rotate_half(q, c, s, rotary), ops_plain.rotate_half(k, c, s, rotary)
    for _ in range(1):
        k_pages, v_pages, table, _, _ = paged_cache(lengths, kv_heads, head_dim, page_size, torch.bfloat16, DEV, seed=4)
        before_k = k_pages.clone()
        out = ops.linear_qkv_rope_store(taken if not isinstance(taken, torch.Tensor) else taken.to(DEV), w.to(DEV),
                                        bias.to(DEV), None if cos is None else cos.to(DEV),
                                        None if sin is None else sin.to(DEV), rotary, positions, seq_of_token, table,
                                        k_pages, v_pages, heads, kv_heads, head_dim)
        ops.check_status()
        assert rel_error(out[:, :heads * head_dim].reshape(T, heads, head_dim), q_ref) < TOL[torch.bfloat16]
        touched = torch.zeros_like(before_k, dtype=torch.bool)
        for t in range(T):
            page = int(table[int(seq_of_token[t]), int(pos[t]) // page_size])
            slot = int(pos[t]) % page_size
            assert rel_error(k_pages[page, :, slot], k_ref[t]) < TOL[torch.bfloat16]
            assert rel_error(v_pages[page, :, slot], v[t]) < TOL[torch.bfloat16]
            touched[page, :, slot] = True
        assert torch.equal(k_pages[~touched], before_k[~touched]), "a slot outside the step's positions was written"


# ---------------------------------------------------------------------------
# attention
# ---------------------------------------------------------------------------
def _attention_case(ops, dtype, heads, kv_heads, head_dim, q_lens, starts, window=0, split=0, force_simt=False,
                    page_size=16, spike=None, decode_prefix=0, known=None, longest=0):
    lengths = [s + n for s, n in zip(starts, q_lens)]
    k_pages, v_pages, table, k_list, v_list = paged_cache(lengths, kv_heads, head_dim, page_size, dtype, DEV, seed=9)
    positions, seq_of_token, q_start, start_pos = batch_index(q_lens, starts, DEV)
    T = sum(q_lens)
    gen = torch.Generator().manual_seed(17)
    stride = heads * head_dim + 24          # rows wider than the queries, as inside a fused qkv buffer
    buf = torch.randn(T, stride, generator=gen).to(dtype)
    if spike is not None:
        # make one (far) key of request 0 dominate the first query head of its last row
        seq, key_pos = spike
        row = sum(q_lens[:seq + 1]) - 1
        direction = k_list[seq][key_pos, 0].float()
        buf[row, :head_dim] = (direction / direction.norm() * 60.0).to(dtype)
    scale = 1.0 / math.sqrt(head_dim)
    dq = buf.to(DEV)
    out = ops.attention(dq[:, :heads * head_dim], k_pages, v_pages, table, q_start, start_pos, positions,
                        seq_of_token, len(q_lens), longest or max(q_lens), max(lengths), heads, kv_heads, head_dim, scale,
                        window=window, split_tokens=split, force_simt=force_simt, decode_prefix=decode_prefix, **(known or {}))
    ops.check_status()
    q = buf[:, :heads * head_dim].view(T, heads, head_dim)
    refs = []
    for s, (n, start) in enumerate(zip(q_lens, starts)):
        begin = sum(q_lens[:s])
        refs.append(ops_plain.attention_rows(q[begin:begin + n], k_list[s], v_list[s], range(start, start + n),
                                             scale, window))
    ref = torch.cat(refs).reshape(T, heads * head_dim)
    return rel_error(out, ref), out, ref


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(6, 2, 48), (3, 1, 32), (4, 4, 16), (7, 1, 128), (2, 2, 100)])
def test_attention_simt(ops, dtype, heads, kv_heads, head_dim):
    err, _, _ = _attention_case(ops, dtype, heads, kv_heads, head_dim, [5, 1, 37, 2], [30, 150, 0, 63],
                                force_simt=True)
    assert err < TOL[dtype]


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size,window", [
    (7, 1, 128, 16, 0), (12, 2, 64, 64, 0), (3, 1, 32, 16, 100), (4, 2, 16, 5, 0), (34, 2, 128, 16, 300), (4, 4, 128, 64, 1)])
def test_attention_float32_rows_do_not_depend_on_the_step(ops, heads, kv_heads, head_dim, page_size, window):
    """The tiled float32 kernel: lengths at the edges of its tiles (64 keys) and runs (256), and one request whole, in
    portions and token by token (16 and 64 rows to a block, runs inside a block and merged) to the same bits."""
    case = lambda q_lens, starts, **kw: _attention_case(ops, torch.float32, heads, kv_heads, head_dim, q_lens, starts,
                                                        page_size=page_size, window=window, **kw)
    err, out, ref = case([1, 1, 9, 65, 1, 257], [0, 63, 64, 190, 256, 511])
    simt, _, _ = case([1, 1, 9, 65, 1, 257], [0, 63, 64, 190, 256, 511], force_simt=True)
    # 64 keys are summed before they join the rest and a score in four parts, so no more error than key by key;
    # a quarter more for rounding's luck
    assert err < TOL[torch.float32] and err <= 1.25 * simt + 1e-8
    if page_size != 16:
        return
    # the same keys and queries in other cuts
    lengths = 600
    k_pages, v_pages, table, _k, _v = paged_cache([lengths], kv_heads, head_dim, page_size, torch.float32, DEV, seed=3)
    q = torch.randn(lengths, heads * head_dim, generator=torch.Generator().manual_seed(4)).to(DEV)

    def rows(start, count, bound=lengths):
        positions, seq_of_token, q_start, start_pos = batch_index([count], [start], DEV)
        return ops.attention(q[start:start + count], k_pages, v_pages, table, q_start, start_pos, positions, seq_of_token, 1,
                             count, bound, heads, kv_heads, head_dim, head_dim ** -0.5, window=window)
    whole = rows(0, lengths)
    for start, count in ((0, 1), (63, 1), (64, 2), (255, 3), (256, 1), (300, 30), (599, 1), (410, 190)):
        assert torch.equal(rows(start, count), whole[start:start + count]), (start, count)
    assert torch.equal(rows(520, 1, bound=4096), whole[520:521])
    ops.check_status()


@pytest.mark.parametrize("group,counts", [(1, (16, 17, 32, 33, 64, 65)), (7, (2, 3, 4, 5, 9)), (16, (1, 2, 3)), (17, (1, 2)), (32, (1, 2)), (33, (1, 2)), (64, (1, 2))])
def test_attention_float32_rows_have_the_bits_of_any_block(ops, group, counts):
    """Portions around the lines between 16, 32 and 64 rows to a block, alone (blocks find an SM each) and repeated in a step of many
    requests (they do not), against the whole prompt in one step."""
    length, head_dim = 330, 64
    k_pages, v_pages, table, _k, _v = paged_cache([length], 2, head_dim, 16, torch.float32, DEV, seed=3)
    q = torch.randn(length, 2 * group * head_dim, generator=torch.Generator().manual_seed(4)).to(DEV)

    def rows(starts, count):
        positions, seq_of_token, q_start, start_pos = batch_index([count] * len(starts), starts, DEV)
        return ops.attention(torch.cat([q[s:s + count] for s in starts]), k_pages, v_pages, table.expand(len(starts), -1).contiguous(), q_start,
                             start_pos, positions, seq_of_token, len(starts), count, length, 2 * group, 2, head_dim, 0.1)
    whole = rows([0], length)
    for count in counts:
        starts = [0, 63, 255, length - count] * 50
        alone, many = rows(starts[:1], count), rows(starts, count)
        assert torch.equal(alone, whole[:count])
        for i, s in enumerate(starts[:4]):
            assert torch.equal(many[i * count:(i + 1) * count], whole[s:s + count]), (count, s)
        assert torch.equal(many.view(50, -1), many.view(50, -1)[:1].expand(50, -1))
    ops.check_status()


@pytest.mark.parametrize("heads,kv_heads,head_dim,page_size,window,q_lens,starts", [
    (28, 4, 128, 16, 0, [1500, 37, 1], [0, 300, 70]), (40, 8, 64, 64, 200, [1030, 260], [15, 0]), (16, 8, 32, 16, 0, [900, 333, 300], [1, 64, 0]),
    (28, 4, 128, 16, 0, [1024], [0]), (28, 4, 128, 64, 0, [250], [5]), (28, 4, 128, 16, 0, [300], [4100]), (12, 2, 128, 64, 0, [130] * 9, [0] * 9)])
def test_attention_prefill_on_both_sides_of_the_two_tile_rule(ops, heads, kv_heads, head_dim, page_size, window, q_lens, starts):
    """Portions that take two query tiles to a block (many blocks or long keys) and portions that take one."""
    err, _, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, q_lens, starts, page_size=page_size, window=window)
    assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("heads,kv_heads,head_dim,count,length", [
    (12, 2, 128, 32, 64), (12, 2, 128, 8, 300), (28, 4, 128, 20, 64), (40, 8, 128, 6, 128), (4, 4, 128, 40, 200), (14, 2, 64, 40, 17)])
def test_attention_of_short_prompts_on_both_sides_of_the_rule_for_waves(ops, heads, kv_heads, head_dim, count, length):
    """Many short prompts: one query tile to a block unless that takes twice the waves of two, the last prompt longer than the rest."""
    err, _, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, [length] * (count - 1) + [length + 9], [0] * count, page_size=64)
    assert err < TOL[torch.bfloat16]


def test_leading_single_tokens_deep_in_long_contexts_get_splits_of_their_own(ops):
    """A mixed step: nine single tokens at contexts of about 4,000 beside a prompt of 300 tokens.  The prompt's
    keys are not cut; the single tokens, a decode batch of their own, have theirs cut (the choice is automatic
    here), and one far key dominates a row so that a split lost in the merge would show."""
    starts = [4000 + 37 * i for i in range(9)] + [0]
    err, _, _ = _attention_case(ops, torch.bfloat16, 14, 2, 128, [1] * 9 + [300], starts, decode_prefix=9, spike=(0, 123))
    assert err < TOL[torch.bfloat16]
    assert ops.choose_attention_split(9, 9, 1, 4400, 14, 2, bound=4400) > 0          # the single tokens' keys are cut
    starts = [4000 + 37 * i for i in range(9)] + [2900]                                # ... also beside a long portion
    err, _, _ = _attention_case(ops, torch.bfloat16, 14, 2, 128, [1] * 9 + [1500], starts, decode_prefix=9, spike=(0, 123))
    assert err < TOL[torch.bfloat16]
    assert ops.choose_attention_split(1509, 10, 1500, 4400, 14, 2, bound=4400) == 0  # whose keys are not cut


@pytest.mark.parametrize("heads,kv_heads,head_dim,window", [(14, 2, 128, 0), (8, 2, 64, 0), (6, 2, 48, 0), (20, 1, 128, 0), (14, 2, 128, 300)])
@pytest.mark.parametrize("lead,portions,starts", [
    ([1800, 3, 900, 64, 63, 1200, 65, 5], [70], [0]), ([40, 30, 20, 10, 5, 4, 3, 2], [200, 3], [0, 700]), ([1500] * 9, [17, 300], [128, 0])])
def test_mixed_steps_whose_lengths_are_known(ops, heads, kv_heads, head_dim, window, lead, portions, starts):
    """Single tokens cut at an SM's share of their keys or not at all, beside portions that are served by their own longest context: the
    longest request among the single tokens, among the portions, all alike; a group too large for the decode kernel, pages of a
    head size that goes without tensor maps, a window."""
    q_lens, begins = [1] * len(lead) + portions, lead + starts
    known = dict(lead_keys=sum(lead) + len(lead), lead_longest=max(lead) + 1, rest_ctx_len=max(s + n for s, n in zip(starts, portions)))
    err, _, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, q_lens, begins, window=window, decode_prefix=len(lead), known=known,
                                spike=(0, lead[0] - 1))
    assert err < TOL[torch.bfloat16]


def test_side_by_side_attention_is_done_before_what_follows(ops):
    """The two attention kernels of a mixed step run side by side; the kernels behind them (here products over their rows, and the next step's
    attention into the same buffer) find both done, every time."""
    lead = [int(n) for n in torch.randint(50, 3000, (40,), generator=torch.Generator().manual_seed(1))]
    q_lens, starts = [1] * len(lead) + [90], lead + [0]
    k_pages, v_pages, table, _k, _v = paged_cache([a + n for a, n in zip(starts, q_lens)], 4, 128, 64, torch.bfloat16, DEV, seed=5)
    positions, seq_of_token, q_start, start_pos = batch_index(q_lens, starts, DEV)
    gen = torch.Generator().manual_seed(6)
    q = [torch.randn(sum(q_lens), 28 * 128, generator=gen).to(torch.bfloat16).to(DEV) for _ in range(2)]
    w = (torch.randn(256, 28 * 128, generator=gen) * 0.02).to(torch.bfloat16).to(DEV)
    out = torch.zeros_like(q[0])
    first = [None, None]
    for i in range(40):
        ops.attention(q[i % 2], k_pages, v_pages, table, q_start, start_pos, positions, seq_of_token, len(q_lens), 90, max(lead) + 1, 28, 4, 128,
                      128 ** -0.5, decode_prefix=len(lead), lead_keys=sum(lead) + 40, lead_longest=max(lead) + 1, rest_ctx_len=90, out=out)
        rows = ops.linear(out, w, None, ops.GEMM_STORE_F32, settled=True)
        if first[i % 2] is None:
            first[i % 2] = rows
        assert torch.equal(rows, first[i % 2]), i
    ops.check_status()


@pytest.mark.parametrize("tokens,longest", [(8, 4), (30, 2)])
def test_a_step_of_single_tokens_whose_bound_says_more(ops, tokens, longest):
    """All portions single tokens, as ``decode_prefix`` says, under a looser bound of their length: no portion is left behind them."""
    err, _, _ = _attention_case(ops, torch.bfloat16, 14, 2, 128, [1] * tokens, [2300] + [40] * (tokens - 1), decode_prefix=tokens, longest=longest)
    assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("lead,portions,starts,lead_is_cut,rest_is_cut", [
    (list(range(100, 4001, 100)), [90], [0], True, False),          # singles cut, their states merged behind both kernels
    (list(range(60, 640, 20)), [64], [4000], False, True),          # the portion's keys cut beside them
    (list(range(300, 940, 80)), [1187], [0], False, False)])      # a prompt for blocks of two query tiles, its rows from a kernel of another kind
@pytest.mark.parametrize("captured", [False, True])
def test_side_by_side_attention_sees_what_the_kernels_in_front_have_just_written(ops, lead, portions, starts, lead_is_cut, rest_is_cut, captured):
    """Queries, keys and values come out of the product and store right in front, other ones in every turn.  Expected: the single tokens and the
    portions in calls of their own, everything waited for.  In a captured graph, whose replays repeat one launch, the kernels wait."""
    from aegean_tge_b200.parts.rope import rotary_tables
    heads, kv_heads, head_dim, hidden, page_size = 28, 4, 128, 256, 64
    q_lens, begins, n = [1] * len(lead) + portions, lead + starts, len(lead)
    lengths = [a + m for a, m in zip(begins, q_lens)]
    known = dict(lead_keys=sum(lengths[:n]), lead_longest=max(lengths[:n]), rest_ctx_len=max(lengths[n:]))
    lead_cut = ops.choose_leading_split(n, known["lead_keys"], known["lead_longest"], kv_heads, max(lengths))
    rest_cut = ops.choose_attention_split(sum(portions), len(portions), max(portions), known["rest_ctx_len"], heads, kv_heads, bound=known["rest_ctx_len"])
    assert (lead_cut > 0) == lead_is_cut and (rest_cut > 0) == rest_is_cut
    k_pages, v_pages, table, _k, _v = paged_cache(lengths, kv_heads, head_dim, page_size, torch.bfloat16, DEV, seed=5)
    positions, seq_of_token, q_start, start_pos = batch_index(q_lens, begins, DEV)
    cos, sin = (t.to(DEV) for t in rotary_tables(10000.0, head_dim, 4096))
    gen = torch.Generator().manual_seed(6)
    tokens, turns = sum(q_lens), 6
    x = [torch.randn(tokens, hidden, generator=gen).to(torch.bfloat16).to(DEV) for _ in range(turns)]
    w = (torch.randn((heads + 2 * kv_heads) * head_dim, hidden, generator=gen) * 0.1).to(torch.bfloat16).to(DEV)
    w_o = (torch.randn(256, heads * head_dim, generator=gen) * 0.02).to(torch.bfloat16).to(DEV)
    attended, results = torch.zeros(tokens, heads * head_dim, dtype=torch.bfloat16, device=DEV), torch.zeros(turns, tokens, 256, device=DEV)

    def store(i):
        return ops.linear_qkv_rope_store(x[i], w, None, cos, sin, head_dim, positions, seq_of_token, table, k_pages, v_pages, heads, kv_heads, head_dim)

    def turn(i):
        qkv = store(i)
        ops.attention(qkv[:, :heads * head_dim], k_pages, v_pages, table, q_start, start_pos, positions, seq_of_token, len(q_lens), max(q_lens),
                      max(lengths), heads, kv_heads, head_dim, head_dim ** -0.5, decode_prefix=n, out=attended, **known)
        ops.linear(attended, w_o, None, ops.GEMM_STORE_F32, out=results[i])

    # positions and q_start of a call count from the call's first token
    wanted = []
    rest = batch_index(portions, starts, DEV)
    for i in range(turns):
        qkv = store(i)
        torch.cuda.synchronize()
        rows = torch.zeros_like(attended)
        ops.attention(qkv[:n, :heads * head_dim], k_pages, v_pages, table[:n].contiguous(), q_start[:n + 1], start_pos[:n], positions[:n],
                      seq_of_token[:n], n, 1, known["lead_longest"], heads, kv_heads, head_dim, head_dim ** -0.5, out=rows[:n])
        torch.cuda.synchronize()
        ops.attention(qkv[n:, :heads * head_dim], k_pages, v_pages, table[n:].contiguous(), rest[2], rest[3], rest[0], rest[1], len(portions),
                      max(portions), known["rest_ctx_len"], heads, kv_heads, head_dim, head_dim ** -0.5, out=rows[n:])
        torch.cuda.synchronize()
        wanted.append(ops.linear(rows, w_o, None, ops.GEMM_STORE_F32))
        torch.cuda.synchronize()
    if captured:
        turn(0)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for i in range(turns):
                turn(i)
        run = graph.replay
    else:
        run = lambda: [turn(i) for i in range(turns)]
    for _ in range(4):
        results.zero_()
        run()
        for i in range(turns):
            assert rel_error(results[i], wanted[i]) < TOL[torch.bfloat16], i
    ops.check_status()


def test_leading_single_tokens_that_fill_the_chip_are_not_cut(ops, monkeypatch):
    """A mixed step whose single tokens occupy the SMs as they are: cut, they would cost more states to write and to merge than
    the parallel runs give back, and with kept first tokens scratch memory for runs of the whole context.  They have the
    bits of the uncut walk, and the step asks for no scratch memory."""
    for heads, kv_heads, starts, options in ((28, 4, [900] * 40, {}), (28, 4, [1500 + 3 * i for i in range(38)], dict(window=300, keep_first=64))):
        q_lens = [1] * len(starts) + [70]
        k_pages, v_pages, table, _k, _v = paged_cache([s + n for s, n in zip(starts + [0], q_lens)], kv_heads, 128, 64, torch.bfloat16, DEV, seed=5)
        positions, seq_of_token, q_start, start_pos = batch_index(q_lens, starts + [0], DEV)
        q = torch.randn(sum(q_lens), heads * 128, generator=torch.Generator().manual_seed(6)).to(torch.bfloat16).to(DEV)
        run = lambda **kw: ops.attention(q, k_pages, v_pages, table, q_start, start_pos, positions, seq_of_token, len(q_lens), 70,
                                         max(starts) + 1, heads, kv_heads, 128, 128 ** -0.5, decode_prefix=len(starts), **options, **kw)
        with monkeypatch.context() as patch:
            patch.setattr(ops, "_scratch", {})
            chosen = run()
            assert not ops._scratch
        assert torch.equal(chosen, run(split_tokens=1 << 20))
    ops.check_status()


@pytest.mark.parametrize("split,window", [(256, 0), (128, 0), (64, 0), (64, 700)])
def test_attention_merges_many_splits(ops, split, window):
    """Single tokens deep in a context, their keys cut into 14, 28 and 55 splits: the merging kernel hands round the splits'
    weights lane by lane, up to four to a lane, and asks for sixteen states at a time; with a window most splits hold no
    visible key.  One far key is made to dominate, so a split dropped or counted twice would show."""
    err, _, _ = _attention_case(ops, torch.bfloat16, 14, 2, 128, [1, 1, 1], [3499, 1200, 65], window=window, split=split,
                                spike=(0, 3000 if window else 17))
    assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("heads,kv_heads,head_dim,start,window", [
    (7, 1, 128, 8191, 0), (7, 1, 128, 8192, 0), (4, 1, 64, 9100, 0), (2, 1, 32, 12000, 0), (7, 1, 128, 9000, 8300)])
def test_attention_merges_more_splits_than_a_warp_holds(ops, heads, kv_heads, head_dim, start, window):
    """Keys in splits of 64: 128 of them, the most whose weights a warp holds, and more, which are walked one by one; far keys
    at both ends of the walk dominate in turn."""
    for spike in ((0, 5 if not window else start - window + 3), (0, start - 1)):
        err, _, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, [1, 1], [start, 70], window=window, split=64, spike=spike)
        assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(7, 1, 128), (28, 4, 64), (6, 2, 48), (40, 2, 16)])
@pytest.mark.parametrize("page_size,split,window", [(16, 0, 0), (64, 128, 0), (4, 64, 0), (16, 0, 40), (32, 64, 100)])
def test_attention_routes_leading_single_tokens_to_the_decode_kernel(ops, heads, kv_heads, head_dim, page_size, split,
                                                                     window):
    """A step whose first ten sequences bring one token each and whose last two bring portions: told so, the
    tensor-core path serves the ten with its decode kernel and the rest with its prefill kernel (with and without
    a cut of the keys, whose partial results share one scratch buffer); untold, one kernel serves all.  Both are
    right, and they agree to rounding.  One single token sits at position 0, one far into its sequence; with a
    window some splits hold no visible key."""
    q_lens = [1] * 10 + [70, 3]
    starts = [0, 199, 64, 5, 130, 17, 63, 64, 255, 1] + [200, 15]
    routed, out_routed, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, q_lens, starts, split=split,
                                            page_size=page_size, decode_prefix=10, window=window)
    plain_way, out_plain, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, q_lens, starts, split=split,
                                              page_size=page_size, window=window)
    assert routed < TOL[torch.bfloat16] and plain_way < TOL[torch.bfloat16]
    assert rel_error(out_routed, out_plain.float()) < TOL[torch.bfloat16]


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(6, 2, 48), (3, 1, 32), (4, 4, 16), (7, 1, 128), (28, 4, 64),
                                                     (5, 5, 80), (40, 2, 16), (4, 2, 256), (6, 2, 192)])
@pytest.mark.parametrize("q_lens,starts", [([5, 1, 37, 2], [30, 150, 0, 63]), ([1, 1, 1], [0, 199, 64]),
                                           ([130], [0]), ([70, 3], [200, 15])])
def test_attention_mma(ops, heads, kv_heads, head_dim, q_lens, starts):
    err, _, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, q_lens, starts)
    assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("split", [64, 128, 192])
@pytest.mark.parametrize("q_lens,starts", [([1, 1, 1, 1], [700, 3, 255, 256]), ([40, 1], [300, 129])])
def test_attention_mma_split_keys(ops, split, q_lens, starts):
    err, _, _ = _attention_case(ops, torch.bfloat16, 7, 1, 128, q_lens, starts, split=split)
    assert err < TOL[torch.bfloat16]
    err, _, _ = _attention_case(ops, torch.bfloat16, 6, 2, 48, q_lens, starts, split=split)
    assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(28, 4, 128), (10, 2, 64), (16, 1, 128)])
@pytest.mark.parametrize("split,window", [(128, 0), (512, 0), (256, 300), (64, 0), (192, 77)])
def test_attention_decode_splits(ops, heads, kv_heads, head_dim, split, window):
    """Single tokens with two to sixteen key splits, some of them without keys for the short requests."""
    err, _, _ = _attention_case(ops, torch.bfloat16, heads, kv_heads, head_dim, [1, 1, 1, 1, 1], [1000, 0, 511, 512, 130],
                                window=window, split=split)
    assert err < TOL[torch.bfloat16]


@pytest.mark.parametrize("dtype,simt", [(torch.float32, True), (torch.bfloat16, True), (torch.bfloat16, False)])
def test_attention_reads_a_far_key(ops, dtype, simt):
    """One key hundreds of positions back carries almost all the weight: the output must be its value."""
    err, out, ref = _attention_case(ops, dtype, 4, 2, 64, [1, 3], [600, 20], force_simt=simt, spike=(0, 7))
    assert err < TOL[dtype]


@pytest.mark.parametrize("dtype,simt", [(torch.float32, True), (torch.bfloat16, False)])
@pytest.mark.parametrize("window", [1, 16, 40, 65])
def test_attention_window_edge(ops, dtype, simt, window):
    """With a window the key just outside it must not count, however strong; the one just inside must."""
    for key_offset in (window, window - 1):           # just outside / just inside (distance from the query)
        start = 300
        if key_offset > start:
            continue
        err, out, ref = _attention_case(ops, dtype, 4, 2, 64, [1, 5], [start, 100], window=window, force_simt=simt,
                                        spike=(0, start - key_offset))
        assert err < TOL[dtype]
    err, _, _ = _attention_case(ops, dtype, 4, 2, 64, [33, 2], [60, 10], window=window, force_simt=simt, split=64 if not simt else 0)
    assert err < TOL[dtype]


# ---------------------------------------------------------------------------
# sampling
# ---------------------------------------------------------------------------
def test_sample_greedy_takes_the_first_maximum(ops):
    logits = torch.zeros(3, 1000)
    logits[0, 17] = 5.0
    logits[0, 800] = 5.0                         # a tie: the lower index wins (sampling.cpp:198-207)
    logits[1, 999] = 1.0
    logits[2, :] = -3.0                          # all equal: index 0
    ids = ops.sample(logits.to(DEV), torch.zeros(3, device=DEV), torch.zeros(3, device=DEV))
    assert ids.cpu().tolist() == [17, 999, 0]


@pytest.mark.parametrize("vocab", [331, 4097, 152064])
def test_sample_temperature_lands_where_the_draw_points(ops, vocab):
    """The chosen index is the one whose slice of the exact (float64) cumulative distribution holds the
    draw u.  Float32 sums over n terms are exact to about n * 2^-24 of the total, so the draw may sit
    that far outside the chosen slice, no further; on a small vocabulary the kernel must also agree
    with the sequential float32 walk of the reference."""
    from plain.qwen2_plain import sample_plain
    import numpy as np
    gen = torch.Generator().manual_seed(vocab)
    rows = 6
    logits = torch.randn(rows, vocab, generator=gen) * 2.0
    temps = [0.8, 1.0, 0.3, 2.0, 0.8, 0.05]
    uniforms = [0.37, 0.9991, 0.0004, 0.5, 0.73, 0.11]
    ids = ops.sample(logits.to(DEV), torch.tensor(temps, device=DEV), torch.tensor(uniforms, device=DEV)).cpu().tolist()
    slack = vocab * 2.0 ** -24

    class Fixed:
        def __init__(self, u): self.u = u
        def next(self): return np.float32(self.u)
    for r in range(rows):
        z = logits[r].double()
        e = torch.exp((z - z.max()) / temps[r])
        cdf = torch.cumsum(e, 0) / e.sum()
        lower = float(cdf[ids[r] - 1]) if ids[r] > 0 else 0.0
        assert lower - slack <= uniforms[r] <= float(cdf[ids[r]]) + slack, (r, ids[r], lower, float(cdf[ids[r]]))
        if vocab <= 4097:
            assert ids[r] == sample_plain(logits[r].numpy(), temps[r], Fixed(uniforms[r]))


def test_sample_histogram_follows_the_distribution(ops):
    """Many draws from a small distribution: observed frequencies within a chi-square bound."""
    from aegean_tge_b200.sampling import XorShift32
    probs = torch.tensor([0.5, 0.25, 0.125, 0.0625, 0.0625])
    logits = torch.log(probs)[None, :].repeat(4000, 1)
    rng = XorShift32(123)
    uniforms = torch.tensor([rng.next_uniform() for _ in range(4000)])
    ids = ops.sample(logits.to(DEV), torch.ones(4000, device=DEV), uniforms.to(DEV)).cpu()
    counts = torch.bincount(ids.long(), minlength=5).double()
    expected = probs.double() * 4000
    chi2 = float(((counts - expected) ** 2 / expected).sum())
    assert chi2 < 20.5          # 4 degrees of freedom, p ~ 4e-4


def test_a_bounded_wait_gives_up_and_leaves_the_device_usable():
    """The product kernels wait on barriers with a time limit; when it runs out they set a status bit and
    unwind instead of hanging.  A one-thread kernel makes that wait run out on purpose (a barrier nothing
    arrives at, a limit of 1 ms): the launch returns, the status word says so once, and a product right
    afterwards is exact."""
    from aegean_tge_b200 import ops
    ops.check_status()
    arrived, took = ops.wait_gives_up(1_000_000)
    torch.cuda.synchronize()
    assert not arrived and 1_000_000 <= took < 50_000_000, (arrived, took)
    with pytest.raises(ops.DeviceStatusError, match="wait gave up"):
        ops.check_status()
    ops.check_status()                                  # reading it cleared it
    with pytest.raises(ops.KernelError):
        ops.wait_gives_up(10**9)                        # long limits are refused outright
    x = torch.randint(-3, 4, (24, 256), device="cuda").to(torch.bfloat16)
    w = torch.randint(-3, 4, (384, 256), device="cuda").to(torch.bfloat16)
    out = ops.linear(x, w, None, ops.GEMM_STORE_F32)
    assert torch.equal(out, x.float() @ w.float().T)    # small integers: exact in bfloat16 products and float32 sums
    ops.check_status()
