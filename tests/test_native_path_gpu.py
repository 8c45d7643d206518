"""The native call path (csrc/host.cpp) against the Python path of the same operators, bit for bit (an explicit stream
argument selects the latter), and the rows a grouped call has to clear itself."""
import pytest
import torch

import tilelang_ascend_b200 as q
from oracle import qgemm_oracle as oc

pytestmark = pytest.mark.gpu


def _dirty(nbytes):
    """Leave memory of this size in the caching allocator that does not hold zeros."""
    t = torch.full((nbytes,), 0x55, dtype=torch.uint8, device="cuda")
    del t


@pytest.mark.parametrize("total,blocks", [
    (90, [(0, 0, 40), (1, 60, 30)]),                                      # a hole in the middle
    (300, [(0, 5, 100), (7, 105, 50), (1, 290, 10), (1, 4000, 10)]),      # holes at both ends, entries outside the tensors
    (40000, [(0, 128 * i, 127) for i in range(300)]),                     # more rows than one pass of the grid, one row each open
    (1, [(0, 0, 0)]),                                                     # nothing covered
    (20011, [(1, 19000, 100)]),                                           # two tiles, rows to clear for every SM
    (5000, [(i % 2, 5 * i, 3) for i in range(1000)] + [(0, 4999, 1)]),    # a long table of short blocks
])
def test_grouped_clears_uncovered_rows(total, blocks):
    K, N, G = 32, 48, 2
    gen = torch.Generator().manual_seed(total)
    A = torch.randint(-128, 128, (total, K), dtype=torch.int8, generator=gen).cuda()
    B = torch.randint(-128, 128, (G, K, N), dtype=torch.int8, generator=gen).cuda()
    s = (torch.rand((G, N), generator=gen) * 0.02).cuda()
    meta = torch.tensor(blocks, dtype=torch.int32, device="cuda")
    _dirty(total * N * 2)
    C = q.grouped_quant_matmul(A, B, meta, s, out_dtype="float16")
    ref = torch.zeros((total, N), dtype=torch.float16)
    for g, m0, rows in blocks:
        if g < G and m0 < total and rows:
            acc = A[m0:m0 + rows].cpu().to(torch.int32) @ B[g].cpu().to(torch.int32)
            ref[m0:m0 + rows] = (acc.float() * s[g].cpu()).half()
    assert torch.equal(C.cpu(), ref)


@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_same_results_as_the_python_path(dt):
    here = torch.cuda.current_stream()
    A, B, sa, sb = None, None, None, None
    A, B, sa, sb = [t.cuda() for t in oc.make_w8a8_inputs(2, 70, 96, 80, seed=3)]
    args = dict(scale_a=sa, out_dtype=dt)
    assert torch.equal(q.quant_matmul(A, B, sb, **args), q.quant_matmul(A, B, sb, stream=here, **args))
    k = q.simple_quant_batch_matmul(2, 70, 80, 96, "N", 128, 256, 64, out_dtype=dt)
    assert torch.equal(k(A, B, sb, sa), k(A, B, sb, sa, stream=here))
    X = torch.randn((3, 7, 64), generator=torch.Generator().manual_seed(1)).to(getattr(torch, dt)).cuda()
    for a, b in zip(q.act_quant(X), q.act_quant(X, stream=here)):
        assert a.shape == b.shape and torch.equal(a, b)
    Aw, P, S = [t.cuda() for t in oc.make_w4a16_inputs(9, 512, 48, dt, 128, seed=4)]
    Z = torch.randint(0, 16, S.shape, generator=torch.Generator().manual_seed(2)).to(torch.float16).cuda()
    for kw in (dict(), dict(zeros=Z, zeros_mode="quantized"), dict(zeros=Z, zeros_mode="rescale"), dict(out_dtype="float16")):
        assert torch.equal(q.w4a16_gemm(Aw, P, S, **kw), q.w4a16_gemm(Aw, P, S, stream=here, **kw))
    assert torch.equal(q.w4a16_gemm(Aw, P), q.w4a16_gemm(Aw, P, stream=here))
    Xq, W, C = X.view(21, 64), torch.empty((4096, 64), dtype=torch.int8, device="cuda"), [torch.empty((21, 4096), dtype=torch.int32, device="cuda") for _ in range(2)]
    qB = torch.randint(0, 256, (4096, 32), dtype=torch.uint8, generator=torch.Generator().manual_seed(5)).cuda()
    a8, s8 = q.act_quant(Xq)
    q.w4a8_gemm_cv(21, 4096, 64)(a8, qB, W, C[0])
    q.w4a8_gemm_cv(21, 4096, 64)(a8, qB, W, C[1], stream=here)
    assert torch.equal(C[0], C[1])


def test_runs_on_the_current_stream_and_rejects_as_before():
    A, B, sa, sb = [t.cuda() for t in oc.make_w8a8_inputs(1, 64, 128, 64, seed=6)]
    A, B, sb = A[0], B[0], sb.view(-1)[:64].contiguous()
    want = q.quant_matmul(A, B, sb)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        A2 = A.clone()
        got = q.quant_matmul(A2, B, sb)
    side.synchronize()
    assert torch.equal(got, want)
    with pytest.raises(ValueError, match="contiguous"):
        q.quant_matmul(A.t(), B, sb)
    with pytest.raises(ValueError, match="dtype mismatch"):
        q.quant_matmul(A.float(), B, sb)
    with pytest.raises(ValueError, match="scale"):
        q.quant_matmul(A, B, sb[:5].contiguous())
    with pytest.raises(ValueError, match="device mismatch"):
        q.quant_matmul(A, B, sb.cpu())
    assert q.quant_matmul(A[:0], B, sb).shape == (0, 64)


def test_function_transforms_are_refused_in_torch_words():
    """Under vmap and jvp the arguments are wrappers without storage: every operator raises, as on the Python path, and the
    process goes on (the exception is met while the interpreter lock is released)."""
    A, B, sa, sb = [t.cuda() for t in oc.make_w8a8_inputs(2, 16, 64, 32, seed=9)]
    X = torch.randn((2, 16, 64), device="cuda").half()
    P = torch.zeros((32, 32), dtype=torch.uint8, device="cuda")
    W, C = torch.empty((32, 64), dtype=torch.int8, device="cuda"), torch.empty((16, 32), dtype=torch.int32, device="cuda")
    meta = q.build_block_metadata((16,), 128, "cuda")
    calls = [(lambda a: q.quant_matmul(a, B[0], sb[0]), A), (q.act_quant, X), (lambda x: q.w4a16_gemm(x, P), X),
             (lambda a: q.w4a8_gemm_cv(16, 32, 64)(a, P, W, C), A), (lambda x: q.w4a8_gemm_act_quant(16, 32, 64)(x, P, W, C), X),
             (lambda a: q.grouped_quant_matmul(a, B[:1], meta, sb[0]), A)]
    for call, arg in calls:
        with pytest.raises(RuntimeError):
            torch.vmap(call)(arg)
    for call in (q.act_quant, lambda x: q.w4a16_gemm(x, P)):
        with pytest.raises(RuntimeError):
            torch.func.jvp(call, (X[0],), (X[1],))
    assert q.quant_matmul(A[0], B[0], sb[0]).shape == (16, 32)


def test_integral_floats_in_a_factory():
    """A factory takes its shape by value, so 16.0 is 16; and a shape that does not fit is refused either way."""
    A, P, S = [t.cuda() for t in oc.make_w4a16_inputs(16, 512, 256, "float16", 128, seed=8)]
    want = q.w4a16_gemm(A, P, S)
    assert torch.equal(q.dequant_gemm_fp16_wrapper(16.0, 256.0, 512.0, 128, 256, 64)(A, P, S), want)
    with pytest.raises(ValueError, match="shape mismatch"):
        q.dequant_gemm_fp16_wrapper(17.0, 256, 512, 128, 256, 64)(A, P, S)
    y, s = q.act_quant_kernel_int8_optimized(512.0)(A)
    y0, s0 = q.act_quant(A)
    assert torch.equal(y, y0) and torch.equal(s, s0.view(-1))
    with pytest.raises(ValueError, match="shape"):
        q.act_quant_kernel_int8_optimized(256.0)(A)
