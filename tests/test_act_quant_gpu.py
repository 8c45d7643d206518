"""GPU parity of the per-token activation quantiser (examples/deepseek_v4/act_quant.py) through the C ABI."""
import pytest
import torch

import tilelang_ascend_b200 as q
from oracle import qgemm_oracle as oc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,round_scale,bf16", [("act_quant_2d", False, ("x",)),
                                                   ("act_quant_3d_round", True, ("x",)),
                                                   ("act_quant_f16", False, ())])
def test_reference_vectors(golden, name, round_scale, bf16):
    c = golden.case(name, bf16=bf16)
    y, s = q.act_quant(c["x"].cuda(), round_scale=round_scale)
    assert y.shape == c["y"].shape and s.shape == c["s"].shape
    assert torch.equal(y.cpu(), c["y"])
    assert torch.equal(s.cpu(), c["s"])


# rows of 8 .. 16392 elements: one warp per row up to a whole block per row, and the re-read path beyond
SHAPES = [(1, 8), (7, 264), (64, 1024), (33, 2056), (130, 4096), (48, 7168), (5, 16384), (3, 16392), (2, 40000)]


@pytest.mark.parametrize("M,N", SHAPES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_matches_oracle_bit_for_bit(M, N, dtype):
    g = torch.Generator().manual_seed(M * 100003 + N)
    x = (torch.randn(M, N, generator=g) * torch.rand(M, 1, generator=g) * 8).to(dtype)
    y_ref, s_ref = oc.act_quant_torch_ref(x)
    y, s = q.act_quant(x.cuda())
    assert torch.equal(s.cpu(), s_ref)
    assert torch.equal(y.cpu(), y_ref)


def test_round_scale_is_a_power_of_two_not_below_amax_over_127():
    g = torch.Generator().manual_seed(3)
    x = (torch.randn(200, 512, generator=g) * 5).to(torch.bfloat16)
    x[0] = 0
    x[1, :] = 127.0  # amax / 127 == 1 exactly: the power of two is 1, not 2
    y, s = q.act_quant(x.cuda(), round_scale=True)
    y_ref, s_ref = oc.act_quant_torch_ref(x, round_scale=True)
    assert torch.equal(s.cpu(), s_ref) and torch.equal(y.cpu(), y_ref)
    m, e = torch.frexp(s.cpu())
    assert torch.all(m == 0.5)
    assert float(s[1]) == 1.0 and torch.all(y[1] == 127)


def test_zero_rows_and_empty_input():
    x = torch.zeros(4, 64, dtype=torch.bfloat16, device="cuda")
    y, s = q.act_quant(x)
    assert torch.all(y == 0)
    assert torch.equal(s.cpu(), torch.full((4, 1), 1e-4, dtype=torch.float32) / 127.0)
    y, s = q.act_quant(torch.empty(0, 64, dtype=torch.bfloat16, device="cuda"))
    assert y.shape == (0, 64) and s.shape == (0, 1)


def test_feeds_the_w8a8_gemm():
    """act_quant -> quant_matmul(A, B, scale_b, scale_a) equals the oracle chain on the same inputs."""
    g = torch.Generator().manual_seed(11)
    M, K, N = 96, 512, 272
    x = torch.randn(M, K, generator=g).to(torch.bfloat16)
    B = torch.randint(-128, 128, (K, N), dtype=torch.int8, generator=g)
    sb = torch.rand(N, generator=g) * 0.02 + 0.001
    a8, sa = q.act_quant(x.cuda())
    C = q.quant_matmul(a8, B.cuda(), sb.cuda(), scale_a=sa.view(-1), out_dtype="bfloat16")
    a8_ref, sa_ref = oc.act_quant_torch_ref(x)
    C_ref = oc.quant_matmul_ref(a8_ref, B, sb, "bfloat16", scale_a=sa_ref.view(-1))
    assert torch.equal(C.cpu(), C_ref)


def test_factory_signature_and_errors():
    kernel = q.act_quant_kernel_int8_optimized(256, block_M=16, block_N=256, round_scale=False)
    x = torch.randn(20, 256).to(torch.bfloat16)
    y, s = kernel(x.cuda())
    y_ref, s_ref = oc.act_quant_torch_ref(x)
    assert s.shape == (20,) and torch.equal(y.cpu(), y_ref) and torch.equal(s.cpu(), s_ref.view(-1))
    with pytest.raises(ValueError):
        kernel(torch.zeros(4, 128, dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(ValueError):
        q.act_quant_kernel_int8_optimized(100)
    with pytest.raises(ValueError):
        q.act_quant(torch.zeros(4, 64, dtype=torch.float32, device="cuda"))
    with pytest.raises(q.QGemmError):
        q.act_quant(torch.zeros(4, 12, dtype=torch.bfloat16, device="cuda"))


@pytest.mark.parametrize("M,K,N,dtype,round_scale", [(1, 1024, 4096, torch.bfloat16, False), (16, 8192, 1024, torch.bfloat16, False),
                                                     (37, 4096, 2560, torch.float16, True), (128, 2048, 10240, torch.bfloat16, False),
                                                     (5, 16384 + 256, 272, torch.float16, False)])
def test_quantiser_fused_into_the_w4a8_operator(M, K, N, dtype, round_scale):
    """bf16 / f16 activations straight into the W4A8 operator: scales and int32 results are those of the oracle's
    act_quant followed by its W4A8 GEMM, bit for bit, and of the two separate device calls."""
    g = torch.Generator().manual_seed(M + K + N)
    x = (torch.randn(M, K, generator=g) * torch.rand(M, 1, generator=g) * 4).to(dtype)
    qB = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g)
    a8_ref, sa_ref = oc.act_quant_torch_ref(x, round_scale=round_scale)
    C_ref = oc.w4a8_gemm_ref(a8_ref, qB)
    ws = torch.empty((N, K), dtype=torch.int8, device="cuda")
    C = torch.empty((M, N), dtype=torch.int32, device="cuda")
    kernel = q.w4a8_gemm_act_quant(M, N, K, round_scale=round_scale)
    C, sa = kernel(x.cuda(), qB.cuda(), ws, C)
    assert torch.equal(sa.cpu(), sa_ref.view(-1))
    assert torch.equal(C.cpu(), C_ref)
    a8, sa2 = q.act_quant(x.cuda(), round_scale=round_scale)
    C2 = q.w4a8_gemm_cv(M, N, K)(a8, qB.cuda(), ws, torch.empty_like(C))
    assert torch.equal(C, C2) and torch.equal(sa, sa2.view(-1))


def test_fused_quantiser_needs_room_for_its_scratch_in_the_workspace():
    """The [N, K] int8 workspace is the only scratch the operator gets; a weight matrix smaller than the kernel's own
    scratch (a few MB) is rejected with a message instead of being overrun."""
    M, K, N = 4, 256, 128
    kernel = q.w4a8_gemm_act_quant(M, N, K)
    with pytest.raises(q.QGemmError, match="workspace is too small"):
        kernel(torch.zeros((M, K), dtype=torch.bfloat16, device="cuda"), torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda"),
               torch.empty((N, K), dtype=torch.int8, device="cuda"), torch.empty((M, N), dtype=torch.int32, device="cuda"))


def test_fused_quantiser_rejects_more_than_128_tokens():
    M, K, N = 129, 256, 128
    kernel = q.w4a8_gemm_act_quant(M, N, K)
    with pytest.raises(q.QGemmError, match="M <= 128"):
        kernel(torch.zeros((M, K), dtype=torch.bfloat16, device="cuda"), torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda"),
               torch.empty((N, K), dtype=torch.int8, device="cuda"), torch.empty((M, N), dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("M,K,layers", [(1, 2048, 24), (24, 4096, 12), (40, 16384 + 256, 4)])
def test_chain_of_quantisers_and_few_token_gemms(M, K, layers):
    """Quantiser and few-token W8A8 kernel are programmatic dependents of each other: a chain in which each call reads what the
    one in front has just written is bit-identical to the same chain with the device drained between the calls."""
    g = torch.Generator().manual_seed(M + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).cuda()
    W = torch.randint(-128, 128, (K, K), dtype=torch.int8, generator=g).cuda()
    scale = (torch.rand(K, generator=g) / (0.577 * 74 * K ** 0.5)).cuda()  # a layer keeps its input's magnitude

    def chain(drain):
        h = x
        for _ in range(layers):
            a, sa = q.act_quant(h)
            if drain:
                torch.cuda.synchronize()
            h = q.quant_matmul(a, W, scale, scale_a=sa.view(-1), out_dtype="bfloat16")
            if drain:
                torch.cuda.synchronize()
        return h

    want = chain(True)
    for _ in range(3):
        assert torch.equal(chain(False), want)
    assert torch.isfinite(want.float()).all() and want.float().abs().max() > 0.1


@pytest.mark.parametrize("M", [8, 40])
def test_scales_written_in_front_of_the_quantiser(M):
    """The int4 GEMM reads its scales without waiting for the kernel directly in front of it.  Here that is the quantiser, and the
    kernel in front of the quantiser writes the scales: the chain is bit-identical to the one with the device drained between the
    calls."""
    K, N, rows = 4096, 4096, 32  # 32 groups of 128
    g = torch.Generator(device="cuda").manual_seed(M)
    a = torch.randint(-128, 128, (rows, K), dtype=torch.int8, generator=g, device="cuda")
    Ws = [torch.randint(-128, 128, (K, N), dtype=torch.int8, generator=g, device="cuda") for _ in range(3)]
    P = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    x = torch.randn((M, K), generator=g, device="cuda").half()
    scale = torch.full((1,), 1e-8, device="cuda")

    def chain(drain):
        step = torch.cuda.synchronize if drain else lambda: None
        out = []
        for i in range(12):
            S = q.quant_matmul(a, Ws[i % 3], scale, out_dtype="float16")
            step()
            y, s = q.act_quant(x)
            step()
            out += [q.w4a16_gemm(x, P, S, 8, 128), y, s]
            step()
        return out

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(u, v) for u, v in zip(chain(False), want))
    assert not torch.equal(want[0], want[3])


# On 148 SMs: tiles of 128 x 128, grouped ones of 128 x 256 in several rounds, tiles of two CTAs; more and fewer quantiser blocks than
# SMs.  (130 x 8192 by tiles of 128 x 128 too: its K is not cut, see the test below.)
@pytest.mark.parametrize("M,K,layers,layout", [(300, 1024, 12, "KN"), (130, 8192, 6, "KN"), (1150, 4096, 6, "NK"), (1200, 4096, 6, "KN"),
                                               (4096, 2048, 6, "NK"), (777, 512, 12, "KN")])
@pytest.mark.parametrize("grouped", [False, True])
def test_chain_of_quantisers_and_tile_gemms(M, K, layers, layout, grouped):
    """The tile kernels are programmatic dependents too, of the quantiser and of each other, and let the quantiser start early: a
    chain whose steps read what the one in front has just written - every other step two products in a row, into buffers that the
    allocator hands out again at once - is bit-identical to the same chain with the device drained between the calls."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    scale = torch.rand(K, generator=g, device="cuda") / (0.577 * 74 * K ** 0.5)  # a layer keeps its input's magnitude
    if grouped:
        sizes = (M // 3, 0, M - M // 3 - 7, 7)
        W = torch.randint(-128, 128, (4, K, K), dtype=torch.int8, generator=g, device="cuda")
        kernel = q.grouped_quant_gemm(sizes, K, K, out_dtype="bfloat16")
        meta, scales = kernel.block_metadata("cuda"), scale.expand(4, K).contiguous()
        product = lambda a, sa: kernel(a, W, meta, scales, sa)
    else:
        W = torch.randint(-128, 128, (K, K), dtype=torch.int8, generator=g, device="cuda")
        product = lambda a, sa: q.quant_matmul(a, W, scale, scale_a=sa, out_dtype="bfloat16", b_layout=layout)

    def chain(drain):
        step = torch.cuda.synchronize if drain else lambda: None
        h, first = x, None
        for i in range(layers):
            a, sa = q.act_quant(h)
            step()
            if i % 2:
                first = product(a, sa.view(-1))
                step()
            h = product(a, sa.view(-1))
            step()
        return h, first

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(u, v) for u, v in zip(chain(False), want))
    assert torch.isfinite(want[0].float()).all() and want[0].float().abs().max() > 0.1


# On 148 SMs the tile kernels' other forms: a K cut over two CTAs (even and odd number of k blocks; with accumulators only), tiles of
# 128 x 256 with a tail of half-width ones, grouped ones of exactly one round.
@pytest.mark.parametrize("form,M,K,layers", [("split", 100, 6400, 6), ("split", 128, 6528, 6), ("whole", 9500, 288, 10), ("grouped", 4600, 1024, 8)])
def test_chain_through_the_other_forms_of_the_tile_gemm(form, M, K, layers):
    """These start early behind the quantiser and behind each other too, and let the next kernel start: same chain, same bits."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    scale = torch.rand(K, generator=g, device="cuda") / (0.577 * 74 * K ** 0.5)
    if form == "grouped":
        W = torch.randint(-128, 128, (4, K, K), dtype=torch.int8, generator=g, device="cuda")
        kernel = q.grouped_quant_gemm((M // 3, 0, M - M // 3 - 7, 7), K, K, out_dtype="bfloat16")
        meta, scales = kernel.block_metadata("cuda"), scale.expand(4, K).contiguous()
        product = lambda a, sa: (kernel(a, W, meta, scales, sa),)
    else:
        W = torch.randint(-128, 128, (K, K), dtype=torch.int8, generator=g, device="cuda")
        product = lambda a, sa: q.quant_matmul(a, W, scale, scale_a=sa, out_dtype="bfloat16", return_accumulators=True) if form == "split" \
            else (q.quant_matmul(a, W, scale, scale_a=sa, out_dtype="bfloat16"),)

    def chain(drain):
        step = torch.cuda.synchronize if drain else lambda: None
        h, first = (x,), (x,)
        for i in range(layers):
            a, sa = q.act_quant(h[0])
            step()
            if i % 2:
                first = product(a, sa.view(-1))
                step()
            h = product(a, sa.view(-1))
            step()
        return (*h, *first)

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(u, v) for u, v in zip(chain(False), want))
    assert torch.isfinite(want[0].float()).all() and want[0].float().abs().max() > 0.1


# one, two, four and eight chunks of eight per thread; rows shared by 32 .. 1024 threads, full and one chunk over; the last number of
# rows that is spread on 148 SMs (rows x threads <= 1100 x 148), and the next
@pytest.mark.parametrize("M,N", [(3, 256), (3, 264), (318, 4096), (317, 4104), (5, 4096), (5, 4104), (158, 8192), (159, 8192), (159, 8200),
                                 (160, 8200), (7, 16384), (7, 16392), (636, 2048), (637, 2048), (1271, 2056), (1273, 2056), (5089, 256),
                                 (5088, 512), (5089, 512), (317, 4096), (635, 2048), (158, 8200), (635, 2056), (636, 2056), (5087, 512), (5087, 256),
                                 (5088, 256), (317, 8192), (318, 8192)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("round_scale", [False, True])
def test_threads_per_row(M, N, dt, round_scale):
    g = torch.Generator().manual_seed(M + N)
    x = torch.randn(M, N, generator=g).to(dt)
    x[M // 2] = 0
    x[M - 1, N - 1] = 60.0
    y, s = q.act_quant(x.cuda(), round_scale)
    y_ref, s_ref = oc.act_quant_torch_ref(x, round_scale)
    assert torch.equal(y.cpu(), y_ref) and torch.equal(s.cpu().view(-1), s_ref.view(-1))
