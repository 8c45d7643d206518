"""GPU parity tests for the W8A8 path: CUDA kernels (through libqgemm.so) against the CPU oracle.

Bars (from the reference's own checks): int32 accumulators bit-exact
(examples/dequantize_gemm/example_dequant_gemm_fine_grained.py:373-374), fp16/bf16 outputs within
rtol = atol = 1e-2 (examples/quant_batch_matmul/example_quant_batch_matmul.py:116).  Because the
epilogue is one fp32 multiply per scale after an exact integer sum, outputs are also compared bit for bit.
"""
import pytest
import torch

from oracle import qgemm_oracle as oc

pytestmark = pytest.mark.gpu


def _q():
    import tilelang_ascend_b200 as q
    return q


def _cmp(C, ref, exact=True):
    torch.testing.assert_close(C.cpu().float(), ref.float(), rtol=1e-2, atol=1e-2)
    if exact:
        assert torch.equal(C.cpu(), ref), f"not bit-exact: {(C.cpu() != ref).sum().item()} of {ref.numel()} differ"


@pytest.mark.parametrize("name,odt", [("w8a8_b_s1_f16", "float16"), ("w8a8_b_sN_bf16", "bfloat16"),
                                      ("w8a8_u_s1_bf16", "bfloat16"), ("w8a8_u_sN_f16", "float16")])
def test_golden_vectors(golden, name, odt):
    """Reference-produced vectors (its check_case recipe: randint(-128, 127), scale = randn)."""
    q = _q()
    c = golden.case(name, bf16=("C",) if odt == "bfloat16" else ())
    A, B, s = c["A"].cuda(), c["B"].cuda(), c["scale"].cuda()
    if A.dim() == 3:
        k = q.simple_quant_batch_matmul(A.shape[0], A.shape[1], B.shape[2], A.shape[2], "N" if s.numel() > 1 else "1",
                                        128, 256, 64, out_dtype=odt)
    else:
        k = q.simple_quant_matmul(A.shape[0], B.shape[1], A.shape[1], "N" if s.numel() > 1 else 1, 128, 256, 64,
                                  out_dtype=odt)
    _cmp(k(A, B, s), c["C"])


def test_two_scale_golden_nk_layout(golden):
    """examples/deepseek_v4/int8_gemm.py golden: B stored [N, K], per-token and per-channel scales."""
    q = _q()
    c = golden.case("w8a8_two_scale_bf16", bf16=("C",))
    C = q.quant_matmul(c["A"].cuda(), c["B_nk"].cuda(), c["scale_b"].squeeze(1).contiguous().cuda(),
                       scale_a=c["scale_a"].squeeze(1).contiguous().cuda(), out_dtype=torch.bfloat16, b_layout="NK")
    torch.testing.assert_close(C.cpu().float(), c["C"].float(), rtol=1e-2, atol=1e-2)
    ref = oc.quant_matmul_ref(c["A"], c["B_nk"].t().contiguous(), c["scale_b"].squeeze(1), "bfloat16",
                              scale_a=c["scale_a"].squeeze(1))
    assert torch.equal(C.cpu(), ref)


SHAPES = [
    # batch (0 = unbatched), M, K, N
    (0, 128, 128, 128),
    (0, 128, 128, 256),
    (0, 1, 16, 16),
    (0, 7, 48, 80),
    (0, 129, 272, 400),
    (0, 300, 1040, 528),
    (3, 65, 144, 272),
    (2, 256, 2048, 1024),
    (0, 1024, 1024, 1024),
    (8, 1024, 1024, 1024),  # the reference example's default case (example_quant_batch_matmul.py:120-133)
    (20, 300, 272, 528),    # enough 256 x 256 tiles for the two-CTA kernel, ragged in M, N and K
    (0, 2304, 528, 2320),
]


@pytest.mark.parametrize("batch,M,K,N", SHAPES)
@pytest.mark.parametrize("odt", ["float16", "bfloat16"])
def test_accumulators_and_output_exact(batch, M, K, N, odt):
    q = _q()
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=batch * 7 + M)
    ref, acc_ref = oc.quant_matmul_ref(A, B, sb, odt, scale_a=sa, return_acc=True)
    C, acc = q.quant_matmul(A.cuda(), B.cuda(), sb.cuda(), scale_a=sa.cuda(), out_dtype=odt, return_accumulators=True)
    assert torch.equal(acc.cpu(), acc_ref), "int32 accumulators differ"
    _cmp(C, ref)


@pytest.mark.parametrize("batch,M,K,N", [(0, 96, 160, 144), (2, 130, 512, 272), (0, 512, 4096, 256), (24, 260, 144, 528)])
def test_nk_layout_and_int32_output(batch, M, K, N):
    q = _q()
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=5)
    acc_ref = oc.int_matmul_exact(A, B)
    B_nk = B.transpose(-1, -2).contiguous()
    acc = q.quant_matmul(A.cuda(), B_nk.cuda(), None, out_dtype=torch.int32, b_layout="NK")
    assert torch.equal(acc.cpu(), acc_ref)
    acc2 = q.quant_matmul(A.cuda(), B.cuda(), None, out_dtype=torch.int32)
    assert torch.equal(acc2.cpu(), acc_ref)


def test_single_scale_and_shared_scales():
    q = _q()
    A, B, sa, sb = oc.make_w8a8_inputs(4, 100, 256, 208, seed=11)
    one = sb[0, :1].contiguous()
    ref = oc.quant_matmul_ref(A, B, one, "float16")
    _cmp(q.quant_matmul(A.cuda(), B.cuda(), one.cuda()), ref)
    shared = sb[0].contiguous()
    ref = oc.quant_matmul_ref(A, B, shared, "bfloat16", scale_a=sa[0].contiguous())
    _cmp(q.quant_matmul(A.cuda(), B.cuda(), shared.cuda(), scale_a=sa[0].contiguous().cuda(), out_dtype="bfloat16"), ref)


def test_extreme_values_large_k():
    """All operands at -128 with K = 4096: accumulators reach 2**26 and the int32 -> fp32 conversion rounds."""
    q = _q()
    M, K, N = 130, 4096, 144
    A = torch.full((M, K), -128, dtype=torch.int8)
    B = torch.full((K, N), -128, dtype=torch.int8)
    B[::3] = 127
    s = torch.full((N,), 1e-4)
    ref, acc_ref = oc.quant_matmul_ref(A, B, s, "float16", return_acc=True)
    C, acc = q.quant_matmul(A.cuda(), B.cuda(), s.cuda(), return_accumulators=True)
    assert torch.equal(acc.cpu(), acc_ref)
    _cmp(C, ref)


def test_config1_and_reference_recipe():
    """BASELINE config 1 (1 x 256 x 1024 x 1024 -> fp16) and the reference's own input recipe on it."""
    q = _q()
    A, B, sa, sb = oc.make_config_inputs("cfg1")
    ref = oc.quant_matmul_ref(A, B, sb, "float16", scale_a=sa)
    k = q.simple_quant_batch_matmul(1, 256, 1024, 1024, "N", 128, 256, 64)
    _cmp(k(A.cuda(), B.cuda(), sb.cuda(), sa.cuda()), ref)
    torch.manual_seed(0)
    A = torch.randint(-128, 127, [1, 256, 1024], dtype=torch.int8)
    B = torch.randint(-128, 127, [1, 1024, 1024], dtype=torch.int8)
    scale = torch.randn([1024])
    _cmp(k(A.cuda(), B.cuda(), scale.cuda()), oc.quant_matmul_ref(A, B, scale, "float16"))


def test_config4_batched_full_size():
    """BASELINE config 4 (16 x 512 x 7168 x 2048 -> bf16), full size, accumulators bit-exact."""
    q = _q()
    A, B, sa, sb = oc.make_config_inputs("cfg4")
    ref, acc_ref = oc.quant_matmul_ref(A, B, sb, "bfloat16", scale_a=sa, return_acc=True)
    C, acc = q.quant_matmul(A.cuda(), B.cuda(), sb.cuda(), scale_a=sa.cuda(), out_dtype="bfloat16",
                            return_accumulators=True)
    assert torch.equal(acc.cpu(), acc_ref)
    _cmp(C, ref)


def test_config3_full_size_properties():
    """BASELINE config 3 (4096 x 4096 x 14336 -> bf16) at full size: exact on a band of rows and columns
    against the oracle, plus size-independent properties over the whole output (linearity in A:
    acc(A1) + acc(A2) == acc(A1 + A2) for operands that do not overflow int8; a checksum of columns)."""
    q = _q()
    A, B, sa, sb = oc.make_config_inputs("cfg3")
    Ad, Bd = A.cuda(), B.cuda()
    C, acc = q.quant_matmul(Ad, Bd, sb.cuda(), scale_a=sa.cuda(), out_dtype="bfloat16", return_accumulators=True)
    rows = torch.cat([torch.arange(0, 160), torch.arange(2000, 2100), torch.arange(4000, 4096)])
    ref, acc_ref = oc.quant_matmul_ref(A[rows], B, sb, "bfloat16", scale_a=sa[rows], return_acc=True)
    assert torch.equal(acc[rows.cuda()].cpu(), acc_ref)
    assert torch.equal(C[rows.cuda()].cpu(), ref)
    # column checksum: sum_n acc[m, n] == A[m, :] . (sum_n B[:, n])   (int64, exact)
    colsum = B.to(torch.int64).sum(dim=1)
    want = (A.to(torch.int64) * colsum[None, :]).sum(dim=1)
    assert torch.equal(acc.to(torch.int64).sum(dim=1).cpu(), want)
    # linearity: halves of A (arithmetic shift keeps them in range) recombine exactly
    A1 = (A >> 1)
    A2 = A - A1
    acc1 = q.quant_matmul(A1.cuda(), Bd, None, out_dtype=torch.int32)
    acc2 = q.quant_matmul(A2.cuda(), Bd, None, out_dtype=torch.int32)
    assert torch.equal(acc1 + acc2, acc)


# (with accumulators; without them the few-token form takes these shapes)
SPLITK_SHAPES = [(0, 256, 6400, 1024), (2, 200, 6416, 528), (0, 130, 7168, 272), (3, 256, 6544, 1024), (0, 200, 6288, 2064),
                 (2, 300, 7296, 1040), (0, 129, 8192, 144)]
# too short a K, or too many tiles
UNSPLIT_SHAPES = [(0, 256, 4096, 1024), (2, 200, 4224, 528), (3, 256, 4608, 1024), (0, 200, 4112, 2064), (2, 300, 4096, 1040),
                  (0, 256, 6272, 1024), (2, 300, 6400, 1680)]


@pytest.mark.parametrize("batch,M,K,N", SPLITK_SHAPES + UNSPLIT_SHAPES)
def test_k_split_over_cta_pairs_is_exact(batch, M, K, N):
    """Few tiles and a long K: the kernel runs in clusters of two CTAs that each accumulate half of K and exchange
    halves of the tile through distributed shared memory, for weights [K, N] and at least 50 k blocks.  Ragged M, N and K, even
    and odd numbers of k blocks, batches, shapes on the other side of the rule, and [N, K] weights, whose K is never cut:
    accumulators and outputs bit-exact against the oracle."""
    q = _q()
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=M + K)
    ref, acc_ref = oc.quant_matmul_ref(A, B, sb, "bfloat16", scale_a=sa, return_acc=True)
    C, acc = q.quant_matmul(A.cuda(), B.cuda(), sb.cuda(), scale_a=sa.cuda(), out_dtype="bfloat16", return_accumulators=True)
    assert torch.equal(acc.cpu(), acc_ref) and torch.equal(C.cpu(), ref)
    assert torch.equal(q.quant_matmul(A.cuda(), B.cuda(), sb.cuda(), scale_a=sa.cuda(), out_dtype="bfloat16").cpu(), ref)
    acc2 = q.quant_matmul(A.cuda(), B.transpose(-1, -2).contiguous().cuda(), None, out_dtype=torch.int32, b_layout="NK")
    assert torch.equal(acc2.cpu(), acc_ref)


def test_k_split_and_unsplit_kernels_give_the_same_bits():
    """The same shapes with the K split switched off (QGEMM_W8_SPLITK=0 is read once per process, hence a child
    process): the accumulators keep all of them off the few-token form, so that unsplit tiles take the split ones'
    place, with identical results."""
    import os
    import subprocess
    import sys
    code = r"""
import torch
from oracle import qgemm_oracle as oc
import tilelang_ascend_b200 as q
for batch, M, K, N in %r:
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=M + K)
    ref, acc_ref = oc.quant_matmul_ref(A, B, sb, "bfloat16", scale_a=sa, return_acc=True)
    C, acc = q.quant_matmul(A.cuda(), B.cuda(), sb.cuda(), scale_a=sa.cuda(), out_dtype="bfloat16", return_accumulators=True)
    assert torch.equal(C.cpu(), ref) and torch.equal(acc.cpu(), acc_ref), (batch, M, K, N)
print("unsplit ok")
""" % (SPLITK_SHAPES,)
    env = dict(os.environ, QGEMM_W8_SPLITK="0")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "unsplit ok" in r.stdout, r.stdout + r.stderr


def test_rejects_bad_arguments():
    q = _q()
    k = q.simple_quant_matmul(64, 64, 64, "N", 128, 256, 64)
    A = torch.zeros(64, 64, dtype=torch.int8, device="cuda")
    s = torch.ones(64, device="cuda")
    with pytest.raises(ValueError, match="contiguous"):
        k(A.t(), A, s)
    with pytest.raises(ValueError, match="dtype mismatch"):
        k(A.float(), A, s)
    with pytest.raises(ValueError, match="device mismatch"):
        k(A, A.cpu(), s)
    with pytest.raises(ValueError, match="shape mismatch"):
        k(A[:32].contiguous(), A, s)
    with pytest.raises(q.QGemmError, match="multiples of 16"):
        q.quant_matmul(torch.zeros(8, 24, dtype=torch.int8, device="cuda"),
                       torch.zeros(24, 40, dtype=torch.int8, device="cuda"), torch.ones(40, device="cuda"))
    # the context is still usable after rejected calls
    assert torch.equal(k(A, A, s).cpu(), torch.zeros(64, 64, dtype=torch.float16))


def test_empty_inputs_give_empty_outputs():
    """No rows / no tokens: an empty result, no launch (the reference wrapper allocates the output with torch.empty)."""
    q = _q()
    B = torch.zeros(128, 64, dtype=torch.int8, device="cuda")
    sb = torch.ones(64, device="cuda")
    C = q.quant_matmul(torch.zeros(0, 128, dtype=torch.int8, device="cuda"), B, sb)
    assert C.shape == (0, 64) and C.dtype == torch.float16
    Cb = q.quant_matmul(torch.zeros(0, 5, 128, dtype=torch.int8, device="cuda"), torch.zeros(0, 128, 64, dtype=torch.int8, device="cuda"), sb)
    assert Cb.shape == (0, 5, 64)
    P = torch.zeros(64, 64, dtype=torch.uint8, device="cuda")
    C4 = q.w4a16_gemm(torch.zeros(0, 128, dtype=torch.float16, device="cuda"), P, None)
    assert C4.shape == (0, 64)


@pytest.mark.parametrize("batch,M,K,N", [
    (0, 1, 16, 16),          # one CTA, one ragged block
    (0, 16, 1024, 144),      # K over eight CTAs: shares of four tokens
    (0, 33, 1040, 4112),     # shares that are no multiple of 16, ragged K and N
    (0, 64, 2064, 14336),    # a cluster of two
    (3, 17, 512, 8192),      # one or two CTAs per tile, batched
    (40, 64, 128, 1024),     # more tiles than CTAs fit at once
    (0, 129, 1024, 1040), (0, 512, 256, 1024), (2, 300, 272, 256),  # several token tiles
    (0, 192, 4112, 2064),
    (0, 300, 4112, 272), (2, 260, 2064, 256), (0, 500, 1040, 528),  # ... with K cut over eight or four CTAs
    (0, 112, 1152, 1040), (0, 128, 512, 4112), (3, 96, 2048, 8192),   # on either side of the choice of the form
])
@pytest.mark.parametrize("layout", ["KN", "NK"])
@pytest.mark.parametrize("odt", ["float16", "bfloat16"])
def test_few_tokens_exact(batch, M, K, N, layout, odt):
    """The few-token form at the edges of its token tiles and K cuts: bit-exact (an exact integer sum, then one fp32
    multiplication per scale), with every form of the scales."""
    q = _q()
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=M + K)
    Bd = (B if layout == "KN" else B.transpose(-1, -2).contiguous()).cuda()
    for a, b in ((sa, sb), (None, sb), (sa.reshape(-1)[:M].contiguous(), sb.reshape(-1)[:N].contiguous()),
                 (None, sb.reshape(-1)[:1].contiguous())):
        ref = oc.quant_matmul_ref(A, B, b, odt, scale_a=a)
        C = q.quant_matmul(A.cuda(), Bd, b.cuda(), scale_a=None if a is None else a.cuda(), out_dtype=odt, b_layout=layout)
        _cmp(C, ref)


def test_few_tokens_behind_the_quantiser():
    """The quantiser lets the product behind it start early: a chain in which each step reads what the step in front has
    just written - the activations and, [N, K], the weights - gives what the same chain gives with the device drained
    between the steps."""
    q = _q()
    g = torch.Generator().manual_seed(3)
    X = [torch.randn((48, 2048), generator=g).to(torch.bfloat16).cuda() for _ in range(4)]
    W = [torch.randn((2048, 2048), generator=g).to(torch.bfloat16).cuda() for _ in range(4)]

    def chain(sync):
        x = X[0]
        for i in range(12):
            b, sb = q.act_quant(W[i % 4])
            if sync:
                torch.cuda.synchronize()
            a, sa = q.act_quant(x)
            if sync:
                torch.cuda.synchronize()
            x = q.quant_matmul(a, b, sb.view(-1), scale_a=sa.view(-1), out_dtype="bfloat16", b_layout="NK") * 0.02
            if sync:
                torch.cuda.synchronize()
            y = q.quant_matmul(a, q.act_quant(W[(i + 1) % 4])[0], sb.view(-1), scale_a=sa.view(-1), out_dtype="bfloat16",
                               b_layout="NK")
            if sync:
                torch.cuda.synchronize()
            x = x + y * 0.01
        return x

    ref = chain(True)
    for _ in range(5):
        assert torch.equal(chain(False), ref)


# Tiles of 256 x 256 made by two CTAs: one round of them and two, with the last one cut in half-width items; rows that end in the
# first or in the second CTA's half of a tile, one row into it or with it; columns that end in either CTA's half of B; K with a
# remainder of 16; several problems.
@pytest.mark.parametrize("batch,M,K,N", [(0, 1300, 3072, 2064), (0, 1281, 3088, 2304), (0, 1409, 4096, 2192),
                                         (0, 2200, 3072, 2320), (3, 520, 4112, 2048), (9, 256, 3072, 2320)])
@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_tiles_of_two_ctas_are_exact(batch, M, K, N, layout):
    q = _q()
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=M + N)
    odt = "bfloat16" if layout == "KN" else "float16"
    ref, acc_ref = oc.quant_matmul_ref(A, B, sb, odt, scale_a=sa, return_acc=True)
    Bd = (B if layout == "KN" else B.transpose(-1, -2).contiguous()).cuda()
    C = q.quant_matmul(A.cuda(), Bd, sb.cuda(), scale_a=sa.cuda(), out_dtype=odt, b_layout=layout)
    _cmp(C, ref)
    acc = q.quant_matmul(A.cuda(), Bd, sb.cuda(), out_dtype="int32", b_layout=layout)
    assert torch.equal(acc.cpu(), acc_ref)


@pytest.mark.parametrize("hook,codes", [(1, [3]), (3, [1, 2, 3]), (4, [1, 2, 3])])
@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_tiles_of_two_ctas_give_up_cleanly(layout, hook, codes):
    """Bounded waits of the two-CTA form, made to run out in the safe way in its last pair: the last accumulators are never
    handed over (1), or one of the two CTAs copies nothing while the other one fills its ring (3, 4).  The launch ends by itself,
    without the code of a copy that never landed, and the next call is exact."""
    q = _q()
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    A, B, sa, sb = (t.cuda() for t in oc.make_w8a8_inputs(0, 1300, 3072, 2064, seed=1))
    if layout == "NK":
        B = B.transpose(-1, -2).contiguous()
    want = q.quant_matmul(A, B, sb, scale_a=sa, b_layout=layout)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        lib.qgemm_set_wait_limit_ms(20)
        lib.qgemm_debug_withhold_commit(hook)
        q.quant_matmul(A, B, sb, scale_a=sa, b_layout=layout, status=status)
        torch.cuda.synchronize()  # returns: the kernel gave up by itself
        assert int(status.item()) in codes
    finally:
        lib.qgemm_debug_withhold_commit(0)
        lib.qgemm_set_wait_limit_ms(2000)
    status.zero_()
    assert torch.equal(q.quant_matmul(A, B, sb, scale_a=sa, b_layout=layout, status=status), want)
    assert int(status.item()) == 0


def test_switch_for_tiles_of_two_ctas():
    """QGEMM_W8_PAIR=0 (read once per process, hence a child process): single CTAs make the tiles, so that the test hook of the
    two-CTA form changes nothing, with the same bits."""
    import os
    import subprocess
    import sys
    code = r"""
import torch
from oracle import qgemm_oracle as oc
import tilelang_ascend_b200 as q
from tilelang_ascend_b200 import _lib
_lib.load().qgemm_debug_withhold_commit(1)
for batch, M, K, N in [(0, 1300, 3072, 2064), (3, 520, 4112, 2048)]:
    A, B, sa, sb = oc.make_w8a8_inputs(batch, M, K, N, seed=M + N)
    ref, acc_ref = oc.quant_matmul_ref(A, B, sb, "bfloat16", scale_a=sa, return_acc=True)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    C, acc = q.quant_matmul(A.cuda(), B.cuda(), sb.cuda(), scale_a=sa.cuda(), out_dtype="bfloat16", return_accumulators=True, status=status)
    assert torch.equal(C.cpu(), ref) and torch.equal(acc.cpu(), acc_ref) and int(status.item()) == 0, (batch, M, K, N)
print("single ok")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, QGEMM_W8_PAIR="0"), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "single ok" in r.stdout, r.stdout + r.stderr


# On 148 SMs: one CTA each that fits an SM or shares it; a cut in two from eight k blocks on, in four from six, in eight from 32 and up
# to 14 clusters, and the sizes at either side of each; clusters of four on 136 and 140 SMs; 96 and 208 KB of pipeline, a K that the
# shorter one just holds and one block more, more k blocks than stages, up to 128 tokens, and one token more.
@pytest.mark.parametrize("batch,M,K,N", [
    (0, 32, 896, 9472), (0, 33, 1024, 9472), (0, 17, 1024, 9488), (0, 48, 640, 4352), (0, 16, 768, 4480), (0, 8, 4096, 4352), (0, 40, 2048, 18944),
    (0, 5, 1536, 18960), (0, 24, 4080, 1168), (0, 60, 8192, 1168), (0, 128, 4096, 2048), (0, 12, 4096, 1792), (0, 30, 1024, 8192), (0, 48, 1056, 8192), (0, 16, 640, 9488), (0, 16, 656, 9488), (0, 100, 4112, 1808), (0, 129, 1152, 1040), (3, 72, 4864, 6016),
    (2, 1, 4224, 1024)])
@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_plans_for_few_tokens_are_exact(batch, M, K, N, layout):
    g = torch.Generator(device="cuda").manual_seed(K + M + N)
    lead = (batch,) if batch else ()
    A = torch.randint(-128, 128, lead + (M, K), dtype=torch.int8, generator=g, device="cuda")
    B = torch.randint(-128, 128, lead + ((K, N) if layout == "KN" else (N, K)), dtype=torch.int8, generator=g, device="cuda")
    sb, sa = torch.rand(lead + (N,), generator=g, device="cuda"), torch.rand(lead + (M,), generator=g, device="cuda")
    acc = A.double() @ (B if layout == "KN" else B.transpose(-1, -2)).double()
    want = ((acc.float() * sa.unsqueeze(-1)) * sb.unsqueeze(-2)).to(torch.bfloat16)
    import tilelang_ascend_b200 as q
    assert torch.equal(q.quant_matmul(A, B, sb, scale_a=sa, out_dtype="bfloat16", b_layout=layout), want)


# Tiles of two CTAs at short K, down to fewer k blocks than pipeline stages, and tiles of 128 x 128 or 128 x 256 where these are taken
# instead, on 148 SMs.
@pytest.mark.parametrize("batch,M,K,N", [(0, 3100, 288, 1296), (0, 3100, 400, 3600), (0, 1300, 640, 2320), (0, 2310, 1024, 2576),
                                         (12, 640, 672, 560), (0, 169, 800, 4400), (0, 602, 2048, 6896), (0, 4096, 16, 2320)])
@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_short_k_is_exact(batch, M, K, N, layout):
    import tilelang_ascend_b200 as q
    g = torch.Generator(device="cuda").manual_seed(K + M + N)
    lead = (batch,) if batch else ()
    A = torch.randint(-128, 128, lead + (M, K), dtype=torch.int8, generator=g, device="cuda")
    B = torch.randint(-128, 128, lead + ((K, N) if layout == "KN" else (N, K)), dtype=torch.int8, generator=g, device="cuda")
    sb, sa = torch.rand(lead + (N,), generator=g, device="cuda"), torch.rand(lead + (M,), generator=g, device="cuda")
    acc = (A.double() @ (B if layout == "KN" else B.transpose(-1, -2)).double()).float()  # below 2^24: exact
    C = q.quant_matmul(A, B, sb, scale_a=sa, out_dtype="float16", b_layout=layout)
    assert torch.equal(C, ((acc * sa.unsqueeze(-1)) * sb.unsqueeze(-2)).to(torch.float16))


# K cut over two CTAs: at least 50 k blocks, weights [K, N], accumulators wanted.  Ragged M, N and K, and beyond the limits: too short a
# K, too many tiles, weights [N, K].
@pytest.mark.parametrize("batch,M,K,N", [(0, 256, 6400, 1024), (2, 200, 6416, 528), (0, 130, 8192, 2064), (3, 256, 6272, 1024), (0, 1100, 6544, 1040)])
@pytest.mark.parametrize("layout", ["KN", "NK"])
def test_long_k_of_few_tiles_is_exact(batch, M, K, N, layout):
    import tilelang_ascend_b200 as q
    g = torch.Generator(device="cuda").manual_seed(K + M + N)
    lead = (batch,) if batch else ()
    A = torch.randint(-128, 128, lead + (M, K), dtype=torch.int8, generator=g, device="cuda")
    B = torch.randint(-128, 128, lead + ((K, N) if layout == "KN" else (N, K)), dtype=torch.int8, generator=g, device="cuda")
    sb, sa = torch.rand(lead + (N,), generator=g, device="cuda"), torch.rand(lead + (M,), generator=g, device="cuda")
    want = A.double() @ (B if layout == "KN" else B.transpose(-1, -2)).double()
    C, acc = q.quant_matmul(A, B, sb, scale_a=sa, out_dtype="float16", b_layout=layout, return_accumulators=True)
    assert torch.equal(acc.double(), want)
    assert torch.equal(C, ((want.float() * sa.unsqueeze(-1)) * sb.unsqueeze(-2)).to(torch.float16))
