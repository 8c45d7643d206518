"""GPU parity tests for the W4A16 / W4A8 paths: CUDA kernels (through libqgemm.so) against the CPU oracle.

Bars: fp16/bf16 outputs within rtol = atol = 1e-2
(examples/dequantize_gemm/example_dequant_gemm_fine_grained.py:341-344); int32 outputs exact (:373-374,
examples/dequantize_gemm/example_dequant_gemm_w4a8.py:182).  The kernel accumulates exact f16 x f16
products in fp32 in a different order than the CPU matmul, so float results are close, not identical.
"""
import pytest
import torch

from oracle import qgemm_oracle as oc

pytestmark = pytest.mark.gpu


def _q():
    import tilelang_ascend_b200 as q
    return q


def _close(C, ref):
    assert C.dtype == ref.dtype
    torch.testing.assert_close(C.cpu().float(), ref.float(), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("name,dt", [("dq_f16", "float16"), ("dq_bf16", "bfloat16")])
def test_golden_unscaled(golden, name, dt):
    """Reference-produced vectors of ref_program_fp16 (unsigned nibbles, no scale, no zero point)."""
    q = _q()
    bf = ("A", "C") if dt == "bfloat16" else ()
    c = golden.case(name, bf16=bf)
    M, K = c["A"].shape
    N = c["packed"].shape[0]
    if K % 32 != 0 or N % 8 != 0:
        pytest.skip("shape below the kernel's granularity")
    w = q.dequant_gemm_fp16_wrapper(M, N, K, 128, 256, 64, dt, dt)
    C = w(c["A"], c["packed"])  # CPU in -> CPU out, like the reference wrapper
    assert not C.is_cuda
    _close(C, c["C"])


def test_reference_known_answer_through_kernel():
    """The reference's nibble-order vector [[0x12, 0x34]] -> [2, 1, 4, 3], observed through the GEMM:
    with A = identity rows the output row m is column m of the unpacked weights."""
    q = _q()
    K, N = 32, 8
    packed = torch.zeros(N, K // 2, dtype=torch.uint8)
    packed[0, 0], packed[0, 1] = 0x12, 0x34
    A = torch.eye(K, dtype=torch.float16)[:4]
    C = q.w4a16_gemm(A.cuda(), packed.cuda()).cpu()
    assert C[:, 0].tolist() == [2.0, 1.0, 4.0, 3.0]
    assert torch.equal(C.float(), oc.unpack_uint4(packed).float().t()[:4])


W4_SHAPES = [
    # M, K, N, group
    (16, 256, 128, 128),
    (1, 32, 8, 32),
    (5, 96, 40, 32),
    (16, 1024, 256, 128),
    (8, 4096, 512, 128),
    (33, 640, 264, 64),
    (64, 2048, 384, 128),
    (100, 512, 136, 256),
    (256, 1024, 256, 128),
    (300, 768, 520, -1),
    # two blocks of 128 tokens per tile (above 128 tokens): ragged second block, odd and even block counts, split K
    (130, 512, 272, 128),
    (200, 2048, 136, 32),
    (513, 1024, 264, 64),
    (640, 4096, 384, 128),
]


@pytest.mark.parametrize("M,K,N,group", W4_SHAPES)
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_scaled_against_oracle(M, K, N, group, dt):
    q = _q()
    g = K if group == -1 else group
    A, packed, scales = oc.make_w4a16_inputs(M, K, N, dt, g, seed=M + N)
    ref = oc.dequant_gemm_fp16_ref(A, packed, dt, scales, 8, g)
    C = q.w4a16_gemm(A.cuda(), packed.cuda(), scales.cuda(), 8, group)
    _close(C, ref)
    # a second, tighter bar than the reference's: error relative to the output scale
    err = (C.cpu().float() - ref.float()).abs().max().item()
    assert err <= 2e-2 * max(1.0, ref.float().abs().max().item()) * (1 if dt == "float16" else 4)


@pytest.mark.parametrize("M,K,N", [(16, 512, 128), (256, 256, 256), (512, 512, 512)])
def test_unscaled_reference_semantics(M, K, N):
    """scales=None: raw unsigned nibble values, exactly the reference example (its 256^3 / 512^3 ladder)."""
    q = _q()
    g = torch.Generator().manual_seed(0)
    A = torch.randn(M, K, generator=g).half()
    packed = torch.randint(0, 255, (N, K // 2), dtype=torch.uint8, generator=g)
    w = q.dequant_gemm_fp16_wrapper(M, N, K, 128, 256, 64)
    C = w(A.cuda(), packed.cuda())
    assert C.is_cuda
    _close(C, oc.dequant_gemm_fp16_ref(A, packed, "float16"))


def test_dequant_is_exact_via_identity_activations():
    """With A = I (K x K) the GEMM returns W^T: every dequantised weight must equal the oracle's fp16 value
    bit for bit ((q - 8) is exact, the product with the scale rounds once)."""
    q = _q()
    K, N = 256, 136
    _, packed, scales = oc.make_w4a16_inputs(1, K, N, "float16", 128, seed=3)
    A = torch.eye(K, dtype=torch.float16)
    C = q.w4a16_gemm(A.cuda(), packed.cuda(), scales.cuda(), 8, 128).cpu()
    W = oc.dequant_weight_ref(packed, scales, 8, 128)  # [N, K]
    assert torch.equal(C, W.t())
    for zero in (0, 3, 15):
        C = q.w4a16_gemm(A.cuda(), packed.cuda(), scales.cuda(), zero, 128).cpu()
        assert torch.equal(C, oc.dequant_weight_ref(packed, scales, zero, 128).t())


def test_split_k_is_deterministic_and_counters_stay_clean():
    q = _q()
    A, packed, scales = oc.make_config_inputs("cfg2")
    Ad, Pd, Sd = A.cuda(), packed.cuda(), scales.cuda()
    ref = oc.dequant_gemm_fp16_ref(A, packed, "float16", scales, 8, 128)
    outs = [q.w4a16_gemm(Ad, Pd, Sd, 8, 128) for _ in range(5)]
    _close(outs[0], ref)
    for o in outs[1:]:
        assert torch.equal(o, outs[0])


@pytest.mark.parametrize("batch,M,K,N,dt", [(3, 5, 512, 264, "float16"), (4, 16, 1024, 256, "bfloat16"),
                                             (2, 70, 256, 384, "float16"), (6, 1, 2048, 128, "bfloat16")])
def test_batched_matches_oracle_and_single_calls(batch, M, K, N, dt):
    """Independent problems of one shape in one launch: every batch entry must match the oracle and the
    same problem launched on its own (identical arithmetic per element, possibly another fp32 split order)."""
    q = _q()
    ins = [oc.make_w4a16_inputs(M, K, N, dt, 128, seed=100 + b) for b in range(batch)]
    A = torch.stack([i[0] for i in ins]).cuda()
    P = torch.stack([i[1] for i in ins]).cuda()
    S = torch.stack([i[2] for i in ins]).cuda()
    C = q.w4a16_gemm(A, P, S, 8, 128)
    assert C.shape == (batch, M, N)
    for b in range(batch):
        ref = oc.dequant_gemm_fp16_ref(ins[b][0], ins[b][1], dt, ins[b][2], 8, 128)
        _close(C[b], ref)
        single = q.w4a16_gemm(A[b].contiguous(), P[b].contiguous(), S[b].contiguous(), 8, 128)
        torch.testing.assert_close(C[b].float(), single.float(), rtol=2e-3, atol=2e-3)
    C2 = q.w4a16_gemm(A, P, None)  # unscaled, batched
    for b in range(batch):
        _close(C2[b], oc.dequant_gemm_fp16_ref(ins[b][0], ins[b][1], dt))


@pytest.mark.parametrize("M", [1, 8, 64])
def test_config5_decode_full_size(M):
    """BASELINE config 5 decode shapes at full size (K = 8192, N = 28672, bf16): a band of output columns
    against the oracle plus linearity in A over the whole output (f(A) + f(2A) == f(3A) up to rounding)."""
    q = _q()
    A, packed, scales = oc.make_config_inputs("cfg5", M=M)
    Ad, Pd, Sd = A.cuda(), packed.cuda(), scales.cuda()
    C = q.w4a16_gemm(Ad, Pd, Sd, 8, 128)
    cols = torch.cat([torch.arange(0, 256), torch.arange(14000, 14200), torch.arange(28672 - 200, 28672)])
    ref = oc.dequant_gemm_fp16_ref(A, packed[cols], "bfloat16", scales[:, cols].contiguous(), 8, 128)
    _close(C[:, cols.cuda()], ref)
    C2 = q.w4a16_gemm((Ad * 2), Pd, Sd, 8, 128)
    torch.testing.assert_close(C2.float(), C.float() * 2, rtol=1e-2, atol=1e-2)  # exact power-of-two scaling in fp32
    assert torch.isfinite(C.float()).all()


def test_config5_prefill_m512_band():
    q = _q()
    A, packed, scales = oc.make_config_inputs("cfg5", M=512)
    C = q.w4a16_gemm(A.cuda(), packed.cuda(), scales.cuda(), 8, 128)
    cols = torch.cat([torch.arange(0, 128), torch.arange(20000, 20128)])
    ref = oc.dequant_gemm_fp16_ref(A, packed[cols], "bfloat16", scales[:, cols].contiguous(), 8, 128)
    _close(C[:, cols.cuda()], ref)


@pytest.mark.parametrize("M,N,K", [(64, 64, 256), (128, 128, 512), (256, 256, 1024)])
def test_w4a8_signed_exact(M, N, K):
    """The reference's three W4A8 levels (example_dequant_gemm_w4a8.py:202-208), exact int32."""
    q = _q()
    g = torch.Generator().manual_seed(42)
    A = torch.randint(-8, 8, (M, K), dtype=torch.int8, generator=g)
    Bi = torch.randint(-8, 8, (N, K), dtype=torch.int8, generator=g)
    qB = oc.pack_int4_signed(Bi)
    kernel = q.w4a8_gemm_cv(M, N, K)
    ws = torch.zeros(N, K, dtype=torch.int8, device="cuda")
    C = torch.zeros(M, N, dtype=torch.int32, device="cuda")
    out = kernel(A.cuda(), qB.cuda(), ws, C)
    assert torch.equal(ws.cpu(), Bi)
    assert torch.equal(out.cpu(), oc.w4a8_gemm_ref(A, qB))


def test_w4a8_golden(golden):
    q = _q()
    c = golden.case("w4a8")
    M, K = c["A"].shape
    N = c["qB"].shape[0]
    ws = torch.zeros(N, K, dtype=torch.int8, device="cuda")
    C = torch.zeros(M, N, dtype=torch.int32, device="cuda")
    q.w4a8_gemm_cv(M, N, K)(c["A"].cuda(), c["qB"].cuda(), ws, C)
    assert torch.equal(ws.cpu(), c["conv"])
    assert torch.equal(C.cpu(), c["C_nm"].t())


@pytest.mark.parametrize("M,N,K,odt", [(256, 256, 256, "int32"), (512, 512, 512, "int32"), (512, 512, 512, "float16")])
def test_int8_mode_unsigned_exact(M, N, K, odt):
    """dequant_gemm_int8_wrapper ladder (example_dequant_gemm_fine_grained.py:459-469)."""
    q = _q()
    g = torch.Generator().manual_seed(0)
    A = torch.randint(-128, 127, (M, K), dtype=torch.int8, generator=g)
    packed = torch.randint(0, 255, (N, K // 2), dtype=torch.uint8, generator=g)
    C = q.dequant_gemm_int8_wrapper(M, N, K, 128, 128, 64, odt)(A, packed)
    ref = oc.dequant_gemm_int8_ref(A, packed, odt)
    if odt == "int32":
        assert torch.equal(C, ref)
    else:
        torch.testing.assert_close(C, ref, rtol=1e-2, atol=1e-2)


def test_unpack_kernel_matches_oracle_on_ragged_sizes():
    q = _q()
    g = torch.Generator().manual_seed(1)
    for N, K in [(1, 2), (3, 34), (17, 96), (64, 1000)]:
        packed = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g)
        assert torch.equal(q.unpack_int4(packed.cuda()).cpu(), oc.unpack_uint4(packed).to(torch.int8))
        assert torch.equal(q.unpack_int4(packed.cuda(), signed=True).cpu(), oc.unpack_int4_signed(packed))


def test_rejects_bad_arguments():
    q = _q()
    A = torch.zeros(4, 64, dtype=torch.float16, device="cuda")
    P = torch.zeros(16, 32, dtype=torch.uint8, device="cuda")
    with pytest.raises(ValueError, match="dtype mismatch"):
        q.w4a16_gemm(A.float(), P)
    with pytest.raises(ValueError, match="shape mismatch"):
        q.w4a16_gemm(A, P[:, :16].contiguous())
    with pytest.raises(q.QGemmError, match="multiple of 32"):
        q.w4a16_gemm(A[:, :48].contiguous(), P[:, :24].contiguous())
    with pytest.raises(q.QGemmError, match="group"):
        q.w4a16_gemm(A, P, torch.ones(4, 16, dtype=torch.float16, device="cuda"), 8, 16)
    assert torch.equal(q.w4a16_gemm(A, P).cpu(), torch.zeros(4, 16, dtype=torch.float16))


@pytest.mark.parametrize("M,K,N,dt,group", [
    (17, 256, 128, "float16", 128), (40, 512, 272, "bfloat16", 64), (200, 1024, 528, "float16", 32),
    (130, 768, 2320, "bfloat16", 256), (300, 512, 144, "float16", 512), (129, 2048, 1024, "bfloat16", 128)])
def test_small_ragged_shapes_scaled_and_unscaled(M, K, N, dt, group):
    """Every group size on small ragged shapes (up to 64 tokens with wide groups the group-sum kernel, otherwise wide
    tiles, whole or cut along K), with scales and with the raw nibble values."""
    q = _q()
    A, P, S = oc.make_w4a16_inputs(M, K, N, dt, group, seed=M + K)
    _close(q.w4a16_gemm(A.cuda(), P.cuda(), S.cuda(), 8, group), oc.dequant_gemm_fp16_ref(A, P, dt, S, 8, group))
    _close(q.w4a16_gemm(A.cuda(), P.cuda(), None), oc.dequant_gemm_fp16_ref(A, P, dt))


def test_wide_tiles_read_dequantised_weights_back_exactly():
    """Unit activations, 256 tokens: half(q - zero) * s bit for bit with groups of 64."""
    q = _q()
    K, N, group = 256, 144, 64
    _, P, S = oc.make_w4a16_inputs(1, K, N, "float16", group, seed=3)
    W = q.w4a16_gemm(torch.eye(K, dtype=torch.float16).cuda(), P.cuda(), S.cuda(), 8, group)  # [K, N], transposed
    assert torch.equal(W.cpu().t().contiguous(), oc.dequant_weight_ref(P, S, 8, group).half())


@pytest.mark.parametrize("M", [48, 100])
def test_batched_ragged(M):
    q = _q()
    ins = [oc.make_w4a16_inputs(M, 512, 272, "float16", 128, seed=s) for s in range(3)]
    A, P, S = [torch.stack([x[i] for x in ins]).cuda() for i in range(3)]
    C = q.w4a16_gemm(A, P, S, 8, 128)
    for b in range(3):
        _close(C[b], oc.dequant_gemm_fp16_ref(ins[b][0], ins[b][1], "float16", ins[b][2], 8, 128))


def test_config5_prefill_m4096_band_and_linearity():
    """Config 5 at 4096 tokens, on wide tiles of 256 tokens: bands of output columns against the oracle, and f(2A) == 2 f(A)
    over the whole output."""
    q = _q()
    A, packed, scales = oc.make_config_inputs("cfg5", M=4096)
    Ad, Pd, Sd = A.cuda(), packed.cuda(), scales.cuda()
    C = q.w4a16_gemm(Ad, Pd, Sd, 8, 128)
    cols = torch.cat([torch.arange(0, 64), torch.arange(20000, 20064), torch.arange(28672 - 64, 28672)])
    ref = oc.dequant_gemm_fp16_ref(A, packed[cols], "bfloat16", scales[:, cols].contiguous(), 8, 128)
    _close(C[:, cols.cuda()], ref)
    C2 = q.w4a16_gemm(Ad * 2, Pd, Sd, 8, 128)
    torch.testing.assert_close(C2.float(), C.float() * 2, rtol=1e-2, atol=1e-2)


def _cfg5_column_sum_of_weights(packed, scales, zero=8, group=128):
    """sum over n of the dequantised weights W[n, k] = half(q - zero) * s[k / g, n], in float64, group by group."""
    N, K = packed.shape[0], packed.shape[1] * 2
    q = oc.unpack_uint4(packed).to(torch.float32)  # [N, K]
    wsum = torch.empty(K, dtype=torch.float64)
    for g in range(K // group):
        w = ((q[:, g * group:(g + 1) * group] - zero).half() * scales[g, :, None]).double()  # one f16 rounding, as the operator's contract says
        wsum[g * group:(g + 1) * group] = w.sum(dim=0)
    return wsum


@pytest.fixture(scope="module")
def cfg5_weights():
    _, packed, scales = oc.make_config_inputs("cfg5", M=1)
    return packed, scales, _cfg5_column_sum_of_weights(packed, scales), packed.cuda(), scales.cuda()


@pytest.mark.parametrize("M", [1, 8, 16, 64, 512, 4096])
def test_config5_whole_output_identity(cfg5_weights, M):
    """An identity every output tile takes part in, at full size: sum_n C[m, n] == A[m, :] . sum_n W[n, :].
    A tile written to the wrong place, left out or added twice (a lost or duplicated split-K hand-over) moves a
    row sum by about sqrt(128) * |C|, far outside the bar, which is the rounding of 28672 bf16 outputs."""
    q = _q()
    packed, scales, wsum, Pd, Sd = cfg5_weights
    A, _, _ = oc.make_config_inputs("cfg5", M=M)
    C = q.w4a16_gemm(A.cuda(), Pd, Sd, 8, 128)
    got = C.double().sum(dim=1).cpu()
    want = A.half().double() @ wsum  # the operator converts bf16 activations to f16 first, as the reference wrapper does
    N = packed.shape[0]
    cmax = C.float().abs().max().item()
    bar = 6.0 * (N ** 0.5) * cmax * 2.0 ** -9 + 1e-3 * want.abs().max().item()
    assert (got - want).abs().max().item() <= bar, ((got - want).abs().max().item(), bar)
    assert torch.isfinite(C.float()).all()


def test_kernels_on_either_side_of_a_switch_agree():
    """Up to 64 tokens the group scale multiplies the group's fp32 sum, above that every weight is scaled in f16
    first: the same token row through both kernels differs by at most that f16 product's rounding, 2^-11
    relative per term - far inside the operator's tolerance, and the bar here."""
    q = _q()
    M, K, N = 65, 2048, 512
    A, packed, scales = oc.make_w4a16_inputs(M, K, N, "float16", 128, seed=11)
    Ad, Pd, Sd = A.cuda(), packed.cuda(), scales.cuda()
    C65 = q.w4a16_gemm(Ad, Pd, Sd, 8, 128)                      # per-weight scale (tcgen05 kernel, 128-token tile)
    C64 = q.w4a16_gemm(Ad[:64].contiguous(), Pd, Sd, 8, 128)    # group-sum kernel, 64-token tile
    C32 = q.w4a16_gemm(Ad[:32].contiguous(), Pd, Sd, 8, 128)    # group-sum kernel, 32-token tile
    C8 = q.w4a16_gemm(Ad[:8].contiguous(), Pd, Sd, 8, 128)      # group-sum kernel, 16-token tile
    ref = oc.dequant_gemm_fp16_ref(A, packed, "float16", scales, 8, 128)
    _close(C65, ref)
    _close(C64, ref[:64])
    # the group-sum kernel does the same arithmetic per row whatever the token count and tile height ...
    assert torch.equal(C32, C64[:32])
    # ... up to the order in which the K ranges of a split tile are added in fp32 (the single-launch form of small
    # problems cuts K over a cluster, the two-launch form over the persistent grid)
    torch.testing.assert_close(C8.float(), C64[:8].float(), rtol=2e-3, atol=2e-3)
    # |sum_k a w (1 + e_k)| with |e_k| <= 2^-11: bounded by 2^-11 * sum |a w|, plus the output's own rounding
    W = oc.dequant_weight_ref(packed, scales, 8, 128).float()
    bound = (A.float().abs() @ W.abs().t()) * 2.0 ** -11 + ref.float().abs() * 2.0 ** -9 + 1e-3
    assert ((C65[:64].float() - C64.float()).abs().cpu() <= bound[:64]).all()


def test_bounded_wait_expires_cleanly_and_the_next_call_is_exact():
    """The time-out path end to end, without faulting or hanging anything: with the test hook on, one
    accumulator hand-over of the launch is never signalled, so one wait of the epilogue runs into its limit
    (20 ms here).  The kernel must return by itself with QGEMM_ST_TIMEOUT_EPILOGUE in the status word, and the
    next ordinary call on the same device must be correct."""
    q = _q()
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    A, packed, scales = oc.make_w4a16_inputs(16, 1024, 256, "float16", 128, seed=5)
    Ad, Pd, Sd = A.cuda(), packed.cuda(), scales.cuda()
    ref = oc.dequant_gemm_fp16_ref(A, packed, "float16", scales, 8, 128)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        lib.qgemm_set_wait_limit_ms(20)
        lib.qgemm_debug_withhold_commit(1)
        q.w4a16_gemm(Ad, Pd, Sd, 8, 128, status=status)
        torch.cuda.synchronize()  # returns: the kernel gave up by itself
        assert int(status.item()) == 3  # QGEMM_ST_TIMEOUT_EPILOGUE
        with pytest.raises(q.QGemmError, match="bounded wait ran out"):
            q.w4a16_gemm(Ad, Pd, Sd, 8, 128, check_status=True)
    finally:
        lib.qgemm_debug_withhold_commit(0)
        lib.qgemm_set_wait_limit_ms(2000)
    status.zero_()
    C = q.w4a16_gemm(Ad, Pd, Sd, 8, 128, status=status)
    _close(C, ref)
    assert int(status.item()) == 0
    C2 = q.w4a16_gemm(Ad, Pd, Sd, 8, 128, check_status=True)
    assert torch.equal(C, C2)


def test_back_to_back_calls_that_feed_each_other():
    """Calls issued back to back overlap: a call's pre-pass is resident and its GEMM kernel is already streaming
    weights while the call in front still runs.  Here every call reads the previous call's output as its
    activations and all calls share one scratch area (the built-in one), so any step taken too early shows: the
    chain must be bit-identical to the same chain with the device drained between calls, and match the oracle."""
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    M, K, layers = 16, 2048, 6
    g = torch.Generator().manual_seed(77)
    A0, _, _ = oc.make_w4a16_inputs(M, K, K, "float16", 128, seed=70)
    Ws = []
    for l in range(layers):
        _, P, S = oc.make_w4a16_inputs(M, K, K, "float16", 128, seed=71 + l)
        # keep the chain's magnitude steady: rescale so that one layer maps unit-variance rows to about unit variance
        W = oc.dequant_weight_ref(P, S, 8, 128).float()
        gain = (torch.randn(64, K, generator=g) @ W.t()).std().item()
        Ws.append((P, (S.float() / gain).to(torch.float16)))
    dev = [(P.cuda(), S.cuda()) for P, S in Ws]
    stream = torch.cuda.current_stream().cuda_stream

    def chain(drain):
        x = A0.cuda()
        outs = []
        for P, S in dev:
            C = torch.empty((M, K), dtype=torch.float16, device="cuda")
            rc = lib.qgemm_w4a16_noalloc(x.data_ptr(), P.data_ptr(), S.data_ptr(), 8, 128, C.data_ptr(), M, K, K,
                                         _lib.DT_F16, _lib.DT_F16, None, stream)
            assert rc == 0, _lib.last_error()
            if drain:
                torch.cuda.synchronize()
            outs.append(C)
            x = C
        torch.cuda.synchronize()
        return outs

    want = chain(drain=True)
    for _ in range(3):
        got = chain(drain=False)
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    x = A0
    for (P, S), c in zip(Ws, want):
        ref = oc.dequant_gemm_fp16_ref(x, P, "float16", S, 8, 128)
        _close(c, ref)
        x = c.cpu()


SMALL_SHAPES = [
    # M, K, N, group, dtype, batch: clusters of 1 (K <= 1024), 2 and 4 CTAs, K beyond the form's range, ragged N, batches
    (16, 1024, 256, 128, "float16", None), (5, 512, 136, 128, "bfloat16", None), (16, 2048, 512, 128, "float16", None),
    (9, 4096, 1024, 128, "bfloat16", None), (16, 4096, 4096, 128, "float16", None), (1, 8192, 2048, 128, "float16", None),
    (16, 8192, 2304, 256, "bfloat16", None), (12, 4096, 264, 4096, "float16", None), (16, 2048, 384, 128, "float16", 3),
]


@pytest.mark.parametrize("M,K,N,group,dt,batch", SMALL_SHAPES)
def test_single_launch_form_of_small_problems(M, K, N, group, dt, batch):
    """Problems of at most four slabs per CTA run as one launch (activations prepared inside the kernel, K cut over a
    thread-block cluster whose CTAs add their sums through distributed shared memory): results against the oracle,
    one-hot rows bit for bit, the interleaved layout identical, and two runs identical."""
    q = _q()
    if batch is None:
        A, P, S = oc.make_w4a16_inputs(M, K, N, dt, group, seed=M + N)
        ref = oc.dequant_gemm_fp16_ref(A, P, dt, S, 8, group)
    else:
        parts = [oc.make_w4a16_inputs(M, K, N, dt, group, seed=40 + i) for i in range(batch)]
        A, P, S = [torch.stack([p[i] for p in parts]) for i in range(3)]
        ref = torch.stack([oc.dequant_gemm_fp16_ref(*p[:2], dt, p[2], 8, group) for p in parts])
    C = q.w4a16_gemm(A.cuda(), P.cuda(), S.cuda(), 8, group)
    _close(C, ref)
    assert torch.equal(C, q.w4a16_gemm(A.cuda(), P.cuda(), S.cuda(), 8, group))
    if batch is None:
        Pi = q.interleave_weight(P, 4, "float16").view(torch.uint8)
        assert torch.equal(C, q.w4a16_gemm(A.cuda(), Pi.cuda(), S.cuda(), 8, group, weight_layout="interleaved"))
        W = oc.dequant_weight_ref(P, S, 8, group)
        for k0 in (0, K // 2 - 3, K - M):
            hot = torch.zeros((M, K), dtype=A.dtype)
            hot[torch.arange(M), k0 + torch.arange(M)] = 1
            Wt = q.w4a16_gemm(hot.cuda(), P.cuda(), S.cuda(), 8, group, out_dtype=torch.float16)
            assert torch.equal(Wt.cpu(), W[:, k0:k0 + M].t().contiguous())


def test_single_launch_form_gives_up_cleanly_when_a_cluster_signal_is_missing():
    """The bounded wait of the single-launch form, made to expire in the safe way: with the test hook at 2, CTA 1 of
    the last cluster writes its sums but keeps its signal back, so the first CTA's wait runs into the limit (20 ms).
    The kernel must return by itself with QGEMM_ST_TIMEOUT_EPILOGUE, and the next ordinary call must be exact."""
    q = _q()
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    A, packed, scales = oc.make_w4a16_inputs(16, 4096, 512, "float16", 128, seed=9)  # four clusters of four CTAs
    Ad, Pd, Sd = A.cuda(), packed.cuda(), scales.cuda()
    ref = oc.dequant_gemm_fp16_ref(A, packed, "float16", scales, 8, 128)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        lib.qgemm_set_wait_limit_ms(20)
        lib.qgemm_debug_withhold_commit(2)
        C_bad = q.w4a16_gemm(Ad, Pd, Sd, 8, 128, status=status)
        torch.cuda.synchronize()  # returns: the kernel gave up by itself
        assert int(status.item()) == 3  # QGEMM_ST_TIMEOUT_EPILOGUE
        # the clusters whose signals all arrived wrote their tiles
        _close(C_bad[:, :384], ref[:, :384])
    finally:
        lib.qgemm_debug_withhold_commit(0)
        lib.qgemm_set_wait_limit_ms(2000)
    status.zero_()
    C = q.w4a16_gemm(Ad, Pd, Sd, 8, 128, status=status)
    _close(C, ref)
    assert int(status.item()) == 0


@pytest.mark.parametrize("M,K,N,zeros", [
    (3, 1024, 256, None),       # one launch, K over a cluster
    (16, 8192, 264, None),      # tiles shared by several CTAs
    (1, 512, 128 * 160, None),  # whole tiles
    (33, 1024, 128 * 150, None), (64, 4096, 144, "tensor"), (20, 2048, 272, "tensor"),
])
@pytest.mark.parametrize("fmt", ["sequential", "interleaved"])
def test_non_finite_activations(M, K, N, zeros, fmt):
    """An infinite activation gives +inf, -inf or (where q == zero) NaN per output feature, and leaves the other rows alone."""
    q = _q()
    A, packed, scales = oc.make_w4a16_inputs(M, K, N, "bfloat16", 128, seed=M + N)
    clean = A.clone()
    A[0, K // 2 + 5] = float("inf")
    A[0, 7] = 1.0e38  # beyond f16: the operator's 16-bit activations make it an infinity
    if M > 2:
        A[M - 1, K - 1] = float("-inf")
        A[M // 2, 3] = float("nan")
    kw = {}
    if zeros == "tensor":
        kw["zeros_mode"] = "quantized"
        z = torch.randint(0, 16, scales.shape, generator=torch.Generator().manual_seed(1)).to(torch.float16)
    else:
        z = 8
    W = (oc.dequant_weight_zeros_ref(packed, scales, z, 128, "quantized") if zeros == "tensor"
         else oc.dequant_weight_ref(packed, scales, 8, 128)).double()
    B = oc.interleave_int4_f16_ref(packed) if fmt == "interleaved" else packed
    if fmt == "interleaved":
        kw["weight_layout"] = "interleaved"
    call = lambda a: q.w4a16_gemm(a.cuda(), B.cuda(), scales.cuda(), z.cuda() if zeros else z, 128, out_dtype="float16", **kw).cpu()
    C, C0 = call(A), call(clean)
    rows = sorted({0} | ({M - 1, M // 2} if M > 2 else set()))
    torch.testing.assert_close(C[rows].double(), A[rows].half().double() @ W.t(), equal_nan=True)  # +-inf and NaN only
    other = [m for m in range(M) if m not in rows]
    assert torch.equal(C[other], C0[other])


@pytest.mark.parametrize("M,K,N,group,zeros", [
    (65, 256, 8, 128, None),        # one tile of 80 tokens, one slab
    (128, 4096, 136, 32, None),     # K cut over CTAs, two accumulators
    (129, 1056, 272, 32, "rescale"),    # K not a multiple of 64
    (256, 8192, 128, 64, None),     # the tallest tile, cut along K
    (257, 512, 128 * 75, 128, None),    # two token tiles, whole tiles and a cut remainder
    (17, 2048, 144, 64, "quantized"), (9, 512, 2064, 128, "original"), (1, 1024, 16, 32, "rescale"),
    (700, 768, 1040, 768, "original"),
])
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_wide_tiles(M, K, N, group, zeros, dt):
    """The wide tiles at the edges of their token tiles, K slabs and cuts; once more with the scratch of 128-token tiles
    (no tile is split then).  Sums of f16 x f16 products in fp32 against float64: the output's rounding and 2^-24 per
    addition of at most K terms, of the sum of magnitudes."""
    q = _q()
    from tilelang_ascend_b200 import _lib
    A, packed, scales = oc.make_w4a16_inputs(M, K, N, dt, group, seed=M + N)
    if zeros is None:
        z, W = 7, oc.dequant_weight_ref(packed, scales, 7, group)
    else:
        z = torch.randint(0, 16, scales.shape, generator=torch.Generator().manual_seed(M)).to(torch.float16)
        W = oc.dequant_weight_zeros_ref(packed, scales, z, group, zeros)
    A64, W64 = A.half().double(), W.double()
    ref = A64 @ W64.t()
    bound = (2.0 ** -11 if dt == "float16" else 2.0 ** -8) * ref.abs() + K * 2.0 ** -24 * (A64.abs() @ W64.abs().t()) + 1e-6
    Ac, P, S = A.cuda(), packed.cuda(), scales.cuda()
    Z = z.cuda() if zeros else None
    C = q.w4a16_gemm(Ac, P, S, Z if zeros else 7, group, zeros_mode=zeros or "original")
    assert bool(((C.cpu().double() - ref).abs() <= bound).all())
    lib = _lib.load()
    mode = {None: 0, "original": 0, "rescale": 1, "quantized": 2}[zeros]
    code = q.ops._ABI_DT[Ac.dtype]
    small = lib.qgemm_w4a16_call_workspace_bytes(1, M, N, K, group, 1, 1 if zeros else 0, mode)
    if M > 64:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        small = min(small, lib.qgemm_w4a16_counter_bytes() + sms * 2 * 128 * 128 * 4 + M * K * 2)
    ws = torch.empty(small, dtype=torch.uint8, device="cuda")
    C2 = torch.full((M, N), float("nan"), dtype=Ac.dtype, device="cuda")
    args = (Ac.data_ptr(), P.data_ptr(), S.data_ptr(), Z.data_ptr() if zeros else 0, 7, mode, 0, group, C2.data_ptr(), ws.data_ptr())
    call = lambda size: lib.qgemm_w4a16_ex(*args, size, 1, M, N, K, code, code, 0, torch.cuda.current_stream().cuda_stream)
    assert call(small - 1) != 0  # refused
    assert call(small) == 0, _lib.last_error()
    assert bool(((C2.cpu().double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("K", [96, 160, 192, 224])
@pytest.mark.parametrize("M,mode", [(70, None), (1800, None), (5, "original"), (33, "rescale"), (70, "quantized")])
def test_one_group_shorter_than_a_slab(K, M, mode):
    """One group of the whole K, K below a slab of 256 and no divisor of it, on the wide tiles: only the scale rows that
    were fetched may be read.  A call before it leaves NaN in the places where further rows would be."""
    q = _q()
    N, g = 272, torch.Generator().manual_seed(K + M)
    junk = [t.cuda() for t in oc.make_w4a16_inputs(70, 256, 148 * 128, "float16", 32, seed=1)]
    nan = torch.full_like(junk[2], float("nan"))
    q.w4a16_gemm(junk[0], junk[1], nan, nan, 32, zeros_mode="original")
    q.w4a16_gemm(junk[0], junk[1], nan, 8, 32)
    A, P, S = oc.make_w4a16_inputs(M, K, N, "float16", K, seed=K)
    if mode is None:
        W, zeros = oc.dequant_weight_ref(P, S, 8, K), 8
        C = q.w4a16_gemm(A.cuda(), P.cuda(), S.cuda(), 8, K)
    else:
        zeros = torch.randint(0, 16, (1, N), generator=g).half()
        W = oc.dequant_weight_zeros_ref(P, S, zeros, K, mode)
        C = q.w4a16_gemm(A.cuda(), P.cuda(), S.cuda(), zeros.cuda(), K, zeros_mode=mode)
    _close(C, (A.float() @ W.float().t()).half())


def _float64_ref(A, packed, scales, zeros, group):
    """C and the sum of the terms' magnitudes in float64: sum over k of a * (q - zero) * s, zeros an int or [K/g, N]."""
    qv = oc.unpack_uint4(packed).double()  # [N, K]
    z = zeros if isinstance(zeros, int) else zeros.double().t().repeat_interleave(group, 1)
    W = (qv - z) * scales.double().t().repeat_interleave(group, 1)
    A = A.half().double()
    return A @ W.t(), A.abs() @ W.abs().t()


@pytest.mark.parametrize("M,K,group,zeros,dt", [
    (1, 1024, 128, 8, "float16"), (16, 1024, 1024, 3, "bfloat16"),  # the single-launch form
    (5, 8192, 128, 8, "float16"), (24, 1024, 256, 15, "float16"), (64, 1024, 128, 8, "bfloat16"),  # pre-pass, three tile heights
    (16, 1024, 128, None, "float16"), (24, 1024, 1024, None, "bfloat16"), (40, 2048, 128, None, "float16"),  # zero tensors
])
def test_large_activations_at_the_zero_point(M, K, group, zeros, dt):
    """Large activations that face weights at the zero point contribute nothing, so they must not cost the other terms
    precision: (q - zero) is formed exactly before anything is multiplied.  Bar: the rounding of the output (8 or 11 bits)
    and of an fp32 sum of K terms, K * 2^-24 of the sum of the terms' magnitudes."""
    q = _q()
    N = 264 if zeros is not None else 272
    g = torch.Generator().manual_seed(M + K)
    A = (torch.randn((M, K), generator=g) * 0.02).to(getattr(torch, dt))
    A[:, 5::64] = torch.tensor([60000.0, -31000.0]).repeat(K // 128).to(A.dtype)
    nib = torch.randint(0, 16, (N, K), generator=g)
    z = torch.full((K // group, N), zeros) if zeros is not None else torch.randint(0, 16, (K // group, N), generator=g)
    nib[:, 5::64] = z.t().repeat_interleave(group, 1)[:, 5::64]
    packed = (nib[:, 0::2] | (nib[:, 1::2] << 4)).to(torch.uint8)
    scales = (torch.rand((K // group, N), generator=g) * 0.02 + 0.005).half()
    zt = zeros if zeros is not None else z.half()
    ref, mag = _float64_ref(A, packed, scales, zt, group)
    C = q.w4a16_gemm(A.cuda(), packed.cuda(), scales.cuda(), zt if zeros is not None else zt.cuda(), group,
                     zeros_mode="original" if zeros is not None else "quantized")
    bound = ref.abs() * 2.0 ** (-11 if dt == "float16" else -8) + mag * (K * 2.0 ** -24) + 1e-7
    err = (C.cpu().double() - ref).abs()
    assert (err <= bound).all(), (err / bound).max().item()


@pytest.mark.parametrize("M,K,N,n_dst", [
    (16, 1024, 264, 2), (33, 2048, 128, 8),            # group-sum kernel: whole tiles and tiles cut along K
    (100, 512, 272, 3), (128, 8192, 256, 2),           # wide tiles: whole ones; a few of long K, cut
    (300, 1024, 128 * 75, 2), (1800, 256, 272, 1),     # whole tiles and a cut remainder; many tokens, N no multiple of 64
])
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_gathered_form_writes_every_destination(M, K, N, n_dst, dt):
    """The gathered form with buffers of this GPU as destinations: the plain call's bits in columns [col0, col0 + N) of each,
    nothing beside them."""
    from tilelang_ascend_b200.ops import w4a16_gemm_gather
    q = _q()
    A, P, S = [t.cuda() for t in oc.make_w4a16_inputs(M, K, N, dt, 128, seed=M + N)]
    want = q.w4a16_gemm(A, P, S, 8, 128)
    ldc, col0 = N + 24, 8
    dst = [torch.full((M, ldc), 7.0, dtype=A.dtype, device="cuda") for _ in range(n_dst)]
    w4a16_gemm_gather(A, P, S, 8, 128, [d.data_ptr() for d in dst], ldc, col0)
    for d in dst:
        # (16 tokens: the plain call may be the single launch, which adds the K ranges in another order)
        if M <= 16:
            torch.testing.assert_close(d[:, col0:col0 + N].float(), want.float(), rtol=2e-3, atol=2e-3)
        else:
            assert torch.equal(d[:, col0:col0 + N], want)
        assert bool((d[:, :col0] == 7).all()) and bool((d[:, col0 + N:] == 7).all())


@pytest.mark.parametrize("M", [17, 31, 32, 33, 48, 49, 63, 64])
@pytest.mark.parametrize("K,N", [(512, 40), (2304, 1008), (4096, 20480)])
def test_each_token_gets_its_own_sums(M, K, N):
    """The drain sets share a tile's tokens: with one-hot activations token m reads weight column k(m) back, (q - 8) * s rounded
    once, bit for bit, whether its tile is whole or cut along K over several CTAs."""
    q = _q()
    _, packed, scales = oc.make_w4a16_inputs(M, K, N, "float16", 128, seed=M)
    k = (torch.arange(M) * 2654435761) % K
    A = torch.zeros(M, K, dtype=torch.float16)
    A[torch.arange(M), k] = 1.0
    C = q.w4a16_gemm(A.cuda(), packed.cuda(), scales.cuda(), 8, 128)
    byte = packed[:, k // 2].to(torch.int32)
    nibble = torch.where(k % 2 == 0, byte & 15, byte >> 4)              # [N, M]
    want = ((nibble - 8).float() * scales[k // 128].float().T).T.half()  # the product of two f16 values is exact in fp32
    assert torch.equal(C.cpu(), want)


# Wide tiles made by two CTAs (256 weight rows): whole tiles and tiles cut along K; tokens that fill a tile or end in the first or
# the second CTA's half of it; weight rows that end in either CTA's half; scale groups of 64 and 128; a zeros tensor.
@pytest.mark.parametrize("M,K,N,group,zeros", [(500, 8192, 14344, 128, False), (1000, 3328, 20488, 128, False), (430, 8192, 9472, 128, False),
                                               (860, 6144, 6016, 64, True), (1047, 4864, 3720, 128, False), (1588, 4608, 2992, 128, False)])
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_wide_tiles_of_two_ctas(M, K, N, group, zeros, dt):
    """One-hot activations read columns of half(q - zero) * s (f16) back bit for bit, for every token and weight row; dense ones
    agree with float64 within the fp32 sums' bound and the output's rounding."""
    q = _q()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    P = torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8)
    S = (torch.rand(K // group, N, generator=g, device="cuda") * 0.015 + 0.005).half()
    Z = torch.randint(0, 16, (K // group, N), generator=g, device="cuda").half() if zeros else 8
    nib = torch.stack([P & 15, P >> 4], dim=-1).view(N, K).half()
    rep = lambda t: t.T.repeat_interleave(group, dim=1)  # noqa: E731
    W = (nib - (rep(Z) if zeros else 8)) * rep(S)        # the difference is exact, the product rounds once
    out = torch.float16 if dt == "float16" else torch.bfloat16
    kw = dict(zeros_mode="quantized") if zeros else {}
    k = (torch.arange(M, device="cuda") * 2654435761) % K
    A = torch.zeros(M, K, dtype=out, device="cuda")
    A[torch.arange(M, device="cuda"), k] = 1.0
    assert torch.equal(q.w4a16_gemm(A, P, S, Z, group, **kw), W[:, k].T.to(out))
    A = torch.randn(M, K, generator=g, device="cuda").to(out)
    C = q.w4a16_gemm(A, P, S, Z, group, **kw).double()
    a = A.half().double()
    ref, mag = a @ W.double().T, a.abs() @ W.double().abs().T
    eps = 2.0 ** -11 if dt == "float16" else 2.0 ** -8
    assert ((C - ref).abs() <= eps * ref.abs() + K * 2.0 ** -24 * mag + 1e-7).all()


@pytest.mark.parametrize("hook,codes", [(1, [3]), (3, [1, 2, 3, 4]), (4, [1, 2, 3, 4])])
def test_wide_tiles_of_two_ctas_give_up_cleanly(hook, codes):
    """Bounded waits of the two-CTA wide tiles, made to run out in the safe way in the last pair: the last accumulators are never
    handed over (1), or one of the two CTAs copies no activations while the other one fills its ring (3, 4).  The launch ends by
    itself, without the code of a copy that never landed, and the next call is right."""
    q = _q()
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    A, P, S = (t.cuda() for t in oc.make_w4a16_inputs(430, 8192, 9472, "float16", 128, seed=1))
    want = q.w4a16_gemm(A, P, S, 8, 128)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        lib.qgemm_set_wait_limit_ms(20)
        lib.qgemm_debug_withhold_commit(hook)
        q.w4a16_gemm(A, P, S, 8, 128, status=status)
        torch.cuda.synchronize()  # returns: the kernel gave up by itself
        assert int(status.item()) in codes
    finally:
        lib.qgemm_debug_withhold_commit(0)
        lib.qgemm_set_wait_limit_ms(2000)
    status.zero_()
    assert torch.equal(q.w4a16_gemm(A, P, S, 8, 128, status=status), want)
    assert int(status.item()) == 0


def _call_workspaces(shapes, pair):
    """qgemm_w4a16_call_workspace_bytes of (M, K, N), groups of 128, in a process with pairs of CTAs switched on or off."""
    import json
    import os
    import subprocess
    import sys
    code = ("import json, sys; from tilelang_ascend_b200 import _lib; lib = _lib.load(); "
            "print(json.dumps([lib.qgemm_w4a16_call_workspace_bytes(1, M, N, K, 128, 1, 0, 0) for M, K, N in json.loads(sys.argv[1])]))")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    res = subprocess.run([sys.executable, "-c", code, json.dumps(shapes)], cwd=root, env={**os.environ, "QGEMM_W4_PAIR": pair},
                         capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stderr
    return json.loads(res.stdout.splitlines()[-1])


def test_token_counts_of_two_cta_tiles():
    """An MMA over two CTAs takes tokens in steps of 32: where pairs change a tile's height (read off the scratch that a call
    needs), the height is a multiple of it."""
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shapes = [(M, K, N) for K, N in [(6144, 6664), (3328, 4384), (8192, 12896), (3072, 8704), (5120, 6960)]
              for M in range(190, 2400, 53)]
    height = lambda s, need: (need - lib.qgemm_w4a16_counter_bytes() - 2 * s[0] * s[1]) // (sms * 2 * 128 * 4)  # noqa: E731
    changed = 0
    for s, one, two in zip(shapes, _call_workspaces(shapes, "0"), _call_workspaces(shapes, "1")):
        if one != two:
            changed += 1
            assert height(s, two) % 32 == 0, (s, height(s, two))
    assert changed >= 5


def test_short_k_stays_with_single_ctas():
    """Below thirteen slabs of K a pair of CTAs gains nothing or is the slower one: the plan is the one without pairs."""
    shapes = [(M, K, N) for K in (1024, 1536, 2048, 3072) for N in (1088, 4096, 13792, 25408) for M in (250, 700, 1152, 2221, 3468)]
    assert _call_workspaces(shapes, "1") == _call_workspaces(shapes, "0")


@pytest.mark.parametrize("M,K,N", [(211, 6400, 12768), (218, 8192, 12896)])
def test_scratch_for_single_ctas_is_enough(M, K, N):
    """Where pairs of CTAs would take taller tiles, and so more scratch, the scratch that single CTAs need is still accepted,
    a byte less is refused as it is without pairs, and the results agree within the fp32 sums' bound and the output's rounding."""
    q = _q()
    from tilelang_ascend_b200 import _lib
    lib = _lib.load()
    (small,), (large,) = _call_workspaces([(M, K, N)], "0"), _call_workspaces([(M, K, N)], "1")
    assert small < large  # otherwise the shape shows nothing
    A, P, S = (t.cuda() for t in oc.make_w4a16_inputs(M, K, N, "float16", 128, seed=M))
    want = q.w4a16_gemm(A, P, S, 8, 128).double()
    code = q.ops._ABI_DT[torch.float16]
    ws = torch.empty(small, dtype=torch.uint8, device="cuda")
    C = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    call = lambda size: lib.qgemm_w4a16_ex(A.data_ptr(), P.data_ptr(), S.data_ptr(), 0, 8, 0, 0, 128, C.data_ptr(), ws.data_ptr(),  # noqa: E731
                                           size, 1, M, N, K, code, code, 0, torch.cuda.current_stream().cuda_stream)
    assert call(small - 1) != 0
    assert call(small) == 0, _lib.last_error()
    # both ways add the same products in fp32, in another order: K 2^-24 of the sum of magnitudes each
    nib = torch.stack([P & 15, P >> 4], dim=-1).view(N, K).half()
    W = ((nib - 8) * S.T.repeat_interleave(128, dim=1)).double()
    mag = A.double().abs() @ W.abs().T
    assert ((C.double() - want).abs() <= 2.0 ** -10 * want.abs() + 2 * K * 2.0 ** -24 * mag + 1e-7).all()


def test_switch_for_wide_tiles_of_two_ctas():
    """QGEMM_W4_PAIR=0 (read once per process, hence a child process): single CTAs make the tiles, so that the test hook of the
    two-CTA form changes nothing; one-hot activations read columns of (q - 8) * s back bit for bit."""
    import os
    import subprocess
    import sys
    code = r"""
import torch
from oracle import qgemm_oracle as oc
import tilelang_ascend_b200 as q
from tilelang_ascend_b200 import _lib
_lib.load().qgemm_debug_withhold_commit(1)
M, K, N = 430, 8192, 9472
_, P, S = (t.cuda() for t in oc.make_w4a16_inputs(16, K, N, "float16", 128, seed=1))
W = (torch.stack([P & 15, P >> 4], dim=-1).view(N, K).half() - 8) * S.T.repeat_interleave(128, dim=1)
k = (torch.arange(M, device="cuda") * 2654435761) % K
A = torch.zeros(M, K, dtype=torch.float16, device="cuda")
A[torch.arange(M, device="cuda"), k] = 1.0
status = torch.zeros(1, dtype=torch.int32, device="cuda")
assert torch.equal(q.w4a16_gemm(A, P, S, 8, 128, status=status), W[:, k].T) and int(status.item()) == 0
print("single ok")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, QGEMM_W4_PAIR="0"), capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "single ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("batch,M,K,N", [
    # one (row, slab) per warp of the pre-pass, one and a few rows; a last slab that is cut; two in registers; three and ten in shared
    # memory; rounds of several, the last one partly filled; a block for every round, one and several waves of them; and, up to 16
    # tokens of a short K, no pre-pass
    (1, 1, 8192, 40), (1, 5, 8224, 64), (1, 16, 8224, 64), (3, 13, 6432, 64), (60, 15, 4128, 40),
    (13, 64, 8192, 40), (75, 37, 6432, 40),
    (1, 1, 288, 40), (3, 5, 1312, 64), (1, 48, 4384, 72), (2, 33, 6432, 40), (23, 16, 4096, 48), (40, 16, 4096, 64), (9, 64, 8192, 40),
    (1, 64, 8224, 128), (19, 61, 5152, 40)])
@pytest.mark.parametrize("dt", ["float16", "bfloat16"])
def test_pre_pass_of_the_group_sum_kernel(batch, M, K, N, dt):
    """Small integer activations and scales of one: the fp32 sums are exact, so the result is the float64 product rounded once.
    The scratch starts as NaN: activation rows beyond M are not written and must not reach an output."""
    q = _q()
    g = torch.Generator(device="cuda").manual_seed(K + 64 * M + batch)
    A = torch.randint(-3, 4, (batch, M, K), generator=g, device="cuda").to(getattr(torch, dt))
    P = torch.randint(0, 256, (batch, N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    S = torch.ones((batch, 1, N), dtype=torch.float16, device="cuda")
    W = torch.stack([P & 15, P >> 4], dim=-1).view(batch, N, K).double() - 8
    want = (A.double() @ W.transpose(1, 2)).to(getattr(torch, dt))
    if batch == 1:
        A, P, S, want = A[0], P[0], S[0], want[0]
    poison = torch.full((1 << 24,), float("nan"), device="cuda")  # the scratch comes from this block
    del poison
    assert torch.equal(q.w4a16_gemm(A, P, S, 8, K), want)


# On 148 SMs, slabs per CTA and the tiles they belong to: fewer than the activation stages (one, two, three), as many, one more; a change
# of tile after one slab, after two, after three, with a batch, and from a shared tile to a whole one; one token and M below the tile.
@pytest.mark.parametrize("batch,M,K,N", [
    (1, 1, 8192, 560), (1, 1, 1792, 6288), (1, 3, 3584, 4096), (1, 16, 1024, 20000), (1, 9, 1280, 20000), (1, 2, 512, 30000),
    (1, 1, 768, 24000), (3, 13, 2304, 7296), (19, 5, 512, 1072)])
@pytest.mark.parametrize("zeros", ["scalar", "tensor"])
def test_first_activations_of_a_cta(batch, M, K, N, zeros):
    """Small integer activations and scales of one, as above: the fp32 sums are exact."""
    q = _q()
    g = torch.Generator(device="cuda").manual_seed(K + 64 * M + batch)
    A = torch.randint(-3, 4, (batch, M, K), generator=g, device="cuda").to(torch.bfloat16)
    P = torch.randint(0, 256, (batch, N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    S = torch.ones((batch, K // 256, N), dtype=torch.float16, device="cuda")
    Z = torch.randint(0, 16, (batch, K // 256, N), generator=g, device="cuda").to(torch.float16)
    W = torch.stack([P & 15, P >> 4], dim=-1).view(batch, N, K).double()
    W -= 8 if zeros == "scalar" else Z.double().transpose(1, 2).repeat_interleave(256, dim=2)
    want = (A.double() @ W.transpose(1, 2)).to(torch.bfloat16)
    for _ in range(2):  # the second call starts beside the first one
        got = [q.w4a16_gemm(A, P, S, 8, 256) if zeros == "scalar" else q.w4a16_gemm(A, P, S, Z, 256, zeros_mode="quantized") for _ in range(3)]
        assert all(torch.equal(x, want) for x in got)


# On 148 SMs: every tile's K in equal ranges, one per CTA.  Whole tiles on 61 and 66 CTAs, on 60 with 8.9 slabs a CTA more than an even
# deal has, on 60 with 10.1 more (not taken), on 59 (not taken); ranges of two on 99 and 108, of three on 99; halves with 4.9 and with
# 5.1 slabs more (not taken).
@pytest.mark.parametrize("batch,M,K,N", [
    (1, 64, 1280, 7728), (1, 40, 2816, 8400), (1, 20, 3840, 7680), (1, 20, 4352, 7680), (1, 17, 1280, 7504), (1, 16, 4608, 1312),
    (1, 32, 3072, 2256), (1, 3, 6912, 1312), (1, 12, 5632, 5248), (4, 12, 5632, 1280)])
def test_equal_ranges_of_k(batch, M, K, N):
    """Small integer activations and scales of one: the fp32 sums are exact whatever the cut."""
    q = _q()
    g = torch.Generator(device="cuda").manual_seed(K + 64 * M + batch)
    A = torch.randint(-3, 4, (batch, M, K), generator=g, device="cuda").half()
    P = torch.randint(0, 256, (batch, N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    S = torch.ones((batch, K // 128, N), dtype=torch.float16, device="cuda")
    W = torch.stack([P & 15, P >> 4], dim=-1).view(batch, N, K).double() - 8
    want = (A.double() @ W.transpose(1, 2)).half()
    for _ in range(2):
        assert all(torch.equal(x, want) for x in [q.w4a16_gemm(A, P, S, 8, 128) for _ in range(3)])
