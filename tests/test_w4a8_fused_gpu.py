"""GPU parity of the fused W4A8 kernel (int4 weights unpacked on the way to the tensor core, up to 128 tokens)
through the C ABI entry qgemm_w4a8, exact int32 against the CPU oracle."""
import pytest
import torch

import tilelang_ascend_b200 as q
from oracle import qgemm_oracle as oc

pytestmark = pytest.mark.gpu

# (M, N, K): every token-tile height (16 / 32 / 64 / 128), ragged N and K (K not a multiple of the 256-wide slab),
# sizes large enough for the kernel's scratch to fit into the caller's [N, K] workspace
CASES = [(1, 1024, 4096), (16, 1040, 4128), (17, 2048, 4096), (32, 2064, 4064), (40, 4096, 4096),
         (64, 4112, 4096), (100, 4096, 8192), (128, 4096, 8224)]


@pytest.mark.parametrize("M,N,K", CASES)
def test_signed_nibbles_exact_and_no_int8_copy(M, N, K):
    g = torch.Generator().manual_seed(M * 7 + N)
    A = torch.randint(-128, 128, (M, K), dtype=torch.int8, generator=g)
    Bi = torch.randint(-8, 8, (N, K), dtype=torch.int8, generator=g)
    qB = oc.pack_int4_signed(Bi)
    ws = torch.full((N, K), 0x55, dtype=torch.int8, device="cuda")
    C = torch.zeros(M, N, dtype=torch.int32, device="cuda")
    out = q.w4a8_gemm_cv(M, N, K)(A.cuda(), qB.cuda(), ws, C)
    assert torch.equal(out.cpu(), oc.w4a8_gemm_ref(A, qB))
    # the fused kernel uses only the head of the workspace as scratch: the int8 copy of the weights is never written
    assert torch.all(ws[-1] == 0x55) and not torch.equal(ws[-1].cpu(), Bi[-1])
    # a second call on the same (dirty) workspace gives the same result
    out2 = q.w4a8_gemm_cv(M, N, K)(A.cuda(), qB.cuda(), ws, torch.zeros_like(C))
    assert torch.equal(out2, out)


@pytest.mark.parametrize("M,N,K", [(8, 1024, 4096), (48, 4096, 4096)])
def test_unsigned_nibbles_int8_mode_exact(M, N, K):
    g = torch.Generator().manual_seed(K + M)
    A = torch.randint(-128, 128, (M, K), dtype=torch.int8, generator=g)
    P = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g)
    C = q.dequant_gemm_int8_wrapper(M, N, K, 128, 128, 64, "int32")(A.cuda(), P.cuda())
    assert torch.equal(C.cpu(), oc.dequant_gemm_int8_ref(A, P, "int32"))


def test_extreme_values():
    M, N, K = 16, 1024, 4096
    A = torch.full((M, K), -128, dtype=torch.int8)
    Bi = torch.full((N, K), -8, dtype=torch.int8)
    Bi[::2] = 7
    qB = oc.pack_int4_signed(Bi)
    ws = torch.zeros(N, K, dtype=torch.int8, device="cuda")
    C = torch.zeros(M, N, dtype=torch.int32, device="cuda")
    out = q.w4a8_gemm_cv(M, N, K)(A.cuda(), qB.cuda(), ws, C)
    assert torch.equal(out.cpu(), oc.w4a8_gemm_ref(A, qB))


# Weight tiles for a number of SMs, and whether there are whole ones in the form for few tokens and K of at least 24 slabs: a round
# of whole tiles and nothing cut; a remainder of at least half a round, cut; two rounds and one tile, cut with one of the rounds; and
# one round and one tile, all of which are cut.
TILES = [(lambda sms: sms, True), (lambda sms: sms + (sms + 1) // 2 + 2, True), (lambda sms: 2 * sms + 1, True), (lambda sms: sms + 1, False)]


@pytest.mark.parametrize("tiles,whole", TILES)
@pytest.mark.parametrize("M,K", [(16, 6144), (1, 6176), (7, 5888), (17, 6144)])
@pytest.mark.parametrize("form", ["signed", "unsigned", "quantised"])
def test_whole_tiles_behind_cut_ones(form, M, K, tiles, whole):
    """Few tokens, long K and at least a round of tiles: the remainder's tiles are cut along K first, whole ones follow.  K = 5888
    (23 slabs) and 17 tokens stay with the other form.  Exact, against float64 sums."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = tiles(sms)
    assert (n // sms - (1 if 0 < 2 * (n % sms) < sms else 0) > 0) == whole
    N = 128 * n - 48
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    qB = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    W = torch.stack([qB & 15, qB >> 4], dim=-1).view(N, K).double()
    if form != "unsigned":
        W = torch.where(W >= 8, W - 16, W)
    ws, C = torch.empty((N, K), dtype=torch.int8, device="cuda"), torch.empty((M, N), dtype=torch.int32, device="cuda")
    if form == "quantised":
        x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
        A, scale = q.act_quant(x)
        C, s = q.w4a8_gemm_act_quant(M, N, K)(x, qB, ws, C)
        assert torch.equal(s.view(-1), scale.view(-1))
    else:
        A = torch.randint(-128, 128, (M, K), dtype=torch.int8, generator=g, device="cuda")
        C = q.w4a8_gemm_cv(M, N, K)(A, qB, ws, C) if form == "signed" else q.dequant_gemm_int8_wrapper(M, N, K, 128, 128, 64)(A, qB)
    assert torch.equal(C.double(), A.double() @ W.T)


@pytest.mark.parametrize("M,K,N", [(1, 2048, 2048), (48, 4096, 4096), (2, 16384 + 256, 1024)])
@pytest.mark.parametrize("fused", [True, False])
def test_behind_the_kernels_that_write_its_activations(M, K, N, fused):
    """The pre-pass starts early behind the few-token W8A8 kernel and the quantiser, which still write the activations then: a
    chain is bit-identical to the same chain with the device drained between the calls."""
    import tilelang_ascend_b200 as q
    g = torch.Generator(device="cuda").manual_seed(M + K)
    a0 = torch.randint(-128, 128, (M, K), dtype=torch.int8, generator=g, device="cuda")
    Ws = [torch.randint(-128, 128, (K, K), dtype=torch.int8, generator=g, device="cuda") for _ in range(3)]
    scale = torch.full((K,), 1e-4, device="cuda")
    qB = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    ws = torch.empty((N, K), dtype=torch.int8, device="cuda")
    kernel = q.w4a8_gemm_act_quant(M, N, K) if fused else q.w4a8_gemm_cv(M, N, K)

    def chain(drain):
        step = torch.cuda.synchronize if drain else lambda: None
        out, a = [], a0
        for i in range(9):
            h = q.quant_matmul(a, Ws[i % 3], scale, out_dtype="bfloat16")
            step()
            C = torch.empty((M, N), dtype=torch.int32, device="cuda")
            if fused:
                C, s = kernel(h, qB, ws, C)
                out.append(s)
                step()
            a, s = q.act_quant(h)
            step()
            if not fused:
                C = kernel(a, qB, ws, C)
                step()
            out += [C, s]
        return out

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(chain(False), want))
    assert len({int(c.view(-1)[0]) for c in want if c.dtype == torch.int32}) > 1  # the steps differ


# blocks per row of the pre-pass: eight, as many as leave one per SM, one; rows of more chunks than it keeps in shared memory; parts
# that are not whole multiples of a block's threads
@pytest.mark.parametrize("M,K", [(1, 4128), (18, 4128), (19, 8224), (37, 8192), (49, 8224), (74, 4096), (75, 4128), (128, 8224), (5, 16416)])
@pytest.mark.parametrize("dt", ["bfloat16", "float16"])
def test_parts_of_the_pre_pass(M, K, dt):
    """Quantised activations and their row sums, made by several blocks per row: exact against the quantiser's int8 values, with
    weights whose sums the row sums decide."""
    N = 5120
    g = torch.Generator(device="cuda").manual_seed(K + M)
    x = (torch.randn((M, K), generator=g, device="cuda") + 0.5).to(getattr(torch, dt))
    x[:, -1] = 7.0  # the largest value of a row belongs to its last part
    qB = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    W = torch.stack([qB & 15, qB >> 4], dim=-1).view(N, K).double()
    W = torch.where(W >= 8, W - 16, W)
    ws = torch.full((N, K), 0x55, dtype=torch.int8, device="cuda")
    C = torch.empty((M, N), dtype=torch.int32, device="cuda")
    A, scale = q.act_quant(x)
    want = A.double() @ W.T
    got, s = q.w4a8_gemm_act_quant(M, N, K)(x, qB, ws, C)
    assert torch.equal(s.view(-1), scale.view(-1)) and torch.equal(got.double(), want)
    assert torch.equal(q.w4a8_gemm_cv(M, N, K)(A, qB, ws, torch.empty_like(C)).double(), want)
