"""The hand-written tcgen05 GEMM against an fp32 PyTorch reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,bn", [(128, 256, 64, 256), (128, 128, 128, 128), (256, 512, 256, 0), (300, 520, 200, 0),
                                      (1024, 1024, 1024, 256), (1024, 1024, 1024, 128), (4096, 6144, 4096, 0)])
def test_gemm_bf16_tn_matches_fp32(M, N, K, bn):
    from rocm_systems_b200.ops import train_ops as ops

    torch.manual_seed(M + N + K)
    a = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    b = torch.randn(N, K, device="cuda").to(torch.bfloat16)
    out = ops.gemm_bf16_tn(a, b, bn=bn)
    torch.cuda.synchronize()
    assert ops.gemm_take_error() == 0
    ref = a.float() @ b.float().t()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)


@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K,bn", [(256, 256, 64, 256), (256, 128, 128, 128), (512, 512, 256, 0), (304, 520, 200, 0), (1000, 328, 72, 0),
                                      (1024, 1024, 1024, 256), (1024, 1024, 1024, 128), (4096, 6144, 4096, 0)])
def test_gemm_on_cta_pairs_matches_fp32_for_every_operand_order(M, N, K, bn, ta, tb):
    """The CTA-pair kernel with each operand stored K-major (row-major [rows, K]) or MN-major (the transpose view of a
    row-major [K, rows]): the forward, input-gradient and weight-gradient forms of a linear layer."""
    from rocm_systems_b200.ops import train_ops as ops

    torch.manual_seed(M + N + K)
    a = (torch.randn(K, M, device="cuda").to(torch.bfloat16).t() if ta else torch.randn(M, K, device="cuda").to(torch.bfloat16))
    b = (torch.randn(K, N, device="cuda").to(torch.bfloat16).t() if tb else torch.randn(N, K, device="cuda").to(torch.bfloat16))
    out = ops.gemm(a, b, bn=bn)
    torch.cuda.synchronize()
    assert ops.gemm_take_error() == 0
    ref = a.float() @ b.float().t()
    err = (out.float() - ref).abs().max().item()
    scale = ref.abs().max().item()
    assert err <= 1e-2 * scale + 1e-2, (err, scale)


def test_gemm_on_cta_pairs_writes_into_a_strided_view():
    from rocm_systems_b200.ops import train_ops as ops

    torch.manual_seed(5)
    a = torch.randn(384, 256, device="cuda").to(torch.bfloat16)
    b = torch.randn(200, 256, device="cuda").to(torch.bfloat16)
    big = torch.full((384, 512), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm(a, b, out=big[:, 64:264])
    torch.cuda.synchronize()
    assert ops.gemm_take_error() == 0
    ref = a.float() @ b.float().t()
    assert (big[:, 64:264].float() - ref).abs().max().item() <= 1e-2 * ref.abs().max().item() + 1e-2
    assert bool((big[:, :64] == 7).all()) and bool((big[:, 264:] == 7).all())     # nothing outside the view was written


@pytest.mark.parametrize("wt", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (1, 1000, 8), (16, 6144, 4096), (17, 136, 200), (33, 4096, 14336), (64, 28672, 512), (65, 1032, 1000),
                                   (128, 264, 328), (129, 4096, 1024), (300, 520, 4096), (512, 1024, 520)])
def test_gemm_of_few_rows_matches_fp32(M, N, K, wt):
    """Sizes that take the kernel with output features as MMA rows and K split over a cluster (one token up to four token tiles, ragged
    edges in every direction, fewer 64-step slices than splits). Bound: one bf16 rounding of the result (within 2^-8 of its size), and
    one fp32 truncation (2^-23 of the running sum) per 16 reduction steps of an MMA, K / 16 of them; the running sum of K products
    of unit variance stays below 6 sqrt(K)."""
    from rocm_systems_b200.ops import train_ops as ops

    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    w = torch.randn(K, N, device="cuda").to(torch.bfloat16).t() if wt else torch.randn(N, K, device="cuda").to(torch.bfloat16)
    big = torch.full((M + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.gemm(x, w, out=big[:M, :N])
    torch.cuda.synchronize()
    assert ops.gemm_take_error() == 0
    ref = x.double() @ w.double().t()
    err = (big[:M, :N].double() - ref).abs()
    assert bool((err <= ref.abs() * 2.0 ** -8 + 6 / 16 * K ** 1.5 * 2.0 ** -23).all()), float((err - ref.abs() * 2.0 ** -8).max())
    assert bool((big[M:] == 7).all()) and bool((big[:, N:] == 7).all())     # nothing outside the view was written


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (1, 1000, 256), (16, 6144, 4096), (17, 136, 384), (32, 4096, 14336), (33, 4096, 1152), (64, 28672, 512),
                                   (65, 1032, 640), (65, 1032, 1152), (128, 264, 4096), (192, 512, 8192), (257, 640, 384), (16, 136, 16512), (40, 2056, 640), (20, 6152, 512), (1, 520, 896)])
def test_fp8_linear_of_few_rows_matches_the_oracle(M, N, K):
    """The block-scaled kernel with output features as MMA rows (one to four token tiles, ragged edges, more splits than blocks of K, a K
    whose scales just do not fit), behind the quantiser it may overlap. Products of codes are exact in fp32; bound: the bf16 rounding of
    the result and one fp32 rounding per block and split of a sum that stays below the sum of magnitudes."""
    from rocm_systems_b200.ops import fp8
    from rocm_systems_b200.ops import train_ops as ops

    torch.manual_seed(M + N + K)
    x = torch.randn(M, K, device="cuda").to(torch.bfloat16)
    wq, ws = fp8.quantize_weight((torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16))
    xq, xs = fp8.quantize_act(x)
    rq, rs = fp8.ref_quantize_act(x)
    assert torch.equal(xq.view(torch.uint8), rq.view(torch.uint8)) and torch.equal(xs, rs)
    a, b = fp8.ref_dequantize_act(xq, xs).double(), fp8.ref_dequantize_weight(wq, ws).double()
    ref = a @ b.t()
    tol = ref.abs() * 2.0 ** -8 + (a.abs() @ b.abs().t()) * 2.0 ** -24 * (K // 128 + 16)
    for out in (fp8.linear(x, wq, ws), fp8.gemm(xq, xs, wq, ws)):
        torch.cuda.synchronize()
        assert ops.gemm_take_error() == 0
        assert bool(((out.double() - ref).abs() <= tol).all())


@pytest.mark.parametrize("size", [1e-30, 1e-12, 1.0, 1e30])
def test_quantiser_codes_are_those_of_an_ieee_division(size):
    """Every bf16 significand over scales drawn from the data: codes and scales of both quantisers are bit-equal to the oracles', which divide."""
    from rocm_systems_b200.ops import fp8

    torch.manual_seed(1)
    x = (torch.randn(1500, 2176, device="cuda") * size).to(torch.bfloat16)
    x[0, :128] = 0
    x[1, 3] = float("inf")
    for got, want in ((fp8.quantize_act(x), fp8.ref_quantize_act(x)), (fp8.quantize_weight(x[2:]), fp8.ref_quantize_weight(x[2:]))):
        assert torch.equal(got[0].view(torch.uint8) & 0x7f == 0x7f, want[0].view(torch.uint8) & 0x7f == 0x7f)   # NaN (inf / inf) in the same places
        ok = want[0].view(torch.uint8) & 0x7f != 0x7f
        assert torch.equal(got[0].view(torch.uint8)[ok], want[0].view(torch.uint8)[ok]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("amax", [0.0, 2.0 ** -133, 1e-20, 1.0, 3e38])
def test_quantisers_keep_the_sign_of_zeros_and_of_what_rounds_to_zero(amax):
    """-0, the smallest negative numbers and quotients below half a code step become the code 0x80 as they do in a division; the expert layer's
    dispatch quantises the same way (its bf16 copy of the rows holds -0 there). Whole codes are compared."""
    from rocm_systems_b200.comm import Communicator, get_unique_id
    from rocm_systems_b200.ops import fp8
    from rocm_systems_b200.parallel.ep import MoELayer, dequantize_e4m3_per128, quantize_e4m3_per128

    E, H = 32, 1024
    g = torch.Generator(device="cuda").manual_seed(3)
    small = torch.tensor([-0.0, 0.0, -(2.0 ** -133), 2.0 ** -133, -(2.0 ** -126), 2.0 ** -126, -1e-30, 1e-30], device="cuda")
    x = small[torch.randint(0, len(small), (E, H), device="cuda", generator=g)].to(torch.bfloat16)
    x[:, ::128] = amax
    x[1::2, ::128] = -amax
    assert bool((x.view(torch.int16) == -32768).any())      # -0 is in there
    for got, want in ((fp8.quantize_act(x), fp8.ref_quantize_act(x)), (fp8.quantize_weight(x), fp8.ref_quantize_weight(x))):
        assert torch.equal(got[0].view(torch.uint8), want[0].view(torch.uint8)) and torch.equal(got[1], want[1])
    comm = Communicator(0, 1, get_unique_id(), 0)
    moe = MoELayer(comm, E, H, 128, 1, E, capacity=128, seed=5)
    moe.forward(x, 4.0 * torch.eye(E, device="cuda"))       # token e is the one row of expert e
    rows = moe.xb.view(E, 128, H)[:, 0]
    torch.cuda.synchronize()
    assert torch.equal(rows.view(torch.int16), dequantize_e4m3_per128(*quantize_e4m3_per128(x)).view(torch.int16))
    moe.free()
    comm.destroy()


@pytest.mark.parametrize("M,N,K", [(1000, 8200, 1152), (129, 28680, 1152), (513, 8192, 1152), (2049, 8200, 640), (4096, 6144, 512), (4097, 4104, 512), (513, 4232, 1152), (2049, 7176, 640)])
def test_fp8_gemm_on_cta_pairs_equals_the_one_cta_kernel(M, N, K):
    """Sizes that the rule sends to CTA pairs (ragged rows, columns and an odd number of blocks of K): every partial product is folded in the
    same order with the same operations, so the results are bit-equal to the kernel that a CTA limit asks for. Strided output; nothing else is written."""
    from rocm_systems_b200.ops import fp8
    from rocm_systems_b200.ops import train_ops as ops

    torch.manual_seed(M + N + K)
    xq, xs = fp8.quantize_act(torch.randn(M, K, device="cuda").to(torch.bfloat16))
    wq, ws = fp8.quantize_weight((torch.randn(N, K, device="cuda") * 0.05).to(torch.bfloat16))
    big = torch.full((M + 1, N + 8), 7.0, dtype=torch.bfloat16, device="cuda")
    fp8.gemm(xq, xs, wq, ws, out=big[:M, :N])
    want = fp8.gemm(xq, xs, wq, ws, max_ctas=148)
    torch.cuda.synchronize()
    assert ops.gemm_take_error() == 0
    assert torch.equal(big[:M, :N], want)
    assert bool((big[M:] == 7).all()) and bool((big[:, N:] == 7).all())
