"""The expert GEMMs of the mixture-of-experts layer where their tiles end: few rows (features as MMA rows), for fp8 a middle range (a CTA
per 128 x 128 tile), many (CTA pairs), experts without any, one expert with all, counts around the edges of 16, 32, 64, 128 and 256 rows, forward and backward."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm():
    from rocm_systems_b200.comm import Communicator, get_unique_id

    torch.cuda.set_device(0)
    c = Communicator(0, 1, get_unique_id(), 0)
    yield c
    c.destroy()


def _logits(counts, E, k):
    """Logits that send every token to k experts, expert e to counts[e] tokens in all (counts sum to T * k, none above T)."""
    T = sum(counts) // k
    out = torch.full((T, E), -4.0)
    slots = [e for e in range(E) for _ in range(counts[e])]
    for i, e in enumerate(slots):      # consecutive slots of one expert go to different tokens
        out[i % T, e] = 1.0 + 0.01 * ((i * 7) % 13)
    return out.cuda()


# (hidden, ffn, k, rows of the experts)
CASES = [
    (1024, 128, 1, [1]),
    (1024, 256, 1, [15, 16, 17, 0, 31, 32, 33]),
    (2048, 384, 2, [63, 64, 65, 0, 40, 80, 80]),
    (1024, 256, 1, [127, 128, 129, 0, 1]),
    (1024, 640, 1, [255, 256, 257, 0, 511, 512, 513, 900]),
    (3072, 128, 2, [1000, 1000]),
    (1024, 128, 1, [0, 127, 128, 129, 300, 1, 0, 640, 255, 256, 257, 384, 385, 1200]),     # more than 112 rows per expert on average
]


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("hidden,ffn,k,rows", CASES)
def test_experts_match_float64(comm, hidden, ffn, k, rows, fp8):
    """Forward (bf16 or fp8 gate/up weights) and, in bf16, backward against float64 on the dequantised rows. Bounds relative to the
    2-norm: four bf16 roundings of 2^-9 rms each in a chain (pre-activation, activation, row, sum) stay below 2^-6; dropped capacity never occurs."""
    from rocm_systems_b200.ops import train_ops as ops
    from rocm_systems_b200.parallel.ep import MoELayer, dequantize_e4m3_per128, quantize_e4m3_per128

    E = 32
    counts = rows + [0] * (E - len(rows))
    T = sum(counts) // k
    moe = MoELayer(comm, E, hidden, ffn, k, T, capacity=max(max(counts), 128), seed=5, fp8_experts=fp8)
    try:
        g = torch.Generator(device="cuda").manual_seed(hidden + ffn)
        logits = _logits(counts, E, k)
        for trial in range(2):         # both parities of the counters, and buffers that hold an earlier call's rows
            x = torch.randn(T, hidden, device="cuda", generator=g).to(torch.bfloat16)
            dy = torch.randn(T, hidden, device="cuda", generator=g).to(torch.bfloat16)
            if trial == 0 and not fp8:  # whatever an earlier program left in the scratch buffers must not matter
                moe.xb.fill_(float("nan"))
                moe.act.fill_(float("nan"))
            y = moe.forward(x, logits).clone()
            assert moe.counts() == (counts, 0)
            xq = dequantize_e4m3_per128(*quantize_e4m3_per128(x)).double()
            wg, wu = (w.double().requires_grad_(True) for w in ((moe._w_gate_ref, moe._w_up_ref) if fp8 else (moe.w_gate, moe.w_up)))
            wd, xl, ll = moe.w_down.double().requires_grad_(True), xq.clone().requires_grad_(True), logits.double().requires_grad_(True)
            tv, ti = torch.topk(ll, k, dim=-1)
            tw = torch.softmax(tv, -1)
            ref = torch.zeros_like(xl)
            for e in range(E):
                t, r = (ti == e).nonzero(as_tuple=True)
                if t.numel():
                    ref = ref.index_add(0, t, tw[t, r].unsqueeze(-1) * ((torch.nn.functional.silu(xl[t] @ wg[e].t()) * (xl[t] @ wu[e].t())) @ wd[e].t()))
            pairs = [(y, ref.detach())]
            if not fp8:
                ref.backward(dy.double())
                dx, dlogits = moe.backward(dy)
                dg, du, dd = moe.expert_weight_grads()
                pairs += [(dx, xl.grad), (dg, wg.grad), (du, wu.grad), (dd, wd.grad)]
                if k > 1:
                    pairs.append((dlogits, ll.grad))
                else:
                    assert bool((dlogits == 0).all())      # a softmax over one value
                for e in range(E):
                    if counts[e] == 0:
                        assert not bool(dg[e].any() or du[e].any() or dd[e].any())
            torch.cuda.synchronize()
            assert ops.gemm_take_error() == 0
            for i, (a, b) in enumerate(pairs):
                assert float((a.double() - b).norm()) <= 2.0 ** -6 * float(b.norm()), (trial, i)
    finally:
        moe.free()


@pytest.mark.parametrize("rows", [[1, 40, 0, 128, 33], [97, 256, 0, 511, 2300]])      # few rows per expert on average, and more than 96
@pytest.mark.parametrize("w_rows,K", [(128, 200), (384, 1000), (640, 64), (1024, 1032)])
def test_grouped_gemm_matches_float64(comm, rows, w_rows, K):
    """The grouped GEMM a program can call by itself, with weight rows that end inside a 256-column tile and reductions that end inside a 64-step slice.
    Nothing is written past an expert's rows, and what lies past them in the input does not matter. 1024 weight rows: the result
    goes to the window, where combine with unit weights finds it. Bound: the bf16 rounding of the result and one fp32 truncation per 16
    steps of a sum that stays below the sum of magnitudes."""
    from rocm_systems_b200 import _lib
    from rocm_systems_b200.ops import train_ops as ops
    from rocm_systems_b200.parallel.ep import MoELayer, _lib_ep

    E, H = 32, 1024
    counts = rows + [0] * (E - len(rows))
    T = sum(counts)
    moe = MoELayer(comm, E, H, 128, 1, T, capacity=max(max(counts), 128), seed=5)
    try:
        g = torch.Generator(device="cuda").manual_seed(w_rows + K)
        moe.forward(torch.randn(T, H, device="cuda", generator=g).to(torch.bfloat16), _logits(counts, E, 1))
        assert moe.counts() == (counts, 0)
        a = torch.randn(E, moe.cap, K, device="cuda", generator=g).to(torch.bfloat16)
        for e in range(E):
            a[e, counts[e]:] = float("nan")
        w = torch.randn(E, w_rows, K, device="cuda", generator=g).to(torch.bfloat16)
        out = torch.full((E, moe.cap, w_rows), 7.0, dtype=torch.bfloat16, device="cuda")
        to_window = w_rows == H
        _lib.check(_lib_ep().b200collEpGroupedGemm(comm.handle, moe._win.ptr, a.data_ptr(), w.data_ptr(), None if to_window else out.data_ptr(), w_rows, K, *moe._args(),
                                                   ops._s()), "b200collEpGroupedGemm")
        if to_window:
            y, ones = torch.empty(T, H, dtype=torch.bfloat16, device="cuda"), torch.ones(T, 1, device="cuda")
            _lib.check(_lib_ep().b200collEpCombine(comm.handle, moe._win.ptr, moe.top_idx.data_ptr(), ones.data_ptr(), moe.sent.data_ptr(), y.data_ptr(), T, 1, *moe._args(),
                                                   ops._s()), "b200collEpCombine")
            out[moe.top_idx[:, 0].long(), moe.sent[:, 0].long()] = y
        torch.cuda.synchronize()
        assert ops.gemm_take_error() == 0
        for e in range(E):
            x, ww, got = a[e, :counts[e]].double(), w[e].double(), out[e]
            ref = x @ ww.t()
            tol = ref.abs() * 2.0 ** -8 + (x.abs() @ ww.abs().t()) * 2.0 ** -23 * (K // 16 + 1)
            assert bool(((got[:counts[e]].double() - ref).abs() <= tol).all()), e
            assert bool((got[counts[e]:] == 7).all()), e
    finally:
        moe.free()


@pytest.mark.parametrize("T,E,k", [(1, 32, 1), (33, 32, 8), (1000, 64, 2), (9, 1024, 8), (257, 256, 5)])
def test_router_gradient_matches_its_oracle(T, E, k):
    """Against the formula in float64; bound: k products and sums of fp32 in the dot product, two more operations behind it."""
    from rocm_systems_b200 import _lib
    from rocm_systems_b200.ops import train_ops as ops
    from rocm_systems_b200.parallel.ep import _lib_ep, router_backward

    g = torch.Generator(device="cuda").manual_seed(T + E)
    idx = torch.argsort(torch.randn(T, E, device="cuda", generator=g), dim=-1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn(T, k, device="cuda", generator=g), -1)
    d = torch.randn(T, k, device="cuda", generator=g)
    out = torch.full((T, E), 7.0, device="cuda")
    _lib.check(_lib_ep().b200collEpRouterGrad(w.data_ptr(), idx.data_ptr(), d.data_ptr(), out.data_ptr(), T, E, k, ops._s()), "b200collEpRouterGrad")
    torch.cuda.synchronize()
    ref = router_backward(w.double(), idx, d.double(), E)
    size = (d.abs() + (d * w).abs().sum(-1, keepdim=True)).double().amax(-1, keepdim=True)
    assert bool(((out.double() - ref).abs() <= (k + 3) * 2.0 ** -23 * size).all())
    selected = torch.zeros(T, E, dtype=torch.bool, device="cuda").scatter_(1, idx.long(), True)
    assert not bool(out[~selected].any())
