"""The expert GEMMs of the mixture-of-experts layer where their tiles end: few rows (features as MMA rows), many (CTA pairs), experts
without any, one expert with all, counts around the edges of 16, 32, 64, 128 and 256 rows, forward and backward."""
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
