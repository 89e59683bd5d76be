"""AdamW of an embedding table split into rows with and without a token, against the dense update."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab,H,T,repeat", [(5, 8, 1, False), (1000, 1032, 300, False), (64, 64, 64, False), (3000, 4096, 513, True), (7, 2048, 100, True)])
def test_row_updates_match_the_dense_update(vocab, H, T, repeat):
    """Distinct tokens: bit-equal to the dense update. Repeated ones: the gradient g is an fp32 sum of up to T terms of one sign in an order
    that varies, so two sums differ by at most d = 2 T 2^-24 g; then the first moments differ by 0.1 d, the second by 0.05 (2 g + d) d,
    plus fp32 roundings. The weights only follow them (their step is lr m / sqrt(v), here below 3 lr, with relative changes of 4 d / g at most)."""
    from rocm_systems_b200.ops import train_ops as ops

    g = torch.Generator(device="cuda").manual_seed(vocab + T)
    tok = torch.randint(0, vocab, (T,), device="cuda", generator=g) if repeat else torch.randperm(vocab, device="cuda", generator=g)[:T]
    dout = torch.randn(T, H, device="cuda", generator=g).abs().to(torch.bfloat16)     # of one sign: no cancellation in the sums
    n, pad = vocab * H, 64
    state = [torch.randn(n + pad, device="cuda", generator=g) for _ in range(3)]
    state[2] = state[2].abs()
    a, b = [s.clone() for s in state], [s.clone() for s in state]
    pa, pb = (torch.zeros(n + pad, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    hyper = dict(lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, step=3)
    dense = torch.zeros(vocab, H, device="cuda")
    ops.embedding_bwd_(tok, dout, dense)
    ops.adamw_(a[0][:n], a[1][:n], a[2][:n], dense.view(-1), pa[:n], **hyper)
    owner = ops.embedding_owner(tok, vocab)
    want = torch.full((vocab,), 0x7F7F7F7F, dtype=torch.int64)
    for t in range(T - 1, -1, -1):
        want[int(tok[t])] = t
    assert torch.equal(owner.cpu().long(), want)
    ops.adamw_rows_(b[0], b[1], b[2], pb, owner, H, **hyper)
    drows = torch.zeros(T, H, device="cuda")
    ops.embedding_bwd_owned_(tok, dout, owner, drows)
    ops.adamw_rows_(b[0], b[1], b[2], pb, owner, H, **hyper, tokens=tok, drows=drows)
    torch.cuda.synchronize()
    gmax = float(dense.max())
    d = 2 * T * 2.0 ** -24 * gmax
    bounds = [3e-2 * 4 * 2 * T * 2.0 ** -24 + 1e-6, 0.1 * d + 1e-6, 0.05 * (2 * gmax + d) * d + 1e-6 * gmax * gmax, 2.0 ** -5]   # bf16 copy: one step of a weight below 8
    for x, y, start, tol in zip(a + [pa], b + [pb], state + [torch.zeros_like(pa)], bounds):
        if repeat:
            assert float((x.double() - y.double()).abs().max()) <= tol
        else:
            assert torch.equal(x, y)
        assert torch.equal(y[n:], start[n:])
