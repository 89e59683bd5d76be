"""AdamW of an embedding table split into rows with and without a token, against the dense update: the kernels by themselves and inside
the training step, where the rows without a token are updated on the communication stream beside the backward pass."""
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


def _embedding_after(rows_from, batches, overlap):
    from rocm_systems_b200.models.llama import LlamaConfig, LlamaTrainer
    from rocm_systems_b200.parallel.fsdp import AdamWConfig

    cfg = LlamaConfig.tiny(64)
    t = LlamaTrainer(cfg, None, torch.device("cuda", 0), opt=AdamWConfig(lr=1e-2, weight_decay=0.1), seed=3, overlap=overlap)
    assert t.engine.updates_rows
    t.engine.rows_from = rows_from
    losses = [t.step(tok.pin_memory(), tgt.pin_memory()) for tok, tgt in batches]
    torch.cuda.synchronize()
    return losses, [x.clone() for x in (t.embed.master, t.embed.m, t.embed.v, t.embed.shard)]


@pytest.mark.parametrize("overlap", [True, False])
def test_training_steps_with_row_updates_equal_those_with_the_dense_update(overlap):
    """Four steps whose batches hold each id once, out of ids that come and go between the steps (a row is idle in one step and owned in the
    next, with moments that decay and weights that decay): master, moments and bf16 weights of the embedding are bit-equal."""
    g = torch.Generator().manual_seed(1)
    batches = [(torch.randperm(400, generator=g)[:128].view(2, 64), torch.randint(0, 1024, (2, 64), generator=g)) for _ in range(4)]
    assert any(set(a[0].flatten().tolist()) & set(b[0].flatten().tolist()) for a, b in zip(batches, batches[1:]))
    dense, rows = _embedding_after(float("inf"), batches, overlap), _embedding_after(0, batches, overlap)
    assert dense[0] == rows[0]
    for x, y in zip(dense[1], rows[1]):
        assert torch.equal(x, y)


def test_a_training_step_with_repeated_ids():
    """One step of a batch of few ids, each many times: the rows without a token are bit-equal to the dense update's, the others are rows whose
    fp32 sums depend on the order of the atomics on both paths (bounded in the test of the kernels) and have all moved."""
    g = torch.Generator().manual_seed(2)
    tok = torch.randint(0, 7, (2, 64), generator=g)
    batches = [(tok, torch.randint(0, 1024, (2, 64), generator=g))]
    (_, dense), (_, rows) = _embedding_after(float("inf"), batches, True), _embedding_after(0, batches, True)
    owned = torch.zeros(1024, dtype=torch.bool)
    owned[tok.flatten().unique()] = True
    n = 1024 * 256
    for x, y in zip(dense, rows):
        a, b = x[:n].view(1024, 256)[~owned.cuda()], y[:n].view(1024, 256)[~owned.cuda()]
        assert torch.equal(a, b)
    for x in (dense[1], rows[1]):                     # first moments
        assert bool((x[:n].view(1024, 256)[owned.cuda()] != 0).any(1).all()) and not bool(x[:n].view(1024, 256)[~owned.cuda()].any())
