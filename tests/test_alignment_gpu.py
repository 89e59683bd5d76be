"""Misaligned buffers of the grouped and one-rank GEMM entry points: the host refuses them, before anything is launched."""
import pytest
import torch

pytestmark = pytest.mark.gpu

INVALID_ARGUMENT = 4


@pytest.fixture(scope="module")
def comm():
    from rocm_systems_b200.comm import Communicator, get_unique_id

    torch.cuda.set_device(0)
    c = Communicator(0, 1, get_unique_id(), 0)
    yield c
    c.destroy()


@pytest.fixture(scope="module", params=[8, 128])    # rows per expert on average: the few-row kernels, CTA pairs
def layers(comm, request):
    from rocm_systems_b200.parallel.ep import MoELayer

    T = 32 * request.param
    x = torch.randn(T, 1024, device="cuda").to(torch.bfloat16)
    logits = torch.randn(T, 32, device="cuda")
    made = [MoELayer(comm, 32, 1024, 128, 1, T, seed=5, fp8_experts=fp8) for fp8 in (False, True)]
    for m in made:
        m.forward(x, logits)
    made[0].backward(x)
    torch.cuda.synchronize()
    yield made
    for m in made:
        m.free()


def _refused(fn, args, which):
    """`fn` refuses `args` with any one of the pointers numbered in `which` moved by one bf16 element."""
    for i in which:
        moved = list(args)
        moved[i] = moved[i] + 2
        assert fn(*moved) == INVALID_ARGUMENT, i


def test_expert_gemms_refuse_misaligned_buffers(comm, layers):
    from rocm_systems_b200.ops import train_ops as ops
    from rocm_systems_b200.parallel.ep import _lib_ep

    lib, s = _lib_ep(), ops._s()
    m, m8 = layers
    h, dims = comm.handle, m._args()
    dw13, dw2 = (torch.empty_like(t) for t in (m.w13, m.w2))
    p = [t.data_ptr() for t in (m.d_out, m.w13, m.w2, m.xb, m.act, m.gu, m.d_act, dw13, dw2)]
    _refused(lib.b200collEpExpertsBackward, [h, m._win.ptr, *p, *dims, s], range(2, 11))
    _refused(lib.b200collEpExperts, [h, m._win.ptr, m.w13.data_ptr(), m.w2.data_ptr(), m.xb.data_ptr(), m.act.data_ptr(), *dims, s], range(2, 6))
    _refused(lib.b200collEpExpertsFp8, [h, m8._win.ptr, m8.w13_q.data_ptr(), m8.w13_s.data_ptr(), m8.w2.data_ptr(), m8.act.data_ptr(), *dims, s], (2, 4, 5))
    _refused(lib.b200collEpGatherGrad, [h, m._win.ptr, m.out.data_ptr(), m.top_w.data_ptr(), m.d_out.data_ptr(), m.T, m.k, *dims, s], (2, 4))
    _refused(lib.b200collEpGateGrad, [h, m._win.ptr, m.out.data_ptr(), m.top_idx.data_ptr(), m.sent.data_ptr(), m.d_gate.data_ptr(), m.T, m.k, *dims, s], (2,))
    _refused(lib.b200collEpGroupedGemm, [h, m._win.ptr, m.d_out.data_ptr(), m.w13.data_ptr(), m.gu.data_ptr(), 2 * m.ffn, m.hidden, *dims, s], (2, 3, 4))
    torch.cuda.synchronize()
    assert ops.gemm_take_error() == 0


@pytest.mark.parametrize("rows", [128, 640])    # the few-row kernels, CTA pairs
def test_one_rank_gemms_refuse_misaligned_buffers(comm, rows):
    from rocm_systems_b200.ops import train_ops as ops
    from rocm_systems_b200.parallel.tp import TensorParallelMLP, TensorParallelMLPFp8, _lib_tp

    lib, s, h = _lib_tp(), ops._s(), comm.handle
    mlp = TensorParallelMLP(comm, rows, 1024, 512, seed=3)
    x, w13, act, w2, y = (t.data_ptr() for t in (mlp.x_full, mlp.w13, mlp.act, mlp.w2, mlp.y))
    for swiglu in (0, 1):
        _refused(lib.b200collAgGemm, [h, x, w13, act, rows, 1024 if swiglu else 512, 1024, swiglu, 0, s], (1, 2, 3))
    _refused(lib.b200collGemmRs, [h, act, w2, mlp._ws.ptr, y, rows, 1024, 512, s], (1, 2, 4))
    mlp.free()
    m8 = TensorParallelMLPFp8(comm, rows, 1024, 512, seed=3)
    q, qs, out = m8.x_q.data_ptr(), m8.x_s.data_ptr(), m8.act.data_ptr()
    for swiglu in (0, 1):
        _refused(lib.b200collAgGemmFp8, [h, q, qs, m8.w13_q.data_ptr(), m8.w13_s.data_ptr(), out, rows, 1024 if swiglu else 512, 1024, swiglu, 0, s], (1, 3, 5))
    _refused(lib.b200collGemmRsFp8, [h, q, qs, m8.w2_q.data_ptr(), m8.w2_s.data_ptr(), m8._ws.ptr, m8.y.data_ptr(), rows, 1024, 512, s], (1, 3, 6))
    torch.cuda.synchronize()
    m8.free()
    assert ops.gemm_take_error() == 0
