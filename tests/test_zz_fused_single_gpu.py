"""The fused tensor-parallel and expert-parallel paths on ONE GPU (a communicator of one rank): the tcgen05 GEMM with the
all-gather→GEMM policy and SwiGLU epilogue, the GEMM→reduce-scatter epilogue, staging and reducer, the expert-parallel
dispatch (route, fp8 quantise, row reservation by atomics, stores), grouped expert GEMMs and combine — all against their
plain PyTorch compositions, through the same workers the multi-GPU tests use. The collective part degenerates (nothing
crosses a link), the kernels and their schedules are the real ones.

One rank on its own takes the plain GEMMs for its tensor-parallel calls. So these tests run twice: as a program does, and with
B200COLL_FUSED_ONE_RANK=1, which asks for the kernels of several ranks. The workers check by name that the kernels meant did run.

Each runs in a child process; every device-side wait is limited to 5 s. One rank holds all experts, and the router
kernel wants a multiple of 32 of them, so the expert-parallel runs use 32 local experts."""
import pytest

from test_gpu_fused_multi import _launch

pytestmark = pytest.mark.gpu


def _tp(fused, port, worker, *args, fused_kernels, plain_kernels):
    _launch(1, port, worker, "--expect-kernels", fused_kernels if fused else plain_kernels, *args, timeout=600, extra_env={"B200COLL_FUSED_ONE_RANK": str(int(fused))})


FUSED = pytest.mark.parametrize("fused", [False, True])


@FUSED
def test_tensor_parallel_mlp_on_one_rank(fused):
    """256 and 512 rows (the few-row kernels as plain GEMMs); a gate/up weight in tiles of 128 columns."""
    bf16 = dict(fused_kernels="agGemmKernel,gemmRsKernel", plain_kernels="gemmNarrowKernel")
    _tp(fused, 29881, "tp_worker.py", **bf16)
    _tp(fused, 29882, "tp_worker.py", "--rows", "512", "--hidden", "2048", "--ffn", "1024", **bf16)
    _tp(fused, 29892, "tp_worker.py", "--rows", "128", "--hidden", "1152", "--ffn", "576", **bf16)


@FUSED
def test_tensor_parallel_mlp_fp8_on_one_rank(fused):
    """Both fused kernels on block-scaled e4m3 operands against the PyTorch statement of the same arithmetic."""
    fused_kernels = "agGemmFp8Kernel,gemmRsFp8Kernel"
    _tp(fused, 29885, "tp_worker.py", "--fp8", fused_kernels=fused_kernels, plain_kernels="gemmNarrowFp8Kernel")
    _tp(fused, 29886, "tp_worker.py", "--fp8", "--rows", "512", "--hidden", "2048", "--ffn", "1024", fused_kernels=fused_kernels,
        plain_kernels="agGemmFp8Kernel,gemmFp8BlockKernel")     # neither few rows nor enough tiles for pairs


@FUSED
def test_tensor_parallel_layer_forward_and_backward_on_one_rank(fused):
    """Forward and backward of the whole tensor-parallel layer, and of the MLP half at a second shape, against float64 autograd."""
    bf16 = dict(fused_kernels="agGemmKernel,gemmRsKernel", plain_kernels="gemmNarrowKernel")
    _tp(fused, 29888, "tp_layer_worker.py", **bf16)
    _tp(fused, 29889, "tp_layer_worker.py", "--what", "mlp", "--rows", "512", "--hidden", "2048", "--ffn", "1024", **bf16)


def test_expert_parallel_layer_on_one_rank():
    _launch(1, 29883, "ep_worker.py", "--experts-local", "32", timeout=600)


def test_expert_parallel_layer_backward_on_one_rank():
    _launch(1, 29880, "ep_worker.py", "--experts-local", "32", "--backward", timeout=600)


def test_expert_parallel_layer_with_fp8_experts_on_one_rank():
    """The first expert GEMM on the received e4m3 rows and block-quantised weights (no dequantisation pass)."""
    _launch(1, 29887, "ep_worker.py", "--experts-local", "32", "--fp8-experts", timeout=600)


def test_device_initiated_layer_on_one_pe():
    """put+signal to itself, the atomics on its own words, the barrier of one: the device API's code paths on one GPU."""
    _launch(1, 29884, "shmem_worker.py", timeout=600)


@FUSED
def test_tensor_parallel_mlp_on_one_rank_at_the_plain_gemms_sizes(fused):
    """Sizes that the plain CTA-pair GEMMs with the SwiGLU epilogue take on one rank (more than a round of 256 x 256 tiles, an odd number of
    128-row blocks, a reduction that is no multiple of 256)."""
    _tp(fused, 29890, "tp_worker.py", "--rows", "640", "--hidden", "1152", "--ffn", "4224", fused_kernels="agGemmKernel,gemmRsKernel", plain_kernels="gemmPairKernel")
    _tp(fused, 29891, "tp_worker.py", "--fp8", "--rows", "1152", "--hidden", "1152", "--ffn", "3200", fused_kernels="agGemmFp8Kernel,gemmRsFp8Kernel",
        plain_kernels="gemmFp8PairKernel")
