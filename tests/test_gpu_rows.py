"""The GEMMs for few rows per group (csrc/gemm_fp8_rows.cu) against the 128-token tiles of csrc/gemm_fp8.cu, which the
other test files compare with the oracle."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows per group: none, one, around the 16-token steps, a full 64-token chunk and its neighbours
ROWS = [0, 1, 15, 16, 17, 0, 33, 48, 49, 63, 64, 65, 3]


def _operands(rows, N, K, seed):
    from llm_kernels_b200.quantization import fp8_kernel
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    W, M = len(rows), sum(rows)
    a, a_s = fp8_kernel.act_quant(torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16))
    b, b_s = fp8_kernel.weight_quant(torch.randn(W * N, K, generator=g, device=dev) * 0.02)
    seg = torch.tensor([0] + torch.tensor(rows).cumsum(0).tolist(), dtype=torch.int64, device=dev)
    widx = torch.randperm(W, generator=g, device=dev)
    return a, a_s, b.view(W, N, K), b_s.view(W, N // 128, K // 128), seg, widx


@pytest.mark.parametrize("N,K", [(128, 128), (384, 640), (512, 1152)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_rows_kernel_plain_is_bit_identical(N, K, dtype):
    """Same promotion (one FMA per value and K block, in K order), so the same bits."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    a, a_s, b, b_s, seg, widx = _operands(ROWS, N, K, 1)
    c = torch.empty(a.shape[0], N, dtype=dtype, device=a.device)
    want = torch.empty_like(c)
    G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, c)
    with G.gemm_options():
        G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, want)
    assert torch.equal(c, want)


@pytest.mark.parametrize("epilogue", [1, 4])
@pytest.mark.parametrize("N,K", [(256, 128), (768, 640)])
def test_rows_kernel_fused_is_bit_identical(N, K, epilogue):
    from llm_kernels_b200.moe import group_gemm_kernel as G
    a, a_s, b, b_s, seg, widx = _operands(ROWS, N, K, 2)
    M = a.shape[0]
    out = [(torch.empty(M, N // 2, dtype=torch.uint8, device=a.device), torch.empty(M, N // 256, device=a.device)) for _ in range(2)]
    G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, *out[0], epilogue=epilogue)
    with G.gemm_options():
        G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, *out[1], epilogue=epilogue)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
