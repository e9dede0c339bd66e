"""The GEMMs for few rows per group (csrc/gemm_fp8_rows.cu, csrc/gemm_w4a16.cu) against the 128-token tiles of
csrc/gemm_fp8.cu, which the other test files compare with the oracle."""
import os
import re

import pytest
import torch

pytestmark = pytest.mark.gpu

# rows per group: none, one, around the 16-token steps, a full 64-token chunk and its neighbours; two chunks and a rest
ROWS = [0, 1, 15, 16, 17, 0, 33, 48, 49, 63, 64, 65, 3, 0, 1, 0, 130, 1, 0, 2, 32, 31, 0, 0, 1, 0]
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "llm_kernels_b200", "csrc")


def _limit():
    """Rows per group on average up to which fp8 products take the kernel under test."""
    return int(re.search(r"kMaxRowsPerGroup = (\d+);", open(os.path.join(CSRC, "gemm_rows.cuh")).read()).group(1))


def _bits(t):
    return t.view({2: torch.int16, 4: torch.int32}[t.element_size()])


def _operands(rows, N, K, seed):
    """Every eleventh row is zero, whose e4m3 codes are NaN with a scale of zero."""
    from llm_kernels_b200.quantization import fp8_kernel
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    W, M = len(rows), sum(rows)
    x = torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
    x[5::11] = 0
    a, a_s = fp8_kernel.act_quant(x)
    b, b_s = fp8_kernel.weight_quant(torch.randn(W * N, K, generator=g, device=dev) * 0.02)
    seg = torch.tensor([0] + torch.tensor(rows).cumsum(0).tolist(), dtype=torch.int64, device=dev)
    widx = torch.randperm(W, generator=g, device=dev)
    return a, a_s, b.view(W, N, K), b_s.view(W, N // 128, K // 128), seg, widx


@pytest.mark.parametrize("N,K", [(128, 128), (384, 640), (512, 1152)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
def test_rows_kernel_plain_is_bit_identical(N, K, dtype):
    """Same promotion (one FMA per value and K block, in K order), so the same bits."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    assert sum(ROWS) <= _limit() * len(ROWS)                     # else both calls run the same kernel
    a, a_s, b, b_s, seg, widx = _operands(ROWS, N, K, 1)
    c = torch.empty(a.shape[0], N, dtype=dtype, device=a.device)
    want = torch.empty_like(c)
    G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, c)
    with G.gemm_options():
        G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, want)
    assert torch.equal(_bits(c), _bits(want))


@pytest.mark.parametrize("groups", [1, 3])
@pytest.mark.parametrize("more", [0, 1])
def test_rows_kernel_at_its_limit(groups, more):
    """The last number of rows that takes the kernel and the first that does not, against 64-bit sums: e4m3 products are exact,
    so what is left are the roundings of K / 128 scaled block sums and of the f32 sum inside the tensor core."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    rows = [_limit()] * groups
    rows[-1] += more
    a, a_s, b, b_s, seg, widx = _operands(rows, 384, 640, 5)
    a = torch.where(a_s.repeat_interleave(128, -1) > 0, a.float(), 0.0).to(a.dtype)
    c = G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, torch.empty(a.shape[0], 384, device=a.device))
    wide = lambda t, s: t.double() * s.double().repeat_interleave(128, -1)
    for i in range(groups):
        w = int(widx[i])
        want = wide(a[seg[i]:seg[i + 1]], a_s[seg[i]:seg[i + 1]]) @ wide(b[w], b_s[w].repeat_interleave(128, 0)).t()
        assert float((c[seg[i]:seg[i + 1]] - want).norm() / want.norm()) < 1e-4


@pytest.mark.parametrize("epilogue", [1, 4])
@pytest.mark.parametrize("N,K", [(256, 128), (768, 640)])
def test_rows_kernel_fused_is_bit_identical(N, K, epilogue):
    from llm_kernels_b200.moe import group_gemm_kernel as G
    assert sum(ROWS) <= _limit() * len(ROWS)
    a, a_s, b, b_s, seg, widx = _operands(ROWS, N, K, 2)
    M = a.shape[0]
    out = [(torch.empty(M, N // 2, dtype=torch.uint8, device=a.device), torch.empty(M, N // 256, device=a.device)) for _ in range(2)]
    G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, *out[0], epilogue=epilogue)
    with G.gemm_options():
        G.grouped_gemm_fp8(a, a_s, b, b_s, seg, widx, *out[1], epilogue=epilogue)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(_bits(out[0][1]), _bits(out[1][1]))


@pytest.mark.parametrize("whole_zeros", [True, False])
@pytest.mark.parametrize("rows", [ROWS, [0, 129, 64, 200, 128, 17, 127, 0]])
@pytest.mark.parametrize("N,K", [(128, 128), (384, 640), (512, 1024)])
def test_w4a16_kernel_is_bit_identical(N, K, rows, whole_zeros):
    """Both token-chunk widths, K with and without a half-filled 256-k slot, whole zero points (one subtraction per pair)
    and others (the general conversion): the same bf16 weights and the same K order, so the same bits as expanding the
    weights first."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    from llm_kernels_b200.quantization import w4a16_kernel
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(3)
    W, M = len(rows), sum(rows)
    packed = torch.randint(-2 ** 31, 2 ** 31, (W, N, K // 8), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    sc = (torch.rand(W, N, K // 128, generator=g, device=dev) * 0.02 + 1e-3).to(torch.bfloat16)
    zp = torch.randint(0, 16, (W, N, K // 128), generator=g, device=dev).to(torch.bfloat16)
    if not whole_zeros:
        zp[:, ::3] += 0.375
        zp[:, 1::7] = -21.0
        sc[:, 2::5] = 2.0 ** -124
    a = torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16)
    seg = torch.tensor([0] + torch.tensor(rows).cumsum(0).tolist(), dtype=torch.int64, device=dev)
    widx = torch.randperm(W, generator=g, device=dev)
    pairs, full = G.pair_scales_t(sc, zp), w4a16_kernel.expand_bf16(packed, sc, zp)
    for epi, cols, dt in ((0, N, torch.float32), (0, N, torch.float16), (2, N // 2, torch.bfloat16), (5, N // 2, torch.bfloat16)):
        if epi and N % 256:
            continue
        c, want = (torch.full((M, cols), float("nan"), dtype=dt, device=dev) for _ in range(2))
        G.grouped_gemm_w4a16(a, packed, pairs, seg, widx, c, epilogue=epi)
        G.grouped_gemm_bf16(a, full, seg, widx, want, epilogue=epi) if dt != torch.float16 else \
            want.copy_(G.grouped_gemm_bf16(a, full, seg, widx, torch.empty(M, cols, dtype=torch.float32, device=dev)))
        assert torch.equal(c, want)


@pytest.mark.parametrize("rows", [ROWS, [128, 0, 129, 95, 1, 32]])
@pytest.mark.parametrize("N,K", [(128, 128), (384, 640), (512, 1152)])
def test_w4a8_kernel_is_bit_identical(N, K, rows):
    """Raw nibbles with the zero point taken off the dot product in exact f32 arithmetic against weights expanded to int8:
    the same bits, with scales and zero points up to the ends of what keeps (q - z) * s inside int8."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    from llm_kernels_b200.quantization import w4a8_kernel
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(4)
    W, M = len(rows), sum(rows)
    packed = torch.randint(-2 ** 31, 2 ** 31, (W, N // 8, K), generator=g, device=dev, dtype=torch.int64).to(torch.int32)
    s4 = torch.randint(-8, 9, (W, N, K // 128), generator=g, device=dev).to(torch.int8)
    z4 = torch.randint(0, 16, (W, N, K // 128), generator=g, device=dev).to(torch.int8)
    s4[:, ::5], z4[:, ::5] = 1, -112                        # 112 .. 127
    s4[:, 1::5], z4[:, 1::5] = 1, 127                       # -127 .. -112
    s4[:, 2::5], z4[:, 2::5] = -1, -112                     # -127 .. -112
    a = torch.randint(-128, 128, (M, K), generator=g, device=dev).to(torch.int8)
    a[::3] = -128                                           # the largest sums
    a_s = torch.rand(M, K // 128, generator=g, device=dev) * 0.01 + 1e-3
    b_s = torch.rand(W, N // 128, K // 128, generator=g, device=dev) * 0.01 + 1e-3
    seg = torch.tensor([0] + torch.tensor(rows).cumsum(0).tolist(), dtype=torch.int64, device=dev)
    widx = torch.randperm(W, generator=g, device=dev)
    for dt in (torch.float32, torch.bfloat16, torch.float16):
        c, want = (torch.full((M, N), float("nan"), dtype=dt, device=dev) for _ in range(2))
        G.grouped_gemm_w4a8(a, a_s, packed, G.pair_scales_t(s4, z4), b_s, seg, widx, c)
        G.grouped_gemm_i8(a, a_s, w4a8_kernel.expand_int8(packed, s4, z4), b_s, seg, widx, want)
        assert torch.equal(c, want)


def test_w4a8_range_check_matches_the_host_form():
    """One scale group at a time is pushed over the end of int8, by its largest, its smallest or no nibble that it holds."""
    from types import SimpleNamespace
    from llm_kernels_b200.moe.all2all_moe import DeepseekV3MoE
    g = torch.Generator().manual_seed(5)
    for n, s, z, lo, hi, want in ((0, 9, 0, 0, 14, True), (9, 9, 0, 0, 15, False), (255, -9, 0, 0, 15, False), (131, 9, 15, 1, 15, True),
                                  (131, 9, 15, 0, 15, False), (7, 1, -113, 0, 14, True), (7, 1, -113, 0, 15, False), (200, -128, 3, 3, 4, True), (200, -128, 3, 2, 3, False)):
        q = torch.randint(0, 16, (1, 256, 384), generator=g)
        q[0, n, 128:256] = torch.randint(lo, hi + 1, (128,), generator=g)
        q[0, n, 130], q[0, n, 255] = lo, hi
        s4 = torch.ones(1, 256, 3, dtype=torch.int8)
        z4 = torch.full((1, 256, 3), 8, dtype=torch.int8)
        s4[0, n, 1], z4[0, n, 1] = s, z
        words = sum(q.view(1, 32, 8, 384)[:, :, i] << (4 * i) for i in range(8))
        packed = torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)
        for dev in ("cpu", "cuda"):
            fake = SimpleNamespace(w13_qweight=packed.to(dev), w13_s4=s4.to(dev), w13_z4=z4.to(dev), _buffers_cache={})
            assert DeepseekV3MoE._raw_nibbles_ok(fake, "w13") == want, (n, s, z, lo, hi, dev)


@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (24, 4096, 7168), (100, 1152, 640), (128, 512, 2048), (129, 512, 2048)])
def test_w4a8_gemm_splits_against_64_bits(M, N, K):
    """The K splits of few rows and the single launch of more: integer dot products are exact, so what is left is the f32
    scaling and sum of K / 128 blocks, at most about sqrt(K / 128) roundings of 6e-8 in the 2-norm."""
    from llm_kernels_b200.quantization import w4a8_kernel
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(6)
    packed, s, s4, z4 = w4a8_kernel.weight_quant(torch.randn(N, K, generator=g, device=dev) * 0.02)
    a, a_s = w4a8_kernel.act_quant(torch.randn(M, K, generator=g, device=dev).to(torch.bfloat16))
    c = w4a8_kernel.w4a8_gemm(a, a_s, packed, s, s4, z4, out_dtype=torch.float32)
    w = w4a8_kernel.expand_int8(packed, s4, z4).double() * s.double().repeat_interleave(128, 0).repeat_interleave(128, 1)
    want = (a.double() * a_s.double().repeat_interleave(128, 1)) @ w.t()
    assert float((c - want).norm() / want.norm()) < 6e-8 * max(4.0, (K / 128) ** 0.5)
