"""The launches around the GEMMs at the sizes where their routes and tiles change (csrc/router.cu, route.cu, permute.cu, quant.cu,
w4.cu), and the compiled call paths (csrc/calls.cpp) against the Python functions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.contiguous().view({1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[t.element_size()])


# one launch up to 65536 slots, chunks of 1024; three launches beyond.  Some ids lie outside [0, E).
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025, 5000, 65535, 65536, 65537])
@pytest.mark.parametrize("E", [1, 7, 256, 1024])
def test_sort_is_stable_at_its_chunk_edges(n, E):
    from llm_kernels_b200.moe import group_gemm_kernel as G
    g = torch.Generator().manual_seed(n + E)
    ids = torch.randint(-1, E + 1, (n,), generator=g)
    ids[::3] = int(torch.randint(0, E, (1,), generator=g))          # one expert with a third of the slots
    order, dst, seg = (t.cpu() for t in G.run_moe_ep_preproess(ids.cuda(), E))
    ok = (ids >= 0) & (ids < E)
    slots = ok.nonzero().view(-1)
    rows = slots[torch.sort(ids[slots], stable=True)[1]]
    want = torch.full((n,), -1, dtype=torch.int32)
    want[rows] = torch.arange(len(rows), dtype=torch.int32)
    assert torch.equal(dst, want) and torch.equal(order[:len(rows)], ids[rows])
    assert torch.equal(seg, torch.cat([torch.zeros(1, dtype=torch.int64), torch.bincount(ids[slots], minlength=E).cumsum(0)]))


def test_sort_opts_in_to_shared_memory_in_time():
    """Static and dynamic shared memory together leave the default limit at 681 experts.  A process of its own: once a kernel has
    been opted in, the limit stays raised."""
    import os
    import subprocess
    import sys
    code = ("import torch\n"
            "from llm_kernels_b200.moe import group_gemm_kernel as G\n"
            "for E in (680, 681, 682, 683):\n"
            "    ids = torch.arange(64).mul(37) % E\n"
            "    order, dst, seg = (t.cpu() for t in G.run_moe_ep_preproess(ids.cuda(), E))\n"
            "    want, rows = torch.sort(ids, stable=True)\n"
            "    assert torch.equal(order, want) and torch.equal(dst[rows], torch.arange(64, dtype=torch.int32)), E\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr


def test_a_refused_launch_is_not_reported_by_the_next():
    from llm_kernels_b200 import _native as N
    lib = N.lib()
    x = torch.randn(2, 2048, device="cuda").to(torch.bfloat16)
    y, s = torch.zeros(2, 2048, dtype=torch.uint8, device="cuda"), torch.zeros(2, 16, device="cuda")

    def quant(rows):
        return lib.b200moe_act_quant_fp8(x.data_ptr(), N.BF16, rows, 2048, y.data_ptr(), 2048, s.data_ptr(), 16, N.stream())
    assert quant(1 << 33) == 6              # 2^32 blocks, which a 32-bit count holds as none: the runtime launches nothing
    assert not y.any() and quant(2) == 0 and y.any()


# registers per lane 1, 8 and 32; groups that do and do not divide the 32 lanes; more splits than loads in flight
@pytest.mark.parametrize("T", [1, 8, 9])
@pytest.mark.parametrize("E,groups,kept,k,splits", [(8, 1, 1, 2, 1), (32, 4, 2, 4, 9), (48, 3, 2, 5, 3), (256, 8, 4, 8, 16),
                                                    (257, 1, 1, 8, 2), (1024, 32, 7, 32, 1)])
@pytest.mark.parametrize("scoring", [0, 1])
def test_selection_from_partial_sums(T, E, groups, kept, k, splits, scoring):
    from llm_kernels_b200 import _native as N
    g = torch.Generator().manual_seed(E + T)
    stride = E + 3
    part = torch.randn(splits, T, stride, generator=g) * 0.01
    bias = torch.randint(-40, 40, (E,), generator=g) / 4.0
    idx = torch.empty(T, k, dtype=torch.int64, device="cuda")
    w = torch.empty(T, k, device="cuda")
    pc, bc = part.cuda(), bias.cuda()
    N.check(N.lib().b200moe_router_select(pc.data_ptr(), splits, stride, bc.data_ptr(), T, E, k, groups, kept, scoring, 1, 1.5,
                                          idx.data_ptr(), w.data_ptr(), N.stream()))
    logits = part[..., :E].double().sum(0)
    score = logits.sigmoid() if scoring == 0 else logits.softmax(-1)
    choice = score + bias.double()
    sure = torch.ones(T, dtype=torch.bool)
    if groups > 1:
        gs = choice.view(T, groups, -1).topk(2, dim=-1)[0].sum(-1)
        best, order = torch.sort(gs, dim=-1, descending=True, stable=True)
        sure = best[:, kept - 1] - best[:, kept] > 1e-5             # f32 could keep either group otherwise
        keep = torch.zeros_like(gs, dtype=torch.bool).scatter_(1, order[:, :kept], True)
        choice = torch.where(keep.repeat_interleave(E // groups, 1), choice, 0.0)
    gap, want = torch.sort(choice, dim=-1, descending=True, stable=True)
    for t in range(T):
        # picks are compared up to the first pair that f32 could order either way
        close = ((gap[t, :k] - gap[t, 1:k + 1]) < 1e-5).nonzero().view(-1) if k < E else torch.tensor([], dtype=torch.int64)
        n = (int(close[0]) if len(close) else k) if sure[t] else 0
        got = idx[t].cpu()
        assert torch.equal(got[:n], want[t, :n])
        ref = score[t, got] / (score[t, got].sum() + 1e-20) * 1.5
        # a few f32 roundings of the scores and of their sum of up to 32 terms
        assert float(((w[t].cpu().double() - ref) / ref).abs().max()) < 40 * 2 ** -23


# a thread per expert for one token (or what fits beside it), a warp per token otherwise; 1, 8, 16 and 32 experts a lane
@pytest.mark.parametrize("E,groups,kept", [(8, 1, 1), (33, 1, 1), (64, 4, 2), (128, 1, 1), (255, 5, 2), (256, 8, 4), (257, 1, 1), (384, 1, 1),
                                           (512, 8, 4), (513, 1, 1), (1024, 32, 7)])
@pytest.mark.parametrize("splits", [1, 3, 16])
@pytest.mark.parametrize("scoring", [0, 1])
def test_selection_does_not_depend_on_the_batch(E, groups, kept, splits, scoring):
    """The sums run in the order of the splits in either form: the same bits."""
    from llm_kernels_b200 import _native as N
    g = torch.Generator(device="cuda").manual_seed(E)
    T, k, stride = 13, min(8, E), E + 3
    part = torch.randn(splits, T, stride, generator=g, device="cuda")
    bias = torch.randn(E, generator=g, device="cuda")

    def select(part):
        n = part.shape[1]
        idx, w = torch.full((n, k), -1, dtype=torch.int64, device="cuda"), torch.full((n, k), -1.0, device="cuda")
        N.check(N.lib().b200moe_router_select(part.data_ptr(), splits, stride, bias.data_ptr(), n, E, k, groups, kept, scoring, 1, 2.5,
                                              idx.data_ptr(), w.data_ptr(), N.stream()))
        return idx, w
    whole = select(part)
    for n in (1, 2, 3, 5):
        for t in range(0, T - n + 1, n):
            for a, b in zip(whole, select(part[:, t:t + n].contiguous())):
                assert torch.equal(_bits(a[t:t + n]), _bits(b))


@pytest.mark.parametrize("T", [1, 2])
@pytest.mark.parametrize("H,E", [(64, 128), (1088, 128), (7168, 256)])
def test_router_logits_of_few_tokens(T, H, E):
    """Against 64 bits.  The f32 weight is exactly the sum of its parts; a lane adds H / 128 products, then 8 sums follow: as many
    roundings of partial sums at most, each below the sum of the products' sizes."""
    from llm_kernels_b200 import _native as N
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16)
    w = torch.randn(E, H, generator=g) * 0.02
    hi = w.to(torch.bfloat16)
    mid = (w - hi.float()).to(torch.bfloat16)
    lo = (w - hi.float() - mid.float()).to(torch.bfloat16)
    w3 = torch.cat([hi, mid, lo], 1).cuda()
    assert N.lib().b200moe_router_ksplits(T, H, E) == 1
    part = torch.full((T, E), float("nan"), device="cuda")
    xc = x.cuda()
    N.check(N.lib().b200moe_router_logits_bf16x3(xc.data_ptr(), w3.data_ptr(), part.data_ptr(), T, H, E, 1, N.stream()))
    exact = x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t()
    assert float(((part.cpu().double() - exact).abs() / size).max()) < (H / 128 + 9) * 2 ** -24


# a block per round of columns, one block per token from 1025 (quantizers) or 4097 tokens on; rows that end inside a warp
@pytest.mark.parametrize("T", [1, 3, 511, 512, 1024, 1025, 4096, 4097])
@pytest.mark.parametrize("H", [128, 2176, 7168])
@pytest.mark.parametrize("topk", [1, 5, 8])
def test_permute_and_unpermute(T, H, topk):
    from llm_kernels_b200 import _native as N
    from llm_kernels_b200.quantization import fp8_kernel, int8_kernel
    g = torch.Generator(device="cuda").manual_seed(H)
    E, S = 16, T * topk
    x = torch.randn(T, H, generator=g, device="cuda").to(torch.bfloat16)
    ids = torch.rand(T, E, generator=g, device="cuda").topk(topk, dim=1)[1]
    dst = torch.randperm(S, generator=g, device="cuda").to(torch.int32).view(T, topk)
    lo, hi = 2, 13                                                   # some slots belong to other ranks
    here = (ids >= lo) & (ids <= hi)
    rows = dst[here].long()
    src = torch.arange(T, device="cuda").view(T, 1).expand(T, topk)[here]
    for name, quant, stride in (("fp8", fp8_kernel.act_quant, H + 8), ("fp8", fp8_kernel.act_quant, H + 16),
                                ("int8", lambda v: int8_kernel.act_quant(v, rounding="floor_half"), H + 8)):
        out = torch.zeros(S, stride, dtype=torch.uint8, device="cuda")
        s = torch.zeros(S, H // 128 + 1, device="cuda")
        fn = getattr(N.lib(), f"b200moe_permute_quant_{name}")
        tail = (1,) if name == "int8" else ()
        N.check(fn(x.data_ptr(), N.BF16, dst.data_ptr(), ids.data_ptr(), lo, hi, T, topk, H, out.data_ptr(), stride, s.data_ptr(),
                   H // 128 + 1, *tail, N.stream()))
        q, qs = quant(x)
        want = torch.zeros_like(out)
        want[rows, :H] = _bits(q)[src]
        want_s = torch.zeros_like(s)
        want_s[rows, :H // 128] = qs.float()[src]
        assert torch.equal(out, want) and torch.equal(s, want_s)
    down = torch.randn(S, H, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.rand(T, topk, generator=g, device="cuda")
    y = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().b200moe_post_reorder(down.data_ptr(), N.BF16, y.data_ptr(), dst.data_ptr(), ids.data_ptr(), w.data_ptr(), lo, hi,
                                         T, topk, H, N.stream()))
    acc = torch.zeros(T, H, dtype=torch.float64, device="cuda")
    for j in range(topk):                                            # the kernel's f32 multiply-adds, in 64 bits and rounded
        acc = torch.where(here[:, j:j + 1], (acc + down[dst[:, j].long()].double() * w[:, j:j + 1].double()).float().double(), acc)
    assert torch.equal(y, acc.float().to(torch.bfloat16))


@pytest.mark.parametrize("rows,cols", [(1, 128), (3, 384), (129, 2176)])
@pytest.mark.parametrize("pad", [0, 8, 16])
def test_fp8_quantizer_rows_of_any_stride(rows, cols, pad):
    from llm_kernels_b200 import _native as N
    from oracle import restate as R
    x = torch.randn(rows, cols, generator=torch.Generator().manual_seed(cols)).to(torch.bfloat16)
    xc = x.cuda()
    y = torch.zeros(rows, cols + pad, dtype=torch.uint8, device="cuda")
    s = torch.zeros(rows, cols // 128 + (pad > 0), device="cuda")
    N.check(N.lib().b200moe_act_quant_fp8(xc.data_ptr(), N.BF16, rows, cols, y.data_ptr(), cols + pad, s.data_ptr(), s.shape[1], N.stream()))
    q, qs = R.act_quant_fp8(x)
    assert torch.equal(y[:, :cols].cpu(), _bits(q)) and torch.equal(s[:, :cols // 128].cpu(), qs)
    assert not y[:, cols:].any() and not s[:, cols // 128:].any()


@pytest.mark.parametrize("N_,K", [(8, 128), (40, 384), (264, 2176)])
def test_int4_expansions_for_every_scale(N_, K):
    """All int8 scales and zero points (the products wrap), and the asymmetric format with zero points that are no whole numbers."""
    from llm_kernels_b200.quantization import w4a8_kernel, w4a16_kernel
    g = torch.Generator().manual_seed(K)
    q = torch.randint(0, 16, (N_, K), generator=g)
    s4, z4 = (torch.randint(-128, 128, (N_, K // 128), dtype=torch.int8, generator=g) for _ in range(2))
    packed = sum(q.view(N_ // 8, 8, K)[:, c] << (4 * c) for c in range(8)).to(torch.int32)
    want = ((q - z4.long().repeat_interleave(128, 1)) * s4.long().repeat_interleave(128, 1)).to(torch.int8)
    assert torch.equal(w4a8_kernel.expand_int8(packed.cuda(), s4.cuda(), z4.cuda()).cpu(), want)
    words = sum(q.view(N_, K // 8, 8)[..., j] << (4 * j) for j in range(8)).to(torch.int32)
    sc, zp = (torch.rand(N_, K // 128, generator=g) * m for m in (0.1, 15.0))
    sc, zp = sc.to(torch.bfloat16), zp.to(torch.bfloat16)
    wide = lambda t: t.float().repeat_interleave(128, 1)
    want = ((q.float() - wide(zp)) * wide(sc)).to(torch.bfloat16)
    assert torch.equal(w4a16_kernel.expand_bf16(words.cuda(), sc.cuda(), zp.cuda()).cpu(), want)


@pytest.mark.parametrize("M", [1, 24, 128, 129])
@pytest.mark.parametrize("N_,K", [(256, 128), (384, 1152)])
def test_compiled_calls_give_what_the_python_functions_give(M, N_, K, monkeypatch):
    from llm_kernels_b200 import _native as N
    from llm_kernels_b200.quantization import fp8_kernel, w4a8_kernel

    class NotTaken:
        def __getattr__(self, name):
            return lambda *args: None

    def run():
        out = []
        g = torch.Generator(device="cuda").manual_seed(3)
        x = torch.randn(2, M, K, generator=g, device="cuda").to(torch.bfloat16)
        w = torch.randn(N_, K, generator=g, device="cuda") * 0.02
        for mod, gemm in ((fp8_kernel, fp8_kernel.fp8_gemm), (w4a8_kernel, w4a8_kernel.w4a8_gemm)):
            q, s = mod.act_quant(x)
            weight = mod.weight_quant(w)
            out += [q, s, gemm(q, s, *weight, out_dtype=torch.bfloat16), gemm(q[:1].contiguous(), s[:1].contiguous(), *weight)]
            if mod is w4a8_kernel:
                out.append(gemm(q, s.float(), weight[0], weight[1].float(), *weight[2:], out_dtype=torch.float16))
        return out
    fast = run()
    monkeypatch.setattr(N, "_calls_module", NotTaken())
    for a, b in zip(fast, run()):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(_bits(a), _bits(b))


def test_compiled_calls_leave_what_they_do_not_take():
    from llm_kernels_b200 import _native as N
    f8 = torch.float8_e4m3fn
    x = torch.zeros(4, 256, device="cuda", dtype=torch.bfloat16)
    a, s, b, bs = x.to(f8), torch.ones(4, 2, device="cuda"), torch.zeros(256, 256, device="cuda").to(f8), torch.ones(2, 2, device="cuda")
    c = N.calls()
    assert c.act_quant(x, 0) is not None and c.fp8_gemm(a, s, b, bs, torch.bfloat16, 1) is not None
    for bad in (x.cpu(), x.t(), x[:, ::2], x.double(), x[:, :100].contiguous(), None, x[0, 0]):
        assert c.act_quant(bad, 0) is None
    for i, bad in ((0, a.t()), (0, x), (1, s.double()), (2, b.t()), (3, bs.cpu()), (4, torch.int8), (4, None), (0, a[:0])):
        args = [a, s, b, bs, torch.bfloat16, 1]
        args[i] = bad
        assert c.fp8_gemm(*args) is None
    assert type(c.fp8_gemm(a, s, b, bs, torch.bfloat16, 3)) is int          # an empty split: the library's status
    for ks in (2 ** 31, 2 ** 70, -2 ** 70, 2.0, None):                      # no C int
        assert c.fp8_gemm(a, s, b, bs, torch.bfloat16, ks) is None


@pytest.mark.parametrize("kind", ["act_quant", "fp8_gemm", "w4a8_gemm"])
def test_compiled_calls_let_other_threads_run(kind):
    """A launch that waits for room in the queue does so without the interpreter.  The queue is held by a sleep of about 0.8 s; a
    second thread notes the longest time that it could not run."""
    import threading
    import time
    from llm_kernels_b200.quantization import fp8_kernel, w4a8_kernel
    x = torch.randn(16, 256, device="cuda").to(torch.bfloat16)
    w = torch.randn(256, 256, device="cuda")
    mod = w4a8_kernel if kind == "w4a8_gemm" else fp8_kernel
    q, s = mod.act_quant(x)
    weight = mod.weight_quant(w)
    call = {"act_quant": lambda: mod.act_quant(x), "fp8_gemm": lambda: fp8_kernel.fp8_gemm(q, s, *weight),
            "w4a8_gemm": lambda: w4a8_kernel.w4a8_gemm(q, s, *weight)}[kind]
    call()
    torch.cuda.synchronize()
    done, longest_gap = threading.Event(), [0.0]

    def ticker():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.002)
            now = time.perf_counter()
            longest_gap[0], last = max(longest_gap[0], now - last), now
    thread = threading.Thread(target=ticker)
    thread.start()
    torch.cuda._sleep(1_500_000_000)
    waited, began = 0.0, time.perf_counter()
    while waited < 0.1 and time.perf_counter() - began < 3:       # until one call has waited for the queue
        t = time.perf_counter()
        call()
        waited = time.perf_counter() - t
    done.set()
    thread.join()
    torch.cuda.synchronize()
    assert waited >= 0.1, "no call met a full queue"
    assert longest_gap[0] < waited / 2
