"""The launches around the GEMMs at the sizes where their routes and tiles change (csrc/router.cu, route.cu, permute.cu, quant.cu,
w4.cu), and the compiled call paths (csrc/calls.cpp) against the Python functions."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _bits(t):
    return t.contiguous().view({1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[t.element_size()])


def _select(part, bias, E, k, groups, kept, scoring):
    """b200moe_router_select on partial sums [splits, T, stride] -> (idx, weights) on the host."""
    from llm_kernels_b200 import _native as N
    splits, T, stride = part.shape
    pc, bc = part.cuda(), bias.cuda()
    idx, w = torch.full((T, k), -1, dtype=torch.int64, device="cuda"), torch.full((T, k), -1.0, device="cuda")
    N.check(N.lib().b200moe_router_select(pc.data_ptr(), splits, stride, bc.data_ptr(), T, E, k, groups, kept, scoring, 1, 1.5,
                                          idx.data_ptr(), w.data_ptr(), N.stream()))
    return idx.cpu(), w.cpu()


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
    """The biases are spread far wider than f32 rounds, and positive, so that masked experts (0) are out of the question."""
    g = torch.Generator().manual_seed(E + T)
    stride = E + 3
    part = torch.randn(splits, T, stride, generator=g)
    bias = torch.linspace(0.5, 4.5, E)[torch.randperm(E, generator=g)]
    idx, w = _select(part, bias, E, k, groups, kept, scoring)
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
    compared = 0
    for t in range(T):
        assert len(set(idx[t].tolist())) == k
        # a few f32 roundings of the scores and of their sum of up to 32 terms
        ref = score[t, idx[t]] / (score[t, idx[t]].sum() + 1e-20) * 1.5
        assert float(((w[t].double() - ref) / ref).abs().max()) < 40 * 2 ** -23
        if not sure[t]:
            continue
        assert bool((choice[t, idx[t]] > 0).all())                  # of the groups that were kept
        # picks are compared up to the first pair that f32 could order either way
        close = (gap[t, :k] - gap[t, 1:k + 1] < 1e-5).nonzero().view(-1)
        n = int(close[0]) if len(close) else k
        assert torch.equal(idx[t, :n], want[t, :n])
        compared += n == k
    assert compared >= max(1, T - 1)


@pytest.mark.parametrize("T", [1, 9])
@pytest.mark.parametrize("E,groups,kept,k", [(8, 1, 1, 4), (32, 4, 2, 8), (255, 5, 2, 8), (384, 1, 1, 32), (1024, 32, 7, 32)])
@pytest.mark.parametrize("scoring", [0, 1])
def test_selection_takes_the_lower_id_of_equals(T, E, groups, kept, k, scoring):
    """Three different logits over all experts: almost every comparison, of experts and of groups, is a tie."""
    g = torch.Generator().manual_seed(E)
    level = torch.tensor([-1.0, 0.0, 2.0])
    which = torch.randint(0, 3, (1, T, E + 3), generator=g)
    idx, _ = _select(level[which], torch.zeros(E), E, k, groups, kept, scoring)
    choice = (level.sigmoid() if scoring == 0 else level.exp())[which[0, :, :E]]     # orders as the scores do
    if groups > 1:
        gs = choice.view(T, groups, -1).topk(2, dim=-1)[0].sum(-1)
        order = torch.sort(gs, dim=-1, descending=True, stable=True)[1][:, :kept]
        keep = torch.zeros(T, groups, dtype=torch.bool).scatter_(1, order, True)
        choice = torch.where(keep.repeat_interleave(E // groups, 1), choice, 0.0)
    assert torch.equal(idx, torch.sort(choice, dim=-1, descending=True, stable=True)[1][:, :k])


# a thread per expert for one token (or what fits beside it), a warp per token otherwise; 1, 8, 16 and 32 experts a lane
@pytest.mark.parametrize("E,groups,kept", [(8, 1, 1), (33, 1, 1), (64, 4, 2), (128, 1, 1), (255, 5, 2), (256, 8, 4), (257, 1, 1), (384, 1, 1),
                                           (512, 8, 4), (513, 1, 1), (1024, 32, 7)])
@pytest.mark.parametrize("splits", [1, 3, 16])
@pytest.mark.parametrize("scoring", [0, 1])
def test_selection_does_not_depend_on_the_batch(E, groups, kept, splits, scoring):
    """The sums run in the order of the splits in either form: the same bits."""
    g = torch.Generator().manual_seed(E)
    T, k = 13, min(8, E)
    part = torch.randn(splits, T, E + 3, generator=g)
    bias = torch.randn(E, generator=g)
    whole = _select(part, bias, E, k, groups, kept, scoring)
    for n in (1, 2, 3, 5):
        for t in range(0, T - n + 1, n):
            for a, b in zip(whole, _select(part[:, t:t + n].contiguous(), bias, E, k, groups, kept, scoring)):
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


def _split_calls(seed):
    """Quantizers and split GEMMs of a linear layer, their scratch freed as they return: -> a function that gives the outputs."""
    from llm_kernels_b200.quantization import fp8_kernel, w4a8_kernel
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(24, 1152, generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn(384, 1152, generator=g, device="cuda") * 0.02
    up = torch.randn(1152, 384, generator=g, device="cuda") * 0.02
    weights = [(fp8_kernel.weight_quant(w), fp8_kernel.weight_quant(up)), (w4a8_kernel.weight_quant(w), w4a8_kernel.weight_quant(up))]

    def run():
        out = []
        for mod, gemm, pair in ((fp8_kernel, fp8_kernel.fp8_gemm, weights[0]), (w4a8_kernel, w4a8_kernel.w4a8_gemm, weights[1])):
            y = gemm(*mod.act_quant(x), *pair[0], out_dtype=torch.bfloat16)
            out.append(gemm(*mod.act_quant(y), *pair[1], out_dtype=torch.bfloat16))
        return out
    return run


def _alone(run):
    """The same with the device idle between any two launches' calls."""
    from llm_kernels_b200 import _native as N
    calls = N.calls()

    class Waiting:
        def __getattr__(self, name):
            def call(*args):
                out = getattr(calls, name)(*args)
                torch.cuda.synchronize()
                return out
            return call
    N._calls_module = Waiting()
    try:
        return run()
    finally:
        N._calls_module = calls


def test_dependent_launches_keep_the_order_of_the_stream():
    """Short launches one after another, whose scratch and intermediate results are freed and taken again at once: a kernel that
    started before its predecessor was through would read or overwrite what that one still uses.  Eager and captured."""
    run = _split_calls(5)
    want = _alone(run)
    got = [run() for _ in range(50)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = [run() for _ in range(5)]
    for _ in range(10):
        graph.replay()
        got += [[t.clone() for t in out] for out in outs]
    torch.cuda.synchronize()
    for out in got:
        for a, b in zip(out, want):
            assert torch.equal(_bits(a), _bits(b))


@pytest.mark.parametrize("own_streams", [False, True])
def test_split_gemms_of_two_threads_have_scratch_of_their_own(own_streams):
    """Compiled calls of two threads, on one stream or two, with other inputs each: the launches of the two come in any order."""
    import threading
    runs = [_split_calls(seed) for seed in (7, 8)]
    want = [_alone(run) for run in runs]
    got, start = [[], []], threading.Barrier(2)
    torch.cuda.synchronize()

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream() if own_streams else torch.cuda.default_stream()):
            start.wait()
            got[i] = [runs[i]() for _ in range(100)]
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        assert len(got[i]) == 100
        for out in got[i]:
            for a, b in zip(out, want[i]):
                assert torch.equal(_bits(a), _bits(b))
