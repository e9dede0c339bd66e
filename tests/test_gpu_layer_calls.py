"""The one-call layer pass against the separate launches, and where passes, streams and graphs meet."""
from dataclasses import replace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(method="fp8_block", act="silu", shared=0, tokens=37, hidden=512, inter=256, seed=3):
    """(layer with seeded weights, tokens)."""
    from llm_kernels_b200 import workloads as WL
    from llm_kernels_b200.moe.all2all_moe import DeepseekV3MoE
    dev = torch.device("cuda:0")
    shape = replace(WL.CONFIG0, tokens=tokens, hidden=hidden, inter=inter, seed=seed, method=method)
    cfg = WL.make_config(shape)
    cfg.hidden_act, cfg.n_shared_experts = act, shared
    layer = DeepseekV3MoE(cfg, device=dev).eval()
    WL.fill_layer_cpu_seeded(layer, shape)
    if shared:
        g = torch.Generator().manual_seed(seed)
        wide = inter * shared
        layer.load_shared_experts(*[(torch.randn(*s, generator=g) * 0.05).to(torch.bfloat16).to(dev)
                                    for s in ((wide, hidden), (wide, hidden), (hidden, wide))])
    return layer, WL.tokens(shape).to(dev).view(1, tokens, hidden)


def _separate(layer, x):
    """The same pass as one launch after the other."""
    layer.stage_events = []
    y = layer(x).clone()
    assert any(name == "post_reorder" for name, _ in layer.stage_events)
    layer.stage_events = None
    return y


@pytest.mark.parametrize("method", ["fp8_block", "w4a16", "w4a8"])
@pytest.mark.parametrize("act,shared", [("silu", 0), ("gelu", 0), ("silu", 2), ("gelu", 1)])
@pytest.mark.parametrize("tokens", [1, 37, 130, 768])
def test_one_call_pass_is_bit_identical_to_separate_launches(method, act, shared, tokens):
    """One row in all, few and many rows per expert, shared experts in single CTAs and in pairs (768 rows, hidden 2048)."""
    layer, x = _layer(method, act, shared, tokens, hidden=2048 if tokens == 768 else 512)
    y = layer(x).clone()
    assert layer._native is not None
    layer._native = None
    assert torch.equal(y, _separate(layer, x)) and layer._native is None
    layer.check_status()


def test_one_call_pass_after_changes():
    """Weights loaded in place, a replaced router weight and a changed setting: the next pass has them."""
    layer, x = _layer("w4a8")
    other, _ = _layer("w4a8", seed=8)
    seen = [layer(x).clone()]
    for name, t in layer.named_buffers():
        t.copy_(dict(other.named_buffers())[name])
    seen.append(layer(x).clone())
    layer.gate.weight = torch.nn.Parameter(other.gate.weight.detach().clone())
    seen.append(layer(x).clone())
    assert torch.equal(seen[-1], other(x))
    layer.gate.routed_scaling_factor = 2.0
    seen.append(layer(x).clone())
    assert torch.equal(seen[-1], _separate(layer, x))
    assert not any(torch.equal(a, b) for a, b in zip(seen, seen[1:]))
    layer.w13_s4[0, 0, 0], layer.w13_z4[0, 0, 0] = 127, 0         # (q - 0) * 127 leaves int8: only expansion is right
    layer.w13_qweight[0, 0, 0] |= 0xF
    y = layer(x).clone()
    layer.w4_fused_rows_per_group = 0
    assert torch.equal(y, layer(x)) and not layer._raw_nibbles_ok("w13")
    layer.check_status()


def test_refused_pass_leaves_the_side_stream_joined():
    """A launch is refused by the host checks after the shared experts' gate/up has been forked off: a capture around it
    can only end if the side stream has been joined again."""
    layer, x = _layer(shared=1)
    layer(x)
    w = layer.w13_weight
    odd = torch.empty(w.numel() + 16, dtype=torch.uint8, device=w.device)[1:1 + w.numel()]      # contiguous, not 16-byte aligned
    layer.w13_weight = odd.view(w.dtype).view(w.shape)
    with pytest.raises(AssertionError, match="aligned"):
        layer(x)
    graph = torch.cuda.CUDAGraph()
    with pytest.raises(AssertionError, match="aligned"):
        with torch.cuda.graph(graph):
            layer(x)
    layer.w13_weight = w
    assert torch.isfinite(layer(x)).all()
    layer.check_status()


@pytest.mark.parametrize("method", ["fp8_block", "w4a16", "w4a8"])
@pytest.mark.parametrize("what", ["router", "expert"])
def test_graph_follows_weights_loaded_in_place(method, what):
    """The split router weight and the int4 pairs are made from the weights: a replay must not go on with the old ones, nor
    read memory that an eager pass after the change has freed."""
    layer, x = _layer(method)
    other, _ = _layer(method, seed=4)
    run = layer.make_graphed(x)
    out = run.static_output
    before = run(x).clone()
    if what == "router":
        with torch.no_grad():
            layer.gate.weight.copy_(other.gate.weight)
    else:
        for name, t in layer.named_buffers():
            t.copy_(dict(other.named_buffers())[name])
    got = run(x)
    assert got is out
    got = got.clone()
    want = layer(x).clone()
    assert torch.equal(got, want) and not torch.equal(got, before)
    junk = [torch.full((1 << 20,), float("nan"), device=x.device) for _ in range(8)]      # freed memory would be taken by these
    assert torch.equal(run(x), want) and len(junk) == 8
    layer.check_status()


@pytest.mark.parametrize("shared", [0, 1])
def test_passes_of_two_threads_and_streams(shared):
    """Two threads, each on a stream of its own, run one layer on different tokens; a graph of it is replayed beside them."""
    import threading
    layer, x = _layer(shared=shared, tokens=96)
    xs = [x, x.flip(1).contiguous(), x.roll(5, 1).contiguous()]
    want = [layer(t).clone() for t in xs]
    run = layer.make_graphed(xs[2])
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                y = run(xs[2]) if i == 2 else layer(xs[i])
                torch.cuda.current_stream().synchronize()
                if not torch.equal(y, want[i]):
                    wrong.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    layer.check_status()


@pytest.mark.parametrize("tokens", [40, 400])
def test_w4a8_first_pass_can_be_captured(tokens):
    """10 and 100 rows per expert: whether the weights fit the fused GEMMs is not known yet and cannot be asked during a
    capture, so the graph expands them; the bits are the same."""
    layer, x = _layer("w4a8", tokens=tokens)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = layer(x)
    graph.replay()
    torch.cuda.synchronize()
    got = y.clone()
    assert torch.equal(got, layer(x)) and layer._native is not None
    layer.check_status()
