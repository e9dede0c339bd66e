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
