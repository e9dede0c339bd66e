"""What the Python layer hands to the library, seen on the host: the launches are replaced by a recorder (or, where only the
library's argument checks matter, reach the library itself, which checks before it launches)."""
import pytest
import torch


@pytest.fixture
def host(monkeypatch):
    """CPU tensors pass for the current device's."""
    from llm_kernels_b200 import _native as N, build
    build.build()
    monkeypatch.setattr(N, "require_cuda", lambda *tensors: None)
    monkeypatch.setattr(N, "stream", lambda: 0)
    return N


class Recorder:
    """Stands in for the loaded library: every entry point succeeds and is noted; `on` maps names to replacements."""

    def __init__(self, **on):
        self.calls, self.on = [], on

    def __getattr__(self, name):
        def call(*args):
            self.calls.append((name, args))
            return self.on[name](*args) if name in self.on else 0
        return call

    def names(self):
        return [n for n, _ in self.calls]


def _w4a8_operands(M, K, kw, scale_cols):
    """int8 rows of K, a weight of 256 channels x kw, `scale_cols` activation scales per row."""
    return (torch.zeros(M, K, dtype=torch.int8), torch.ones(M, scale_cols), torch.zeros(32, kw, dtype=torch.int32),
            torch.ones(2, kw // 128), torch.ones(256, kw // 128, dtype=torch.int8), torch.ones(256, kw // 128, dtype=torch.int8))


@pytest.mark.parametrize("M", [24, 200])
@pytest.mark.parametrize("K,kw,scale_cols", [(1024, 512, 8), (512, 1024, 4), (1024, 1024, 4)])
def test_w4a8_gemm_refuses_operands_that_disagree(host, monkeypatch, M, K, kw, scale_cols):
    """A weight of another K, or too few activation scales, is refused for few rows as for many."""
    from llm_kernels_b200.quantization import w4a8_kernel
    monkeypatch.setattr(w4a8_kernel, "expand_int8", lambda b, s4, z4: torch.zeros(8 * b.shape[0], b.shape[1], dtype=torch.int8))
    with pytest.raises(AssertionError):
        w4a8_kernel.w4a8_gemm(*_w4a8_operands(M, K, kw, scale_cols))


@pytest.mark.parametrize("M", [24, 200])
def test_w4a8_gemm_reads_wider_scales_by_their_own_stride(host, monkeypatch, M):
    from llm_kernels_b200.quantization import w4a8_kernel
    lib = Recorder()
    monkeypatch.setattr(host, "_lib", lib)
    w4a8_kernel.w4a8_gemm(*_w4a8_operands(M, 1024, 1024, 11))
    name, args = lib.calls[-1]
    assert name == "b200moe_grouped_gemm_i8" and args[3] == 11


@pytest.fixture
def layer_host(host, monkeypatch):
    """make(method) -> (layer on the host, bf16 tokens, recorder of its launches)."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    from llm_kernels_b200.moe.all2all_moe import DeepseekV3MoE
    from llm_kernels_b200.workloads import LayerShape, make_config
    monkeypatch.setattr(G, "_workspace", lambda device, nbytes: torch.empty(1024, dtype=torch.uint8))

    def make(method="fp8_block", cls=DeepseekV3MoE, config={}, **on):
        lib = Recorder(b200moe_layer_workspace_bytes=lambda d, T: 4096, b200moe_router_ksplits=lambda T, H, E: 1, **on)
        monkeypatch.setattr(host, "_lib", lib)
        shape = LayerShape("host", 4, 256, 128, 8, 2, 1, 1, "sigmoid", 1.0, 0, method=method)
        cfg = make_config(shape)
        for name, value in config.items():
            setattr(cfg, name, value)
        layer = cls(cfg, device="cpu").eval()
        return layer, torch.zeros(1, 4, 256, dtype=torch.bfloat16), lib
    return make


@pytest.mark.parametrize("method", ["fp8_block", "w4a16", "w4a8"])
def test_layer_pass_is_one_call(layer_host, method):
    layer, x, lib = layer_host(method)
    assert layer(x).shape == x.shape and lib.names()[-1] == "b200moe_layer_forward"
    assert not any(n.startswith("b200moe_grouped") for n in lib.names())


@pytest.mark.parametrize("method,name,change", [
    ("fp8_block", "w13_weight_scale", lambda t: t.to(torch.bfloat16)),
    ("fp8_block", "w2_weight_scale", lambda t: t.double()),
    ("fp8_block", "w13_weight", lambda t: torch.cat([t.view(torch.uint8)] * 2, dim=2).view(t.dtype)),
    ("w4a16", "w2_scale", lambda t: t.float()),
    ("w4a16", "w13_qweight", lambda t: t.to(torch.int64)),
    ("w4a8", "w2_weight_scale", lambda t: t.half()),
    ("w4a8", "w13_s4", lambda t: torch.cat([t, t], dim=2))])
def test_layer_refuses_weights_of_another_type_or_shape(layer_host, method, name, change):
    """The one-call pass reads raw pointers: what the separate launches refuse must not reach it."""
    layer, x, lib = layer_host(method)
    layer(x)
    setattr(layer, name, change(getattr(layer, name)))
    lib.calls.clear()
    with pytest.raises((AssertionError, RuntimeError)):
        layer(x)
    assert "b200moe_layer_forward" not in lib.names()


def test_layer_refuses_weights_of_another_device_in_every_pass(layer_host, host, monkeypatch):
    """x on the current device is not enough, also once a pass has gone through."""
    layer, x, lib = layer_host()
    current = [x, layer._status, *layer.state_dict(keep_vars=True).values()]

    def require_cuda(*tensors):
        if not all(t is None or any(t.data_ptr() == c.data_ptr() for c in current) for t in tensors):
            raise RuntimeError("not on the current device")
    monkeypatch.setattr(host, "require_cuda", require_cuda)
    layer(x)
    x = torch.ones_like(x)
    current = [x]                                    # the caller has moved on to another device
    with pytest.raises(RuntimeError, match="current device"):
        layer(x)


def test_layer_passes_gemm_options_on(layer_host):
    """gemm_options around a layer reaches its grouped GEMMs."""
    from llm_kernels_b200.moe import group_gemm_kernel as G
    layer, x, lib = layer_host()
    with G.gemm_options(max_ctas=7):
        layer(x)
    gemms = [args for n, args in lib.calls if n == "b200moe_grouped_gemm_fp8"]
    assert len(gemms) == 2 and all(args[-2]._obj.max_ctas == 7 for args in gemms)


def _hook(seen):
    return lambda *a: seen.append(1)


@pytest.mark.parametrize("how", ["forward hook", "pre-forward hook", "global hook", "instance forward", "gate class", "infer override", "infer on the instance"])
def test_layer_runs_what_replaces_its_gate_or_pipeline(layer_host, how):
    from llm_kernels_b200.moe.all2all_moe import DeepseekV3MoE, MoEGate
    seen = []

    class Other(DeepseekV3MoE):
        def triton_group_gemm_moe_infer(self, x, idx, w):
            seen.append(1)
            return super().triton_group_gemm_moe_infer(x, idx, w)

    class OtherGate(MoEGate):
        def forward(self, x):
            seen.append(1)
            return super().forward(x)

    layer, x, lib = layer_host(cls=Other if how == "infer override" else DeepseekV3MoE)
    if how != "infer override":
        layer(x)                                     # a pass before the change must not decide for the ones after it
    handle, gate_forward, infer = None, layer.gate.forward, layer.triton_group_gemm_moe_infer
    if how == "forward hook":
        layer.gate.register_forward_hook(_hook(seen))
    elif how == "pre-forward hook":
        layer.gate.register_forward_pre_hook(_hook(seen))
    elif how == "global hook":
        handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(1) if m is layer.gate else None)
    elif how == "instance forward":
        layer.gate.forward = lambda h: (seen.append(1), gate_forward(h))[1]
    elif how == "gate class":
        layer.gate.__class__ = OtherGate
    elif how == "infer on the instance":
        layer.triton_group_gemm_moe_infer = lambda *a: (seen.append(1), infer(*a))[1]
    try:
        layer(x)
    finally:
        if handle is not None:
            handle.remove()
    assert seen == [1]


@pytest.mark.parametrize("name,value", [("topk_method", "greedy"), ("topk_method", "group_limited_greedy"), ("scoring_func", "relu")])
def test_layer_names_an_unsupported_router(layer_host, name, value):
    """Such a gate has no correction bias for the layer to read."""
    layer, x, lib = layer_host(config={name: value})
    with pytest.raises(NotImplementedError, match=value if name == "topk_method" else "scoring"):
        layer(x)


def test_layer_takes_weights_made_under_inference_mode(layer_host):
    """Inference tensors have no version to compare."""
    layer, x, lib = layer_host()
    with torch.inference_mode():
        for name in ("w13_weight", "w13_weight_scale", "w2_weight", "w2_weight_scale"):
            setattr(layer, name, getattr(layer, name).clone())
    layer(x)
    layer(x)
    assert lib.names().count("b200moe_layer_forward") == 2


def test_layer_structure_follows_weights_and_settings(layer_host):
    """What the library reads in a pass is what the layer holds at that moment."""
    from ctypes import POINTER, cast
    from llm_kernels_b200 import _native as N
    seen = []
    layer, x, lib = layer_host("w4a16", b200moe_layer_forward=lambda d, *a: seen.append(N.Layer.from_buffer_copy(cast(d, POINTER(N.Layer))[0])) or 0)
    layer(x)
    layer(x)
    assert bytes(seen[0]) == bytes(seen[1])
    layer.w2_zero += 1                                     # in place: another copy of the pairs
    old = layer.w13_qweight
    layer.w13_qweight = old.clone()
    layer.gate.routed_scaling_factor = 3.5
    layer.gate.weight.data.add_(1.0)
    with torch.no_grad():
        layer.gate.weight.add_(1.0)
    layer(x)
    d = seen[2]
    assert d.w13 == layer.w13_qweight.data_ptr() != old.data_ptr() and d.scaling == 3.5
    assert d.w2 == layer.w2_qweight.data_ptr() and d.router_bias == layer.gate.e_score_correction_bias.data_ptr()
    assert torch.equal(layer._pairs("w2", "_scale", "_zero")[..., 1], layer.w2_zero.transpose(1, 2))
    assert d.w2_pairs == layer._pairs("w2", "_scale", "_zero").data_ptr() and d.router_w3 == layer.gate._w3.data_ptr()
    assert torch.equal(layer.gate._w3[:8].float().view(8, 3, 256).sum(1), layer.gate.weight)


def _twice(layer, x, lib, entry, note):
    """Runs a second pass of the layer in the middle of the first one's call of `entry`; returns what `note` made of the
    arguments of both, the outer one first."""
    seen = []

    def outer(*args):
        seen.append(note(*args))
        if len(seen) == 1:
            layer(x)
        return 0
    lib.on[entry] = outer
    layer(x)
    return seen


def test_layer_passes_that_overlap_have_workspaces_of_their_own(layer_host):
    """Another stream or thread, or a captured graph, can be in the middle of a pass."""
    layer, x, lib = layer_host()
    a, b = _twice(layer, x, lib, "b200moe_layer_forward", lambda d, x, y, T, ws, nbytes, stream: range(ws, ws + nbytes))
    assert a.stop <= b.start or b.stop <= a.start


def test_layer_keeps_the_last_rows_for_the_gemm_timing(layer_host):
    """_last_rows describes the last pass, whichever path it took."""
    layer, x, lib = layer_host()

    def layout(d, T, send, seg):
        send._obj.value, seg._obj.value = 0, 3584
        return 0
    lib.on["b200moe_layer_workspace_layout"] = layout
    layer(x)
    buf, rows, seg, widx = layer._last_rows()
    assert rows == 8 and buf.shape == (8, 272) and seg.shape == (9,) and widx is None
    layer.stage_events = []
    layer._mark = lambda name: None
    layer(x)
    assert layer._last_rows()[0] is layer._last[0] and layer._last_rows()[0].data_ptr() != buf.data_ptr()


def test_layer_passes_that_overlap_share_no_events(layer_host, monkeypatch):
    """With shared experts a pass orders two streams; an event recorded again by another pass would order the wrong work.
    The library makes them, so none is handed over."""
    from ctypes import POINTER, cast
    from types import SimpleNamespace
    from llm_kernels_b200 import _native as N
    handles = iter(range(1, 100))
    monkeypatch.setattr(torch.cuda, "Stream", lambda device=None: SimpleNamespace(cuda_stream=next(handles)))
    monkeypatch.setattr(torch.cuda, "Event", lambda: SimpleNamespace(cuda_event=next(handles), record=lambda: None))
    layer, x, lib = layer_host(config={"n_shared_experts": 1})
    a, b = _twice(layer, x, lib, "b200moe_layer_forward", lambda d, *rest: N.Layer.from_buffer_copy(cast(d, POINTER(N.Layer))[0]))
    assert a.side_stream == b.side_stream == 1 and a.shared_inter == 128
    assert not {a.fork_event, a.join_event} & {b.fork_event, b.join_event} - {None}


def test_layer_pass_keeps_what_its_structure_points_to(layer_host):
    """A pass after a change of the weights, in another thread, must not free what a pass in flight reads: the structure
    itself, the split router weight, the pairs."""
    import gc
    import weakref
    layer, x, lib = layer_host("w4a16")
    layer(x)
    held = [weakref.ref(layer._native[1]), *(weakref.ref(t) for t in (layer.gate._w3, layer._pairs("w2", "_scale", "_zero")))]
    alive = []

    def note(*args):
        if alive:
            gc.collect()
            alive.append([r() is not None for r in held])
        else:
            alive.append(None)
            layer.w2_zero += 1
            with torch.no_grad():
                layer.gate.weight.add_(1.0)
    _twice(layer, x, lib, "b200moe_layer_forward", note)
    assert alive[1] == [True] * 3
    gc.collect()
    assert [r() is not None for r in held] == [False] * 3


@pytest.mark.parametrize("method", ["fp8_block", "w4a8"])
def test_layer_can_be_copied_after_a_pass(layer_host, method):
    import copy
    import io
    layer, x, lib = layer_host(method)
    layer(x)
    file = io.BytesIO()
    torch.save(layer, file)
    file.seek(0)
    for twin in (copy.deepcopy(layer), torch.load(file, weights_only=False)):
        assert twin._native is None and twin._last_pass is None
        twin(x)
        assert twin._native[1].w13 == next(iter(twin.buffers())).data_ptr() != layer._native[1].w13


def test_layer_saved_by_an_earlier_version_runs(layer_host):
    layer, x, lib = layer_host()
    for name in ("_native", "_last_pass", "_layout", "_sizes"):
        del layer.__dict__[name]
    layer(x)
    assert lib.names().count("b200moe_grouped_gemm_fp8") == 2


@pytest.mark.parametrize("kind", ["fp8", "w4a8"])
def test_split_gemms_that_overlap_have_partials_of_their_own(host, monkeypatch, kind):
    """The product and the sum of its splits are two launches: another thread's call can come between them."""
    from llm_kernels_b200.quantization import fp8_kernel, w4a8_kernel
    f8 = torch.float8_e4m3fn
    seen = []

    def call():
        if kind == "w4a8":
            return w4a8_kernel.w4a8_gemm(*_w4a8_operands(24, 1024, 1024, 8))
        return fp8_kernel.fp8_gemm(torch.zeros(24, 1024, dtype=f8), torch.ones(24, 8), torch.zeros(256, 1024, dtype=f8), torch.ones(2, 8))

    def outer(*args):
        seen.append(range(args[10], args[10] + args[11]))
        if len(seen) == 1:
            call()
        return 0
    monkeypatch.setattr(host, "_lib", Recorder(b200moe_gemm_i8_block_splitk=outer, b200moe_gemm_fp8_block_splitk=outer))
    call()
    a, b = seen
    assert len(a) == 8 * 24 * 256 * 4 and (a.stop <= b.start or b.stop <= a.start)


def test_grouped_gemms_refuse_a_missing_group_table(host):
    """Also for one group, and before anything else decides that there is nothing to do (no rows)."""
    lib, bf = host.lib(), host.BF16
    assert lib.b200moe_grouped_gemm_i8(16, 128, 16, 1, 16, 16, 16, bf, 256, 0, 128, 128, 1, 1, None, None, None, None, None) == 4
    for fn, tail in ((lib.b200moe_grouped_gemm_bf16, (0, None, None, None)), (lib.b200moe_grouped_gemm_f16, (None, None, None))):
        assert fn(16, 256, 16, 16, bf, 256, 0, 128, 128, 1, 1, None, None, *tail) == 4
        assert fn(16, 256, 16, 16, bf, 256, 0, 128, 128, 1, 1, 16, None, *tail) == 0


def test_package_imports_on_a_torch_without_cuda():
    """The host-only parts (configurations, bit packing on the CPU, plans) need no CUDA in torch."""
    import os
    import subprocess
    import sys
    code = ("import torch\n"
            "for name in [n for n in dir(torch._C) if n.startswith('_cuda_get')]:\n"
            "    delattr(torch._C, name)\n"
            "import llm_kernels_b200._native, llm_kernels_b200.moe.all2all_moe, llm_kernels_b200.workloads\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr


def test_layer_moved_to_another_device_is_refused(layer_host, host, monkeypatch):
    """Module.to moves weights and buffers; the layer's scratch and status word stay on the device that it was made for."""
    layer, x, lib = layer_host()
    elsewhere = layer._status

    def require_cuda(*tensors):
        if any(t is elsewhere for t in tensors):
            raise RuntimeError("not on the current device")
    monkeypatch.setattr(host, "require_cuda", require_cuda)
    with pytest.raises(RuntimeError, match="current device"):
        layer(x)


def test_quantized_calls_do_without_their_compiled_module(host, monkeypatch, tmp_path):
    """It is missing, or belongs to another torch: the Python functions serve the call and make their own checks."""
    from llm_kernels_b200 import build
    from llm_kernels_b200.quantization import fp8_kernel, w4a8_kernel
    assert build.calls_fit() and not build.needs_build()
    for patch in (lambda m: m.setattr(build, "CALLS", str(tmp_path / "_calls.so")),
                  lambda m: m.setattr(build, "calls_stamp", lambda: "built for another torch")):
        with monkeypatch.context() as m:
            lib = Recorder()
            m.setattr(host, "_lib", lib)
            m.setattr(host, "_calls_module", None)
            patch(m)
            with pytest.warns(RuntimeWarning, match="take longer"):
                fp8_kernel.act_quant(torch.zeros(2, 128))
            w4a8_kernel.act_quant(torch.zeros(2, 128))
            fp8_kernel.fp8_gemm(torch.zeros(200, 256, dtype=torch.float8_e4m3fn), torch.ones(200, 2),
                                torch.zeros(256, 256, dtype=torch.float8_e4m3fn), torch.ones(2, 2))
            w4a8_kernel.w4a8_gemm(*_w4a8_operands(200, 256, 256, 2))
            assert lib.names() == ["b200moe_act_quant_fp8", "b200moe_act_quant_int8", "b200moe_gemm_fp8_block",
                                   "b200moe_w4a8_gemm_operands", "b200moe_gemm_i8_block"]
            assert build.needs_build()


def test_library_is_built_without_the_compiled_calls(monkeypatch, tmp_path):
    """Other hosts need the library alone: no torch with CUDA, or none with headers."""
    from llm_kernels_b200 import build
    build.build()
    monkeypatch.setattr(build, "CALLS", str(tmp_path / "_calls.so"))
    monkeypatch.setattr(build, "_calls_possible", lambda: False)
    assert not build.needs_build() and build.build() == build.LIB and not (tmp_path / "_calls.so").exists()
