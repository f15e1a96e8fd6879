"""Host side of the ops, without a device: the launches are answered by a stand-in for the library."""

import importlib

import pytest
import torch

import generative_recommenders_b200 as G

HC = importlib.import_module("generative-recommenders_b200.hstu_compute")


class _Library:
    """Answers the fused uvqk launch; ``rc`` is its return code, ``during`` runs inside the call."""

    def __init__(self):
        self.rc, self.during, self.prepared = 0, None, []

    def b200_hstu_ln_linear_workspace_bytes(self, D, N):
        return 4096

    def b200_hstu_ln_linear_silu_fwd(self, a, stream):
        self.prepared.append(a.weights_prepared)
        if self.during is not None:
            run, self.during = self.during, None
            run()
        return self.rc


@pytest.fixture
def uvqk(monkeypatch):
    """(library, parameters, call): ``call()`` queues the fused stage on the parameters in the list."""
    lib = _Library()

    def check(rc, what):
        if rc != 0:
            raise RuntimeError(what)

    class _Device:
        def __enter__(self):
            return None

        def __exit__(self, *exc):
            return False

    monkeypatch.setattr(HC._cabi, "lib", lambda: lib)
    monkeypatch.setattr(HC._cabi, "check", check)
    monkeypatch.setattr(HC, "stream_ptr", lambda device: 0)
    monkeypatch.setattr(HC, "on_device", lambda device: _Device())
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    HC.clear_prepared_weights()
    D, N, hv = 16, 32, 8
    params = [torch.nn.Parameter(torch.ones(n, dtype=torch.bfloat16), requires_grad=False) for n in (D, D)]
    params += [torch.nn.Parameter(torch.ones(s, dtype=torch.bfloat16), requires_grad=False) for s in ((D, N), (N,))]
    x = torch.ones(4, D, dtype=torch.bfloat16)
    yield lib, params, lambda: HC._fused_uqvk_launch(x, params[0], params[1], 1e-6, params[2], params[3], hv, True)
    HC.clear_prepared_weights()


def test_prepared_weights_are_kept_while_the_parameters_are_unchanged(uvqk):
    lib, params, call = uvqk
    call(), call()
    with torch.no_grad():
        params[2].mul_(2)
    call(), call()
    assert lib.prepared == [0, 1, 0, 1]


def test_failed_launch_leaves_no_prepared_weights(uvqk):
    # the workspace of a call that returned an error holds nothing
    lib, params, call = uvqk
    lib.rc = 1
    with pytest.raises(RuntimeError, match="ln_linear"):
        call()
    lib.rc = 0
    call(), call()
    assert lib.prepared == [0, 0, 1]


def test_prepared_weights_are_shared_after_their_preparation_is_queued(uvqk):
    # another thread's call may come between the lookup of this one and its launch: it must not take a
    # workspace whose preparation is not in the stream yet
    lib, params, call = uvqk
    lib.during = call
    call()
    assert lib.prepared == [0, 0]
    call()
    assert lib.prepared == [0, 0, 1]


def test_weights_forgotten_during_a_call_stay_forgotten(uvqk):
    lib, params, call = uvqk
    lib.during = HC.clear_prepared_weights
    call(), call()
    assert lib.prepared == [0, 0]


@pytest.mark.parametrize("which", range(4))
def test_replaced_parameter_is_not_the_prepared_one(uvqk, monkeypatch, which):
    # an id, an address and a version can all come back with a new parameter once the old one is gone
    lib, params, call = uvqk
    monkeypatch.setattr(HC, "id", lambda t: 7, raising=False)
    call()
    storage = params[which].detach()
    params[which] = None
    params[which] = torch.nn.Parameter(storage, requires_grad=False)
    call()
    assert lib.prepared == [0, 0]


def test_parameters_made_in_inference_mode_are_not_remembered(uvqk):
    # they carry no version counter, so nothing would tell a changed one
    lib, params, call = uvqk
    with torch.inference_mode():
        params[:] = [torch.nn.Parameter(p.detach().clone(), requires_grad=False) for p in params]
        call(), call()
    assert lib.prepared == [0, 0]


def test_span_and_the_autograd_rule_are_seen_through_by_the_compiler():
    common = importlib.import_module("generative-recommenders_b200.common")

    def step(x):
        with common.span("## step ##"):
            y = x + 1
        return y * 2 if common.outside_autograd(y) else y * 3

    x = torch.ones(3)
    # (under the compiler a call keeps its autograd node)
    assert torch.equal(torch.compile(step, fullgraph=True, backend="eager")(x), torch.full((3,), 6.0))
    assert torch.equal(step(x), torch.full((3,), 4.0))


@pytest.mark.parametrize("device", [1, None, "cuda:1", torch.device("cuda", 1), torch.device("cuda")])
def test_on_device_takes_what_the_device_context_takes(device, monkeypatch):
    common = importlib.import_module("generative-recommenders_b200.common")
    entered = []
    monkeypatch.setattr(torch.cuda, "device", entered.append)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: 0, raising=False)
    common.on_device(device)
    assert entered == [device]
    with common.on_device(torch.device("cuda", 0)):
        pass
    assert entered == [device]


@pytest.mark.parametrize("rows", [0, 6])
def test_full_kv_offsets_are_the_callers_own(rows, monkeypatch):
    # what the caller does to the offsets it got must not change those of the cache, new rows or none
    stu = importlib.import_module("generative-recommenders_b200.stu")
    monkeypatch.setattr(stu, "concat_2D_jagged", lambda values_left, **kw: values_left)
    layer = G.STULayer(G.STULayerConfig(embedding_dim=16, num_heads=1, hidden_dim=16, attention_dim=16))
    layer.k_cache = layer.v_cache = torch.zeros(9, 16)
    layer.kv_caching_offsets, layer.max_kv_caching_len = torch.tensor([0, 4, 9], dtype=torch.int32), 5
    delta = torch.zeros(rows, 16)
    _, _, longest, offsets = layer.construct_full_kv(delta, delta)
    n = rows // 2
    assert longest == 5 + n and offsets.dtype == torch.int64 and offsets.tolist() == [0, 4 + n, 9 + 2 * n]
    offsets.zero_()
    assert layer.kv_caching_offsets.tolist() == [0, 4, 9]


@pytest.fixture
def fp8(monkeypatch):
    """(module, seen): ``seen`` collects the block offsets, as int32, that the launches are given; before they
    are read, the memory that a dropped tensor would have left is written over."""
    import ctypes

    module = importlib.import_module("generative-recommenders_b200.hstu_attention_fp8")
    seen = []

    def read(address, n):
        keep = [torch.full((n,), -1, dtype=torch.int32) for _ in range(64)]
        seen.append(list((ctypes.c_int32 * n).from_address(address)))
        del keep
        return 0

    class Library:
        def b200_hstu_attn_workspace_bytes(self, a, which):
            return 0

        def b200_hstu_attn_fwd_fp8(self, fa, stream):
            return read(fa.block_offsets, fa.base.B + 1)

        def b200_hstu_quantize_e4m3_block(self, *args):
            return read(args[7], args[8] + 1)

    monkeypatch.setattr(module._cabi, "lib", Library)
    monkeypatch.setattr(module, "require_cuda", lambda *tensors: None)
    monkeypatch.setattr(module, "stream_ptr", lambda device: 0)
    monkeypatch.setattr(module, "on_device", lambda device: importlib.import_module("contextlib").nullcontext())
    return module, seen


# a caller may hold them in any integer type and layout
_BLOCKS = [torch.tensor([0, 1, 3], dtype=torch.int32), torch.tensor([0, 1, 3]),
           torch.tensor([[0, 1, 3], [9, 9, 9]], dtype=torch.int32).t().contiguous()[:, 0]]


@pytest.mark.parametrize("blocks", _BLOCKS)
def test_block_offsets_reach_the_fp8_forward(fp8, blocks):
    module, seen = fp8
    x8, scale = torch.zeros(300, 1, 64).to(torch.float8_e4m3fn), torch.ones(4, 1)
    module.hstu_mha_fp8(256, 1.0, x8, x8, x8, scale, scale, scale, blocks, torch.tensor([0, 100, 300]))
    assert seen == [[0, 1, 3]]


@pytest.mark.parametrize("blocks", _BLOCKS)
def test_block_offsets_reach_the_quantiser(fp8, blocks):
    module, seen = fp8
    _, _, out = module.quantize_e4m3_block(torch.zeros(300, 1, 64), torch.tensor([0, 100, 300]), blocks)
    assert seen == [[0, 1, 3]]
    assert out is blocks


class _OnDevice(torch.Tensor):
    is_cuda = True


@pytest.mark.parametrize("autocast", [False, True])
def test_separate_stages_go_one_by_one_under_autocast(monkeypatch, autocast):
    """Autocast changes the type between LayerNorm, linear and attention: each op has to see the tensor it gets.
    The one native call, whose kernels are all told the type of x, is for calls without it."""
    D, H, d, M = 24, 2, 4, 6
    made = [torch.zeros(s).as_subclass(_OnDevice) for s in ((M, D), (D,), (D,), (D, 4 * H * d), (4 * H * d,))]
    offsets = torch.tensor([0, M]).as_subclass(_OnDevice)
    taken = []

    class _Host:
        def separate_attention_inference(self, *args):
            taken.append("one call")
            return (made[0],) * 4

    def uqvk(**kwargs):
        taken.append("uqvk")
        return (torch.zeros(M, H * d),) + (torch.zeros(M, H, d),) * 3

    def attention(**kwargs):
        taken.append("attention")
        return torch.zeros(M, H, d)

    monkeypatch.setattr(HC._cabi, "host", lambda: _Host())
    monkeypatch.setattr(HC, "hstu_compute_uqvk", uqvk)
    monkeypatch.setattr(HC, "hstu_mha", attention)
    before = torch.is_autocast_enabled("cuda")
    torch.set_autocast_enabled("cuda", autocast)
    try:
        with torch.no_grad():
            HC.hstu_preprocess_and_attention(made[0], made[1], made[2], 1e-6, H, d, d, made[3], made[4], M, offsets, 0.5,
                                             True, None, 0, 0, False, False, False)
    finally:
        torch.set_autocast_enabled("cuda", before)
    assert taken == (["uqvk", "attention"] if autocast else ["one call"])


class _Sees(torch.utils._python_dispatch.TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


@pytest.mark.parametrize("replaced, on_class", [(name, on_class) for name in ("forward", "cached_forward", "construct_full_kv")
                                               for on_class in (False, True)] + [("__call__", True)])
def test_replaced_methods_of_a_layer_are_called_for_every_layer(monkeypatch, replaced, on_class):
    stu = importlib.import_module("generative-recommenders_b200.stu")
    cfg = G.STULayerConfig(embedding_dim=16, num_heads=1, hidden_dim=16, attention_dim=16)
    layers = [G.STULayer(cfg) for _ in range(3)]
    stack = G.STUStack(layers)
    for layer in layers:
        layer.k_cache = layer.v_cache = torch.zeros(5, 16)
        layer.kv_caching_offsets, layer.max_kv_caching_len = torch.tensor([0, 2, 5]), 3
    taken = []
    shortcuts = {"forward": "_forward", "cached_forward": "_cached_forward", "__call__": "_forward"}
    if replaced in shortcuts:
        monkeypatch.setattr(stu.STULayer, shortcuts[replaced], lambda self, *a, **kw: taken.append("own") or torch.zeros(2, 16))
    else:
        monkeypatch.setattr(stu, "hstu_cached_attention", lambda *a: taken.append("own"))
        monkeypatch.setattr(stu.STULayer, "_cached_attention_of_ops", lambda self, *a: (None, None))
        monkeypatch.setattr(stu, "_compute_output", lambda **kw: kw["x"])

    def run():
        taken.clear()
        with torch.no_grad():
            if replaced in ("forward", "__call__"):
                stack(torch.zeros(2, 16), None, None, 2, None)
            else:
                stack.cached_forward(torch.zeros(2, 16), None)
        return list(taken)

    assert run() == ["own"] * 3
    if replaced == "__call__":
        own = torch.nn.Module.__call__
        monkeypatch.setattr(torch.nn.Module, "__call__", lambda self, *a, **kw: (
            own(self, *a, **kw) if self is stack else taken.append("replaced") or torch.zeros(2, 16)))
    else:
        def replacement(*args, **kwargs):
            taken.append("replaced")
            return torch.zeros(2, 16)
        if on_class:
            monkeypatch.setattr(stu.STULayer, replaced, replacement)
        else:
            for layer in layers:
                setattr(layer, replaced, replacement)
    if replaced == "construct_full_kv":
        assert run() == []     # (the ops one by one, which call it)
    else:
        assert run() == ["replaced"] * 3


def test_layers_are_called_as_modules_where_someone_looks_on():
    stu = importlib.import_module("generative-recommenders_b200.stu")
    layer = G.STULayer(G.STULayerConfig(embedding_dim=16, num_heads=1, hidden_dim=16, attention_dim=16))
    with torch.no_grad():
        assert stu._nobody_looks_on() and stu._unobserved(layer, "forward") and stu._unobserved(layer, "cached_forward")
        with _Sees():
            assert not stu._nobody_looks_on()
    assert not stu._nobody_looks_on()     # (gradients: nothing may be overwritten)
    layer.register_forward_hook(lambda *a: None)
    assert not stu._unobserved(layer, "forward")


def _cached_call(monkeypatch, host, targets):
    """``hstu_cached_attention`` of two sequences with one new row each; ``host`` answers the native calls."""
    D = 16
    on = lambda *s, dtype=torch.bfloat16: torch.zeros(s, dtype=dtype).as_subclass(_OnDevice)  # noqa: E731
    monkeypatch.setattr(HC, "_prepared_workspace", lambda *a: (torch.zeros(4096, dtype=torch.uint8), False, None))
    monkeypatch.setattr(HC._cabi, "lib", lambda: _Library())
    monkeypatch.setattr(HC._cabi, "host", lambda: host)
    offsets = torch.tensor([0, 2, 5]).as_subclass(_OnDevice)
    targets = None if targets is None else torch.ones(targets, dtype=torch.int64).as_subclass(_OnDevice)
    with torch.no_grad():
        return HC.hstu_cached_attention(on(2, D), on(D), on(D), 1e-6, 1, D, D, on(D, 4 * D), on(4 * D), on(5, D), on(5, D),
                                        offsets, targets, 4, 0.1, 0, 0)


class _Native:
    """The native calls, the choice of path answered by yes."""

    def __init__(self):
        self.native = G._cabi.host()

    def cached_attention(self, *args):
        return self.native.cached_attention(*args)

    def cached_supported(self, *args):
        return True


def test_attention_of_new_rows_refuses_missing_target_counts(monkeypatch):
    """The kernels read ``num_targets[b]`` of every sequence."""
    rows = torch.zeros(2, 1, 16).as_subclass(_OnDevice)
    offsets, targets = (torch.tensor(t).as_subclass(_OnDevice) for t in ([0, 1, 2], [1]))
    with pytest.raises(RuntimeError, match="one entry per sequence"):
        G.delta_hstu_mha(2, 0.1, rows, rows, rows, offsets, targets)
    q8 = rows.to(torch.float8_e4m3fn).as_subclass(_OnDevice)
    with pytest.raises(RuntimeError, match="one entry per sequence"):
        G.hstu_mha_fp8(2, 0.1, q8, q8, q8, rows, rows, rows, offsets, offsets, targets)
    with pytest.raises(RuntimeError, match="one entry per sequence"):
        _cached_call(monkeypatch, _Native(), 1)


@pytest.mark.parametrize("k_rows, v_rows", [(5, 5), (5, 4), (5, 6)])
def test_cached_attention_reads_k_and_v_of_as_many_rows(k_rows, v_rows):
    """One launch appends to both and takes one row count; other caches go to the separate ops, and a V of fewer
    rows than K is refused where both are read together."""
    t = lambda *s: torch.zeros(s, dtype=torch.bfloat16)  # noqa: E731
    offsets = torch.tensor([0, 2, 5])
    assert G._cabi.host().cached_supported(t(2, 64), t(64, 256), 64, 64, t(k_rows, 64), t(v_rows, 64), offsets) == (
        k_rows == v_rows)
    if v_rows < k_rows:
        rows = torch.zeros(k_rows, 1, 16).as_subclass(_OnDevice)
        with pytest.raises(AssertionError, match="wrong v shape"):
            G.delta_hstu_mha(k_rows, 0.1, rows[:1], rows, rows[:v_rows], torch.tensor([0, k_rows]).as_subclass(_OnDevice))


def test_cached_attention_in_one_call_takes_what_it_can_read():
    """16-bit rows, contiguous caches of the same type and of the heads' widths, int64 offsets."""
    t = lambda *s, dtype=torch.bfloat16: torch.zeros(s, dtype=dtype)  # noqa: E731
    good = {"x": t(2, 64), "w": t(64, 256), "hv": 64, "ha": 64, "k": t(5, 64), "v": t(5, 64), "offsets": torch.tensor([0, 2, 5])}
    supported = lambda **kw: G._cabi.host().cached_supported(*dict(good, **kw).values())  # noqa: E731
    assert supported()
    for name, other in (("x", t(2, 64, dtype=torch.float32)), ("x", t(0, 64)), ("x", t(2, 128)[:, ::2]), ("x", t(2, 1, 64)),
                        ("k", t(5, 64, dtype=torch.float16)), ("v", t(5, 64, dtype=torch.float32)), ("k", t(5, 63)),
                        ("v", t(5, 128)[:, :64]), ("v", t(5, 1, 64)), ("k", t(5)),
                        ("offsets", torch.tensor([0, 2, 5], dtype=torch.int32)), ("offsets", torch.arange(6)[::2])):
        assert not supported(**{name: other}), name


@pytest.mark.parametrize("on", [False, True])
def test_status_check_reaches_cached_attention(monkeypatch, on):
    """Checked or not, the same path runs."""
    asked = []

    class _Host(_Native):
        def cached_attention(self, *args):
            asked.append(args[-1])
            return "taken"

        def attention_forward(self, *args):
            asked.append(args[-1])
            return args[0], None

    HA = importlib.import_module("generative-recommenders_b200.hstu_attention")
    monkeypatch.setattr(HA, "_CHECK_STATUS", on)
    assert _cached_call(monkeypatch, _Host(), None) == "taken"
    rows = torch.zeros(2, 1, 16).as_subclass(_OnDevice)
    G.delta_hstu_mha(2, 0.1, rows, rows, rows, torch.tensor([0, 1, 2]).as_subclass(_OnDevice))
    assert asked == [on, on]


def test_host_module_is_built_anew_for_another_torch(tmp_path, monkeypatch):
    build = importlib.import_module("generative-recommenders_b200.build")
    runs = []

    def run(cmd, **kw):
        runs.append(cmd)
        (tmp_path / "_host.so").write_text("")
        return importlib.import_module("subprocess").CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build, "BUILD", str(tmp_path))
    monkeypatch.setattr(build, "HOST", str(tmp_path / "_host.so"))
    monkeypatch.setattr(build, "subprocess", type("S", (), {"run": staticmethod(run)}))
    for expected in (1, 1):
        build._build_host(False, False)
        assert len(runs) == expected
    monkeypatch.setattr(torch, "__version__", "0.0.0")
    build._build_host(False, False)
    assert len(runs) == 2


@pytest.mark.parametrize("width, norm, rows, bias", [(24, 16, 16, 64), (8, 16, 16, 64), (16, 8, 16, 64), (16, 16, 16, 63)])
def test_fused_uvqk_stage_refuses_parameters_of_another_width(width, norm, rows, bias):
    """The kernel reads them, and sizes its workspace, by the width of x."""
    t = lambda *s: torch.zeros(s, dtype=torch.bfloat16)  # noqa: E731
    x, nw, w, b, ws = t(2, width), t(norm), t(rows, 64), t(bias), torch.zeros(4096, dtype=torch.uint8)
    with pytest.raises(RuntimeError, match="another width"):
        HC._fused_uqvk_launch(x, nw, nw, 1e-6, w, b, 16, True)
    with pytest.raises(RuntimeError, match="another width"):
        G._cabi.host().cached_attention(x, nw, nw, w, b, 1e-6, 1, 16, 16, ws, False, t(5, 16), t(5, 16),
                                        torch.tensor([0, 2, 5]), None, 4, 0.1, 0, 0, 0, G._cabi.BF16, False)
