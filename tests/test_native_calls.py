"""Native autograd nodes and the native forward pass give what the Python operators and modules give, bit for bit, and
leave to those what something else watches."""
import contextlib

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bf16(*shape):
    return torch.randn(*shape, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("kind", ["2d", "3d", "transposed", "sliced", "one row"])
@pytest.mark.parametrize("needs", [(True, True), (True, False), (False, True)])
def test_linear_node_matches_the_python_function(kind, needs):
    from picotron_b200 import ops
    from picotron_b200.ops import gemm
    torch.manual_seed(0)
    x = {"2d": lambda: _bf16(70, 64), "3d": lambda: _bf16(3, 35, 64), "transposed": lambda: _bf16(64, 72).t(),
         "sliced": lambda: _bf16(5, 40, 76)[:, 1:38, 4:68], "one row": lambda: _bf16(1, 64)}[kind]()
    x.requires_grad_(needs[0])
    w = _bf16(136, 64).requires_grad_(needs[1])
    dy = _bf16(136, *x.shape[:-1]).movedim(0, -1) if kind != "one row" else _bf16(1, 136)     # not contiguous
    wanted = [t for t in (x, w) if t.requires_grad]
    before = ops.launches()
    y = gemm.linear(x, w)
    assert "LinearNode" in y.grad_fn.name()
    got = torch.autograd.grad(y, wanted, dy)
    assert ops.launches() - before == 1 + len(wanted)
    ref = gemm._LinearFn.apply(x, w)
    for a, b in zip(got, torch.autograd.grad(ref, wanted, dy)):
        assert a.shape == b.shape and torch.equal(a, b)
    assert torch.equal(y, ref)
    ops.check_status()


def test_linear_node_leaves_main_grad_and_postponed_gradients_to_python():
    from picotron_b200.ops import gemm
    torch.manual_seed(1)
    x, w, dy = _bf16(40, 64).requires_grad_(), torch.nn.Parameter(_bf16(72, 64)), _bf16(40, 72)
    with gemm.defer_wgrad() as queue:
        gemm.linear(x, w).backward(dy)
    assert w.grad is None and len(queue) == 1
    gemm.run_deferred(queue)
    late = w.grad.clone()
    w.grad = None
    y = gemm.linear(x, w)
    w.main_grad = torch.zeros(72, 64, device="cuda")             # looked up when the gradient is there, not before
    ready = []
    w.grad_ready_hook = lambda: ready.append(1)
    y.backward(dy)
    assert w.grad is None and ready == [1]
    want = dy.double().t() @ x.detach().double()
    assert (w.main_grad.double() - want).norm() <= 1e-5 * want.norm()
    assert (late.double() - want).norm() <= 2 ** -8 * want.norm()


def _main_grad(w):
    w.main_grad = torch.zeros(w.shape, device="cuda")
    w.calls = []
    w.grad_ready_hook = lambda: w.calls.append(1)
    return w.main_grad


@pytest.mark.parametrize("how", ["grad", "backward"])
@pytest.mark.parametrize("where", ["main_grad", "queue"])
@pytest.mark.parametrize("learns", [True, False])
def test_a_backward_for_the_input_alone_keeps_the_weight_gradient(how, where, learns):
    """The weight's gradient goes into main_grad, or into the queue, whether or not this backward asks for it, as long as
    the weight learns: as with the Python function."""
    from picotron_b200.ops import gemm
    torch.manual_seed(4)
    x, dy = _bf16(40, 64).requires_grad_(), _bf16(40, 72)
    w = torch.nn.Parameter(_bf16(72, 64), requires_grad=learns)
    results = []
    for call in (gemm.linear, gemm._LinearFn.apply):
        buf = _main_grad(w)
        x.grad = None
        with contextlib.ExitStack() as stack:
            queue = stack.enter_context(gemm.defer_wgrad()) if where == "queue" else []
            y = call(x, w)
            dx = torch.autograd.grad(y, x, dy)[0] if how == "grad" else y.backward(dy, inputs=[x]) or x.grad
        assert len(queue) == int(learns and where == "queue")
        gemm.run_deferred(queue)
        assert len(w.calls) == int(learns) and bool(buf.any()) == learns and w.grad is None
        results.append((dx, buf))
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("b,s,H,Hkv,d,causal", [(1, 33, 3, 1, 64, False), (2, 130, 4, 4, 128, True)])
def test_attention_node_matches_the_python_function(b, s, H, Hkv, d, causal):
    """One to two key blocks per query: dQ has at most two addends and repeats bit for bit. Slices of a fused buffer."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    torch.manual_seed(2)
    heads = _bf16(b, s, H + 2 * Hkv, d).requires_grad_()
    q, k, v = heads[:, :, :H], heads[:, :, H:H + Hkv], heads[:, :, H + Hkv:]
    go = _bf16(b, H, s, d).transpose(1, 2)
    before = ops.launches()
    out = A.attention(q, k, v, causal, 0.2)
    assert "AttentionNode" in out.grad_fn.name()
    got = torch.autograd.grad(out, (q, k, v), go)
    assert ops.launches() - before == 4
    ref = A._FlashAttnFn.apply(q, k, v, causal, 0.2)
    for a, r in zip(got, torch.autograd.grad(ref, (q, k, v), go)):
        assert torch.equal(a, r)
    assert torch.equal(out, ref)
    ops.check_status()


def test_nodes_keep_saved_tensor_hooks_and_refuse_a_second_pass():
    from picotron_b200.ops import attention as A
    from picotron_b200.ops import gemm
    x, w = _bf16(24, 64).requires_grad_(), _bf16(64, 64).requires_grad_()
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        y = gemm.linear(x, w)
        o = A.attention(*(t.view(1, 24, 1, 64) for t in (y, y, y)), True)
    assert len(seen) == 2 + 5
    o.sum().backward()
    assert x.grad is not None and w.grad is not None
    with pytest.raises(RuntimeError):
        o.sum().backward()


def test_watched_calls_take_the_python_functions():
    """Transforms are refused as before; under a forward-mode level the Python function answers."""
    from picotron_b200.ops import gemm
    x, w = _bf16(24, 64), _bf16(64, 64)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: gemm.linear(t, w).float().sum())(x)
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: gemm.linear(t, w))(x.view(2, 12, 64))
    with torch.autograd.forward_ad.dual_level():
        y = gemm.linear(x.requires_grad_(), w)
        assert "_LinearFn" in y.grad_fn.name()


def _model(name, layers, seq, widths=None):
    """``widths``: those of the layers' MLPs, where they differ."""
    from picotron_b200.config import MODEL_SHAPES
    from picotron_b200.models.llama import MLP, Llama
    from picotron_b200.param_store import ParamStore
    from types import SimpleNamespace
    shape = dict(MODEL_SHAPES["HuggingFaceTB/SmolLM-135M"], num_hidden_layers=layers, max_position_embeddings=seq,
                 init_std=0.05, **name)
    torch.manual_seed(3)
    config = SimpleNamespace(**shape)
    with torch.device("cuda"):
        model = Llama(config)
        for layer, width in zip(model.decoder_layers, widths or ()):
            layer.mlp = MLP(config, width)
    model.reset_parameters()
    model = model.to(torch.bfloat16)
    return model, ParamStore(model)


@pytest.mark.parametrize("b,s", [(1, 1), (1, 33), (3, 130)])
def test_native_forward_matches_the_modules(b, s):
    from picotron_b200 import ops
    model, _ = _model({}, 2, 130)
    ids = torch.randint(0, 49152, (b, s), device="cuda")
    with torch.no_grad():
        assert model._native_layers(ids) is not None
        native = model(ids)
        seen = []
        for mod in (model.decoder_layers[1], model.decoder_layers[0].mlp.down_proj, model.final_norm):
            handle = mod.register_forward_hook(lambda *a: seen.append(1))
            assert model._native_layers(ids) is None
            assert torch.equal(model(ids), native)
            handle.remove()
        assert len(seen) == 3
    ops.check_status()
    assert native.shape == (b, s, 49152) and native.grad_fn is None
    assert model(ids).grad_fn is not None                       # with gradients the modules run


@pytest.mark.parametrize("b,s,shape,in_epilogue,parts", [
    (2, 500, dict(intermediate_size=2048, num_attention_heads=8, num_key_value_heads=4), True, False),
    (1, 33, dict(intermediate_size=8192, num_attention_heads=8, num_key_value_heads=2), False, True),
    (2, 200, dict(intermediate_size=8192, num_attention_heads=16, num_key_value_heads=16), True, True),
    (1, 7, dict(intermediate_size=6144, num_attention_heads=8, num_key_value_heads=8), False, True)])
def test_native_forward_with_every_layout_of_its_memory(b, s, shape, in_epilogue, parts):
    """The activation in the gate-up product (no room for gate | up) and by itself, the down projection whole and in
    parts of K (slabs in the same allocation), head_dim 64 and 128; three layers, so every buffer is used again."""
    from picotron_b200 import ops
    model, _ = _model(dict(hidden_size=1024, vocab_size=4096, **shape), 3, 600)
    inter = shape["intermediate_size"]
    assert ops.ext().gemm_swiglu_pays(b * s, inter, 1024, False, False) == in_epilogue
    assert (ops.ext().gemm_parts_of_k(b * s, 1024, inter) > 0) == parts
    ids = torch.randint(0, 4096, (b, s), device="cuda")
    with torch.no_grad():
        assert model._native_layers(ids) is not None
        native = [model(ids) for _ in range(2)]
        handle = model.final_norm.register_forward_hook(lambda *a: None)
        assert model._native_layers(ids) is None
        modules = model(ids)
        handle.remove()
    ops.check_status()
    assert all(torch.equal(n, modules) for n in native) and modules.float().std() > 0.01


def test_native_forward_is_left_where_it_does_not_apply():
    ids = torch.randint(0, 49152, (1, 20), device="cuda")
    model, _ = _model({}, 2, 32)
    model.rope.pos_offset = 4
    with torch.no_grad():
        native = model(ids)
        handle = model.final_norm.register_forward_hook(lambda *a: None)
        assert torch.equal(model(ids), native)
        handle.remove()
        with pytest.raises(RuntimeError, match="position table too short"):
            model(torch.randint(0, 49152, (1, 29), device="cuda"))
        model.decoder_layers[1].attention.core = lambda q, k, v, causal: q       # as context parallelism installs one
        assert model._native_layers(ids) is None
    parallel, _ = _model(dict(parallel_block=True), 2, 32)
    loose, _ = _model({}, 1, 32)
    for m in loose.modules():                                    # weights that are not stored side by side
        m.__dict__.pop("_fused_group", None)
    uneven, _ = _model({}, 2, 32, widths=(1536, 768))
    with torch.no_grad():
        for other in (parallel, loose, uneven):
            assert other._native_layers(ids) is None and other(ids).shape == (1, 20, 49152)


@pytest.mark.parametrize("where", ["instance", "class"])
@pytest.mark.parametrize("owner,method", [("MLP", "hidden"), ("MLP", "forward"), ("Linear", "forward"),
                                          ("Attention", "_fused_local"), ("RMSNorm", "forward"),
                                          ("DecoderLayer", "forward")])
def test_replaced_methods_are_called(monkeypatch, where, owner, method):
    """A program that replaces a method of a module or of its class sees it called, with gradients and without."""
    from picotron_b200.models import llama
    model, _ = _model({}, 2, 32)
    ids = torch.randint(0, 49152, (1, 20), device="cuda")
    cls, layer = getattr(llama, owner), model.decoder_layers[1]
    mod = {"MLP": layer.mlp, "Linear": layer.mlp.down_proj, "Attention": layer.attention,
           "RMSNorm": layer.post_attention_layernorm, "DecoderLayer": layer}[owner]
    plain, seen = getattr(cls, method), []

    def instead(self, *a, **k):
        seen.append(self)
        return plain(self, *a, **k)
    if where == "class":
        monkeypatch.setattr(cls, method, instead)
    else:
        setattr(mod, method, lambda *a, **k: instead(mod, *a, **k))
    for grad in (True, False):
        seen.clear()
        with torch.set_grad_enabled(grad):
            model(ids)
        assert any(m is mod for m in seen)


def test_subclass_of_the_mlp_keeps_its_own_hidden():
    from types import SimpleNamespace
    from picotron_b200.models.llama import MLP
    from picotron_b200.param_store import ParamStore

    class Doubled(MLP):
        def hidden(self, x):
            return 2 * super().hidden(x)
    torch.manual_seed(5)
    with torch.device("cuda"):
        mlp = Doubled(SimpleNamespace(hidden_size=64, intermediate_size=128, init_std=0.05)).to(torch.bfloat16)
    ParamStore(mlp)
    x = _bf16(20, 64)
    y, want = mlp(x), torch.nn.functional.linear(mlp.hidden(x), mlp.down_proj.weight)
    assert (y.float() - want.float()).norm() <= 2 ** -7 * want.float().norm()
