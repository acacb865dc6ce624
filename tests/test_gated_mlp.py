"""The gated MLP with the activation inside the GEMMs, against 64-bit products of the same bf16 values."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(got, want, mag, k):
    """fp32 sums of k exact products (2^-24 of their magnitudes each), one rounding to bf16 (2^-8 of the value, with
    room for the activation's fp32 arithmetic)."""
    err = (got.double() - want).abs()
    bound = want.abs() * 2 ** -8 + mag * (k + 2) * 2.0 ** -24 + 1e-30
    assert (err <= bound).all(), (err / bound).max()


@pytest.mark.parametrize("rows,inter,hidden", [(1, 8, 8), (33, 1536, 576), (128, 136, 64), (129, 120, 72),
                                               (300, 264, 520), (4200, 1160, 200)])
@pytest.mark.parametrize("pitch", [0, 16])
def test_products_with_swiglu(rows, inter, hidden, pitch):
    """Less than a tile, half a pair, ragged rows and columns, a gate tile that reaches into the up rows, more tiles
    than pairs; operands with a row pitch."""
    from picotron_b200 import ops
    torch.manual_seed(1)
    dev = dict(device="cuda")
    x = torch.randn(rows, hidden + pitch, **dev).to(torch.bfloat16)[:, :hidden]
    w = (torch.randn(2 * inter, hidden + pitch, **dev) / hidden ** 0.5).to(torch.bfloat16)[:, :hidden]
    gu, act, _ = ops.ext().gemm_swiglu(x, w, True, 1)
    none, act_only, _ = ops.ext().gemm_swiglu(x, w, False, 1)
    ops.check_status()
    _close(gu, x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t(), hidden)
    g, u = gu.double().chunk(2, -1)
    _close(act, torch.nn.functional.silu(g) * u, torch.zeros_like(g), 0)
    assert none.numel() == 0 and torch.equal(act_only, act)
    dy = torch.randn(rows, hidden + pitch, **dev).to(torch.bfloat16)[:, :hidden]
    wd = (torch.randn(hidden, inter + pitch, **dev) / inter ** 0.5).to(torch.bfloat16)[:, :inter]
    dgu, _ = ops.ext().gemm_swiglu_bwd(dy, wd, gu, 1)
    ops.check_status()
    d, mag = dy.double() @ wd.double(), dy.double().abs() @ wd.double().abs()
    sg = torch.sigmoid(g)
    dg_of, du_of = u * sg * (1 + g * (1 - sg)), g * sg
    dg, du = dgu.chunk(2, -1)
    # 1 + g (1 - sigmoid) cancels for g near -1.28: its terms are at most 1 + |g|, a few 2^-24 of the factors around it
    slack = 16 * 2.0 ** -24 * d.abs() * u.abs() * sg * (1 + g.abs())
    err = (dg.double() - d * dg_of).abs()
    bound = (d * dg_of).abs() * 2 ** -8 + mag * dg_of.abs() * (hidden + 2) * 2 ** -24
    assert (err <= bound + slack + 1e-30).all()
    _close(du, d * du_of, mag * du_of.abs(), hidden)


@pytest.mark.parametrize("rows", [75, 2560])
@pytest.mark.parametrize("keep_grad_of_x", [True, False])
def test_mlp_module_takes_the_one_op_and_matches_the_separate_ones(keep_grad_of_x, rows):
    """Few rows (products and a pass) and enough for the fused epilogues: gradients accumulate in main_grad; a hook on
    the down projection selects the separate ops."""
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200.models.llama import MLP
    from picotron_b200.param_store import ParamStore
    torch.manual_seed(2)
    with torch.device("cuda"):
        mlp = MLP(SimpleNamespace(hidden_size=1024, intermediate_size=2064, init_std=0.05)).to(torch.bfloat16)
    store = ParamStore(mlp)
    for backward in (False, True):
        assert ops.ext().gemm_swiglu_pays(2 * rows, 2064, 1024, True, backward) == (rows > 75)
    x = torch.randn(2, rows, 1024, device="cuda").to(torch.bfloat16).requires_grad_(keep_grad_of_x)
    dy = torch.randn(2, rows, 1024, device="cuda").to(torch.bfloat16)
    got = []
    for separate in (False, True):
        seen = []
        handle = mlp.down_proj.register_forward_hook(lambda *a: seen.append(1)) if separate else None
        store.zero_grads()
        x.grad = None
        y = mlp(x)
        y.backward(dy)
        with torch.no_grad():
            assert torch.equal(mlp(x), y)
        assert bool(seen) == separate
        if handle is not None:
            handle.remove()
        got.append((y.detach().clone(), store.flat_grads.clone(), x.grad.clone() if keep_grad_of_x else None))
    ops.check_status()
    assert torch.equal(got[0][0], got[1][0])
    # the separate path rounds the gradient of the activation to bf16 (2^-9 each): sums of such errors
    for a, b in zip(got[0][1:], got[1][1:]):
        if a is not None:
            assert (a.float() - b.float()).norm() <= 2 ** -8 * b.float().norm()
    assert all(p.grad is None for p in mlp.parameters())


def _tiles(counts, spare):
    """Group of every 128-row tile for groups of these many tiles, and `spare` tiles of no group behind them."""
    return torch.tensor([g for g, c in enumerate(counts) for _ in range(c)] + [-1] * spare, dtype=torch.int32).cuda()


@pytest.mark.parametrize("counts,spare,inter,hidden", [([1, 7, 16], 0, 64, 64), ([3, 0, 8, 1, 4], 9, 136, 128),
                                                       ([33, 31, 1], 2, 320, 192), ([0, 0, 12], 13, 264, 64),
                                                       ([2] * 40 + [9] * 40, 0, 192, 128)])
def test_row_groups_on_pairs(counts, spare, inter, hidden):
    """Odd and even segments, empty groups, tiles of no group, segments across the stretches of 32 tiles in which pairs
    are listed, more pairs than the chip has: plain products and those with the activation, each row against its group's
    matrix in 64 bits. Rows of no group keep what was there."""
    from picotron_b200 import ops
    torch.manual_seed(sum(counts))
    G, tg = len(counts), _tiles(counts, spare)
    P = tg.numel() * 128
    assert ops.ext().gemm_rows_on_pairs(P, G)
    group = tg.long().repeat_interleave(128)
    x = torch.randn(P, hidden, device="cuda").to(torch.bfloat16)
    dy = torch.randn(P, hidden, device="cuda").to(torch.bfloat16)
    wg = (torch.randn(G, 2 * inter, hidden, device="cuda") / hidden ** 0.5).to(torch.bfloat16)
    wd = (torch.randn(G, hidden, inter, device="cuda") / inter ** 0.5).to(torch.bfloat16)
    gu, act = ops.ext().grouped_swiglu(x, wg.view(-1, hidden), tg, G)
    dgu = ops.ext().grouped_swiglu_bwd(dy, wd.view(-1, inter), gu, tg, G)
    plain = torch.full((P, 2 * inter), 7.0, device="cuda", dtype=torch.bfloat16)
    back = torch.full((P, inter), 7.0, device="cuda", dtype=torch.bfloat16)
    ops.ext().gemm_grouped(x, wg.view(-1, hidden), plain, P, 2 * inter, hidden, hidden, hidden, 2 * inter, False, False,
                           0, 0, tg, G, 2 * inter)
    ops.ext().gemm_grouped(dy, wd.view(-1, inter), back, P, inter, hidden, hidden, inter, inter, False, True, 0, 0, tg,
                           G, hidden)
    ops.check_status()
    assert (plain[group < 0] == 7).all() and (back[group < 0] == 7).all()
    for g, c in enumerate(counts):
        if c == 0:
            continue
        r = group == g
        xs, w, ds, v = x[r].double(), wg[g].double(), dy[r].double(), wd[g].double()
        _close(plain[r], xs @ w.t(), xs.abs() @ w.abs().t(), hidden)
        _close(back[r], ds @ v, ds.abs() @ v.abs(), hidden)
        assert torch.equal(gu[r], plain[r])
        ga, up = gu[r].double().chunk(2, -1)
        _close(act[r], torch.nn.functional.silu(ga) * up, torch.zeros_like(ga), 0)
        d, mag, sg = ds @ v, ds.abs() @ v.abs(), torch.sigmoid(ga)
        dga, dup = dgu[r].chunk(2, -1)
        _close(dup, d * ga * sg, mag * (ga * sg).abs(), hidden)
        of = up * sg * (1 + ga * (1 - sg))
        slack = 16 * 2.0 ** -24 * d.abs() * up.abs() * sg * (1 + ga.abs())
        bound = (d * of).abs() * 2 ** -8 + mag * of.abs() * (hidden + 2) * 2.0 ** -24 + slack + 1e-30
        assert ((dga.double() - d * of).abs() <= bound).all()


@pytest.mark.parametrize("counts,spare,N,K,on_pairs", [([5, 0, 9, 1, 13, 3], 1, 2048, 1024, True),
                                                       ([11, 12, 1], 0, 2184, 2048, True),
                                                       ([2] * 40 + [9] * 40, 3, 1032, 704, True),
                                                       ([11, 12, 1], 0, 512, 512, False),
                                                       ([33, 0, 91], 2, 1024, 192, False)])
@pytest.mark.parametrize("b_mn_major", [False, True])
def test_plain_products_with_row_groups(counts, spare, N, K, on_pairs, b_mn_major):
    """Either side of the rule between the one-CTA kernel and pairs: odd and empty segments, ragged columns, tiles of no
    group, several rounds."""
    from picotron_b200 import ops
    torch.manual_seed(N + K)
    G, tg = len(counts), _tiles(counts, spare)
    P = tg.numel() * 128
    assert ops.ext().gemm_rows_plan(0, P, N, K, G) == on_pairs
    group = tg.long().repeat_interleave(128)
    x = torch.randn(P, K, device="cuda").to(torch.bfloat16)
    w = (torch.randn(G, *((K, N) if b_mn_major else (N, K)), device="cuda") / K ** 0.5).to(torch.bfloat16)
    out = torch.full((P, N), 7.0, device="cuda", dtype=torch.bfloat16)
    w2 = w.view(-1, w.shape[-1])
    ops.ext().gemm_grouped(x, w2, out, P, N, K, K, w2.shape[1], N, False, b_mn_major, 0, 0, tg, G,
                           K if b_mn_major else N)
    ops.check_status()
    assert (out[group < 0] == 7).all()
    for g, c in enumerate(counts):
        if c:
            a, b = x[group == g].double(), w[g].double() if b_mn_major else w[g].double().t()
            _close(out[group == g], a @ b, a.abs() @ b.abs(), K)


def test_expert_layer_with_the_activation_inside_matches_the_separate_ops(monkeypatch):
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.ops import grouped_gemm
    from picotron_b200.param_store import ParamStore
    from picotron_b200.parallel.expert_parallel import MoELayer
    if pgm.process_group_manager is None:
        pgm.setup_process_group_manager(1, 1, 1, 1, 1)
    torch.manual_seed(5)
    cfg = SimpleNamespace(hidden_size=256, intermediate_size=192, num_experts=4, num_experts_per_tok=2, init_std=0.05)
    with torch.device("cuda"):
        layer = MoELayer(cfg).to(torch.bfloat16)
    layer.train()
    store = ParamStore(layer)
    x = torch.randn(1, 1500, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    dy = torch.randn_like(x)
    got = []
    for separate in (False, True):
        if separate:
            monkeypatch.setattr(grouped_gemm, "grouped_mlp", lambda *a: None)
        store.zero_grads()
        x.grad = None
        before = ops.launches()
        y = layer(x)
        y.backward(dy)
        got.append((y.detach().clone(), x.grad.clone(), store.flat_grads.clone(), ops.launches() - before))
    ops.check_status()
    assert torch.equal(got[0][0], got[1][0]) and got[0][3] == got[1][3] - 2
    # the separate path rounds the activation's gradient; then the roundings of gate | up's gradient, of the routed
    # rows' and of their sum fall differently on the two sides: 2^-9 of the value each, three of them on either side
    for a, b in zip(got[0][1:3], got[1][1:3]):
        assert (a.float() - b.float()).norm() <= (1 + 2 * 3) * 2 ** -9 * b.float().norm()


def _expert_layer():
    from types import SimpleNamespace
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.param_store import ParamStore
    from picotron_b200.parallel.expert_parallel import MoELayer
    if pgm.process_group_manager is None:
        pgm.setup_process_group_manager(1, 1, 1, 1, 1)
    cfg = SimpleNamespace(hidden_size=256, intermediate_size=192, num_experts=4, num_experts_per_tok=2, init_std=0.05)
    with torch.device("cuda"):
        layer = MoELayer(cfg).to(torch.bfloat16)
    layer.train()
    return layer, ParamStore(layer)


def _nodes(fn, seen=None):
    """Names of all nodes of a graph."""
    seen = {} if seen is None else seen
    if fn is not None and fn not in seen:
        seen[fn] = fn.name()
        for nxt, _ in fn.next_functions:
            _nodes(nxt, seen)
    return " ".join(seen.values())


def test_down_projections_of_experts_are_ready_before_the_products_of_gate_and_up(monkeypatch):
    """A data-parallel reduction that a down projection's hook starts runs beside the rest of the backward pass: its
    hooks come before the input gradient and the weight gradient of gate and up, as with the separate operators."""
    from picotron_b200 import ops
    from picotron_b200.ops import grouped_gemm
    torch.manual_seed(6)
    layer, store = _expert_layer()
    x = torch.randn(1, 1500, 256, device="cuda").to(torch.bfloat16).requires_grad_()
    events = []
    for name, p in layer.named_parameters():
        p.grad_ready_hook = lambda kind=name.split(".")[-2]: events.append(kind)
    for name in ("grouped_gemm_nn", "grouped_gemm_tn"):
        plain = getattr(grouped_gemm, name)
        monkeypatch.setattr(grouped_gemm, name, lambda *a, _f=plain, _n=name, **k: (events.append(_n), _f(*a, **k))[1])
    y = layer(x)
    assert "GroupedMLP" in _nodes(y.grad_fn)
    y.backward(torch.randn_like(y))
    ops.check_status()
    events = [e for e in events if e != "gate"]                   # the router's
    assert events[:1] + events[5:7] == ["grouped_gemm_tn", "grouped_gemm_nn", "grouped_gemm_tn"]
    assert events[1:5] == ["down_proj"] * 4 and sorted(events[7:]) == ["gate_proj"] * 4 + ["up_proj"] * 4


@pytest.mark.parametrize("grouped", [False, True])
@pytest.mark.parametrize("learns", ["down", "up and down", "input"])
def test_gate_and_up_that_no_gradient_reaches_get_none(grouped, learns):
    """Frozen gate and up projections of an input that needs no gradient stay out of the backward pass, as with the
    separate operators: nothing is added to their main_grad and their hooks stay silent."""
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200.models.llama import MLP
    from picotron_b200.ops import grouped_gemm
    from picotron_b200.param_store import ParamStore
    torch.manual_seed(7)
    if grouped:
        layer, store = _expert_layer()
        experts = list(layer.local_experts)
        layout = grouped_gemm.GroupLayout.uniform(4, 1024, "cuda")
        x = torch.randn(4096, 256, device="cuda").to(torch.bfloat16)
    else:
        with torch.device("cuda"):
            layer = MLP(SimpleNamespace(hidden_size=256, intermediate_size=192, init_std=0.05)).to(torch.bfloat16)
        store, experts = ParamStore(layer), [layer]
        x = torch.randn(300, 256, device="cuda").to(torch.bfloat16)
    gate_up = [m for e in experts for m in (e.gate_proj, e.up_proj)]
    downs = [e.down_proj for e in experts]
    called = set()
    for m in gate_up + downs:
        m.weight.grad_ready_hook = lambda m=m: called.add(m)
    for m in gate_up:
        m.weight.requires_grad_(learns == "up and down" and any(m is e.up_proj for e in experts))
    x.requires_grad_(learns == "input")
    y = grouped_gemm.grouped_mlp(x, gate_up, downs, layout) if grouped else layer(x)
    assert "MLPFn" in y.grad_fn.name()
    y.backward(torch.randn_like(y))
    ops.check_status()
    assert all(m.weight.main_grad.any() for m in downs) and called >= set(downs)
    reached = learns != "down"            # one product accumulates for both of the pair
    assert all(bool(m.weight.main_grad.any()) == reached and (m in called) == reached for m in gate_up)
