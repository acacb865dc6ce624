"""Routing ops of the mixture-of-experts layer (``ops.moe_route``): the PyTorch restatements against
the layer's own eager routing code on CPU, and the kernels against the restatements on the GPU
(router forward / backward, slot assignment, weighted combine forward / backward)."""
import pytest
import torch


def _routing_case(T=96, E=16, k=3, seed=0):
    g = torch.Generator().manual_seed(seed)
    logits = torch.randn(T, E, generator=g) * 2.0
    bias = torch.randn(E, generator=g) * 0.1
    return logits, bias


def test_reference_router_matches_the_layer_code():
    from picotron_b200.ops import moe_route as mr
    logits, bias = _routing_case()
    for b in (None, bias):
        for renorm in (True, False):
            probs, idx, w, counts = mr.route_ref(logits, b, 3, renorm)
            p = torch.softmax(logits, -1, dtype=torch.float32)
            sc = p + b if b is not None else p
            want_idx = torch.topk(sc, 3, dim=-1).indices
            assert torch.equal(idx, want_idx)
            ww = p.gather(-1, want_idx)
            if renorm:
                ww = ww / ww.sum(-1, keepdim=True)
            assert torch.allclose(w, ww) and torch.allclose(probs, p)
            assert counts.sum().item() == idx.numel() and torch.equal(counts, torch.bincount(idx.reshape(-1), minlength=16))


def test_reference_slots_and_combine_match_the_capacity_path():
    from picotron_b200.ops import moe_route as mr
    from picotron_b200.parallel.capacity_moe import slot_assignment
    g = torch.Generator().manual_seed(1)
    T, E, k, C, d = 64, 8, 2, 10, 16
    idx = torch.randint(0, E, (T, k), generator=g)
    pos, table = mr.slots_ref(idx, E, C)
    assert torch.equal(pos, slot_assignment(idx.reshape(-1), E))
    rows = torch.arange(T * k)
    for r in rows.tolist():
        e, ps = idx.reshape(-1)[r].item(), pos[r].item()
        if ps < C:
            assert table[e * C + ps].item() == r
    assert (table >= 0).sum().item() == (pos < C).sum().item()
    out = torch.randn(E * C, d, generator=g)
    w = torch.rand(T, k, generator=g)
    y = mr.combine_ref(out, idx, pos.view(T, k), w, C)
    want = torch.zeros(T, d)
    for t in range(T):
        for j in range(k):
            ps = pos.view(T, k)[t, j].item()
            if ps < C:
                want[t] += w[t, j] * out[idx[t, j].item() * C + ps]
    assert torch.allclose(y, want, atol=1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("E,k,renorm,use_bias", [(64, 6, True, True), (8, 2, True, False), (16, 1, False, True),
                                                (200, 8, False, False)])
def test_route_kernel_matches_reference(E, k, renorm, use_bias):
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    torch.manual_seed(E + k)
    T = 777
    # every row is a random permutation of E distinct values that bf16 represents exactly: no ties, so the
    # selection is unambiguous (which of two equal scores wins is not part of the contract)
    step = 1.0 / 32 if E > 64 else 1.0 / 8
    perm = torch.rand(T, E, device="cuda").argsort(dim=-1).float()
    logits = ((perm - E / 2) * step).to(torch.bfloat16).requires_grad_(True)
    assert torch.equal(logits.detach().float(), (perm - E / 2) * step)
    bias = (torch.randn(E, device="cuda") * 0.001) if use_bias else None
    probs, idx, w, counts = mr.route(logits, bias, k, renorm)
    ref_logits = logits.detach().float().requires_grad_(True)
    rp, ri, rw, rc = mr.route_ref(ref_logits, bias, k, renorm)
    assert idx.dtype == torch.int32 and torch.equal(idx.long(), ri), "selected experts differ"
    assert torch.allclose(probs, rp, atol=1e-6, rtol=1e-4) and torch.allclose(w, rw, atol=1e-6, rtol=1e-4)
    assert torch.equal(counts.long(), rc)
    # backward: gradient through the weights and a dense gradient w.r.t. the probabilities (aux loss)
    gw = torch.randn_like(rw)
    gp = torch.randn_like(rp) * 0.1
    ((w * gw).sum() + (probs * gp).sum()).backward()
    ((rw * gw).sum() + (rp * gp).sum()).backward()
    err = (logits.grad.float() - ref_logits.grad).abs().max().item()
    scale = ref_logits.grad.abs().max().item()
    assert err <= 1e-2 * scale + 1e-6, (err, scale)      # bf16 rounding of the returned gradient
    ops.check_status("moe route")


@pytest.mark.gpu
@pytest.mark.parametrize("E,k", [(8, 2), (8, 8), (33, 3), (64, 6), (256, 8)])
@pytest.mark.parametrize("use_bias", [False, True])
def test_route_kernel_stays_in_range_for_rows_that_are_not_finite(E, k, use_bias):
    """A token whose logits hold NaN or infinities still gets k different experts of the E there are (the tables that
    follow are indexed with them), weights that carry the NaN, and leaves the other tokens' choices alone."""
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    torch.manual_seed(E * 10 + k)
    T, inf, nan = 300, float("inf"), float("nan")
    perm = torch.rand(T, E, device="cuda").argsort(dim=-1).float()
    logits = ((perm - E / 2) / 32).to(torch.bfloat16)
    bias = torch.randn(E, device="cuda") * 1e-4 if use_bias else None
    _, clean_idx, clean_w, _ = mr.route(logits, bias, k, True)
    bad = {3: nan, 64: inf, 65: -inf}                       # one entry: NaN, +inf (softmax NaN), -inf (softmax fine)
    for row, value in bad.items():
        logits[row, E // 2] = value
    logits[100], logits[101], logits[102] = nan, inf, -inf   # whole rows: no score compares
    not_finite = torch.zeros(T, dtype=torch.bool, device="cuda")
    not_finite[[3, 64, 100, 101, 102]] = True
    logits.requires_grad_()
    probs, idx, w, counts = mr.route(logits, bias, k, True)
    ops.check_status("moe route")
    assert idx.min().item() >= 0 and idx.max().item() < E
    assert (idx.long().sort(dim=1).values.diff(dim=1) > 0).all(), "an expert twice"
    assert torch.equal(counts.long(), torch.bincount(idx.reshape(-1).long(), minlength=E)) and counts.numel() == E
    assert torch.equal(torch.isnan(probs).all(dim=1), not_finite) and torch.equal(torch.isnan(w).all(dim=1), not_finite)
    assert (idx[not_finite].long() == torch.arange(k, device="cuda")).all()
    same = ~not_finite
    same[65] = False
    assert torch.equal(idx[same], clean_idx[same]) and torch.equal(w[same], clean_w[same])
    assert probs[65, E // 2].item() == 0 and w[65].isfinite().all()
    (w * torch.randn_like(w)).sum().backward()
    assert torch.equal(logits.grad.isfinite().all(dim=1), ~not_finite)


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,k,C", [(512, 8, 2, 100), (4096, 64, 6, 300), (100, 4, 1, 1000)])
def test_slots_kernel_matches_reference(T, E, k, C):
    from picotron_b200.ops import moe_route as mr
    g = torch.Generator(device="cuda").manual_seed(T)
    idx = torch.randint(0, E, (T, k), device="cuda", generator=g, dtype=torch.int32)
    pos, table = mr.slots(idx, E, C)
    rpos, rtable = mr.slots_ref(idx.long(), E, C)
    assert torch.equal(pos.long(), rpos) and torch.equal(table, rtable)


@pytest.mark.gpu
def test_combine_kernel_matches_reference():
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    torch.manual_seed(3)
    T, E, k, C, d = 600, 16, 4, 120, 256
    idx = torch.randint(0, E, (T, k), device="cuda", dtype=torch.int32)
    pos, table = mr.slots(idx, E, C)
    out = torch.randn(E * C, d, device="cuda").to(torch.bfloat16).requires_grad_(True)
    w = torch.rand(T, k, device="cuda").requires_grad_(True)
    y = mr.combine(out, idx, pos.view(T, k), w, table, C)
    ro, rw = out.detach().float().requires_grad_(True), w.detach().clone().requires_grad_(True)
    ry = mr.combine_ref(ro, idx.long(), pos.view(T, k).long(), rw, C)
    assert (y.float() - ry).abs().max().item() <= 2e-2 * ry.abs().max().item()
    g = torch.randn(T, d, device="cuda").to(torch.bfloat16)
    y.backward(g)
    ry.backward(g.float())
    assert (out.grad.float() - ro.grad).abs().max().item() <= 2e-2 * ro.grad.abs().max().item() + 1e-6
    assert (w.grad - rw.grad).abs().max().item() <= 2e-2 * rw.grad.abs().max().item() + 1e-6
    assert (pos >= C).any(), "the case should contain rows over capacity"
    ops.check_status("moe combine")


def test_reference_layout_orders_and_pads():
    from picotron_b200.ops import moe_route as mr
    idx = torch.tensor([[2, 0], [2, 1], [0, 2]])
    slot, table, seg, owner = mr.layout_ref(idx, 4)
    assert seg.tolist() == [0, 128, 256, 384, 384] and owner.tolist() == [0, 1, 2, -1, -1]
    assert slot.tolist() == [256, 0, 257, 128, 1, 258]
    assert all(table[s].item() == r for r, s in enumerate(slot.tolist())) and (table >= 0).sum() == 6


@pytest.mark.parametrize("rows,E", [(1, 256), (8, 256), (255, 256), (300, 256), (129, 1), (1000, 7), (4096, 64)])
def test_layout_buffers_hold_every_routing_and_little_more(rows, E):
    """Enough tiles for the routing that pads most (single rows in as many experts as there are, the rest in one), and
    never a tile for an expert that cannot have a row."""
    from picotron_b200.ops import moe_route as mr
    n = min(rows, E)
    counts = [1] * (n - 1) + [rows - (n - 1)]
    worst = sum((c + 127) // 128 for c in counts)
    assert worst <= mr.max_tiles(rows, E) <= worst + (rows + 127) // 128
    idx = torch.tensor([e for e, c in enumerate(counts) for _ in range(c)])
    slot, table, seg, owner = mr.layout_ref(idx, E)
    assert table.numel() == 128 * mr.max_tiles(rows, E) == 128 * owner.numel() and seg[-1] == 128 * worst


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,k", [(1, 256, 8), (3, 256, 1), (40, 64, 6)])
def test_layout_kernel_with_more_experts_than_rows(T, E, k):
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    idx = torch.stack([torch.randperm(E, device="cuda")[:k] for _ in range(T)]).int()
    counts = torch.bincount(idx.reshape(-1), minlength=E).int()
    slot, table, layout = mr.local_layout(idx, counts)
    ops.check_status("moe layout")
    rslot, rtable, rseg, rowner = mr.layout_ref(idx, E)
    used = rseg[-1].item()
    assert torch.equal(slot, rslot) and torch.equal(table[:used], rtable[:used])
    assert torch.equal(layout.seg_start, rseg) and torch.equal(layout.tile_group, rowner)


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,k,skew", [(1, 4, 1, 0), (777, 64, 6, 0), (4096, 256, 8, 2), (2731, 8, 6, 3), (8192, 64, 6, 1)])
def test_layout_kernel_matches_reference(T, E, k, skew):
    """Row counts around the 16 rows of a thread and the 16384 rows of a pass, experts without rows, one that has
    most of them."""
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    g = torch.Generator(device="cuda").manual_seed(T + E)
    idx = (torch.rand(T, k, device="cuda", generator=g) ** (1 + skew) * E).int().clamp_(max=E - 1)
    counts = torch.bincount(idx.reshape(-1), minlength=E).int()
    slot, table, layout = mr.local_layout(idx, counts)
    ops.check_status("moe layout")
    rslot, rtable, rseg, rowner = mr.layout_ref(idx, E)
    used = rseg[-1].item()
    assert torch.equal(slot, rslot) and torch.equal(table[:used], rtable[:used])
    assert torch.equal(layout.seg_start, rseg) and torch.equal(layout.tile_group, rowner) and layout.rows == rtable.numel()


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,k,latent", [(5, 8, 2, 0), (300, 8, 1, 0), (1000, 16, 6, 256)])
def test_local_experts_layer_matches_the_tensor_path(T, E, k, latent, monkeypatch):
    """The device-routed layer against the same layer on sorted, padded tensors (weights rounded to bf16 there: the
    outputs may differ by that and by their own rounding, 2^-8 each)."""
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.parallel.expert_parallel import MoELayer
    if pgm.process_group_manager is None:
        pgm.setup_process_group_manager(1, 1, 1, 1, 1)
    torch.manual_seed(T)
    with torch.device("cuda"):
        layer = MoELayer(SimpleNamespace(hidden_size=512, intermediate_size=256, num_experts=E, num_experts_per_tok=k,
                                         moe_latent_dim=latent, shared_expert_intermediate_size=256)).to(torch.bfloat16)
    x0 = torch.randn(T, 512, device="cuda", dtype=torch.bfloat16)
    dy = torch.randn(T, 512, device="cuda", dtype=torch.bfloat16)
    got = []
    for flag in ("1", "0"):
        monkeypatch.setenv("PICO_MOE_DEVICE_ROUTING", flag)
        x = x0.clone().requires_grad_()
        assert layer._local_routed_ok(x) == (flag == "1")
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        y.backward(dy)
        got.append([y.detach(), x.grad] + [p.grad.clone() for p in layer.parameters() if p.grad is not None])
    ops.check_status("moe layer")
    assert len(got[0]) == len(got[1])
    for a, b in zip(*got):
        assert ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-6)).item() < 2 ** -6


@pytest.mark.gpu
def test_layout_reports_rows_that_it_cannot_place():
    """Indices that name no expert and counts that disagree with the indices: everything read later stays inside the
    tables (slot -1, row -1), the other rows lie where they would, and the status words say so."""
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    T, E, k, d = 300, 4, 2, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    idx = torch.randint(0, E, (T, k), device="cuda", generator=g, dtype=torch.int32)
    good = idx.clone()
    idx[7, 1], idx[8, 0], idx[299, 1] = E, -1, 2 ** 31 - 1
    placed = ((idx >= 0) & (idx < E)).reshape(-1)
    counts = torch.bincount(idx.reshape(-1)[placed], minlength=E).int()
    slot, table, layout = mr.local_layout(idx, counts)
    with pytest.raises(RuntimeError, match="bounds"):
        ops.check_status()
    want, fill = [], [0] * E
    for e in idx.reshape(-1).tolist():
        want.append(layout.seg_start[e].item() + fill[e] if 0 <= e < E else -1)
        if 0 <= e < E:
            fill[e] += 1
    assert slot.tolist() == want
    used = layout.seg_start[-1].item()
    rows = torch.arange(T * k, device="cuda", dtype=torch.int32)[placed]
    assert torch.equal(table[slot[placed].long()], rows) and (table[:used] >= 0).sum().item() == rows.numel()
    # the sums: NaN for the tokens with such a row, the others as always
    x = torch.randn(T, d, device="cuda", generator=g).to(torch.bfloat16).requires_grad_()
    w = torch.rand(T, k, device="cuda", generator=g).requires_grad_()
    out = mr.gather_rows(x, slot, table, layout, k)
    y = mr.combine_rows(out, w, slot, table, layout)
    y.backward(torch.ones_like(y))
    bad = torch.zeros(T, dtype=torch.bool, device="cuda")
    bad[[7, 8, 299]] = True
    assert torch.equal(torch.isnan(y).all(dim=1), bad) and torch.equal(torch.isnan(x.grad).all(dim=1), bad)
    assert torch.allclose(y[~bad].float(), (x * w.sum(1, keepdim=True))[~bad].float(), rtol=2 ** -7)
    assert (w.grad.reshape(-1)[~placed] == 0).all() and w.grad.isfinite().all()
    # counts below and above what the indices hold, and far beyond the tables
    for wrong in ([0, 0, 0, 0], [1, 600, 0, 300], [2 ** 31 - 1] * E, [-5] * E):
        slot, table, layout = mr.local_layout(good, torch.tensor(wrong, device="cuda", dtype=torch.int32))
        with pytest.raises(RuntimeError, match="bounds"):
            ops.check_status()
        used = layout.seg_start[-1].item()
        assert 0 <= used <= layout.rows and slot.max().item() < used and slot.min().item() >= -1
        assert used == 0 or (table[:used].max().item() < T * k and table[:used].min().item() >= -1)
        assert layout.tile_group.max().item() < E and layout.tile_group.min().item() >= -1
        assert (layout.seg_start.diff() >= 0).all()


@pytest.mark.gpu
def test_gather_of_more_rows_than_32_bits_count_threads_for():
    """A warp per row from 2^27 rows on: 2^32 threads and more."""
    from picotron_b200 import ops
    n, d, k = 2 ** 27 + 5, 8, 2
    x = torch.randn(1024, d, device="cuda").to(torch.bfloat16)
    row = torch.arange(n, device="cuda", dtype=torch.int32) % (1024 * k)
    row[::1000] = -1
    out = torch.empty(n, d, device="cuda", dtype=torch.bfloat16)
    ops.ext().moe_gather(x, row, torch.tensor([n], device="cuda", dtype=torch.int32), out, k)
    ops.check_status()
    for lo in range(0, n, 2 ** 24):
        r = row[lo:lo + 2 ** 24]
        want = x[r.clamp(min=0).long() // k].masked_fill((r < 0)[:, None], 0)
        assert torch.equal(out[lo:lo + 2 ** 24], want)


@pytest.mark.gpu
@pytest.mark.parametrize("E,k", [(8, 2), (64, 6)])
def test_tokens_that_are_not_finite_stay_among_themselves(E, k):
    """A diverging token through the whole layer: NaN in its own outputs and input gradient, the others as without it."""
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.parallel.expert_parallel import MoELayer
    if pgm.process_group_manager is None:
        pgm.setup_process_group_manager(1, 1, 1, 1, 1)
    torch.manual_seed(E)
    with torch.device("cuda"):
        layer = MoELayer(SimpleNamespace(hidden_size=512, intermediate_size=256, num_experts=E,
                                         num_experts_per_tok=k)).to(torch.bfloat16)
    clean = torch.randn(257, 512, device="cuda", dtype=torch.bfloat16)
    dirty = clean.clone()
    dirty[3, 17], dirty[200] = float("nan"), float("inf")
    dy = torch.randn_like(clean)
    got = []
    for x in (clean, dirty):
        x.requires_grad_()
        assert layer._local_routed_ok(x)
        y = layer(x)
        y.backward(dy)
        got.append((y.detach(), x.grad))
    ops.check_status("moe layer")
    same = torch.ones(257, dtype=torch.bool, device="cuda")
    same[[3, 200]] = False
    for a, b in zip(*got):
        assert torch.isnan(b[~same]).all() and torch.equal(a[same], b[same])


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["hook", "module"])
def test_a_gate_that_gives_fp32_logits_keeps_its_route(how, monkeypatch):
    """Logits that are not bf16 (a forward hook, a gate of the user's own without a ``weight``) are routed in fp32 by
    the tensor path, as before the local experts had kernels of their own."""
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.parallel.expert_parallel import MoELayer
    if pgm.process_group_manager is None:
        pgm.setup_process_group_manager(1, 1, 1, 1, 1)
    torch.manual_seed(11)
    with torch.device("cuda"):
        layer = MoELayer(SimpleNamespace(hidden_size=256, intermediate_size=256, num_experts=8,
                                         num_experts_per_tok=2)).to(torch.bfloat16)
    if how == "hook":
        layer.gate.register_forward_hook(lambda mod, args, out: out.float() * 1.0009765625)
    else:
        class Gate(torch.nn.Module):
            def __init__(self):
                super().__init__()
                self.table = torch.nn.Parameter(torch.randn(256, 8, device="cuda"))

            def forward(self, x):
                return x.float() @ self.table
        layer.gate = Gate()
    x = torch.randn(300, 256, device="cuda", dtype=torch.bfloat16)
    got = []
    for flag in ("1", "0"):
        monkeypatch.setenv("PICO_MOE_DEVICE_ROUTING", flag)
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        y.float().square().sum().backward()
        got.append([y.detach()] + [p.grad.clone() for p in layer.parameters()])
    ops.check_status("moe layer")
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.gpu
@pytest.mark.parametrize("renorm,aux,bias_rate", [(False, 0.0, 0.0), (True, 0.01, 0.0), (True, 0.0, 0.05), (False, 0.02, 0.1)])
def test_local_experts_layer_balances_like_the_tensor_path(renorm, aux, bias_rate, monkeypatch):
    """Raw router probabilities as weights, the auxiliary loss (its dense gradient enters the router beside the
    weights') and the loss-free bias (selection by probability + bias, update from the kernel's counts): outputs,
    gradients, loss and bias against the layer on sorted, padded tensors over three steps. The tensor path rounds the
    weights to bf16, so outputs and gradients may differ by that and their own rounding, 2^-8 each."""
    from types import SimpleNamespace
    from picotron_b200 import ops
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.parallel.expert_parallel import MoELayer
    if pgm.process_group_manager is None:
        pgm.setup_process_group_manager(1, 1, 1, 1, 1)
    torch.manual_seed(7)
    with torch.device("cuda"):
        layer = MoELayer(SimpleNamespace(hidden_size=256, intermediate_size=256, num_experts=16, num_experts_per_tok=3,
                                         norm_topk_prob=renorm, router_aux_loss_coef=aux,
                                         router_bias_update_rate=bias_rate)).to(torch.bfloat16)
    layer.train()
    layer.expert_bias = layer.expert_bias.float()
    xs = [torch.randn(700, 256, device="cuda", dtype=torch.bfloat16) for _ in range(3)]
    dy = torch.randn(700, 256, device="cuda", dtype=torch.bfloat16)
    got = []
    for flag in ("1", "0"):
        monkeypatch.setenv("PICO_MOE_DEVICE_ROUTING", flag)
        layer.expert_bias.zero_()
        layer.zero_grad(set_to_none=True)
        values, exact = [], []
        for x0 in xs:
            x = x0.clone().requires_grad_()
            assert layer._local_routed_ok(x) == (flag == "1")
            y = layer(x)
            loss = (y * dy).float().sum()
            assert (layer.aux_loss is not None) == (aux > 0)
            if aux > 0:
                values.append(layer.aux_loss.detach().reshape(1))
                loss = loss + 1000.0 * layer.aux_loss
            loss.backward()
            values += [y.detach(), x.grad]
            exact.append(layer.expert_bias.clone())
        got.append((values + [p.grad.clone() for p in layer.parameters()], exact))
    ops.check_status("moe layer")
    for a, b in zip(got[0][0], got[1][0]):
        assert ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-6)).item() < 2 ** -6
    assert all(torch.equal(a, b) for a, b in zip(got[0][1], got[1][1])) and (got[0][1][-1].any().item() == (bias_rate > 0))


@pytest.mark.gpu
@pytest.mark.parametrize("T,E,k", [(1, 8, 8), (700, 32, 8), (5000, 64, 8), (300, 65, 3), (300, 128, 8), (300, 129, 8)])
def test_route_kernel_at_the_edges_of_its_lanes(T, E, k):
    """One, two, four and eight experts per lane at their limits, more tokens than warps: the choice and the counts are
    exact (distinct logits), probabilities and weights fp32 (1e-6)."""
    from picotron_b200 import ops
    from picotron_b200.ops import moe_route as mr
    g = torch.Generator().manual_seed(E)
    logits = torch.stack([torch.randperm(E, generator=g) for _ in range(T)]).float().div(16).to(torch.bfloat16).cuda()
    probs, idx, w, counts = mr.route(logits, None, k, True)
    ops.check_status()
    want = torch.softmax(logits.double(), -1)
    chosen = torch.sort(logits.float(), dim=-1, descending=True, stable=True).indices[:, :k]
    ww = want.gather(1, chosen)
    if k > 1:
        ww = ww / ww.sum(-1, keepdim=True)
    assert torch.equal(idx.long(), chosen) and torch.equal(counts.long(), torch.bincount(chosen.flatten(), minlength=E))
    assert torch.allclose(probs.double(), want, atol=1e-6) and torch.allclose(w.double(), ww, atol=1e-6)
