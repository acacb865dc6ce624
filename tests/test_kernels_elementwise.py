"""Memory-bound kernels against fp32 torch restatements of the same ops."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


@pytest.mark.parametrize("rows,H", [(64, 256), (1000, 2048), (33, 4096), (7, 8192), (5, 520)])
def test_rmsnorm_fwd_bwd(rows, H):
    from picotron_b200 import ops
    from picotron_b200.ops import norm
    torch.manual_seed(0)
    x = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = (1 + 0.1 * torch.randn(H, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    y = norm.rmsnorm(x, w, 1e-5)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    yr = norm.rmsnorm_ref(xr, wr, 1e-5)
    yr.backward(g.float())
    ops.check_status()
    assert _rel(y, yr) < 1e-2
    assert _rel(x.grad, xr.grad) < 1e-2
    assert _rel(w.grad, wr.grad) < 2e-2


def test_add_rmsnorm_and_main_grad():
    from picotron_b200.ops import norm
    torch.manual_seed(1)
    rows, H = 300, 2048
    x = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.nn.Parameter((1 + 0.1 * torch.randn(H, device="cuda")).to(torch.bfloat16))
    w.main_grad = torch.zeros(H, device="cuda", dtype=torch.float32)
    y, h = norm.add_rmsnorm(x, r, w, 1e-5)
    gy, gh = torch.randn_like(y), torch.randn_like(h)
    torch.autograd.backward([y, h], [gy, gh])
    xr = x.detach().float().requires_grad_(True)
    rr = r.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    # the kernel rounds the summed stream to bf16 before normalising (straight-through here)
    hr = (xr + rr) + ((xr + rr).to(torch.bfloat16).float() - (xr + rr)).detach()
    yr = norm.rmsnorm_ref(hr, wr, 1e-5)
    torch.autograd.backward([yr, hr], [gy.float(), gh.float()])
    assert _rel(y, yr) < 1e-2 and _rel(h, hr) < 1e-2
    assert _rel(x.grad, xr.grad) < 1e-2 and _rel(r.grad, rr.grad) < 1e-2
    assert w.grad is None and _rel(w.main_grad, wr.grad) < 2e-2


@pytest.mark.parametrize("d", [64, 128])
def test_rope(d):
    from picotron_b200.ops import rope
    torch.manual_seed(2)
    b, s, nh = 2, 48, 6
    cos, sin = rope.get_cos_sin(128, d, base=10000.0, device="cuda")
    x = torch.randn(b, s, nh, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = rope.apply_rope(x, cos, sin, pos_offset=16)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_(True)
    yr = rope.apply_rope_ref(xr, cos, sin, pos_offset=16)
    yr.backward(g.float())
    assert _rel(y, yr) < 1e-2 and _rel(x.grad, xr.grad) < 1e-2


def test_swiglu():
    from picotron_b200.ops import swiglu
    torch.manual_seed(3)
    gu = torch.randn(5, 37, 2 * 688, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = swiglu.swiglu(gu)
    g = torch.randn_like(y)
    y.backward(g)
    gr = gu.detach().float().requires_grad_(True)
    yr = swiglu.swiglu_ref(gr)
    yr.backward(g.float())
    assert _rel(y, yr) < 1e-2 and _rel(gu.grad, gr.grad) < 1e-2


def test_swiglu_with_device_side_row_count():
    """Rows at or past a fill level that lives on the device are skipped, forward and backward."""
    from picotron_b200.ops import swiglu
    torch.manual_seed(5)
    gu = torch.randn(300, 2 * 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    n = torch.tensor([129], device="cuda", dtype=torch.int32)
    y = swiglu.swiglu(gu, rows_in_use=n)
    g = torch.randn_like(y)
    y[:129].backward(g[:129])
    gr = gu.detach().float().requires_grad_(True)
    yr = swiglu.swiglu_ref(gr)
    yr[:129].backward(g[:129].float())
    assert _rel(y[:129], yr[:129]) < 1e-2 and _rel(gu.grad[:129], gr.grad[:129]) < 1e-2


@pytest.mark.parametrize("rows,V", [(64, 4096), (300, 49152), (17, 32000)])
def test_cross_entropy(rows, V):
    from picotron_b200.ops import cross_entropy as ce
    torch.manual_seed(4)
    logits = (3 * torch.randn(rows, V, device="cuda")).to(torch.bfloat16).requires_grad_(True)
    t = torch.randint(0, V, (rows,), device="cuda")
    lr = logits.detach().float().requires_grad_(True)
    loss_r = ce.cross_entropy_ref(lr, t)
    loss_r.mean().backward()
    loss = ce.cross_entropy(logits * 1.0, t, inplace=True)
    loss.mean().backward()
    assert torch.allclose(loss, loss_r, atol=2e-3, rtol=2e-3)
    assert _rel(logits.grad, lr.grad) < 2e-2


def test_cross_entropy_vocab_shards_combine():
    """Two column shards evaluated separately and merged by hand equal the dense loss."""
    from picotron_b200 import ops
    torch.manual_seed(5)
    rows, V = 50, 1024
    logits = (2 * torch.randn(rows, V, device="cuda")).to(torch.bfloat16)
    t = torch.randint(0, V, (rows,), device="cuda")
    e = ops.ext()
    stats = []
    for r in range(2):
        sh = logits[:, r * 512:(r + 1) * 512].contiguous()
        st = torch.empty(rows, 3, device="cuda")
        e.ce_stats(sh, 512, t, st, rows, 512, r * 512)
        stats.append(st)
    g = torch.stack(stats)
    m = g[..., 0].max(0).values
    s = (g[..., 1] * torch.exp(g[..., 0] - m)).sum(0)
    tl = g[..., 2].sum(0)
    loss = s.log() + m - tl
    ref = torch.nn.functional.cross_entropy(logits.float(), t, reduction="none")
    assert torch.allclose(loss, ref, atol=2e-3, rtol=2e-3)


def test_adamw_matches_torch():
    from picotron_b200.ops.adamw import FlatAdamW
    torch.manual_seed(6)
    n = 100_003
    p = torch.randn(n, device="cuda").to(torch.bfloat16)
    g = torch.randn(n, device="cuda")
    ref_p = torch.nn.Parameter(p.float().clone())
    opt_ref = torch.optim.AdamW([ref_p], lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1)
    opt = FlatAdamW(p, g.clone(), lr=1e-2, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.1, master_weights=True)
    for i in range(3):
        opt.grads.copy_(g * (i + 1))
        ref_p.grad = (g * (i + 1)) * 0.5
        opt.step(grad_scale=0.5, zero_grad=True)
        opt_ref.step()
    assert opt.grads.abs().sum().item() == 0
    assert torch.allclose(opt.master, ref_p.detach(), atol=1e-5, rtol=1e-5)
    assert _rel(p, ref_p.detach()) < 1e-2


def test_embedding():
    from picotron_b200.ops import embedding as emb
    torch.manual_seed(7)
    V, H = 1000, 256
    w = torch.nn.Parameter(torch.randn(V, H, device="cuda", dtype=torch.bfloat16))
    ids = torch.randint(0, 2 * V, (4, 33), device="cuda")
    out = emb.embedding(ids, w, vocab_start=500)
    ref = emb.embedding_ref(ids, w.detach().float(), vocab_start=500)
    assert _rel(out, ref) < 1e-3
    g = torch.randn_like(out)
    out.backward(g)
    wr = w.detach().float().requires_grad_(True)
    emb.embedding_ref(ids, wr, vocab_start=500).backward(g.float())
    assert _rel(w.grad, wr.grad) < 1e-2


@pytest.mark.parametrize("rows,H", [(1, 8), (3, 512), (129, 576), (1200, 8), (1300, 960), (5, 1032), (700, 1544), (2049, 2048), (7, 2056)])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm_row_widths_against_64_bits(rows, H, residual):
    """Both directions at the widths where the thread count changes. Outputs are rounded once to bf16 (half of the last
    of 8 bits, 2^-9 of the value on average size and at most 2^-8 of it); the weight gradient is a sum of ``rows``
    fp32 products of bf16 numbers, rounded to bf16 at the end."""
    from picotron_b200 import ops
    from picotron_b200.ops import norm
    torch.manual_seed(rows + H)
    x = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    r = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16, requires_grad=True) if residual else None
    w = torch.randn(H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16)
    y, h = norm.add_rmsnorm(x, r, w, 1e-5)
    grads = torch.autograd.grad((y, h) if residual else (y,), (x, w), (dy, dy) if residual else (dy,))
    ops.check_status("rmsnorm")
    h6 = (x.detach() + r.detach() if residual else x.detach()).double().requires_grad_()
    w6 = w.detach().double().requires_grad_()
    y6 = h6 * torch.rsqrt(h6.pow(2).mean(-1, keepdim=True) + 1e-5) * w6
    want = torch.autograd.grad((y6, h6) if residual else (y6,), (h6, w6), (dy.double(),) * (2 if residual else 1))
    for got, exp in ((y, y6.detach()), (grads[0], want[0]), (grads[1], want[1])):
        scale = exp.abs().clamp_min(exp.pow(2).mean().sqrt())
        assert ((got.double() - exp).abs() / scale).max().item() < 2 ** -8 + 1e-5


@pytest.mark.parametrize("rows,H", [(1, 576), (3, 960), (301, 2048), (5, 4096), (5, 1032), (7, 2056)])
def test_rmsnorm_backward_keeps_infinities_where_they_are(rows, H):
    """An infinity in the last row's gradient (rows are worked on two at a time) makes its own column of the weight
    gradient infinite, not NaN, and leaves the other columns and rows alone."""
    from picotron_b200 import ops
    from picotron_b200.ops import norm
    torch.manual_seed(H)
    x = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16).abs_().add_(0.5).requires_grad_()
    w = torch.ones(H, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    dy = torch.randn(rows, H, device="cuda", dtype=torch.bfloat16)
    clean = torch.autograd.grad(norm.rmsnorm(x, w, 1e-5), (x, w), dy)
    dy[-1, 5] = float("inf")
    dx, dw = torch.autograd.grad(norm.rmsnorm(x, w, 1e-5), (x, w), dy)
    ops.check_status("rmsnorm")
    others = torch.arange(H, device="cuda") != 5
    assert dw[5].item() == float("inf") and torch.equal(dw[others], clean[1][others])
    assert torch.equal(dx[:-1], clean[0][:-1]) and not dx[-1].isfinite().any()


@pytest.mark.parametrize("rows,V", [(3, 8), (5, 24), (700, 4104), (301, 49152), (2, 57344), (3, 57352)])
def test_cross_entropy_rows_in_one_pass(rows, V):
    """Rows shorter than the copies they arrive in, more rows than CTAs, the longest row of the one-pass kernel and the
    first of the two-pass one; targets at both ends and outside, -inf logits. fp32 sums of exact bf16 inputs: 1e-5;
    gradients are rounded to bf16 once: 2^-8 of the value, and 1e-5 of the largest for the fp32 part of small ones."""
    from picotron_b200 import ops
    from picotron_b200.ops import cross_entropy as ce
    torch.manual_seed(9)
    logits = (4 * torch.randn(rows, V, device="cuda")).to(torch.bfloat16)
    logits[0, 1::2] = -float("inf")
    t = torch.randint(0, V, (rows,), device="cuda")
    t[0], t[-1] = 0, V - 1
    t[1] = -100                       # no target in this shard: log-sum-exp alone
    ref = logits.double()
    lse = torch.logsumexp(ref, -1)
    inside = (t >= 0) & (t < V)
    hit = torch.zeros_like(ref)
    hit[inside, t[inside]] = 1
    want = lse - torch.where(inside, ref.gather(1, t.clamp(0, V - 1)[:, None])[:, 0], torch.zeros_like(lse))
    dwant = ((ref - lse[:, None]).exp() - hit) / rows
    loss = torch.empty(rows, device="cuda")
    for d in (torch.empty_like(logits), logits):          # beside the logits, then over them
        ce._stats_loss_grad(logits, t, loss, d, 1.0 / rows, 0, None)
        ops.check_status()
        assert torch.allclose(loss.double(), want, rtol=1e-5, atol=1e-5)
        assert ((d.double() - dwant).abs() <= dwant.abs() * 2 ** -8 + 1e-5 / rows).all()


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("rows,H", [(1, 8), (777, 576)])
def test_embedding_gradient_of_repeated_ids(rows, H, offset):
    """Few ids, many rows; a gradient buffer at 16-byte alignment and one off it. fp32 sums of at most 777 bf16 values:
    777 * 2^-24 of the sum of their magnitudes."""
    from picotron_b200 import ops
    torch.manual_seed(10)
    V = 7
    dout = torch.randn(rows, H, device="cuda").to(torch.bfloat16)
    ids = torch.randint(0, V + 2, (rows,), device="cuda")         # two of them outside the shard
    dw = torch.zeros(V * H + offset, device="cuda")[offset:].view(V, H)
    ops.ext().embedding_bwd(dout, ids, dw, rows, H, V, 0)
    keep = ids < V
    want = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids[keep], dout[keep].double())
    mag = torch.zeros(V, H, device="cuda", dtype=torch.float64).index_add_(0, ids[keep], dout[keep].double().abs())
    assert ((dw.double() - want).abs() <= mag * rows * 2 ** -24).all()
