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
    """Less than a tile, half a pair, ragged rows and columns, a gate tile that reaches into the up rows, more tiles than
    pairs; operands with a row pitch."""
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
    err, bound = (dg.double() - d * dg_of).abs(), (d * dg_of).abs() * 2 ** -8 + mag * dg_of.abs() * (hidden + 2) * 2 ** -24
    assert (err <= bound + slack + 1e-30).all()
    _close(du, d * du_of, mag * du_of.abs(), hidden)


@pytest.mark.parametrize("rows", [75, 2560])
@pytest.mark.parametrize("keep_grad_of_x", [True, False])
def test_mlp_module_takes_the_one_op_and_matches_the_separate_ones(keep_grad_of_x, rows):
    """Few rows (products and a pass) and enough for the fused epilogues: gradients accumulate in main_grad; a hook on the
    down projection selects the separate ops."""
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
