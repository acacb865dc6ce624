"""tcgen05 flash attention against the fp32 torch restatement (``ops.attention.attention_block``):
causal and full, grouped-query heads, ragged sequence lengths, strided q/k/v views of a fused
projection, and the position-offset form that ring attention uses."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


def _run_fwd(q, k, v, causal, q_pos0=0, k_pos0=0):
    from picotron_b200 import ops
    b, sq, H, d = q.shape
    out = torch.empty((b, sq, H, d), device=q.device, dtype=q.dtype)
    lse = torch.empty((b, H, sq), device=q.device, dtype=torch.float32)
    ops.ext().attention_fwd(q, k, v, out, lse, d ** -0.5, causal, q_pos0, k_pos0, None)
    ops.check_status("attention fwd")
    return out, lse


CASES = [  # b, sq, sk, H, Hkv, d, causal
    (2, 128, 128, 4, 4, 64, True), (1, 256, 256, 4, 2, 64, True), (2, 384, 384, 8, 8, 64, False),
    (1, 200, 200, 4, 4, 64, True), (1, 1000, 1000, 2, 1, 64, True), (1, 256, 256, 2, 2, 128, True),
    (2, 130, 130, 4, 2, 128, False), (1, 2048, 2048, 4, 4, 64, True),
]


@pytest.mark.parametrize("b,sq,sk,H,Hkv,d,causal", CASES)
def test_attention_fwd(b, sq, sk, H, Hkv, d, causal):
    from picotron_b200.ops import attention as A
    torch.manual_seed(0)
    q = torch.randn(b, sq, H, d, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(b, sk, Hkv, d, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(b, sk, Hkv, d, device="cuda", dtype=torch.bfloat16)
    out, lse = _run_fwd(q, k, v, causal)
    ref, ref_lse = A.attention_block(q.float(), k.float(), v.float(), causal)
    assert _rel(out, ref) < 1e-2
    assert torch.allclose(lse, ref_lse, atol=2e-2, rtol=1e-3)


def test_attention_fwd_strided_views_of_fused_qkv():
    from picotron_b200.ops import attention as A
    torch.manual_seed(1)
    b, s, H, Hkv, d = 2, 256, 8, 4, 64
    qkv = torch.randn(b, s, (H + 2 * Hkv) * d, device="cuda", dtype=torch.bfloat16)
    q = qkv[..., :H * d].view(b, s, H, d)
    k = qkv[..., H * d:(H + Hkv) * d].view(b, s, Hkv, d)
    v = qkv[..., (H + Hkv) * d:].view(b, s, Hkv, d)
    out, _ = _run_fwd(q, k, v, True)
    ref, _ = A.attention_block(q.float(), k.float(), v.float(), True)
    assert _rel(out, ref) < 1e-2


@pytest.mark.parametrize("q_pos0,k_pos0", [(256, 0), (256, 256), (0, 256), (128, 256)])
def test_attention_fwd_block_offsets(q_pos0, k_pos0):
    """A ring-attention step: queries at global positions q_pos0.., keys at k_pos0..; rows that see
    no key return 0 with lse = -inf."""
    from picotron_b200.ops import attention as A
    torch.manual_seed(2)
    b, s, H, d = 1, 256, 2, 64
    q = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    out, lse = _run_fwd(q, k, v, True, q_pos0, k_pos0)
    ref, ref_lse = A.attention_block(q.float(), k.float(), v.float(), True, None, q_offset=q_pos0, k_offset=k_pos0)
    dead = torch.isinf(ref_lse)
    assert torch.equal(torch.isinf(lse), dead)
    assert _rel(out, ref) < 1e-2 if ref.abs().sum() > 0 else out.abs().sum() == 0
    assert torch.allclose(lse[~dead], ref_lse[~dead], atol=2e-2, rtol=1e-3)


BWD_CASES = [  # b, s, H, Hkv, d, causal
    (2, 128, 2, 2, 64, True), (1, 256, 4, 2, 64, True), (1, 384, 4, 4, 64, False), (1, 200, 2, 1, 64, True),
    (1, 256, 2, 2, 128, True), (1, 300, 4, 2, 128, False), (1, 1024, 4, 4, 64, True),
]


@pytest.mark.parametrize("b,s,H,Hkv,d,causal", BWD_CASES)
def test_attention_autograd(b, s, H, Hkv, d, causal):
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    torch.manual_seed(3)
    q = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(b, s, Hkv, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(b, s, Hkv, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    go = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    out = A.attention(q, k, v, causal)
    out.backward(go)
    ops.check_status("attention bwd")
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = A.attention_ref(qr, kr, vr, causal)
    ref.backward(go.float())
    assert _rel(out, ref) < 1e-2
    assert _rel(q.grad, qr.grad) < 2e-2
    assert _rel(k.grad, kr.grad) < 2e-2
    assert _rel(v.grad, vr.grad) < 2e-2


def test_attention_backward_block_offsets():
    """Backward of one ring step given the merged out / lse of the whole row."""
    from picotron_b200.ops import attention as A
    torch.manual_seed(4)
    b, s, H, d = 1, 256, 2, 64
    q = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    k = torch.randn(b, 2 * s, H, d, device="cuda", dtype=torch.bfloat16)
    v = torch.randn(b, 2 * s, H, d, device="cuda", dtype=torch.bfloat16)
    go = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    # queries are the second half of a 2*s sequence; full causal attention over both key blocks
    out, lse = A.attention_block(q.float(), k.float(), v.float(), True, None, q_offset=s, k_offset=0)
    out = out.to(torch.bfloat16)
    for blk in range(2):
        kb, vb = k[:, blk * s:(blk + 1) * s].contiguous(), v[:, blk * s:(blk + 1) * s].contiguous()
        dq, dk, dv = A.flash_attention_backward(go, q, kb, vb, out, lse, True, None, q_pos0=s, k_pos0=blk * s)
        rq, rk, rv = A.attention_block_backward(go, q, kb, vb, out, lse, True, None, q_offset=s, k_offset=blk * s)
        assert _rel(dq, rq) < 2e-2 and _rel(dk, rk) < 2e-2 and _rel(dv, rv) < 2e-2


@pytest.mark.parametrize("acc_dtype", [torch.float32, torch.bfloat16])
def test_merge_kernel_matches_eager_merge(acc_dtype):
    """Online-softmax merge of two partial results: the kernel against the eager formula, including
    rows that have seen no key on one side or on both (lse = -inf)."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    torch.manual_seed(0)
    b, s, H, d = 2, 300, 6, 64
    out_a = torch.randn(b, s, H, d, device="cuda").to(acc_dtype)
    out_b = torch.randn(b, s, H, d, device="cuda").to(torch.bfloat16)
    lse_a = torch.randn(b, H, s, device="cuda") * 3
    lse_b = torch.randn(b, H, s, device="cuda") * 3
    lse_a[0, 0, :10] = float("-inf")
    lse_b[0, 1, :10] = float("-inf")
    lse_a[1, 2, 5:9] = float("-inf")
    lse_b[1, 2, 5:9] = float("-inf")
    with torch.enable_grad():       # the eager formula is what runs when gradients are recorded
        want_out, want_lse = A.merge_attention_blocks(out_a.clone().requires_grad_(True), lse_a, out_b, lse_b)
    with torch.no_grad():
        got_out, got_lse = A.merge_attention_blocks(out_a.clone(), lse_a.clone(), out_b, lse_b)
    ops.check_status("attn merge")
    assert got_out.dtype == torch.float32
    assert torch.equal(torch.isinf(got_lse), torch.isinf(want_lse))
    fin = ~torch.isinf(want_lse)
    assert torch.allclose(got_lse[fin], want_lse[fin], atol=1e-5, rtol=1e-5)
    assert torch.allclose(got_out, want_out.detach(), atol=2e-3, rtol=1e-3)
    assert got_out[1, 5:9, 2].abs().max().item() == 0.0        # no key on either side: stays zero


def _close(a, b, atol, rtol):
    """Per-element check next to the norm ratio: |a - b| <= atol + rtol * |b| everywhere."""
    return bool(((a.float() - b.float()).abs() <= atol + rtol * b.float().abs()).all())


def test_attention_head_dim_128_at_2048_tokens():
    """head_dim 128 at a training-size sequence (forward and backward), norm ratio and per-element bounds."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    torch.manual_seed(11)
    b, s, H, Hkv, d = 1, 2048, 4, 2, 128
    q = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(b, s, Hkv, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(b, s, Hkv, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    go = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    out = A.attention(q, k, v, True)
    out.backward(go)
    ops.check_status("attention d128 s2048")
    qr, kr, vr = (t.detach().float().requires_grad_(True) for t in (q, k, v))
    ref = A.attention_ref(qr, kr, vr, True)
    ref.backward(go.float())
    assert _rel(out, ref) < 1e-2 and _close(out, ref, atol=2e-2, rtol=2e-2)
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        assert _rel(got, want) < 2e-2
        assert _close(got, want, atol=0.05 * want.abs().max().item(), rtol=5e-2)


def test_attention_long_context_shape_against_library_attention():
    """The long-context benchmark's per-rank shape (16384 tokens, 32 query / 8 KV heads, head_dim 64,
    causal). The fp32 restatement would need a 16384 x 16384 score matrix per head, so the oracle here
    is PyTorch's library attention on the same bf16 inputs (K/V heads repeated for it); forward and
    backward."""
    import torch.nn.functional as F
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    torch.manual_seed(12)
    b, s, H, Hkv, d = 1, 16384, 32, 8, 64
    q = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    k = torch.randn(b, s, Hkv, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    v = torch.randn(b, s, Hkv, d, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    go = torch.randn(b, s, H, d, device="cuda", dtype=torch.bfloat16)
    out = A.attention(q, k, v, True)
    out.backward(go)
    ops.check_status("attention long context")
    qr, kr, vr = (t.detach().clone().requires_grad_(True) for t in (q, k, v))
    rep = H // Hkv
    ref = F.scaled_dot_product_attention(qr.transpose(1, 2), kr.repeat_interleave(rep, dim=2).transpose(1, 2),
                                         vr.repeat_interleave(rep, dim=2).transpose(1, 2), is_causal=True)
    ref = ref.transpose(1, 2)
    ref.backward(go)
    assert _rel(out, ref) < 2e-2
    for got, want in ((q.grad, qr.grad), (k.grad, kr.grad), (v.grad, vr.grad)):
        assert _rel(got, want) < 3e-2


# one tile of a pair without the other, key blocks that outnumber the score buffers, every ragged end
TILE_EDGES = [  # sq, sk, H, Hkv, d, causal, q_pos0
    (44, 700, 2, 1, 64, False, 0), (44, 700, 2, 2, 128, False, 0), (129, 513, 2, 1, 64, False, 0),
    (300, 300, 4, 2, 128, False, 0), (641, 641, 3, 3, 128, True, 0), (1333, 1333, 3, 1, 64, True, 0),
    (255, 257, 2, 2, 64, False, 0), (384, 256, 2, 2, 128, True, 256), (129, 900, 2, 1, 64, True, 771),
]


@pytest.mark.parametrize("sq,sk,H,Hkv,d,causal,q_pos0", TILE_EDGES)
def test_attention_tile_edges_against_64_bits(sq, sk, H, Hkv, d, causal, q_pos0):
    """Forward and gradients against torch in 64 bits. bf16 has 8 significant bits: a result rounded once is
    2^-9 / sqrt(3) = 1.1e-3 off (root mean square); P rounded to bf16 adds as much to the output, P, dS and
    the output's own rounding (through delta) to the gradients. The limits are twice the sums."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    torch.manual_seed(sq + sk + d)
    q, k, v, go = (torch.randn(2, s, n, d, device="cuda", dtype=torch.bfloat16)
                   for s, n in ((sq, H), (sk, Hkv), (sk, Hkv), (sq, H)))
    out, lse = A.flash_attention_forward(q, k, v, causal, None, q_pos0, 0)
    grads = A.flash_attention_backward(go, q, k, v, out, lse, causal, None, q_pos0, 0)
    ops.check_status("attention tile edges")
    q6, k6, v6 = (t.double().requires_grad_() for t in (q, k, v))
    rep = H // Hkv
    s6 = torch.einsum("bqhd,bkhd->bhqk", q6, k6.repeat_interleave(rep, 2)) * d ** -0.5
    if causal:
        hidden = torch.arange(sk, device="cuda")[None] > torch.arange(sq, device="cuda")[:, None] + q_pos0
        s6 = s6.masked_fill(hidden, float("-inf"))
    ref = torch.einsum("bhqk,bkhd->bqhd", s6.softmax(-1), v6.repeat_interleave(rep, 2))
    want = torch.autograd.grad(ref, (q6, k6, v6), go.double())

    def off(a, b):
        return ((a.double() - b).norm() / b.norm()).item()
    assert off(out, ref.detach()) < 4.4e-3
    assert torch.allclose(lse.double(), torch.logsumexp(s6, -1).detach(), atol=1e-4, rtol=1e-5)
    for got, exp in zip(grads, want):
        assert off(got, exp) < 6.6e-3


@pytest.mark.parametrize("b,s,H,Hkv,d,offset", [(1, 1, 1, 1, 64, 0), (2, 129, 4, 2, 64, 5), (1, 300, 3, 1, 128, 0),
                                                (3, 97, 2, 2, 128, 31)])
def test_rotary_attention_gradients_against_64_bits(b, s, H, Hkv, d, offset):
    """dq and dk leave the attention backward rotated back (both halves of a head, ragged lengths, a position offset).
    Values are bf16 roundings of rotated q and k forward (2^-9 each) and of the gradients: 2-norm within 1.5 %."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    from picotron_b200.ops import rope as R
    torch.manual_seed(s + d)
    qkv = torch.randn(b, s, (H + 2 * Hkv) * d, device="cuda").to(torch.bfloat16)
    cos, sin = R.get_cos_sin(s + offset + 3, d, 10000.0, device="cuda")
    ch, sh = R.rope_tables_for_kernel(cos, sin)
    x = qkv.clone().requires_grad_()
    go = torch.randn(b, s, H * d, device="cuda").to(torch.bfloat16)
    (g,) = torch.autograd.grad(A.rope_attention_fused(x * 1, H, Hkv, d, ch, sh, offset), x, go)
    ops.check_status()
    xr = qkv.double().requires_grad_()
    heads = xr.view(b, s, H + 2 * Hkv, d)
    c, n = (t[offset:offset + s].double()[None, :, None] for t in (ch, sh))
    lo, hi = heads.chunk(2, -1)
    turned = torch.cat([lo * c - hi * n, hi * c + lo * n], -1)
    q, k, v = turned[:, :, :H], turned[:, :, H:H + Hkv], heads[:, :, H + Hkv:]
    k, v = (t.repeat_interleave(H // Hkv, dim=2) for t in (k, v))
    score = torch.einsum("bqhd,bkhd->bhqk", q, k) / d ** 0.5
    score = score.masked_fill(torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    out = torch.einsum("bhqk,bkhd->bqhd", score.softmax(-1), v).reshape(b, s, H * d)
    (want,) = torch.autograd.grad(out, xr, go.double())
    for lo_, hi_ in ((0, H), (H, H + Hkv), (H + Hkv, H + 2 * Hkv)):
        a, w = g[..., lo_ * d:hi_ * d].double(), want[..., lo_ * d:hi_ * d]
        if s > 1 or lo_ > H:                       # one token: its probability is 1 and dq, dk are rounding noise
            assert (a - w).norm() <= 0.015 * w.norm()


@pytest.mark.parametrize("b,s,H,Hkv,d,causal,shared", [(1, 300, 1, 1, 64, True, False), (1, 1100, 8, 1, 64, True, True),
                                                       (2, 513, 3, 1, 128, False, True), (1, 129, 2, 2, 128, True, False)])
def test_key_blocks_shared_by_several_ctas(b, s, H, Hkv, d, causal, shared):
    """Few key blocks: where they have enough steps the steps of each are split. dK and dV are sums of the shares in
    order, the same bits on each run; 2-norm of bf16 roundings of P and dS (2^-9 each) and of the results against 64
    bits."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    assert (ops.ext().attention_bwd_splits(b, s, s, H, Hkv, d, causal, 0, 0) > 1) == shared
    torch.manual_seed(s)
    q, go = (torch.randn(b, s, H, d, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(b, s, Hkv, d, device="cuda").to(torch.bfloat16) for _ in range(2))
    out, lse = A.flash_attention_forward(q, k, v, causal)
    first = [t.clone() for t in A.flash_attention_backward(go, q, k, v, out, lse, causal)]
    for _ in range(3):
        dq, dk, dv = A.flash_attention_backward(go, q, k, v, out, lse, causal)
        assert torch.equal(dk, first[1]) and torch.equal(dv, first[2])
    ops.check_status()
    qr, kr, vr = (t.double().requires_grad_() for t in (q, k, v))
    score = torch.einsum("bqhd,bkhd->bhqk", qr, kr.repeat_interleave(H // Hkv, 2)) / d ** 0.5
    if causal:
        score = score.masked_fill(torch.ones(s, s, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = torch.einsum("bhqk,bkhd->bqhd", score.softmax(-1), vr.repeat_interleave(H // Hkv, 2))
    for got, want in zip(first, torch.autograd.grad(ref, (qr, kr, vr), go.double())):
        assert (got.double() - want).norm() <= 3 * 2 ** -9 * want.norm()


@pytest.mark.parametrize("splits", [0, 1, 2, 3, 16])
@pytest.mark.parametrize("b,sq,sk,H,Hkv,d,causal,q0,k0,rope", [
    (1, 300, 300, 1, 1, 64, True, 0, 0, False), (2, 129, 129, 4, 2, 128, True, 0, 0, True),
    (3, 257, 257, 3, 1, 64, True, 0, 0, True), (1, 640, 640, 3, 3, 64, False, 0, 0, True),
    (2, 200, 330, 4, 2, 64, True, 130, 0, False), (1, 1024, 1024, 8, 2, 64, True, 1024, 0, False),
    (1, 300, 300, 2, 1, 128, True, 0, 200, False)])
def test_any_number_of_shares(b, sq, sk, H, Hkv, d, causal, q0, k0, rope, splits):
    """One to 16 shares of a key block's steps, uneven ones and more than there are steps, several batches; steps of a
    ring, where the keys lie behind the queries or ahead of some (rows without a key); rotated q and k, whose gradients
    are rotated back from the slabs. Against 64 bits: roundings of P and dS to bf16 and of the results (2^-9 each), one
    more where dK is rounded before it is rotated."""
    from picotron_b200 import ops
    from picotron_b200.ops import attention as A
    from picotron_b200.ops import rope as R
    torch.manual_seed(sq + sk)
    q, go = (torch.randn(b, sq, H, d, device="cuda").to(torch.bfloat16) for _ in range(2))
    k, v = (torch.randn(b, sk, Hkv, d, device="cuda").to(torch.bfloat16) for _ in range(2))
    tables = ()
    if rope:
        tables = (*R.rope_tables_for_kernel(*R.get_cos_sin(sk + 9, d, 10000.0, device="cuda")), 4)
    out, lse = A.flash_attention_forward(q, k, v, causal, None, q0, k0)

    def run():
        return ops.ext().attention_bwd_new(go, q, k, v, out, lse, d ** -0.5, causal, q0, k0, *(tables or (None, None, 0)),
                                           splits)
    grads = [t.clone() for t in run()]
    again = run()
    assert torch.equal(again[1], grads[1]) and torch.equal(again[2], grads[2])
    ops.check_status()
    q6, k6, v6, g6 = (t.double().transpose(1, 2) for t in (q, k.repeat_interleave(H // Hkv, 2),
                                                           v.repeat_interleave(H // Hkv, 2), go))
    score = q6 @ k6.transpose(-1, -2) * d ** -0.5
    if causal:
        hidden = torch.arange(sk, device="cuda")[None] + k0 > torch.arange(sq, device="cuda")[:, None] + q0
        score = score.masked_fill(hidden, float("-inf"))
    p = score.softmax(-1).nan_to_num(0.0)
    ds = p * (g6 @ v6.transpose(-1, -2) - (g6 * (p @ v6)).sum(-1, keepdim=True)) * d ** -0.5
    want = [ds @ k6, ds.transpose(-1, -2) @ q6, p.transpose(-1, -2) @ g6]
    want = [t.transpose(1, 2) if i == 0 else t.transpose(1, 2).unflatten(2, (Hkv, -1)).sum(3) for i, t in enumerate(want)]
    if rope:
        for i in (0, 1):
            lo, hi = want[i].chunk(2, -1)
            c, n = (t[4:4 + want[i].shape[1]].double()[None, :, None] for t in tables[:2])
            want[i] = torch.cat([lo * c + hi * n, hi * c - lo * n], -1)
    for got, w in zip(grads, want):
        assert (got.double() - w).norm() <= (4 if rope else 3) * 2 ** -9 * w.norm()


def test_wrong_numbers_of_shares_are_refused():
    from picotron_b200 import ops
    q = torch.zeros(1, 64, 1, 64, device="cuda", dtype=torch.bfloat16)
    lse = torch.zeros(1, 1, 64, device="cuda")
    for splits in (-1, 17):
        with pytest.raises(RuntimeError, match="splits"):
            ops.ext().attention_bwd_new(q, q, q, q, q, lse, 1.0, True, 0, 0, None, None, 0, splits)
