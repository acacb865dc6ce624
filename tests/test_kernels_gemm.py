"""tcgen05 GEMM against an fp32 torch reference: all operand layouts, output modes, ragged
shapes (M, N, K not multiples of the tile) and strided views."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops():
    from picotron_b200 import ops
    from picotron_b200.ops import gemm
    return ops, gemm


def _rel_err(a, b):
    return ((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-12)).item()


SHAPES = [(128, 256, 64), (256, 512, 128), (1024, 2048, 512), (200, 264, 72), (8, 64, 2048),
          (4096, 1536, 2048), (136, 136, 200), (384, 128, 4096), (64, 8192, 256)]


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_nt(M, N, K):
    ops, gemm = _ops()
    torch.manual_seed(0)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    out = gemm.gemm_nt(a, b)
    ref = a.float() @ b.float().t()
    ops.check_status()
    assert _rel_err(out, ref) < 1e-2
    out32 = gemm.gemm_nt(a, b, out_dtype=torch.float32)
    ops.check_status()
    assert _rel_err(out32, ref) < 1e-5


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_nn(M, N, K):
    ops, gemm = _ops()
    torch.manual_seed(1)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    out = gemm.gemm_nn(a, b)
    ops.check_status()
    assert _rel_err(out, a.float() @ b.float()) < 1e-2


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_tn_and_accumulate(M, N, K):
    ops, gemm = _ops()
    torch.manual_seed(2)
    a = torch.randn(K, M, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    ref = a.float().t() @ b.float()
    out = gemm.gemm_tn(a, b)
    ops.check_status()
    assert _rel_err(out, ref) < 1e-2
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    base = acc.clone()
    gemm.gemm_tn(a, b, out=acc, accumulate=True)
    gemm.gemm_tn(a, b, out=acc, accumulate=True)
    ops.check_status()
    assert _rel_err(acc, base + 2 * ref) < 1e-5


def test_gemm_strided_views():
    ops, gemm = _ops()
    torch.manual_seed(3)
    big = torch.randn(512, 1024, device="cuda", dtype=torch.bfloat16)
    a = big[:, 256:768]                      # row stride 1024, K = 512
    w = torch.randn(384, 512, device="cuda", dtype=torch.bfloat16)
    outbuf = torch.zeros(512, 1024, device="cuda", dtype=torch.bfloat16)
    out = outbuf[:, 128:512]
    gemm.gemm_nt(a, w, out=out)
    ops.check_status()
    assert _rel_err(out, a.float() @ w.float().t()) < 1e-2
    assert outbuf[:, :128].abs().sum().item() == 0 and outbuf[:, 512:].abs().sum().item() == 0


def test_linear_autograd_matches_torch():
    ops, gemm = _ops()
    torch.manual_seed(4)
    x = torch.randn(4, 96, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.randn(512, 256, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    y = gemm.linear(x, w)
    g = torch.randn_like(y)
    y.backward(g)
    xr = x.detach().float().requires_grad_(True)
    wr = w.detach().float().requires_grad_(True)
    yr = torch.nn.functional.linear(xr, wr)
    yr.backward(g.float())
    ops.check_status()
    assert _rel_err(y, yr) < 1e-2
    assert _rel_err(x.grad, xr.grad) < 1e-2
    assert _rel_err(w.grad, wr.grad) < 1e-2


def test_linear_main_grad_accumulation():
    ops, gemm = _ops()
    torch.manual_seed(5)
    x = torch.randn(256, 128, device="cuda", dtype=torch.bfloat16, requires_grad=True)
    w = torch.nn.Parameter(torch.randn(64, 128, device="cuda", dtype=torch.bfloat16))
    w.main_grad = torch.zeros(64, 128, device="cuda", dtype=torch.float32)
    for _ in range(3):
        gemm.linear(x, w).sum().backward()
    ops.check_status()
    assert w.grad is None
    ref = 3 * torch.ones(256, 64, device="cuda").t() @ x.detach().float()
    assert _rel_err(w.main_grad, ref) < 1e-5


# ---------------------------------------------------------------------------------------------
# grouped GEMM over the local experts of a mixture-of-experts layer
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("counts,d_in,d_out", [([128, 256, 128], 128, 256), ([5, 0, 300, 129], 256, 384),
                                                ([1000, 17, 64, 512, 3, 250, 0, 77], 512, 1024)])
def test_grouped_gemm_forward_dgrad_wgrad(counts, d_in, d_out):
    ops, _ = _ops()
    from picotron_b200.ops import grouped_gemm as gg
    torch.manual_seed(3)
    G = len(counts)
    n = sum(counts)
    layout = gg.GroupLayout.from_counts(counts, "cuda")
    assert layout.rows % 128 == 0 and layout.tile_group.numel() == max(layout.rows // 128, 1)
    x = torch.randn(n, d_in, device="cuda", dtype=torch.bfloat16)
    w = torch.randn(G * d_out, d_in, device="cuda", dtype=torch.bfloat16) * 0.1
    xp = layout.pad(x)
    # forward
    y = layout.unpad(gg.grouped_gemm_nt(xp, w, layout, d_out))
    ops.check_status()
    ref, off = [], 0
    for e, c in enumerate(counts):
        ref.append(x[off:off + c].float() @ w[e * d_out:(e + 1) * d_out].float().t())
        off += c
    ref = torch.cat(ref)
    assert _rel_err(y, ref) < 1e-2
    # input gradient
    dy = torch.randn(n, d_out, device="cuda", dtype=torch.bfloat16)
    dyp = layout.pad(dy)
    dx = layout.unpad(gg.grouped_gemm_nn(dyp, w, layout, d_out))
    ops.check_status()
    ref, off = [], 0
    for e, c in enumerate(counts):
        ref.append(dy[off:off + c].float() @ w[e * d_out:(e + 1) * d_out].float())
        off += c
    assert _rel_err(dx, torch.cat(ref)) < 1e-2
    # weight gradient, accumulated into fp32; experts without rows keep their old values
    acc = torch.randn(G * d_out, d_in, device="cuda", dtype=torch.float32)
    base = acc.clone()
    gg.grouped_gemm_tn(dyp, xp, layout, acc, accumulate=True)
    ops.check_status()
    off = 0
    for e, c in enumerate(counts):
        want = base[e * d_out:(e + 1) * d_out] + dy[off:off + c].float().t() @ x[off:off + c].float()
        got = acc[e * d_out:(e + 1) * d_out]
        assert _rel_err(got, want) < 1e-4, (e, c)
        off += c


def test_moe_layer_grouped_experts_match_per_expert_loop():
    """The MoE layer on the grouped-GEMM path (stacked expert weights in a ParamStore, gradients
    accumulated into main_grad) against the same layer run expert by expert in plain PyTorch."""
    import copy
    import types
    ops, _ = _ops()
    from picotron_b200 import process_group_manager as pgm
    from picotron_b200.param_store import ParamStore
    from picotron_b200.parallel.expert_parallel import MoELayer
    pgm.process_group_manager = None
    cfg = types.SimpleNamespace(hidden_size=256, intermediate_size=128, num_experts=8, num_experts_per_tok=2,
                                init_std=0.05, num_shared_experts=1)
    torch.manual_seed(0)
    layer = MoELayer(cfg, ep_group=False).to("cuda", torch.bfloat16)
    ref = copy.deepcopy(layer)
    store = ParamStore(layer)
    assert any(len(g.mods) == 16 for g in store.fused_groups) and any(len(g.mods) == 8 for g in store.fused_groups)
    x = torch.randn(2, 192, 256, device="cuda", dtype=torch.bfloat16)
    xr = x.clone().requires_grad_(True)
    x.requires_grad_(True)
    before = ops.launches()
    y = layer(x)
    y.float().square().mean().backward()
    ops.check_status()
    assert ops.launches() - before > 0
    import os
    os.environ["PICO_REFERENCE_OPS"] = "1"
    try:
        yr = ref(xr)
        yr.float().square().mean().backward()
    finally:
        os.environ["PICO_REFERENCE_OPS"] = "0"
    assert _rel_err(y, yr) < 2e-2
    assert _rel_err(x.grad, xr.grad) < 3e-2
    for (n, p), (_, q) in zip(layer.named_parameters(), ref.named_parameters()):
        g = p.main_grad if getattr(p, "main_grad", None) is not None and p.grad is None else p.grad
        assert _rel_err(g, q.grad) < 5e-2, n


@pytest.mark.parametrize("my_rank", [0, 1, 3])
def test_dropless_ep_layout_kernel_matches_reference(my_rank):
    """The device-side layout of the dropless expert-parallel exchange (offsets of outgoing blocks,
    padded expert segments, tile -> expert array, return blocks) against its Python restatement, with
    empty experts, experts that are exact multiples of the tile, and a table that does not fit."""
    ops, _ = _ops()
    from picotron_b200.ops.fused_ep_var import var_layout_ref
    ep, L = 4, 3
    E = ep * L
    g = torch.Generator().manual_seed(7)
    table = torch.randint(0, 300, (ep, E), generator=g, dtype=torch.int32)
    table[:, 2] = 0                  # an expert nobody routes to
    table[:, 5] = 32                 # 4 x 32 = exactly one tile
    for max_rows in (128 * 40, 128 * 6):      # roomy, and too small for some experts
        dev = table.cuda()
        send = torch.empty((E, 4), device="cuda", dtype=torch.int32)
        ret = torch.empty((ep * L, 4), device="cuda", dtype=torch.int32)
        seg_start = torch.empty(L + 1, device="cuda", dtype=torch.int32)
        seg_len = torch.empty(L, device="cuda", dtype=torch.int32)
        tiles = torch.empty(max_rows // 128, device="cuda", dtype=torch.int32)
        ops.ext().ep_var_layout(dev, ep, L, my_rank, max_rows, send, ret, seg_start, seg_len, tiles)
        r_send, r_ret, r_seg, r_len, r_tiles = var_layout_ref(table.tolist(), L, my_rank, max_rows)
        assert send.cpu().tolist() == r_send
        got_ret, want_ret = ret.cpu().tolist(), r_ret
        for a, b in zip(got_ret, want_ret):
            assert a[0] == b[0] and a[2:] == b[2:] and (a[0] == 0 or a[1] == b[1]), (a, b)
        assert seg_start.cpu().tolist() == r_seg and seg_len.cpu().tolist() == r_len
        assert tiles.cpu().tolist() == r_tiles
        words = ops.ext().status_fetch()       # the small table reports the rows it could not place
        assert (words[0] != 0) == (max_rows == 128 * 6)


# ---------------------------------------------------------------------------------------------
# CTA-pair tiles: sizes whose modelled time chooses them, with ragged ends in every dimension
# ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K", [(4000, 4104, 520), (4104, 4000, 72), (8192, 2056, 1000)])
def test_pair_tiles_all_layouts(M, N, K):
    """bf16 results of fp32 sums: within the output's rounding of the 64-bit product, 2^-8 of the value (half of the
    last of its 8 bits), plus the sum's error, sqrt(K) 2^-24 of the row's size, against the 1e-2 floor: 2e-4."""
    ops, gemm = _ops()
    torch.manual_seed(M + K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    ref = a.double() @ b.double().t()
    scale = ref.abs().clamp_min(ref.pow(2).mean().sqrt() * 1e-2)
    for out in (gemm.gemm_nt(a, b), gemm.gemm_nn(a, b.t().contiguous()),
                gemm.gemm_tn(a.t().contiguous(), b.t().contiguous())):
        ops.check_status("pair gemm")
        assert ((out.double() - ref).abs() / scale).max().item() < 2 ** -8 + 2e-4


@pytest.mark.parametrize("M,N,K,max_ctas", [(4000, 4104, 520, 0), (8192, 2056, 1000, 0), (1016, 1528, 8, 2),
                                            (504, 760, 72, 2), (512, 744, 384, 7), (496, 504, 392, 5), (1488, 760, 1000, 37)])
def test_pair_tiles_with_pitched_operands_and_limited_grids(M, N, K, max_ctas):
    """Column slices of wider matrices as operands and results (fused projections have them), one pair, an odd number of
    CTAs, from one K block to more than the six stages. Limits as in test_pair_tiles_all_layouts; what lies beside a
    result stays."""
    ops, gemm = _ops()
    plan = ops.ext().gemm_plan
    for a_mn, b_mn, mode in ((False, False, 0), (False, True, 0), (True, True, 0), (True, True, 2)):
        pairs, bn, tiles, whole = plan(0, M, N, K, a_mn, b_mn, mode, max_ctas)
        assert pairs > 0 and (max_ctas == 0 or (pairs == max_ctas // 2 and whole == tiles))
    torch.manual_seed(M + K)

    def sliced(rows, cols, dtype=torch.bfloat16):
        return torch.randn(rows, (cols + 31) // 8 * 8, device="cuda").to(dtype)[:, 16:16 + cols]
    a, b = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.randn(N, K, device="cuda").to(torch.bfloat16)
    a_k, a_m, b_k, b_n = sliced(M, K), sliced(K, M), sliced(N, K), sliced(K, N)
    for view, dense in ((a_k, a), (a_m, a.t()), (b_k, b), (b_n, b.t())):
        view.copy_(dense)
    ref = a.double() @ b.double().t()
    scale = ref.abs().clamp_min(ref.pow(2).mean().sqrt() * 1e-2)
    for product, x, y in ((gemm.gemm_nt, a_k, b_k), (gemm.gemm_nn, a_k, b_n), (gemm.gemm_tn, a_m, b_n)):
        wide = torch.full((M, N + 24), 7.0, device="cuda", dtype=torch.bfloat16)
        product(x, y, out=wide[:, 8:8 + N], max_ctas=max_ctas)
        ops.check_status("pair gemm")
        assert ((wide[:, 8:8 + N].double() - ref).abs() / scale).max().item() < 2 ** -8 + 2e-4
        assert (wide[:, :8] == 7).all() and (wide[:, 8 + N:] == 7).all()
    acc = sliced(M, N, torch.float32)
    want = acc.double() + ref
    gemm.gemm_tn(a_m, b_n, out=acc, accumulate=True, max_ctas=max_ctas)
    ops.check_status("pair gemm accumulate")
    assert ((acc.double() - want).norm() / want.norm()).item() < 1e-5


def test_sizes_of_the_pair_tests_run_on_pairs():
    """The tests of the pair kernel that take their kernel from the size rule, and the cut ones from its cut."""
    ops, _ = _ops()
    plan = ops.ext().gemm_plan
    for M, N, K in ((4000, 4104, 520), (4104, 4000, 72), (8192, 2056, 1000)):
        assert all(plan(0, M, N, K, a, b, 0, 0)[0] > 0 for a, b in ((False, False), (False, True), (True, True)))
    for M, N, K in ((520, 776, 4096), (5120, 960, 8192), (576, 264, 16384)):
        pairs, _, tiles, whole = plan(0, M, N, K, True, True, 2, 0)
        assert pairs > 0 and whole < tiles
    pairs, _, tiles, whole = plan(0, 2048, 2048, 1999, True, True, 2, 0)       # 64 tiles on 74 pairs: as they are
    assert pairs > 0 and whole == tiles


@pytest.mark.parametrize("M,N,K", [(520, 776, 4096), (2048, 2048, 1999), (5120, 960, 8192), (576, 264, 16384)])
def test_pair_tiles_accumulate_with_a_cut_last_round(M, N, K):
    """The last round's tiles are cut along K and added in pieces: fp32 sums, 1e-5 of the 64-bit result, and
    what D held before stays in it."""
    ops, gemm = _ops()
    torch.manual_seed(M + K)
    a = torch.randn(K, M, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(K, N, device="cuda", dtype=torch.bfloat16)
    acc = torch.randn(M, N, device="cuda", dtype=torch.float32)
    ref = acc.double() + 2 * (a.double().t() @ b.double())
    for _ in range(2):
        gemm.gemm_tn(a, b, out=acc, accumulate=True)
    ops.check_status("pair gemm accumulate")
    assert ((acc.double() - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.parametrize("M,N,K", [(6144, 2048, 8192), (960, 960, 8192), (5120, 960, 8192), (516, 771, 4096),
                                   (512, 512, 16384), (3072, 2040, 7000)])
def test_cut_last_round_gives_the_same_bits_on_each_run(M, N, K):
    """Pieces of a tile come from different pairs, two to eighteen of them: D, the first piece and the others are added
    in that order whoever is done first. Column slices of wider buffers, N without a factor of 4; another stream's
    work moves the pairs' finishing order about. fp32 sums: 1e-5 of the 64-bit result, nothing beside the slice."""
    ops, gemm = _ops()
    pairs, _, tiles, whole = ops.ext().gemm_plan(0, M, N, K, True, True, 2, 0)
    assert pairs and whole < tiles
    torch.manual_seed(M + K)
    a = torch.randn(K, (M + 63) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, 32:32 + M]
    b = torch.randn(K, (N + 15) // 8 * 8, device="cuda", dtype=torch.bfloat16)[:, :N]
    before = torch.randn(M, (N + 7) // 4 * 4 + 4, device="cuda")
    wide, side, noise = before.clone(), torch.cuda.Stream(), torch.randn(2 ** 24, device="cuda")
    first = None
    for run in range(6):
        wide.copy_(before)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(run):
                noise.mul_(1.0)
        launched = ops.launches()
        gemm.gemm_tn(a, b, out=wide[:, 4:4 + N], accumulate=True)
        assert ops.launches() - launched == 2            # the product and the kernel that adds the pieces
        torch.cuda.current_stream().wait_stream(side)
        first = wide.clone() if first is None else first
        assert torch.equal(wide, first)
    ops.check_status("pair gemm, cut")
    ref = before.double()
    ref[:, 4:4 + N] += a.double().t() @ b.double()
    assert torch.equal(first[:, :4], before[:, :4]) and torch.equal(first[:, 4 + N:], before[:, 4 + N:])
    assert ((first.double() - ref).norm() / ref.norm()).item() < 1e-5


@pytest.mark.parametrize("M,N,K", [(128, 576, 49152), (1, 64, 8192), (33, 960, 20000), (1000, 520, 32768), (130, 136, 6400)])
def test_products_summed_in_parts_of_k(M, N, K):
    """Few tiles and a long reduction: parts of K added in fp32 in order, rounded once; the same bits again: 2^-8 of the value for the rounding. The
    sums: K / 16 adds of a running sum up to 4 times the result's size, each cut off at 2^-23 of it (the tensor cores
    do not round), relative to the value or the results' root mean square, whichever is larger."""
    ops, gemm = _ops()
    torch.manual_seed(M + K)
    a = torch.randn(M, K, device="cuda", dtype=torch.bfloat16)
    b = torch.randn(N, K, device="cuda", dtype=torch.bfloat16)
    assert gemm._parts_of_k(M, N, K) >= 2
    ref = a.double() @ b.double().t()
    scale = ref.abs().clamp_min(ref.pow(2).mean().sqrt())
    wide = torch.zeros(M, N + 8, device="cuda", dtype=torch.bfloat16)
    for out in (gemm.gemm_nt(a, b), gemm.gemm_nn(a, b.t().contiguous()), gemm.gemm_nt(a, b, out=wide[:, 8:])):
        ops.check_status("gemm in parts")
        assert ((out.double() - ref).abs() / scale).max().item() < 2 ** -8 + K / 16 * 4 * 2 ** -23
    assert wide[:, :8].abs().max().item() == 0
    assert torch.equal(gemm.gemm_nt(a, b), gemm.gemm_nt(a, b))


@pytest.mark.parametrize("counts,M,N", [([64, 0, 192, 0] * 40, 128, 520), ([0, 640, 64] * 13, 384, 1000),
                                        ([0, 0], 256, 38000), ([128] * 150, 128, 264), ([320, 64], 256, 38003),
                                        ([64, 0, 192, 0], 128, 136)])
def test_grouped_weight_gradients_on_pairs(counts, M, N):
    """Blocks of half a pair tile, ragged columns, empty first and last groups, nothing but empty groups, four and more
    rounds of tiles, and one shape of the one-CTA kernel. fp32 sums of exact products: 2^-24 per addition of the sum
    of the magnitudes."""
    ops, _ = _ops()
    torch.manual_seed(11)
    G, K = len(counts), max(sum(counts), 64)
    starts = [0]
    for c in counts:
        starts.append(starts[-1] + c)
    seg = torch.tensor(starts, device="cuda", dtype=torch.int32)
    a = torch.randn(K, M, device="cuda").to(torch.bfloat16)
    b = torch.randn(K, (N + 7) // 8 * 8, device="cuda").to(torch.bfloat16)[:, :N]
    wide = torch.randn(G * M, (N + 3) // 4 * 4 + 4, device="cuda")
    before, acc = wide.clone(), wide[:, :N]
    base = acc.double()
    ops.ext().gemm_grouped(a, b, acc, M, N, K, M, b.stride(0), acc.stride(0), True, True, 2, 1, seg, G, 0)
    ops.check_status()
    assert torch.equal(wide[:, N:], before[:, N:])
    for g, c in enumerate(counts):
        rows = slice(starts[g], starts[g + 1])
        x, y = a[rows].double(), b[rows].double()
        want = base[g * M:(g + 1) * M] + x.t() @ y
        mag = base[g * M:(g + 1) * M].abs() + x.abs().t() @ y.abs()
        assert ((acc[g * M:(g + 1) * M].double() - want).abs() <= mag * (c + 2) * 2.0 ** -24).all()
