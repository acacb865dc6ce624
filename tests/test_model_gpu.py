"""Whole-model check on the GPU: the hand-written kernel path (fused QKV/RoPE/attention, tcgen05
GEMMs, fused norms, fused cross entropy, flat AdamW) against the plain PyTorch restatement of the
same bf16 model (``PICO_REFERENCE_OPS=1``) — losses over a few optimizer steps must agree."""
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


def _losses(reference: bool, steps=4, kv_heads=4, graph=True):
    from picotron_b200 import ops, process_group_manager as pgm
    from picotron_b200.engine import TrainEngine
    os.environ["PICO_REFERENCE_OPS"] = "1" if reference else "0"
    pgm.process_group_manager = None
    cfg = {"distributed": dict(tp_size=1, dp_size=1),
           "model": dict(name="tiny-llama-test", init_std=0.02, dtype="bfloat16", num_hidden_layers=2,
                         hidden_size=512, intermediate_size=1024, num_attention_heads=8, num_key_value_heads=kv_heads),
           "training": dict(seed=0, learning_rate=1e-3, seq_length=256, micro_batch_size=2,
                            gradient_accumulation_steps=2, num_samples=512, cuda_graph=graph),
           "dataset": dict(name="synthetic")}
    eng = TrainEngine(cfg, device=torch.device("cuda", 0))
    out = [eng.train_step().item() for _ in range(steps)]
    if not reference:
        ops.check_status("model test")
        assert (eng._mb_graph not in (None, False)) == graph, "CUDA-graph replay was (not) used as asked"
    os.environ["PICO_REFERENCE_OPS"] = "0"
    return out


@pytest.mark.parametrize("kv_heads", [8, 4])
def test_kernel_path_matches_torch_path(kv_heads):
    a = _losses(False, kv_heads=kv_heads)
    b = _losses(True, kv_heads=kv_heads)
    for x, y in zip(a, b):
        assert abs(x - y) < 3e-2, (a, b)
    assert a[-1] < a[0]


def test_graph_replay_equals_eager_launches():
    """The micro-batch replayed from a CUDA graph runs the same kernels in the same order as eager
    launches: the losses of several optimizer steps are bit-identical."""
    a = _losses(False, steps=5, graph=True)
    b = _losses(False, steps=5, graph=False)
    assert a == b, (a, b)


@pytest.mark.parametrize("batch,seq", [(1, 33), (2, 200)])
def test_logits_without_gradients_are_the_same_bits(batch, seq):
    """The forward pass without autograd functions around the kernels runs the same kernels."""
    from picotron_b200 import ops
    from picotron_b200.engine import TrainEngine
    engine = TrainEngine({
        "distributed": dict(tp_size=1, dp_size=1),
        "model": dict(name="tiny-llama-test", init_std=0.02, dtype="bfloat16", hidden_size=512, intermediate_size=1024,
                      num_attention_heads=8, num_key_value_heads=4, num_hidden_layers=2),
        "training": dict(seed=0, seq_length=seq, micro_batch_size=batch, num_samples=64),
        "dataset": dict(name="synthetic")}, device=torch.device("cuda", 0))
    ids = torch.randint(0, 4096, (batch, seq), device="cuda")
    with_grad = engine.model(ids).detach()
    with torch.no_grad():
        without = engine.model(ids)
    ops.check_status("forward")
    assert not without.requires_grad and torch.equal(with_grad, without)


@pytest.mark.parametrize("captured", [False, True])
def test_launches_ahead_keep_the_order_of_forked_streams(captured):
    """Kernels set up beside their predecessor wait for everything their stream waits for: a long product, a fork to
    another stream that reads it, work on both, and a join, launched right behind the event waits as the captured
    tensor-parallel micro-batches do. Eager and replayed, with new inputs each time, against one stream with a
    synchronisation after every step (the same kernels, so the same bits)."""
    from picotron_b200 import ops
    from picotron_b200.ops import gemm, norm, swiglu
    torch.manual_seed(0)
    d = 2048

    def new():
        return torch.randn(d, d, device="cuda", dtype=torch.bfloat16)
    x, w1, w2, w3, scale = new(), new() * 0.02, new() * 0.02, new() * 0.02, torch.ones(d, device="cuda", dtype=torch.bfloat16)
    side = torch.cuda.Stream()
    big = torch.randn(6144, 6144, device="cuda", dtype=torch.bfloat16)

    def steps(fork, join, sync):
        with torch.no_grad():
            out = []
            for _ in range(3):
                gemm.gemm_nt(big, big)                   # holds the SMs while the next ones are set up
                a = gemm.gemm_nt(x, w1)
                sync()
                with fork():
                    b = norm.rmsnorm(a, scale, 1e-5)     # launched ahead behind an event wait only
                    c = gemm.gemm_nt(b, w2)
                e = swiglu.swiglu(a)
                f = gemm.gemm_nt(a, w3)
                sync()
                join()
                g = gemm.gemm_nt(c, f)                   # launched ahead behind a kernel of each stream
                h, r = norm.add_rmsnorm(g, c, scale, 1e-5)
                sync()
                out += [a, b, c, e, f, g, h, r]
            return out

    class on_side:
        def __enter__(self):
            side.wait_stream(torch.cuda.current_stream())
            self.ctx = torch.cuda.stream(side)
            self.ctx.__enter__()

        def __exit__(self, *args):
            self.ctx.__exit__(*args)

    def back():
        torch.cuda.current_stream().wait_stream(side)

    def forked():
        return steps(on_side, back, lambda: None)

    def alone():
        import contextlib
        return steps(contextlib.nullcontext, lambda: None, torch.cuda.synchronize)
    forked()
    torch.cuda.synchronize()
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            held = forked()
    for _ in range(4):
        x.copy_(new())
        want = [t.clone() for t in alone()]
        if captured:
            graph.replay()
            got = held
        else:
            got = forked()
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(want, got))
    ops.check_status("forked streams")
