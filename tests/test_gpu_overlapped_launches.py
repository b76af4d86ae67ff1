"""Kernels whose launch overlaps the end of the kernel before them: chains in which memory that one kernel reads is written by another shortly
before and again shortly after, on a side stream and in a captured graph."""
import pytest
import torch

from conftest import free_port, require_cuda

pytestmark = pytest.mark.gpu

HIDDEN, FFN, EXPERTS, TOP_K, STEPS = 1024, 640, 8, 4, 6


@pytest.fixture(scope="module")
def txr():
    require_cuda()
    import tilexr_b200

    return tilexr_b200


def _chain(txr, comm, weights, x, after):
    """Every operator of a feed-forward and of an MoE exchange that is launched this way; `after` is called behind each.  What it makes on the way is
    released at its end, so the next call writes to the same memory."""
    gemm, quant, ep = txr.gemm, txr.quant, txr.ep
    gate, (w13, s13), (w2, s2), experts, wide = weights

    def done(result):
        after()
        return result

    logits = done(quant.router_logits(x, gate))
    d = done(ep.dispatch(comm, x, gate_logits=logits, num_experts=EXPERTS, top_k=TOP_K, quant_mode=ep.QUANT_FP8_1X128))
    rows = done(quant.fp8_dequant_1x128(d.expand_x, d.dynamic_scales))
    hidden = done(quant.swiglu(done(gemm.grouped_matmul(rows, experts, d.expert_token_nums))))
    mixed = done(ep.combine(comm, done(gemm.matmul(hidden, wide)), d, expert_scales=d.topk_weights))
    q, s = done(quant.fp8_quant_1x128(mixed))
    q, s = done(quant.swiglu_fp8_quant_1x128(done(gemm.matmul_fp8_block(q, s, w13, s13))))
    y = done(gemm.matmul_fp8_block(q, s, w2, s2))
    m, e = done(quant.mxfp8_quant(y))
    return logits, rows.sum(dim=1, dtype=torch.float64), mixed, y, done(quant.mxfp8_dequant(m, e))


@pytest.mark.parametrize("tokens", [17, 64, 600])
def test_chain_of_overlapped_launches(txr, tokens):
    g = torch.Generator().manual_seed(tokens)

    def randn(*shape):
        return torch.randn(*shape, generator=g).mul_(shape[-1] ** -0.5).to(torch.bfloat16).cuda()

    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        weights = (torch.randn(EXPERTS, HIDDEN, generator=g).cuda(), txr.gemm.quantize_weight_128x128(randn(2 * FFN, HIDDEN)),
                   txr.gemm.quantize_weight_128x128(randn(HIDDEN, FFN)), randn(EXPERTS, 2 * FFN, HIDDEN), randn(HIDDEN, FFN))
        batches = [torch.randn(tokens, HIDDEN, generator=g).to(torch.bfloat16).cuda() for _ in range(2 * STEPS)]
        want = [_chain(txr, comm, weights, x, torch.cuda.synchronize) for x in batches]
        assert all(torch.isfinite(w[3].float()).all() and w[3].any() for w in want)

        def check(got, expected):
            torch.cuda.synchronize()
            assert comm.device_status() == 0
            for step, (a, b) in enumerate(zip(got, expected)):
                for i, (u, v) in enumerate(zip(a, b)):
                    assert torch.equal(u, v), (step, i)

        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.cuda._sleep(100_000_000)               # some 50 ms: the launches queue up behind it
            got = [_chain(txr, comm, weights, x, lambda: None) for x in batches]
        check(got, want)

        inputs = [x.clone() for x in batches[:STEPS]]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            outs = [_chain(txr, comm, weights, x, lambda: None) for x in inputs]
        for first in (0, STEPS):
            for static, x in zip(inputs, batches[first:first + STEPS]):
                static.copy_(x)
            for _ in range(3):
                graph.replay()
            check(outs, want[first:first + STEPS])
        del graph
    finally:
        comm.destroy()
