"""The Megatron-Core style token dispatcher over the fused dispatch / combine kernels, against a dense PyTorch MoE."""
import pytest
import torch

from conftest import free_port, require_cuda

pytestmark = pytest.mark.gpu


def test_dispatcher_round_trip_matches_dense_moe():
    require_cuda()
    import tilexr_b200 as txr
    from tilexr_b200.integrations.megatron_dispatcher import TileXRTokenDispatcher

    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        s, b, h, E, K = 24, 2, 256, 8, 2
        g = torch.Generator().manual_seed(4)
        hidden = torch.randn(s, b, h, generator=g).to(torch.bfloat16).cuda()
        logits = torch.randn(s * b, E, generator=g)
        probs, idx = torch.softmax(logits, -1).topk(K, dim=-1)
        probs = (probs / probs.sum(-1, keepdim=True)).cuda()
        idx = idx.cuda()
        w = (torch.randn(E, h, h, generator=g) / h ** 0.5).to(torch.bfloat16).cuda()

        disp = TileXRTokenDispatcher(comm, E, K, h)
        for _ in range(2):
            rows, counts = disp.token_permutation(hidden, probs, idx)
            torch.cuda.synchronize()
            assert counts.tolist() == torch.bincount(idx.reshape(-1).cpu(), minlength=E).tolist()
            assert disp.ctx() is not None and int(disp.ctx().recv_total.item()) == s * b * K
            out_rows = torch.zeros_like(rows)
            first = 0
            for e, n in enumerate(counts.tolist()):          # what a grouped GEMM does with the sorted rows
                out_rows[first:first + n] = rows[first:first + n] @ w[e].t()
                first += n
            y, _ = disp.token_unpermutation(out_rows)
            torch.cuda.synchronize()
            assert comm.device_status() == 0
        x = hidden.reshape(-1, h).float()
        ref = torch.zeros_like(x)
        for k in range(K):
            per_tok = torch.stack([(x[t].to(torch.bfloat16) @ w[idx[t, k]].t()).float() for t in range(x.shape[0])])
            ref += probs[:, k:k + 1].float() * per_tok
        assert y.shape == hidden.shape
        assert torch.allclose(y.float().reshape(-1, h), ref, rtol=3e-2, atol=3e-2)
        with pytest.raises(RuntimeError):
            disp.token_unpermutation(out_rows)
    finally:
        comm.destroy()


def test_dispatcher_backward_matches_dense_moe():
    """Loss gradients with respect to the hidden states, the router probabilities and the expert outputs through the two
    autograd functions (dispatch and combine in swapped roles), against a dense MoE under PyTorch autograd."""
    require_cuda()
    import tilexr_b200 as txr
    from tilexr_b200.integrations.megatron_dispatcher import TileXRTokenDispatcher

    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        tokens, h, E, K = 64, 256, 8, 2
        g = torch.Generator().manual_seed(8)
        x = torch.randn(tokens, h, generator=g).to(torch.bfloat16).cuda().requires_grad_(True)
        logits = torch.randn(tokens, E, generator=g).cuda().requires_grad_(True)
        w = (torch.randn(E, h, h, generator=g) / h ** 0.5).to(torch.bfloat16).cuda()
        target = torch.randn(tokens, h, generator=g).cuda()

        probs, idx = torch.softmax(logits, -1).topk(K, dim=-1)
        disp = TileXRTokenDispatcher(comm, E, K, h)
        rows, counts = disp.token_permutation(x, probs, idx)
        pieces, first = [], 0
        for e, n in enumerate(counts.tolist()):
            pieces.append(rows[first:first + n] @ w[e].t())
            first += n
        out = torch.cat(pieces + [rows[first:] * 0])
        y, _ = disp.token_unpermutation(out)
        (y.float() * target).sum().backward()
        torch.cuda.synchronize()
        assert comm.device_status() == 0
        gx, gl = x.grad.float().clone(), logits.grad.clone()

        x.grad = logits.grad = None
        probs2, idx2 = torch.softmax(logits, -1).topk(K, dim=-1)
        dense = torch.zeros(tokens, h, device="cuda")
        for k in range(K):
            per_tok = torch.bmm(x.unsqueeze(1), w[idx2[:, k]].transpose(1, 2)).squeeze(1).float()
            dense = dense + probs2[:, k:k + 1] * per_tok
        (dense * target).sum().backward()
        assert torch.allclose(y.float(), dense, rtol=3e-2, atol=3e-2)
        assert torch.allclose(gx, x.grad.float(), rtol=5e-2, atol=5e-2), (gx - x.grad.float()).abs().max()
        assert torch.allclose(gl, logits.grad, rtol=5e-2, atol=2e-2), (gl - logits.grad).abs().max()
    finally:
        comm.destroy()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,hidden,top_k,capacity", [(1, 8, 1, 1), (5, 264, 3, 19), (130, 1032, 8, 1040)])
def test_combine_backward_rows_match_the_unfused_form(tokens, hidden, top_k, capacity, dtype):
    """Row gradients and gate-weight dot products of one pass against plain PyTorch, with rows nobody uses at the end."""
    import dataclasses

    from tilexr_b200.ops import ep

    gen = torch.Generator().manual_seed(tokens)
    n = tokens * top_k
    g = torch.randn(capacity, hidden, generator=gen).to(dtype).cuda()
    out = torch.randn(capacity, hidden, generator=gen).to(dtype).cuda()
    w = torch.rand(capacity, generator=gen).cuda()
    assist = torch.zeros(capacity, 4, dtype=torch.int32)
    assist[:, 2] = torch.arange(capacity) % top_k
    d = ep.DispatchResult(**{f.name: None for f in dataclasses.fields(ep.DispatchResult) if f.default is dataclasses.MISSING})
    d.expand_x, d.expand_scales, d.assist = g, w, assist.cuda()
    d.recv_total = torch.tensor([n], dtype=torch.int32, device="cuda")
    width = max(16, (2 * top_k + 7) // 8 * 8)
    grad, wide = ep.combine_backward_rows(d, out, top_k, width)
    want = (g[:n].float() * w[:n, None]).to(dtype)
    assert torch.equal(grad[:n], want) and not grad[n:].any()
    dots = (g[:n].double() * out[:n].double()).sum(dim=1)
    cols = (2 * assist[:n, 2].long().cuda())[:, None]
    got = wide[:n].double().gather(1, cols) + wide[:n].double().gather(1, cols + 1)
    # the pair keeps 16 bits of the fp32 sum, whose own error is below hidden * 2^-24 of the sum of magnitudes
    bound = dots.abs() * 2.0 ** -15 + (g[:n].double() * out[:n].double()).abs().sum(dim=1) * hidden * 2.0 ** -24
    assert ((got.squeeze(1) - dots).abs() <= bound).all()
    rest = wide[:n].clone().scatter_(1, cols, 0).scatter_(1, cols + 1, 0)
    assert not rest.any()
    only_grad, none = ep.combine_backward_rows(d, None, top_k, width)
    assert none is None and torch.equal(only_grad, grad)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,hidden,top_k,extra", [(1, 8, 1, 0), (5, 264, 3, 19), (130, 1032, 8, 1)])
def test_combine_backward_on_one_rank(tokens, hidden, top_k, extra, dtype):
    """Row gradients and gate-weight gradients from the output gradient where it is; inactive routes, rows that no route fills."""
    require_cuda()
    import tilexr_b200 as txr
    from tilexr_b200.ops import ep

    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        gen = torch.Generator().manual_seed(tokens)
        experts = 11
        x = torch.randn(tokens, hidden, generator=gen).to(dtype).cuda()
        ids = torch.stack([torch.randperm(experts, generator=gen)[:top_k] for _ in range(tokens)]).to(torch.int32)
        if tokens > 1:
            ids[torch.rand(tokens, top_k, generator=gen) < 0.2] = -1
        w = torch.rand(tokens, top_k, generator=gen).cuda()
        d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids.cuda(), max_recv_rows=tokens * top_k + extra)
        out = torch.randn(d.expand_x.shape, generator=gen).to(dtype).cuda()
        gy = torch.randn(tokens, hidden, generator=gen).to(dtype).cuda()
        grad, gw = ep.combine_backward_local(comm, d, gy, out, w, True)
        rows = d.route_rows.long()
        want, filled = torch.zeros_like(out), torch.zeros(out.shape[0], dtype=torch.bool, device="cuda")
        t, k = torch.nonzero(rows >= 0, as_tuple=True)
        want[rows[t, k]] = (w[t, k, None] * gy[t].float()).to(dtype)
        filled[rows[t, k]] = True
        assert torch.equal(grad, want) and not grad[~filled].any() and int(filled.sum()) == int(d.recv_total)
        terms = gy[t].double() * out[rows[t, k]].double()
        dots = torch.zeros(tokens, top_k, dtype=torch.float64, device="cuda")
        bound = torch.zeros_like(dots)
        dots[t, k], bound[t, k] = terms.sum(dim=1), terms.abs().sum(dim=1) * hidden * 2.0 ** -24
        assert ((gw.double() - dots).abs() <= bound).all()
        only, none = ep.combine_backward_local(comm, d, gy, out, w, False)
        assert none is None and torch.equal(only, grad)
        assert ep.combine_backward_local(comm, d, gy.float(), out, w, True) is None        # not the kernel's types
    finally:
        comm.destroy()
