"""Expert-parallel dispatch / combine and the local hot ops against fp32 PyTorch references."""
import pytest
import torch

from conftest import require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def txr():
    require_cuda()
    import tilexr_b200

    return tilexr_b200


@pytest.mark.parametrize("score_func,renorm,bias", [(0, True, False), (1, True, False), (1, False, True)])
def test_routing_topk(txr, score_func, renorm, bias):
    from tilexr_b200.utils import oracle

    g = torch.Generator().manual_seed(0)
    logits = torch.randn(333, 256, generator=g)
    b = torch.randn(256, generator=g) * 0.1 if bias else None
    ids, w = txr.quant.routing_topk(logits.cuda(), 8, score_func, renorm, 2.5, None if b is None else b.cuda())
    rids, rw = oracle.routing_topk_ref(logits, 8, score_func, renorm, 2.5, b)
    assert torch.equal(ids.cpu(), rids)
    assert torch.allclose(w.cpu(), rw, rtol=1e-5, atol=1e-7)


def test_fp8_quant_1x128_matches_reference(txr):
    from tilexr_b200.utils import oracle

    g = torch.Generator().manual_seed(1)
    x = (torch.randn(257, 7168, generator=g) * 3).to(torch.bfloat16)
    x[5] = 0       # an all-zero row hits the amax floor
    q, s = txr.quant.fp8_quant_1x128(x.cuda())
    rq, rs = oracle.fp8_quant_1x128_ref(x)
    assert torch.equal(s.cpu(), rs)
    assert torch.equal(q.cpu().view(torch.uint8), rq.view(torch.uint8))
    back = txr.quant.fp8_dequant_1x128(q, s, torch.bfloat16)
    ref_back = oracle.fp8_dequant_1x128_ref(rq, rs).to(torch.bfloat16)
    assert torch.equal(back.cpu(), ref_back)
    rel = (back.cpu().float() - x.float()).abs().max() / x.float().abs().max()
    assert rel < 0.07


@pytest.mark.parametrize("e5m2", [False, True])
def test_mxfp8_matches_reference(txr, e5m2):
    from tilexr_b200.utils import oracle

    g = torch.Generator().manual_seed(2)
    x = (torch.randn(64, 1000, generator=g) * torch.logspace(-3, 3, 1000)).to(torch.float16)
    q, s = txr.quant.mxfp8_quant(x.cuda(), e5m2)
    rq, rs = oracle.mxfp8_quant_ref(x, e5m2)
    assert torch.equal(s.cpu(), rs)
    assert torch.equal(q.cpu().view(torch.uint8), rq.view(torch.uint8))
    back = txr.quant.mxfp8_dequant(q, s, torch.float16)
    assert torch.allclose(back.cpu().float(), oracle.mxfp8_dequant_ref(rq, rs).to(torch.float16).float(), rtol=0, atol=0)


@pytest.mark.parametrize("with_residual", [False, True])
def test_rmsnorm(txr, with_residual):
    from tilexr_b200.utils import oracle

    g = torch.Generator().manual_seed(3)
    x = torch.randn(37, 8192, generator=g).to(torch.bfloat16)
    gamma = (1 + 0.1 * torch.randn(8192, generator=g)).to(torch.bfloat16)
    res = torch.randn(37, 8192, generator=g).to(torch.bfloat16) if with_residual else None
    res_dev = res.cuda() if with_residual else None
    y = txr.quant.rmsnorm(x.cuda(), gamma.cuda(), 1e-6, res_dev)
    ry, rres = oracle.rmsnorm_ref(x, gamma, 1e-6, res)
    assert torch.allclose(y.cpu().float(), ry.float(), rtol=2e-2, atol=2e-2)
    assert (y.cpu().float() - ry.float()).abs().mean() < 2e-3
    if with_residual:
        assert torch.equal(res_dev.cpu(), rres)


def _ep_case(txr, ranks, bs, h, experts, top_k, quant, fused_routing, masks=False, zero_copy=False, dtype=torch.bfloat16,
             dedup=None, scales_at_dispatch=False):
    from tilexr_b200.ops import ep
    from tilexr_b200.utils import oracle

    world = txr.init_emulated_world(ranks, device=0, buffer_mb=128)
    g = torch.Generator().manual_seed(11)
    xs = [torch.randn(bs, h, generator=g).to(dtype) for _ in range(ranks)]
    logits = [torch.randn(bs, experts, generator=g) for _ in range(ranks)]
    routed = [oracle.routing_topk_ref(l, top_k, 1, True, 1.0) for l in logits]
    ids = [r[0] for r in routed]
    ws = [r[1] for r in routed]
    mask = None
    if masks:
        mask = [(torch.rand(bs, generator=g) > 0.3) for _ in range(ranks)]
    max_rows = bs * ranks * min(top_k, experts // ranks)
    outs = world.symm_empty((max_rows, h), torch.float8_e4m3fn if quant else dtype) if zero_copy else [None] * ranks
    for _ in range(2):
        def call(c, r):
            kw = dict(num_experts=experts, top_k=top_k, quant_mode=ep.QUANT_FP8_1X128 if quant else ep.QUANT_NONE,
                      score_func=1, renormalize=True, max_recv_rows=max_rows, expand_x_out=outs[r],
                      active_mask=None if mask is None else mask[r].cuda(), dedup=dedup)
            if scales_at_dispatch:
                kw["expert_scales"] = ws[r].cuda()
            if fused_routing:
                return ep.dispatch(c, xs[r].cuda(), gate_logits=logits[r].cuda(), **kw)
            return ep.dispatch(c, xs[r].cuda(), expert_ids=ids[r].cuda(), **kw)
        res = world.run(call)
        world.check()
    ref = oracle.ep_dispatch_ref(xs, ids, experts, mask)
    expert_outs = []
    for r in range(ranks):
        d = res[r]
        n = int(d.recv_total.item())
        assert n == len(ref[r]["rows"])
        assert torch.equal(d.assist[:n].cpu(), ref[r]["assist"])
        assert torch.equal(d.expert_token_nums.cpu(), ref[r]["token_nums"])
        assert torch.equal(d.send_counts.cpu(), ref[r]["send_counts"])
        if fused_routing or scales_at_dispatch:
            # the gate weight of every received row travelled with it
            a = ref[r]["assist"].long()
            want_w = torch.stack([ws[int(s)][int(t), int(k)] for s, t, k, _ in a.tolist()]) if n else torch.empty(0)
            assert torch.allclose(d.expand_scales[:n].cpu(), want_w, rtol=1e-5, atol=1e-7)
        if fused_routing:
            assert torch.equal(d.topk_ids.cpu(), ids[r])
            assert torch.allclose(d.topk_weights.cpu(), ws[r], rtol=1e-5, atol=1e-7)
        if quant:
            rq, rs = oracle.fp8_quant_1x128_ref(ref[r]["expand_x"]) if n else (None, None)
            if n:
                assert torch.equal(d.expand_x[:n].cpu().view(torch.uint8), rq.view(torch.uint8))
                assert torch.equal(d.dynamic_scales[:n].cpu(), rs)
            rows = txr.quant.fp8_dequant_1x128(d.expand_x, d.dynamic_scales, dtype)
        else:
            assert torch.equal(d.expand_x[:n].cpu(), ref[r]["expand_x"])
            rows = d.expand_x
        # stand-in expert: scale by (1 + local expert index / 8)
        e_local = (d.assist[:, 3] % (experts // ranks)).clamp(min=0).float().cuda()
        out = (rows.float() * (1 + e_local / 8).unsqueeze(1)).to(dtype)
        expert_outs.append(out)

    ys = world.run(lambda c, r: ep.combine(c, expert_outs[r], res[r], expert_scales=ws[r].cuda(),
                                           active_mask=None if mask is None else mask[r].cuda()))
    world.check()
    ref_outs = [expert_outs[r][: len(ref[r]["rows"])].cpu() for r in range(ranks)]
    yref = oracle.ep_combine_ref(ref, ref_outs, ids, ws, dtype)
    for r in range(ranks):
        got = ys[r].cpu().float()
        want = yref[r].float()
        if mask is not None:
            want = want * mask[r].unsqueeze(1).float()
        assert torch.allclose(got, want, rtol=2e-2, atol=2e-2), (got - want).abs().max()
        assert (got - want).abs().mean() < 1e-3
    world.destroy()


def test_ep_bf16_explicit_ids(txr):
    _ep_case(txr, ranks=4, bs=48, h=256, experts=16, top_k=2, quant=False, fused_routing=False)


def test_ep_fp8_fused_routing(txr):
    _ep_case(txr, ranks=4, bs=40, h=1024, experts=32, top_k=4, quant=True, fused_routing=True)


def test_ep_token_mask(txr):
    _ep_case(txr, ranks=2, bs=33, h=512, experts=8, top_k=2, quant=True, fused_routing=False, masks=True)


def test_ep_zero_copy_output(txr):
    _ep_case(txr, ranks=4, bs=64, h=512, experts=16, top_k=4, quant=True, fused_routing=True, zero_copy=True)


def test_ep_eight_ranks_fp16(txr):
    _ep_case(txr, ranks=8, bs=24, h=512, experts=64, top_k=8, quant=False, fused_routing=True, dtype=torch.float16)


def test_ep_dedup_explicit_ids_with_scales(txr):
    # top-8 over 2 ranks: nearly every token has several experts on the remote rank
    _ep_case(txr, ranks=2, bs=40, h=512, experts=16, top_k=8, quant=True, fused_routing=False, scales_at_dispatch=True,
             zero_copy=True)


def test_ep_dedup_staged_output_and_masks(txr):
    _ep_case(txr, ranks=4, bs=37, h=256, experts=32, top_k=6, quant=False, fused_routing=True, masks=True)


def test_ep_large_batch_overlapped_combine(txr):
    # enough routes for combine's bucketed send order with dedicated reducer blocks
    _ep_case(txr, ranks=2, bs=1536, h=512, experts=16, top_k=8, quant=True, fused_routing=True, zero_copy=True)


def test_ep_dedup_off_matches(txr):
    _ep_case(txr, ranks=4, bs=40, h=1024, experts=32, top_k=4, quant=True, fused_routing=True, dedup=False)


@pytest.mark.parametrize("e5m2", [False, True])
def test_ep_dispatch_fused_mxfp8(txr, e5m2):
    """quantMode 3 / 4: rows arrive as MXFP8 with one E8M0 exponent byte per 32 elements, bit-exact vs the reference."""
    from tilexr_b200.ops import ep
    from tilexr_b200.utils import oracle

    ranks, bs, h, experts, top_k = 4, 36, 1024, 16, 4
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    g = torch.Generator().manual_seed(21)
    xs = [(torch.randn(bs, h, generator=g) * (1 + 3 * torch.rand(bs, 1, generator=g))).to(torch.bfloat16) for _ in range(ranks)]
    xs[0][0, :40] = 0                                  # an all-zero block
    logits = [torch.randn(bs, experts, generator=g) for _ in range(ranks)]
    ids = [oracle.routing_topk_ref(l, top_k, 1, True, 1.0)[0] for l in logits]
    mode = ep.QUANT_MXFP8_E5M2 if e5m2 else ep.QUANT_MXFP8_E4M3
    res = world.run(lambda c, r: ep.dispatch(c, xs[r].cuda(), gate_logits=logits[r].cuda(), num_experts=experts, top_k=top_k,
                                             quant_mode=mode, score_func=1))
    world.check()
    ref = oracle.ep_dispatch_ref(xs, ids, experts, None)
    for r in range(ranks):
        d = res[r]
        n = int(d.recv_total.item())
        assert n == len(ref[r]["rows"]) and n > 0
        assert d.expand_x.dtype == (torch.float8_e5m2 if e5m2 else torch.float8_e4m3fn)
        assert d.dynamic_scales.dtype == torch.uint8 and tuple(d.dynamic_scales.shape[1:]) == (h // 32,)
        rq, rs = oracle.mxfp8_quant_ref(ref[r]["expand_x"], e5m2)
        assert torch.equal(d.expand_x[:n].cpu().view(torch.uint8), rq.view(torch.uint8))
        assert torch.equal(d.dynamic_scales[:n].cpu(), rs)
    world.destroy()


@pytest.mark.parametrize("dynamic,smooth", [(True, False), (True, True), (False, True)])
def test_ep_dispatch_int8_modes(txr, dynamic, smooth):
    """quantMode 1 (static) and 2 (per-row dynamic) int8, with per-expert smoothing scales."""
    from tilexr_b200.ops import ep
    from tilexr_b200.utils import oracle

    ranks, bs, h, experts, top_k = 2, 20, 512, 8, 3
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    g = torch.Generator().manual_seed(31)
    xs = [torch.randn(bs, h, generator=g).to(torch.bfloat16) for _ in range(ranks)]
    ids = [torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(bs)]).to(torch.int32) for _ in range(ranks)]
    ws = [torch.rand(bs, top_k, generator=g) for _ in range(ranks)]
    smooth_scales = (0.5 + torch.rand(experts, h, generator=g)) * (1.0 if dynamic else 20.0) if smooth else None
    mode = ep.QUANT_DYNAMIC_INT8 if dynamic else ep.QUANT_STATIC_INT8
    res = world.run(lambda c, r: ep.dispatch(c, xs[r].cuda(), expert_ids=ids[r].cuda(), expert_scales=ws[r].cuda(),
                                             num_experts=experts, top_k=top_k, quant_mode=mode,
                                             scales=None if smooth_scales is None else smooth_scales.cuda()))
    world.check()
    ref = oracle.ep_dispatch_ref(xs, ids, experts, None)
    for r in range(ranks):
        d = res[r]
        n = int(d.recv_total.item())
        assert n == len(ref[r]["rows"]) and d.expand_x.dtype == torch.int8
        v = ref[r]["expand_x"].float()
        if smooth_scales is not None:
            v = v * smooth_scales[ref[r]["assist"][:, 3].long()]
        if dynamic:
            amax = v.abs().amax(dim=1)
            inv = torch.where(amax > 0, torch.full_like(amax, 127.0) / amax, torch.ones_like(amax))   # tensor / tensor: IEEE division
            want = torch.round(v * inv.unsqueeze(1)).clamp(-128, 127).to(torch.int8)
            assert torch.equal(d.dynamic_scales[:n].cpu(), torch.where(amax > 0, amax / 127.0, torch.ones_like(amax)))
        else:
            want = torch.round(v).clamp(-128, 127).to(torch.int8)
            assert d.dynamic_scales is None
        assert torch.equal(d.expand_x[:n].cpu(), want)
        assert d.dedup == (smooth_scales is None)
    world.destroy()


def test_ep_shared_expert_ranks(txr):
    """Two leading ranks hold the shared expert (one copy each), two hold the routed experts: every token also
    goes to its copy of the shared expert (slot top_k, weight 1), cf. the reference's destination rule."""
    from tilexr_b200.ops import ep
    from tilexr_b200.utils import oracle

    ranks, shared_ranks, shared_experts, bs, h, experts, top_k = 4, 2, 1, 24, 256, 8, 2
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    g = torch.Generator().manual_seed(41)
    xs = [torch.randn(bs, h, generator=g).to(torch.bfloat16) for _ in range(ranks)]
    logits = [torch.randn(bs, experts, generator=g) for _ in range(ranks)]
    routed = [oracle.routing_topk_ref(l, top_k, 1, True, 1.0) for l in logits]
    ids, ws = [r[0] for r in routed], [r[1] for r in routed]
    res = world.run(lambda c, r: ep.dispatch(c, xs[r].cuda(), gate_logits=logits[r].cuda(), num_experts=experts, top_k=top_k,
                                             score_func=1, shared_expert_num=shared_experts, shared_expert_rank_num=shared_ranks))
    world.check()
    per_shared = shared_ranks // shared_experts
    moe_per_rank = experts // (ranks - shared_ranks)
    # expected rows per destination: local expert major, then source rank, then token order
    for dst in range(ranks):
        want = []      # (src, token, slot, expert id)
        local = [None] if dst < shared_ranks else list(range((dst - shared_ranks) * moe_per_rank, (dst - shared_ranks + 1) * moe_per_rank))
        for e in local:
            for src in range(ranks):
                for t in range(bs):
                    if e is None:
                        if src % per_shared + 0 * per_shared == dst:
                            want.append((src, t, top_k, 0))
                    else:
                        for k in range(top_k):
                            if int(ids[src][t, k]) == e:
                                want.append((src, t, k, e))
        d = res[dst]
        n = int(d.recv_total.item())
        assert n == len(want), (dst, n, len(want))
        assert d.assist[:n].cpu().tolist() == [list(w) for w in want]
        rows = torch.stack([xs[s][t] for s, t, _, _ in want]) if want else torch.empty(0, h, dtype=torch.bfloat16)
        assert torch.equal(d.expand_x[:n].cpu(), rows)
        assert d.expert_token_nums.numel() == (1 if dst < shared_ranks else moe_per_rank)
    # identity experts: y = sum_k w_k x + x (the shared expert's copy)
    ys = world.run(lambda c, r: ep.combine(c, res[r].expand_x, res[r], expert_scales=ws[r].cuda()))
    world.check()
    for r in range(ranks):
        want = (xs[r].float() * (ws[r].sum(dim=1, keepdim=True) + 1.0))
        assert torch.allclose(ys[r].cpu().float(), want, rtol=2e-2, atol=2e-2)
    world.destroy()


def test_ep_overflow_is_reported_not_written(txr):
    from tilexr_b200.ops import ep

    world = txr.init_emulated_world(2, device=0, buffer_mb=64)
    x = [torch.randn(16, 256).to(torch.bfloat16).cuda() for _ in range(2)]
    ids = [torch.zeros(16, 2, dtype=torch.int32).cuda() for _ in range(2)]     # every route to expert 0
    ids[0][:, 1] = 1
    ids[1][:, 1] = 1
    world.run(lambda c, r: ep.dispatch(c, x[r], expert_ids=ids[r], num_experts=4, top_k=2, max_recv_rows=8))
    torch.cuda.synchronize()
    assert all(c.device_status() == 4 for c in world.comms)      # TILEXR_DEV_BAD_ARGUMENT on every rank
    for c in world.comms:
        c.reset_status()
    world.destroy()


def test_reset_status_keeps_flags_meaningful(txr):
    """After a failed launch and reset_status the next launches must still WAIT for their flags: the reset keeps
    the launch epoch, so flags left by earlier launches stay older than anything a new launch waits for."""
    from tilexr_b200.ops import ep
    from tilexr_b200.utils import oracle

    ranks = 4
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    g = torch.Generator().manual_seed(5)
    # a few launches first, so that flags and done epochs of earlier launches exist
    for i in range(5):
        xs = [torch.randn(3000, generator=g).cuda() for _ in range(ranks)]
        outs = world.run(lambda c, r: txr.all_reduce(c, xs[r]))
        world.check()
        assert torch.allclose(outs[0], sum(xs), rtol=1e-5, atol=1e-5)
    epoch_before = [c.dfx()[0] for c in world.comms]
    x = [torch.randn(16, 256, generator=g).to(torch.bfloat16).cuda() for _ in range(ranks)]
    ids = [torch.zeros(16, 2, dtype=torch.int32).cuda() for _ in range(ranks)]
    for r in range(ranks):
        ids[r][:, 1] = 1
    world.run(lambda c, r: ep.dispatch(c, x[r], expert_ids=ids[r], num_experts=8, top_k=2, max_recv_rows=8))
    torch.cuda.synchronize()
    assert all(c.device_status() == 4 for c in world.comms)
    for c in world.comms:
        c.reset_status()
    assert all(c.device_status() == 0 for c in world.comms)
    for i in range(3):
        xs = [torch.randn(5000, generator=g).cuda() for _ in range(ranks)]
        outs = world.run(lambda c, r: txr.all_reduce(c, xs[r]))
        gathered = world.run(lambda c, r: txr.all_gather(c, xs[r]))
        world.check()
        for r in range(ranks):
            assert torch.allclose(outs[r], sum(xs), rtol=1e-5, atol=1e-5)
            assert torch.equal(gathered[r], torch.stack(xs))
    assert all(c.dfx()[0] > e for c, e in zip(world.comms, epoch_before))      # the epoch went on, it did not restart
    xs = [torch.randn(24, 256, generator=g).to(torch.bfloat16) for _ in range(ranks)]
    ids = [torch.randint(0, 8, (24, 2), generator=g, dtype=torch.int32) for _ in range(ranks)]
    for t in ids:
        t[:, 1] = (t[:, 0] + 1 + t[:, 1] % 7) % 8                                # two different experts per token
    res = world.run(lambda c, r: ep.dispatch(c, xs[r].cuda(), expert_ids=ids[r].cuda(), num_experts=8, top_k=2))
    world.check()
    ref = oracle.ep_dispatch_ref(xs, ids, 8, None)
    for r in range(ranks):
        n = int(res[r].recv_total.item())
        assert n == len(ref[r]["rows"])
        assert torch.equal(res[r].assist[:n].cpu(), ref[r]["assist"])
        assert torch.equal(res[r].expand_x[:n].cpu(), ref[r]["expand_x"])
    world.destroy()


@pytest.mark.parametrize("fp8", [False, True])
def test_moe_layer_matches_a_dense_reference(txr, fp8):
    """The MoE block (routing, dispatch, expert FFN on the tcgen05 GEMM, combine) against plain PyTorch in fp32."""
    from conftest import free_port
    from tilexr_b200.models import ExpertParallelMoE, MoEConfig
    from tilexr_b200.utils import oracle

    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    cfg = MoEConfig(hidden=512, ffn=256, num_experts=8, top_k=2, fp8_dispatch=fp8)
    layer = ExpertParallelMoE(comm, cfg, seed=3)
    g = torch.Generator().manual_seed(9)
    x = torch.randn(96, cfg.hidden, generator=g).to(torch.bfloat16)
    y = layer(x.cuda())
    torch.cuda.synchronize()
    assert comm.device_status() == 0
    logits = x.float() @ layer.gate.detach().cpu().t()
    ids, ws = oracle.routing_topk_ref(logits, cfg.top_k, cfg.score_func, cfg.renormalize, cfg.routed_scale)
    xin = x.float()
    if fp8:
        q, s = oracle.fp8_quant_1x128_ref(x)
        xin = oracle.fp8_dequant_1x128_ref(q, s).to(torch.bfloat16).float()
    w13, w2 = layer.w13.detach().cpu().float(), layer.w2.detach().cpu().float()
    want = torch.zeros(96, cfg.hidden)
    for t in range(96):
        for k in range(cfg.top_k):
            e = int(ids[t, k])
            gu = xin[t] @ w13[e].t()                                  # gate and up rows interleaved; the activation runs in fp32
            hmid = (torch.nn.functional.silu(gu[0::2]) * gu[1::2]).to(torch.bfloat16).float()
            want[t] += float(ws[t, k]) * (hmid @ w2[e].t()).to(torch.bfloat16).float()
    got = y.cpu().float()
    assert torch.allclose(got, want, rtol=3e-2, atol=3e-3), (got - want).abs().max()
    comm.destroy()


@pytest.mark.parametrize("dedup", [False, True])
def test_ep_with_tensor_parallel_groups(txr, dedup):
    """tpWorldSize 2 on four ranks: two expert groups of two ranks.  Every route reaches both ranks of its group, sorted
    by local expert; the lane counts come back; combine adds the two partial outputs of every row."""
    from tilexr_b200.ops import ep
    from tilexr_b200.utils import oracle

    ranks, T, bs, h, experts, top_k = 4, 2, 24, 512, 8, 2
    groups, per = ranks // T, experts // (ranks // T)
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    g = torch.Generator().manual_seed(5)
    xs = [torch.randn(bs, h, generator=g).to(torch.bfloat16) for _ in range(ranks)]
    routed = [oracle.routing_topk_ref(torch.randn(bs, experts, generator=g), top_k, 1, True, 1.0) for _ in range(ranks)]
    ids, ws = [r[0] for r in routed], [r[1] for r in routed]
    ids[1][3, 1] = -1                                     # an inactive route
    res = world.run(lambda c, r: ep.dispatch(c, xs[r].cuda(), expert_ids=ids[r].cuda(), expert_scales=ws[r].cuda(),
                                             num_experts=experts, top_k=top_k, tp_world_size=T, dedup=dedup))
    world.check()
    # the same dispatch stated on lane experts: route (t, k) -> slots k * T + l on expert ((group * T + l) * per + local)
    wide = []
    for r in range(ranks):
        e = ids[r].long()
        lane = torch.arange(T).view(1, 1, T)
        v = ((e // per).unsqueeze(-1) * T + lane) * per + (e % per).unsqueeze(-1)
        v = torch.where(e.unsqueeze(-1) >= 0, v, torch.full_like(v, -1))
        wide.append(v.reshape(bs, top_k * T).to(torch.int32))
    ref = oracle.ep_dispatch_ref(xs, wide, experts * T)
    for r in range(ranks):
        d = res[r]
        n = int(d.recv_total.item())
        assert n == len(ref[r]["rows"]) and n > 0
        assert torch.equal(d.assist[:n].cpu(), ref[r]["assist"])
        assert torch.equal(d.expand_x[:n].cpu(), ref[r]["expand_x"])
        assert torch.equal(d.expert_token_nums.cpu(), ref[r]["token_nums"]) and d.expert_token_nums.numel() == per
        assert torch.equal(d.send_counts.cpu(), ref[r]["send_counts"])
        by_lane = [sum(1 for (s, _, _, _) in ref[r]["rows"] if s % T == l) for l in range(T)]
        assert d.tp_recv_counts.cpu().tolist() == by_lane
        # both ranks of a group hold the same rows
        mate = res[r ^ 1]
        assert torch.equal(mate.expand_x[:n].cpu(), d.expand_x[:n].cpu())
    # each rank returns its "partial output": the row scaled by a factor of its own
    factor = [1.0 + r / 8 for r in range(ranks)]
    outs = [(res[r].expand_x.float() * factor[r]).to(torch.bfloat16) for r in range(ranks)]
    ys = world.run(lambda c, r: ep.combine(c, outs[r], res[r], expert_scales=ws[r].cuda()))
    world.check()
    for r in range(ranks):
        want = torch.zeros(bs, h)
        for t in range(bs):
            for k in range(top_k):
                e = int(ids[r][t, k])
                if e < 0:
                    continue
                for l in range(T):
                    owner = (e // per) * T + l
                    want[t] += float(ws[r][t, k]) * (xs[r][t].float() * factor[owner]).to(torch.bfloat16).float()
        got = ys[r].cpu().float()
        assert torch.allclose(got, want, rtol=2e-2, atol=2e-2), (got - want).abs().max()
    world.destroy()


@pytest.mark.parametrize("quant_mode", ["none", "fp8", "mxfp8", "int8"])
@pytest.mark.parametrize("tokens,experts,top_k", [(1, 8, 2), (17, 40, 8), (300, 256, 4), (1009, 5, 3)])
def test_dispatch_of_a_single_rank_stores_rows_at_their_place(txr, tokens, experts, top_k, quant_mode):
    """One rank: rows, scales and tuples go to the outputs without the window.  Expert ids with inactive routes, an active
    mask, more capacity than rows; blocks without tokens at the smallest batch."""
    from conftest import free_port

    ep, quant = txr.ep, txr.quant
    h = 512
    g = torch.Generator().manual_seed(tokens)
    x = (torch.randn(tokens, h, generator=g) * 2).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32)
    ids[0, top_k - 1] = -1
    mask = torch.rand(tokens, generator=g) > 0.2
    mask[0] = True
    weights = torch.rand(tokens, top_k, generator=g)
    mode = {"none": ep.QUANT_NONE, "fp8": ep.QUANT_FP8_1X128, "mxfp8": ep.QUANT_MXFP8_E4M3, "int8": ep.QUANT_DYNAMIC_INT8}[quant_mode]
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        for _ in range(2):        # the second launch finds what the first one left in the control block
            d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids.cuda(), expert_scales=weights.cuda(), active_mask=mask.cuda(),
                            quant_mode=mode, max_recv_rows=tokens * top_k + 3)
            torch.cuda.synchronize()
            assert comm.device_status() == 0
        active = (ids >= 0) & mask[:, None]
        flat = torch.where(active, ids, torch.full_like(ids, experts)).reshape(-1).long()
        order = torch.sort(flat, stable=True).indices[:int(active.sum())]
        token, slot, n = order // top_k, order % top_k, order.numel()
        assert int(d.recv_total) == n and d.tp_recv_counts.tolist() == [0]
        assert torch.equal(d.assist[:n].cpu(), torch.stack((torch.zeros_like(token), token, slot, flat[order]), 1).int())
        assert torch.equal(d.expert_token_nums.cpu(), torch.bincount(flat[order], minlength=experts)[:experts])
        assert torch.equal(d.expand_scales[:n].cpu(), weights.reshape(-1)[order])
        rows = torch.full((tokens * top_k,), -1, dtype=torch.int32)
        rows[order] = torch.arange(n, dtype=torch.int32)
        assert torch.equal(d.route_rows.cpu().reshape(-1), rows)
        sent = x[token.cuda()]
        if quant_mode == "none":
            assert torch.equal(d.expand_x[:n], sent)
        elif quant_mode == "int8":
            amax = sent.float().abs().amax(dim=1, keepdim=True)
            want = torch.round(sent.float() * (torch.full_like(amax, 127.0) / amax)).clamp(-128, 127).to(torch.int8)
            assert torch.equal(d.expand_x[:n], want) and torch.equal(d.dynamic_scales[:n], (amax / torch.full_like(amax, 127.0)).squeeze(1))
        else:
            want, scales = quant.fp8_quant_1x128(sent) if quant_mode == "fp8" else quant.mxfp8_quant(sent)
            assert torch.equal(d.expand_x[:n].view(torch.uint8), want.view(torch.uint8)) and torch.equal(d.dynamic_scales[:n], scales)
    finally:
        comm.destroy()


@pytest.mark.parametrize("ranks", [1, 2])
def test_dispatch_into_an_output_off_the_16_byte_grid(txr, ranks):
    """A caller's output that starts between 16-byte boundaries takes the way through the window."""
    ep = txr.ep
    h, tokens, experts, top_k = 64, 37, 8, 3
    g = torch.Generator().manual_seed(7)
    xs = [torch.randn(tokens, h, generator=g).to(torch.bfloat16).cuda() for _ in range(ranks)]
    ids = [torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32).cuda() for _ in range(ranks)]
    cap = tokens * ranks * top_k
    outs = [torch.zeros(cap * h + 8, dtype=torch.bfloat16, device="cuda")[3:3 + cap * h].view(cap, h) for _ in range(ranks)]
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    try:
        ds = world.run(lambda c, r: ep.dispatch(c, xs[r], expert_ids=ids[r], num_experts=experts, top_k=top_k, max_recv_rows=cap, expand_x_out=outs[r]))
        world.check()
        for r, d in enumerate(ds):
            assert d.expand_x.data_ptr() % 16 != 0
            n = int(d.recv_total)
            tuples = d.assist[:n].cpu().tolist()
            assert n > 0 and torch.equal(d.expand_x[:n], torch.stack([xs[s][t] for s, t, _, _ in tuples]))
    finally:
        world.destroy()


def test_dispatch_of_ranks_with_slightly_different_batches(txr):
    """The ranks of an emulated world share one launch: batches that differ a little must come out at one grid."""
    ep = txr.ep
    h, experts, top_k, sizes = 64, 8, 2, (290, 300)
    g = torch.Generator().manual_seed(11)
    xs = [torch.randn(n, h, generator=g).to(torch.bfloat16).cuda() for n in sizes]
    ids = [torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(n)]).to(torch.int32).cuda() for n in sizes]
    cap = sum(sizes) * top_k
    world = txr.init_emulated_world(2, device=0, buffer_mb=64)
    try:
        ds = world.run(lambda c, r: ep.dispatch(c, xs[r], expert_ids=ids[r], num_experts=experts, top_k=top_k, max_recv_rows=cap))
        world.check()
        assert sum(int(d.recv_total) for d in ds) == cap
        for d in ds:
            n = int(d.recv_total)
            tuples = d.assist[:n].cpu().tolist()
            assert torch.equal(d.expand_x[:n], torch.stack([xs[s][t] for s, t, _, _ in tuples]))
    finally:
        world.destroy()


def test_dispatch_in_a_window_with_room_for_few_blocks(txr, port):
    """Every block of a dispatch keeps a row of counts in the window: a window that the rows nearly fill still takes the batch."""
    ep = txr.ep
    h, experts, top_k, tokens = 256, 1024, 2, 1024
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=16, device=0)
    try:
        # what sixteen tokens to a block need fits (64 blocks of 1024 counts), what four to a block need does not
        rows = (comm.data_half_bytes - 64 * experts * 4 - 2048) // (h * 2 + 16 + 8)
        g = torch.Generator().manual_seed(12)
        x = torch.randn(tokens, h, generator=g).to(torch.bfloat16).cuda()
        ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32).cuda()
        d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids, max_recv_rows=rows)
        torch.cuda.synchronize()
        n = tokens * top_k
        assert comm.device_status() == 0 and int(d.recv_total) == n
        assert torch.equal(d.expand_x[:n], x[d.assist[:n, 1].long()])
        with pytest.raises(RuntimeError):
            ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids, max_recv_rows=rows + 128)
    finally:
        comm.destroy()


def test_lane_counts_are_zero_whatever_becomes_of_a_dispatch(txr, port):
    """One tensor-parallel lane: its count is zero after a launch that gave up on too many rows, too, and the C entry leaves the
    caller's buffer alone."""
    import ctypes

    ep = txr.ep
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=16, device=0)
    try:
        x = torch.randn(16, 256).to(torch.bfloat16).cuda()
        ids = torch.zeros(16, 2, dtype=torch.int32).cuda()
        ids[:, 1] = 1
        for cap, status in ((64, 0), (8, 4)):            # 4: TILEXR_DEV_BAD_ARGUMENT, 32 rows do not fit 8
            used = [torch.full((1,), 7, dtype=torch.int32, device="cuda") for _ in range(64)]
            del used                                     # the dispatch's small outputs come from this memory
            d = ep.dispatch(comm, x, expert_ids=ids, num_experts=4, top_k=2, max_recv_rows=cap)
            torch.cuda.synchronize()
            assert comm.device_status() == status and d.tp_recv_counts.tolist() == [0]
        comm.reset_status()

        pointer, i64 = ctypes.c_void_p, ctypes.c_int64

        class Params(ctypes.Structure):                  # TileXREpDispatchParams
            _fields_ = ([(n, pointer) for n in ("x", "expertIds", "gateLogits", "selectionBias", "xActiveMask")] +
                        [(n, i64) for n in ("activeMaskType", "bs", "h", "topK", "moeExpertNum", "quantMode", "scoreFunc", "renormalize")] +
                        [("routedScalingFactor", ctypes.c_float), ("expertTokenNumsType", i64), ("maxRecvRows", i64)] +
                        [(n, pointer) for n in ("topkIdsOut", "topkWeightsOut", "expandXOut", "dynamicScalesOut", "assistInfoForCombineOut",
                                                "expertTokenNumsOut", "sendCountsOut", "recvTotalOut")] +
                        [("dtype", ctypes.c_int), ("routeRowsOut", pointer), ("expertScales", pointer), ("expandScalesOut", pointer), ("dedup", i64),
                         ("assistExtOut", pointer), ("scales", pointer), ("sharedExpertNum", i64), ("sharedExpertRankNum", i64), ("tpWorldSize", i64),
                         ("tpRankId", i64), ("tpRecvCountsOut", pointer)])

        out = {n: torch.zeros(size, dtype=t, device="cuda") for n, size, t in (
            ("expandXOut", (64, 256), torch.bfloat16), ("assistInfoForCombineOut", (64, 4), torch.int32),
            ("expertTokenNumsOut", (4,), torch.int64), ("sendCountsOut", (4,), torch.int32), ("recvTotalOut", (1,), torch.int32))}
        mine = torch.full((1,), 7, dtype=torch.int32, device="cuda")
        p = Params(x=x.data_ptr(), expertIds=ids.data_ptr(), bs=16, h=256, topK=2, moeExpertNum=4, maxRecvRows=64, dtype=11, tpWorldSize=1,
                   tpRecvCountsOut=mine.data_ptr(), **{n: t.data_ptr() for n, t in out.items()})
        from pathlib import Path
        lib = ctypes.CDLL(str(Path(txr.__file__).parent / "lib" / "libtilexr.so"))
        assert lib.TileXRMoeEpDispatchFused(ctypes.byref(p), pointer(comm.handle), pointer(torch.cuda.current_stream().cuda_stream)) == 0
        torch.cuda.synchronize()
        assert comm.device_status() == 0 and int(out["recvTotalOut"]) == 32 and out["expertTokenNumsOut"].sum() > 0 and int(mine) == 7
    finally:
        comm.destroy()


@pytest.mark.parametrize("score_func", [0, 1])
@pytest.mark.parametrize("experts,top_k", [(5, 5), (33, 8), (256, 8), (500, 6), (1000, 32)])
def test_routing_topk_of_equal_and_invalid_scores(txr, experts, top_k, score_func):
    """Equal scores go to the lower expert; an expert whose score is NaN or minus infinity is never picked, and slots without a candidate
    have weight zero and an id that no expert has."""
    g = torch.Generator().manual_seed(experts)
    logits = torch.randint(-2, 3, (64, experts), generator=g).float()          # five values: ties in every row
    bias = torch.zeros(experts)
    logits[1] = 0.5                                                            # all equal
    if score_func == 1:
        bias = torch.randint(0, 2, (experts,), generator=g) * 0.25 - 0.5       # sums below, at and above zero
        bias[::7] = float("-inf")
        logits[2, 1::2] = float("nan")
        logits[3, 1:] = float("nan")                                           # at most one valid expert
        logits[4] = float("nan")
        logits[5, 0], logits[5, 1] = float("inf"), float("-inf")
    ids, w = txr.quant.routing_topk(logits.cuda(), top_k, score_func, True, 2.0, bias.cuda() if score_func == 1 else None)
    ids, w = ids.cpu(), w.cpu()
    scores = torch.softmax(logits, -1) if score_func == 0 else torch.sigmoid(logits)
    sel = scores + bias
    for t in range(64):
        valid = [e for e in range(experts) if sel[t, e] > float("-inf")]
        want = sorted(valid, key=lambda e: (-float(sel[t, e]), e))[:top_k]
        assert ids[t, :len(want)].tolist() == want, t
        assert all(i == 0x7fffffff for i in ids[t, len(want):].tolist())
        if want:
            picked = scores[t, want]
            assert torch.allclose(w[t, :len(want)], picked / picked.sum() * 2.0, rtol=1e-5, atol=0)
            assert not w[t, len(want):].any()


def test_dispatch_of_tokens_with_few_valid_experts(txr, port):
    """Routing fused into the dispatch: a slot without a candidate is an inactive route."""
    ep = txr.ep
    g = torch.Generator().manual_seed(9)
    tokens, experts, top_k = 40, 16, 4
    logits = torch.randn(tokens, experts, generator=g)
    for t in range(tokens):
        logits[t, torch.randperm(experts, generator=g)[:experts - t % 6]] = float("nan")      # t % 6 valid experts
    x = torch.randn(tokens, 64, generator=g).to(torch.bfloat16).cuda()
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=16, device=0)
    try:
        d = ep.dispatch(comm, x, gate_logits=logits.cuda(), num_experts=experts, top_k=top_k, score_func=1)
        torch.cuda.synchronize()
        assert comm.device_status() == 0
        want = [(e, t) for t in range(tokens) for e in torch.argsort(logits[t].nan_to_num(-100.0), descending=True)[:min(top_k, t % 6)].tolist()]
        n = len(want)
        assert int(d.recv_total) == n and [(e, t) for _, t, _, e in d.assist[:n].tolist()] == sorted(want)
        assert torch.equal(d.expand_x[:n], x[[t for _, t in sorted(want)]])
        assert ((d.route_rows >= 0).sum(dim=1).cpu() == torch.tensor([min(top_k, t % 6) for t in range(tokens)])).all()
    finally:
        comm.destroy()


@pytest.mark.parametrize("blocks,tokens,experts,top_k", [(8, 600, 40, 8), (1, 37, 8, 8), (3, 1, 5, 2), (37, 1200, 1024, 8), (296, 4099, 257, 2)])
def test_dispatch_of_a_single_rank_over_block_counts(txr, monkeypatch, blocks, tokens, experts, top_k):
    """The counts of a block take one byte, or two where it has more than 255 routes; fewer blocks than a vector of counts, and more."""
    from conftest import free_port

    ep = txr.ep
    monkeypatch.setenv("TILEXR_EP_BLOCKS", str(blocks))
    g = torch.Generator().manual_seed(tokens)
    x = torch.randn(tokens, 64, generator=g).to(torch.bfloat16).cuda()
    ids = torch.randint(-1, experts, (tokens, top_k), generator=g).to(torch.int32)
    ids[: tokens // 3] = 1                                  # one expert with far more routes than the others, several per token
    weights = torch.rand(tokens, top_k, generator=g)
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        for _ in range(2):
            d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids.cuda(), expert_scales=weights.cuda(), max_recv_rows=tokens * top_k)
        torch.cuda.synchronize()
        assert comm.device_status() == 0
        flat = torch.where(ids >= 0, ids, torch.full_like(ids, experts)).reshape(-1).long()
        order = torch.sort(flat, stable=True).indices[:int((ids >= 0).sum())]
        n, counts = order.numel(), torch.bincount(flat[order], minlength=experts)
        assert int(d.recv_total) == n and torch.equal(d.expert_token_nums.cpu(), counts)
        assert torch.equal(d.send_counts.cpu().long(), counts.cumsum(0))
        assert torch.equal(d.expand_x[:n], x[(order // top_k).cuda()])
        assert torch.equal(d.assist[:n, 1:].cpu(), torch.stack((order // top_k, order % top_k, flat[order]), 1).int())
        assert torch.equal(d.assist_ext[:n, 1].cpu().view(torch.float32), weights.reshape(-1)[order]) and not d.assist_ext[:n, 0].any()
    finally:
        comm.destroy()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,hidden,experts,top_k", [(1, 8, 3, 1), (5, 264, 7, 3), (130, 1032, 40, 8), (33, 512, 40, 11), (300, 7168, 64, 17)])
def test_combine_on_one_rank(txr, tokens, hidden, experts, top_k, dtype):
    """Inactive routes, masks, shared expert outputs, more than eight routes, rows of any length; against 64 bits."""
    from conftest import free_port

    ep = txr.ep
    g = torch.Generator().manual_seed(tokens + hidden)
    x = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32)
    ids[torch.rand(tokens, top_k, generator=g) < 0.1] = -1
    weights = torch.rand(tokens, top_k, generator=g).cuda()
    shared = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    mask = (torch.rand(tokens, generator=g) > 0.2).cuda()
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=256, device=0)
    try:
        d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids.cuda(), max_recv_rows=tokens * top_k)
        out = torch.randn(d.expand_x.shape, generator=g).to(dtype).cuda()
        rows = d.route_rows.long()
        picked = torch.where((rows >= 0)[..., None], out.double()[rows.clamp_min(0)], torch.zeros((), dtype=torch.float64, device="cuda"))
        for scales, sx, m in ((weights, None, None), (None, shared, None), (weights, shared, mask)):
            y = ep.combine(comm, out, d, expert_scales=scales, shared_expert_x=sx, active_mask=m)
            torch.cuda.synchronize()
            assert comm.device_status() == 0
            terms = picked * (scales.double()[..., None] if scales is not None else 1.0)
            if m is not None:
                terms = terms * m[:, None, None]
            want = terms.sum(dim=1) + (sx.double() if sx is not None else 0.0)
            # the fp32 sum of top_k + 1 terms, rounded once to the 16-bit type
            size = terms.abs().sum(dim=1) + (sx.double().abs() if sx is not None else 0.0)
            bound = want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) + size * (top_k + 1) * 2.0 ** -23 + 2.0 ** -24
            assert ((y.double() - want).abs() <= bound).all()
    finally:
        comm.destroy()


def test_combine_of_a_route_that_the_dispatch_did_not_place(txr, port):
    """Ids that name a route without a row: reported, as in a world with peers, and the communicator goes on after a reset."""
    ep = txr.ep
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=16, device=0)
    try:
        x = torch.randn(9, 64).to(torch.bfloat16).cuda()
        ids = torch.arange(9, dtype=torch.int32).view(9, 1).cuda() % 4
        ids[3] = -1
        d = ep.dispatch(comm, x, num_experts=4, top_k=1, expert_ids=ids)
        y = ep.combine(comm, d.expand_x, d)
        torch.cuda.synchronize()
        assert comm.device_status() == 0 and torch.equal(y, torch.where((ids >= 0), x, torch.zeros_like(x)))
        run_status, launch_count, finished, failed = 3, 10, 0x0D0E, 0xDEAD         # words of the failure record, two values
        assert comm.dfx()[run_status] == finished
        launches = comm.dfx()[launch_count]
        d.topk_ids = ids.clone().fill_(1)
        ep.combine(comm, d.expand_x, d)
        torch.cuda.synchronize()
        assert comm.device_status() != 0 and comm.dfx()[run_status] == failed and comm.dfx()[launch_count] == launches + 1
        comm.reset_status()
        d.topk_ids = ids
        assert torch.equal(ep.combine(comm, d.expand_x, d), y) and comm.device_status() == 0
    finally:
        comm.destroy()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,hidden,experts", [(1, 512, 8), (33, 1536, 40), (700, 7168, 256)])
def test_dispatch_through_fp8_and_back(txr, port, tokens, hidden, experts, dtype):
    """One pass gives what quantised rows and their dequantisation give, bit for bit."""
    ep = txr.ep
    g = torch.Generator().manual_seed(tokens)
    x = (torch.randn(tokens, hidden, generator=g) * torch.logspace(-4, 2, hidden)).to(dtype).cuda()
    x[0, :128] = 0
    logits = torch.randn(tokens, experts, generator=g).cuda()
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=128, device=0)
    try:
        args = dict(gate_logits=logits, num_experts=experts, top_k=4, quant_mode=ep.QUANT_FP8_1X128, max_recv_rows=tokens * 4)
        d = ep.dispatch(comm, x, **args)
        r = ep.dispatch(comm, x, round_trip=True, **args)
        torch.cuda.synchronize()
        assert comm.device_status() == 0 and r.dynamic_scales is None and r.expand_x.dtype == dtype
        assert torch.equal(r.expand_x.view(torch.int16), txr.quant.fp8_dequant_1x128(d.expand_x, d.dynamic_scales, dtype).view(torch.int16))
        for name in ("assist", "expert_token_nums", "send_counts", "recv_total", "topk_ids", "topk_weights", "route_rows", "expand_scales"):
            assert torch.equal(getattr(d, name), getattr(r, name)), name
        with pytest.raises(RuntimeError):
            ep.dispatch(comm, x, round_trip=True, **dict(args, quant_mode=ep.QUANT_NONE))
    finally:
        comm.destroy()


def test_dispatches_of_a_single_rank_in_turn(txr):
    """The barrier's count runs on from launch to launch: large and small grids, and clusters, which do not use it, on one communicator."""
    from conftest import free_port

    ep, experts, top_k, g = txr.ep, 24, 4, torch.Generator().manual_seed(9)
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        for tokens in (3000, 65, 64, 300, 1, 3000, 129, 1009, 65, 592, 593, 1036, 1037, 1184, 1185):
            x = torch.randn(tokens, 64, generator=g).to(torch.bfloat16).cuda()
            ids = torch.randint(0, experts, (tokens, top_k), generator=g).to(torch.int32)
            d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids.cuda(), expert_scales=torch.ones(tokens, top_k).cuda(),
                            max_recv_rows=tokens * top_k)
            flat = ids.reshape(-1).long()
            order = torch.sort(flat, stable=True).indices
            assert torch.equal(d.expert_token_nums.cpu(), torch.bincount(flat, minlength=experts))
            assert torch.equal(d.expand_x[:tokens * top_k], x[(order // top_k).cuda()])
        assert comm.device_status() == 0
    finally:
        comm.destroy()


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("aligned_first", [True, False])
def test_dispatches_of_a_single_rank_on_and_off_the_16_byte_grid_in_turn(txr, fp8, aligned_first):
    """Outputs on and off the 16-byte grid take different kernels: on one communicator, in grids that grow and shrink, with a combine in
    between and without, neither leaves anything behind that the other reads."""
    from conftest import free_port

    ep, h, experts, top_k, g = txr.ep, 512, 24, 4, torch.Generator().manual_seed(21)
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        aligned = aligned_first
        for step, tokens in enumerate((65, 1009, 300, 3000, 65, 65, 3000, 1009, 1009, 300, 64, 3000, 16, 300)):
            n = tokens * top_k
            x = torch.randn(tokens, h, generator=g).to(torch.bfloat16).cuda()
            ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32)
            row_type = torch.float8_e4m3fn if fp8 else torch.bfloat16
            out = torch.zeros(n * h + 16, dtype=row_type, device="cuda")[0 if aligned else 1:][:n * h].view(n, h)
            assert (out.data_ptr() % 16 == 0) == aligned
            d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids.cuda(), expert_scales=torch.ones(tokens, top_k).cuda(),
                            quant_mode=ep.QUANT_FP8_1X128 if fp8 else ep.QUANT_NONE, max_recv_rows=n, expand_x_out=out)
            torch.cuda.synchronize()
            assert comm.device_status() == 0
            flat = ids.reshape(-1).long()
            order = torch.sort(flat, stable=True).indices
            counts = torch.bincount(flat, minlength=experts)
            assert int(d.recv_total) == n and torch.equal(d.expert_token_nums.cpu(), counts) and torch.equal(d.send_counts.cpu().long(), counts.cumsum(0))
            assert torch.equal(d.route_rows.cpu().reshape(-1)[order].long(), torch.arange(n))
            src = (order // top_k).cuda()
            want = x[src]
            if fp8:
                want, scales = txr.quant.fp8_quant_1x128(want)
                assert torch.equal(d.dynamic_scales, scales)
            assert torch.equal(out.view(torch.uint8) if fp8 else out, want.view(torch.uint8) if fp8 else want)
            if step % 3 == 1:
                y = ep.combine(comm, x[src], d)
                torch.cuda.synchronize()
                # top_k equal rows with weight one: four times the value, exact in bf16
                assert comm.device_status() == 0 and torch.equal(y, x * top_k)
            aligned = not aligned
    finally:
        comm.destroy()


@pytest.mark.parametrize("registered", [False, True])
@pytest.mark.parametrize("mode", ["none", "fp8", "mxfp8", "int8"])
@pytest.mark.parametrize("ranks,dedup", [(1, False), (2, False), (3, True)])
def test_dispatch_into_any_output_off_the_16_byte_grid(txr, ranks, dedup, mode, registered):
    """Every transport, tokens with several experts on one rank, ordinary and registered memory: as into an output on the grid.  Rows of an odd number of
    16-byte pieces where the transport allows it."""
    ep = txr.ep
    modes = {"none": ep.QUANT_NONE, "fp8": ep.QUANT_FP8_1X128, "mxfp8": ep.QUANT_MXFP8_E4M3, "int8": ep.QUANT_DYNAMIC_INT8}
    row_type = {"none": torch.bfloat16, "fp8": torch.float8_e4m3fn, "mxfp8": torch.float8_e4m3fn, "int8": torch.int8}[mode]
    h, tokens, experts, top_k = {"none": 1032, "fp8": 512, "mxfp8": 512, "int8": 1040}[mode], 75, 6, 4
    g = torch.Generator().manual_seed(ranks)
    xs = [torch.randn(tokens, h, generator=g).to(torch.bfloat16).cuda() for _ in range(ranks)]
    ids = [torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32).cuda() for _ in range(ranks)]
    weights = torch.rand(tokens, top_k, generator=g).cuda()
    cap = tokens * ranks * top_k
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    try:
        if registered:
            memory = world.symm_empty((cap * h + 16,), row_type)
        else:
            memory = [torch.zeros(cap * h + 16, dtype=row_type, device="cuda") for _ in range(ranks)]
        results = []
        for offset in (0, 1):
            outs = [m[offset:offset + cap * h].view(cap, h) for m in memory]
            results.append(world.run(lambda c, r: ep.dispatch(c, xs[r], expert_ids=ids[r], expert_scales=weights, num_experts=experts, top_k=top_k,
                                                              quant_mode=modes[mode], max_recv_rows=cap, expand_x_out=outs[r], dedup=dedup)))
            world.check()
            if offset == 0:
                rows = [d.expand_x[:int(d.recv_total)].clone() for d in results[0]]
                for m in memory:
                    m.view(torch.uint8).zero_()
        for d, e, want in zip(*results, rows):
            n = int(d.recv_total)
            assert e.expand_x.data_ptr() % 16 != 0 and int(e.recv_total) == n > 0
            assert torch.equal(e.expand_x[:n].view(torch.uint8) if mode != "none" else e.expand_x[:n], want.view(torch.uint8) if mode != "none" else want)
            assert torch.equal(e.assist[:n], d.assist[:n]) and torch.equal(e.route_rows, d.route_rows)
            if mode != "none":
                assert torch.equal(e.dynamic_scales[:n], d.dynamic_scales[:n])
    finally:
        world.destroy()


def test_tensors_off_the_16_byte_grid_that_the_kernels_read_in_16_byte_pieces(txr, port):
    """Refused on the host, before a launch; tokens that are only copied may start anywhere."""
    ep, h, tokens, experts, top_k = txr.ep, 512, 9, 8, 2
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=16, device=0)
    try:
        def off(rows):
            return torch.randn(rows * h + 8, generator=torch.Generator().manual_seed(rows)).to(torch.bfloat16).cuda()[1:1 + rows * h].view(rows, h)

        ids = (torch.arange(tokens * top_k, dtype=torch.int32).view(tokens, top_k) % experts).cuda()
        x = off(tokens)
        args = dict(num_experts=experts, top_k=top_k, expert_ids=ids)
        for mode in (ep.QUANT_FP8_1X128, ep.QUANT_MXFP8_E5M2, ep.QUANT_DYNAMIC_INT8):
            with pytest.raises(RuntimeError):
                ep.dispatch(comm, x, quant_mode=mode, **args)
        d = ep.dispatch(comm, x, **args)
        n = int(d.recv_total)
        assert n == tokens * top_k and torch.equal(d.expand_x[:n], x[d.assist[:n, 1].long()])
        rows = d.expand_x.shape[0]
        for kw in (dict(expert_out=off(rows)), dict(shared_expert_x=x)):
            with pytest.raises(RuntimeError):
                ep.combine(comm, kw.pop("expert_out", d.expand_x), d, **kw)
        assert torch.equal(ep.combine(comm, d.expand_x, d), x * top_k) and comm.device_status() == 0
    finally:
        comm.destroy()


@pytest.mark.parametrize("cap", [1, 20, None])
def test_blocks_of_a_single_rank_under_the_switch(txr, monkeypatch, tmp_path, cap):
    """TILEXR_EP_BLOCKS caps the blocks of a dispatch and of a combine, whichever kernel they take; the results are the same."""
    import json

    from conftest import free_port

    from tilexr_b200.utils.stage_profile import stage_profile

    ep, h, tokens, experts, top_k = txr.ep, 512, 400, 16, 2
    g = torch.Generator().manual_seed(3)
    x = torch.randn(tokens, h, generator=g).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(experts, generator=g)[:top_k] for _ in range(tokens)]).to(torch.int32).cuda()
    if cap is not None:
        monkeypatch.setenv("TILEXR_EP_BLOCKS", str(cap))
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{free_port()}", buffer_mb=64, device=0)
    try:
        with stage_profile(str(tmp_path)):
            d = ep.dispatch(comm, x, num_experts=experts, top_k=top_k, expert_ids=ids)
            y = ep.combine(comm, d.expand_x, d)
        assert comm.device_status() == 0 and torch.equal(y, x * top_k)
        blocks = [json.loads(p.read_text())["blocks"] for p in sorted(tmp_path.rglob("trace.json"))]
        assert len(blocks) == 2 and (min(blocks) > 20 if cap is None else max(blocks) <= cap), blocks
    finally:
        comm.destroy()
