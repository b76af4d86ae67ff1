"""The work this framework is timed on: single-GPU passes through its public entry points.

Six kinds of work, each over the sizes it meets in use:

* ``ep``       expert-parallel dispatch -> dequantisation -> combine, the exchange of an MoE block with the expert itself
               left out (the workload of ``bench.py``); decode batches to prefill, fp8 / MXFP8 / 16-bit transport, routing
               fused into the dispatch or given as expert ids;
* ``moe``      a whole ``ExpertParallelMoE`` block: router, dispatch, grouped SwiGLU experts, combine;
* ``linear``   one projection: ``gemm.matmul`` in bf16 / fp16, or quantisation and ``gemm.matmul_fp8_block``;
* ``mlp``      a ``SequenceParallelMLP`` block (all-gather GEMM, SwiGLU, GEMM reduce-scatter);
* ``train``    the token dispatcher's permutation and unpermutation, forward and backward;
* ``norm``     ``all_reduce_rmsnorm`` of a tensor-parallel layer on an emulated world.

A communicator, and a receive buffer in registered memory where one is used, are made once per process, as a program does.
"""
from __future__ import annotations

import functools
import math
import socket
import weakref

import torch

import tilexr_b200 as txr
from tilexr_b200.integrations.megatron_dispatcher import TileXRTokenDispatcher
from tilexr_b200.models import ExpertParallelMoE, MoEConfig
from tilexr_b200.models.tp_mlp import SequenceParallelMLP, TPMlpConfig
from tilexr_b200.ops import collectives, ep, gemm, quant

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
QUANT = {"none": ep.QUANT_NONE, "fp8": ep.QUANT_FP8_1X128, "mxfp8": ep.QUANT_MXFP8_E4M3}
MAX_ROWS, MAX_ROW_BYTES = 4096 * 8, 7168


def listed():
    return [
        # a decode step of a few requests: launches and the latency of the count exchange
        dict(name="ep_decode_16", kind="ep", tokens=16, hidden=7168, experts=256, top_k=8, quant="fp8", routing="logits", registered=False),
        # a ragged batch of a smaller model whose framework routes by itself and sends 16-bit rows
        dict(name="ep_ragged_1009", kind="ep", tokens=1009, hidden=4096, experts=64, top_k=6, quant="none", routing="ids", registered=False),
        # prefill, the headline workload of bench.py: 4096 x 7168 tokens, 256 experts, top-8, fp8 rows into registered memory
        dict(name="ep_prefill_4096", kind="ep", tokens=4096, hidden=7168, experts=256, top_k=8, quant="fp8", routing="logits", registered=True),
        # a decode step of an MoE block: every touched expert's weights are read for a handful of rows
        dict(name="moe_decode_32", kind="moe", tokens=32, hidden=2048, ffn=1024, experts=64, top_k=8),
        # prefill of an MoE block with one GPU's share of 256 experts
        dict(name="moe_prefill_4096", kind="moe", tokens=4096, hidden=7168, ffn=2048, experts=32, top_k=8),
        # one projection of a decode step: the weight is read once for 17 rows
        dict(name="linear_decode_17", kind="linear", m=17, n=7168, k=2048, dtype="bf16", fp8=False),
        # a projection of a ragged chunk, sizes off every tile
        dict(name="linear_ragged_1000", kind="linear", m=1000, n=4104, k=2056, dtype="fp16", fp8=False),
        # a square product of training size
        dict(name="linear_large_8192", kind="linear", m=8192, n=8192, k=8192, dtype="bf16", fp8=False),
        # a block-scaled fp8 projection of a prefill chunk, activations quantised on the way
        dict(name="linear_fp8_block_2048", kind="linear", m=2048, n=7168, k=4096, dtype="bf16", fp8=True),
        # the feed-forward of a tensor-parallel layer (one rank's columns), block-scaled fp8
        dict(name="mlp_fp8_2048", kind="mlp", tokens=2048, hidden=4096, ffn=7168, fp8=True),
        # the token exchange of a training step, forward and backward with gradients of activations and gate weights
        dict(name="train_2048", kind="train", tokens=2048, hidden=4096, experts=64, top_k=8),
        # the sum and the norm behind a row-parallel projection, four ranks
        dict(name="norm_4x256", kind="norm", ranks=4, tokens=256, hidden=7168),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ep", "ep", "ep", "moe", "moe", "linear", "linear", "linear", "mlp", "train", "norm"])
    if kind == "ep":
        q = rng.choice(["fp8", "fp8", "mxfp8", "none"])
        registered = q != "mxfp8" and rng.random() < 0.3
        experts = rng.choice([32, 64, 160, 256, 384])
        top_k = rng.choice([2, 4, 6, 8])
        hidden = rng.choice([1024, 2048, 4096, 5120, 7168])
        if q == "none":
            hidden = min(hidden // (2 if registered else 1) + 8 * rng.randrange(0, 16), MAX_ROW_BYTES // 2 if registered else MAX_ROW_BYTES)
        return dict(kind=kind, tokens=_log(rng, 1, 4096), hidden=hidden, experts=experts, top_k=top_k, quant=q,
                    routing=rng.choice(["logits", "ids"]), registered=registered)
    if kind == "moe":
        return dict(kind=kind, tokens=_log(rng, 1, 3000), hidden=rng.choice([1024, 2048, 4096]), ffn=rng.choice([512, 768, 1024, 1408]),
                    experts=rng.choice([8, 16, 60, 64, 128]), top_k=rng.choice([2, 4, 6, 8]))
    if kind == "linear":
        if rng.random() < 0.35:
            return dict(kind=kind, m=_log(rng, 1, 8192), n=8 * _log(rng, 32, 1024), k=128 * _log(rng, 4, 64), dtype="bf16", fp8=True)
        return dict(kind=kind, m=_log(rng, 1, 8192), n=8 * _log(rng, 16, 1024), k=8 * _log(rng, 16, 1024), dtype=rng.choice(["bf16", "bf16", "fp16"]),
                    fp8=False)
    if kind == "mlp":
        return dict(kind=kind, tokens=256 * _log(rng, 1, 16), hidden=512 * _log(rng, 2, 14), ffn=128 * _log(rng, 6, 112), fp8=rng.random() < 0.6)
    if kind == "train":
        return dict(kind=kind, tokens=_log(rng, 16, 4096), hidden=8 * _log(rng, 64, 640), experts=rng.choice([16, 64, 128]), top_k=rng.choice([2, 4, 8]))
    return dict(kind=kind, ranks=rng.choice([2, 4, 8]), tokens=_log(rng, 1, 1024), hidden=8 * _log(rng, 128, 1024))


# ---- what a program keeps -------------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _comm():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    return txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=1024, device=0)


@functools.lru_cache(maxsize=None)
def _receive_buffer():
    return _comm().symm_empty([MAX_ROWS * MAX_ROW_BYTES], torch.uint8)


@functools.lru_cache(maxsize=None)
def _world(ranks):
    return txr.init_emulated_world(ranks, device=0, buffer_mb=64)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, dtype=torch.bfloat16, scale=1.0):
    return torch.randn(*shape, generator=g, device="cuda").mul_(scale).to(dtype)


def _route_inputs(case, g):
    t, e, k = case["tokens"], case["experts"], case["top_k"]
    logits = torch.randn(t, e, generator=g, device="cuda")
    weights, ids = torch.softmax(logits, dim=1).topk(k, dim=1)
    return logits, weights.contiguous(), ids.to(torch.int32).contiguous()


def _ep_inputs(case, seed):
    g = _generator(seed)
    x = _randn(g, case["tokens"], case["hidden"])
    return (x,) + _route_inputs(case, g)


def _moe_inputs(case, seed):
    g = _generator(seed)
    h, f, e = case["hidden"], case["ffn"], case["experts"]
    x = _randn(g, case["tokens"], h)
    gate = _randn(g, e, h, dtype=torch.float32, scale=h ** -0.5)
    w13 = torch.empty(e, 2 * f, h, device="cuda", dtype=torch.bfloat16)
    w2 = torch.empty(e, h, f, device="cuda", dtype=torch.bfloat16)
    for i in range(e):
        w13[i] = _randn(g, 2 * f, h, scale=h ** -0.5)
        w2[i] = _randn(g, h, f, scale=f ** -0.5)
    return x, gate, w13, w2


def _linear_inputs(case, seed):
    g = _generator(seed)
    dtype = DTYPES[case["dtype"]]
    return _randn(g, case["m"], case["k"], dtype=dtype), _randn(g, case["n"], case["k"], dtype=dtype, scale=case["k"] ** -0.5)


def _mlp_inputs(case, seed):
    g = _generator(seed)
    h, f = case["hidden"], case["ffn"]
    return _randn(g, case["tokens"], h), _randn(g, 2 * f, h, scale=h ** -0.5), _randn(g, h, f, scale=f ** -0.5)


def _norm_inputs(case, seed):
    g = _generator(seed)
    xs = [_randn(g, case["tokens"], case["hidden"]) for _ in range(case["ranks"])]
    return xs, (1.0 + 0.1 * torch.randn(case["hidden"], generator=g, device="cuda")).to(torch.bfloat16)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case)
    if kind == "ep":
        x, logits, weights, ids = _ep_inputs(case, seed)
        state.update(comm=_comm(), x=x, logits=logits, weights=weights, ids=ids, recv=None)
        if case["registered"]:
            # the receive buffer of this size, in registered memory: senders write the rows where they stay
            rows, dtype = case["tokens"] * case["top_k"], torch.float8_e4m3fn if case["quant"] == "fp8" else x.dtype
            flat = _receive_buffer()[: rows * case["hidden"] * dtype.itemsize]
            state["recv"] = flat.view(dtype).view(rows, case["hidden"])
    elif kind == "moe":
        x, gate, w13, w2 = _moe_inputs(case, seed)
        cfg = MoEConfig(hidden=case["hidden"], ffn=case["ffn"], num_experts=case["experts"], top_k=case["top_k"])
        layer = ExpertParallelMoE(_comm(), cfg, with_experts=False)
        layer.gate.data.copy_(gate)
        layer.w13, layer.w2 = torch.nn.Parameter(w13), torch.nn.Parameter(w2)
        state.update(layer=layer, x=x)
    elif kind == "linear":
        a, b = _linear_inputs(case, seed)
        state.update(a=a, b=b)
        if case["fp8"]:
            state["b"], state["scale_b"] = gemm.quantize_weight_128x128(b)
    elif kind == "mlp":
        x, w13, w2 = _mlp_inputs(case, seed)
        comm = _comm()
        cfg = TPMlpConfig(hidden=case["hidden"], ffn=case["ffn"], tokens=case["tokens"], fp8_block=case["fp8"])
        layer = SequenceParallelMLP(comm, cfg, w13, w2)
        for buffer in (layer.stage_rows, layer.stage_out) + ((layer.stage_scales,) if case["fp8"] else ()):
            weakref.finalize(layer, comm.symm_free, buffer).atexit = False
        state.update(layer=layer, x=x)
    elif kind == "train":
        x, _, weights, ids = _ep_inputs(case, seed)
        state.update(x=x.requires_grad_(), probs=weights.requires_grad_(), ids=ids, grad=_randn(_generator(seed + 1), *x.shape),
                     dispatcher=TileXRTokenDispatcher(_comm(), case["experts"], case["top_k"], case["hidden"]))
    else:
        xs, gamma = _norm_inputs(case, seed)
        state.update(world=_world(case["ranks"]), xs=xs, gamma=gamma)
    return state


def run(state):
    kind = state["kind"]
    if kind == "ep":
        comm, q = state["comm"], QUANT[state["quant"]]
        routed = (dict(gate_logits=state["logits"], score_func=quant.SCORE_SIGMOID) if state["routing"] == "logits" else
                  dict(expert_ids=state["ids"], expert_scales=state["weights"]))
        d = ep.dispatch(comm, state["x"], num_experts=state["experts"], top_k=state["top_k"], quant_mode=q, expand_x_out=state["recv"], **routed)
        rows = d.expand_x
        if state["quant"] == "fp8":
            rows = quant.fp8_dequant_1x128(rows, d.dynamic_scales, torch.bfloat16)
        elif state["quant"] == "mxfp8":
            rows = quant.mxfp8_dequant(rows, d.dynamic_scales, torch.bfloat16)
        weights = d.topk_weights if state["routing"] == "logits" else state["weights"]
        y = ep.combine(comm, rows, d, expert_scales=weights)
        out = dict(y=y, weights=weights, ids=d.topk_ids, counts=d.expert_token_nums, assist=d.assist, expand_x=d.expand_x)
        if state["quant"] != "none":
            out.update(expand_x=d.expand_x.view(torch.uint8), scales=d.dynamic_scales)
        return out
    if kind == "moe":
        return state["layer"](state["x"])
    if kind == "linear":
        if not state["fp8"]:
            return gemm.matmul(state["a"], state["b"])
        a, scale_a = quant.fp8_quant_1x128(state["a"])
        return gemm.matmul_fp8_block(a, scale_a, state["b"], state["scale_b"])
    if kind == "mlp":
        return state["layer"](state["x"])
    if kind == "train":
        rows, counts = state["dispatcher"].token_permutation(state["x"], state["probs"], state["ids"])
        y, _ = state["dispatcher"].token_unpermutation(rows)
        grad_x, grad_probs = torch.autograd.grad(y, (state["x"], state["probs"]), state["grad"])
        return dict(y=y.detach(), rows=rows.detach(), counts=counts, grad_x=grad_x, grad_probs=grad_probs)
    xs, gamma = state["xs"], state["gamma"]
    return state["world"].run(lambda c, r: collectives.all_reduce_rmsnorm(c, xs[r], gamma))


# ---- what a pass cannot do without --------------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("ep", "train"):
        t, h, routes = case["tokens"], case["hidden"], case["tokens"] * case["top_k"]
        tokens, rows = t * h * 2, routes * h * 2
        if kind == "train":
            # permutation, unpermutation, the gradient of the rows (read beside the rows themselves) and that of the tokens
            return {"bytes": (tokens + rows) + (rows + tokens) + (tokens + 2 * rows) + (rows + tokens), "flops": 6.0 * routes * h}
        sent = {"none": rows, "fp8": routes * (h + h // 128 * 4), "mxfp8": routes * (h + h // 32)}[case["quant"]]
        logits = t * case["experts"] * 4 if case["routing"] == "logits" else routes * 8
        stand_in = 0 if case["quant"] == "none" else sent + rows
        return {"bytes": tokens + logits + sent + routes * 28 + stand_in + rows + tokens, "flops": 2.0 * routes * h}
    if kind == "moe":
        t, h, f, e, k = case["tokens"], case["hidden"], case["ffn"], case["experts"], case["top_k"]
        touched = e * (1.0 - (1.0 - k / e) ** t)
        return {"bytes": int(2 * t * h * 2 + e * h * 4 + touched * 3 * h * f * 2), "flops": 2.0 * t * h * e + 6.0 * t * k * h * f}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        weight = n * k * (1 if case["fp8"] else 2)
        return {"bytes": m * k * 2 + weight + m * n * 2, "flops": 2.0 * m * n * k}
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * t * h * 2 + 3 * h * f * (1 if case["fp8"] else 2), "flops": 6.0 * t * h * f}
    n = case["ranks"] * case["tokens"] * case["hidden"] * 2
    return {"bytes": 2 * n + case["hidden"] * 2, "flops": (case["ranks"] + 4.0) * case["ranks"] * case["tokens"] * case["hidden"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "ep":
        # two roundings to bf16 of fp32 sums; a share of whole values for scores and quantised elements that lie on a tie
        return {"rel": 1e-2, "max": 5e-2, "differ": 1e-3}
    if kind == "moe":
        # a token whose eighth and ninth expert score alike may take the other; fp8 elements on a tie take the neighbour
        return {"rel": 2e-2}
    if kind == "linear":
        return {"rel": 1e-3 if case["dtype"] == "fp16" else 1e-2}
    if kind == "mlp":
        # the activation is rounded to bf16 and then to fp8, whose neighbours are 6 % apart
        return {"rel": 4e-2 if case["fp8"] else 1.5e-2}
    if kind == "train":
        return {"rel": 1e-2, "max": 5e-2, "differ": 0.0}
    return {"rel": 1e-2, "max": 5e-2}


# ---- the same results in 64 bits ---------------------------------------------------------------------------------------


def _fp8_blocks(x):
    """x [rows, h] in 64 bits -> (e4m3 values in 64 bits, scales [rows, h / 128]): one scale per 128 elements."""
    blocks = x.view(x.shape[0], -1, 128)
    amax = blocks.abs().amax(dim=2, keepdim=True).clamp_min(1e-4)
    q = (blocks * (448.0 / amax)).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return q.view(x.shape), (amax / 448.0).squeeze(2)


def _mx_blocks(x):
    """MXFP8: 32 elements share the exponent floor(log2(amax)) - 8; -> (e4m3 values, exponent bytes [rows, h / 32])."""
    blocks = x.view(x.shape[0], -1, 32)
    amax = blocks.abs().amax(dim=2, keepdim=True)
    e = torch.where(amax > 0, torch.frexp(amax.float())[1].double() - 1.0 - 8.0, torch.full_like(amax, -127.0)).clamp(-127.0, 127.0)
    q = (blocks * torch.exp2(-e)).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return q.view(x.shape), (e + 127.0).squeeze(2).to(torch.uint8)


def _expand(q, scales, width):
    return (q.double().view(q.shape[0], -1, width) * scales.unsqueeze(2)).view(q.shape)


def _exact_ep(case, seed):
    x, logits, weights, ids = _ep_inputs(case, seed)
    t, k = case["tokens"], case["top_k"]
    if case["routing"] == "logits":
        weights, ids = torch.sigmoid(logits.double()).topk(k, dim=1)
        weights = weights / weights.sum(dim=1, keepdim=True)
        ids = ids.to(torch.int32)
    flat = ids.reshape(-1).long()
    order = torch.sort(flat, stable=True).indices          # rows by expert, then by token and slot
    token = torch.div(order, k, rounding_mode="floor")
    counts = torch.bincount(flat, minlength=case["experts"])
    assist = torch.stack((torch.zeros_like(token), token, order % k, flat[order]), dim=1).to(torch.int32)
    if case["quant"] == "none":
        y = x.double() * weights.double().sum(dim=1, keepdim=True)
        return dict(y=y, weights=weights, ids=ids, counts=counts, assist=assist, expand_x=x[token])
    if case["quant"] == "fp8":
        q, s = _fp8_blocks(x.double())
        deq = _expand(q, s, 128)
    else:
        q, s = _mx_blocks(x.double())
        deq = _expand(q, torch.exp2(s.double() - 127.0), 32)
    y = deq * weights.double().sum(dim=1, keepdim=True)
    return dict(y=y, weights=weights, ids=ids, counts=counts, assist=assist, expand_x=q.view(torch.uint8)[token], scales=s[token])


def _exact_moe(case, seed):
    x, gate, w13, w2 = _moe_inputs(case, seed)
    weights, ids = torch.sigmoid(x.double() @ gate.double().t()).topk(case["top_k"], dim=1)
    weights = weights / weights.sum(dim=1, keepdim=True)
    q, s = _fp8_blocks(x.double())
    rows = _expand(q, s, 128)
    y = torch.zeros_like(rows)
    for e in range(case["experts"]):
        token, slot = torch.nonzero(ids == e, as_tuple=True)
        if token.numel():
            up = rows[token] @ w13[e].double().t()
            act = torch.nn.functional.silu(up[:, 0::2]) * up[:, 1::2]
            y.index_add_(0, token, (act @ w2[e].double().t()) * weights[token, slot].unsqueeze(1))
    return y


def _weight_blocks(w):
    """quantize_weight_128x128 and back, in 64 bits; the scales are fp32 numbers by definition of the format."""
    n, k = w.shape
    nb = -(-n // 128)
    blocks = torch.nn.functional.pad(w.float(), (0, 0, 0, nb * 128 - n)).view(nb, 128, k // 128, 128)
    scale = (blocks.abs().amax(dim=(1, 3)).clamp_min(1e-4) / 448.0)[:, None, :, None]
    q = (blocks / scale).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
    return (q.double() * scale.double()).view(nb * 128, k)[:n]


def _fp8_rows(x):
    return _expand(*_fp8_blocks(x), 128)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ep":
        return _exact_ep(case, seed)
    if kind == "moe":
        return _exact_moe(case, seed)
    if kind == "linear":
        a, b = _linear_inputs(case, seed)
        if case["fp8"]:
            return _fp8_rows(a.double()) @ _weight_blocks(b).t()
        return a.double() @ b.double().t()
    if kind == "mlp":
        x, w13, w2 = _mlp_inputs(case, seed)
        f = case["ffn"]
        if case["fp8"]:
            up = _fp8_rows(x.double()) @ _weight_blocks(w13).t()
            act = torch.nn.functional.silu(up[:, :f]) * up[:, f:]
            return _fp8_rows(act) @ _weight_blocks(w2).t()
        up = x.double() @ w13.double().t()
        return (torch.nn.functional.silu(up[:, :f]) * up[:, f:]) @ w2.double().t()
    if kind == "train":
        x, _, weights, ids = _ep_inputs(case, seed)
        grad = _randn(_generator(seed + 1), *x.shape).double()
        flat = ids.reshape(-1).long()
        token = torch.div(torch.sort(flat, stable=True).indices, case["top_k"], rounding_mode="floor")
        total = weights.double().sum(dim=1, keepdim=True)
        dots = (grad * x.double()).sum(dim=1, keepdim=True)
        return dict(y=x.double() * total, rows=x[token], counts=torch.bincount(flat, minlength=case["experts"]), grad_x=grad * total,
                    grad_probs=dots.expand(-1, case["top_k"]))
    xs, gamma = _norm_inputs(case, seed)
    total = sum(x.double() for x in xs)
    y = total * torch.rsqrt(total.square().mean(dim=1, keepdim=True) + 1e-6) * gamma.double()
    return [y] * case["ranks"]
