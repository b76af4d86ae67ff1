"""Elementwise kernels beside the GEMMs and the exchange, against plain PyTorch at the edges of their tiling."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def txr():
    import tilexr_b200 as t

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return t


def _gate_up(rows, f, dtype, seed=3):
    g = torch.Generator().manual_seed(seed)
    x = (torch.randn(rows, 2 * f, generator=g) * 3.0).to(dtype).cuda()
    x[0, 0], x[0, f] = float("inf"), 2.0          # an infinite gate, a zero, a NaN, a row of zeros
    x[-1, 1], x[-1, f + 2] = 0.0, float("nan")
    if rows > 2:
        x[1] = 0.0
    return x


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,f", [(1, 8), (3, 24), (33, 40), (257, 128), (1000, 7168)])
def test_swiglu_matches_the_unfused_form(txr, rows, f, dtype):
    x = _gate_up(rows, f, dtype)
    want = (torch.nn.functional.silu(x[:, :f].float()) * x[:, f:].float()).to(dtype)
    got = txr.quant.swiglu(x)
    assert got.shape == want.shape and got.dtype == dtype
    # both round an fp32 value once; the fp32 values may differ in their last bits (exp, the order of * and /), which moves
    # a rounding by one unit in the last place at most
    ulp = torch.finfo(dtype).eps
    finite = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(torch.isinf(got), torch.isinf(want))
    diff = (got.float() - want.float()).abs()
    assert (diff[finite] <= ulp * want.float().abs()[finite] + torch.finfo(dtype).smallest_normal * ulp).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,f", [(1, 128), (3, 384), (31, 896), (1000, 7168)])
def test_swiglu_fp8_quant_is_the_quantised_swiglu(txr, rows, f, dtype):
    x = _gate_up(rows, f, dtype)
    q, s = txr.quant.swiglu_fp8_quant_1x128(x)
    want_q, want_s = txr.quant.fp8_quant_1x128(txr.quant.swiglu(x))
    assert torch.equal(q.view(torch.uint8), want_q.view(torch.uint8)) and torch.equal(s, want_s)


@pytest.mark.parametrize("rows,h", [(1, 128), (5, 128), (7, 384), (33, 640)])
def test_fp8_quant_rows_that_do_not_fill_a_warp(txr, rows, h):
    """A 128-element block is eight threads, wherever its row starts in the launch."""
    from tilexr_b200.utils import oracle

    x = (torch.randn(rows, h, generator=torch.Generator().manual_seed(rows)) * 5).to(torch.bfloat16)
    q, s = txr.quant.fp8_quant_1x128(x.cuda())
    want_q, want_s = oracle.fp8_quant_1x128_ref(x)
    assert torch.equal(s.cpu(), want_s) and torch.equal(q.cpu().view(torch.uint8), want_q.view(torch.uint8))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,h", [(1, 128), (3, 128), (9, 384), (130, 7168)])
def test_fp8_dequant_at_the_edges_of_a_launch(txr, rows, h, dtype):
    x = (torch.randn(rows, h, generator=torch.Generator().manual_seed(h)) * 4).to(dtype).cuda()
    q, s = txr.quant.fp8_quant_1x128(x)
    got = txr.quant.fp8_dequant_1x128(q, s, dtype)
    assert torch.equal(got, (q.float().view(rows, -1, 128) * s[:, :, None]).view(rows, h).to(dtype))


@pytest.mark.parametrize("e5m2", [False, True])
@pytest.mark.parametrize("rows,h", [(1, 8), (3, 40), (5, 33), (7, 100), (130, 4096)])
def test_mxfp8_dequant_rows_of_any_length(txr, rows, h, e5m2):
    """Rows of a multiple of eight elements take eight at a time, the others one; a row may end inside its last block."""
    x = (torch.randn(rows, h, generator=torch.Generator().manual_seed(h)) * 4).to(torch.bfloat16).cuda()
    q, s = txr.quant.mxfp8_quant(x, e5m2)
    got = txr.quant.mxfp8_dequant(q, s)
    scale = torch.exp2(s.float() - 127).repeat_interleave(32, dim=1)[:, :h]
    assert torch.equal(got, (q.float() * scale).to(torch.bfloat16))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens,h,experts", [(1, 8, 1), (32, 2048, 64), (63, 264, 33), (65, 2048, 32), (130, 1032, 60), (1000, 7168, 256)])
def test_router_logits_in_fp32(txr, tokens, h, experts, dtype):
    """K shorter than a chunk, parts of K that are empty or ragged, tokens and experts off the tile."""
    g = torch.Generator().manual_seed(h)
    x = torch.randn(tokens, h, generator=g).to(dtype).cuda()
    gate = (torch.randn(experts, h, generator=g) * h ** -0.5).cuda()
    got = txr.quant.router_logits(x, gate)
    want = x.double() @ gate.double().t()
    # a chain of at most 32 * ceil(h / 256) multiply-adds per warp and 15 additions behind it, each half an fp32 unit of a partial sum
    steps = 32 * ((h + 255) // 256) + 16
    bound = (x.double().abs() @ gate.double().abs().t()) * steps * 2.0 ** -24
    assert got.dtype == torch.float32 and ((got.double() - want).abs() <= bound).all()


def _router(experts=8, h=64):
    from types import SimpleNamespace

    from tilexr_b200.models import ExpertParallelMoE, MoEConfig

    return ExpertParallelMoE(SimpleNamespace(world_size=1, rank=0), MoEConfig(hidden=h, num_experts=experts), with_experts=False).requires_grad_(False)


@pytest.mark.parametrize("how", ["forward_mode", "vmap", "jvp", "jit_trace", "make_fx"])
def test_route_logits_under_transforms_and_tracing(txr, how):
    """The router's kernel is not an operator of torch: transforms and tracers must see the matmul it stands for."""
    layer = _router()
    g = torch.Generator().manual_seed(4)
    x = torch.randn(5, 64, generator=g).to(torch.bfloat16).cuda()
    t = torch.randn(5, 64, generator=g).to(torch.bfloat16).cuda()
    plain = lambda v: v.float() @ layer.gate.t()      # noqa: E731
    close = dict(rtol=1e-5, atol=1e-5)                # fp32 sums of 64 products of order 1/50
    with torch.no_grad():
        if how == "forward_mode":
            with torch.autograd.forward_ad.dual_level():
                out = layer.route_logits(torch.autograd.forward_ad.make_dual(x, t))
                tangent = torch.autograd.forward_ad.unpack_dual(out).tangent
            assert tangent is not None and torch.allclose(tangent, plain(t), **close)
        elif how == "jvp":
            out, tangent = torch.func.jvp(layer.route_logits, (x,), (t,))
            assert torch.allclose(out, plain(x), **close) and torch.allclose(tangent, plain(t), **close)
        elif how == "vmap":
            out = torch.func.vmap(layer.route_logits)(torch.stack((x, t)))
            assert torch.allclose(out, torch.stack((plain(x), plain(t))), **close)
        elif how == "jit_trace":
            traced = torch.jit.trace(lambda v: layer.route_logits(v), x, check_trace=False)
            assert torch.allclose(traced(t), plain(t), **close)
        else:
            from torch.fx.experimental.proxy_tensor import make_fx

            traced = make_fx(lambda v: layer.route_logits(v))(x)
            assert torch.allclose(traced(t), plain(t), **close)


def test_router_logits_and_swiglu_on_another_device(txr):
    """Both stand for torch operators, which follow their tensors' device: the current one does not matter, nor which came first."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two devices in one process")
    g = torch.Generator().manual_seed(6)
    x, gate = torch.randn(40, 2048, generator=g).to(torch.bfloat16), torch.randn(64, 2048, generator=g) / 64
    with torch.cuda.device(0):
        got = [(txr.quant.router_logits(x.to(d), gate.to(d)).cpu(), txr.quant.swiglu(x.to(d)).cpu()) for d in ("cuda:0", "cuda:1")]
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
