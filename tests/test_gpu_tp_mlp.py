"""The sequence-parallel feed-forward on one rank: the fused GEMMs, SwiGLU and quantisation kernels behind it against a product in 64 bits of
the same weights, with roundings where the layer rounds.  (Several ranks: tests/test_tp_mlp_cpu.py for the layer, tests/test_gpu_gemm.py for the kernels.)"""
import types

import pytest
import torch

from conftest import require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def txr():
    require_cuda()
    import tilexr_b200

    return tilexr_b200


def _off_the_grid(gemm):
    """The GEMM module with a first product that starts between 16-byte boundaries."""
    def moved(result):
        flat = torch.empty(result.numel() + 8, dtype=result.dtype, device=result.device)
        view = flat[3:3 + result.numel()].view(result.shape)
        view.copy_(result)
        assert view.is_contiguous() and view.data_ptr() % 16 != 0
        return view

    names = {n: getattr(gemm, n) for n in ("matmul_reduce_scatter", "matmul_reduce_scatter_fp8_block", "quantize_weight_128x128")}
    return types.SimpleNamespace(all_gather_matmul=lambda *a: moved(gemm.all_gather_matmul(*a)),
                                 all_gather_matmul_fp8_block=lambda *a: moved(gemm.all_gather_matmul_fp8_block(*a)), **names)


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("fp8,dtype,tokens,hidden,ffn", [(False, torch.bfloat16, 256, 512, 264), (False, torch.float16, 512, 264, 1032),
                                                         (True, torch.bfloat16, 512, 1024, 896), (True, torch.float16, 256, 512, 2944)])
def test_sequence_parallel_mlp_on_one_rank(txr, port, fp8, dtype, tokens, hidden, ffn, aligned):
    from tilexr_b200.models.tp_mlp import SequenceParallelMLP, TPMlpConfig, shard_weights
    from tilexr_b200.ops import gemm
    from tilexr_b200.utils import oracle

    g = torch.Generator().manual_seed(hidden)
    x = torch.randn(tokens, hidden, generator=g).to(dtype).cuda()
    wg, wu, wd = [(torch.randn(*s, generator=g) * s[1] ** -0.5).to(dtype).cuda() for s in ((ffn, hidden), (ffn, hidden), (hidden, ffn))]
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=64, device=0)
    try:
        w13, w2 = shard_weights(wg, wu, wd, 0, 1)
        cfg = TPMlpConfig(hidden=hidden, ffn=ffn, tokens=tokens, dtype=dtype, fp8_block=fp8)
        layer = SequenceParallelMLP(comm, cfg, w13, w2, ops=None if aligned else _off_the_grid(gemm))
        for _ in range(2):
            y = layer(x)
        torch.cuda.synchronize()
        assert comm.device_status() == 0 and y.shape == x.shape and y.dtype == dtype

        def rounded(v):
            """Activations as a product gets them."""
            v = v.to(dtype)
            if not fp8:
                return v.double()
            return oracle.fp8_dequant_1x128_ref(*oracle.fp8_quant_1x128_ref(v)).double().cuda()

        def weight(w, s):
            return w.double() if not fp8 else w.double() * s.double().repeat_interleave(128, 0)[:w.shape[0]].repeat_interleave(128, 1)

        gu = (rounded(x) @ weight(layer.w13, getattr(layer, "s13", None)).t()).to(dtype).double()
        act = torch.nn.functional.silu(gu[:, :ffn]) * gu[:, ffn:]
        want = rounded(act) @ weight(layer.w2, getattr(layer, "s2", None)).t()
        # three roundings to 16 bits of at most eps / 2 each on either side; with fp8 a last bit of the product can move a quantised
        # activation by one step (an eighth of its value at most), one in a hundred of them at the very most: 1/8 * sqrt(1/100)
        bound = 3 * torch.finfo(dtype).eps + (0.0125 if fp8 else 0.0)
        assert (y.double() - want).norm() <= bound * want.norm()
    finally:
        comm.destroy()
