"""tcgen05 GEMM and its all-gather / reduce-scatter fusions against an fp32 PyTorch matmul."""
import pytest
import torch

from conftest import require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def txr():
    require_cuda()
    import tilexr_b200

    return tilexr_b200


def _close(got, want, k):
    got, want = got.float().cpu(), want.float().cpu()
    tol = 2e-2 * max(1.0, (k ** 0.5) / 8)
    assert torch.allclose(got, want, rtol=2e-2, atol=tol), (got - want).abs().max()
    assert (got - want).abs().mean() < 0.02 * want.abs().mean() + 1e-3


@pytest.mark.parametrize("m,n,k,dtype", [
    (128, 256, 64, torch.bfloat16),
    (512, 512, 256, torch.bfloat16),
    (300, 264, 200, torch.bfloat16),        # ragged in every dimension
    (2048, 2048, 1024, torch.float16),
    (1024, 7168, 2048, torch.bfloat16),     # more tiles than SMs: both accumulator buffers, ring wrap
])
def test_matmul(txr, m, n, k, dtype):
    g = torch.Generator().manual_seed(m + n + k)
    a = (torch.randn(m, k, generator=g) * 0.5).to(dtype).cuda()
    b = (torch.randn(n, k, generator=g) * 0.5).to(dtype).cuda()
    for _ in range(2):
        c = txr.gemm.matmul(a, b)
    torch.cuda.synchronize()
    _close(c, a.float() @ b.float().t(), k)


@pytest.mark.parametrize("m,n,k,fmt", [
    (256, 256, 128, torch.float8_e4m3fn),
    (1000, 520, 400, torch.float8_e4m3fn),      # ragged in every dimension
    (2048, 4096, 2048, torch.float8_e5m2),
    (4096, 2048, 7168, torch.float8_e4m3fn),    # more tiles than CTA pairs, long K
])
def test_matmul_fp8(txr, m, n, k, fmt):
    """fp8 operands on the kind::f8f6f4 tensor-core path against an fp32 product of the same fp8 values."""
    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g).to(fmt).cuda()
    b = torch.randn(n, k, generator=g).to(fmt).cuda()
    alpha = 0.37
    for _ in range(2):
        c = txr.gemm.matmul_fp8(a, b, alpha)
    torch.cuda.synchronize()
    want = alpha * (a.float() @ b.float().t())
    got = c.float()
    # fp32 accumulation of exact fp8 products: only the final bf16 rounding differs
    assert torch.allclose(got, want, rtol=1e-2, atol=1e-2 * (k ** 0.5)), (got - want).abs().max()
    assert (got - want).abs().mean() < 4e-3 * want.abs().mean() + 1e-4


@pytest.mark.parametrize("ranks,shard_rows,n,k", [(2, 128, 256, 256), (2, 256, 512, 1024), (4, 128, 768, 512), (4, 512, 1024, 512)])
def test_all_gather_matmul(txr, ranks, shard_rows, n, k):
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    g = torch.Generator().manual_seed(7)
    shards = [(torch.randn(shard_rows, k, generator=g) * 0.5).to(torch.bfloat16).cuda() for _ in range(ranks)]
    bs = [(torch.randn(n, k, generator=g) * 0.5).to(torch.bfloat16).cuda() for _ in range(ranks)]
    staging = world.symm_empty((ranks * shard_rows, k), torch.bfloat16)
    full = torch.cat(shards).float()
    for _ in range(3):
        outs = world.run(lambda c, r: txr.gemm.all_gather_matmul(c, shards[r], bs[r], staging[r]))
        world.check()
    for r in range(ranks):
        _close(outs[r], full @ bs[r].float().t(), k)
    world.destroy()


@pytest.mark.parametrize("ranks,shard_rows,n,k", [(2, 128, 256, 128), (2, 256, 512, 512), (4, 128, 512, 256), (4, 512, 1024, 768)])
def test_matmul_reduce_scatter(txr, ranks, shard_rows, n, k):
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    g = torch.Generator().manual_seed(9)
    m = ranks * shard_rows
    a = [(torch.randn(m, k, generator=g) * 0.5).to(torch.bfloat16).cuda() for _ in range(ranks)]
    b = [(torch.randn(n, k, generator=g) * 0.5).to(torch.bfloat16).cuda() for _ in range(ranks)]
    staging = world.symm_empty((m, n), torch.bfloat16)
    # partial products travel as bf16 and are summed in rank order in fp32
    partial = [(a[r].float() @ b[r].float().t()).to(torch.bfloat16).float() for r in range(ranks)]
    want = partial[0]
    for p in partial[1:]:
        want = want + p
    for _ in range(3):
        outs = world.run(lambda c, r: txr.gemm.matmul_reduce_scatter(c, a[r], b[r], staging[r]))
        world.check()
    for r in range(ranks):
        _close(outs[r], want[r * shard_rows:(r + 1) * shard_rows], k * ranks)
    world.destroy()


def test_matmul_all_reduce(txr):
    """GEMM with the reduce-scatter in its epilogue, then an all-gather of the reduced shards: every rank ends with the sum."""
    ranks, shard_rows, n, k = 2, 128, 256, 256
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    g = torch.Generator().manual_seed(21)
    m = ranks * shard_rows
    a = [(torch.randn(m, k, generator=g) * 0.5).to(torch.bfloat16).cuda() for _ in range(ranks)]
    b = [(torch.randn(n, k, generator=g) * 0.5).to(torch.bfloat16).cuda() for _ in range(ranks)]
    staging = world.symm_empty((m, n), torch.bfloat16)
    want = sum((a[r].float() @ b[r].float().t()).to(torch.bfloat16).float() for r in range(ranks))
    for _ in range(2):
        outs = world.run(lambda c, r: txr.gemm.matmul_all_reduce(c, a[r], b[r], staging[r]))
        world.check()
    for r in range(ranks):
        _close(outs[r], want, k * ranks)
    world.destroy()


@pytest.mark.parametrize("m,n,k", [(128, 256, 128), (256, 256, 512), (300, 384, 1024), (1024, 2048, 7168), (96, 128, 256)])
def test_matmul_fp8_block_scaled(txr, m, n, k):
    """Block-scaled fp8 (1 x 128 activation scales, 128 x 128 weight scales, fp32) against the fp32 product of the
    dequantised operands.  Rows are given very different magnitudes, and so are the weight blocks, so that a scale
    applied to the wrong row, column group or block of K shows."""
    from tilexr_b200.utils import oracle

    g = torch.Generator().manual_seed(31)
    a = torch.randn(m, k, generator=g) * (0.25 + 4.0 * torch.rand(m, 1, generator=g)) * (0.5 + torch.rand(1, k // 128, generator=g)).repeat_interleave(128, dim=1)
    w = torch.randn(n, k, generator=g) * 0.5
    nb = (n + 127) // 128
    w = w * (0.2 + 3.0 * torch.rand(nb, k // 128, generator=g)).repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
    qa, sa = txr.quant.fp8_quant_1x128(a.to(torch.bfloat16).cuda())
    qw, sw = txr.gemm.quantize_weight_128x128(w.cuda())
    got = txr.gemm.matmul_fp8_block(qa, sa, qw, sw).float().cpu()
    torch.cuda.synchronize()
    da = oracle.fp8_dequant_1x128_ref(qa.cpu(), sa.cpu())
    dw = qw.cpu().float().view(-1, k) * sw.cpu().repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
    want = da @ dw.t()
    assert torch.allclose(got, want, rtol=1e-2, atol=1e-2 * want.abs().max().item()), (got - want).abs().max()
    assert (got - want).abs().mean() < 4e-3 * want.abs().mean() + 1e-4


@pytest.mark.parametrize("counts,n,k,swiglu", [
    ([300, 0, 17, 256, 1, 700], 512, 256, False),          # empty group, groups smaller and larger than a tile, ragged starts
    ([300, 0, 17, 256, 1, 700], 512, 256, True),
    ([5] * 70, 264, 128, False),                             # more groups than one launch holds, N not a multiple of the tile
    ([2000, 3000, 100, 4000], 4096, 1024, True),             # more tiles than CTA pairs
])
def test_grouped_matmul(txr, counts, n, k, swiglu):
    """One launch over all groups, row counts read on the device, against fp32 PyTorch; rows past the counts untouched."""
    g = torch.Generator().manual_seed(sum(counts) + n)
    total = sum(counts)
    rows = (torch.randn(total + 40, k, generator=g) * 0.5).to(torch.bfloat16).cuda()
    w = (torch.randn(len(counts), n, k, generator=g) * 0.2).to(torch.bfloat16).cuda()
    group_rows = torch.tensor(counts, dtype=torch.int64).cuda()
    epi = txr.gemm.EPILOGUE_SWIGLU if swiglu else txr.gemm.EPILOGUE_STORE
    out = torch.full((total + 40, n // 2 if swiglu else n), 7.0, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):
        got = txr.gemm.grouped_matmul(rows, w, group_rows, epilogue=epi, out=out)
    torch.cuda.synchronize()
    want = txr.gemm.grouped_matmul_ref(rows, w, group_rows, epi)
    _close(got[:total], want[:total], k)
    assert torch.all(got[total:] == 7.0)


def _block_operands(txr, rows, n, k, seed):
    g = torch.Generator().manual_seed(seed)
    a = torch.randn(rows, k, generator=g) * (0.25 + 4.0 * torch.rand(rows, 1, generator=g))
    w = torch.randn(n, k, generator=g) * 0.5
    qa, sa = txr.quant.fp8_quant_1x128(a.to(torch.bfloat16).cuda())
    qw, sw = txr.gemm.quantize_weight_128x128(w.cuda())
    return qa, sa, qw, sw


def _block_product(qa, sa, qw, sw):
    k = qa.shape[1]
    da = qa.float().cpu().view(qa.shape[0], k // 128, 128) * sa.cpu().unsqueeze(-1)
    dw = qw.float().cpu() * sw.cpu().repeat_interleave(128, dim=0)[:qw.shape[0]].repeat_interleave(128, dim=1)
    return da.view(qa.shape[0], k) @ dw.t()


@pytest.mark.parametrize("ranks,shard_rows,n,k", [(2, 256, 256, 512), (2, 512, 640, 1024), (4, 256, 512, 1536)])
def test_all_gather_matmul_fp8_block(txr, ranks, shard_rows, n, k):
    """Block-scaled fp8 GEMM fused with the all-gather of A: every rank's rows AND scales travel into the others' staging
    buffers during the launch; three launches in a row reuse the buffers behind the reuse guard."""
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    ops = [_block_operands(txr, shard_rows, n, k, 50 + r) for r in range(ranks)]
    a_staging = world.symm_empty((ranks * shard_rows, k), torch.float8_e4m3fn)
    s_staging = world.symm_empty((ranks * shard_rows, k // 128), torch.float32)
    for _ in range(3):
        outs = world.run(lambda c, r: txr.gemm.all_gather_matmul_fp8_block(c, ops[r][0], ops[r][1], a_staging[r], s_staging[r], ops[r][2], ops[r][3]))
        world.check()
    qa_all = torch.cat([o[0] for o in ops])
    sa_all = torch.cat([o[1] for o in ops])
    for r in range(ranks):
        want = _block_product(qa_all, sa_all, ops[r][2], ops[r][3])
        got = outs[r].float().cpu()
        assert torch.allclose(got, want, rtol=1e-2, atol=1e-2 * want.abs().max().item()), (got - want).abs().max()
        assert (got - want).abs().mean() < 4e-3 * want.abs().mean() + 1e-4
    world.destroy()


@pytest.mark.parametrize("ranks,shard_rows,n,k", [(2, 256, 256, 256), (2, 256, 768, 1024), (4, 256, 512, 512)])
def test_matmul_reduce_scatter_fp8_block(txr, ranks, shard_rows, n, k):
    """Block-scaled fp8 GEMM fused with the reduce-scatter of its result: partial tiles travel as bf16 and are added in
    rank order in fp32."""
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    m = ranks * shard_rows
    ops = [_block_operands(txr, m, n, k, 70 + r) for r in range(ranks)]
    staging = world.symm_empty((m, n), torch.bfloat16)
    partial = [_block_product(*ops[r]).to(torch.bfloat16).float() for r in range(ranks)]
    want = partial[0]
    for p in partial[1:]:
        want = want + p
    for _ in range(3):
        outs = world.run(lambda c, r: txr.gemm.matmul_reduce_scatter_fp8_block(c, ops[r][0], ops[r][1], ops[r][2], ops[r][3], staging[r]))
        world.check()
    for r in range(ranks):
        got = outs[r].float().cpu()
        ref = want[r * shard_rows:(r + 1) * shard_rows]
        assert torch.allclose(got, ref, rtol=2e-2, atol=2e-2 * ref.abs().max().item()), (got - ref).abs().max()
        assert (got - ref).abs().mean() < 6e-3 * ref.abs().mean() + 1e-4
    world.destroy()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (1, 128, 64), (16, 120, 72), (17, 7168, 2048), (33, 136, 2056), (64, 8200, 2048), (65, 4096, 320),
                                   (65, 264, 4096), (128, 264, 4104), (129, 512, 4100 // 8 * 8), (300, 1024, 4096), (1000, 512, 4096), (5, 40960, 136)])
def test_matmul_few_rows(txr, m, n, k, dtype):
    """Tiles of 128 columns by 16 to 128 rows: remainders of both, K split over one to eight CTAs with a ragged last part,
    more tiles than places."""
    g = torch.Generator().manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g).to(dtype).cuda()
    b = (torch.randn(n, k, generator=g) * k ** -0.5).to(dtype).cuda()
    want = a.double() @ b.double().t()
    for _ in range(2):
        got = txr.gemm.matmul(a, b).double()
        # fp32 sums of k products (k eps of the sum of magnitudes at the very most), rounded once to the output type
        bound = want.abs() * torch.finfo(dtype).eps / 2 + (a.double().abs() @ b.double().abs().t()) * k * 2.0 ** -24 + 2.0 ** -24
        assert ((got - want).abs() <= bound).all()


@pytest.mark.parametrize("epilogue", [0, 1])
@pytest.mark.parametrize("groups,n,k,counts", [(3, 144, 72, [0, 5, 0]), (5, 256, 128, [1, 0, 40, 2, 17]), (70, 272, 64, None), (300, 128, 64, None)])
def test_grouped_matmul_few_rows_per_group(txr, groups, n, k, counts, epilogue):
    """Empty groups, a group of several row chunks, more groups than one launch takes, rows behind the last group."""
    g = torch.Generator().manual_seed(groups)
    if counts is None:
        counts = torch.randint(0, 6, (groups,), generator=g).tolist()
        counts[groups // 2] = 50
    total = sum(counts)
    rows = torch.randn(total + 7, k, generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn(groups, n, k, generator=g) * k ** -0.5).to(torch.bfloat16).cuda()
    out = torch.full((total + 7, n // 2 if epilogue else n), 3.0, dtype=torch.bfloat16, device="cuda")
    got = txr.gemm.grouped_matmul(rows, w, torch.tensor(counts, dtype=torch.int64, device="cuda"), epilogue=epilogue, out=out)
    want = txr.gemm.grouped_matmul_ref(rows, w, torch.tensor(counts), epilogue)
    # one rounding to bf16 of a value of order one
    assert torch.allclose(got[:total].float(), want[:total], rtol=2.0 ** -7, atol=2.0 ** -7)
    assert (got[total:] == 3.0).all()


@pytest.mark.parametrize("m,n,k", [(260, 264, 128 * 65), (130, 256, 128 * 130), (4100, 5128, 128), (1300, 7176, 128 * 3), (100, 256, 128 * 260)])
def test_matmul_fp8_block_scales_in_segments(txr, m, n, k):
    """More blocks of K than a CTA holds scales for, one block only, several tiles per CTA (the next tile's scales are fetched while
    one is stored), more blocks than the weight's shared-memory table has places."""
    g = torch.Generator().manual_seed(k)
    a = torch.randn(m, k, generator=g).cuda() * (0.25 + 4.0 * torch.rand(m, 1, generator=g).cuda())
    a *= (0.5 + torch.rand(1, k // 128, generator=g).cuda()).repeat_interleave(128, dim=1)
    w = torch.randn(n, k, generator=g).cuda() * (0.2 + torch.rand((n + 127) // 128, k // 128, generator=g).cuda()).repeat_interleave(
        128, dim=0)[:n].repeat_interleave(128, dim=1)
    qa, sa = txr.quant.fp8_quant_1x128(a.to(torch.bfloat16))
    qw, sw = txr.gemm.quantize_weight_128x128(w)
    da = (qa.double().view(m, -1, 128) * sa.double()[:, :, None]).view(m, k)
    dw = qw.double() * sw.double().repeat_interleave(128, dim=0)[:n].repeat_interleave(128, dim=1)
    want = da @ dw.t()
    got = txr.gemm.matmul_fp8_block(qa, sa, qw, sw).double()
    # fp32 sums of k products of fp8 values, one rounding to bf16
    bound = want.abs() * 2.0 ** -8 + (da.abs() @ dw.abs().t()) * k * 2.0 ** -24
    assert ((got - want).abs() <= bound).all()


def _exact_block_operands(rows, n, k, seed):
    """Small whole numbers with scales that are powers of two from 2^-2 to 2^2, so that every sum is exact: products are multiples of
    2^-4, and sums of them that stay below 2^20 (_exact_block_product asserts it) fit 24 bits.  Neighbouring blocks have different scales."""
    g = torch.Generator().manual_seed(seed)
    kb, nb = k // 128, (n + 127) // 128
    qa = torch.randint(-2, 3, (rows, k), generator=g).float().to(torch.float8_e4m3fn).cuda()
    qw = torch.randint(-1, 2, (n, k), generator=g).float().to(torch.float8_e4m3fn).cuda()
    exponent = lambda r: (torch.randint(0, 5, (r, 1), generator=g) + torch.cumsum(torch.randint(1, 5, (r, kb), generator=g), 1)) % 5 - 2      # noqa: E731
    return qa, torch.exp2(exponent(rows).float()).cuda(), qw, torch.exp2(exponent(nb).float()).cuda()


def _exact_block_product(qa, sa, qw, sw):
    """The product in 64 bits, checked to be one that 32-bit sums give exactly in any order."""
    rows, k = qa.shape
    da = (qa.double().view(rows, -1, 128) * sa.double()[:, :, None]).view(rows, k)
    dw = qw.double() * sw.double().repeat_interleave(128, dim=0)[:qw.shape[0]].repeat_interleave(128, dim=1)
    want = da @ dw.t()
    assert (da.abs() @ dw.abs().t()).max() < 2.0 ** 20 and torch.equal(want * 16, (want * 16).round())
    return want


@pytest.mark.parametrize("m,n,k", [(260, 264, 128 * 65), (130, 256, 128 * 130), (4100, 5128, 128), (1300, 7176, 128 * 3), (100, 256, 128 * 260)])
def test_matmul_fp8_block_scales_exactly(txr, m, n, k):
    """The sizes of the test above with operands whose product is exact: one wrong scale of one block of K shows."""
    ops = _exact_block_operands(m, n, k, k + m)
    assert torch.equal(txr.gemm.matmul_fp8_block(*ops), _exact_block_product(*ops).to(torch.bfloat16))


@pytest.mark.parametrize("ranks,shard_rows,n,k", [(4, 256, 2568, 128 * 68), (2, 512, 2824, 512), (2, 256, 136, 128 * 132)])
def test_all_gather_matmul_fp8_block_exactly(txr, ranks, shard_rows, n, k):
    """Several tiles per CTA pair, own and peers' in turn (the next tile's scales are fetched ahead for own rows only), and more blocks of K than
    a CTA holds scales for, with operands whose product is exact."""
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    try:
        ops = [_exact_block_operands(shard_rows, n, k, 90 + r) for r in range(ranks)]
        a_staging = world.symm_empty((ranks * shard_rows, k), torch.float8_e4m3fn)
        s_staging = world.symm_empty((ranks * shard_rows, k // 128), torch.float32)
        qa, sa = torch.cat([o[0] for o in ops]), torch.cat([o[1] for o in ops])
        for _ in range(2):
            outs = world.run(lambda c, r: txr.gemm.all_gather_matmul_fp8_block(c, ops[r][0], ops[r][1], a_staging[r], s_staging[r], ops[r][2], ops[r][3]))
            world.check()
            for r in range(ranks):
                assert torch.equal(outs[r], _exact_block_product(qa, sa, ops[r][2], ops[r][3]).to(torch.bfloat16))
                assert torch.equal(a_staging[r].view(torch.uint8), qa.view(torch.uint8)) and torch.equal(s_staging[r], sa)
    finally:
        world.destroy()


@pytest.mark.parametrize("rows,n,k,ctas", [(256, 136, 512, None), (512, 2568, 1536, None), (1280, 5128, 512, None), (512, 520, 1536, "3")])
def test_all_gather_matmul_fp8_block_on_one_rank(txr, port, monkeypatch, rows, n, k, ctas):
    """A rank without peers: the product of its own rows, exactly, and all rows and scales in the staging buffers; then of rows that are there already."""
    if ctas is not None:
        monkeypatch.setenv("TILEXR_GEMM_CTAS", ctas)
    comm = txr.init_process(0, 1, comm_id=f"127.0.0.1:{port}", buffer_mb=64, device=0)
    try:
        qa, sa, qw, sw = _exact_block_operands(rows, n, k, rows + n)
        want = _exact_block_product(qa, sa, qw, sw).to(torch.bfloat16)
        a_staging, s_staging = comm.symm_empty((rows, k), torch.float8_e4m3fn), comm.symm_empty((rows, k // 128), torch.float32)
        for a, s in ((qa, sa), (a_staging, s_staging)):
            got = txr.gemm.all_gather_matmul_fp8_block(comm, a, s, a_staging, s_staging, qw, sw)
            assert torch.equal(got, want)
            assert torch.equal(a_staging.view(torch.uint8), qa.view(torch.uint8)) and torch.equal(s_staging, sa)
        if k % 512 == 0:
            off = comm.symm_empty((rows * (k // 128) + 4,), torch.float32)[1:1 + rows * (k // 128)].view(rows, k // 128)
            with pytest.raises(RuntimeError):                  # the scales travel in 16-byte pieces
                txr.gemm.all_gather_matmul_fp8_block(comm, qa, sa, a_staging, off, qw, sw)
        assert comm.device_status() == 0
    finally:
        comm.destroy()


@pytest.mark.parametrize("ranks,shard_rows,n,k", [(4, 256, 2568, 128 * 65), (2, 512, 2824, 128), (2, 256, 136, 128 * 129)])
def test_matmul_reduce_scatter_fp8_block_exactly(txr, ranks, shard_rows, n, k):
    """Several tiles per CTA pair (a tile's staging shares its memory with the next tile's scales) and more blocks of K than a CTA holds
    scales for, with operands whose partial products are exact."""
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    try:
        m = ranks * shard_rows
        ops = [_exact_block_operands(m, n, k, 110 + r) for r in range(ranks)]
        staging = world.symm_empty((m, n), torch.bfloat16)
        want = sum(_exact_block_product(*o).to(torch.bfloat16).float() for o in ops)        # in rank order, as the owner adds them
        for _ in range(2):
            outs = world.run(lambda c, r: txr.gemm.matmul_reduce_scatter_fp8_block(c, ops[r][0], ops[r][1], ops[r][2], ops[r][3], staging[r]))
            world.check()
            for r in range(ranks):
                assert torch.equal(outs[r], want[r * shard_rows:(r + 1) * shard_rows].to(torch.bfloat16))
    finally:
        world.destroy()


def test_matmul_few_rows_under_the_switches_of_the_other_kernels(txr, monkeypatch):
    """TILEXR_GEMM_PAIR=0 asks for the one-CTA kernel, whose sums run over K in one piece; a cap on the CTAs leaves the result as it is."""
    g = torch.Generator().manual_seed(2)
    a = torch.randn(17, 2048, generator=g).to(torch.bfloat16).cuda()
    b = (torch.randn(7168, 2048, generator=g) / 45).to(torch.bfloat16).cuda()
    w = (torch.randn(6, 512, 2048, generator=g) / 45).to(torch.bfloat16).cuda()
    counts = torch.tensor([3, 0, 9, 1, 0, 4], dtype=torch.int64, device="cuda")
    with monkeypatch.context() as env:
        env.setenv("TILEXR_GEMM_SKINNY", "0")
        one_piece = txr.gemm.matmul(a, b)
        env.delenv("TILEXR_GEMM_SKINNY")
        env.setenv("TILEXR_GEMM_PAIR", "0")
        assert torch.equal(txr.gemm.matmul(a, b), one_piece)
    want, grouped = a.double() @ b.double().t(), txr.gemm.grouped_matmul(a, w, counts)
    bound = want.abs() * 2.0 ** -8 + (a.double().abs() @ b.double().abs().t()) * 2048 * 2.0 ** -24
    for ctas in ("1", "7", "64"):
        monkeypatch.setenv("TILEXR_GEMM_CTAS", ctas)
        assert ((txr.gemm.matmul(a, b).double() - want).abs() <= bound).all()
        assert torch.equal(txr.gemm.grouped_matmul(a, w, counts), grouped)        # never split: the cap changes no order of sums


def _small_ints(g, *shape, dtype=torch.bfloat16):
    return torch.randint(-2, 3, shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("m", [129, 160, 161, 255, 256, 257, 288, 289, 384, 385, 479, 481, 511, 513])
@pytest.mark.parametrize("n,k", [(8, 64), (264, 200), (512, 328), (4104, 136)])
def test_matmul_of_partial_tiles_exactly(txr, m, n, k):
    """Row and column blocks that are not full: the operand with less left becomes the instruction's N, in steps of 32.  Small whole
    numbers (|sum| <= 4 k, exact in fp32), so the only rounding is the one of the output."""
    g = torch.Generator(device="cuda").manual_seed(m + n)
    a, b = _small_ints(g, m, k), _small_ints(g, n, k)
    want = (a.double() @ b.double().t()).to(torch.bfloat16)
    assert torch.equal(txr.gemm.matmul(a, b), want)
    assert torch.equal(txr.gemm.matmul(a.half(), b.half()), (a.double() @ b.double().t()).half())
    if k % 16 == 0:
        f8 = torch.float8_e4m3fn
        assert torch.equal(txr.gemm.matmul_fp8(a.to(f8), b.to(f8), 1.0), want)


@pytest.mark.parametrize("m,n", [(1160, 19208), (1249, 9480)])
def test_matmul_of_partial_tiles_in_many_waves(txr, m, n):
    """More than four tiles per CTA pair: row blocks of more than 128 rows are computed as C^T, too."""
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = _small_ints(g, m, 72), _small_ints(g, n, 72)
    assert torch.equal(txr.gemm.matmul(a, b), (a.double() @ b.double().t()).to(torch.bfloat16))


@pytest.mark.parametrize("epilogue", [0, 1])
@pytest.mark.parametrize("n,k,counts", [(272, 136, [257, 0, 33, 512, 200, 1, 480]), (512, 64, [300, 31, 32, 225, 224]), (16, 72, [129, 600]),
                                        (9488, 64, [700, 0, 161, 400, 224, 225, 96])])
def test_grouped_matmul_of_partial_tiles(txr, n, k, counts, epilogue):
    """Groups that end inside a row block, computed as C^T where fewer rows than columns are left; rows behind the last group stay."""
    g = torch.Generator(device="cuda").manual_seed(n + k)
    total = sum(counts)
    rows, w = _small_ints(g, total + 3, k), _small_ints(g, len(counts), n, k)
    nums = torch.tensor(counts, dtype=torch.int64, device="cuda")
    out = torch.full((total + 3, n // 2 if epilogue else n), 7.0, dtype=torch.bfloat16, device="cuda")
    got = txr.gemm.grouped_matmul(rows, w, nums, epilogue, out)
    prod = torch.cat([r.double() @ w[i].double().t() for i, r in enumerate(rows[:total].split(counts))])
    if epilogue == 0:
        assert torch.equal(got[:total], prod.to(torch.bfloat16))
    else:
        want = torch.nn.functional.silu(prod[:, 0::2]) * prod[:, 1::2]
        # one rounding to bf16 (2^-9) of an fp32 value whose exponential and division are a few ulp of fp32 off
        assert torch.allclose(got[:total].double(), want, rtol=2 ** -8, atol=1e-6)
    assert torch.equal(got[total:], torch.full_like(got[total:], 7.0))


@pytest.mark.parametrize("m,n,k", [(300, 9480, 256), (6401, 776, 128 * 29), (100, 7176, 384), (257, 2184, 128 * 57)])
def test_matmul_fp8_block_slices_exactly(txr, m, n, k):
    """One tile or two behind a wave of whole ones (slices of 32 columns, the last of them past N), and few tiles altogether (slices of
    128 and of 64 columns)."""
    ops = _exact_block_operands(m, n, k, k + m)
    assert torch.equal(txr.gemm.matmul_fp8_block(*ops), _exact_block_product(*ops).to(torch.bfloat16))


def test_staging_buffers_off_the_16_byte_grid(txr):
    """Partial tiles travel in 16-byte pieces: refused on the host, before a launch."""
    rows, n, k, ranks = 256, 136, 512, 2
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    try:
        a, b = torch.zeros(ranks * rows, k, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, k, dtype=torch.bfloat16, device="cuda")
        qa, sa, qw, sw = _exact_block_operands(ranks * rows, n, k, 1)
        stagings = [s[1:1 + ranks * rows * n].view(ranks * rows, n) for s in world.symm_empty((ranks * rows * n + 8,), torch.bfloat16)]
        with pytest.raises(RuntimeError):
            world.run(lambda c, r: txr.gemm.matmul_reduce_scatter(c, a, b, stagings[r]))
        with pytest.raises(RuntimeError):
            world.run(lambda c, r: txr.gemm.matmul_reduce_scatter_fp8_block(c, qa, sa, qw, sw, stagings[r]))
        world.check()
    finally:
        world.destroy()
