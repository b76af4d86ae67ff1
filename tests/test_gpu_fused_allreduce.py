"""All-reduce + residual add + RMSNorm in one kernel, one-shot and two-shot, against fp32 PyTorch."""
import pytest
import torch

from conftest import require_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def txr():
    require_cuda()
    import tilexr_b200

    return tilexr_b200


def _reference(xs, residual, gamma, eps):
    acc = xs[0].float()
    for x in xs[1:]:
        acc = acc + x.float()
    if residual is not None:
        acc = acc + residual.float()
    s = acc.to(xs[0].dtype)
    xf = s.float()
    y = (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * gamma.float()).to(xs[0].dtype)
    return y, s


@pytest.mark.parametrize("ranks,rows,h,algo,with_res,symmetric", [
    (2, 1, 8192, 1, True, False),
    (8, 16, 8192, 1, True, False),
    (4, 256, 4096, 1, False, False),
    (4, 64, 8192, 2, True, False),
    (8, 203, 2048, 2, True, False),       # rows do not divide by the rank count
    (4, 128, 8192, 2, True, True),        # peers write y and the residual directly
    (8, 37, 1024, 0, True, False),
    (8, 1, 2048, 2, True, False),         # two-shot with fewer rows than ranks: most ranks own nothing
    (8, 3, 1024, 2, True, True),
])
def test_all_reduce_rmsnorm(txr, ranks, rows, h, algo, with_res, symmetric):
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=64)
    g = torch.Generator().manual_seed(5)
    xs = [torch.randn(rows, h, generator=g).to(torch.bfloat16) for _ in range(ranks)]
    res = torch.randn(rows, h, generator=g).to(torch.bfloat16) if with_res else None
    gamma = (1 + 0.1 * torch.randn(h, generator=g)).to(torch.bfloat16)
    want_y, want_res = _reference(xs, res, gamma, 1e-6)
    xd = [x.cuda() for x in xs]
    gd = gamma.cuda()
    for rep in range(2):
        if symmetric:
            ys = world.symm_empty((rows, h), torch.bfloat16)
            rd = world.symm_empty((rows, h), torch.bfloat16)
            for r in rd:
                r.copy_(res)
        else:
            ys = [None] * ranks
            rd = [res.cuda() if with_res else None for _ in range(ranks)]
        out = world.run(lambda c, r: txr.collectives.all_reduce_rmsnorm(c, xd[r], gd, 1e-6, residual=rd[r], algo=algo, out=ys[r]))
        world.check()
        for r in range(ranks):
            if with_res:
                assert torch.equal(rd[r].cpu(), want_res), f"rank {r} residual"
            got = out[r].cpu().float()
            assert torch.allclose(got, want_y.float(), rtol=2e-2, atol=2e-2)
            assert torch.equal(out[r].cpu(), out[0].cpu())       # bit-identical on every rank
    world.destroy()


def test_choice_by_size(txr):
    assert txr._C.all_reduce_rmsnorm_choose(16 * 1024, 8) == 1
    assert txr._C.all_reduce_rmsnorm_choose(4 << 20, 8) == 2
    assert txr._C.all_reduce_rmsnorm_choose(4 << 20, 2) == 1


@pytest.mark.parametrize("ranks,rows,h,algo,with_res,symmetric", [
    (4, 2000, 264, 2, True, False),       # several groups of rows per block in every phase, the last one ragged
    (3, 1501, 1032, 2, True, True),
    (2, 700, 9000, 1, False, False),      # rows longer than two 16-byte columns per thread
])
def test_all_reduce_rmsnorm_groups_of_rows(txr, ranks, rows, h, algo, with_res, symmetric):
    test_all_reduce_rmsnorm(txr, ranks, rows, h, algo, with_res, symmetric)


@pytest.mark.parametrize("ranks,rows,h,algo,with_res,symmetric", [
    (2, 9, 8192, 2, False, False),        # the longest rows for two 16-byte columns per thread: all of them used (a grid this small takes the other kernel)
    (2, 9, 8200, 2, True, False),         # the shortest with a third
    (3, 26, 4104, 1, True, False),        # one thread has a second column; an odd row after whole pairs
])
def test_all_reduce_rmsnorm_around_two_columns_per_thread(txr, ranks, rows, h, algo, with_res, symmetric):
    test_all_reduce_rmsnorm(txr, ranks, rows, h, algo, with_res, symmetric)


def test_emulated_world_of_more_ranks_than_travel_with_a_launch():
    """Argument blocks of more ranks than fit the launch's parameters come as a device array."""
    require_cuda()
    import tilexr_b200 as txr
    from tilexr_b200.ops import collectives

    ranks, rows, h = 9, 5, 64
    world = txr.init_emulated_world(ranks, device=0, buffer_mb=16)
    try:
        g = torch.Generator().manual_seed(3)
        xs = [torch.randn(rows, h, generator=g).to(torch.bfloat16).cuda() for _ in range(ranks)]
        gamma = torch.ones(h, dtype=torch.bfloat16, device="cuda")
        for _ in range(3):
            ys = world.run(lambda c, r: collectives.all_reduce_rmsnorm(c, xs[r], gamma))
            world.check()
        total = sum(x.float() for x in xs).to(torch.bfloat16).float()
        want = total * torch.rsqrt(total.square().mean(dim=1, keepdim=True) + 1e-6)
        for y in ys:
            # one rounding to bf16 of an fp32 product whose reciprocal root is a few ulp of fp32 off
            assert torch.allclose(y.float(), want, rtol=2 ** -7, atol=2 ** -7) and torch.equal(y, ys[0])
    finally:
        world.destroy()


@pytest.mark.parametrize("ranks,rows,h,algo,with_res,symmetric", [
    (2, 75, 8192, 1, True, False),        # one row more than there are places with one block to an SM: the form with two, all its columns used
    (2, 74, 8192, 1, True, False),        # the last grid of the other
    (3, 51, 4104, 2, True, True),         # 49 blocks per rank fit one to an SM; one thread has a second column
    (2, 160, 8200, 1, False, False),      # too long for two columns per thread, whatever the grid
])
def test_all_reduce_rmsnorm_around_one_block_per_sm(txr, ranks, rows, h, algo, with_res, symmetric):
    test_all_reduce_rmsnorm(txr, ranks, rows, h, algo, with_res, symmetric)


@pytest.mark.parametrize("blocks", ["1", "9", "100"])
def test_all_reduce_rmsnorm_under_the_switch(txr, monkeypatch, blocks):
    monkeypatch.setenv("TILEXR_AR_NORM_BLOCKS", blocks)
    test_all_reduce_rmsnorm(txr, 2, 130, 2048, 1, True, False)
