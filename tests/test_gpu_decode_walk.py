"""Decode attention in launches whose blocks walk several (row, chunk, kv head) items: the same bits as the kernel with a block per
possible chunk, for rows counted from their positions (up to 256) and more, with chunks that no row reaches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,chunks", [(70, 12), (256, 4), (257, 4), (300, 3)])
@pytest.mark.parametrize("hd,P,window", [(64, 64, None), (64, 8, 300), (128, 32, None)])
def test_walk(M, chunks, hd, P, window):
    from snowllm_b200.ops import kernels
    nh, nkv = 32, 8
    gen = torch.Generator().manual_seed(M + hd)
    longest = (chunks - 1) * 256                         # the last chunk is reached by nobody
    positions = torch.randint(0, longest, (M,), generator=gen)
    positions[:5] = torch.tensor([0, longest - 1, 255, 256, 1])
    width = -(-longest // P)
    pages = 3 * width + 1
    table = torch.stack([torch.randperm(pages, generator=gen)[:width] for _ in range(M)]).to(torch.int32).cuda()
    pool = torch.randn(pages, 2, nkv, P, hd, device="cuda").to(torch.bfloat16)
    q = torch.randn(M + 4, nh, hd, device="cuda").to(torch.bfloat16)
    rows = (torch.randperm(M + 4, generator=gen)[:M]).to(torch.int32).cuda()
    at = torch.zeros(M + 4, dtype=torch.int32)
    seg = torch.zeros(M + 4, dtype=torch.int32)
    at[rows.cpu().long()] = positions.to(torch.int32)
    seg[rows.cpu().long()] = torch.arange(M, dtype=torch.int32)
    outs = []
    for tma in (True, False):
        out = torch.full((M + 4, nh * hd), 7.0, device="cuda").to(torch.bfloat16)
        kernels.attention_decode_mma(q, pool, table, P, at.cuda(), seg.cuda(), hd ** -0.5, chunks, out, window=window,
                                     rows=rows, tma=tma)
        outs.append(out)
    assert torch.equal(*outs)
    assert kernels.attention_decode_status() == 0
    served = torch.zeros(M + 4, dtype=torch.bool)
    served[rows.cpu().long()] = True
    assert (outs[0][~served.cuda()] == 7).all() and outs[0].isfinite().all()


# the line from which a launch walks (32 chunks a row, 16 rounds of possible blocks, up to 256 rows of head size 64), its sides, and
# rows with and without a window; some rows reach one chunk, some nearly all, the last chunk nobody
@pytest.mark.parametrize("M,chunks", [(27, 32), (28, 32), (64, 31), (64, 33), (256, 32), (257, 32)])
@pytest.mark.parametrize("P,window", [(64, None), (8, 300), (256, None)])
def test_walk_at_its_line(M, chunks, P, window):
    test_walk(M, chunks, 64, P, window)
