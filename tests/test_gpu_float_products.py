"""float32 products at the edges of their kernels (chunks of 128 columns, strips of 16, passes of 2 to 16 rows; each of the four
tiles with ragged edges): every output is one thread's sum in order of k, so few rows and many come to the same bits, and so do
bfloat16 operands and the same values in float32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(*shape, seed=0):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


@pytest.mark.parametrize("K", [4, 128, 132, 644, 2048])
@pytest.mark.parametrize("N", [1, 17, 200])
def test_few_rows_and_many(N, K):
    from snowllm_b200.ops import kernels
    a, w = operands(200, K, seed=1), operands(N, K, seed=2)
    many = kernels.gemm_simt(a, w)
    want = a.double() @ w.double().T
    # K roundings of 2^-24, each of a partial sum of at most about 4 sqrt(K)
    assert float((many.double() - want).abs().max()) <= 2.0 ** -24 * K * 4 * K ** 0.5
    for M in (1, 2, 3, 5, 9, 16, 17, 40, 129):
        assert torch.equal(kernels.gemm_simt(a[:M].contiguous(), w), many[:M])
        assert torch.equal(kernels.gemm_simt(a[:M].contiguous(), w, w_ahead=True), many[:M])


@pytest.mark.parametrize("counts", [[1] * 5, [0, 0, 3, 0], [17, 0, 1, 0, 0, 0], [40, 9, 70]])
def test_groups(counts):
    from snowllm_b200.ops import kernels
    G, M, N, K = len(counts), sum(counts), 56, 260
    x, w = operands(2 * M + 1, K, seed=3), operands(G, N, K, seed=4)
    rows = torch.randperm(2 * M, generator=torch.Generator().manual_seed(5))[:M].to(torch.int32).cuda()
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    out = kernels.gemm_simt(x, w, a_rows=rows, a_div=2, offsets=offsets, rows_out=M, max_rows_per_group=M)
    lo = 0
    for e, n in enumerate(counts):
        if n:
            assert torch.equal(out[lo:lo + n], kernels.gemm_simt(x[(rows[lo:lo + n] // 2).long()].contiguous(), w[e]))
        lo += n


# Fewer rows than groups, and more strips of 16 columns over all groups than the SMs hold blocks (five each): a block looks the group
# up that its number stands for (up to 15 rows to 16 groups).  One group of 32 and several of them; empty ones first, last and between; rows in
# one group alone; 30 rows of 32 groups are the last to be looked up, 31 have a block per group.
@pytest.mark.parametrize("N,counts", [
    (3584, [0, 1, 0, 2] * 3 + [0] * 20), (3584, [0] * 31 + [1]), (3584, [1] + [0] * 31), (3584, [0] * 31 + [31]),
    (3584, [1] * 31 + [0]), (3584, [0] + [1] * 30 + [0]), (3584, [0, 17] + [0] * 29 + [9]), (384, [0, 1] * 16),
    (260, [0] * 33 + [1, 0, 3] + [0] * 33 + [2]), (260, [0] * 69 + [1]), (112, [(e % 5 == 3) * (1 + e % 3) for e in range(128)])])
@pytest.mark.parametrize("K", [64, 260])
def test_fewer_rows_than_groups(N, counts, K):
    from snowllm_b200.ops import kernels
    G, M = len(counts), sum(counts)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert M < G and -(-N // 16) * G > 5 * sms
    x, w = operands(M, K, seed=13), operands(G, N, K, seed=14)
    rows = torch.randperm(2 * M, generator=torch.Generator().manual_seed(15))[:M].to(torch.int32).cuda()
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    out = torch.full((M, N), float("nan"), device="cuda")
    kernels.gemm_simt(x, w, a_rows=rows, a_div=2, offsets=offsets, rows_out=M, max_rows_per_group=M, out=out)
    lo = 0
    for e, n in enumerate(counts):
        if n:
            assert torch.equal(out[lo:lo + n], kernels.gemm_simt(x[(rows[lo:lo + n] // 2).long()].contiguous(), w[e]))
        lo += n


def tile_of(M, N, groups, rows):
    from snowllm_b200.ops import kernels
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return kernels.fn("snk_gemm_simt_tile")(M, N, groups, rows, sms)


# tiles 128 x 128, 64 x 128, 64 x 64 and 32 x 64; K in vectors of four, odd (element by element), less than a step of 16
@pytest.mark.parametrize("K", [12, 132, 645])
@pytest.mark.parametrize("M,N,tile", [(300, 6147, 0), (1000, 1999, 0), (509, 2050, 1), (130, 4099, 1), (200, 2049, 2),
                                      (1100, 2051, 2), (33, 130, 3)])
def test_every_tile_at_its_edges(M, N, tile, K):
    from snowllm_b200.ops import kernels
    assert tile_of(M, N, 0, M) == tile
    a, w = operands(M, K, seed=6).to(torch.bfloat16), operands(N, K, seed=7).to(torch.bfloat16)
    out = kernels.gemm_simt(a.float(), w.float())
    want = a.double() @ w.double().T
    assert float((out.double() - want).abs().max()) <= 2.0 ** -24 * K * 4 * K ** 0.5
    for lo in (0, M // 2, M - 16):                     # the few-rows kernel (K a multiple of 4) or a lower tile
        assert torch.equal(kernels.gemm_simt(a[lo:lo + 16].float(), w.float()), out[lo:lo + 16])
    assert torch.equal(kernels.gemm_simt(a, w, out_dtype=torch.float32), out)
    assert torch.equal(kernels.gemm_simt(a, w), out.to(torch.bfloat16))


@pytest.mark.parametrize("N,tile", [(2051, 0), (1027, 1), (515, 2)])
def test_groups_on_the_larger_tiles(N, tile):
    from snowllm_b200.ops import kernels
    counts, K = [300, 0, 517, 129], 132
    G, M = len(counts), sum(counts)
    assert tile_of(M, N, G, M) == tile
    x, w = operands(M, K, seed=8), operands(G, N, K, seed=9)
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    out = kernels.gemm_simt(x, w, offsets=offsets, rows_out=M, max_rows_per_group=M)
    lo = 0
    for e, n in enumerate(counts):
        if n:
            assert torch.equal(out[lo:lo + n], kernels.gemm_simt(x[lo:lo + n], w[e]))
        lo += n
