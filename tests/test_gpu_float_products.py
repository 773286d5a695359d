"""float32 products at the edges of their kernels (chunks of 128 columns, strips of 16, passes of 2 to 16 rows; tiles of 32 to
128): every output is one thread's sum in order of k, so few rows and many come to the same bits."""
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
