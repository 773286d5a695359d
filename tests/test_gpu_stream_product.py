"""The few-rows products: the one that streams W through shared memory, at the edges of its boxes (512 columns), strips (16
rows of W) and passes (8 and 16 rows), against a double-precision product and the kernel without a ring; its bounded waits;
and grouped products with fewer rows than groups, whose blocks look up the groups that own any."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(*shape, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=gen).to(torch.bfloat16)


def slack_of(K):
    """What a float sum of K products of N(0, 1) values may be off by: the sum takes a step per MMA of 16 columns and
    then 16 more (warps, halves), each rounding (or cutting off) 2^-23 of a partial sum of at most about 2 sqrt(K)."""
    return 2.0 ** -23 * (K / 16 + 16) * 2 * K ** 0.5


def off(got, want, K):
    """The largest error over that slack and, for bfloat16 outputs, one rounding of the result."""
    slack = slack_of(K) + (2.0 ** -8 * want.abs() if got.dtype == torch.bfloat16 else 0)
    return float(((got.double() - want).abs() / slack).max())


# K: less than a block (the kernel without a ring), a block, a part of a box, a box, a box and a block, an odd number of
# boxes of a split sum, a deep one
@pytest.mark.parametrize("K", [32, 64, 448, 512, 576, 2048, 2624, 10752])
@pytest.mark.parametrize("M,N", [(1, 16), (8, 17), (9, 200), (16, 2368), (3, 2384), (5, 40)])
def test_plain(M, N, K):
    from snowllm_b200.ops import kernels
    a, w = operands(M, K, seed=1), operands(N, K, seed=2)
    want = a.double() @ w.double().T
    out = kernels.gemm_skinny(a, w, out_dtype=torch.float32)
    assert off(out, want, K) <= 1
    assert off(kernels.gemm_skinny(a, w), want, K) <= 1
    # the kernel without a ring (which takes the rows by a list) comes to the same bits, in one pass and in several
    rows = torch.arange(M, dtype=torch.int32, device="cuda")
    for hint in (8, 64):
        other = kernels.gemm_skinny(a, w, out_dtype=torch.float32, a_rows=rows, rows_hint=hint)
        assert torch.equal(other, out)


@pytest.mark.parametrize("counts", [[1] * 5, [0, 0, 3, 0], [17, 0, 8, 9, 1], [0] * 40 + [2] + [0] * 30 + [33], [16]])
@pytest.mark.parametrize("N,K", [(48, 128), (256, 1792)])
def test_grouped(counts, N, K):
    from snowllm_b200.ops import kernels
    G, M = len(counts), sum(counts)
    x, w = operands(2 * M + 1, K, seed=3), operands(G, N, K, seed=4)
    rows = torch.randperm(2 * M, generator=torch.Generator().manual_seed(5))[:M].to(torch.int32).cuda()
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    for hint in (8, 16):
        out = kernels.gemm_skinny(x, w, out_dtype=torch.float32, a_rows=rows, a_div=2, offsets=offsets, rows_out=M,
                                  rows_hint=hint)
        glu = kernels.gemm_skinny(x, w, a_rows=rows, a_div=2, offsets=offsets, rows_out=M, rows_hint=hint, swiglu=1)
        lo = 0
        for e, n in enumerate(counts):
            if n:
                want = x[(rows[lo:lo + n] // 2).long()].double() @ w[e].double().T
                assert off(out[lo:lo + n], want, K) <= 1
                gate, up = want.view(n, N // 16, 2, 8).unbind(2)
                ref = (gate * torch.sigmoid(gate) * up).reshape(n, N // 2)
                # one rounding, and the float sums' error through the gate (its slope is at most 1.1) and the product
                slack = 2.0 ** -8 * ref.abs() + slack_of(K) * (1.1 * up.abs() + gate.abs() + 1).reshape(n, N // 2)
                assert ((glu[lo:lo + n].double() - ref).abs() <= slack).all()
            lo += n


def test_wait_that_runs_out():
    from snowllm_b200.errors import KernelError
    from snowllm_b200.ops import kernels
    a, w = operands(4, 1024, seed=6), operands(4096, 1024, seed=7)
    good = kernels.gemm_skinny(a, w)
    watch = kernels.StatusWatch()
    kernels.lose_loads(True)
    try:
        kernels.gemm_skinny(a, w)
        watch.peek()
        torch.cuda.synchronize()
    finally:
        kernels.lose_loads(False)
    with pytest.raises(KernelError, match="bounded wait ran out.*gemm_skinny"):
        watch.check()
    assert kernels.gemm_skinny_status() == 0
    assert torch.equal(kernels.gemm_skinny(a, w), good)


def test_a_block_that_gave_up_stays_until_its_copies_have_landed():
    """At most two boxes a block, fewer than stages: the producer is gone when the multiplying warps' wait runs out, and
    they give the copies on their way their 200 us themselves.  The launch takes the wait and those."""
    from snowllm_b200.ops import kernels
    a, w = operands(4, 1024, seed=8), operands(16 * 100, 1024, seed=9)
    kernels.gemm_skinny(a, w)
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    kernels.lose_loads(True)
    try:
        begin.record()
        kernels.gemm_skinny(a, w)
        end.record()
        torch.cuda.synchronize()
    finally:
        kernels.lose_loads(False)
    assert kernels.gemm_skinny_status() == 1
    assert begin.elapsed_time(end) >= 1500 + 0.2


def test_a_slow_kernel_in_front_is_not_a_wait_that_ran_out():
    """The kernel in front takes longer than a wait may: 1.5 s and the time it gives its copies (a tcgen05 product whose
    loads are lost).  The rings of the product behind it are full all the while, and its own waits begin after it."""
    from snowllm_b200.ops import kernels
    a, w = operands(4, 2048, seed=10), operands(16384, 2048, seed=11)      # 7 strips of 4 boxes a block
    x, v = operands(128, 64, seed=12), operands(128, 64, seed=13)
    good = kernels.gemm_skinny(a, w)
    kernels.gemm_tc(x, v)
    assert kernels.gemm_tc_status() == 0 and kernels.gemm_skinny_status() == 0
    lose = kernels.fn("snk_gemm_tc_test_lose_loads")
    lose(1)
    try:
        kernels.gemm_tc(x, v)
        out = kernels.gemm_skinny(a, w, w_ahead=True)
        torch.cuda.synchronize()
    finally:
        lose(0)
    assert kernels.gemm_tc_status() != 0
    assert kernels.gemm_skinny_status() == 0
    assert torch.equal(out, good)


@pytest.mark.parametrize("M,dtype", [(4, torch.bfloat16), (64, torch.bfloat16), (4, torch.float32)])
def test_w_may_come_from_the_kernel_in_front(M, dtype):
    """Without ``w_ahead``, products whose w the launch in front of them writes, replayed without a gap; the numbers of
    the same products launched one by one."""
    from snowllm_b200.ops import linear
    x, v = operands(M, 2048, seed=14).to(dtype), operands(2048, 64, seed=15).to(dtype)
    us = [operands(2048, 64, seed=16 + i).to(dtype) for i in range(4)]
    w = torch.zeros(2048, 2048, dtype=dtype, device="cuda")
    want = []
    for u in us:
        linear(u, v, out=w)
        torch.cuda.synchronize()
        want.append(linear(x, w))
        torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = []
        for u in us:
            linear(u, v, out=w)
            got.append(linear(x, w))
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


# one row tile and two; one sum a warp and four (K of 2,048 on, up to 2,368 rows of W); one to three rounds of strips;
# boxes that end in the middle, an odd number of them
@pytest.mark.parametrize("M,N,K", [(1, 16, 64), (3, 208, 576), (13, 1008, 576), (16, 200, 1088), (5, 2368, 2560), (12, 1776, 4096),
                                   (16, 2352, 2112), (9, 2384, 2048), (8, 4112, 1600), (16, 4752, 2112)])
def test_weights_read_ahead_and_stores_with_a_gate(M, N, K):
    """The streaming product, W read ahead or not, to float, to bfloat16, with a gate and with the square of relu at its
    store, inside an output that is full of NaN: the same bits as the kernel without a ring, nothing beside them."""
    from snowllm_b200.ops import kernels
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert kernels.fn("snk_gemm_skinny_streams")(M, N, K, sms)
    a, w = operands(M, K, seed=20), operands(N, K, seed=21)
    rows = torch.arange(M, dtype=torch.int32, device="cuda")
    stores = [dict(out_dtype=torch.float32), {}, dict(act=kernels.UNARY_CODES["relu2"])]
    stores += [dict(swiglu=code) for code in (1, 2, 3) if N % 16 == 0]
    for store in stores:
        want = kernels.gemm_skinny(a, w, a_rows=rows, **store)
        for ahead in (False, True):
            room = torch.full((want.numel() + 128,), float("nan"), dtype=want.dtype, device="cuda")
            out = room[64:-64].view(want.shape)
            kernels.gemm_skinny(a, w, out=out, w_ahead=ahead, **store)
            assert torch.equal(out, want)
            assert bool(room[:64].isnan().all()) and bool(room[-64:].isnan().all())
    assert kernels.gemm_skinny_status() == 0


@pytest.mark.parametrize("M,N,K", [(17, 64, 1024), (64, 2048, 2048), (130, 520, 200), (200, 6144, 576), (2050, 264, 1088)])
def test_tcgen05_product_with_its_weight_read_ahead(M, N, K):
    """Split along K and whole, one round of tiles and more, more and fewer k-blocks than the ring has stages."""
    from snowllm_b200.ops import kernels
    a, w = operands(M, K, seed=22), operands(N, K, seed=23)
    for store in (dict(out_dtype=torch.float32), {}, dict(swiglu=1)):
        if "swiglu" in store and N % 16:
            continue
        want = kernels.gemm_tc(a, w, **store)
        for _ in range(3):
            assert torch.equal(kernels.gemm_tc(a, w, w_ahead=True, **store), want)
    assert kernels.gemm_tc_status() == 0


@pytest.mark.parametrize("counts", [[0] * 40 + [2] + [0] * 30 + [33], [1] * 5 + [0] * 90, [0] * 99 + [7], [3, 0, 9] + [0] * 120])
def test_grouped_blocks_that_look_their_group_up(counts):
    """Fewer rows than groups and more blocks than the SMs hold at once: against each group's rows as a product of their own."""
    from snowllm_b200.ops import kernels
    G, M, N, K = len(counts), sum(counts), 1024, 256
    assert G > M and N // 16 * G > 8 * torch.cuda.get_device_properties(0).multi_processor_count
    x, w = operands(M, K, seed=24), operands(G, N, K, seed=25)
    offsets = torch.tensor([0] + counts).cumsum(0).to(torch.int32).cuda()
    for hint in (8, 16):
        out = kernels.gemm_skinny(x, w, out_dtype=torch.float32, offsets=offsets, rows_out=M, rows_hint=hint)
        lo = 0
        for e, n in enumerate(counts):
            if n:
                rows = torch.arange(n, dtype=torch.int32, device="cuda")
                assert torch.equal(out[lo:lo + n], kernels.gemm_skinny(x[lo:lo + n].contiguous(), w[e].contiguous(),
                                                                       out_dtype=torch.float32, rows_hint=hint, a_rows=rows))
            lo += n
