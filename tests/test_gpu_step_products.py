"""What the streaming few-rows product does beside multiplying in a step of one-token rows: the gated short convolution at its
store, and the RMS norm in front of it, at the edges of units (16 channels), row shares (1 and 2 rows) and taps."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def draw(*shape, seed, scale=1.0, dtype=BF):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(dtype)


def conv_operands(M, H, K, L, seed=0):
    weight, state = draw(H, L, seed=seed + 2, scale=0.3), draw(M + 3, L - 1, H, seed=seed + 3)
    start = torch.tensor([0 if m % 3 == 1 else 5 + m for m in range(M)], dtype=torch.int32, device="cuda")
    slot = torch.randperm(M + 3, generator=torch.Generator().manual_seed(seed))[:M].to(torch.int32).cuda()
    return draw(3 * H, K, seed=seed + 1, scale=0.02), weight, state, start, slot


def conv_plain(bcx, weight, state, start, slot):
    from snowllm_b200.ops import kernels
    M = bcx.shape[0]
    cu = torch.arange(M + 1, dtype=torch.int32, device="cuda")
    return kernels.short_conv(bcx, weight, state, cu, start, slot, cu[:M])


# one unit per block at the most (2,368 channels) and fewer units than SMs; K of whole and of partial boxes of 512 columns
@pytest.mark.parametrize("H,K", [(2048, 2048), (2368, 2048), (1600, 2624)])
@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("L", [2, 3, 4])
def test_conv_at_the_store(M, H, K, L):
    from snowllm_b200.ops import kernels
    w, weight, state, start, slot = conv_operands(M, H, K, L)
    x, other = draw(M, K, seed=9), state.clone()
    if not kernels.conv_step_ok(x, w, weight, M, M):
        pytest.skip("not a size for this device")
    y = kernels.conv_step(x, w, weight, state, start, slot)
    assert torch.equal(y, conv_plain(kernels.gemm_skinny(x, w), weight, other, start, slot))
    assert torch.equal(state, other)


def test_conv_sizes_refused():
    from snowllm_b200.ops import kernels
    ok = kernels.fn("snk_conv_step_ok")
    assert not any(ok(*s) for s in [(3, 2048, 2048, 3), (0, 2048, 2048, 3), (1, 2048, 2048, 5), (1, 2048, 2048, 1),
                                    (1, 2040, 2048, 3), (1, 2048, 2040, 3), (1, 2048, 512, 3)])


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(2384, 64), (3072, 2048), (6144, 2048), (16384, 1024), (4096, 2624)])
@pytest.mark.parametrize("pieces", [0, 1, 4])
def test_norm_in_front(M, N, K, pieces):
    from snowllm_b200.ops import kernels
    residual, gamma, w = draw(M, K, seed=1, dtype=torch.float32), draw(K, seed=2), draw(N, K, seed=3, scale=0.05)
    delta = None
    if pieces == 1:
        delta = draw(M, K, seed=4, dtype=torch.float32)
    elif pieces:
        pos = torch.randperm(M * pieces, generator=torch.Generator().manual_seed(5)).to(torch.int32).cuda()
        delta = kernels.ExpertSum(draw(M * pieces, K, seed=6, dtype=torch.float32), pos,
                                  torch.rand(M, pieces, device="cuda"))
    if not kernels.PendingNorm.ok(residual, delta, gamma, BF, w):
        pytest.skip("not a size for this device")
    other = residual.clone()
    out = kernels.PendingNorm(residual, delta, gamma, 1e-5).product(w)
    kernels.add_rmsnorm(other, delta, gamma, 1e-5, BF)
    assert torch.equal(residual, other)
    r = residual.double()
    x = r * torch.rsqrt(r.square().mean(-1, keepdim=True) + 1e-5) * gamma.double()
    want = x @ w.double().T
    # every value of the norm is rounded to bfloat16 once (2^-9 of itself, twice that allowed), and so is the result
    bound = 2.0 ** -8 * (x.abs() @ w.double().abs().T) + 2.0 ** -8 * want.abs()
    assert ((out.double() - want).abs() <= bound).all()
    if N % 16 == 0:
        glu = kernels.PendingNorm(other.clone(), None, gamma, 1e-5).product(w, swiglu=1)
        gate, up = out.float().view(M, N // 16, 2, 8).unbind(2)
        ref = (torch.nn.functional.silu(gate.double()) * up.double()).reshape(M, N // 2)
        near = 2.0 ** -7 * (1.1 * gate.abs() * up.abs() + gate.abs() + up.abs()).reshape(M, N // 2) + 1e-6
        assert ((glu.double() - ref).abs() <= near).all()


@pytest.mark.parametrize("M,L", [(1, 3), (1, 4), (2, 3), (2, 2)])
def test_norm_and_conv(M, L):
    """Both at once: the same as the convolution of the product of the norm's own rows, whose bits the product forms again."""
    from snowllm_b200.ops import kernels
    H = K = 2048
    w, weight, state, start, slot = conv_operands(M, H, K, L, seed=20)
    residual, gamma = draw(M, K, seed=31, dtype=torch.float32), draw(K, seed=32)
    delta = draw(M, K, seed=33, dtype=torch.float32)
    pending = kernels.PendingNorm(residual, delta, gamma, 1e-5)
    if not (pending.ok(residual, delta, gamma, BF, w) and kernels.conv_step_ok(pending, w, weight, M, M)):
        pytest.skip("not a size for this device")
    other, plain_state = residual.clone(), state.clone()
    y = kernels.conv_step(pending, w, weight, state, start, slot)
    bcx = kernels.PendingNorm(other, delta, gamma, 1e-5).product(w)
    assert torch.equal(residual, other)
    assert torch.equal(y, conv_plain(bcx, weight, plain_state, start, slot))
    assert torch.equal(state, plain_state)


# Widths at which a thread of the product stands for one, two and four threads of the norm's kernel, whole and in part
@pytest.mark.parametrize("M,K", [(m, k) for m in (1, 2) for k in (64, 448, 512, 960, 1024, 2048)] + [(1, 2624), (1, 4096)])
@pytest.mark.parametrize("pieces", [0, 1, 3])
def test_norm_in_front_is_the_norms_own(M, K, pieces):
    """The rows of a norm that a product forms for itself are the norm's own kernel's, bit for bit: what a request's rows are does not
    depend on how many requests a step has."""
    from snowllm_b200.ops import kernels
    gamma = draw(K, seed=42)
    w = torch.eye(max(K, 2560), K, device="cuda", dtype=BF)                 # the product hands the norm's rows on as they are
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    for seed in range(100):                              # (another order of the sum shows in the last bit of one row in thirty)
        residual, delta = draw(M, K, seed=seed, scale=3.0, dtype=torch.float32), None
        if pieces == 1:
            delta = draw(M, K, seed=1000 + seed, dtype=torch.float32)
        elif pieces:
            pos = torch.randperm(M * pieces, generator=torch.Generator().manual_seed(seed)).to(torch.int32).cuda()
            delta = kernels.ExpertSum(draw(M * pieces, K, seed=2000 + seed, dtype=torch.float32), pos,
                                      draw(M, pieces, seed=3000 + seed, dtype=torch.float32))
        if not kernels.PendingNorm.ok(residual, delta, gamma, BF, w):
            pytest.skip("not a size for this device")
        other = residual.clone()
        out = kernels.PendingNorm(residual, delta, gamma, 1e-5).product(w)
        rows = kernels.add_rmsnorm(other, delta, gamma, 1e-5, BF)
        differ += (residual != other).sum() + (out[:, :K] != rows).sum()
    assert int(differ) == 0
