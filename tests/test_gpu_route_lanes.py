"""The selection of many rows with up to 32 experts (a lane an expert, csrc/moe.cu) against the general one, which 33 experts and more
take: the same picks and weights, bit for bit, ties, zeros of both signs, infinities and biases of -inf included; and what is picked
where scores are NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu
RENORM, TINY = 1, 32


def topk(logits, bias, k, flags, transposed=0):
    """``logits`` [planes, M, E]."""
    from snowllm_b200.ops import kernels
    planes, M, E = logits.shape
    laid = (logits[0].T if transposed else logits).contiguous().cuda()
    bias = None if bias is None else bias.cuda()
    ids = torch.full((M, k), -7, dtype=torch.int32, device="cuda")
    wts = torch.full((M, k), float("nan"), device="cuda")
    kernels.check(kernels.fn("snk_moe_topk")(kernels._ptr(laid), kernels._ptr(bias), kernels._ptr(ids), kernels._ptr(wts), M, E, k, flags,
                                             1.5, transposed, planes, kernels._stream()), "moe_topk")
    torch.cuda.synchronize()
    return ids.cpu(), wts.cpu()


def draw(E, planes, M=70, seed=0):
    gen = torch.Generator().manual_seed(seed + 100 * E + planes)
    x = torch.randn(planes, M, E, generator=gen)
    x[:, 1] = 0.5                                            # every expert equal
    x[:, 2] = torch.randint(-1, 2, (E,), generator=gen).float()                    # few values
    x[:, 3] = torch.where(torch.rand(E, generator=gen) < 0.5, torch.tensor(0.0), torch.tensor(-0.0))
    x[0, 4, ::2] = float("inf")
    x[0, 5, ::3] = float("-inf")
    x[:, 6] = -200.0                                         # every probability 0
    return x, gen


@pytest.mark.parametrize("E,k", [(1, 1), (5, 2), (5, 5), (31, 4), (32, 1), (32, 8), (32, 32)])
@pytest.mark.parametrize("planes,transposed", [(1, 0), (1, 1), (4, 0), (8, 0)])
@pytest.mark.parametrize("flags", [0, RENORM, RENORM | TINY])
def test_the_same_as_the_general_selection(E, k, planes, transposed, flags):
    logits, gen = draw(E, planes)
    wide = 40 - E
    bias = torch.randn(E, generator=gen)
    tied = bias.clone()
    tied[E // 2:] = tied[0]
    barred = bias.clone()
    barred[: (E + 1) // 2] = float("-inf")
    for b in (bias, tied, barred, torch.full((E,), float("-inf")), None):
        # experts that are never picked fill up to 40: a bias of -inf, or (without one) a probability of 0 behind all others
        fill = torch.full((planes, logits.shape[1], wide), float("-inf") if b is None else 0.0)
        more = None if b is None else torch.cat((b, torch.full((wide,), float("-inf"))))
        got, want = topk(logits, b, k, flags, transposed), topk(torch.cat((logits, fill), 2), more, k, flags, transposed)
        assert torch.equal(got[0], want[0])
        assert torch.equal(got[1].view(torch.int32), want[1].view(torch.int32))


def picks(score, k):
    """NaN never wins, ties go to the lower expert, a picked one falls to -inf; where nothing is left, index order."""
    score, ids = list(score), []
    for j in range(k):
        best = None
        for e, s in enumerate(score):
            if s == s and (best is None or s > score[best]):
                best = e
        best = j if best is None else best
        ids.append(best)
        score[best] = float("-inf")
    return ids


@pytest.mark.parametrize("E,k", [(5, 5), (31, 4), (32, 32)])
def test_scores_that_are_nan(E, k):
    logits, gen = draw(E, 1, seed=7)
    logits[0, 10:40][torch.rand(30, E, generator=gen) < 0.5] = float("nan")
    logits[0, 40] = float("nan")
    ids, wts = topk(logits, None, k, 0)
    score = (1 / (1 + torch.exp(-logits[0]))).tolist()
    for m in (10, 11, 20, 39, 40):
        assert ids[m].tolist() == picks(score[m], k), m
        assert torch.equal(wts[m].isnan(), logits[0, m].isnan()[ids[m].long()])
