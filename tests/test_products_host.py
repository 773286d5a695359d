"""Which products may read w while the kernel in front still runs: those whose caller says that w is a weight, no others.
The kernels' wrappers are replaced by ones that write down what they are told."""
import pytest
import torch

from snowllm_b200.errors import KernelError
from snowllm_b200.ops import kernels, linear, linear_glu, linear_swiglu


@pytest.fixture
def told(monkeypatch):
    calls = []
    for name in ("gemm_skinny", "gemm_simt", "gemm_tc"):
        monkeypatch.setattr(kernels, name, lambda x, w, name=name, **kw: calls.append((name, kw["w_ahead"])) or x)
    monkeypatch.setattr(kernels, "gemm_skinny_ok", lambda x, w: x.dtype == torch.bfloat16)
    for name in ("swiglu", "gated_act"):
        monkeypatch.setattr(kernels, name, lambda h, *a, **kw: h)
    return calls


@pytest.mark.parametrize("rows,dtype,kernel", [(3, torch.bfloat16, "gemm_skinny"), (40, torch.bfloat16, "gemm_tc"),
                                               (3, torch.float32, "gemm_simt"), (40, torch.float32, "gemm_simt")])
def test_w_is_read_ahead_only_where_the_caller_says_it_is_a_weight(told, rows, dtype, kernel):
    x, w = torch.zeros(rows, 64, dtype=dtype), torch.zeros(32, 64, dtype=dtype)
    for said in (False, True):
        kw = {"w_ahead": True} if said else {}
        linear(x, w, **kw)
        linear_glu(x, w, True, **kw)
        linear_glu(x, w, False, "relu", **kw)
        linear_swiglu(x, w, True, **kw)
        assert told == [(kernel, said)] * 4
        told.clear()


@pytest.mark.parametrize("entry", ["moe_route", "moe_route_sort"])
def test_a_router_is_read_ahead_only_where_the_caller_says_so(monkeypatch, entry):
    parts = []

    def fn(name):
        return lambda *args: parts.append(args[7]) or 0 if name == "snk_gemm_tc_parts" else 0

    monkeypatch.setattr(kernels, "fn", fn)
    for name in ("_chk", "check"):
        monkeypatch.setattr(kernels, name, lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    monkeypatch.setattr(kernels, "gemm_tc_ok", lambda x, w: True)
    monkeypatch.setattr(kernels, "gemm_tc_is_split", lambda M, N, K: True)
    monkeypatch.setattr(kernels, "_tc_scratch_bytes", lambda *a: 64)
    x, w = torch.zeros(65, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16)
    getattr(kernels, entry)(x, w, None, 2, True, 1.0)
    getattr(kernels, entry)(x, w, None, 2, True, 1.0, w_ahead=True)
    assert parts == [0, 1]


TILES = ((128, 128, 1.0), (64, 128, 0.95), (64, 64, 0.8), (32, 64, 0.6))       # rows, columns, share of the FMA rate


@pytest.mark.parametrize("sms", [148, 132])
def test_the_float_tile_is_the_one_with_the_least_work_on_the_busiest_sm(sms):
    pick = kernels.fn("snk_gemm_simt_tile")
    seen = set()
    for M, N, groups in [(17, 56, 0), (200, 2049, 0), (509, 2050, 0), (509, 8195, 0), (300, 6147, 0), (2048, 2048, 0),
                         (8192, 64, 0), (40, 56, 8), (900, 3584, 32), (4096, 3584, 32)]:
        mean = -(-M // groups) if groups else M
        cost = [-(-(max(groups, 1) * -(-mean // bm) * -(-N // bn)) // sms) * bm * bn / rate for bm, bn, rate in TILES]
        assert pick(M, N, groups, M, sms) == cost.index(min(cost))
        seen.add(pick(M, N, groups, M, sms))
    assert seen == {0, 1, 2, 3}


def test_a_float_product_of_millions_of_rows_keeps_a_tile_that_the_grid_can_hold():
    """25,013 groups of 96 rows on average, one of which may own them all: of 32 x 64 tiles, the cheapest by their count, the
    grid would need 75,039 along y.  A launch of 64-row tiles holds up to 4,194,240 rows."""
    pick = kernels.fn("snk_gemm_simt_tile")
    G, M = 25013, 25013 * 96
    assert TILES[pick(M, 64, G, 1000, 148)][0] == 32
    assert TILES[pick(M, 64, G, M, 148)][0] >= 64
    for rows in (32 * 65535, 32 * 65535 + 1, 64 * 65535):
        assert -(-rows // TILES[pick(rows, 64, rows // 75, rows, 148)][0]) <= 65535


def test_which_few_rows_products_stream_w_through_shared_memory():
    """148 SMs: up to 2,368 rows of W are one round of strips, up to 4,736 two, up to 7,104 three."""
    streams = kernels.fn("snk_gemm_skinny_streams")
    for (N, K), want in {(16, 2560): 1, (16, 2624): 0, (1760, 4096): 0, (1776, 4096): 1, (2368, 12288): 1, (2368, 12352): 0,
                         (2369, 448): 0, (2369, 512): 1, (4736, 65536): 1, (4737, 512): 0, (4737, 2048): 1, (7104, 16384): 1,
                         (7104, 16448): 0, (7105, 2048): 0, (65536, 2048): 0, (2048, 2080): 0}.items():
        for M in (1, 16):
            assert streams(M, N, K, 148) == want, (N, K)
        assert streams(17, N, K, 148) == 0


@pytest.mark.parametrize("product", ["gemm_simt", "gemm_skinny"])
def test_a_row_gather_that_is_too_short_is_refused(monkeypatch, product):
    monkeypatch.setattr(kernels, "_chk", lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "fn", lambda name: pytest.fail("launched"))
    x, w = torch.zeros(9, 64, dtype=torch.bfloat16), torch.zeros(32, 64, dtype=torch.bfloat16)
    for rows_out, listed in ((None, 8), (12, 11)):
        with pytest.raises(KernelError, match="row gather"):
            getattr(kernels, product)(x, w, a_rows=torch.zeros(listed, dtype=torch.int32), rows_out=rows_out)


def test_which_decode_attention_launches_walk():
    """148 SMs hold 444 blocks at once: 16 rounds of them are 7,104 possible blocks."""
    walks = kernels.fn("snk_attention_decode_walks")
    for (M, nkv, chunks, hd), want in {(28, 8, 32, 64): 1, (27, 8, 32, 64): 0, (64, 8, 31, 64): 0, (64, 8, 32, 64): 1, (256, 8, 32, 64): 1,
                                       (257, 8, 32, 64): 0, (64, 8, 64, 128): 0, (1, 8, 888, 64): 1, (1, 8, 887, 64): 0}.items():
        assert walks(M, nkv, chunks, hd, 0, 148) == want, (M, nkv, chunks, hd)
        assert not walks(M, nkv, chunks, hd, 1, 148)                # launches with options do not
