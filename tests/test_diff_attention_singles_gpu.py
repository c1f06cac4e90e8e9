"""Differential attention of single tokens on tensor cores around the edges of its 64-key tiles and of its ring of three, with windows, page sizes that are no power of
two, absent pages, and scores within, across and beyond the range of the cap's polynomial: against the 32-bit kernel on the same inputs."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,DV,heads,kv", [(32, 32, 4, 2), (64, 128, 8, 2), (128, 128, 16, 1), (48, 48, 3, 1)])
@pytest.mark.parametrize("page", [16, 24, 1])
@pytest.mark.parametrize("window", [0, 1, 65, 200])
@pytest.mark.parametrize("cap", [30.0, 1.5, 0.1, 0.0])
def test_single_tokens(D, DV, heads, kv, page, window, cap):
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    g = torch.Generator().manual_seed(D + page)
    lengths = [1, 2, 63, 64, 65, 128, 129, 192, 193, 256, 257, 500]
    most = -(-max(lengths) // page)
    pages = 40 + most
    table = torch.randint(0, pages, (len(lengths), most), generator=g, dtype=torch.int32)
    k = (0.5 * torch.randn(pages, page, kv, 2 * D, generator=g)).bfloat16().cuda()
    v = torch.randn(pages, page, kv, DV, generator=g).bfloat16().cuda()
    q = torch.randn(len(lengths), heads * 2 * D, generator=g).bfloat16().cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    rows = torch.arange(len(lengths), **i32)
    seq_lens = torch.tensor(lengths, **i32)
    ctx = types.SimpleNamespace(qo_indptr=torch.arange(len(lengths) + 1, **i32), seq_lens=seq_lens, tiles={kernels.DIFF_ATTENTION_TILE: (0, rows, rows)},
                                num_decode_rows=len(lengths), decode_rows=rows, decode_tokens=rows, workspace=Workspace("cuda"))
    common = dict(block_table=table.cuda(), num_q_heads=heads, maps=2, scale=D ** -0.5, softcap=cap, window=window, lam=0.4, head_norm_eps=None, out_scale=1.0)
    got = torch.full((len(lengths), heads * DV), float("nan"), dtype=torch.bfloat16, device="cuda")
    kernels.diff_attention_mma(q, got, k, v, ctx=ctx, **common)
    want = torch.empty(len(lengths), heads * DV, device="cuda")
    kernels.diff_attention_generic(q.float(), want, k.float(), v.float(), positions=seq_lens - 1, row_ids=rows, **common)
    # probabilities and the result are rounded to 16 bits: 2^-9 each, of results up to four
    assert (got.float() - want).abs().max() < 3e-2
    # key rows beyond the sequence lie on pages that are not there: the same result
    table[torch.arange(most)[None] > (torch.tensor(lengths)[:, None] - 1) // page] = -1
    again = torch.full_like(got, float("nan"))
    kernels.diff_attention_mma(q, again, k, v, ctx=ctx, **{**common, "block_table": table.cuda()})
    assert torch.equal(got, again)
