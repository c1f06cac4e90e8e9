"""Differential attention over portions on tcgen05: against the maps written out in 64-bit around the edges of its tiles (128 queries, 64 keys), with windows, scores
under and over the cap's polynomial range, and pages that hold numbers nobody wrote; and the mma.sync kernel on the same."""

import types

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,DV,heads,kv,page", [(64, 128, 4, 2, 16), (64, 64, 3, 1, 8), (128, 128, 2, 2, 64), (128, 64, 4, 1, 16)])
@pytest.mark.parametrize("counts,contexts,window", [([127, 2, 128], [0, 63, 1], 0), ([129, 300], [64, 200], 0), ([260, 64], [130, 0], 65), ([65], [500], 1)])
@pytest.mark.parametrize("cap,spread", [(0.0, 1.0), (50.0, 1.0), (5.0, 2.0)])
@pytest.mark.parametrize("norm", [True, False])
def test_portions(D, DV, heads, kv, page, counts, contexts, window, cap, spread, norm):
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    g = torch.Generator().manual_seed(D + DV + page)
    lengths = [c + n for c, n in zip(contexts, counts)]
    need = [-(-length // page) for length in lengths]
    order = (torch.randperm(sum(need), generator=g) + 1).tolist()
    table = torch.full((len(counts), max(need)), -1, dtype=torch.int32)
    k = torch.full((sum(need) + 1, page, kv, 2 * D), 3e4).bfloat16()
    v = torch.full((sum(need) + 1, page, kv, DV), float("nan")).bfloat16()
    k[0] = v[0] = 0
    keys, values = [], []
    for row, length in enumerate(lengths):
        pages, order = order[: need[row]], order[need[row] :]
        table[row, : need[row]] = torch.tensor(pages, dtype=torch.int32)
        keys.append((spread * torch.randn(length, kv, 2 * D, generator=g)).bfloat16())
        values.append(torch.randn(length, kv, DV, generator=g).bfloat16())
        for j in range(length):
            k[pages[j // page], j % page], v[pages[j // page], j % page] = keys[-1][j], values[-1][j]
    T = sum(counts)
    q = (spread * torch.randn(T, heads * 2 * D + 16, generator=g)).bfloat16()
    scale, lam, eps, out_scale = D ** -0.5, 0.37, 1e-5, 0.6
    want, t = torch.zeros(T, heads, DV, dtype=torch.float64), 0
    for row, (c, n) in enumerate(zip(contexts, counts)):
        at, j = torch.arange(c, c + n)[:, None], torch.arange(c + n)[None]
        hidden = (j > at) | ((j <= at - window) if window else (j < 0))
        for h in range(heads):
            a = []
            for m in range(2):
                s = q[t : t + n, (2 * h + m) * D : (2 * h + m + 1) * D].double() @ keys[row][:, h // (heads // kv), m * D : (m + 1) * D].double().T * scale
                s = cap * torch.tanh(s / cap) if cap else s
                a.append(torch.softmax(s.masked_fill(hidden, float("-inf")), -1) @ values[row][:, h // (heads // kv)].double())
            o = a[0] - lam * a[1]
            want[t : t + n, h] = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + eps) * out_scale if norm else o
        t += n
    i32 = dict(dtype=torch.int32, device="cuda")
    starts = [sum(counts[:i]) for i in range(len(counts) + 1)]

    def tiles(size):
        pairs = [(row, s) for row, n in enumerate(counts) for s in range(0, n, size)]
        return len(pairs), torch.tensor([row for row, _ in pairs], **i32), torch.tensor([s for _, s in pairs], **i32)

    short, long = kernels.DIFF_ATTENTION_TILE, kernels.DIFF_ATTENTION_TC5_TILE
    for sizes in ((short,), (short, long)):
        ctx = types.SimpleNamespace(qo_indptr=torch.tensor(starts, **i32), seq_lens=torch.tensor(lengths, **i32), tiles={size: tiles(size) for size in sizes}, num_decode_rows=0,
                                    workspace=Workspace("cuda"))
        out = torch.full((T, heads * DV), float("nan"), dtype=torch.bfloat16, device="cuda")
        flag = torch.zeros(1, **i32)
        before = kernels.launch_count
        kernels.diff_attention_mma(q.cuda()[:, : heads * 2 * D], out, k.cuda(), v.cuda(), ctx=ctx, block_table=table.cuda(), num_q_heads=heads, maps=2, scale=scale, softcap=cap,
                                   window=window, lam=lam, head_norm_eps=eps if norm else None, out_scale=out_scale if norm else 1.0, flag=flag)
        assert flag.item() == 0 and kernels.launch_count == before + 1
        # probabilities and the result rounded to 16 bits: 2^-8 of values of order one to four, and behind the norm of rows whose two maps nearly cancel a few times that
        assert (out.cpu().double().view_as(want) - want).abs().max() < 4e-2, sizes


@pytest.mark.parametrize("rows,length,heads,short", [(8, 30, 32, True), (8, 64, 32, True), (8, 65, 32, False), (1, 192, 16, True), (1, 193, 16, False)])
def test_short_portions_stay_on_mma_sync(rows, length, heads, short):
    """Sequences of one key tile, and of up to 192 keys in few blocks: the same bits as a step that lists no tiles of 128; otherwise the same within rounding."""
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    D = DV = 64
    g = torch.Generator().manual_seed(rows + length)
    k = torch.randn(13 * rows + 1, 16, 4, 2 * D, generator=g).bfloat16().cuda()
    v = torch.randn(13 * rows + 1, 16, 4, DV, generator=g).bfloat16().cuda()
    q = torch.randn(rows * length, heads * 2 * D, generator=g).bfloat16().cuda()
    i32 = dict(dtype=torch.int32, device="cuda")

    def tiles(size):
        pairs = [(row, s) for row in range(rows) for s in range(0, length, size)]
        return len(pairs), torch.tensor([row for row, _ in pairs], **i32), torch.tensor([s for _, s in pairs], **i32)

    results = []
    for sizes in ((kernels.DIFF_ATTENTION_TILE,), (kernels.DIFF_ATTENTION_TILE, kernels.DIFF_ATTENTION_TC5_TILE)):
        ctx = types.SimpleNamespace(qo_indptr=torch.arange(0, rows * length + 1, length, **i32), seq_lens=torch.full((rows,), length, **i32), tiles={size: tiles(size) for size in sizes},
                                    num_decode_rows=0, workspace=Workspace("cuda"), max_portion_seq_len=length)
        out = torch.full((rows * length, heads * DV), float("nan"), dtype=torch.bfloat16, device="cuda")
        kernels.diff_attention_mma(q, out, k, v, ctx=ctx, block_table=torch.arange(1, 13 * rows + 1, **i32).view(rows, 13), num_q_heads=heads, maps=2, scale=D ** -0.5, softcap=50.0,
                                   lam=0.4)
        results.append(out)
    assert torch.equal(*results) == short
    assert (results[0].float() - results[1].float()).abs().max() < 3e-2  # probabilities and results rounded to 16 bits, of values up to four
