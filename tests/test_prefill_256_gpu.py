"""Portions of head size 256 on the tcgen05 kernel: against attention written out in 64-bit around the edges of its tiles (128 queries, 64 keys), with keys
split over blocks, windows, sinks, a gate, keys that serve as values, and pages that hold numbers nobody wrote."""

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 256


@pytest.mark.parametrize("page", [8, 16, 64])
@pytest.mark.parametrize("counts,contexts,window,heads,kv", [([127, 2, 128], [0, 63, 1], 0, 2, 1), ([129, 300, 5], [64, 200, 700], 0, 3, 3), ([260], [130], 65, 4, 2), ([64, 65], [0, 0], 1, 16, 1)])
@pytest.mark.parametrize("extras", [False, True])
def test_portions(counts, contexts, window, heads, kv, page, extras):
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    g = torch.Generator().manual_seed(heads + page)
    lengths = [c + n for c, n in zip(contexts, counts)]
    need = [-(-length // page) for length in lengths]
    order = (torch.randperm(sum(need), generator=g) + 1).tolist()
    table = torch.full((len(counts), max(need)), -1, dtype=torch.int32)
    k = torch.full((sum(need) + 1, page, kv, D), 3e4).bfloat16()  # what nobody wrote
    v = torch.full((sum(need) + 1, page, kv, D), float("nan")).bfloat16()
    k[0] = v[0] = 0
    keys, values = [], []
    for row, length in enumerate(lengths):
        pages, order = order[: need[row]], order[need[row] :]
        table[row, : need[row]] = torch.tensor(pages, dtype=torch.int32)
        keys.append(torch.randn(length, kv, D, generator=g).bfloat16())
        values.append(keys[-1] if extras else torch.randn(length, kv, D, generator=g).bfloat16())
        for j in range(length):
            k[pages[j // page], j % page], v[pages[j // page], j % page] = keys[-1][j], values[-1][j]
    if extras:
        k = torch.where(k == 3e4, torch.zeros(()).bfloat16(), k)
        v = k  # rows that serve as keys and values
    T = sum(counts)
    q = torch.randn(T, heads * D + 8, generator=g).bfloat16()[:, : heads * D]
    sinks = torch.randn(heads, generator=g) if extras else None
    gate = torch.randn(T, heads * D, generator=g).bfloat16() if extras else None
    scale = D ** -0.5
    want, t = torch.zeros(T, heads * D, dtype=torch.float64), 0
    for row, (c, n) in enumerate(zip(contexts, counts)):
        for h in range(heads):
            s = q[t : t + n, h * D : (h + 1) * D].double() @ keys[row][:, h // (heads // kv)].double().T * scale
            at, j = torch.arange(c, c + n)[:, None], torch.arange(c + n)[None]
            s = s.masked_fill((j > at) | ((j <= at - window) if window else (j < 0)), float("-inf"))
            if sinks is not None:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            want[t : t + n, h * D : (h + 1) * D] = torch.softmax(s, -1)[:, : c + n] @ values[row][:, h // (heads // kv)].double()
        t += n
    if gate is not None:
        want *= torch.sigmoid(gate.double())
    i32 = dict(dtype=torch.int32, device="cuda")
    starts = [0]
    for n in counts:
        starts.append(starts[-1] + n)

    def tiles(size):
        pairs = [(row, s) for row, n in enumerate(counts) for s in range(0, n, size)]
        return len(pairs), torch.tensor([row for row, _ in pairs], **i32), torch.tensor([s for _, s in pairs], **i32)

    assert kernels.attention_prefill_wide_tile_rows(D) == 128
    num, rows, firsts = tiles(kernels.attention_prefill_tile_rows(D))
    kc, vc = k.cuda(), v.cuda()
    if extras:
        vc = kc
    for splits in (None, 1, 2, 5):
        out = torch.full((T, heads * D), float("nan"), dtype=torch.bfloat16, device="cuda")
        flag = torch.zeros(1, **i32)
        padded = torch.zeros(T, heads * D + 8, dtype=torch.bfloat16, device="cuda")
        padded[:, : heads * D] = q.cuda()
        kernels.attention_prefill_mma(padded[:, : heads * D], out, kc, vc, qo_indptr=torch.tensor(starts, **i32), seq_lens=torch.tensor(lengths, **i32), block_table=table.cuda(),
                                      tile_rows=rows, tile_starts=firsts, num_tiles=num, num_q_heads=heads, scale=scale, window=window, flag=flag, max_seq_len=max(lengths),
                                      workspace=Workspace("cuda"), num_splits=splits, wide_tiles=tiles(128), sinks=None if sinks is None else sinks.cuda(),
                                      gate=None if gate is None else gate.cuda())
        assert flag.item() == 0
        # probabilities and the result are rounded to 16 bits: 2^-8 of values of order one to four
        assert (out.cpu().double() - want).abs().max() < 2e-2, splits
