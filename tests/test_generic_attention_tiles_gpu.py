"""The 32-bit attention kernel's tiles and segments of keys: against attention written out in 64-bit around their edges, and equal bits whether a token
comes in a prompt, in a portion, as a single token, or as a single token whose keys are spread over blocks."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def case(heads, kv, dim, page, context, seed):
    g = torch.Generator().manual_seed(seed)
    pages = -(-context // page)
    order = torch.randperm(pages, generator=g) + 1
    k, v = (torch.full((pages + 1, page, kv, dim), float("nan")) for _ in range(2))  # what no token wrote is no number
    for j in range(context):
        k[order[j // page], j % page] = torch.randn(kv, dim, generator=g)
        v[order[j // page], j % page] = torch.randn(kv, dim, generator=g)
    return dict(q=torch.randn(context, heads * dim, generator=g), k=k, v=v, table=order.int()[None])


def written_out(c, heads, kv, dim, page, first, scale, window, sinks, value_dim):
    context = c["q"].shape[0]
    places = [(int(c["table"][0, j // page]), j % page) for j in range(context)]
    keys = torch.stack([c["k"][at] for at in places]).double()
    values = torch.stack([c["v"][at] for at in places]).double()[..., :value_dim]
    out = torch.zeros(context - first, heads, value_dim, dtype=torch.float64)
    for t in range(first, context):
        start = max(0, t + 1 - window) if window else 0
        for h in range(heads):
            s = keys[start : t + 1, h // (heads // kv)] @ c["q"][t, h * dim : (h + 1) * dim].double() * scale
            if sinks is not None:
                s = torch.cat([s, sinks[h : h + 1].double()])
            out[t - first, h] = torch.softmax(s, 0)[: t + 1 - start] @ values[start : t + 1, h // (heads // kv)]
    return out.reshape(context - first, -1)


# heads, key/value heads, width, value width, page, positions, window, sinks
CASES = [(4, 2, 64, 64, 16, 70, 0, False), (8, 2, 128, 128, 16, 330, 0, True), (3, 1, 20, 12, 8, 257, 65, False), (2, 2, 256, 192, 32, 300, 0, False),
         (32, 1, 36, 36, 4, 140, 70, True), (6, 6, 100, 100, 16, 520, 300, False), (64, 1, 32, 32, 16, 66, 1, False)]


@pytest.mark.parametrize("heads,kv,dim,value_dim,page,context,window,with_sinks", CASES)
def test_tiles_and_segments(heads, kv, dim, value_dim, page, context, window, with_sinks):
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    c = case(heads, kv, dim, page, context, seed=2)
    scale = dim ** -0.5
    sinks = torch.randn(heads, generator=torch.Generator().manual_seed(3)) if with_sinks else None
    i32 = dict(dtype=torch.int32, device="cuda")
    device = {name: c[name].cuda() for name in ("q", "k", "v", "table")}

    def run(first, stop, workspace=None):
        """Tokens first .. stop - 1 as one portion."""
        out = torch.full((stop - first, heads * value_dim), float("nan"), device="cuda")
        flag = torch.zeros(1, **i32)
        kernels.paged_attention_generic(device["q"][first:stop], out, device["k"], device["v"], positions=torch.arange(first, stop, **i32),
                                        row_ids=torch.zeros(stop - first, **i32), block_table=device["table"], num_q_heads=heads, scale=scale, window=window, flag=flag,
                                        sinks=None if sinks is None else sinks.cuda(), value_dim=value_dim, workspace=workspace)
        assert flag.item() == 0
        return out

    whole = run(0, context)
    want = written_out(c, heads, kv, dim, page, 0, scale, window, sinks, value_dim)
    # 2^-24 over the roundings of a score (its width in sums of 32), a tile's sums and the segments' merges: well under 1e-5 of values of order one
    assert (whole.cpu().double() - want).abs().max() < 1e-5
    cut = context * 3 // 5
    assert torch.equal(torch.cat([run(0, cut), run(cut, context)]), whole)
    for t in {0, 63, 64, cut, min(context - 1, 255), min(context - 1, 256), context - 1}:
        assert torch.equal(run(t, t + 1), whole[t : t + 1]), t
        assert torch.equal(run(t, t + 1, Workspace("cuda")), whole[t : t + 1]), t


@pytest.mark.parametrize("M,N,K", [(1, 5, 7), (16, 33, 64), (17, 130, 300), (64, 64, 256), (65, 129, 257), (300, 257, 513), (700, 3000, 36), (1400, 1900, 20)])
@pytest.mark.parametrize("shift", [0, 1])
def test_products_of_every_tile_shape(M, N, K, shift):
    """Every tile's rows and columns, whole and ragged, rows of whole 16-byte groups and others; a row alone has the bits it has among the others."""
    from kairyu_b200 import kernels

    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K + shift, generator=g)[:, shift:].cuda()
    w, bias = torch.randn(N, K, generator=g).cuda(), torch.randn(N, generator=g).cuda()
    y = torch.empty(M, N, device="cuda")
    kernels.linear(x, w, bias, y)
    want = x.double() @ w.double().T + bias.double()
    # up to 256 additions into one accumulator, each off by at most 2^-24 of a partial sum of at most 5 sqrt(K); their signs are independent, so they add up
    # as the root of their number, and a few thousand outputs show twice that: 2^-24 * 5 sqrt(K) * 16 * 2 = 1e-5 sqrt(K)
    assert (y.double() - want).abs().max() < 1e-5 * K ** 0.5
    for row in {0, M // 2, M - 1}:
        one = torch.empty(1, N, device="cuda")
        kernels.linear(x[row : row + 1], w, bias, one)
        assert torch.equal(one, y[row : row + 1])
