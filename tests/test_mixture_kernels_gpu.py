"""The mixture's plan, row moves and few-pairs products around the groups they take at a time, against torch statements of the same."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,top,experts", [(1, 1, 1), (8, 4, 32), (3, 2, 33), (2048, 4, 32), (2049, 4, 100), (5000, 3, 7), (300, 8, 1000)])
def test_plan(tokens, top, experts):
    from kairyu_b200 import kernels

    g = torch.Generator().manual_seed(tokens)
    ids = torch.stack([torch.randperm(max(experts, top), generator=g)[:top] % experts for _ in range(tokens)]).int() if tokens < 500 else torch.randint(0, experts, (tokens, top), generator=g).int()
    pairs = tokens * top
    plan = kernels.moe_plan(ids.cuda(), experts, torch.full((kernels.moe_plan_size(pairs, experts),), -7, dtype=torch.int32, device="cuda"))
    held = {name: t.cpu() for name, t in plan.items() if isinstance(t, torch.Tensor)}
    counts = torch.bincount(ids.flatten().long(), minlength=experts)
    assert torch.equal(held["ends"].long(), counts.cumsum(0))
    assert torch.equal(held["sorted"].sort().values, torch.arange(pairs, dtype=torch.int32))
    runs = ids.flatten()[held["sorted"].long()]
    assert torch.equal(runs, runs.sort().values)
    assert torch.equal(held["token_of"], held["sorted"] // top)
    assert torch.equal(held["place_of"][held["sorted"].long()], torch.arange(pairs, dtype=torch.int32))
    n = int(held["num_tiles"])
    want = [(e, int(counts[:e].sum()) + first, min(64, int(counts[e]) - first)) for e in range(experts) for first in range(0, int(counts[e]), 64)]
    assert list(zip(held["tile_expert"][:n].tolist(), held["tile_first"][:n].tolist(), held["tile_pairs"][:n].tolist())) == want


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("tokens,top,H", [(1, 1, 8), (5, 3, 24), (7, 4, 2048), (3, 32, 1032), (4, 2, 20), (2, 2, 7)])
@pytest.mark.parametrize("extra", [False, True])
def test_gather_activation_combine(tokens, top, H, extra, dtype):
    from kairyu_b200 import kernels

    g = torch.Generator().manual_seed(H)
    pairs, experts = tokens * top, 4
    x = torch.randn(tokens, H, generator=g).to(dtype).cuda()
    at = torch.randperm(pairs, generator=g).int().cuda()
    rows_of = torch.randint(0, tokens, (pairs,), generator=g).int().cuda()
    gathered = torch.zeros(pairs, H, dtype=dtype, device="cuda")
    kernels.gather_rows(x, rows_of, gathered)
    assert torch.equal(gathered, x[rows_of.long()])
    gate_up = (3 * torch.randn(pairs, 2 * H, generator=g)).to(dtype).cuda()
    y = torch.zeros(pairs, H, dtype=dtype, device="cuda")
    kernels.moe_activation(gate_up, y, limit=2.5, alpha=1.702, shift=1.0)
    a, b = gate_up[:, :H].double().clamp(max=2.5), gate_up[:, H:].double().clamp(-2.5, 2.5)
    want = a * torch.sigmoid(1.702 * a) * (b + 1.0)
    bound = 2 ** -8 if dtype == torch.bfloat16 else 1e-6  # one rounding of a value
    assert ((y.double() - want).abs() <= bound * want.abs() + 1e-6).all()
    weights = torch.rand(tokens, top, generator=g).cuda()
    ids = torch.randint(0, experts + 2, (tokens, top), generator=g).int().cuda()
    shared, shared_gate = (torch.randn(tokens, H, generator=g).to(dtype).cuda(), torch.randn(tokens, 3, generator=g).cuda()[:, 1:2]) if extra else (None, None)
    for rows in ((gathered.float(), gathered) if dtype == torch.bfloat16 else (gathered,)):
        for identity in (False, True):
            out = torch.zeros(tokens, H, dtype=dtype, device="cuda")
            kernels.moe_combine(rows, weights, out, at, **(dict(ids=ids, x=x, experts=experts) if identity else {}), **(dict(extra=shared, extra_gate=shared_gate) if extra else {}))
            each = rows.double()[at.long()].view(tokens, top, H)
            if identity:
                each = torch.where((ids >= experts)[..., None], x.double()[:, None], each)
            want = (each * weights.double()[..., None]).sum(1)
            if extra:
                want = want + torch.sigmoid(shared_gate.double()) * shared.double()
            assert ((out.double() - want).abs() <= bound * want.abs() + 1e-5 * top).all()


@pytest.mark.parametrize("tokens,top,experts,K,N", [(1, 1, 1, 8, 16), (8, 4, 32, 256, 72), (16, 3, 4, 72, 64), (16, 4, 4, 1024, 40), (3, 2, 6, 136, 200), (12, 1, 1, 2048, 64)])
def test_few_pairs(tokens, top, experts, K, N):
    """Both halves of the columns, runs that end in either, more than eight pairs of an expert."""
    from kairyu_b200 import kernels

    g = torch.Generator().manual_seed(K + N)
    ids = torch.stack([torch.randperm(experts, generator=g)[:top] for _ in range(tokens)]).int().cuda()
    pairs = tokens * top
    plan = kernels.moe_plan(ids, experts, torch.zeros(kernels.moe_plan_size(pairs, experts), dtype=torch.int32, device="cuda"))
    x = torch.randn(tokens, K, generator=g).bfloat16().cuda()
    w = (torch.randn(experts, 2 * N, K, generator=g) * K ** -0.5).bfloat16().cuda()
    hidden = torch.zeros(pairs, N, dtype=torch.bfloat16, device="cuda")
    kernels.moe_skinny(x, w, hidden, plan, top=top, gated=True, limit=7.0, alpha=1.702, shift=1.0)
    down = (torch.randn(experts, K, N, generator=g) * N ** -0.5).bfloat16().cuda()
    rows = torch.zeros(pairs, K, device="cuda")
    if N % 8 == 0:
        kernels.moe_skinny(hidden, down, rows, plan, top=top, gated=False)
    for place, pair in enumerate(plan["sorted"].tolist()):
        e, t = int(ids.view(-1)[pair]), pair // top
        both = w[e].double() @ x[t].double()
        a, b = both[:N].clamp(max=7.0), both[N:].clamp(-7.0, 7.0)
        want = a * torch.sigmoid(1.702 * a) * (b + 1.0)
        assert (hidden[place].double() - want).abs().max() < 2e-2 * max(1.0, want.abs().max().item())  # 2^-8 of the largest, and 32-bit sums
        assert (rows[pair].double() - down[e].double() @ hidden[place].double()).abs().max() < 1e-4
