"""The recurrences a chunk of tokens at a time against the recurrence written out in 64-bit, on rows of unequal lengths around a chunk's
edge, with decays that keep, forget and are zero; and that the two forms agree where either may run."""

import pytest
import torch

pytestmark = pytest.mark.gpu

# 32-bit rounding, 2^-24, over sums of a chunk and a state's channels: a few units in the last place of the largest sums
BOUND = 2e-5
SIZES = [(4, 2, 128, 128), (2, 1, 64, 72), (3, 1, 100, 24), (2, 2, 20, 36), (1, 1, 4, 4), (2, 2, 32, 200)]
LENGTHS = [[1, 63, 64, 65, 2], [129, 1, 200]]


def draw(H, KH, D, V, T, channel, delta, decays, seed):
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(T, KH, D, generator=g) * D ** -0.5
    k = torch.nn.functional.normalize(torch.randn(T, KH, D, generator=g), dim=-1)
    v = torch.randn(T, H, V, generator=g)
    beta = torch.rand(T, H, generator=g)
    shape = (T, H, D) if channel else (T, H)
    if decays == "keep":
        decay = torch.exp(-1e-3 * torch.rand(shape, generator=g))
    elif decays == "forget":
        decay = torch.exp(-20 * torch.rand(shape, generator=g) ** 2)
        decay[::7] = 0.0
    else:  # nothing decays and every key is nearly the same: what is written is what the memory lacks, over and over
        decay = torch.ones(shape)
        k = torch.nn.functional.normalize(k[:1] + 0.02 * k, dim=-1)
        beta = torch.ones_like(beta)
    return q, k, v, beta, decay


def written_out(q, k, v, beta, decay, states, lengths, channel, delta):
    q, k, v, beta, decay = (t.double() for t in (q, k, v, beta, decay))
    share = v.shape[1] // k.shape[1]
    q, k = q.repeat_interleave(share, 1), k.repeat_interleave(share, 1)
    outs, final, t0 = [], [], 0
    for row, n in enumerate(lengths):
        S = states[row].double().transpose(1, 2)  # [H, D, V]
        for t in range(t0, t0 + n):
            S = S * (decay[t][:, :, None] if channel else decay[t][:, None, None])
            u = beta[t][:, None] * (v[t] - (torch.einsum("hd,hdv->hv", k[t], S) if delta else 0.0))
            S = S + k[t][:, :, None] * u[:, None]
            outs.append(torch.einsum("hd,hdv->hv", q[t], S))
        final.append(S.transpose(1, 2))
        t0 += n
    return torch.stack(outs), torch.stack(final)


@pytest.mark.parametrize("decays", ["keep", "forget", "same keys"])
@pytest.mark.parametrize("mode", ["head", "channel", "no delta"])
@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("lengths", LENGTHS)
def test_chunks_match_the_recurrence(lengths, sizes, mode, decays, monkeypatch):
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    H, KH, D, V = sizes
    channel, delta = mode == "channel", mode != "no delta"
    if decays == "keep":  # little scratch: the heads go in several groups
        monkeypatch.setattr(kernels, "CHUNKED_SCRATCH_FLOATS", 1)
    T, rows = sum(lengths), len(lengths)
    args = draw(H, KH, D, V, T, channel, delta, decays, seed=3)
    states = 0.3 * torch.randn(rows + 2, H, V, D, generator=torch.Generator().manual_seed(4))
    slots = [(2 * row + 1) % (rows + 2) if rows % 2 else row + 1 for row in range(rows)]
    want, final = written_out(*args, states[slots], lengths, channel, delta)
    i32 = dict(dtype=torch.int32, device="cuda")
    indptr = torch.tensor([sum(lengths[:i]) for i in range(rows + 1)], **i32)
    where = dict(qo_indptr=indptr, state_slots=torch.tensor(slots, **i32))
    flat = [t.reshape(T, -1).contiguous().cuda() for t in args]
    held = states.clone().cuda()
    out = torch.full((T, H * V), float("nan"), device="cuda")
    flag = torch.zeros(1, **i32)
    kernels.chunked_recurrence(*flat, held, out, kv_heads=KH, dim=D, heads=H, vdim=V, workspace=Workspace("cuda"), delta=delta, channel_decay=channel, flag=flag, **where)
    assert flag.item() == 0
    assert (out.cpu().double() - want.reshape(T, -1)).abs().max() < BOUND * max(1.0, want.abs().max().item())
    assert (held.cpu().double()[slots] - final).abs().max() < BOUND * max(1.0, final.abs().max().item())
    others = [slot for slot in range(rows + 2) if slot not in slots]
    assert torch.equal(held.cpu()[others], states[others])
    walked, walked_out = states.clone().cuda(), torch.empty_like(out)
    if delta:
        kernels.delta_recurrence(*flat, walked, walked_out, kv_heads=KH, dim=D, heads=H, vdim=V, channel_decay=channel, **where)
    else:
        kernels.ssm_recurrence(*flat, walked, walked_out, groups=KH, state=D, heads=H, vdim=V, **where)
    assert (out - walked_out).norm() < 2e-6 * walked_out.norm()
    assert (held - walked).norm() < 2e-6 * walked.norm()


def test_a_nan_stays_in_its_row_and_column():
    """A value that is no number reaches the outputs of its own row's later tokens and of its own column, and nothing else."""
    from kairyu_b200 import kernels
    from kairyu_b200.engine.workspace import Workspace

    H, KH, D, V, lengths = 2, 2, 32, 40, [70, 90]
    T = sum(lengths)
    args = draw(H, KH, D, V, T, False, True, "keep", seed=5)
    args[2][10, 1, 7] = float("nan")
    i32 = dict(dtype=torch.int32, device="cuda")
    out = torch.zeros(T, H * V, device="cuda")
    kernels.chunked_recurrence(*(t.reshape(T, -1).contiguous().cuda() for t in args), torch.zeros(2, H, V, D, device="cuda"), out, kv_heads=KH, dim=D, heads=H, vdim=V,
                               workspace=Workspace("cuda"), qo_indptr=torch.tensor([0, 70, 160], **i32), state_slots=torch.tensor([0, 1], **i32))
    bad = out.view(T, H, V).isnan().cpu()
    assert bad[10:70, 1, 7].all()
    bad[10:70, 1, 7] = False
    bad[:10, 1, 7] = False  # earlier tokens of the chunk meet it times a zero
    assert not bad.any()
