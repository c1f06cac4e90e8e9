"""What stands before and behind the recurrences (short convolution, silu, unit norms, decays; gated norms) over rows around the groups of tokens and channels
that the kernels take at a time, against the torch statements of the same, and token by token with equal bits."""

import numpy as np
import pytest
import torch

import makilorn_torch_kernels as delta_ref
import tapasun_torch_kernels as ssm_ref

pytestmark = pytest.mark.gpu

LENGTHS = {"short": [1, 2, 5, 1], "long": [1, 15, 16, 17, 3, 1200, 1]}
# 32-bit: a few roundings of values of order one through exponentials; 16-bit results once more, 2^-9 of a value
CLOSE = {torch.float32: 2e-5, torch.bfloat16: 8e-3}


def near(got, want, dtype=torch.float32):
    want = want.float()
    assert (got.cpu().float() - want).abs().max() < CLOSE[dtype] * max(1.0, want.abs().max().item())


def step(lengths):
    starts = [0, *np.cumsum(lengths).tolist()]
    rows = [row for row, n in enumerate(lengths) for _ in range(n)]
    slots = [(3 * row + 1) % (len(lengths) + 2) if (len(lengths) + 2) % 3 else row for row in range(len(lengths))]
    i32 = dict(dtype=torch.int32)
    return dict(row_ids=torch.tensor(rows, **i32), qo_indptr=torch.tensor(starts, **i32), state_slots=torch.tensor(slots, **i32))


def on_gpu(tensors):
    return {name: t.cuda() if isinstance(t, torch.Tensor) else t for name, t in tensors.items()}


def token_by_token(lengths, where, call):
    """``call(tokens, where of them)`` for every row's i-th token at once, i going up."""
    starts = where["qo_indptr"].tolist()
    for i in range(max(lengths)):
        live = [row for row, n in enumerate(lengths) if i < n]
        call(torch.tensor([starts[row] + i for row in live]).cuda(), on_gpu(dict(
            row_ids=torch.arange(len(live), dtype=torch.int32), qo_indptr=torch.arange(len(live) + 1, dtype=torch.int32), state_slots=where["state_slots"][live])))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("KH,D,H,V,taps,channel", [(2, 128, 4, 128, 4, False), (1, 20, 3, 36, 3, True), (2, 100, 2, 64, 2, False), (1, 4, 1, 4, 1, True), (2, 128, 2, 8, 4, True), (1, 130, 2, 6, 5, False)])
def test_delta_prepare(KH, D, H, V, taps, channel, lengths, dtype):
    from kairyu_b200 import kernels

    lengths = LENGTHS[lengths]
    g = torch.Generator().manual_seed(D + V)
    T, C = sum(lengths), 2 * KH * D + H * V
    where = step(lengths)
    packed = torch.randn(T, C + 8, generator=g).to(dtype)
    inputs = dict(gates=torch.randn(T, H * (1 if channel else 2), generator=g), taps=torch.randn(C, taps, generator=g) * 0.5,
                  kept=torch.randn(len(lengths) + 2, taps - 1, C, generator=g) if taps > 1 else None,
                  a_log=torch.randn(H, generator=g), dt_bias=torch.randn(H * (D if channel else 1), generator=g),
                  channel_a=torch.randn(T, H * D, generator=g) if channel else None)
    sizes = dict(kv_heads=KH, dim=D, heads=H, vdim=V)

    def outputs(rows, device):
        per = D if channel else 1
        return {n: torch.zeros(rows, c, device=device) for n, c in (("q", KH * D), ("k", KH * D), ("v", H * V), ("beta", H), ("decay", H * per))}

    def run(module, device, rows, where, kept):
        out = outputs(len(rows), device)
        on = {n: (t.to(device) if t is not None else None) for n, t in inputs.items()}
        module.delta_prepare(packed.to(device)[rows], on["gates"][rows].contiguous(), on["taps"], kept, a_log=on["a_log"], dt_bias=on["dt_bias"],
                             channel_a=on["channel_a"][rows].contiguous() if channel else None, **out, **where, **sizes)
        return out

    want_kept = inputs["kept"].clone() if taps > 1 else None
    want = run(delta_ref, "cpu", torch.arange(T), where, want_kept)
    kept = inputs["kept"].cuda() if taps > 1 else None
    got = run(kernels, "cuda", torch.arange(T).cuda(), on_gpu(where), kept)
    for name in got:
        near(got[name], want[name])
    if taps > 1:
        near(kept, want_kept)
    kept_single = inputs["kept"].cuda() if taps > 1 else None
    single = outputs(T, "cuda")

    def one(rows, where):
        for name, t in run(kernels, "cuda", rows, where, kept_single).items():
            single[name][rows] = t

    if max(lengths) < 100:
        token_by_token(lengths, where, one)
        assert all(torch.equal(single[name], got[name]) for name in got)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("G,N,H,V,taps,bias,parts", [(2, 128, 4, 64, 4, True, 2), (1, 20, 3, 36, 3, False, 1), (1, 4, 1, 4, 1, True, 1), (3, 12, 6, 100, 2, True, 1), (1, 6, 2, 7, 4, True, 2)])
def test_ssm_prepare_and_norm(G, N, H, V, taps, bias, parts, lengths, dtype):
    from kairyu_b200 import kernels

    lengths = LENGTHS[lengths]
    g = torch.Generator().manual_seed(N + V)
    T, inner = sum(lengths), H * V
    C = inner + 2 * G * N
    where = step(lengths)
    packed = torch.randn(T, inner + C, generator=g).to(dtype)
    dt_raw, tap = torch.randn(T, H, generator=g), torch.randn(C, taps, generator=g) * 0.5
    conv_bias = torch.randn(C, generator=g) if bias else None
    kept0 = torch.randn(len(lengths) + 2, taps - 1, C, generator=g) if taps > 1 else None
    a_log, dt_bias, skip, weight = torch.randn(H, generator=g), torch.randn(H, generator=g), torch.randn(H, generator=g), torch.randn(inner, generator=g)

    def run(module, device):
        out = {n: torch.zeros(T, c, device=device) for n, c in (("x", inner), ("b", G * N), ("c", G * N), ("dt", H), ("decay", H))}
        kept = kept0.clone().to(device) if taps > 1 else None
        rows = packed.to(device)
        module.ssm_prepare(rows[:, inner:], dt_raw.to(device), tap.to(device), conv_bias.to(device) if bias else None, kept, a_log=a_log.to(device), dt_bias=dt_bias.to(device),
                           groups=G, state=N, heads=H, vdim=V, **out, **{n: t.to(device) for n, t in where.items()})
        normed = torch.zeros(T, inner, dtype=dtype, device=device)
        y = (out["x"] * 0.7).flip(0).contiguous()
        module.ssm_gated_norm(y, out["x"], skip.to(device), rows[:, :inner], weight.to(device), 1e-5, normed, heads=H, vdim=V, norm_groups=parts)
        return out, kept, normed

    want, want_kept, want_normed = run(ssm_ref, "cpu")
    got, kept, normed = run(kernels, "cuda")
    for name in got:
        near(got[name], want[name])
    if taps > 1:
        near(kept, want_kept)
    near(normed, want_normed, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,H,V", [(1, 1, 128), (9, 3, 4), (33, 5, 100), (7, 2, 132), (5, 2, 6)])
@pytest.mark.parametrize("activation", ["silu", "sigmoid"])
def test_delta_gated_norm(T, H, V, activation, dtype):
    from kairyu_b200 import kernels

    g = torch.Generator().manual_seed(V)
    o, packed, weight = torch.randn(T, H * V, generator=g), torch.randn(T, H * V + 8, generator=g).to(dtype), torch.randn(V, generator=g)
    for offset in (0, 8):
        want, got = torch.zeros(T, H * V, dtype=dtype), torch.zeros(T, H * V, dtype=dtype, device="cuda")
        delta_ref.delta_gated_norm(o, packed, offset, weight, 1e-5, want, heads=H, vdim=V, gate_activation=activation)
        kernels.delta_gated_norm(o.cuda(), packed.cuda(), offset, weight.cuda(), 1e-5, got, heads=H, vdim=V, gate_activation=activation)
        near(got, want, dtype)
