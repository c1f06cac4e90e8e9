"""The log-probability report at the sizes where its chunks change form: one entry, a chunk that ends with a
block's width, 16 and 32 entries a thread, and more chunks than a block has threads."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,k", [(1, 2), (255, 3), (257, 3), (8192, 1), (131072, 5), (131073, 5), (262145, 4), (2200001, 3)])
def test_report_over_chunk_sizes(V, k):
    from kairyu_b200 import kernels

    logits = torch.randn(2, V, generator=torch.Generator().manual_seed(V)) * 3.0
    logits[0, V // 2] = logits[0, V - 1] = 40.0  # a tie across chunks: the lower index comes first
    logits[1, : V // 3] = -float("inf")  # a masked stretch, with whole chunks of it
    tokens = torch.tensor([V - 1, V // 2], dtype=torch.int32)
    values = torch.full((2, k + 1), float("nan"), device="cuda")
    indices = torch.full((2, k), -7, dtype=torch.int32, device="cuda")
    kernels.logprob_report(logits.cuda(), torch.tensor([0, 1], dtype=torch.int32, device="cuda"), tokens.cuda(), k, values, indices, tokens_by_row=True)
    logp = torch.log_softmax(logits.double(), dim=-1)
    have = min(k, V)
    best, order = torch.sort(logp, dim=-1, descending=True, stable=True)
    # a thread adds at most 32 terms, then 8 warps and V / 8192 chunks are added in turn: some 320 roundings of
    # 2^-24 of the sum at the longest, and as much again for the exponentials
    bound = 4e-5
    for r in range(2):
        assert abs(float(values[r, 0]) - float(logp[r, tokens[r]])) < bound
        assert indices[r, :have].tolist() == order[r, :have].tolist()
        assert (values[r, 1 : 1 + have].cpu().double() - best[r, :have]).abs().max() < bound
        assert (indices[r, have:] == -1).all()
