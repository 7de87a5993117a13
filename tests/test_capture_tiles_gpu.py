"""Controller statistics at the edges of their 128 x 64 tiles, with running tiles moved by TMA (T a multiple of 4) and by
plain copies, and with more samples than one unit of work holds; two batches, so that the second one merges."""
import pytest
import torch

from oracle import saf_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [2, 4, 32, 63, 64, 65, 127, 128, 132, 193, 260])
@pytest.mark.parametrize("B,hd", [(1, 64), (4, 128), (6, 64), (9, 64)])
def test_statistics_tiles(T, B, hd):
    from saf_b200.capture import AttentionMoments, LogitMoments
    U = 2
    gen = torch.Generator().manual_seed(T + B)
    acc = AttentionMoments(U, T, "cuda")
    lg, lm = LogitMoments(U, T, "cuda", with_var=True), LogitMoments(U, T, "cuda")
    state, lstate, negent = (0, None, None), (0, None, None), torch.zeros(U, dtype=torch.float64)
    for n in (B, 2):
        q = torch.randn(n, U, T, hd, generator=gen).bfloat16()
        k = torch.randn(n, U, T, hd, generator=gen).bfloat16()
        att, raw = O.attention_probs(q.double(), k.double()), O.raw_logits(q.double(), k.double())
        state = O.merge_reduced_moments(*state, *O.centered_batch_reduced_moments(att))
        lstate = O.merge_moments(*lstate, *O.centered_batch_moments(raw))
        negent += O.negative_entropy_sum(att)
        for m in (acc, lg, lm):
            m.update(q.cuda(), k.cuda())
    # scores: exact bf16 products summed in fp32; probabilities: the exponential's and the log-sum-exp's fp32 rounding
    # (2^-24 relative to exponents of up to about 10, so a few 1e-6 of a probability)
    assert O.max_abs(acc.mean.cpu().double(), state[1]) <= 1e-4
    assert not acc.mean.triu(1).any()
    assert ((acc.head_m2.cpu() - state[2]).abs() <= 1e-3 * state[2].abs() + 1e-9).all()
    assert ((acc.neg_entropy.cpu() - negent).abs() <= 1e-3 * negent.abs() + 1e-4).all()
    assert torch.equal(lg.mean, lm.mean)
    assert O.max_abs(lg.mean.cpu().double(), lstate[1]) <= 2e-5
    assert O.max_abs(lg.m2.cpu().double(), lstate[2]) <= 1e-4 * lstate[2].abs().max().item()
