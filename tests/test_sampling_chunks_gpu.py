"""The merge of a row's chunk partials by the plain draw: as many chunks as threads at most, one more (a vocabulary beyond a million),
and a chunk that holds a single number."""
import numpy as np
import pytest
import torch

from oracle.model import sample_token

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [1, 31, 4096, 4097, 256 * 4096, 256 * 4096 + 1])
@pytest.mark.parametrize("inv_t", [1.0, 1.0 / 0.7])
def test_draw_over_chunks(cuda, vocab, inv_t):
    rng = np.random.default_rng(vocab)
    rows = 3
    logits = rng.normal(0, 2, size=(rows, vocab)).astype(np.float32)
    if vocab > 4096:
        logits[1, :4095] = -np.inf          # a chunk of one token in front
    u = rng.random(rows).astype(np.float32)
    tok, prob = torch.empty(rows, dtype=torch.int64, device="cuda"), torch.empty(rows, device="cuda")
    assert cuda.sample_tokens(torch.from_numpy(logits).cuda(), torch.from_numpy(u).cuda(), tok, prob, inv_t) == 0
    torch.cuda.synchronize()
    for r in range(rows):
        l = np.maximum(logits[r] * np.float32(inv_t), np.float32(-1e30)).astype(np.float64)
        w = np.exp(l - l.max())
        cdf = np.cumsum(w) / w.sum()
        t = int(tok[r])
        # sums of at most 2^21 positive terms in two levels of fp32: the draw lies within 1e-4 of the token's range
        assert (cdf[t - 1] if t else 0.0) - 1e-4 <= u[r] <= cdf[t] + 1e-4
        assert abs(float(prob[r]) - w[t] / w.sum()) <= 1e-4 * w[t] / w.sum()
    if vocab <= 4097 and vocab > 1:
        want, _ = sample_token(logits[0], inv_t, u[0])
        assert int(tok[0]) == want


def test_argmax_passes_chunks_without_a_number_and_keeps_the_lowest_index(cuda):
    logits = torch.full((2, 9000), -float("inf"), device="cuda")
    logits[0, [5000, 8999]] = 3.0
    out = torch.empty(2, dtype=torch.int64, device="cuda")
    assert cuda.argmax_rows(logits, out) == 0
    assert out.tolist() == [5000, 0]
