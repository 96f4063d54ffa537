"""The nucleus from its list of candidates: as many candidates as the leader block selects alone, one more, as many as the list holds,
one more; ties at the threshold; a row whose tokens all weigh the same."""
import numpy as np
import pytest
import torch

from oracle.model import sample_token_top_p

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 255, 256, 257, 4096, 4097])
@pytest.mark.parametrize("top_p", [0.3, 0.9, 1.0])
def test_candidate_counts(cuda, n, top_p):
    rng = np.random.default_rng(n)
    vocab, rows = 20000, 4
    logits = np.full((rows, vocab), -90.0, np.float32)     # weight zero beside the candidates
    for r in range(rows):
        at = rng.permutation(vocab)[:n]
        logits[r, at] = rng.uniform(4.0, 4.9, n).astype(np.float32) if r else 4.0   # within one of the maximum; row 0: all the same
        if r == 1 and n > 4:
            logits[r, at[: n // 2]] = logits[r, at[0]]      # half of them tied
    u = np.array([0.0, 0.25, 0.7, 0.999999], np.float32)
    tok, prob = torch.empty(rows, dtype=torch.int64, device="cuda"), torch.empty(rows, device="cuda")
    assert cuda.sample_tokens_top_p(torch.from_numpy(logits).cuda(), torch.from_numpy(u).cuda(), tok, prob, 1.0, top_p) == 0
    torch.cuda.synchronize()
    for r in range(rows):
        want, p = sample_token_top_p(logits[r], 1.0, top_p, u[r])
        got = int(tok[r])
        # exp's last bit differs between the device and numpy: a draw on the boundary of two tokens may take the neighbour
        if got != want:
            ids = np.flatnonzero(logits[r] > 0)
            assert abs(int(np.searchsorted(ids, got)) - int(np.searchsorted(ids, want))) == 1
        else:
            assert abs(float(prob[r]) - p) <= 1e-6 * p
