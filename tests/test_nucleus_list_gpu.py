"""The nucleus from its list of candidates: as many candidates as the leader block selects alone, one more, as many as the list holds,
one more; ties at the threshold; a row whose tokens all weigh the same."""
import math

import numpy as np
import pytest
import torch

from oracle.model import nucleus, sample_token_top_p

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
        key, w, thr, z = nucleus(logits[r], 1.0, top_p)
        w = np.where(key >= np.uint32(thr), w, np.uint64(0)).astype(np.int64)
        want, _ = sample_token_top_p(logits[r], 1.0, top_p, u[r])
        got = int(tok[r])
        # exp's last bits differ between the device and numpy, less than 2^-21 of a weight: a draw that near the boundary of two members may take
        # the other one.  (Row 0: the maximum is every candidate's value, its weight exact.)
        if got != want:
            assert r > 0 and w[got] > 0
            end, t = np.cumsum(w)[got], math.floor(float(u[r]) * z)
            slack = 1 + z // 2 ** 21
            assert end - w[got] - slack <= t <= end + slack
        assert abs(float(prob[r]) - w[got] / z) <= 1e-6 * w[got] / z
