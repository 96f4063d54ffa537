"""The top-p kernel's ways to the threshold - a short candidate list, a longer one, a list that overflows, a row that does not
fit the registers - by the shape of the distribution and the size of the vocabulary; against the oracle's restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V,sigma,peaks,top_p", [
    (151936, 2.0, 40, 0.9), (151936, 4.0, 0, 0.5), (151936, 3.0, 0, 0.9), (151936, 0.5, 0, 0.9), (163840, 2.0, 40, 0.95),
    (163841, 2.0, 40, 0.9), (200001, 3.0, 0, 0.9), (33, 1.0, 0, 0.7), (8191, 5.0, 0, 0.999)])
def test_top_p_by_every_way(V, sigma, peaks, top_p):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    from oracle.model import nucleus, sample_token_top_p
    rng = np.random.default_rng(V)
    rows = 3
    logits = rng.normal(0, sigma, (rows, V)).astype(np.float32)
    for r in range(rows):
        logits[r, rng.integers(0, V, peaks)] = rng.uniform(8, 12, peaks).astype(np.float32)
    u = rng.uniform(0, 1, rows).astype(np.float32)
    tok, prob = torch.empty(rows, dtype=torch.int64, device="cuda"), torch.empty(rows, device="cuda")
    inv_t = float(np.float32(1 / 0.7))
    assert ops.sample_tokens_top_p(torch.from_numpy(logits).cuda(), torch.from_numpy(u).cuda(), tok, prob, inv_t, top_p) == 0
    for r in range(rows):
        key, w, thr, z = nucleus(logits[r], inv_t, top_p)
        want_t, want_p = sample_token_top_p(logits[r], inv_t, top_p, u[r])
        got = int(tok[r])
        if got != want_t:
            # exp's last bit differs between the two sides: allowed where the draw lies within 1e-6 of a boundary
            cum = np.cumsum(np.where(key >= np.uint32(thr), w, 0).astype(np.float64))
            assert np.min(np.abs(cum - float(u[r]) * z)) <= 1e-6 * z, (r, got, want_t)
        else:
            assert abs(float(prob[r]) - want_p) <= 1e-5 * want_p
