"""The delta-rule kernel of a decoder step in its four forms: a thread block per head with all of its state in flight or, with
more heads than SMs, several heads per SM; up to four tokens a sequence or up to eight.  Steps with forced drafts against the
CPU oracle, so that all, some and none of the pending updates are replayed; integer results exact, fp16 rows within the few
roundings by which two fp32 summation orders differ (the bound of the other step tests)."""
import numpy as np
import pytest
import torch

from test_spec_decoder_gpu import compare_step, pull_model, pull_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,k,v_heads,k_heads", [(1, 3, 6, 2), (2, 4, 6, 2), (4, 3, 48, 16), (4, 4, 40, 8), (3, 1, 51, 17), (1, 7, 3, 1)])
def test_step_forms_match_oracle(batch, k, v_heads, k_heads):
    from xinfer_b200.spec import Shape, SpecDecoder
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    shape_cfg = Shape(hidden_size=512, intermediate_size=512, num_hidden_layers=4, num_attention_heads=4, num_key_value_heads=2,
                      vocab_size=2048, linear_num_v_heads=v_heads, linear_num_k_heads=k_heads)
    dec = SpecDecoder(shape_cfg, batch=batch, k=k, max_seq=96, seed=17)
    dec.reset(9, seed=6)
    model = pull_model(dec, shape_cfg, k)
    seqs = pull_state(dec, model, shape_cfg, batch, dec.max_seq)
    for keep in (k, 0, k // 2, k):
        overrides = []
        for b in range(batch):
            cont = model.greedy_continuation(seqs[b], k)
            if keep < k:
                cont[keep] = (cont[keep] + 1 + b) % shape_cfg.vocab_size
            overrides.append(cont)
        assert compare_step(dec, model, seqs, shape_cfg, overrides, tag=f"keep{keep}") == [keep] * batch
    dec.close()


@pytest.mark.parametrize("batch,k", [(1, 7), (3, 4)])
def test_drafts_across_a_key_block(batch, k):
    """The head's context length grows with every draft and here passes a multiple of 64 keys inside a step, on a model so small
    that several launches of a draft pass are on the GPU at once: eager and replayed steps give the same drafts, logits and
    hidden rows, and the eager ones the oracle's."""
    from xinfer_b200.spec import Shape, SpecDecoder
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    shape_cfg = Shape(hidden_size=512, intermediate_size=512, num_hidden_layers=4, num_attention_heads=4, num_key_value_heads=2,
                      vocab_size=2048, linear_num_v_heads=6, linear_num_k_heads=2)
    dec = SpecDecoder(shape_cfg, batch=batch, k=k, max_seq=256, seed=3)
    dec.reset(59, seed=8)
    model = pull_model(dec, shape_cfg, k)
    seqs = pull_state(dec, model, shape_cfg, batch, dec.max_seq)
    for i in range(3):
        compare_step(dec, model, seqs, shape_cfg, tag=f"step{i}")

    def run(graph):
        dec.reset(59, seed=8)
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            if graph:
                dec.capture(stream)        # (one eager step, then the capture)
            else:
                dec.step()
            got = [dec.results()]
            for _ in range(12):
                dec.step()
                got.append(dec.results())
        torch.cuda.synchronize()
        return got
    for (e0, n0), (e1, n1) in zip(run(False), run(True)):
        assert np.array_equal(e0, e1) and np.array_equal(n0, n1)
    dec.close()
