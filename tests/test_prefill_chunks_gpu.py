"""A prompt whose rows do not fit one chunk: the last hidden states and the caches are those of one sequence by itself, which does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,tokens", [
    (8, 601),   # two chunks of 304 and 296 positions
    (5, 1701),  # three: 576, 576 and 548
])
def test_chunks_against_one_sequence(cuda, batch, tokens):
    from xinfer_b200.spec import Shape, SpecDecoder
    shape_cfg = Shape(hidden_size=512, intermediate_size=512, num_hidden_layers=4, num_attention_heads=8, num_key_value_heads=2,
                      vocab_size=1024, linear_num_v_heads=3, linear_num_k_heads=1)
    prompts = np.random.default_rng(batch).integers(0, 1024, size=(batch, tokens)).astype(np.int64)
    rows = tokens + 32

    def run(p):
        dec = SpecDecoder(shape_cfg, batch=len(p), k=3, max_seq=rows, seed=4)
        dec.reset(0, seed=2)
        dec.prefill(p)
        got = {"h_last": dec.tensor(-1, "h_last", np.float16).reshape(len(p), -1).astype(np.float64)}
        for layer, name in ((3, "k_cache"), (3, "v_cache"), (4, "k_cache")):  # (layer 4: the draft head's)
            got[layer, name] = dec.tensor(layer, name, np.float16).reshape(len(p), rows, -1)[:, :tokens - 1].astype(np.float64)
        dec.close()
        return got

    whole = run(prompts)
    for b in (0, batch - 1):
        one = run(prompts[b:b + 1])
        for name in one:
            # a few dozen fp16 roundings (2^-12 rms each, relative) on the way, whose sums come in another order
            err = np.sqrt(np.mean((whole[name][b] - one[name][0]) ** 2) / np.mean(one[name][0] ** 2))
            assert err < 36 ** 0.5 * 2.0 ** -11, name
    assert cuda.device_status(0) == 0
