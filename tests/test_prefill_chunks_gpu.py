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


def test_chunks_leave_the_device_most_of_its_memory(cuda):
    """Buffers for more than 512 rows take a quarter of the free memory at most, their own block, which they replace, counted as free;
    with less, chunks are halved, down to 512 rows whatever that leaves."""
    from xinfer_b200.spec import Shape, SpecDecoder
    shape_cfg = Shape(hidden_size=512, intermediate_size=512, num_hidden_layers=4, num_attention_heads=8, num_key_value_heads=2,
                      vocab_size=1024, linear_num_v_heads=3, linear_num_k_heads=1)
    batch, tokens = 4, 1025  # 4096 rows
    prompts = np.random.default_rng(1).integers(0, 1024, size=(batch, tokens)).astype(np.int64)
    dec = SpecDecoder(shape_cfg, batch=batch, k=3, max_seq=tokens + 32, seed=4)

    def run(free):
        dec.set_chunk_hooks(free_bytes=free)
        dec.reset(0, seed=2)
        dec.prefill(prompts)
        return dec.info(8), dec.info(9), dec.tensor(-1, "h_last", np.float16).astype(np.float64)

    chunks, bytes_512, want = run(1)
    assert chunks == 8
    free = 4 * bytes_512
    seen = {}
    while chunks > 1:  # (a little more free memory each time: the chunks get longer one step after the other)
        chunks, taken, got = run(free)
        assert chunks in (1, 2, 4, 8) and chunks <= min(seen, default=8)
        if chunks not in seen and chunks < 8:
            assert 4 * taken <= free + max(seen.values(), default=bytes_512)
            seen[chunks] = taken
        # a few dozen fp16 roundings (2^-12 rms each, relative) on the way, whose sums come in another order
        assert np.sqrt(np.mean((got - want) ** 2) / np.mean(want ** 2)) < 36 ** 0.5 * 2.0 ** -11
        free += free // 8
    assert sorted(seen) == [1, 2, 4]
    assert run(1)[:2] == (1, seen[1])  # (buffers that are there already are used)
    dec.close()
    assert cuda.device_status(0) == 0


@pytest.mark.parametrize("hidden", [2176, 5120])
@pytest.mark.parametrize("most_rows", [32, 64, 112, 240, 304, 592])
def test_norms_of_a_chunk_by_its_rows(cuda, hidden, most_rows):
    """The embedding norm and the two-job norm of a chunk in every form the number of rows gives them, against one chunk of 900 rows (two vectors
    a thread): caches of the first attention layer and of the draft head, which the second one's output goes straight into."""
    from xinfer_b200.spec import Shape, SpecDecoder
    shape_cfg = Shape(hidden_size=hidden, intermediate_size=512, num_hidden_layers=4, num_attention_heads=8, num_key_value_heads=2,
                      vocab_size=1024, linear_num_v_heads=3, linear_num_k_heads=1)
    prompt = np.random.default_rng(1).integers(0, 1024, size=(1, 901)).astype(np.int64)
    dec = SpecDecoder(shape_cfg, batch=1, k=3, max_seq=932, seed=4)
    runs = []
    for rows in (0, most_rows):
        dec.set_chunk_hooks(most_rows=rows)
        dec.reset(0, seed=2)
        dec.prefill(prompt)
        got = {"h_last": dec.tensor(-1, "h_last", np.float16).astype(np.float64)}
        for layer, name in ((3, "k_cache"), (3, "v_cache"), (4, "k_cache"), (4, "v_cache")):
            got[layer, name] = dec.tensor(layer, name, np.float16).reshape(932, -1)[:900].astype(np.float64)
        runs.append((dec.info(8), got))
    dec.close()
    (one, want), (many, got) = runs
    assert one == 1 and many == -(-900 // most_rows)
    for name in want:
        # a few dozen fp16 roundings (2^-12 rms each, relative) on the way, whose sums come in another order
        err = np.sqrt(np.mean((got[name] - want[name]) ** 2) / np.mean(want[name] ** 2))
        assert err < 36 ** 0.5 * 2.0 ** -11, name
    assert cuda.device_status(0) == 0
