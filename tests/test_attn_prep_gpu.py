"""The attention prologue's form for many heads (a warp per head) against its form for few (a block per head): the same sums in
the same order.  A rotation is two products and a sum in fp32, of which one product is rounded; for a pair's second value it is not the
same one beyond 4096 heads, so those results differ in fp16 by one step where they differ at all.  Cache rows of plain copies are equal bit for bit;
with the head norms in front, through a prompt, the two differ by what the projections' own summation order leaves in fp16."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,hq,hkv,rotary", [(129, 24, 4, 64), (300, 24, 4, 64), (700, 5, 1, 256), (4097, 1, 0, 0)])
def test_rope_rows_equal_pieces(rows, hq, hkv, rotary):
    import xinfer_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    q = torch.randn((rows, hq, 256), generator=g, device="cuda").half()
    k = torch.randn((rows, max(hkv, 1), 256), generator=g, device="cuda").half()
    pos = torch.randint(0, 9000, (rows,), generator=g, device="cuda")
    q1, k1 = q.clone(), k.clone()
    assert ops.rope(q1, k1 if hkv else None, rows, hq, hkv, 256, pos, 1.0e7, rotary) == 0
    for a in range(0, rows, 32):  # at most 1024 heads a call, value heads counted too
        n = min(32, rows - a)
        qa, ka, pa = q[a:a + n], k[a:a + n], pos[a:a + n].clone()
        assert ops.rope(qa, ka if hkv else None, n, hq, hkv, 256, pa, 1.0e7, rotary) == 0
    for whole, pieces in ((q1, q), (k1, k)):
        a, b = whole.double(), pieces.double()
        # |x| < 8: a product's fp32 rounding is below 2^-21; one fp16 step is at most 2^-10 of the value
        assert ((a - b).abs() <= 2.0 ** -10 * a.abs() + 2.0 ** -20).all()
        assert (a != b).double().mean() < 0.01  # (a last fp32 bit moves one fp16 rounding in some thousand)


def test_cache_rows_equal_pieces():
    import xinfer_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(3)
    k, v = (torch.randn((1500, 4, 256), generator=g, device="cuda").half() for _ in range(2))
    whole, pieces = ([torch.zeros((1600, 4, 256), device="cuda", dtype=torch.float16) for _ in range(2)] for _ in range(2))
    assert ops.attention_write_kv_cache(*whole, k, v, 7, 1500, 4, 256, 1600) == 0
    for a in range(0, 1500, 100):  # 800 heads a call
        assert ops.attention_write_kv_cache(*pieces, k[a:a + 100], v[a:a + 100], 7 + a, 100, 4, 256, 1600) == 0
    assert torch.equal(whole[0], pieces[0]) and torch.equal(whole[1], pieces[1])


def test_prompt_with_head_norms():
    from xinfer_b200.spec import Shape, SpecDecoder
    shape_cfg = Shape(hidden_size=512, intermediate_size=512, num_hidden_layers=4, num_attention_heads=24, num_key_value_heads=4,
                      vocab_size=1024, linear_num_v_heads=3, linear_num_k_heads=1)
    prompt = np.arange(121, dtype=np.int64) * 7 % 1024
    caches = []
    for batch in (1, 2):  # 120 x 32 and 240 x 32 heads
        dec = SpecDecoder(shape_cfg, batch=batch, k=3, max_seq=160, seed=4)
        dec.reset(0, seed=2)
        dec.prefill(np.stack([prompt] * batch))
        caches.append(dec.tensor(3, "k_cache", np.float16).reshape(batch, 160, 4, 256)[0, :120].astype(np.float64))
        dec.close()
    # a dozen fp16 roundings (2^-12 rms each, relative) in front of the cache
    assert np.sqrt(np.mean((caches[0] - caches[1]) ** 2) / np.mean(caches[0] ** 2)) < 12 ** 0.5 * 2.0 ** -11
