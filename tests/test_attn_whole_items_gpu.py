"""Attention over a prompt on either side of the lines where tiles are left whole: the number of keys that one tile, or the largest of several,
may have, also where blocks are few for the groups; as many tiles as there are groups of CTAs, and one more; batches of chunks by way of the decoder are in its own tests."""
import pytest

from test_attn_tiles_gpu import reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,T,start", [
    (24, 4, 21, 171), (24, 4, 21, 172),     # one tile, three and four blocks of keys
    (24, 4, 22, 171), (24, 4, 77, 0), (24, 4, 77, 499), (24, 4, 77, 500),  # four tiles, nine and ten blocks
    (24, 4, 777, 0), (24, 4, 778, 0),       # 37 tiles of 21 positions, 38
    (8, 2, 64, 384), (8, 2, 64, 385), (8, 2, 64, 512), (8, 2, 64, 513), (1, 1, 512, 0), (8, 8, 300, 100), (32, 1, 600, 3), (1, 1, 129, 0), (32, 1, 5, 130)])
def test_lines(hq, hkv, T, start):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(T + start)
    cap = start + T + 9
    q = torch.randn((T, hq, 256), generator=g, device="cuda").half()
    k, v = (torch.randn((cap, hkv, 256), generator=g, device="cuda").half() for _ in range(2))
    k[start + T:] = float("nan")
    v[start + T:] = float("nan")
    want = reference(torch, q, k, v, start)
    out = [torch.full((T, hq, 256), float("nan"), device="cuda", dtype=torch.float16) for _ in range(2)]
    for o in out:
        assert ops.sdpa_causal_cached(o, q, k, v, start, T, hq, hkv, 256, max_seq_len=cap) == 0
    torch.cuda.synchronize()
    assert ops.device_status(0) == 0
    assert torch.equal(out[0], out[1])
    got = out[0].float()
    # as in test_attention_tiles: probabilities and output are rounded to fp16 once each
    assert ((got - want).norm() / want.norm()).item() <= 2 * 2 ** -11
    rms = want.pow(2).mean().sqrt()
    assert ((got - want).abs() / torch.maximum(want.abs(), rms)).max().item() <= 8 * 2 ** -11
