"""Either side of the line between a block per head and a warp per head where no head norms are asked for (1024 heads a call, value
heads counted too): whole calls against pieces far below it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [32, 33, 36, 37, 77, 128, 129, 300])  # of 24 + 4 + 4 heads: 1024, 1056, ..., 4096, 4128
def test_rope_against_short_pieces(cuda, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    q, k = (torch.randn((rows, h, 256), generator=g, device="cuda").half() for h in (24, 4))
    pos = torch.randint(0, 9000, (rows,), generator=g, device="cuda")
    q1, k1 = q.clone(), k.clone()
    assert cuda.rope(q1, k1, rows, 24, 4, 256, pos, 1.0e7, 64) == 0
    for a in range(0, rows, 9):
        n = min(9, rows - a)
        assert cuda.rope(q[a:a + n], k[a:a + n], n, 24, 4, 256, pos[a:a + n].clone(), 1.0e7, 64) == 0
    for whole, pieces in ((q1, q), (k1, k)):
        if rows <= 128:  # the same rounding in both forms; beyond 4096 heads the second value of a pair takes the other
            assert torch.equal(whole, pieces)
        a, b = whole.double(), pieces.double()
        # |x| < 8: the fp32 rounding of one product is below 2^-21; one fp16 step is 2^-10 of the value
        assert ((a - b).abs() <= 2.0 ** -10 * a.abs() + 2.0 ** -20).all()
        assert (a != b).double().mean() < 0.01


@pytest.mark.parametrize("rows", [128, 129, 512])  # of 8 slots: 1024, 1032, 4096
def test_cache_write_against_short_pieces(cuda, rows):
    g = torch.Generator(device="cuda").manual_seed(rows)
    k, v = (torch.randn((rows, 4, 256), generator=g, device="cuda").half() for _ in range(2))
    whole, pieces = ([torch.zeros((rows + 40, 4, 256), device="cuda", dtype=torch.float16) for _ in range(2)] for _ in range(2))
    assert cuda.attention_write_kv_cache(*whole, k, v, 7, rows, 4, 256, rows + 40) == 0
    for a in range(0, rows, 50):
        n = min(50, rows - a)
        assert cuda.attention_write_kv_cache(*pieces, k[a:a + n], v[a:a + n], 7 + a, n, 4, 256, rows + 40) == 0
    assert torch.equal(whole[0], pieces[0]) and torch.equal(whole[1], pieces[1])
