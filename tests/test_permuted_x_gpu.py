"""Long launches of more than 16 activation rows have X written in the unpack's order by a small launch in front of them; the allocation-free
entry point never has.  The sums are the same in the same order, so the two agree to the bit on either side of the rule's lines."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [16, 17, 24, 31, 32])
@pytest.mark.parametrize("K,N", [
    (12160, 38144),   # 48 stages per CTA (the last of one group), 149 tiles on 148 SMs
    (12032, 38144),   # 47
    (12288, 37888),   # 148 tiles: none is cut
    (5120, 151936),   # an LM head
])
def test_same_bits_as_without(cuda, M, K, N):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8)
    s = torch.rand((N, K // 128), generator=g, device="cuda").mul_(0.01).half()
    x = torch.randn((M, K), generator=g, device="cuda").half()
    got, want = (torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16) for _ in range(2))
    for _ in range(2):  # (twice: the second call's copy of X follows the first call's reads of it)
        assert cuda.linear_int4(got, x, w, s, None, M, N, K) == 0
    assert cuda.linear_int4_noalloc(want, x, w, s, None, M, N, K) == 0
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    assert torch.equal(got, want) and not torch.isnan(got).any()


def test_uncut_launches_share_no_scratch(cuda):
    """7105 tiles of one stage: long enough for the rule, but no tile is cut, so that such launches may run on several streams at once."""
    M, K, N = 32, 256, 7105 * 256
    g = torch.Generator(device="cuda").manual_seed(3)
    w = torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8)
    s = torch.rand((N, K // 128), generator=g, device="cuda").mul_(0.01).half()
    xs = [torch.randn((M, K), generator=g, device="cuda").half() for _ in range(2)]
    want, got = ([torch.empty((M, N), device="cuda", dtype=torch.float16) for _ in range(2)] for _ in range(2))
    for x, y in zip(xs, want):
        assert cuda.linear_int4_noalloc(y, x, w, s, None, M, N, K) == 0
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    for _ in range(5):
        for stream, x, y in zip(streams, xs, got):
            with torch.cuda.stream(stream):
                assert cuda.linear_int4(y, x, w, s, None, M, N, K) == 0
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    assert all(torch.equal(a, b) for a, b in zip(want, got))


def test_x_written_by_the_launch_in_front(cuda):
    """The small launch starts while the norm in front of it, whose output it reads, still runs; every call has another X."""
    M, K, N = 32, 5120, 151936
    g = torch.Generator(device="cuda").manual_seed(9)
    w = torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8)
    s = torch.rand((N, K // 128), generator=g, device="cuda").mul_(0.01).half()
    norm_w = torch.randn(K, generator=g, device="cuda")
    xs = [torch.randn((M, K), generator=g, device="cuda").half() for _ in range(6)]
    normed = torch.empty_like(xs[0])
    got, want = ([torch.empty((M, N), device="cuda", dtype=torch.float16) for _ in xs] for _ in range(2))
    for x, y in zip(xs, got):
        assert cuda.rmsnorm(normed, x, norm_w, M, K) == 0
        assert cuda.linear_int4(y, normed, w, s, None, M, N, K) == 0
    for x, y in zip(xs, want):
        assert cuda.rmsnorm(normed, x, norm_w, M, K) == 0
        torch.cuda.synchronize()
        assert cuda.linear_int4_noalloc(y, normed, w, s, None, M, N, K) == 0
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    assert all(torch.equal(a, b) for a, b in zip(want, got))
