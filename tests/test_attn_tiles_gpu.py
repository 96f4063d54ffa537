"""Attention over the cache at the sizes where its tiling can go wrong: one 64-key block and its neighbours, one tile and the next,
tiles that are not full, tiles cut between CTAs, score ranges that rescale the accumulator, group sizes that do not divide a
tile, and NaN in the cache behind the last key.  Against fp32 PyTorch."""
import pytest

pytestmark = pytest.mark.gpu


def reference(torch, q, k, v, start):
    T, hq, _ = q.shape
    n = start + T
    kk, vv = (x[:n].float().repeat_interleave(hq // x.shape[1], 1) for x in (k, v))
    s = torch.einsum("thd,nhd->htn", q.float(), kk) / 16
    late = torch.arange(n, device="cuda")[None, :] > (start + torch.arange(T, device="cuda"))[:, None]
    return torch.einsum("htn,nhd->thd", s.masked_fill(late[None], float("-inf")).softmax(-1), vv)


@pytest.mark.parametrize("hq,hkv,T,start,amp", [
    (24, 4, 1, 0, 1), (24, 4, 1, 62, 1), (24, 4, 1, 63, 1), (24, 4, 1, 64, 1), (24, 4, 5, 127, 1), (24, 4, 6, 3000, 8),
    (24, 4, 21, 5, 1), (24, 4, 22, 43, 3), (24, 4, 59, 128, 1), (24, 4, 200, 333, 8), (8, 8, 130, 70, 1), (32, 1, 40, 20, 1),
    (12, 2, 5, 2000, 10), (10, 2, 27, 900, 1)])
def test_attention_tiles(hq, hkv, T, start, amp):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(T + start)
    cap = start + T + 9
    q = (torch.randn((T, hq, 256), generator=g, device="cuda") * amp).half()
    k, v = (torch.randn((cap, hkv, 256), generator=g, device="cuda").half() for _ in range(2))
    k[start + T:] = float("nan")
    v[start + T:] = float("nan")
    want = reference(torch, q, k, v, start)
    for lead in (0, 1):  # an output of 16-byte and of 2-byte alignment
        out = torch.full((T * hq * 256 + lead,), float("nan"), device="cuda", dtype=torch.float16)[lead:]
        assert ops.sdpa_causal_cached(out, q, k, v, start, T, hq, hkv, 256, max_seq_len=cap) == 0
        torch.cuda.synchronize()
        assert ops.device_status(0) == 0
        got = out.view(T, hq, 256).float()
        # probabilities and output are rounded to fp16 once each, 2^-11 at most and a third of that in the 2-norm (one element: at most
        # the two roundings, relative to a value or the rms, whichever is larger, times the few sigma of a 256-term tail)
        assert ((got - want).norm() / want.norm()).item() <= 2 * 2 ** -11
        rms = want.pow(2).mean().sqrt()
        assert ((got - want).abs() / torch.maximum(want.abs(), rms)).max().item() <= 8 * 2 ** -11


@pytest.mark.parametrize("T,start", [(1, 3000), (200, 333)])
def test_attention_wait_runs_out_and_is_reported(T, start):
    """The loader withholds the queries: the launch comes back, the merge behind it stays inside its buffers although the table of
    parts was not written, the status reports it once, and the next call is right."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    from xinfer_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(T)
    q = torch.randn((T, 24, 256), generator=g, device="cuda").half()
    k, v = (torch.randn((start + T, 4, 256), generator=g, device="cuda").half() for _ in range(2))

    def call():
        out = torch.full((T, 24, 256), float("nan"), device="cuda", dtype=torch.float16)
        assert ops.sdpa_causal_cached(out, q, k, v, start, T, 24, 4, 256) == 0
        torch.cuda.synchronize()
        return out
    good = call()
    ops.set_wait_hooks(8_000_000, 0)           # about 4 ms
    try:
        call()
    finally:
        ops.set_wait_hooks(0, -1)
    assert ops.device_status(0) == _lib.ERR_DEVICE_TIMEOUT
    assert torch.equal(call(), good)
    assert ops.device_status(0) == 0


@pytest.mark.parametrize("hq,hkv,T,start", [(24, 4, 1, 1023), (8, 2, 1, 1099), (24, 4, 5, 3000), (24, 4, 77, 0), (12, 2, 22, 900)])
def test_attention_repeats_itself(hq, hkv, T, start):
    """The same call gives the same bits whatever ran in between, and a position the same as in a call without those behind it
    where both cut the keys alike (one block)."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(T)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda").half()  # noqa: E731
    q, k, v = 3 * rand(T, hq, 256), rand(start + T, hkv, 256), rand(start + T, hkv, 256)

    def call(q, k, v, T, start):
        out = torch.full((T, hq, 256), float("nan"), device="cuda", dtype=torch.float16)
        assert ops.sdpa_causal_cached(out, q, k, v, start, T, hq, hkv, 256) == 0
        return out
    first = call(q, k, v, T, start)
    for i in range(12):
        for other in (1, 3, 40):  # (other contents of the kernel's shared memory)
            call((2 + i) * rand(other, hq, 256), (1 + i) * rand(500, hkv, 256), rand(500, hkv, 256), other, 500 - other)
        assert torch.equal(call(q, k, v, T, start), first), i
    few = min(T, 5)
    short = call(q[:few].contiguous(), k, v, few, 20)
    for t in range(few):
        assert torch.equal(call(q[t:t + 1].contiguous(), k, v, 1, 20 + t)[0], short[t]), t
