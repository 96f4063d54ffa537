"""The fp32 linear at the edges of its tiles (32 weight rows, 8 activation rows) and of its cut over K (clusters of one to eight
CTAs, groups that do not fill the warps), with activations over a wide range; fused and SwiGLU forms.  Against fp64."""
import pytest

pytestmark = pytest.mark.gpu


def weights(torch, g, n, k):
    w = torch.randint(0, 256, (n, k // 2), generator=g, device="cuda", dtype=torch.uint8)
    s = (torch.randn((n, k // 128), generator=g, device="cuda").abs() * 0.02 / 7).half()
    q = torch.stack([w & 15, w >> 4], -1).reshape(n, k).double()
    q = torch.where(q > 7, q - 16, q)
    return w, s, (q.view(n, -1, 128) * s.double()[..., None]).view(n, k)


@pytest.mark.parametrize("M,K,N", [(1, 128, 1), (1, 128, 32), (7, 256, 33), (8, 1024, 31), (9, 1152, 65), (17, 5120, 100), (2, 17408, 96), (33, 640, 5000)])
def test_linear_f32(M, K, N):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    x = torch.randn((M, K), generator=g, device="cuda") * torch.exp(3 * torch.randn((M, K), generator=g, device="cuda"))
    bias = torch.randn(N, generator=g, device="cuda")
    (w, s, d), (w2, s2, d2) = weights(torch, g, N, K), weights(torch, g, N, K)
    rel = lambda got, want: ((got.double() - want).norm() / want.norm()).item()  # noqa: E731
    # fp32 sums of K products: 2^-24 each step, growing with the root of the number of steps (128 in a group, then the groups)
    bound = 2 ** -24 * (128 + K / 128) ** 0.5 * 2
    y = torch.full((M, N), float("nan"), device="cuda")
    assert ops.linear_int4(y, x, w, s, bias, M, N, K) == 0
    assert rel(y, x.double() @ d.T + bias.double()) <= bound
    ys = [torch.full((M, N), float("nan"), device="cuda") for _ in range(2)]
    assert ops.linear_int4_fused(x, [{"Y": ys[0], "W_int4": w, "scales": s, "N": N}, {"Y": ys[1], "W_int4": w2, "scales": s2, "N": N}], M, K) == 0
    assert rel(ys[0], x.double() @ d.T) <= bound and rel(ys[1], x.double() @ d2.T) <= bound
    x /= x.abs().amax()  # (so that the gate neither vanishes nor overflows)
    assert ops.mlp_gate_up_swiglu_int4(y, x, w, s, w2, s2, M, N, K) == 0
    gate = x.double() @ d.T
    assert rel(y, gate / (1 + torch.exp(-gate)) * (x.double() @ d2.T)) <= 4 * bound


@pytest.mark.parametrize("M,K,N", [(8, 5120, 512), (8, 6144, 512), (2, 17408, 640)])
@pytest.mark.parametrize("spread", [0.0, 3.0])
def test_linear_f32_is_as_close_as_a_chain_of_fmas(M, K, N, spread):
    """Error against 64 bits beside that of fp32 arithmetic in the reference's association - a chain of 128 fused multiply-adds per
    group, a chain over the groups - for activations of one magnitude and of many; mean of four draws."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    ours, chain = 0.0, 0.0
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(seed + K)
        x = torch.randn((M, K), generator=g, device="cuda") * torch.exp(spread * torch.randn((M, K), generator=g, device="cuda"))
        w, s, d = weights(torch, g, N, K)
        y = torch.empty((M, N), device="cuda")
        assert ops.linear_int4(y, x, w, s, None, M, N, K) == 0
        want = x.double() @ d.T
        sd = s.double()
        q = torch.round(d.view(N, -1, 128) / sd.clamp_min(1e-9)[..., None])          # the integers
        xg, dot = x.double().view(M, 1, -1, 128), torch.zeros((M, N, K // 128), device="cuda", dtype=torch.float64)
        for i in range(128):
            dot = (dot + xg[..., i] * q[None, ..., i]).float().double()              # a product is exact in 64 bits: one rounding
        acc = torch.zeros((M, N), device="cuda", dtype=torch.float64)
        for j in range(K // 128):
            acc = (acc + dot[..., j] * sd[:, j]).float().double()
        ours += ((y.double() - want).norm() / want.norm()).item()
        chain += ((acc - want).norm() / want.norm()).item()
    assert ours <= 1.25 * chain, (ours / 4, chain / 4)


def test_linear_f32_carries_infinities_and_nan():
    """An infinite activation gives infinities of the weights' signs, as fp32 arithmetic does, NaN gives NaN, the largest finite
    values neither; other rows stay untouched."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    M, K, N = 6, 256, 40
    g = torch.Generator(device="cuda").manual_seed(1)
    w, s, d = weights(torch, g, N, K)
    w[w & 0x0F == 0] |= 0x01            # (no zero weights: infinity times zero is NaN)
    w[w & 0xF0 == 0] |= 0x10
    q = torch.stack([w & 15, w >> 4], -1).reshape(N, K).double()
    d = (torch.where(q > 7, q - 16, q).view(N, -1, 128) * s.double()[..., None]).view(N, K)
    x = torch.randn((M, K), generator=g, device="cuda")
    x[1, 5], x[2, 200], x[3, 7] = float("inf"), float("-inf"), float("nan")
    x[4, 9] = torch.tensor(0x7F800001, dtype=torch.int32, device="cuda").view(torch.float32)   # a NaN whose leading half is an infinity's
    x[5] *= 1e36
    y = torch.empty((M, N), device="cuda")
    assert ops.linear_int4(y, x, w, s, None, M, N, K) == 0
    want = x.double() @ d.T
    assert torch.equal(y[1:3].double(), want[1:3]) and torch.isinf(y[1:3]).all()
    assert torch.isnan(y[3:5]).all()
    for r in (0, 5):
        assert ((y[r].double() - want[r]).norm() / want[r].norm()).item() <= 2 ** -24 * (128 + K / 128) ** 0.5 * 2
    silu = torch.empty((3, N), device="cuda")
    assert ops.mlp_gate_up_swiglu_int4(silu, x[:3].contiguous(), w, s, w, s, 3, N, K) == 0
    gate = y[1:3]
    assert torch.equal(silu[1:3].isnan(), (gate / (1 + torch.exp(-gate)) * gate).isnan())
