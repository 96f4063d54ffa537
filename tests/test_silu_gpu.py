"""x / (1 + exp(-x)) as the convolution and gate/up finish it: the same bits as that expression in fp32 with an exact division (torch's,
which calls the same expf), rounded to fp16, whichever kernel a call's rows take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TC, SIMT, GEMM = 1, 2, 3


def silu(x):
    return x / (1.0 + torch.exp(-x))


@pytest.mark.parametrize("rows", [1, 9])
@pytest.mark.parametrize("channels", [1 << 20, (1 << 18) + 1])
def test_convolution(cuda, rows, channels):
    """The fourth weight of a channel is the value, its input 1, the other weights 0: any fp32 value reaches the SiLU."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.empty(channels, device="cuda")
    x.normal_(0, 3, generator=g)
    x[: channels // 4].uniform_(-100, 100, generator=g)
    bits = torch.randint(0, 1 << 32, (channels // 4,), generator=g, device="cuda", dtype=torch.int64)
    x[-(channels // 4):] = (bits - (1 << 31)).to(torch.int32).view(torch.float32)
    ends = [0.0, float("inf"), float("-inf"), 3e38, -3e38, 1e-45, -1e-45, -40.0, -87.3, -87.4, -88.7, -88.8, -103.9, -104.1, 88.8]
    x[:len(ends)] = torch.tensor(ends, device="cuda")
    w = torch.zeros((channels, 4), device="cuda")
    w[:, 3] = x
    out = torch.empty((rows, channels), dtype=torch.float16, device="cuda")
    assert cuda.causal_conv1d_silu(out, torch.ones_like(out), w, rows, None, channels) == 0
    want = silu(x + 0.0).half()  # (0 * 0 + -0 is 0)
    assert torch.equal(torch.isnan(out[0]), torch.isnan(want))
    want = want.nan_to_num(7.0)
    for r in range(rows):
        assert torch.equal(out[r].nan_to_num(7.0), want)


@pytest.mark.parametrize("M,path", [(1, TC), (8, TC), (12, TC), (16, TC), (32, TC), (5, SIMT), (40, GEMM), (77, GEMM), (129, GEMM), (256, GEMM)])
@pytest.mark.parametrize("N", [264, 17408])  # clusters that split K; one uncut tile per CTA
def test_gate_up(cuda, M, path, N):
    """One weight a row is not zero: gate and up are products of an activation and a scale, exact in fp32."""
    K = 1024
    g = torch.Generator(device="cuda").manual_seed(M)
    wg, wu = (torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda") for _ in range(2))
    wg[:, 0], wu[:, 0] = 0x01, 0x10
    sg, su = ((torch.rand((N, K // 128), generator=g, device="cuda") * 2).half() for _ in range(2))
    x = (torch.randn((M, K), generator=g, device="cuda") * 3).half()
    x[0, 0] = -88.0  # (products to -176)
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    cuda.set_linear_path(path)
    try:
        assert cuda.mlp_gate_up_swiglu_int4(y, x, wg, sg, wu, su, M, N, K) == 0
        assert cuda.last_linear_path() == path
    finally:
        cuda.set_linear_path(0)
    gate, up = (x[:, i:i + 1].float() * s[:, 0].float() for i, s in ((0, sg), (1, su)))
    assert torch.equal(y.float(), (silu(gate) * up).half().float())
