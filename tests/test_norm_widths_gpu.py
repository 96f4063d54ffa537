"""RMSNorm with one 8-element vector a thread (few rows, or narrow ones), with two and with up to four: on either side of the lines between them, at
widths that leave the last warp, or the last vector, incomplete, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3, 148, 149, 600])
@pytest.mark.parametrize("hidden", [8, 264, 1000, 1028, 2040, 2048, 2056, 5120, 8192, 8200, 8200 * 2])
def test_rows_and_widths(cuda, rows, hidden):
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    x = torch.randn((rows, hidden), generator=g, device="cuda").half()
    d = torch.randn((rows, hidden), generator=g, device="cuda").half()
    w = torch.randn(hidden, generator=g, device="cuda")
    out, res = torch.empty_like(x), x.clone()
    assert cuda.rmsnorm(out, x, w, rows, hidden) == 0
    # fp32 sums of up to 16400 squares, then one rounding to fp16
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(1, keepdim=True) + 1e-6) * w.double()
    assert torch.all((out.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 2.0 ** -24)
    assert cuda.rmsnorm_residual(out, res, d, w, rows, hidden) == 0
    total = (x.float() + d.float()).half()
    assert torch.equal(res, total)
    want = total.double() * torch.rsqrt(total.double().pow(2).mean(1, keepdim=True) + 1e-6) * w.double()
    assert torch.all((out.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 2.0 ** -24)


@pytest.mark.parametrize("rows", [444, 445, 592, 593, 888, 889])
@pytest.mark.parametrize("hidden", [2048, 2056, 2560, 4096, 4104, 5120, 6136, 6144, 6152])
def test_two_vectors_a_thread(cuda, rows, hidden):
    test_rows_and_widths(cuda, rows, hidden)


@pytest.mark.parametrize("rows", [1, 148, 149, 889])
@pytest.mark.parametrize("hidden", [8, 264, 512, 2056, 5120, 8192])
@pytest.mark.parametrize("shift", ["x", "delta", "out", "w"])
def test_rows_off_their_boundary(cuda, rows, hidden, shift):
    """One operand starts behind a vector's boundary: the scalar loop, in whichever form the rule picks."""
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)

    def placed(t, name):
        if name != shift:
            return t
        room = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape)
        return room.copy_(t)

    x, d = (torch.randn((rows, hidden), generator=g, device="cuda").half() for _ in range(2))
    w = placed(torch.randn(hidden, generator=g, device="cuda"), "w")
    x, d, out = placed(x, "x"), placed(d, "delta"), placed(torch.empty_like(x), "out")
    total = (x.float() + d.float()).half()
    assert cuda.rmsnorm(out, x, w, rows, hidden) == 0
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(1, keepdim=True) + 1e-6) * w.double()
    assert torch.all((out.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 2.0 ** -24)
    assert cuda.rmsnorm_residual(out, x, d, w, rows, hidden) == 0
    assert torch.equal(x, total)
    want = total.double() * torch.rsqrt(total.double().pow(2).mean(1, keepdim=True) + 1e-6) * w.double()
    assert torch.all((out.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 2.0 ** -24)
