"""The convolution over a chunk with one and with four channels a thread, on either side of the line between them, with weights that can be
loaded as vectors and with weights that cannot: the same bits, and those of a row-by-row reference within one rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 8, 9, 63, 64, 65, 72, 200])
@pytest.mark.parametrize("channels", [4, 512, 1028, 1030])
def test_rows_and_channels(cuda, rows, channels):
    g = torch.Generator(device="cuda").manual_seed(rows * 7 + channels)
    x = torch.randn((rows, channels), generator=g, device="cuda").half()
    shifted = torch.randn(channels * 4 + 1, generator=g, device="cuda")[1:].view(channels, 4)  # four bytes behind a boundary
    state = torch.randn((3, channels), generator=g, device="cuda")
    out, states = [], []
    for weights, inplace in ((shifted.clone(), False), (shifted, False), (shifted.clone(), True)):
        st = state.clone()
        o = x.clone() if inplace else torch.full_like(x, float("nan"))
        assert cuda.causal_conv1d_silu(o, o if inplace else x, weights, rows, st, channels) == 0
        out.append(o)
        states.append(st)
    assert all(torch.equal(out[0], o) for o in out) and all(torch.equal(states[0], s) for s in states)
    seen = torch.cat([state.double(), x.double()])
    assert torch.equal(states[0], seen[-3:].float())
    y = sum(shifted[:, t].double() * seen[t:t + rows] for t in range(4))
    want = y / (1 + torch.exp(-y))
    bound = sum((shifted[:, t].double() * seen[t:t + rows]).abs() for t in range(4))  # four fp32 roundings of sums this large at most
    assert torch.all((out[0].double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 8 * 2.0 ** -24 * bound + 2.0 ** -24)


@pytest.mark.parametrize("rows", [1, 3])
@pytest.mark.parametrize("inplace", [False, True])
def test_more_channels_than_blocks_of_one_channel_a_thread(cuda, rows, inplace):
    """65535 blocks of 128 channels and four channels more: too many for a grid with one channel a thread, not for one with four."""
    channels = 65535 * 128 + 4
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn((rows, channels), generator=g, device="cuda").half()
    weights = torch.randn((channels, 4), generator=g, device="cuda")
    state = torch.randn((3, channels), generator=g, device="cuda")
    seen = torch.cat([state, x.float()])
    o = x.clone() if inplace else torch.empty_like(x)
    assert cuda.causal_conv1d_silu(o, o if inplace else x, weights, rows, state, channels) == 0
    assert torch.equal(state, seen[-3:])
    terms = [weights[:, t] * seen[t:t + rows] for t in range(4)]
    y = sum(terms).double()
    want = y / (1 + torch.exp(-y))
    bound = sum(t.abs() for t in terms).double()  # four fp32 roundings of sums this large at most, here and in the expectation
    assert torch.all((o.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + 16 * 2.0 ** -24 * bound + 2.0 ** -24)


@pytest.mark.parametrize("rows,channels", [
    (40, 10240), (41, 10240),  # 400 and 480 blocks of 128 channels and eight positions: one channel a thread below 444 of them
    (392, 1028), (393, 1028),  # 441 and 450
    (880, 512), (881, 512),    # 440 and 444
])
def test_number_of_blocks(cuda, rows, channels):
    test_rows_and_channels(cuda, rows, channels)
