"""The GEMM behind 32 activation rows at every width of its tiles: at their edges, at K where the unpacking warps' and the fold threads' turns
begin and end, with output rows that do not pair up (odd N, odd addresses), and with tiles cut between CTAs (K = 4096: several parts)."""
import numpy as np
import pytest
import torch

import oracle
from conftest import synth_linear

pytestmark = pytest.mark.gpu

GEMM = 3
ROWS = [33, 48, 49, 64, 65, 80, 81, 96, 97, 112, 128, 129, 144, 160, 161, 176, 192, 193, 224, 225, 256, 257, 353, 512]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("K,N", [(128, 256), (384, 258), (512, 301), (640, 130), (1152, 700), (4096, 513)])
def test_every_tile_width(cuda, M, K, N):
    X, W, S, _ = synth_linear(M, K, N, seed=M + K)
    bias = np.linspace(-1, 1, N, dtype=np.float32)
    want = oracle.linear_int4_f64(X.astype(np.float32), W, S) + bias
    cuda.set_linear_path(GEMM)
    try:
        y = torch.full((M, N), float("nan"), device="cuda")
        assert cuda.linear_int4(y, dev(X), dev(W), dev(S), dev(bias), M, N, K) == 0
        # fp16 results, at an address that is a multiple of four and at one that is not
        whole = torch.full((M * N + 1,), float("nan"), dtype=torch.float16, device="cuda")
        halves = [whole[:M * N].view(M, N).clone(), whole[1:].view(M, N)]
        for h in halves:
            assert cuda.linear_int4(h, dev(X), dev(W), dev(S), dev(bias), M, N, K) == 0
    finally:
        cuda.set_linear_path(0)
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    # products are exact: K additions in fp32, each off by half a unit of a partial sum of at most sqrt(K) typical terms
    got = y.cpu().numpy()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-6
    assert np.all(np.abs(got - want) <= 2e-5 * np.abs(want).max())
    assert torch.equal(halves[0], y.half()) and torch.equal(halves[1], y.half())  # the same sums, rounded once


def dense(w, s):
    """The weights of a packed projection in 64 bits, on the GPU."""
    q = torch.stack([w & 15, w >> 4], -1).view(w.shape[0], -1).to(torch.int8)
    return torch.where(q >= 8, q - 16, q).double() * s.double().repeat_interleave(128, 1)


def packed(g, N, K):
    return (torch.randint(0, 256, (N, K // 2), generator=g, device="cuda", dtype=torch.uint8),
            torch.rand((N, K // 128), generator=g, device="cuda").mul_(0.01).half())


@pytest.mark.parametrize("M", [33, 47, 48, 49, 64, 65, 79, 80])
@pytest.mark.parametrize("K,N", [
    (1024, 5632), (1152, 5632),    # 8 groups: each fold thread of a row takes half of the columns; 9: they take the groups in turn
    (2048, 5632), (2176, 5632),    # a tile of 16 and 17 groups
    (3072, 19200),                 # in turn, 75 tiles on 74 pairs
    (5120, 1024), (5120, 1100),    # in turn, tiles in equal parts of eight groups, and in unequal ones
    (17408, 5120),                 # in turn, cut tiles of 136 groups
])
def test_fold_threads_in_turn(cuda, M, K, N):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    w, s = packed(g, N, K)
    x = torch.randn((M, K), generator=g, device="cuda").half()
    y = torch.full((M, N), float("nan"), device="cuda")
    cuda.set_linear_path(GEMM)
    try:
        assert cuda.linear_int4(y, x, w, s, None, M, N, K) == 0
    finally:
        cuda.set_linear_path(0)
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    want = x.double() @ dense(w, s).t()
    # as above
    assert ((y - want).norm() / want.norm()).item() <= 2e-6
    assert (y - want).abs().max().item() <= 2e-5 * want.abs().max().item()


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("K,N", [(128, 130), (1152, 331), (5120, 1216)])
def test_swiglu_at_every_tile_width(cuda, M, K, N):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    (wg, sg), (wu, su) = packed(g, N, K), packed(g, N, K)
    x = torch.randn((M, K), generator=g, device="cuda").half()
    y = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
    cuda.set_linear_path(GEMM)
    try:
        assert cuda.mlp_gate_up_swiglu_int4(y, x, wg, sg, wu, su, M, N, K) == 0
    finally:
        cuda.set_linear_path(0)
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    gate, up = x.double() @ dense(wg, sg).t(), x.double() @ dense(wu, su).t()
    want = gate / (1 + torch.exp(-gate)) * up
    # both sums as above, carried through silu (slope below 1.1, |silu(g)| <= |g|), the product's two fp32 roundings, and one to fp16
    err = 2e-5 * torch.maximum(gate.abs().max(), up.abs().max())
    assert torch.all((y.double() - want).abs() <= 2.0 ** -11 * 1.01 * want.abs() + err * (1.1 * up.abs() + gate.abs()) + 2.0 ** -24)
