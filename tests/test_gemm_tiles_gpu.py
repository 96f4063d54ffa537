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
