"""How the decode kernel (at most 32 activation rows) finishes its tiles: whole tiles whose four warps trade halves, K ranges summed by
a thread-block cluster, tiles cut between CTAs.  Against the oracle in 64 bits at the row counts where halves, quarters and the
clusters' blocks of rows begin and end, with weight rows that leave the last tile ragged.  And the GEMM behind 32 rows, at its tile widths."""
import numpy as np
import pytest
import torch

import oracle
from conftest import synth_linear

pytestmark = pytest.mark.gpu

TC, GEMM = 1, 3
ROWS = [1, 8, 9, 10, 15, 16, 17, 23, 24, 25, 31, 32]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("M", ROWS)
@pytest.mark.parametrize("K,N", [
    (2048, 700),      # clusters of eight, the last tile ragged
    (1280, 5000),     # clusters of five
    (256, 37000),     # one tile per CTA, uncut
    (640, 45000),     # tiles cut between CTAs, among them whole ones
])
def test_rows_of_every_block(cuda, M, K, N):
    X, W, S, _ = synth_linear(M, K, N, seed=M + K)
    bias = np.linspace(-1, 1, N, dtype=np.float32)
    y = torch.full((M, N), float("nan"), device="cuda")
    assert cuda.linear_int4(y, dev(X), dev(W), dev(S), dev(bias), M, N, K) == 0
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    rows = np.unique(np.concatenate([np.arange(0, N, 97), np.arange(min(N, 600)), np.arange(N - 300, N)]))
    want = oracle.linear_int4_f64(X.astype(np.float32), W[rows], S[rows]) + bias[rows]
    got = y.cpu().numpy()[:, rows]
    # products are exact: K additions in fp32, each off by half a unit of a partial sum of at most sqrt(K) typical terms
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 2e-6
    assert np.all(np.isfinite(y.cpu().numpy()))
    again = torch.empty_like(y)
    assert cuda.linear_int4(again, dev(X), dev(W), dev(S), dev(bias), M, N, K) == 0
    assert torch.equal(again, y)


@pytest.mark.parametrize("M", ROWS + [33, 64, 77, 128, 129, 200, 256])
@pytest.mark.parametrize("N", [264, 17408])
def test_gate_up_rows_of_every_block(cuda, M, N):
    """The same for gate/up (clusters; one uncut tile per CTA), and for the tile widths of the GEMM behind 32 rows."""
    K = 512
    X, Wg, Sg, _ = synth_linear(M, K, N, seed=M)
    _, Wu, Su, _ = synth_linear(1, K, N, seed=M + 1)
    X[0] *= 8  # gates far from zero, of either sign
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    assert cuda.mlp_gate_up_swiglu_int4(y, dev(X), dev(Wg), dev(Sg), dev(Wu), dev(Su), M, N, K) == 0
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    rows = np.unique(np.concatenate([np.arange(0, N, 61), np.arange(N - 130, N)]))
    g = oracle.linear_int4_f64(X.astype(np.float32), Wg[rows], Sg[rows])
    u = oracle.linear_int4_f64(X.astype(np.float32), Wu[rows], Su[rows])
    want = g / (1 + np.exp(-g)) * u
    got = y.float().cpu().numpy()[:, rows]
    # one fp16 rounding of the result
    assert np.all(np.abs(got - want) <= 2.0 ** -11 * np.abs(want) * 1.01 + 2e-5 * np.abs(want).max())


@pytest.mark.parametrize("M", [9, 16, 17, 31, 32])
@pytest.mark.parametrize("K,N", [(256, 60000), (640, 45000)])
def test_gate_up_of_several_tiles(cuda, M, K, N):
    """Gate/up with more than one tile per CTA: whole ones one after the other, and cut ones among them (K = 640), whose values go through
    the scratch buffer, by a CTA that is the last to arrive or is not."""
    X, Wg, Sg, _ = synth_linear(M, K, N, seed=M)
    _, Wu, Su, _ = synth_linear(1, K, N, seed=M + 1)
    args = dev(X), dev(Wg), dev(Sg), dev(Wu), dev(Su), M, N, K
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    assert cuda.mlp_gate_up_swiglu_int4(y, *args) == 0
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    rows = np.unique(np.concatenate([np.arange(0, N, 61), np.arange(N - 130, N)]))
    g = oracle.linear_int4_f64(X.astype(np.float32), Wg[rows], Sg[rows])
    u = oracle.linear_int4_f64(X.astype(np.float32), Wu[rows], Su[rows])
    want = g / (1 + np.exp(-g)) * u
    # one fp16 rounding of the result
    assert np.all(np.abs(y.float().cpu().numpy()[:, rows] - want) <= 2.0 ** -11 * np.abs(want) * 1.01 + 2e-5 * np.abs(want).max())
    for _ in range(3):  # (the barriers' phases and the tile counters start as they should, and no tile holds another's values)
        again = torch.full_like(y, float("nan"))
        assert cuda.mlp_gate_up_swiglu_int4(again, *args) == 0
        assert torch.equal(again, y)


@pytest.mark.parametrize("M", [33, 64, 65, 96, 97, 128, 129, 192])
@pytest.mark.parametrize("K,N", [(5120, 5000), (5632, 2048)])
def test_gemm_with_cut_tiles(cuda, M, K, N):
    """The GEMM at either side of its tile widths, its rings many times around and its tiles cut between pairs."""
    X, W, S, _ = synth_linear(M, K, N, seed=M)
    _, Wu, Su, _ = synth_linear(1, K, N, seed=M + 1)
    Xd, w, wu = dev(X), (dev(W), dev(S)), (dev(Wu), dev(Su))
    y, y2 = (torch.full((M, N), float("nan"), device="cuda", dtype=t) for t in (torch.float32, torch.float16))
    cuda.set_linear_path(GEMM)
    try:
        assert cuda.linear_int4(y, Xd, *w, None, M, N, K) == 0 and cuda.last_linear_path() == GEMM
        assert cuda.mlp_gate_up_swiglu_int4(y2, Xd, *w, *wu, M, N, K) == 0 and cuda.last_linear_path() == GEMM
    finally:
        cuda.set_linear_path(0)
    torch.cuda.synchronize()
    assert cuda.device_status(0) == 0
    rows = np.unique(np.concatenate([np.arange(0, N, 17), np.arange(N - 130, N)]))
    g = oracle.linear_int4_f64(X.astype(np.float32), W[rows], S[rows])
    u = oracle.linear_int4_f64(X.astype(np.float32), Wu[rows], Su[rows])
    # K additions in fp32 (those of a group truncated), each off by a unit of a partial sum of at most sqrt(K) typical terms
    assert np.linalg.norm(y.cpu().numpy()[:, rows] - g) / np.linalg.norm(g) <= 2e-6
    want = g / (1 + np.exp(-g)) * u
    assert np.all(np.abs(y2.float().cpu().numpy()[:, rows] - want) <= 2.0 ** -11 * np.abs(want) * 1.01 + 2e-5 * np.abs(want).max())


@pytest.mark.parametrize("M,path", [(4, TC), (32, TC), (100, TC), (33, GEMM), (100, GEMM), (300, GEMM)])
def test_swiglu_far_gates(cuda, M, path):
    """Gates beyond the range of exp: x / (1 + exp(-x)) is zero far below and x far above, not NaN."""
    K, N = 128, 512
    W = torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda")
    W[:, 0] = 1                                            # the gate of every feature is X[:, 0], its up value too
    S = torch.ones((N, 1), dtype=torch.float16, device="cuda")
    X = torch.zeros((M, K), dtype=torch.float16, device="cuda")
    gates = torch.tensor([-60000.0, -100.0, -88.5, -87.5, -20.0, 0.0, 20.0, 88.0, 200.0], device="cuda")
    X[:, 0] = gates[torch.arange(M, device="cuda") % len(gates)].half()
    y = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
    cuda.set_linear_path(path)
    try:
        assert cuda.mlp_gate_up_swiglu_int4(y, X, W, S, W, S, M, N, K) == 0
        assert cuda.last_linear_path() == path
    finally:
        cuda.set_linear_path(0)
    g = X[:, :1].double()
    want = (g / (1 + torch.exp(-g)) * g).expand(M, N)
    assert torch.all((y.double() - want).abs() <= 2.0 ** -10 * want.abs() + 1e-7)
