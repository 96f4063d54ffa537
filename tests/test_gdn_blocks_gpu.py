"""The delta rule over longer calls (blocks of 16 tokens on the tensor cores) and the vectorised convolution, at the
sizes where they can go wrong: around the change of kernel, around block edges, strong decay, repeated keys, and a state
carried from call to call.  Against the fp32 restatement of the reference in oracle/."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import xinfer_b200.ops as ops
    return ops


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def delta_rule_f64(qkv, z, b, a, A_log, dt_bias, norm_w, S, hv, hk):
    T = qkv.shape[0]
    f = lambda x: np.asarray(x, np.float64)  # noqa: E731
    q, k = f(qkv[:, :hk * 128]).reshape(T, hk, 128), f(qkv[:, hk * 128:2 * hk * 128]).reshape(T, hk, 128)
    v, zz = f(qkv[:, 2 * hk * 128:]).reshape(T, hv, 128), f(z).reshape(T, hv, 128)
    unit = lambda x: x / np.sqrt((x * x).sum(-1, keepdims=True) + 1e-6)  # noqa: E731
    q, k = np.repeat(unit(q) * 0.08838834764, hv // hk, 1), np.repeat(unit(k), hv // hk, 1)
    beta = 1 / (1 + np.exp(-f(b)))
    g = np.exp(-np.exp(f(A_log)) * np.logaddexp(0, f(a) + f(dt_bias)))
    S, out = f(S).copy(), np.empty((T, hv, 128))
    for t in range(T):
        S *= g[t][:, None, None]
        d = (v[t] - np.einsum("hkd,hk->hd", S, k[t])) * beta[t][:, None]
        S += k[t][:, :, None] * d[:, None, :]
        out[t] = np.einsum("hkd,hk->hd", S, q[t])
    out = out / np.sqrt((out * out).mean(-1, keepdims=True) + 1e-6) * f(norm_w) * zz / (1 + np.exp(-zz))
    return out.reshape(T, hv * 128), S


@pytest.mark.parametrize("T", [1, 16, 17, 31, 32, 33, 77])
@pytest.mark.parametrize("kind", ["plain", "slow decay", "one key"])
def test_delta_rule_blocks(cuda, T, kind):
    import torch
    hv, hk = 6, 2
    rng = np.random.default_rng(T)
    qkv = rng.normal(0, 1, (2 * T, 2 * hk * 128 + hv * 128)).astype(np.float16)
    z, b, a = (rng.normal(0, 1, (2 * T, n)).astype(np.float16) for n in (hv * 128, hv, hv))
    if kind == "slow decay":
        a = (a - 6).astype(np.float16)
    if kind == "one key":
        qkv[:, hk * 128:2 * hk * 128] = qkv[0, hk * 128:2 * hk * 128]
    A_log, dt_bias = (rng.normal(0, 0.5, hv).astype(np.float32) for _ in range(2))
    norm_w = rng.normal(1, 0.02, 128).astype(np.float32)
    S = rng.normal(0, 0.05, (hv, 128, 128)).astype(np.float32)
    want, S_want = delta_rule_f64(qkv, z, b, a, A_log, dt_bias, norm_w, S, hv, hk)
    out, S_d = torch.full((2 * T, hv * 128), float("nan"), dtype=torch.float16, device="cuda"), dev(S)
    args = [dev(x) for x in (qkv, z, b, a)]
    for c in range(2):  # two calls: the second starts from the first one's state
        part = [x[c * T:(c + 1) * T] for x in args]
        assert cuda.recurrent_gated_delta_net(out[c * T:(c + 1) * T], *part, dev(A_log), dev(dt_bias), dev(norm_w), S_d, T, False, hv, hk) == 0
    torch.cuda.synchronize()
    rel = lambda x, y: np.linalg.norm(np.asarray(x, np.float64) - y) / np.linalg.norm(y)  # noqa: E731
    # the output is rounded to fp16 once: 2^-11 at most, a third of that in the 2-norm.  The state: fp32 rounding of some
    # 128-term sums per token, 6e-8 each, which decay forgets after a few tokens (slow decay: adds up over the call).
    assert rel(out.float().cpu().numpy(), want) <= 5e-4
    assert rel(S_d.cpu().numpy(), S_want) <= 6e-8 * 128 ** 0.5 * (T if kind == "slow decay" else 8) ** 0.5


@pytest.mark.parametrize("T", [2, 7, 8, 9, 15])
@pytest.mark.parametrize("zero", [False, True])
def test_delta_rule_short_calls(cuda, T, zero):
    """Calls that a single block of the token-by-token kernel covers, none of them full."""
    import torch
    hv, hk = 9, 3
    rng = np.random.default_rng(T)
    qkv = rng.normal(0, 1, (T, 2 * hk * 128 + hv * 128)).astype(np.float16)
    z, b, a = (rng.normal(0, 1, (T, n)).astype(np.float16) for n in (hv * 128, hv, hv))
    A_log, dt_bias = (rng.normal(0, 0.5, hv).astype(np.float32) for _ in range(2))
    norm_w = rng.normal(1, 0.02, 128).astype(np.float32)
    S = rng.normal(0, 0.05, (hv, 128, 128)).astype(np.float32)
    want, S_want = delta_rule_f64(qkv, z, b, a, A_log, dt_bias, norm_w, 0 * S if zero else S, hv, hk)
    out, S_d = torch.full((T, hv * 128), float("nan"), dtype=torch.float16, device="cuda"), dev(S)
    assert cuda.recurrent_gated_delta_net(out, dev(qkv), dev(z), dev(b), dev(a), dev(A_log), dev(dt_bias), dev(norm_w), S_d, T, zero, hv, hk) == 0
    torch.cuda.synchronize()
    rel = lambda x, y: np.linalg.norm(np.asarray(x, np.float64) - y) / np.linalg.norm(y)  # noqa: E731
    assert rel(out.float().cpu().numpy(), want) <= 5e-4                       # (the bounds of the longer calls)
    assert rel(S_d.cpu().numpy(), S_want) <= 6e-8 * 128 ** 0.5 * 8 ** 0.5


@pytest.mark.parametrize("T", [17, 40])
@pytest.mark.parametrize("kind", ["1e-4", "1e-5", "small beta", "zero keys", "tiny keys", "large state", "large state, small values"])
def test_delta_rule_blocks_range(cuda, T, kind):
    """Magnitudes far from one, head by head: small states and values, keys at and near zero beside large values, states beyond
    fp16's range, a state that grows from zero by small updates."""
    import torch
    hv, hk = 6, 2
    rng = np.random.default_rng(T)
    qkv = rng.normal(0, 1, (T, 2 * hk * 128 + hv * 128))
    k, v = qkv[:, hk * 128:2 * hk * 128], qkv[:, 2 * hk * 128:]
    z, b, a = (rng.normal(0, 1, (T, n)).astype(np.float16) for n in (hv * 128, hv, hv))
    size = 0.05
    if kind in ("1e-4", "1e-5"):
        size = float(kind)
        v *= size
    elif kind == "small beta":
        b, size = (b - 12).astype(np.float16), 0.0
    elif kind == "zero keys":
        k[2::5] = 0
        v *= 1e4
    elif kind == "tiny keys":
        k *= 1e-4
        v *= 100
    else:  # (with the strong decay of the other kinds the large state is gone after a few tokens)
        a, size = (a - 6).astype(np.float16), 1e7
        if kind == "large state, small values":
            v *= 1e-3
    qkv = qkv.astype(np.float16)
    A_log, dt_bias = (rng.normal(0, 0.5, hv).astype(np.float32) for _ in range(2))
    norm_w = rng.normal(1, 0.02, 128).astype(np.float32)
    S = (size * rng.normal(0, 1, (hv, 128, 128))).astype(np.float32)
    want, S_want = delta_rule_f64(qkv, z, b, a, A_log, dt_bias, norm_w, S, hv, hk)
    out, S_d = torch.full((T, hv * 128), float("nan"), dtype=torch.float16, device="cuda"), dev(S)
    assert cuda.recurrent_gated_delta_net(out, dev(qkv), dev(z), dev(b), dev(a), dev(A_log), dev(dt_bias), dev(norm_w), S_d, T, size == 0, hv, hk) == 0
    torch.cuda.synchronize()
    got, S_got = out.double().cpu().numpy(), S_d.double().cpu().numpy()
    # as above, and half a step of fp16's subnormals on every output
    assert np.linalg.norm(got - want) <= 5e-4 * np.linalg.norm(want) + 2 ** -25 * want.size ** 0.5
    for h in range(hv):
        assert np.linalg.norm(S_got[h] - S_want[h]) <= 6e-8 * 128 ** 0.5 * T ** 0.5 * np.linalg.norm(S_want[h]), h


@pytest.mark.parametrize("T,C", [(1, 4), (2, 10), (3, 516), (8, 513), (9, 512), (40, 1028)])
def test_conv1d_spans(cuda, T, C):
    """One and several spans of positions, channel counts with and without vector access, in place, with and without state."""
    import torch
    rng = np.random.default_rng(T + C)
    x, w, st = rng.normal(0, 1, (T, C)).astype(np.float16), rng.normal(0, 0.5, (C, 4)).astype(np.float32), rng.normal(0, 1, (3, C)).astype(np.float32)
    for state in (st, None):
        ref = None if state is None else state.copy()
        want = np.asarray(oracle.conv1d_silu(x, w, ref), np.float32)
        for in_place in (False, True):
            x_d, st_d = dev(x), None if state is None else dev(state)
            y = x_d if in_place else torch.full_like(x_d, float("nan"))
            assert cuda.causal_conv1d_silu(y, x_d, dev(w), T, st_d, C) == 0
            # one fp16 rounding on either side
            assert np.all(np.abs(y.float().cpu().numpy() - want) <= 2 ** -10 * np.maximum(np.abs(want), 2 ** -14))
            if state is not None:
                assert np.array_equal(st_d.cpu().numpy(), ref)


@pytest.mark.parametrize("T", [1, 2, 3, 7, 8, 9, 16, 17, 61])
@pytest.mark.parametrize("C", [512, 515])
def test_conv1d_in_place(cuda, T, C):
    """A thread's walk over all positions against one that takes eight: the same bits."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn((T, C), generator=g, device="cuda").half()
    w, st = torch.randn((C, 4), generator=g, device="cuda"), torch.randn((3, C), generator=g, device="cuda")
    apart, st2 = torch.empty_like(x), st.clone()
    assert cuda.causal_conv1d_silu(apart, x, w, T, st, C) == 0
    assert cuda.causal_conv1d_silu(x, x, w, T, st2, C) == 0
    assert torch.equal(x, apart) and torch.equal(st, st2)


@pytest.mark.parametrize("with_state", [True, False])
def test_conv1d_beyond_32_bit_positions(cuda, with_state):
    """A sequence of more than 2^31 positions (two channels) gives, at its end and at a seam, what that part alone gives."""
    import torch
    C, T, tail, seam = 2, 2 ** 31 + 21, 64, 2 ** 30
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GB")
    x = torch.full((T, C), 0.5, dtype=torch.float16, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(0)
    for at in (seam - 32, T - tail):
        x[at:at + tail] = torch.randn((tail, C), generator=g, device="cuda").half()
    w, st = torch.randn((C, 4), generator=g, device="cuda"), torch.randn((3, C), generator=g, device="cuda")
    y, last = torch.empty_like(x), st.clone() if with_state else None
    assert cuda.causal_conv1d_silu(y, x, w, T, last, C) == 0
    for at in (seam - 32, T - tail):
        y2, st2 = torch.empty((tail, C), dtype=torch.float16, device="cuda"), torch.full_like(st, 0.5)
        assert cuda.causal_conv1d_silu(y2, x[at:at + tail].contiguous(), w, tail, st2, C) == 0
        assert torch.equal(y[at:at + tail], y2)
    if with_state:
        assert torch.equal(last, st2)
    head = torch.empty((64, C), dtype=torch.float16, device="cuda")
    assert cuda.causal_conv1d_silu(head, x[:64].contiguous(), w, 64, st.clone() if with_state else None, C) == 0
    assert torch.equal(y[:64], head)
    del x, y
    torch.cuda.empty_cache()
