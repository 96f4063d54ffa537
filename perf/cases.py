"""Performance cases: the work that a user of this package has it do, through its public entry points.

    cases = listed()                 the named cases
    case = draw(random.Random(0))    one more of the same ranges
    state = prepare(case, seed)      inputs, weights and handles, on the GPU
    outputs = run(state)             one pass
    work(case), tolerance(case)      what a pass cannot do without, and how close two correct results are

Seven kinds of work (`case["kind"]`), all at the layer shapes of the 27B model (hidden 5120, FFN 17408, 24 query and 4
key/value heads of 256, 48 value and 16 key heads of 128, vocabulary 151936):

  step         the speculative decode loop: one captured step of `SpecDecoder` and the read of its tokens
  generate     a request batch from prompt to last token: reset, chunked prefill, decode steps
  attn_layer   one full-attention layer called op by op, for hosts with a forward pass of their own
  delta_layer  one Gated-DeltaNet layer called op by op
  lm_head      logits of some rows and their arg-max on the device
  linear_f32   the fp32 overload of the INT4 linear
  sample       a sampling call on logits that are there: nucleus draw, plain draw, batched acceptance rule, or the
               synchronous acceptance call that takes and returns host values
"""
from __future__ import annotations

import ctypes
import math
from collections import namedtuple

import numpy as np
import torch

import xinfer_b200
import xinfer_b200.ops as ops
from xinfer_b200.spec import Shape, SpecDecoder

MODEL = Shape()
H, F, V = MODEL.hidden_size, MODEL.intermediate_size, MODEL.vocab_size
HQ, HKV, HD = MODEL.num_attention_heads, MODEL.num_key_value_heads, 256
VH, KH = MODEL.linear_num_v_heads, MODEL.linear_num_k_heads
CH, VD = MODEL.conv_channels, MODEL.linear_num_v_heads * 128
GROUP = 128
DEV = "cuda"


def listed():
    return [
        # The reference's own acceptance call (host tokens, host result) for one sequence: the smallest call there is.
        {"name": "accept_one_sequence", "kind": "sample", "op": "accept_host", "rows": 3, "k": 3, "vocab": V},
        # Eight sequences draw their next token under top-p, as a non-speculative server does once per step.
        {"name": "nucleus_8_rows", "kind": "sample", "op": "top_p", "rows": 8, "k": 0, "vocab": V},
        # The fp32 overload on a key/value-sized projection: callers that keep fp32 activations.
        {"name": "linear_f32_8x5120x1024", "kind": "linear_f32", "m": 8, "k": 5120, "n": 1024},
        # Logits of a verify pass's 32 rows, and the greedy tokens.
        {"name": "lm_head_32_rows", "kind": "lm_head", "m": 32},
        # Single-token decode of one sequence through either kind of layer: launches and weight streaming.
        {"name": "attn_layer_decode", "kind": "attn_layer", "m": 1, "start": 1023},
        {"name": "delta_layer_decode", "kind": "delta_layer", "m": 1},
        # A short prompt: more rows than a decode step, fewer than a GEMM tile, and ragged.
        {"name": "attn_layer_77_rows", "kind": "attn_layer", "m": 77, "start": 0},
        # A full 512-row prefill chunk behind a longer context, and a ragged last chunk.
        {"name": "attn_layer_prefill_512", "kind": "attn_layer", "m": 512, "start": 1536},
        {"name": "delta_layer_prefill_509", "kind": "delta_layer", "m": 509},
        # The decode loop, one user with a short context, and the throughput configuration of the benchmark.
        {"name": "step_batch1_ctx1024", "kind": "step", "layers": 16, "batch": 1, "k": 3, "ctx": 1024, "temperature": 0.0, "top_p": 1.0},
        {"name": "step_batch8_ctx8192", "kind": "step", "layers": 64, "batch": 8, "k": 3, "ctx": 8192, "temperature": 0.0, "top_p": 1.0},
        # A batch of requests end to end with sampling: prefill of medium prompts, then some tokens.
        {"name": "generate_batch4_prompt700", "kind": "generate", "layers": 16, "batch": 4, "k": 3, "prompt": 700, "new": 24,
         "temperature": 0.7, "top_p": 0.9},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "generate", "attn_layer", "attn_layer", "delta_layer", "delta_layer", "lm_head", "linear_f32", "sample"])
    if kind == "sample":
        op = rng.choice(["accept_host", "top_p", "draw", "accept"])
        k = rng.randint(1, 4)
        rows = {"accept_host": k, "top_p": _log_int(rng, 1, 32), "draw": _log_int(rng, 1, 32), "accept": rng.randint(1, 32 // (k + 1)) * (k + 1)}[op]
        return {"kind": kind, "op": op, "rows": rows, "k": k if op.startswith("accept") else 0, "vocab": _log_int(rng, 4096, V)}
    if kind == "linear_f32":
        k, n = rng.choice([(5120, 1024), (5120, 6144), (6144, 5120), (1024, 2048), (512, 1536)])
        return {"kind": kind, "m": _log_int(rng, 1, 32), "k": k, "n": n + 8 * rng.randint(0, 16)}
    if kind == "lm_head":
        return {"kind": kind, "m": _log_int(rng, 1, 32)}
    if kind == "attn_layer":
        return {"kind": kind, "m": _log_int(rng, 1, 512), "start": _log_int(rng, 1, 8192) - 1}
    if kind == "delta_layer":
        return {"kind": kind, "m": _log_int(rng, 1, 512)}
    k = rng.randint(1, 4)
    temperature, top_p = rng.choice([(0.0, 1.0), (0.7, 1.0), (0.7, 0.9)])
    case = {"kind": kind, "layers": rng.choice([4, 8, 16]), "batch": rng.randint(1, min(8, 32 // (k + 1))), "k": k}
    if kind == "step":
        case["ctx"] = _log_int(rng, 64, 8192)
    else:
        case["prompt"], case["new"] = _log_int(rng, 16, 768), rng.randint(4, 24)
        case["batch"] = min(case["batch"], 2800 // case["prompt"])
    return {**case, "temperature": temperature, "top_p": top_p}


# ---------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(g, shape, dtype=torch.float16, std=1.0, mean=0.0):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).mul_(std).add_(mean).to(dtype)


def _symmetric_(w):
    """Random packed int4 as a symmetric quantiser leaves it: values -7 .. 7 around a mean of zero, no -8."""
    w.masked_fill_((w & 0x0F) == 0x08, 0)
    return w.masked_fill_((w & 0xF0) == 0x80, 0)


def _int4(g, n, k):
    """A projection in the library's layout: packed int4 rows and one fp16 scale per 128 weights."""
    w = _symmetric_(torch.randint(0, 256, (n, k // 2), generator=g, device=DEV, dtype=torch.uint8))
    s = _normal(g, (n, k // GROUP), torch.float32, 0.02).abs_().div_(7.0).to(torch.float16)
    return w, s


def _int4_bytes(n, k):
    return n * (k // 2) + n * (k // GROUP) * 2


# ------------------------------------------------------------------------------------------------ decoder set-up
class _DeviceView:
    """A decoder's own device tensor as a torch tensor; keeps the decoder alive."""

    def __init__(self, dec, layer, name, typestr, shape=None):
        size = ctypes.c_int64()
        ptr = xinfer_b200.lib().xinfer_spec_decoder_tensor(dec._h, layer, name.encode(), ctypes.byref(size))
        if not ptr:
            raise KeyError(name)
        self.dec = dec
        self.__cuda_array_interface__ = {"shape": tuple(shape or (size.value,)), "typestr": typestr, "data": (ptr, False), "version": 2}


def _view(dec, layer, name, typestr, shape=None):
    return torch.as_tensor(_DeviceView(dec, layer, name, typestr, shape), device=DEV)


def _pack_rows(rows, scale, w_out, s_out):
    """Symmetric INT4-G128 quantisation of fp32 `rows` (times `scale`) into the library's layout."""
    n, k = rows.shape
    grouped = rows.view(n, k // GROUP, GROUP)
    step = grouped.abs().amax(-1, keepdim=True).clamp_min_(1e-6).div_(7.0)
    q = torch.round(grouped / step).to(torch.int8).view(n, k // 2, 2)
    w_out.copy_(((q[..., 0] & 0xF) | ((q[..., 1] & 0xF) << 4)).view(torch.uint8))
    s_out.copy_((step.view(n, k // GROUP) * scale).to(torch.float16))


def _make_predictive(dec, g):
    """Gives a random-init decoder the sharp next-token distributions of a trained one.

    The LM head becomes an INT4 copy of the embedding table under two permutations, one per half of the features, that
    agree on about 70 % of the tokens; the target sees both halves, the MTP head's input projection passes the first one.
    So every distribution has a clear first token, and the drafts are right about as often as a trained head's are."""
    for layer in range(dec.shape.num_hidden_layers + 1):
        mixer = ("q_proj", "k_proj", "v_proj", "o_proj") if dec.is_full(layer) else ("in_qkv", "in_z", "in_b", "in_a", "out_proj")
        for name in mixer + ("gate", "up", "down"):
            _symmetric_(_view(dec, layer, name + ".w", "|u1"))
    _symmetric_(_view(dec, -1, "mtp_fc.w", "|u1"))
    embed = torch.as_tensor(_DeviceView(dec, -1, "embed", "<u2", (V, H)), device=DEV).view(torch.bfloat16)
    embed.mul_(4.0)
    target = torch.randperm(V, generator=g, device=DEV)              # row v answers token target[v]
    draft = target.clone()
    moved = torch.nonzero(torch.rand(V, generator=g, device=DEV) < 0.3).flatten()
    draft[moved] = draft[moved.roll(1)]
    w, s = _view(dec, -1, "lm_head.w", "|u1", (V, H // 2)), _view(dec, -1, "lm_head.s", "<f2", (V, H // GROUP))
    for a in range(0, V, 16384):
        b = min(V, a + 16384)
        rows = torch.cat([embed[draft[a:b], : H // 2].float() * 0.5, embed[target[a:b], H // 2:].float()], 1)
        _pack_rows(rows, 0.004, w[a:b], s[a:b])
    w, s = _view(dec, -1, "mtp_fc.w", "|u1", (H, H)), _view(dec, -1, "mtp_fc.s", "<f2", (H, 2 * H // GROUP))
    i = torch.arange(H // 2, device=DEV)
    for group in range(H // 2 // GROUP):
        rows = slice(group * GROUP, (group + 1) * GROUP)
        w[rows, group * GROUP // 2: (group + 1) * GROUP // 2] = 0
        s[rows, group] = 4.0 / 7.0
    w[i, i // 2] = torch.where(i % 2 == 0, 0x07, 0x70).to(torch.uint8)


def _decoder(case, seed, max_seq):
    shape = Shape(num_hidden_layers=case["layers"])
    dec = SpecDecoder(shape, batch=case["batch"], k=case["k"], max_seq=max_seq, seed=seed)
    _make_predictive(dec, _gen(seed))
    dec.set_sampling(case["temperature"], seed)
    dec.set_top_p(case["top_p"])
    return dec


def _capture(dec):
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        dec.capture(stream)
    torch.cuda.current_stream().wait_stream(stream)


# ------------------------------------------------------------------------------------------------------ kinds
def _prepare_step(case, seed):
    # cache room for some thousand steps past the context, as a server with a longer maximum length keeps
    max_seq = case["ctx"] + 8192
    dec = _decoder(case, seed, max_seq)
    dec.reset(case["ctx"], seed)
    tokens = torch.randint(0, V, (case["batch"],), generator=_gen(seed + 1), device=DEV).cpu().numpy()
    dec.set_tokens(tokens)
    _capture(dec)
    rows = case["batch"] * (case["k"] + 1)
    return {"case": case, "seed": seed, "dec": dec, "tokens": tokens, "room": max_seq - case["ctx"] - (case["k"] + 1),
            "logits": _view(dec, -1, "logits", "<f4", (rows, V)), "hidden": _view(dec, -1, "x", "<f2", (rows, H)),
            "h_last": _view(dec, -1, "h_last", "<f2", (case["batch"], H))}


def _run_step(st):
    dec, per_step = st["dec"], st["case"]["k"] + 1
    if st["room"] < per_step:  # the cache is full: the next request starts
        dec.reset(st["case"]["ctx"], st["seed"])
        dec.set_tokens(st["tokens"])
        st["room"] = dec.max_seq - st["case"]["ctx"]
    st["room"] -= per_step
    dec.step()
    emitted, counts = dec.results()
    return {"emitted": emitted, "counts": counts, "logits": st["logits"], "hidden": st["hidden"], "h_last": st["h_last"]}


def _decoder_step_work(case, ctx):
    rows, b, k = case["batch"] * (case["k"] + 1), case["batch"], case["k"]
    full = case["layers"] // 4
    delta = case["layers"] - full
    mlp = 2 * _int4_bytes(F, H) + _int4_bytes(H, F)
    attn_w = _int4_bytes(HQ * 2 * HD, H) + 2 * _int4_bytes(HKV * HD, H) + _int4_bytes(H, HQ * HD)
    delta_w = _int4_bytes(CH + VD + 2 * VH, H) + _int4_bytes(H, VD)
    head = _int4_bytes(V, H)
    weights = full * attn_w + delta * delta_w + case["layers"] * mlp + head
    draft_w = attn_w + mlp + head + _int4_bytes(H, 2 * H)
    kv = 2 * b * ctx * HKV * HD * 2
    state = delta * b * (2 * VH * 128 * 128 * 4 + 2 * 3 * CH * 4)
    params = lambda nbytes: nbytes / (0.5 + 2 / GROUP)  # noqa: E731  (weights per packed byte)
    flops = 2 * rows * params(weights) + 2 * b * k * params(draft_w) + 4 * ctx * HQ * HD * (rows * full + b * k)
    return {"bytes": weights + k * draft_w + (full + k) * kv + state + 4 * (rows + b * k) * V, "flops": flops}


def _prepare_generate(case, seed):
    max_seq = case["prompt"] + case["new"] + 64
    dec = _decoder(case, seed, max_seq)
    dec.reset(16, seed)
    _capture(dec)
    prompt = torch.randint(0, V, (case["batch"], case["prompt"]), generator=_gen(seed + 1), device=DEV).cpu().numpy()
    return {"case": case, "dec": dec, "prompt": prompt, "seed": seed, "h_last": _view(dec, -1, "h_last", "<f2", (case["batch"], H))}


def _run_generate(st):
    case = st["case"]
    got = st["dec"].generate(st["prompt"], max_new_tokens=case["new"], temperature=case["temperature"], top_p=case["top_p"], seed=st["seed"])
    return {"tokens": [np.array(r.token_ids, np.int64) for r in got], "stopped": [int(r.finish_reason == "stop") for r in got],
            "h_last": st["h_last"]}


def _generate_work(case):
    b, n = case["batch"], case["prompt"] - 1
    step = _decoder_step_work(case, case["prompt"])
    steps = max(1.0, case["new"] / (1 + 0.6 * case["k"]))
    full = case["layers"] // 4
    delta = case["layers"] - full
    weights = (full * (_int4_bytes(HQ * 2 * HD, H) + 2 * _int4_bytes(HKV * HD, H) + _int4_bytes(H, HQ * HD)) +
               delta * (_int4_bytes(CH + VD + 2 * VH, H) + _int4_bytes(H, VD)) + case["layers"] * (2 * _int4_bytes(F, H) + _int4_bytes(H, F)))
    flops = 2 * b * n * weights / (0.5 + 2 / GROUP) + full * 4 * b * n * (n + 1) / 2 * HQ * HD + delta * 8 * b * n * VD * 128
    kv = (full + 1) * 2 * b * n * HKV * HD * 2
    return {"bytes": weights + kv + delta * b * VH * 128 * 128 * 4 + steps * step["bytes"], "flops": flops + steps * step["flops"]}


def _residual(g, m):
    x = torch.randn((m, H), generator=g, device=DEV)
    x[:, ::512] *= 20.0  # the few large channels of a trained residual stream
    return x.to(torch.float16)


def _mlp_weights(g):
    (wg, sg), (wu, su), (wd, sd) = _int4(g, F, H), _int4(g, F, H), _int4(g, H, F)
    return {"wg": wg, "sg": sg, "wu": wu, "su": su, "wd": wd, "sd": sd}


def _common_layer(g, m):
    half = lambda *shape: torch.empty(shape, device=DEV, dtype=torch.float16)  # noqa: E731
    return {"x": _residual(g, m), "norm1": _normal(g, (H,), torch.float32, 0.02, 1.0), "norm2": _normal(g, (H,), torch.float32, 0.02, 1.0),
            "residual": half(m, H), "normed": half(m, H), "proj": half(m, H), "act": half(m, F), "out": half(m, H), **_mlp_weights(g)}


def _mixer_to_output(st, mixed, m):
    """Output projection, residual add and norm, MLP: the second half of either kind of layer."""
    ops.linear_int4(st["proj"], mixed, st["wo"], st["so"], None, m, H, mixed.shape[1])
    ops.rmsnorm_residual(st["normed"], st["residual"], st["proj"], st["norm2"], m, H)
    ops.mlp_gate_up_swiglu_int4(st["act"], st["normed"], st["wg"], st["sg"], st["wu"], st["su"], m, F, H)
    ops.linear_int4(st["out"], st["act"], st["wd"], st["sd"], None, m, H, F)


def _prepare_attn_layer(case, seed):
    g, m, start = _gen(seed), case["m"], case["start"]
    st = _common_layer(g, m)
    cap = start + m + 32
    half = lambda *shape: torch.empty(shape, device=DEV, dtype=torch.float16)  # noqa: E731
    (wq, sq), (wk, sk), (wv, sv), (wo, so) = _int4(g, HQ * HD, H), _int4(g, HKV * HD, H), _int4(g, HKV * HD, H), _int4(g, H, HQ * HD)
    st.update(case=case, cap=cap, wq=wq, sq=sq, wk=wk, sk=sk, wv=wv, sv=sv, wo=wo, so=so, q=half(m, HQ * HD), k=half(m, HKV * HD),
              v=half(m, HKV * HD), mixed=half(m, HQ * HD), k_cache=_normal(g, (cap, HKV, HD)), v_cache=_normal(g, (cap, HKV, HD)),
              positions=torch.arange(start, start + m, device=DEV, dtype=torch.int64))
    return st


def _run_attn_layer(st):
    m, start, cap = st["case"]["m"], st["case"]["start"], st["cap"]
    st["residual"].copy_(st["x"])
    ops.rmsnorm(st["normed"], st["residual"], st["norm1"], m, H)
    ops.linear_int4_fused(st["normed"], [{"Y": st["q"], "W_int4": st["wq"], "scales": st["sq"], "N": HQ * HD},
                                         {"Y": st["k"], "W_int4": st["wk"], "scales": st["sk"], "N": HKV * HD},
                                         {"Y": st["v"], "W_int4": st["wv"], "scales": st["sv"], "N": HKV * HD}], m, H)
    ops.rope(st["q"], st["k"], m, HQ, HKV, HD, st["positions"])
    ops.attention_write_kv_cache(st["k_cache"], st["v_cache"], st["k"], st["v"], start, m, HKV, HD, cap)
    ops.sdpa_causal_cached(st["mixed"], st["q"], st["k_cache"], st["v_cache"], start, m, HQ, HKV, HD, max_seq_len=cap)
    _mixer_to_output(st, st["mixed"], m)
    return {"out": st["out"], "residual": st["residual"], "mixed": st["mixed"], "k_cache": st["k_cache"][start:start + m],
            "v_cache": st["v_cache"][start:start + m]}


def _attn_layer_work(case):
    m, start = case["m"], case["start"]
    weights = _int4_bytes((HQ + 2 * HKV) * HD, H) + _int4_bytes(H, HQ * HD) + 2 * _int4_bytes(F, H) + _int4_bytes(H, F)
    pairs = m * start + m * (m + 1) / 2
    return {"bytes": weights + 2 * (start + m) * HKV * HD * 2 + 2 * m * HKV * HD * 2 + 3 * m * H * 2,
            "flops": 2 * m * weights / (0.5 + 2 / GROUP) + 4 * pairs * HQ * HD}


def _prepare_delta_layer(case, seed):
    g, m = _gen(seed), case["m"]
    st = _common_layer(g, m)
    half = lambda *shape: torch.empty(shape, device=DEV, dtype=torch.float16)  # noqa: E731
    (wi, si), (wz, sz), (wb, sb), (wa, sa), (wo, so) = (_int4(g, n, k) for n, k in ((CH, H), (VD, H), (VH, H), (VH, H), (H, VD)))
    st.update(case=case, wi=wi, si=si, wz=wz, sz=sz, wb=wb, sb=sb, wa=wa, sa=sa, wo=wo, so=so, qkv=half(m, CH), conv=half(m, CH), z=half(m, VD),
              b=half(m, VH), a=half(m, VH), mixed=half(m, VD), conv_w=_normal(g, (CH, 4), torch.float32, 0.5),
              a_log=_normal(g, (VH,), torch.float32, 0.5, 0.5), dt_bias=_normal(g, (VH,), torch.float32, 0.5),
              gdn_norm=_normal(g, (128,), torch.float32, 0.02, 1.0), state=_normal(g, (VH, 128, 128), torch.float32, 0.05),
              conv_state=_normal(g, (3, CH), torch.float32))
    return st


def _run_delta_layer(st):
    m = st["case"]["m"]
    st["residual"].copy_(st["x"])
    ops.rmsnorm(st["normed"], st["residual"], st["norm1"], m, H)
    ops.linear_int4_fused(st["normed"], [{"Y": st["qkv"], "W_int4": st["wi"], "scales": st["si"], "N": CH},
                                         {"Y": st["z"], "W_int4": st["wz"], "scales": st["sz"], "N": VD},
                                         {"Y": st["b"], "W_int4": st["wb"], "scales": st["sb"], "N": VH},
                                         {"Y": st["a"], "W_int4": st["wa"], "scales": st["sa"], "N": VH}], m, H)
    ops.causal_conv1d_silu(st["conv"], st["qkv"], st["conv_w"], m, st["conv_state"], CH)
    ops.recurrent_gated_delta_net(st["mixed"], st["conv"], st["z"], st["b"], st["a"], st["a_log"], st["dt_bias"], st["gdn_norm"],
                                  st["state"], m, False, VH, KH)
    _mixer_to_output(st, st["mixed"], m)
    return {"out": st["out"], "residual": st["residual"], "mixed": st["mixed"], "state": st["state"], "conv_state": st["conv_state"]}


def _delta_layer_work(case):
    m = case["m"]
    weights = _int4_bytes(CH + VD + 2 * VH, H) + _int4_bytes(H, VD) + 2 * _int4_bytes(F, H) + _int4_bytes(H, F)
    return {"bytes": weights + 2 * VH * 128 * 128 * 4 + 2 * 3 * CH * 4 + 3 * m * H * 2,
            "flops": 2 * m * weights / (0.5 + 2 / GROUP) + 8 * m * VD * 128}


def _prepare_lm_head(case, seed):
    g, m = _gen(seed), case["m"]
    w, s = _int4(g, V, H)
    return {"case": case, "x": _normal(g, (m, H)), "w": w, "s": s, "logits": torch.empty((m, V), device=DEV),
            "tokens": torch.empty(m, device=DEV, dtype=torch.int64)}


def _run_lm_head(st):
    ops.linear_int4(st["logits"], st["x"], st["w"], st["s"], None, st["case"]["m"], V, H)
    ops.argmax_rows(st["logits"], st["tokens"])
    return {"logits": st["logits"], "tokens": st["tokens"]}


def _prepare_linear_f32(case, seed):
    g, m, n, k = _gen(seed), case["m"], case["n"], case["k"]
    w, s = _int4(g, n, k)
    return {"case": case, "x": _normal(g, (m, k), torch.float32), "w": w, "s": s, "bias": _normal(g, (n,), torch.float32, 0.1),
            "y": torch.empty((m, n), device=DEV)}


def _run_linear_f32(st):
    case = st["case"]
    ops.linear_int4(st["y"], st["x"], st["w"], st["s"], st["bias"], case["m"], case["n"], case["k"])
    return st["y"]


def _prepare_sample(case, seed):
    g, rows, vocab, k = _gen(seed), case["rows"], case["vocab"], case["k"]
    # a trained model's logits: a wide bulk and a few dozen candidates above it
    logits = torch.randn((rows, vocab), generator=g, device=DEV).mul_(2.0)
    top = torch.rand((rows, vocab), generator=g, device=DEV).topk(40).indices
    logits.scatter_(1, top, 8.0 + 4.0 * torch.rand((rows, 40), generator=g, device=DEV))
    st = {"case": case, "logits": logits}
    if case["op"] in ("top_p", "draw"):
        st.update(uniform=torch.rand(rows, generator=g, device=DEV), tokens=torch.empty(rows, device=DEV, dtype=torch.int64),
                  probs=torch.empty(rows, device=DEV))
        return st
    # drafts: mostly the likeliest token, sometimes another candidate
    per_seq = k if case["op"] == "accept_host" else k + 1
    batch = rows // per_seq
    best = logits.argmax(1).view(batch, per_seq)[:, :k]
    other = top[:, 0].view(batch, per_seq)[:, :k]
    drafts = torch.where(torch.rand((batch, k), generator=g, device=DEV) < 0.7, best, other).contiguous()
    probs = torch.rand((batch, k), generator=g, device=DEV).mul_(0.5).add_(0.05)
    uniform = torch.rand((batch, k), generator=g, device=DEV)
    if case["op"] == "accept_host":
        st.update(drafts=drafts[0].tolist(), probs=probs[0].tolist(), uniform=uniform[0].tolist())
    else:
        st.update(drafts=drafts, probs=probs, uniform=uniform, view=logits.view(batch, per_seq, vocab),
                  records=torch.zeros(batch * ops.ACCEPT_RECORD_BYTES, device=DEV, dtype=torch.uint8))
    return st


def _run_sample(st):
    op = st["case"]["op"]
    if op == "top_p":
        ops.sample_tokens_top_p(st["logits"], st["uniform"], st["tokens"], st["probs"], 1.0 / 0.7, 0.9)
        return {"tokens": st["tokens"], "probs": st["probs"]}
    if op == "draw":
        ops.sample_tokens(st["logits"], st["uniform"], st["tokens"], st["probs"], 1.0 / 0.7)
        return {"tokens": st["tokens"], "probs": st["probs"]}
    if op == "accept":
        ops.speculative_accept_reject_batched(st["drafts"], st["view"], st["probs"], st["uniform"], st["records"], 1.0 / 0.7, st["case"]["k"])
        return st["records"]
    got = ops.speculative_accept_reject(st["drafts"], st["case"]["k"], st["logits"], st["case"]["vocab"], st["probs"], st["uniform"])
    accepted = got["accepted_tokens"] + [-1] * (st["case"]["k"] - len(got["accepted_tokens"]))
    return {"accepted": np.array(accepted, np.int64), **{name: int(v) for name, v in got.items() if name != "accepted_tokens"}}


# ------------------------------------------------------------------------------------------------ the five calls
def _work_lm_head(case):
    m = case["m"]
    return {"bytes": _int4_bytes(V, H) + 2 * m * H + 4 * m * V, "flops": 2 * m * V * H}


def _work_linear_f32(case):
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": _int4_bytes(n, k) + 4 * m * k + 4 * n + 4 * m * n, "flops": 2 * m * n * k}


def _work_sample(case):
    return {"bytes": 4 * case["rows"] * case["vocab"], "flops": 2 * case["rows"] * case["vocab"]}


Kind = namedtuple("Kind", "prepare run work tolerance")
KINDS = {
    # fp16 activations through every layer of the stack: one fp16 rounding per tensor, carried to the logits
    "step": Kind(_prepare_step, _run_step, lambda case: _decoder_step_work(case, case["ctx"]), {"rel": 0.02, "max": 0.5}),
    "generate": Kind(_prepare_generate, _run_generate, _generate_work, {"rel": 0.02, "max": 0.5}),
    # a handful of fp16 roundings between the layer's input and its output
    "attn_layer": Kind(_prepare_attn_layer, _run_attn_layer, _attn_layer_work, {"rel": 0.004, "max": 0.1}),
    "delta_layer": Kind(_prepare_delta_layer, _run_delta_layer, _delta_layer_work, {"rel": 0.004, "max": 0.1}),
    # fp16 x int4 products are exact in fp32; what is left is the order of 5120 fp32 additions
    "lm_head": Kind(_prepare_lm_head, _run_lm_head, _work_lm_head, {"rel": 3e-5}),
    "linear_f32": Kind(_prepare_linear_f32, _run_linear_f32, _work_linear_f32, {"rel": 1e-5}),
    # the tokens are whole numbers; the probabilities are ratios of fp32 sums over the vocabulary
    "sample": Kind(_prepare_sample, _run_sample, _work_sample, {"rel": 1e-5}),
}


def prepare(case, seed):
    kind = KINDS[case["kind"]]
    return {"kind": kind, "inner": kind.prepare(case, seed)}


def run(state):
    return state["kind"].run(state["inner"])


def work(case):
    return KINDS[case["kind"]].work(case)


def tolerance(case):
    return KINDS[case["kind"]].tolerance
