"""The work that users of calibquant_b200 have it do, as measurable cases.

A case is a dict of plain values; ``path`` says which public entry points one pass goes through:

* ``turn``     one attention layer of the patched backbone answers a prompt: ``attention.forward`` on the prompt,
               then on one new token after another, as an eager ``generate`` drives it (projections included);
* ``decode``   ``ops.decode_attention`` on the group format, the attention of one layer and one decode step;
* ``decode8``  ``calibquant.decode_attention``, the same step on the uint8 format;
* ``prefill``  a prompt behind the ``wqkv`` projection: ``ops.prefill_rope_split``, the quantize + pack calls of the
               visual span in either format, ``ops.prefill_attention``;
* ``pack``     ``triton_quantize_and_pack_along_last_dim`` on values and its per-channel counterpart on keys;
* ``qjl_build`` / ``qjl_step``   sketching the keys of a prompt with ``QJLKeyQuantizer``; one decode step on it:
               score estimate, softmax, quantized value product.

Token counts: 41 system tokens, 256 visual tokens per image tile (13 tiles = 3328), head dim 128, 8 KV heads with
4 or 6 query heads each.  Keys carry outlier channels (per-channel lognormal factor) as in ``oracle/generator.py``.
"""

from __future__ import annotations

import math
import os

import torch

D, HKV, SYS, GROUP = 128, 8, 41, 32
DT = {"fp16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # one user, one picture: prompt and a short answer through the patched forward (the eager generate loop)
        dict(name="turn_b1_1bit", path="turn", batch=1, vis=3328, text=64, new=16, rep=4, bits=1, dtype="bf16", fmt="group"),
        # the smallest call: a thumbnail tile and a few words, one request, called eagerly
        dict(name="decode_b1_t256", path="decode", batch=1, vis=256, text=23, rep=4, bits=1, dtype="bf16", mask=False, graph=False),
        # the 7B backbone's serving step (batch 16, 13 tiles, some text generated already), replayed from a CUDA graph
        # with the live token count on the device
        dict(name="decode_b16_t3328_graph", path="decode", batch=16, vis=3328, text=191, rep=4, bits=1, dtype="bf16", mask=False, graph=True),
        # long context, everything quantized: the default workload of bench.py
        dict(name="decode_b8_t32768", path="decode", batch=8, vis=32768, text=0, rep=4, bits=1, dtype="fp16", mask=False, graph=False),
        # the 20B backbone's step: 48 query heads, batch 64, 26 tiles, 2 bits
        dict(name="decode_b64_t6656_48q", path="decode", batch=64, vis=6656, text=228, rep=6, bits=2, dtype="bf16", mask=False, graph=False),
        # a few padded requests (additive mask) with a visual span that is no multiple of a tile, 4 bits
        dict(name="decode_b4_t5152_masked", path="decode", batch=4, vis=5152, text=37, rep=4, bits=4, dtype="fp16", mask=True, graph=False),
        # the uint8 format's serving step
        dict(name="decode8_b16_t3328_graph", path="decode8", batch=16, vis=3328, text=77, rep=4, bits=1, dtype="bf16", mask=False, graph=True),
        # the 7B backbone's prompts at batch 16: everything of a layer's prefill that is not a GEMM
        dict(name="prefill_b16_t3392", path="prefill", batch=16, vis=3328, text=23, rep=4, bits=1, dtype="bf16", fmt="group"),
        # two short prompts of five tiles, odd length, uint8 format at 2 bits
        dict(name="prefill_b2_t1401_u8", path="prefill", batch=2, vis=1280, text=80, rep=4, bits=2, dtype="fp16", fmt="uint8"),
        # quantize + pack of a long context's keys and values
        dict(name="pack_b8_t32768_2bit", path="pack", batch=8, vis=32768, bits=2, dtype="fp16"),
        # QJL keys: sketching four prompts (the span leaves a full-precision remainder)
        dict(name="qjl_build_b4_t6688", path="qjl_build", batch=4, vis=6688, dtype="bf16"),
        # QJL keys: a decode step over a long context, values at 2 bits
        dict(name="qjl_step_b8_t16384", path="qjl_step", batch=8, vis=16384, rep=4, bits=2, dtype="fp16"),
    ]


# per path: share of the draws, batch range, visual tokens, and the largest batch * tokens (what the listed cases reach)
_RANGES = {
    "turn": (2, 1, 4, 256, 6656, 6656),
    "decode": (5, 1, 64, 256, 32768, 8 * 32768),
    "decode8": (2, 1, 32, 256, 16384, 4 * 16384),
    "prefill": (2, 1, 16, 256, 6656, 16 * 3328),
    "pack": (1, 1, 16, 2048, 32768, 8 * 32768),
    "qjl_build": (1, 1, 8, 512, 8192, 8 * 4096),
    "qjl_step": (1, 1, 16, 512, 16384, 8 * 16384),
}


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    names = list(_RANGES)
    path = rng.choices(names, [_RANGES[n][0] for n in names])[0]
    _, b_lo, b_hi, v_lo, v_hi, most = _RANGES[path]
    while True:
        batch, vis = _log_int(rng, b_lo, b_hi), _log_int(rng, v_lo, v_hi)
        # image tiles give multiples of 256; other front ends any multiple of a quantization group
        vis = max(v_lo, vis // 256 * 256) if rng.random() < 0.6 else max(v_lo, vis // GROUP * GROUP)
        if batch * vis <= most and (path != "prefill" or batch * vis * vis <= 16 * 3328 * 3328):
            break
    case = dict(path=path, batch=batch, vis=vis, dtype=rng.choice(["fp16", "bf16"]))
    text = _log_int(rng, 5, 400)
    if path == "turn":
        case.update(text=text, new=_log_int(rng, 4, 16), rep=4, bits=rng.choice([1, 1, 2, 4]), fmt=rng.choice(["group", "group", "uint8"]))
    elif path in ("decode", "decode8"):
        graph = rng.random() < 0.4
        case.update(text=text, rep=rng.choice([4, 4, 6]), bits=rng.choice([1, 1, 2, 4]), graph=graph,
                    mask=not graph and rng.random() < 0.25)
    elif path == "prefill":
        case.update(text=text, rep=4, bits=rng.choice([1, 1, 2, 4]), fmt=rng.choice(["group", "group", "uint8"]))
        if batch * (SYS + vis + text) ** 2 > 16 * 3392 ** 2:
            case["text"] = 5
    elif path == "pack":
        case.update(bits=rng.choice([1, 2, 4]))
    elif path == "qjl_step":
        case.update(rep=4, bits=rng.choice([2, 4]))
    return case


# ---- inputs ------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, dtype, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)


def _keys(g, dtype, *shape):
    """N(0,1) with a few outlier channels: every channel of the last dimension times a lognormal(0,1) factor."""
    factor = torch.exp(torch.randn(shape[-1], generator=g, device="cuda"))
    return _normal(g, dtype, *shape) * factor.to(dtype)


def _decode_inputs(c, g, dtype):
    """Query, full-precision keys / values (system + text, in buffers with room for what is still to be generated
    when the step is replayed from a graph), mask."""
    B, n_fp = c["batch"], (SYS + c["text"] if c["text"] else 0)
    room = n_fp + (256 if c["graph"] else 0)
    s = {"q": _normal(g, dtype, B, HKV * c["rep"], 1, D), "k_fp": _keys(g, dtype, B, HKV, room, D),
         "v_fp": _normal(g, dtype, B, HKV, room, D), "t_sys": SYS if n_fp else 0, "mask": None, "live": None}
    if c["mask"]:      # left padding of a different length in every row
        total = n_fp + c["vis"]
        lengths = torch.randint(0, SYS - 1, (B, 1), generator=g, device="cuda")
        lengths[0] = 0
        hidden = torch.arange(total, device="cuda").unsqueeze(0) < lengths
        s["mask"] = torch.zeros(B, 1, 1, total, dtype=dtype, device="cuda").masked_fill_(hidden.view(B, 1, 1, total), torch.finfo(dtype).min)
    if c["graph"]:
        s["live"] = torch.tensor([n_fp], dtype=torch.int32, device="cuda")
    return s


def _captured(step):
    """A program that generates many tokens captures the step once and replays it."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = step()
    return graph, out


def _layer(c, g, dtype):
    """One attention layer of the 7B backbone with random weights, patched as a user patches the model."""
    from calibquant_b200 import patch_internvl as pi
    from calibquant_b200.internlm2 import ChatModelShell, InternLM2Config
    hidden = HKV * c["rep"] * D
    cfg = InternLM2Config(hidden_size=hidden, num_attention_heads=HKV * c["rep"], num_key_value_heads=HKV,
                          intermediate_size=64, num_hidden_layers=1, vocab_size=64)
    with torch.device("cuda"):
        shell = ChatModelShell(cfg).to(dtype)
    pi.patch_model(shell, "calibquant", kv_format=c["fmt"])
    pi.BITS_KV = c["bits"]
    pi.SCALE_K, pi.SCALE_V = (0.5, 0.3) if c["bits"] == 1 else (1, 1)
    os.environ["IMAGE_TOKEN_NUM"] = str(c["vis"])
    attn = shell.language_model.model.layers[0].attention
    with torch.no_grad():
        for lin in (attn.wqkv, attn.wo):
            lin.weight.copy_(_normal(g, dtype, *lin.weight.shape) * 0.02)
    return attn


def prepare(case, seed):
    c, g, dtype = case, _gen(seed), DT[case["dtype"]]
    B, vis, path = c["batch"], c["vis"], c["path"]
    from calibquant_b200 import calibquant, ops
    s = {"path": path, "case": c}
    if path == "turn":
        attn = _layer(c, g, dtype)
        T = SYS + vis + c["text"]
        s.update(attn=attn, prompt=_normal(g, dtype, B, T, attn.hidden_size),
                 tokens=[_normal(g, dtype, B, 1, attn.hidden_size) for _ in range(c["new"])],
                 prompt_pos=torch.arange(T, device="cuda").unsqueeze(0).expand(B, T),
                 token_pos=[torch.full((B, 1), T + i, device="cuda", dtype=torch.long) for i in range(c["new"])])
    elif path in ("decode", "decode8"):
        s.update(_decode_inputs(c, g, dtype))
        k = _keys(g, dtype, B, HKV, vis, D)
        if path == "decode":
            s["k_pack"] = ops.pack_k_per_channel(k, GROUP, c["bits"])
            s["v_pack"] = ops.pack_v_per_token(_normal(g, dtype, B, HKV, vis, D), GROUP, c["bits"])
        else:
            clip_k, clip_v = (0.5, 0.3) if c["bits"] == 1 else (1, 1)
            enc_k, sk, zk = calibquant.quant_encode(k.transpose(1, 2), c["bits"], scale=clip_k)
            enc_v, sv, zv = calibquant.quant_encode(_normal(g, dtype, B, vis, HKV, D), c["bits"], scale=clip_v)
            s["state"] = {"enc_k": enc_k, "enc_v": enc_v, "scale_key": sk, "zero_point_key": zk,
                          "scale_value": sv, "zero_point_value": zv}
        if c["graph"]:
            s["graph"], s["out"] = _captured(lambda: _decode_step(s))
    elif path == "prefill":
        from calibquant_b200.internlm2 import RotaryEmbedding
        T = SYS + vis + c["text"]
        qkv = _normal(g, dtype, B, T, HKV, c["rep"] + 2, D)
        qkv[:, :, :, c["rep"]] *= torch.exp(torch.randn(D, generator=g, device="cuda")).to(dtype)
        s["qkv"] = qkv.view(B, T, -1)
        s["cos"], s["sin"] = RotaryEmbedding(D, 1e6).to("cuda")(qkv, T)
        s["pos"] = torch.arange(T, device="cuda").unsqueeze(0).expand(B, T).contiguous()
    elif path == "pack":
        s["k"], s["v"] = _keys(g, dtype, B, HKV, vis, D), _normal(g, dtype, B, HKV, vis, D)
    else:
        from calibquant_b200.qjl.qjl_utils import QJLSketch
        s["sketch"] = QJLSketch((D, 256), 256, device=torch.device("cuda"), rng=torch.Generator(device="cuda").manual_seed(1234))
        s["k"] = _keys(g, dtype, B, HKV, vis, D)
        if path == "qjl_step":
            s["keys"] = _quantizer(s)
            s["keys"].build_sketch(s.pop("k"))
            s["v_pack"] = ops.pack_v_per_token(_normal(g, dtype, B, HKV, vis, D), GROUP, c["bits"])
            s["q"] = _normal(g, dtype, B, HKV * c["rep"], 1, D)
    return s


def _quantizer(s):
    from calibquant_b200.qjl.qjl_utils import QJLKeyQuantizer
    return QJLKeyQuantizer(s["sketch"], 32, 128, GROUP, 2)      # outliers, buffer, group, bits: patch_model's defaults


# ---- one pass ----------------------------------------------------------------------------------------------------

def _decode_step(s):
    from calibquant_b200 import calibquant, ops
    c = s["case"]
    if s["path"] == "decode":
        k_fp, v_fp = (s["k_fp"], s["v_fp"]) if s["k_fp"].shape[2] else (None, None)
        return ops.decode_attention(s["q"], s["k_pack"], s["v_pack"], k_fp, v_fp, s["t_sys"], c["bits"],
                                    mask=s["mask"], t_fp_dev=s["live"])
    return calibquant.decode_attention(s["q"], s["state"], s["k_fp"], s["v_fp"], c["bits"], s["t_sys"],
                                       mask=s["mask"], t_fp_dev=s["live"])


def _prefill(s):
    from calibquant_b200 import calibquant, ops
    c, vis = s["case"], s["case"]["vis"]
    B, T = s["qkv"].shape[:2]
    k_cache = torch.empty(B, HKV, T - vis + 256, D, dtype=s["qkv"].dtype, device="cuda")
    v_cache = torch.empty_like(k_cache)
    q, k, v = ops.prefill_rope_split(s["qkv"], s["cos"], s["sin"], s["pos"], HKV, c["rep"], k_cache, v_cache, SYS, vis)
    if c["fmt"] == "group":
        packs = ops.pack_k_per_channel(k.transpose(1, 2)[:, :, SYS:SYS + vis], GROUP, c["bits"]) + \
            ops.pack_v_per_token(v.transpose(1, 2)[:, :, SYS:SYS + vis], GROUP, c["bits"])
    else:
        clip_k, clip_v = (0.5, 0.3) if c["bits"] == 1 else (1, 1)
        packs = calibquant.quant_encode(k[:, SYS:SYS + vis], c["bits"], scale=clip_k) + \
            calibquant.quant_encode(v[:, SYS:SYS + vis], c["bits"], scale=clip_v)
    out = ops.prefill_attention(q, k, v)
    return [out, *packs, k_cache[:, :, :T - vis], v_cache[:, :, :T - vis]]


@torch.no_grad()
def run(state):
    s, path = state, state["path"]
    if path == "turn":
        out, _, past = s["attn"](s["prompt"], position_ids=s["prompt_pos"], use_cache=True)
        outs = [out]
        for x, pos in zip(s["tokens"], s["token_pos"]):
            out, _, past = s["attn"](x, position_ids=pos, past_key_value=past, use_cache=True)
            outs.append(out)
        return outs + list(past)
    if path in ("decode", "decode8"):
        if s["case"]["graph"]:
            s["graph"].replay()
            return s["out"]
        return _decode_step(s)
    if path == "prefill":
        return _prefill(s)
    if path == "pack":
        from calibquant_b200.qjl import new_pack
        bits = s["case"]["bits"]
        return list(new_pack.quantize_and_pack_k_per_channel(s["k"], GROUP, bits) +
                    new_pack.triton_quantize_and_pack_along_last_dim(s["v"], GROUP, bits))
    if path == "qjl_build":
        keys = _quantizer(s)
        keys.build_sketch(s["k"])
        outs = [keys.key_states_quant, keys.key_outliers_quant, keys.key_outliers_norm, keys.key_states_norm]
        return outs if keys.key_residual is None else outs + [keys.key_residual]
    from calibquant_b200.qjl.matmul import cuda_quantized_bmm_dynamic
    scores = s["keys"].attention_score(s["q"])
    att = torch.softmax(scores / D ** 0.5, dim=-1, dtype=torch.float32).to(s["q"].dtype)
    return [scores, cuda_quantized_bmm_dynamic(GROUP, att, *s["v_pack"], s["case"]["bits"])]


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def _pack_bytes(n, bits):
    """Codes, scales and minima of n elements in the group format."""
    return n * bits / 8 + n / GROUP * 4


def work(case):
    c, path, B, vis = case, case["path"], case["batch"], case["vis"]
    n = B * HKV * vis * D                          # elements of the visual span's keys (and of its values)
    hq = HKV * c.get("rep", 4)
    n_fp = SYS + c["text"] if c.get("text") else 0

    def step(tokens_fp, fmt):
        stored = 2 * _pack_bytes(n, c["bits"]) if fmt == "group" else 2 * n * c["bits"] / 8
        return (stored + 2 * B * HKV * tokens_fp * D * 2 + 2 * B * hq * D * 2, 4.0 * B * hq * D * (vis + tokens_fp))

    def prompt(T, fmt):
        attn = 4.0 * B * hq * D * T * T / 2
        stored = 2 * _pack_bytes(n, c["bits"]) if fmt == "group" else 2 * n * c["bits"] / 8
        return stored + 2 * B * HKV * (T - vis) * D * 2, attn

    if path in ("decode", "decode8"):
        b, f = step(n_fp, "group" if path == "decode" else "uint8")
    elif path == "prefill":
        T = vis + n_fp
        b, f = prompt(T, c["fmt"])
        b += B * T * (hq + 2 * HKV) * D * 2 + B * T * hq * D * 2        # projected prompt in, attention out
    elif path == "turn":
        T, hidden = vis + n_fp, hq * D
        b, f = prompt(T, c["fmt"])
        weights = hidden * (hq + 2 * HKV) * D + hq * D * hidden
        b += 2 * weights + 2 * B * T * hidden * 2
        f += 2.0 * B * T * weights
        for i in range(c["new"]):
            bs, fs = step(n_fp + i + 1, c["fmt"])
            b += bs + 2 * weights + 2 * B * hidden * 2
            f += fs + 2.0 * B * weights
    elif path == "pack":
        b, f = 2 * (2 * n + _pack_bytes(n, c["bits"])), 6.0 * n
    elif path == "qjl_build":
        done = B * HKV * (vis - vis % 128)
        b, f = done * D * 2 + done * (32 + 32 + 2 + 2) + done / GROUP * 32, 2.0 * done * 256 * D
    else:
        keys = B * HKV * vis
        b = keys * (32 + 32 + 2 + 2) + keys / GROUP * 32 + _pack_bytes(n, c["bits"]) + B * hq * vis * 4
        f = 2.0 * B * hq * vis * (512 + D)
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """Codes and packed bytes are exact (sign bits of sums at rounding distance of zero aside).  Attention: the results
    are sums of probabilities rounded to the data type of logits rounded to it, and at 1 and 2 bits the calibration
    maps a rounding of the extreme logit onto its whole row: 1e-2 in fp16, 2e-2 in bf16."""
    path, fp16 = case["path"], case["dtype"] == "fp16"
    if path == "pack":
        return "exact"
    if path == "qjl_build":
        return {"rel": 1e-3 if fp16 else 4e-3, "differ": 2e-3}
    if path == "qjl_step":
        return {"rel": 4e-3 if fp16 else 1e-2}
    if path == "prefill":
        return {"rel": 2e-3 if fp16 else 1e-2}
    return {"rel": 1e-2 if fp16 else 2e-2}
