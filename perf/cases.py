"""The work a user of this package has it do, as measurable cases.

Three kinds, all through the public entry points:

  linear   one packed product as the drop-in operator serves it (`t2g128_int8xint2_linear`, int8 rows of a
           decode width) or as the module serves it (`T2LinearKernel.forward`, bf16 rows, any number of them)
  decode   a whole request: prompt in, tokens out, by one of the four decode policies over captured graphs
  pack     freezing and packing a bf16 weight on the device, as the converter does tensor by tensor

Weights are random-init ternary codes and scales of the released geometries (no checkpoint is at hand), prompts
seeded uniform ids.  Random weights accept next to no draft token, so a decode case that stands for long accepted
blocks sets the confidence threshold to 0 (every chain is the whole block), and one that stands for rejected
blocks keeps the default threshold (every block goes to the verifier and commits one or two tokens).
"""
from __future__ import annotations

import math

import torch

from bitmtp_b200 import fast_generate, generate, ops, synthetic
from bitmtp_b200.fast_runtime import GraphAtlas
from bitmtp_b200.model import T2LinearKernel, t2g128_int8xint2_linear

DEVICE = "cuda"
SEGMENTS = (256, 1024, 4096)                     # the runtime's default segment ladder
WIDTHS = {4: (1, 4, 5, 6, 7, 8, 9), 8: (1, 8, 9, 10, 12, 16, 17)}      # replay widths the command line captures
GEOMETRY = {"1p7b": synthetic.BONSAI_1P7B, "4b": synthetic.BONSAI_4B}
POLICY = {"ar": fast_generate.fast_ar_generate, "spec": fast_generate.fast_speculative_generate,
          "hybrid": fast_generate.fast_hybrid_generate, "conf": fast_generate.fast_confidence_generate}


def _decode(name, geometry, policy, block, prompt, new, threshold=0.9, draft="native"):
    return {"name": name, "kind": "decode", "geometry": geometry, "policy": policy, "block": block, "prompt": prompt,
            "new": new, "threshold": threshold, "draft": draft}


def listed():
    return [
        # the smallest call: a key / value projection for one token, all latency
        {"name": "linear_kv_w1", "kind": "linear", "n": 1024, "k": 2048, "rows": 1, "form": "operator"},
        # a down projection at the width of a D8 verifier replay
        {"name": "linear_down_w9", "kind": "linear", "n": 2048, "k": 6144, "rows": 9, "form": "operator"},
        # the wide stress layer at eight tokens: the largest product a decode step sees besides the head
        {"name": "linear_wide_w8", "kind": "linear", "n": 28672, "k": 8192, "rows": 8, "form": "operator"},
        # a prompt of odd length through one gate projection used as a module
        {"name": "module_gate_333rows", "kind": "linear", "n": 6144, "k": 2048, "rows": 333, "form": "module"},
        # the converter's step for one merged gate|up weight
        {"name": "pack_gate_up", "kind": "pack", "n": 12288, "k": 2048},
        # a plain autoregressive request (the command line captures width 1 only for this mode)
        _decode("ar_256_64", "1p7b", "ar", 8, 256, 64),
        # the benchmark's request: whole blocks committed by confidence, draft width 16
        _decode("hybrid_blocks_256_256", "1p7b", "hybrid", 8, 256, 256, threshold=0.0),
        # hybrid with the e4m3 draft head and every block verified: draft width 9, verifier width 9
        _decode("hybrid_fp8_verify_97_48", "1p7b", "hybrid", 8, 97, 48, draft="fp8"),
        # four-token blocks, always verified
        _decode("spec_d4_300_40", "1p7b", "spec", 4, 300, 40),
        # a long document, then a short answer: the prompt forward and attention over a long history
        _decode("conf_2900_80", "1p7b", "conf", 8, 2900, 80, threshold=0.0),
        # the larger geometry in the largest segment
        _decode("hybrid_4b_1100_64", "4b", "hybrid", 8, 1100, 64, threshold=0.0),
        # a short chat turn: time to a handful of tokens
        _decode("hybrid_chat_19_9", "1p7b", "hybrid", 8, 19, 9),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _cost(case):
    w = work(case)
    return w["bytes"] + w["flops"] / 200


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("linear", "linear", "decode", "decode", "decode", "pack"))
        if kind == "pack":
            case = {"kind": "pack", "n": 8 * _log_int(rng, 128, 4096), "k": 128 * rng.randint(4, 76)}
        elif kind == "linear":
            form = rng.choice(("operator", "module"))
            n, k = 8 * _log_int(rng, 64, 4096), rng.choice((2048, 2560, 4096, 6144, 8192, 9728, 128 * rng.randint(2, 76)))
            rows = rng.randint(1, 17) if form == "operator" else _log_int(rng, 1, 2048)
            case = {"kind": "linear", "n": n, "k": k, "rows": rows, "form": form}
        else:
            geometry = rng.choice(("1p7b", "1p7b", "4b"))
            policy = rng.choice(("ar", "spec", "hybrid", "conf"))
            block = 8 if geometry == "4b" else rng.choice((4, 8))
            threshold = {"ar": 0.9, "spec": 0.9, "conf": 0.0}.get(policy, rng.choice((0.0, 0.9)))
            # the dense draft heads where a verifier follows: their summation order may not decide a committed id
            verified = policy == "spec" or (policy == "hybrid" and threshold > 0.0)
            case = _decode("", geometry, policy, block, _log_int(rng, 8, 3000), _log_int(rng, 8, 256), threshold=threshold,
                           draft=rng.choice(("native", "native", "fp8", "bf16")) if verified else "native")
            del case["name"]
        if _cost(case) <= limit:
            return case


# --------------------------------------------------------------------------- what a pass cannot do without
def _replays(case):
    """(width, logit rows, history length) of every graph replay of a decode case."""
    D, prompt, new, policy = case["block"], case["prompt"], case["new"], case["policy"]
    if policy == "ar":
        return [(1, 1, prompt + i) for i in range(new - 1)]
    if policy != "spec" and case["threshold"] == 0.0:
        blocks = math.ceil((new if policy == "conf" else new - 1) / D)
        return [(2 * D if i else D + (policy != "conf"), D, prompt + D * max(i - 1, 0)) for i in range(blocks)]
    # one committed token per verified block
    return [r for i in range(new - 1) for r in ((D + 1, D, prompt + i), (D + 1, D + 1, prompt + i))]


def work(case):
    if case["kind"] == "pack":
        n, k = case["n"], case["k"]
        return {"bytes": 2 * n * k + n * k // 4 + 2 * n * (k // 128), "flops": 2 * n * k}
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["rows"]
        act = m * k + 4 * m if case["form"] == "operator" else 2 * m * k
        return {"bytes": n * k // 4 + 2 * n * (k // 128) + act + 2 * m * n, "flops": 2 * m * n * k}
    g = GEOMETRY[case["geometry"]]
    q, kv = g["n_heads"] * 128, g["n_kv_heads"] * 128
    per_layer = g["dim"] * (q + 2 * kv) + q * g["dim"] + 3 * g["dim"] * g["ffn_dim"]
    params, head, L = g["n_layers"] * per_layer, g["vocab_size"] * g["dim"], g["n_layers"]
    packed = lambda p: p // 4 + 2 * (p // 128)
    kv_row = 2 * L * kv * 2                                     # bytes of one position's K and V
    T = case["prompt"]
    # the prompt: every weight once, K / V rows written, causal scores and products, one row of logits
    nbytes = packed(params) + packed(head) + 2 * T * g["dim"] + T * kv_row
    flops = 2 * params * T + 2 * L * q * T * T + 2 * head
    for width, rows, hist in _replays(case):
        verifier = rows == case["block"] + 1
        head_bytes = packed(head) if case["draft"] == "native" or verifier else head * (1 if case["draft"] == "fp8" else 2)
        nbytes += packed(params) + head_bytes + hist * kv_row + 2 * width * g["dim"]
        flops += 2 * params * width + 2 * head * rows + 4 * L * q * width * hist
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """A packed product: exact integer group sums, fp32 scale sums, one bf16 rounding - another order of the fp32
    sums moves a few results by one bf16 step (at most 2^-7 of a value).  A request's ids are whole values, and its
    K / V rows feed every later id through bf16 roundings, so the package fixes the order of every fp32 sum."""
    if case["kind"] == "linear":
        return {"rel": 1e-3, "max": 8e-3}
    return "exact"


# --------------------------------------------------------------------------- inputs and passes
def _ternary(n, k, gen):
    return synthetic.device_ternary(n, k, gen, DEVICE)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    if case["kind"] == "pack":
        # a trained latent weight: normal, with a spread of its own in every 128-group
        w = torch.randn(case["n"], case["k"] // 128, 128, generator=gen, device=DEVICE)
        w *= torch.rand(case["n"], case["k"] // 128, 1, generator=gen, device=DEVICE) * 0.04 + 0.01
        return {"case": case, "w": w.view(case["n"], case["k"]).to(torch.bfloat16)}
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["rows"]
        packed, scale = _ternary(n, k, gen)
        x = torch.randn(m, k, generator=gen, device=DEVICE).to(torch.bfloat16)
        if case["form"] == "module":
            layer = T2LinearKernel(k, n).to(DEVICE)
            layer.weight.data, layer.weight_scale = packed, scale
            return {"case": case, "layer": layer, "x": x}
        a, s = ops.quant_rows(x)
        return {"case": case, "a": a, "s": s, "packed": packed, "scale": scale}
    D, widths = case["block"], WIDTHS[case["block"]]
    roles = ("ar",)
    if case["policy"] == "ar":
        widths = (1,)
    else:
        roles += ({"native": "draft", "fp8": "draft_fp8", "bf16": "draft_bf16"}[case["draft"]],)
        roles += ("verify",) if case["policy"] != "conf" else ()
    cfg = synthetic.make_config(GEOMETRY[case["geometry"]], block_size=D)
    state = synthetic.device_state(cfg, DEVICE, seed=seed)
    head = state.pop("_head.weight"), state.pop("_head.weight_scale")
    model = generate.model_from_state(generate.args_from_config(cfg), state, DEVICE)
    model._lm_head_t2_w, model._lm_head_t2_scale = head          # the tied head as packed with the checkpoint
    model._lm_head_t2_vocab = model._lm_head_n_pad = cfg["vocab_size"]
    need = case["prompt"] + case["new"] + max(widths)
    segment = next(s for s in SEGMENTS if s >= need)
    model.prepare_merged_weights(max_positions=segment + max(widths))
    atlas = GraphAtlas(model, model.args, torch.device(DEVICE), segment_ladder=(segment,), m_set=widths, roles=roles,
                       capture_verbose=False)
    ids = torch.randint(0, cfg["vocab_size"], (1, case["prompt"]), generator=gen, device=DEVICE)
    return {"case": case, "model": model, "atlas": atlas, "ids": ids, "segment": segment}


def run(state):
    case = state["case"]
    if case["kind"] == "pack":
        return ops.pack_t2_g128(state["w"])
    if case["kind"] == "linear":
        if case["form"] == "module":
            return state["layer"](state["x"])
        return t2g128_int8xint2_linear(state["a"], state["packed"], state["s"], state["scale"])
    options = {}
    if case["policy"] != "ar":
        options = {"use_fp8_draft": case["draft"] == "fp8", "use_bf16_draft": case["draft"] == "bf16"}
        if case["policy"] != "spec":
            options["threshold"] = case["threshold"]
    tokens, _ = POLICY[case["policy"]](state["model"], state["atlas"], state["ids"], max_gen_len=case["new"], eos_ids=(),
                                       **options)
    # the request's K / V history: the prompt's rows and those of the tokens that no later block may revise
    rows = case["prompt"] + max(0, case["new"] - 1 - 2 * case["block"])
    return tokens, state["atlas"].kv_buffers[state["segment"]][:, :, :, :, :rows]
