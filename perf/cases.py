"""The workloads whose speed is measured, over every architecture the package serves.

A case is one of two things a program does with the package:

* ``kind`` "request": a batch of prompts arrives; its sequences are opened, the prompts run in one step (in chunks when
  they are long), then ``steps`` tokens are decoded for the batch, one step each, and the sequences are closed.  With
  ``steps`` 0 only the prompts run (the time to the first token).
* ``kind`` "decode": the sequences of a batch that is being served already hold their history; ``steps`` tokens are
  decoded for each, and the sequences are then set back to where they were (so that every pass does equal work; only
  for models whose sequences are nothing but keys and values).

Token ids, prompts' and decoded ones alike, are given: what a step returns are its logits, and every result of a case
is logits [sequences, vocabulary] (of the prompts' last places, then of each decoded step).  Weights are random, bf16 or
fp32, with spreads that keep scores, gates and routers in their working range (see ``weight``).

``exact`` computes the same logits in 64 bits from the formulas, on whole sequences: it has no cache, no chunks and no
code in common with the package.
"""
from __future__ import annotations

import json
import math
import os
import tempfile
import zlib
from typing import Dict, List

import torch
import torch.nn.functional as F

DEVICE = "cuda:0"
KINDS = {"bf16": torch.bfloat16, "fp32": torch.float32}

# ---------------------------------------------------------------------------------------------------------------------
# models: the sizes that bench.py runs
# ---------------------------------------------------------------------------------------------------------------------

MINICPM = {
    "8b": dict(num_hidden_layers=32, hidden_size=4096, num_attention_heads=32, num_key_value_heads=2, head_dim=128,
               intermediate_size=16384, tie_word_embeddings=False),
    "0.5b": dict(num_hidden_layers=24, hidden_size=1024, num_attention_heads=16, num_key_value_heads=2, head_dim=64,
                 intermediate_size=4096, tie_word_embeddings=True),
}
SPARSE = {"kernel_size": 32, "kernel_stride": 16, "block_size": 64, "init_blocks": 1, "topk": 64, "window_size": 2048,
          "dense_len": 8192}
SIZES = {
    "1k": dict(width=1024, heads=16, kv_heads=4, dim=64, vdim=64, lin_heads=8, lin_dim=64, lin_vdim=128, delta_heads=16,
               delta_qk_heads=8, delta_dim=64, delta_vdim=64, conv=4, experts=32, top=4, groups=4, keep=2, ff=512,
               shared=1024, streams=4, vocab=32000, q_rank=384, kv_rank=192, rot_dim=32, gru_ff=4096, gru_kv_rank=256),
    "2k": dict(width=2048, heads=16, kv_heads=4, dim=128, vdim=128, lin_heads=16, lin_dim=64, lin_vdim=128, delta_heads=16,
               delta_qk_heads=8, delta_dim=128, delta_vdim=128, conv=4, experts=64, top=6, groups=8, keep=4, ff=768,
               shared=1536, streams=4, vocab=32000, q_rank=768, kv_rank=448, rot_dim=64, gru_ff=8192, gru_kv_rank=512),
}
ROUTED = ("Mufevik", "Kipizen", "Lukelorn", "Rabadra")
NESTED = ROUTED + ("Reravik", "Dinutar")


def _minicpm(case: dict) -> dict:
    cfg = dict(MINICPM[case["size"]], num_hidden_layers=case["layers"])
    half = cfg["head_dim"] // 2
    cfg.update(architectures=["MiniCPMForCausalLM"], model_type="minicpm", vocab_size=73448, rope_theta=10000.0,
               max_position_embeddings=65536, rms_norm_eps=1e-6, scale_emb=12, dim_model_base=256, scale_depth=1.4,
               hidden_act="silu", torch_dtype="bfloat16",
               rope_scaling={"rope_type": "longrope", "long_factor": [1.0 + 39.0 * (i / half) ** 2 for i in range(half)],
                             "short_factor": [1.0] * half, "original_max_position_embeddings": 32768})
    if case["sparse"]:
        cfg["sparse_config"] = dict(SPARSE)
    return cfg


def config(case: dict) -> dict:
    """The config.json of the case's model."""
    if case["model"] == "MiniCPM4":
        return _minicpm(case)
    z, name = SIZES[case["size"]], case["model"]
    base = {"architecture": name, "vocab": z["vocab"], "width": z["width"], "norm": {"eps": 1e-5}}
    scale = z["dim"] ** -0.5
    if name == "Reravik":
        dense = {"kind": "dense", "ff": z["gru_ff"]}
        att = {"type": "latent_attention", "mlp": dense,
               "mixer": {"heads": z["heads"], "dim": z["dim"], "vdim": z["vdim"], "q_rank": z["q_rank"],
                         "kv_rank": z["gru_kv_rank"], "scale": scale, "mask": {"size": z["width"]}}}
        gru = {"type": "mingru", "mixer": {"width": z["width"]}, "mlp": dense}
        return dict(base, embedding={"scale": 12.0}, layers=[att, gru, gru, att, att, gru, gru, att],
                    loop={"start": 2, "stop": 6, "times": 2})
    if name == "Mufevik":
        mlp = {"kind": "moe", "router": {"experts": z["experts"], "top": z["top"],
                                         "groups": {"count": z["groups"], "keep": z["keep"]}},
               "expert": {"ff": z["ff"]}, "shared": {"ff": z["shared"]}}
        par = {"type": "parallel", "mlp": mlp,
               "mixer": {"left": {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": z["dim"], "vdim": z["vdim"],
                                  "scale": scale, "rot": {"dims": z["dim"], "base": 10000.0}},
                         "right": {"heads": z["lin_heads"], "dim": z["lin_dim"], "vdim": z["lin_vdim"], "tau": 8.0, "rank": 32}}}
        delta = {"type": "delta", "mlp": mlp,
                 "mixer": {"heads": z["delta_heads"], "kv_heads": z["delta_qk_heads"], "dim": z["delta_dim"],
                           "vdim": z["delta_vdim"], "conv": z["conv"]}}
        return dict(base, streams=z["streams"], logit_scale=1.0, layers=[delta, par, par, delta, delta, par, par, delta])
    if name == "Kipizen":
        mlp = {"kind": "moe", "router": {"experts": z["experts"], "top": z["top"]}, "expert": {"ff": z["ff"]}}
        n = z["lin_heads"]
        lin = {"type": "lightning", "mlp": mlp,
               "mixer": {"heads": n, "dim": z["lin_dim"], "vdim": z["lin_vdim"],
                         "decay": [1.0 - 2.0 ** (-1 - 7 * i / max(1, n - 1)) for i in range(n)]}}

        def attention(kv_from=None):
            m = {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": z["dim"], "vdim": z["vdim"], "scale": scale,
                 "softcap": 30.0, "mask": {"size": 1024},
                 "rot": {"dims": z["dim"] // 2, "base": 10000.0, "scaling": {"factor": 2.0}}}
            return {"type": "attention", "mlp": mlp, "mixer": m if kv_from is None else dict(m, kv_from=kv_from)}
        return dict(base, embedding={"scale": 1.0},
                    layers=[lin, attention(), attention(1), lin, lin, attention(), attention(5), lin])
    if name == "Lukelorn":
        moe = {"kind": "moe", "router": {"experts": z["experts"], "top": z["top"]}, "expert": {"ff": z["ff"]}}
        att = {"type": "attention", "mlp": moe,
               "mixer": {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": z["dim"], "vdim": z["vdim"], "scale": scale,
                         "softcap": 30.0, "mask": {"size": 1024, "keep_first": 64},
                         "rot": {"dims": z["dim"], "base": 500000.0,
                                 "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
        delta = {"type": "channel_delta", "mlp": moe,
                 "mixer": {"heads": z["delta_heads"], "kv_heads": z["delta_qk_heads"], "dim": z["delta_dim"],
                           "vdim": z["delta_vdim"], "conv": z["conv"], "decay_rank": 32, "gate_rank": 32}}
        latent = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": z["ff"] * z["top"]},
                  "mixer": {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot_dim"], "vdim": z["vdim"],
                            "q_rank": z["q_rank"], "kv_rank": z["kv_rank"], "scale": (z["dim"] + z["rot_dim"]) ** -0.5,
                            "mask": {"size": 1024}, "rot": {"dims": z["rot_dim"], "base": 10000.0}}}
        return dict(base, residual_mult=0.5, layers=[delta, att, dict(att, weights_of=1), latent,
                                                     delta, att, dict(att, weights_of=5), latent])
    if name == "Dinutar":
        n, mlp = z["delta_heads"], {"kind": "dense", "ff": z["ff"] * z["top"]}
        ret = {"type": "retention", "mlp": mlp,
               "mixer": {"heads": n, "dim": z["delta_dim"], "vdim": z["delta_vdim"],
                         "decay": [1.0 - 2.0 ** (-5 - 7 * i / max(1, n - 1)) for i in range(n)],
                         "rot": {"dims": z["delta_dim"], "base": 10000.0}}}

        def latent(kv_from=None):
            m = {"heads": z["heads"], "dim": z["dim"], "rot_dim": z["rot_dim"], "vdim": z["vdim"], "kv_rank": z["kv_rank"],
                 "scale": (z["dim"] + z["rot_dim"]) ** -0.5,
                 "rot": {"dims": z["rot_dim"], "base": 10000.0,
                         "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
            return {"type": "latent_attention", "mlp": mlp, "mixer": m if kv_from is None else dict(m, kv_from=kv_from)}
        return dict(base, postln_alpha=2.0, embedding={"scale": 1.0, "bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 17}},
                    layers=[ret, latent(), ret, latent(1), ret, latent(), ret, latent(5)])
    layer = {"type": "attention",
             "mixer": {"heads": z["heads"], "kv_heads": z["kv_heads"], "dim": z["dim"], "vdim": z["vdim"], "scale": scale,
                       "rot": {"dims": z["dim"], "base": 500000.0}},
             "mlp": {"kind": "moe", "expert": {"ff": z["ff"], "limit": 7.0}, "shared": {"ff": z["shared"], "limit": 7.0},
                     "router": {"experts": z["experts"], "top": z["top"], "scale": 2.0,
                                "groups": {"count": z["groups"], "keep": z["keep"]}}}}
    return dict(base, logit_softcap=25.0, layers=[layer] * 6 + [dict(layer, weights_of=0), dict(layer, weights_of=1)])


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------

def _case(name, kind, model, size, batch, longest, shortest, steps, dtype="bf16", layers=0, sparse=False, chunk=2048) -> dict:
    c = {"kind": kind, "model": model, "size": size, "layers": layers, "sparse": sparse, "dtype": dtype, "batch": batch,
         "longest": longest, "shortest": shortest, "steps": steps, "chunk": chunk}
    return dict(c, name=name) if name else c


def listed() -> List[dict]:
    return [
        # one short turn of a chat on the small model: latency of every launch
        _case("turn_half_b", "request", "MiniCPM4", "0.5b", 1, 61, 61, 16, layers=24),
        # the time to the first token of the headline model: one prompt of 2,048 tokens
        _case("prompt_8b", "request", "MiniCPM4", "8b", 1, 2048, 2048, 0, layers=32),
        # the headline model serving eight conversations of unequal lengths
        _case("decode_8b", "decode", "MiniCPM4", "8b", 8, 4085, 513, 8, layers=32),
        # many long conversations on the small model
        _case("decode_half_b_64", "decode", "MiniCPM4", "0.5b", 64, 8000, 500, 8, layers=24),
        # a long document under block-sparse attention, layers of the headline model, then its answer
        _case("document_sparse", "request", "MiniCPM4", "8b", 1, 12345, 12345, 8, layers=8, sparse=True),
        # the 32-bit path: three prompts in one step and a few more tokens
        _case("replay_fp32", "request", "MiniCPM4", "0.5b", 3, 400, 50, 4, dtype="fp32", layers=24),
        # the other designs: a batch of prompts of unequal lengths, then tokens; in the order of their sizes a crowd of short
        # requests, ordinary ones, long ones
        _case("crowd_mufevik", "request", "Mufevik", "1k", 16, 200, 20, 32),
        _case("batch_reravik", "request", "Reravik", "2k", 4, 1900, 90, 16),
        _case("batch_dinutar", "request", "Dinutar", "2k", 8, 700, 100, 32),
        _case("batch_lukelorn", "request", "Lukelorn", "2k", 3, 2500, 700, 16),
        _case("batch_rabadra", "request", "Rabadra", "2k", 4, 3000, 500, 16),
        _case("long_kipizen", "request", "Kipizen", "2k", 1, 4096, 4096, 16),
    ]


def draw(rng) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    steps = log(1, 32)
    chunk = rng.choice([1024, 2048])
    which = rng.choice(("MiniCPM4", "MiniCPM4", "MiniCPM4") + NESTED + NESTED)
    if which != "MiniCPM4":
        batch, longest = log(1, 16), log(16, 4096)
        longest = min(longest, 8192 // batch)
        return _case(None, "request", which, rng.choice(["1k", "2k"]), batch, longest, max(8, log(max(8, longest // 20), longest)),
                     steps, chunk=chunk)
    form = rng.choice(["request", "decode", "sparse", "fp32"])
    if form == "fp32":
        longest = log(8, 500)
        return _case(None, "request", "MiniCPM4", "0.5b", log(1, 4), longest, log(8, longest), min(steps, 8), dtype="fp32",
                     layers=24, chunk=chunk)
    if form == "sparse":
        longest = log(2000, 14000)
        return _case(None, "request", "MiniCPM4", "8b", 1, longest, longest, min(steps, 16), layers=8, sparse=True, chunk=2048)
    size = rng.choice(["0.5b", "8b"])
    layers = 24 if size == "0.5b" else 32
    if form == "decode":
        batch = log(1, 64 if size == "0.5b" else 12)
        longest = log(64, 4096)
        return _case(None, "decode", "MiniCPM4", size, batch, longest, log(32, longest), min(steps, 8), layers=layers, chunk=chunk)
    batch, longest = log(1, 8), log(8, 2048)
    longest = max(8, min(longest, (4096 if size == "0.5b" else 2048) // batch))
    return _case(None, "request", "MiniCPM4", size, batch, longest, log(8, longest), steps if size == "0.5b" else min(steps, 4),
                 layers=layers, chunk=chunk)


def lengths(case: dict) -> List[int]:
    """The sequences' lengths, from the longest to the shortest in equal ratios."""
    n, a, b = case["batch"], case["longest"], min(case["shortest"], case["longest"])
    return [int(round(a * (b / a) ** (i / max(1, n - 1)))) for i in range(n)]


def _vocab(case: dict) -> int:
    return 73448 if case["model"] == "MiniCPM4" else SIZES[case["size"]]["vocab"]


def tokens(case: dict, seed: int) -> List[List[int]]:
    """Every sequence's prompt or history, with the decoded tokens behind it."""
    g = torch.Generator().manual_seed(seed * 7919 + 17)
    return [torch.randint(0, _vocab(case), (n + case["steps"],), generator=g).tolist() for n in lengths(case)]


#: Weights by the end of their name: (mean, spread).  Matrices and biases are N(0, 0.02), norm weights N(1, 0.02); the
#: projections back into a deep model's stream are smaller.
SPREAD = {"o_proj.weight": (0.0, 0.008), "down_proj.weight": (0.0, 0.008), ".b": (0.0, 0.02), ".correction": (0.0, 0.02), ".sink": (0.0, 1.0), ".conv": (0.3, 0.1), ".A_log": (0.3, 0.3),
          ".dt_bias": (0.3, 0.3), ".shift": (0.5, 0.2), "loop.step": (0.0, 0.02), ".norm1": (1.0, 0.02), ".norm2": (1.0, 0.02),
          ".norm1b": (1.0, 0.02), ".norm2b": (1.0, 0.02), ".norm": (1.0, 0.02), "norm.weight": (1.0, 0.02),
          ".out": (1.0, 0.02), ".ls1": (1.0, 0.02), ".ls2": (1.0, 0.02), ".temp": (1.0, 0.02)}


def weight(case: dict, seed: int, name: str, shape) -> torch.Tensor:
    """A random weight, the same for the same seed and name.  Models of routed experts are given what makes a trained
    router's choice firm, so that a rounding that lets a token take another expert last moves its output little:
    projections back into the residual stream of smaller spread, tokens that share a direction in the stream, and routers
    of three times the spread that look away from it (most experts score near zero, the last chosen one little)."""
    g = torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFFFFFFFFFF)
    mean, spread = next((v for end, v in sorted(SPREAD.items(), key=lambda e: -len(e[0])) if name.endswith(end)), (0.0, 0.02))
    if case["model"] == "Lukelorn" and (name.endswith(".norm1") or name == "final.norm"):
        mean = 0.0                                     # stored around zero
    routed = case["model"] in ROUTED
    if routed and name.endswith((".o", ".down", "embed", ".router")):
        back = 0.004 if case["model"] == "Rabadra" else 0.01          # its experts' weights add up to two
        spread = {"o": back, "down": back, "embed": 1.0, "router": 0.06}[name.rsplit(".", 1)[-1]]
    if case["sparse"] and name.endswith(("q_proj.weight", "k_proj.weight")):
        spread = 0.01                                  # no single key decides: a block chosen otherwise moves little
    t = torch.randn(tuple(shape), generator=g, device=DEVICE) * spread + mean
    if routed and name.endswith(("embed", ".router")):
        t[:, ::2] += 0.5 if name == "embed" else -13.0 / shape[1]
        t[:, 1::2] -= 0.5 if name == "embed" else -13.0 / shape[1]
    if name.endswith((".hc1.mix", ".hc2.mix", ".talk")):
        t += torch.eye(shape[0], device=DEVICE)
    if name.endswith((".hc1.in", ".hc2.in")):
        t += 1.0 / shape[0]
    return t.to(KINDS[case["dtype"]])


# ---------------------------------------------------------------------------------------------------------------------
# the measured path
# ---------------------------------------------------------------------------------------------------------------------

class _State:
    pass


def prepare(case: dict, seed: int):
    """A serving program: a model with its weights, a cache, the decode runner, recorded graphs; the requests."""
    from cpmcu_b200 import LLM, SamplingParams
    from cpmcu_b200.engine import SequenceStep
    from cpmcu_b200.engine.decode import DecodeRunner

    st = _State()
    st.case, st.step_type, st.greedy = case, SequenceStep, SamplingParams()
    ids = tokens(case, seed)
    n, k = case["batch"], case["steps"]
    most = max(4096, max(map(len, ids))) + 64
    with tempfile.TemporaryDirectory() as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(config(case), f)
        st.llm = LLM(folder, dtype=KINDS[case["dtype"]], chunk_length=case["chunk"], cuda_graph=True,
                     max_tokens=sum(len(s) + 128 for s in ids) + 256, max_seq_tokens=most)
    st.llm.init_storage()
    st.llm.load_tensors({name: weight(case, seed, name, spec.shape) for name, spec in st.llm.model.weight_specs().items()})
    st.runner = DecodeRunner(st.llm.stepper, use_graph=True, seed=seed)
    st.prompts = [s[:len(s) - k] for s in ids]
    st.fed = [[s[len(s) - k + j] for s in ids] for j in range(k)]
    if case["kind"] == "decode":
        st.slots = st.llm.stepper.open(n)
        for slot, prompt in zip(st.slots, st.prompts):
            st.llm.step([SequenceStep(slot, prompt, [])])
    run(st)                                            # graphs are recorded once in a program's life
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return st


def _decode(st, slots) -> List[torch.Tensor]:
    runner, n, out = st.runner, len(slots), []
    for j, fed in enumerate(st.fed):
        if j == 0:
            runner.start(slots, fed, list(range(n)), [1] * n, [st.greedy] * n)
        else:
            runner.feed(fed)
        runner.step()
        out.append(runner.logits().clone())
    return out


def run(st):
    case, stepper = st.case, st.llm.stepper
    if case["kind"] == "decode":
        steps = _decode(st, st.slots)
        for slot, prompt in zip(st.slots, st.prompts):
            stepper.cache.set_length(slot, len(prompt))
        return {"steps": steps}
    slots = stepper.open(case["batch"])
    first = st.llm.step([st.step_type(s, p, [len(p) - 1]) for s, p in zip(slots, st.prompts)])
    steps = _decode(st, slots)
    for s in slots:
        stepper.close(s)
    return {"prompts": first, "steps": steps}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------

def work(case: dict) -> dict:
    """Weights are read once a step (of a mixture, the experts that its tokens are expected to choose), the keys and values
    or the state of every sequence once a decoded step, logits are written; products and attention are counted for the
    tokens that need them."""
    cfg, es, k, n = config(case), 2 if case["dtype"] == "bf16" else 4, case["steps"], case["batch"]
    lens = lengths(case)
    if case["model"] == "MiniCPM4":
        h, d, H, G, L = (cfg[x] for x in ("hidden_size", "head_dim", "num_attention_heads", "num_key_value_heads", "num_hidden_layers"))
        head = cfg["vocab_size"] * h
        layers = [dict(dense=(2 * H + 2 * G) * d * h + 3 * h * cfg["intermediate_size"], row=2 * G * d, pair=4 * H * d,
                       reach=(SPARSE["topk"] * 64 + SPARSE["window_size"]) if case["sparse"] else 0)] * L
    else:
        z, W = SIZES[case["size"]], SIZES[case["size"]]["width"]
        head, layers = z["vocab"] * W, []
        order = list(range(len(cfg["layers"])))
        if "loop" in cfg:
            a, b, times = cfg["loop"]["start"], cfg["loop"]["stop"], cfg["loop"]["times"]
            order = order[:a] + order[a:b] * times + order[b:]
        for i in order:
            layer, e = cfg["layers"][i], dict(dense=0, row=0, pair=0, reach=0, state=0, experts=0, top=0, per=0)
            m, mlp = layer["mixer"], layer["mlp"]
            for t, p in ((layer["type"], m),) if layer["type"] != "parallel" else (("attention", m["left"]), ("lightning", m["right"])):
                if t == "mingru":
                    e["dense"] += 4 * W * W
                    e["state"] += W
                    continue
                H, d, dv = p["heads"], p["dim"], p["vdim"]
                if t == "attention":
                    G = p["kv_heads"]
                    own = 0 if "kv_from" in p else G * (d + dv) * W
                    e["dense"] += H * d * W + own + H * dv * W
                    e.update(row=G * (d + dv), pair=2 * H * (d + dv), reach=(p.get("mask") or {}).get("size", 0))
                elif t == "latent_attention":
                    R, dr = p["kv_rank"], p.get("rot_dim", 0)
                    q = p["q_rank"] * (W + H * (d + dr)) if "q_rank" in p else W * H * (d + dr)
                    e["dense"] += q + W * (R + dr) * ("kv_from" not in p) + R * H * (d + dv) + H * dv * W
                    e.update(row=R + dr, pair=2 * H * (d + dr + dv), reach=(p.get("mask") or {}).get("size", 0))
                else:
                    Hk = p.get("kv_heads", H)
                    e["dense"] += 2 * Hk * d * W + 3 * H * dv * W
                    e["state"] += H * d * dv
            if mlp["kind"] == "moe":
                mats = 2 if case["model"] == "Lukelorn" else 3
                e.update(experts=z["experts"], top=z["top"], per=mats * z["ff"] * W)
                e["dense"] += z["experts"] * W + 3 * W * (mlp.get("shared") or {}).get("ff", 0)
            else:
                e["dense"] += (2 if case["model"] == "Dinutar" else 3) * W * mlp["ff"]
            layers.append(e)
    nbytes = flops = 0.0

    def products(rows: int, steps: int):
        nonlocal nbytes, flops
        for e in layers:
            hit = e.get("experts", 0) * (1.0 - (1.0 - e["top"] / e["experts"]) ** rows) if e.get("experts") else 0
            nbytes += steps * es * (e["dense"] + hit * e.get("per", 0))
            flops += steps * 2.0 * rows * (e["dense"] + e.get("top", 0) * e.get("per", 0))
        nbytes += steps * (es * head + 4 * n * _vocab(case))
        flops += steps * 2.0 * n * head

    if case["kind"] == "request":
        products(sum(lens), 1)
        for e in layers:
            for length in lens:
                reach = min(length, e["reach"] or length)
                seen = reach * (reach + 1) / 2 + (length - reach) * reach
                nbytes += es * length * e["row"] + 4 * e.get("state", 0)
                flops += seen * e["pair"] + 4.0 * length * e.get("state", 0)
    products(n, k)
    for e in layers:
        for length in lens:
            reach = min(length + k / 2, e["reach"] or length + k / 2)
            nbytes += k * (es * reach * e["row"] + 8 * e.get("state", 0))
            flops += k * (reach * e["pair"] + 4.0 * e.get("state", 0))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case: dict) -> dict:
    """About four times what the path was seen to be off ``exact``: 1.2e-6 to 2.5e-6 in fp32; in bf16 0.002 to 0.016, and more in a row
    whose token is given another last expert, or another last block, by a rounding."""
    if case["dtype"] == "fp32":
        return {"rel": 1e-5, "max": 4e-4}
    return {"rel": 0.03, "max": 0.9 if case["model"] in ROUTED or case["sparse"] else 0.4}


# ---------------------------------------------------------------------------------------------------------------------
# the same logits in 64 bits
# ---------------------------------------------------------------------------------------------------------------------

def _rms(x, weight=None, eps=1e-5):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _layer_norm(x, weight, bias, eps=1e-5):
    c = x - x.mean(-1, keepdim=True)
    return c * torch.rsqrt((c * c).mean(-1, keepdim=True) + eps) * weight + bias


def _angles(T, freq, magnitude=1.0):
    a = torch.arange(T, dtype=torch.float64, device=DEVICE)[:, None] * freq[None]
    return (torch.cos(a) * magnitude)[:, None, :], (torch.sin(a) * magnitude)[:, None, :]


def _turn_halves(x, freq, magnitude=1.0):
    """x [B, T, heads, d]: column i < n is paired with column i + n, n the number of frequencies."""
    n = freq.numel()
    c, s = _angles(x.shape[1], freq, magnitude)
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], dim=-1)


def _turn_pairs(x, freq):
    """x [B, T, heads, d]: columns 2i and 2i + 1 are a pair."""
    n = freq.numel()
    c, s = _angles(x.shape[1], freq)
    u, v = x[..., 0:2 * n:2], x[..., 1:2 * n:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2), x[..., 2 * n:]], dim=-1)


def _frequencies(rot, kind=""):
    dims, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEVICE)
    f = base ** (-2.0 * i / dims)
    if kind == "Kipizen" and sc:
        f = f / sc["factor"]
    if kind == "Lukelorn" and sc:
        wave = 2.0 * math.pi / f
        blend = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
        mid = (1.0 - blend) * f / sc["factor"] + blend * f
        f = torch.where(wave < sc["original"] / sc["high"], f, torch.where(wave > sc["original"] / sc["low"], f / sc["factor"], mid))
    if kind == "Dinutar" and sc:
        lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * sc[k])) / (2 * math.log(base)) for k in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0), min(math.ceil(hi), dims - 1)
        ramp = torch.clamp((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
        f = f / sc["factor"] * ramp + f * (1.0 - ramp)
    return f


def _attend(q, k, v, scale, cap=0.0, window=0, keep=0, sink=None, mix=None, allowed=None):
    """q [B, T, H, d], k [B, T, G, d], v [B, T, G, dv] -> [B, T, H, dv], causal, 512 queries at a time.  ``sink`` [H]: the
    score of a key without a value; ``mix`` [H, H]: weights mixed over heads after the softmax; ``allowed(first, last)``
    -> [queries, G, T] bool: keys a query may see besides those of the last rules."""
    B, T, H, d = q.shape
    rep = H // k.shape[2]
    kk, vv = k.repeat_interleave(rep, 2).permute(0, 2, 3, 1), v.repeat_interleave(rep, 2).transpose(1, 2)
    out = []
    for a in range(0, T, 512):
        b = min(T, a + 512)
        i, j = torch.arange(a, b, device=DEVICE)[:, None], torch.arange(b, device=DEVICE)[None]
        seen = j <= i
        if window:
            seen = seen & ((i - j < window) | (j < keep))
        if allowed is not None:
            seen = seen & allowed(a, b)[:, :, :b].repeat_interleave(rep, 1).transpose(0, 1)
        s = (q[:, a:b].transpose(1, 2) @ kk[..., :b]) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[None, :, None, None].expand(B, H, b - a, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., :b]
        if mix is not None:
            p = torch.einsum("hg,bgij->bhij", mix, p)
        out.append((p @ vv[:, :, :b]).transpose(1, 2))
    return torch.cat(out, dim=1)


def _recur(q, k, v, decay, beta=None):
    """S <- decay S; u = v, or beta (v - S^T k); S <- S + k u^T; o = S^T q; q, k [B, T, H, d], v [B, T, H, dv], decay
    broadcast over [B, T, H, d]."""
    B, T, H, d = q.shape
    S = torch.zeros(B, H, d, v.shape[-1], dtype=q.dtype, device=q.device)
    decay, out = decay.expand(B, T, H, decay.shape[-1]), torch.empty_like(v)
    for t in range(T):
        S = S * decay[:, t, :, :, None]
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - (k[:, t, :, None, :] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
    return out


class _Exact:
    def __init__(self, case, seed):
        self.case, self.seed, self.cfg, self.kind = case, seed, config(case), case["model"]

    def w(self, name, *shape):
        return weight(self.case, self.seed, name, shape).double()

    def lin(self, x, name, n):
        return x @ self.w(name, n, x.shape[-1]).T

    def heads(self, x, name, n, d):
        return self.lin(x, name, n * d).unflatten(-1, (n, d))

    def vec(self, name, n):
        return self.w(name, n)

    # ---- MiniCPM4 ----
    def minicpm(self, ids):
        c = self.cfg
        h, H, G, d, ff = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["intermediate_size"]
        eps, rs, sc = c["rms_norm_eps"], c["scale_depth"] / math.sqrt(c["num_hidden_layers"]), c["rope_scaling"]
        i = torch.arange(0, d, 2, dtype=torch.float64, device=DEVICE) / d
        f = 1.0 / (torch.tensor(sc["long_factor"], dtype=torch.float64, device=DEVICE) * c["rope_theta"] ** i)
        orig = sc["original_max_position_embeddings"]
        mag = math.sqrt(1.0 + math.log(c["max_position_embeddings"] / orig) / math.log(orig))
        table = self.w("model.embed_tokens.weight", c["vocab_size"], h)
        x = table[ids] * c["scale_emb"]
        del table
        for n in range(c["num_hidden_layers"]):
            p = f"model.layers.{n}."
            y = _rms(x, self.vec(p + "input_layernorm.weight", h), eps)
            q = _turn_halves(self.heads(y, p + "self_attn.q_proj.weight", H, d), f, mag)
            k = _turn_halves(self.heads(y, p + "self_attn.k_proj.weight", G, d), f, mag)
            v = self.heads(y, p + "self_attn.v_proj.weight", G, d)
            allowed = self.blocks(q, k, d ** -0.5) if "sparse_config" in c else None
            o = _attend(q, k, v, d ** -0.5, allowed=allowed).flatten(-2)
            x = x + rs * self.lin(o, p + "self_attn.o_proj.weight", h)
            y = _rms(x, self.vec(p + "post_attention_layernorm.weight", h), eps)
            a = F.silu(self.lin(y, p + "mlp.gate_proj.weight", ff)) * self.lin(y, p + "mlp.up_proj.weight", ff)
            x = x + rs * self.lin(a, p + "mlp.down_proj.weight", h)
        name = "model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight"
        return lambda rows: self.lin(_rms(x[:, rows], self.vec("model.norm.weight", h), eps) * (c["dim_model_base"] / h),
                                     name, c["vocab_size"])

    def blocks(self, q, k, scale):
        """Which keys the block-sparse rule lets a query see: [queries a to b, G, T]."""
        s, T, G = self.cfg["sparse_config"], k.shape[1], k.shape[2]
        ks, st, bs, per = s["kernel_size"], s["kernel_stride"], s["block_size"], s["block_size"] // s["kernel_stride"]
        reach = ks // st - 1
        pooled = k[0].unfold(0, ks, st).mean(-1)                                    # [N, G, d]
        N, nb = pooled.shape[0], (T + bs - 1) // bs

        def allowed(a, b):
            p = torch.arange(a, b, device=DEVICE)
            vis = torch.clamp((p + 1 - ks) // st + 1, min=0)
            sc = torch.einsum("tgrd,ngd->tgrn", q[0, a:b].unflatten(1, (G, -1)), pooled) * scale
            hidden = torch.arange(N, device=DEVICE)[None] >= vis[:, None]
            pr = torch.softmax(sc.masked_fill(hidden[:, None, None], float("-inf")), dim=-1).nan_to_num(0.0).sum(2)
            pr = pr.masked_fill(hidden[:, None], float("-inf"))
            pr = F.pad(pr, (reach, nb * per - N), value=float("-inf"))
            best = F.max_pool1d(pr, per + reach, per)[..., :nb]                     # [t, G, blocks]
            blk = torch.arange(nb, device=DEVICE)[None]
            last = (p // bs - s["window_size"] // bs)[:, None]
            can = (blk >= s["init_blocks"]) & (blk <= last)
            best = best.masked_fill(~can[:, None], float("-inf"))
            top = best.topk(min(s["topk"] - s["init_blocks"], nb), dim=-1)
            on = torch.zeros_like(best, dtype=torch.bool).scatter(-1, top.indices, top.values > float("-inf"))
            on = on | (blk < s["init_blocks"])[:, None] | (blk > last)[:, None] | (p + 1 <= s["dense_len"])[:, None, None]
            return on.repeat_interleave(bs, dim=-1)[..., :T]
        return allowed

    # ---- mixers of the other designs ----
    def latent(self, h, p, m, rows=None):
        H, d, dr, dv, R = m["heads"], m["dim"], m.get("rot_dim", 0), m["vdim"], m["kv_rank"]
        turn = (lambda x: x) if not dr else (lambda x: _turn_pairs(x, _frequencies(m["rot"]))) if self.kind == "Lukelorn" else \
            (lambda x: _turn_halves(x, _frequencies(m["rot"], "Dinutar"), 0.1 * math.log(m["rot"]["scaling"]["factor"]) + 1.0))
        if "q_rank" in m:
            q = self.heads(_rms(self.lin(h, p + "dq", m["q_rank"]), self.vec(p + "dq.norm", m["q_rank"])), p + "uq", H, d + dr)
        else:
            q = self.heads(h, p + "q", H, d + dr)
        if rows is None:
            down = self.lin(h, p + "dkv", R + dr)
            rows = (_rms(down[..., :R], self.vec(p + "dkv.norm", R)), turn(down[..., None, R:]))
        c, turned = rows
        k = torch.cat([self.heads(c, p + "uk", H, d), turned.expand(*turned.shape[:2], H, dr)], dim=-1)
        q = torch.cat([q[..., :d], turn(q[..., d:])], dim=-1)
        o = _attend(q, k, self.heads(c, p + "uv", H, dv), m["scale"], window=(m.get("mask") or {}).get("size", 0))
        if self.kind == "Lukelorn":
            o = o * torch.sigmoid(self.lin(h, p + "g", H))[..., None]
        return self.lin(o.flatten(-2), p + "o", h.shape[-1]), rows

    def attention(self, h, p, m, kept=None):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        W, rot, mask = h.shape[-1], m.get("rot"), m.get("mask") or {}
        q, f = self.lin(h, p + "q", H * d), _frequencies(rot, self.kind)
        turn = _turn_pairs if self.kind in ("Lukelorn", "Rabadra") else _turn_halves
        if self.kind == "Kipizen":
            q = q + self.vec(p + "q.b", H * d)
        if self.kind == "Rabadra":
            q = _rms(q, self.vec(p + "q.norm", H * d))
        q = turn(q.unflatten(-1, (H, d)), f)
        if kept is None:
            k, v = self.lin(h, p + "k", G * d), self.lin(h, p + "v", G * dv)
            if self.kind == "Kipizen":
                k, v = k + self.vec(p + "k.b", G * d), v + self.vec(p + "v.b", G * dv)
            if self.kind == "Rabadra":
                k = _rms(k, self.vec(p + "k.norm", G * d))
            k = turn(k.unflatten(-1, (G, d)), f)
            kept = (_rms(k) if self.kind == "Kipizen" else k, v.unflatten(-1, (G, dv)))
        if self.kind == "Kipizen":
            q = _rms(q)
        sink = mix = None
        if self.kind == "Kipizen":
            sink = torch.zeros(H, dtype=torch.float64, device=DEVICE)
        elif self.kind in ("Lukelorn", "Rabadra"):
            sink = self.vec(p + "sink", H)
        elif self.kind == "Mufevik":
            mix = self.w(p + "talk", H, H)
            q = q * self.vec(p + "temp", H)[:, None]
        o = _attend(q, *kept, m["scale"], m.get("softcap", 0.0), mask.get("size", 0), mask.get("keep_first", 0), sink, mix)
        if self.kind == "Lukelorn":
            o = o * torch.sigmoid(self.lin(h, p + "g", H))[..., None]
        return self.lin(o.flatten(-2), p + "o", W), kept

    def convolved(self, h, name, n, taps):
        x, w = self.lin(h, name, n), self.w(name + ".conv", n, taps)
        return F.silu(sum(F.pad(x, (0, 0, j, 0))[:, :x.shape[1]] * w[:, taps - 1 - j] for j in range(taps)))

    def delta(self, h, p, m):
        H, G, d, dv, W = m["heads"], m["kv_heads"], m["dim"], m["vdim"], h.shape[-1]
        q, k = (self.convolved(h, p + x, G * d, m["conv"]).unflatten(-1, (G, d)) for x in "qk")
        v = self.convolved(h, p + "v", H * dv, m["conv"]).unflatten(-1, (H, dv))
        q, k = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        q, k = (q * d ** -0.5).repeat_interleave(H // G, 2), k.repeat_interleave(H // G, 2)
        beta, rate = torch.sigmoid(self.lin(h, p + "b", H)), torch.exp(self.vec(p + "A_log", H))[:, None]
        if self.kind == "Mufevik":
            dt = F.softplus(self.lin(h, p + "a", H) + self.vec(p + "dt_bias", H), threshold=30)[..., None]
            gate = F.silu(self.lin(h, p + "g", H * dv))
        else:
            dt = F.softplus(self.lin(self.lin(h, p + "a1", m["decay_rank"]), p + "a2", H * d) + self.vec(p + "dt_bias", H * d),
                            threshold=30).unflatten(-1, (H, d))
            gate = torch.sigmoid(self.lin(self.lin(h, p + "g1", m["gate_rank"]), p + "g2", H * dv))
        o = _rms(_recur(q, k, v, torch.exp(-rate * dt), beta), self.vec(p + "norm", dv)).flatten(-2)
        return self.lin(o * gate, p + "o", W)

    def linear(self, h, p, m):
        H, d, dv, W = m["heads"], m["dim"], m["vdim"], h.shape[-1]
        q, k, v = self.heads(h, p + "q", H, d), self.heads(h, p + "k", H, d), self.heads(h, p + "v", H, dv)
        if self.kind == "Mufevik":
            z = self.lin(self.lin(h, p + "a1", m["rank"]), p + "a2", H * d) + self.vec(p + "a2.b", H * d)
            o = _recur(q * d ** -0.5, k, v, (torch.sigmoid(z) ** (1.0 / m["tau"])).unflatten(-1, (H, d)))
            return self.lin(_rms(o, self.vec(p + "norm", dv)).flatten(-2) * F.silu(self.lin(h, p + "g", H * dv)), p + "o", W)
        decay = torch.tensor(m["decay"], dtype=torch.float64, device=DEVICE)[None, None, :, None]
        if self.kind == "Dinutar":
            f = _frequencies(m["rot"])
            o = _recur(_turn_halves(q, f), _turn_halves(k, f) * d ** -0.5, v, decay)
            return self.lin(_rms(o).flatten(-2) * F.silu(self.lin(h, p + "g", H * dv)), p + "o", W)
        o = _recur(F.silu(q), F.silu(k), F.silu(v), decay).flatten(-2)
        return self.lin(_rms(o, self.vec(p + "norm", H * dv)) * torch.sigmoid(self.lin(h, p + "g", H * dv)), p + "o", W)

    def gru(self, h, p):
        W = h.shape[-1]
        z = torch.sigmoid(self.lin(h, p + "z", W) + self.vec(p + "z.b", W))
        u = self.lin(h, p + "x", W) + self.vec(p + "x.b", W)
        add = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        S, out = torch.zeros_like(z[:, 0]), torch.empty_like(z)
        for t in range(z.shape[1]):
            S = (1.0 - z[:, t]) * S + add[:, t]
            out[:, t] = S
        return self.lin(out * F.silu(self.lin(h, p + "g", W)), p + "o", W)

    # ---- feed-forwards ----
    def expert(self, h, p, ff, limit=None):
        W, u = h.shape[-1], self.lin(h, p + "up", ff)
        if self.kind in ("Lukelorn", "Dinutar") and (self.kind == "Dinutar" or ".e" in p):
            return self.lin(torch.relu(u) ** 2, p + "down", W)
        g = self.lin(h, p + "gate", ff)
        if limit is not None:
            g, u = torch.clamp(g, max=limit), torch.clamp(u, -limit, limit)
            return self.lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), p + "down", W)
        return self.lin((F.gelu(g, approximate="tanh") if self.kind == "Reravik" else F.silu(g)) * u, p + "down", W)

    def feed_forward(self, h, p, mlp):
        if mlp["kind"] == "dense":
            return self.expert(h, p, mlp["ff"])
        shape, h = h.shape, h.flatten(0, 1)
        r, E, limit = mlp["router"], mlp["router"]["experts"], mlp["expert"].get("limit")
        z = self.lin(h, p + "router", E)
        if self.kind == "Kipizen":
            val, idx = torch.topk(z + self.vec(p + "router.b", E), r["top"], dim=-1)
            wt = torch.softmax(val, dim=-1)
        else:
            s = torch.softmax(z, dim=-1) if self.kind == "Mufevik" else torch.sigmoid(z)
            choice = s + self.vec(p + "correction", E) if self.kind == "Mufevik" else s
            if "groups" in r:
                by_group = choice.unflatten(-1, (r["groups"]["count"], -1))
                score = by_group.amax(-1) if self.kind == "Mufevik" else by_group.topk(2, dim=-1).values.sum(-1)
                kept = torch.zeros_like(score, dtype=torch.bool).scatter(1, score.topk(r["groups"]["keep"], dim=-1).indices, True)
                choice = by_group.masked_fill(~kept[..., None], float("-inf")).flatten(-2)
            idx = choice.topk(r["top"], dim=-1).indices
            wt = torch.gather(s, 1, idx)
            if self.kind == "Rabadra":
                wt = wt / (wt.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = torch.zeros_like(h)
        for e in range(E):
            rows, place = (idx == e).nonzero(as_tuple=True)
            if rows.numel():
                g = wt[rows, place][:, None]
                x = h[rows] * g if self.kind == "Lukelorn" else h[rows]
                y = self.expert(x, f"{p}e{e}.", mlp["expert"]["ff"], limit)
                out[rows] += y if self.kind == "Lukelorn" else y * g
        if mlp.get("shared"):
            y = self.expert(h, p + "shared.", mlp["shared"]["ff"], mlp["shared"].get("limit"))
            out = out + (y * torch.sigmoid(self.lin(h, p + "shared.sg", 1)) if self.kind == "Mufevik" else y)
        return out.view(shape)

    # ---- the other designs ----
    def mixer(self, h, p, layer, i, kept):
        m, t = layer["mixer"], layer["type"]
        if t == "attention" or t == "latent_attention":
            o, kept[i] = (self.attention if t == "attention" else self.latent)(h, p, m, kept.get(m["kv_from"]) if "kv_from" in m else None)
            return o
        if t == "mingru":
            return self.gru(h, p)
        if t == "parallel":
            W = h.shape[-1]
            a, b = self.attention(h, p + "left.", m["left"])[0], self.linear(h, p + "right.", m["right"])
            return 0.5 * (_rms(a, self.vec(p + "left.out", W)) + _rms(b, self.vec(p + "right.out", W)))
        return self.delta(h, p, m) if "delta" in t else self.linear(h, p, m)

    def nested(self, ids):
        cfg, kind, W, V = self.cfg, self.kind, self.cfg["width"], self.cfg["vocab"]
        T, vec, lin, kept = ids.shape[1], self.vec, self.lin, {}
        x = self.w("embed", V, W)[ids] * (cfg.get("embedding") or {}).get("scale", 1.0)
        if kind == "Reravik":
            i = torch.arange(W // 2, dtype=torch.float64, device=DEVICE)
            a = torch.arange(T, dtype=torch.float64, device=DEVICE)[:, None] * (10000.0 ** (-2.0 * i / W))[None]
            x = x + torch.stack([torch.sin(a), torch.cos(a)], dim=-1).flatten(-2)
        elif kind == "Dinutar":
            b = cfg["embedding"]["bigram"]
            row = (F.pad(ids, (1, 0))[:, :-1] * b["mul_prev"] + ids * b["mul_cur"]) % b["buckets"]
            row[:, 0] = b["buckets"]
            x = _rms(x + self.w("bigram", b["buckets"] + 1, W)[row], vec("embed.norm", W))
        elif kind == "Rabadra":
            x = _layer_norm(x, vec("embed.norm", W), 0.0)
        embedded, order = x, [(i, None) for i in range(len(cfg["layers"]))]
        if kind == "Reravik":
            a, b, times = cfg["loop"]["start"], cfg["loop"]["stop"], cfg["loop"]["times"]
            order = order[:a] + [(i, t if i == a else None) for t in range(times) for i in range(a, b)] + order[b:]
        if kind == "Mufevik":
            x = x[:, :, None, :].repeat(1, 1, cfg["streams"], 1)
        for i, enters in order:
            layer = cfg["layers"][i]
            p = f"l{layer.get('weights_of', i)}."
            mix, feed = (lambda h: self.mixer(h, p + "mix.", layer, i, kept)), (lambda h: self.feed_forward(h, p + "mlp.", layer["mlp"]))
            if kind == "Reravik":
                if enters is not None:
                    x = x + (embedded if enters else 0.0) + self.w("loop.step", cfg["loop"]["times"], W)[enters]
                norm = lambda y, n: _layer_norm(y, vec(p + n, W), vec(p + n + ".b", W))  # noqa: E731
                h = norm(x, "norm1")
                h = h + (F.pad(h, (0, 0, 1, 0))[:, :-1] - h) * vec(p + "shift", W)
                x = x + norm(mix(h), "norm1b")
                x = x + norm(feed(norm(x, "norm2")), "norm2b")
            elif kind == "Mufevik":
                for n, part in (("1", mix), ("2", feed)):
                    S, q = cfg["streams"], f"{p}hc{n}."
                    u = torch.einsum("s,btsw->btw", vec(q + "in", S), x)
                    y = part(_rms(u) * self.w(p + "norm" + n))
                    x = torch.einsum("sr,btsw->btrw", self.w(q + "mix", S, S), x) + vec(q + "out", S)[:, None] * y[:, :, None, :]
            elif kind == "Dinutar":
                for n, part in (("1", mix), ("2", feed)):
                    x = _rms(cfg["postln_alpha"] * x + vec(p + "ls" + n, W) * part(x), vec(p + "norm" + n, W))
            elif kind == "Kipizen":
                x = x + mix(_rms(x, vec(p + "norm1", W)))
                x = x + feed(_rms(x, vec(p + "norm2", W)))
            elif kind == "Lukelorn":
                h = _rms(x, vec(p + "norm1", W) + 1.0)
                x = x + cfg["residual_mult"] * (mix(h) + feed(h))
            else:
                x = x + mix(_layer_norm(x, vec(p + "norm1", W), 0.0)) + feed(_layer_norm(x, vec(p + "norm2", W), 0.0))
        if kind == "Mufevik":
            x = x.sum(2)

        def logits(rows):
            y = x[:, rows]
            if kind == "Reravik":
                y = _layer_norm(y, vec("final.norm", W), vec("final.norm.b", W))
            elif kind == "Rabadra":
                y = _layer_norm(y, vec("final.norm", W), 0.0)
            elif kind == "Mufevik":
                y = _rms(y) * self.w("final.norm")
            else:
                y = _rms(y, vec("final.norm", W) + (1.0 if kind == "Lukelorn" else 0.0))
            z = lin(y, "embed" if kind == "Dinutar" else "head", V)
            cap = cfg.get("logit_softcap")
            return cap * torch.tanh(z / cap) if cap else z * cfg.get("logit_scale", 1.0)
        return logits


def exact(case: dict, seed: int):
    """What ``run`` returns, in 64 bits.  The sequences run one by one where that is cheaper, else side by side, the shorter
    ones filled up behind their end (no place sees a later one)."""
    model, ids, k = _Exact(case, seed), tokens(case, seed), case["steps"]
    alone = case["model"] == "MiniCPM4"
    rows: Dict[int, torch.Tensor] = {}
    if alone:
        for b, s in enumerate(ids):
            at = model.minicpm(torch.tensor([s], device=DEVICE))
            rows[b] = at(torch.arange(len(s) - k - 1, len(s), device=DEVICE))[0]
    else:
        most = max(map(len, ids))
        at = model.nested(torch.tensor([s + [0] * (most - len(s)) for s in ids], device=DEVICE))
        for b, s in enumerate(ids):
            rows[b] = at(torch.arange(len(s) - k - 1, len(s), device=DEVICE))[b]
    out = torch.stack([rows[b] for b in range(len(ids))], dim=1)                   # [1 + steps, sequences, vocabulary]
    steps = list(out[1:].unbind(0))
    return {"steps": steps} if case["kind"] == "decode" else {"prompts": out[0], "steps": steps}
