"""What this framework is timed on: rounds of serving through the ragged engine.

A case is one round: prompts of some sessions enter ``put`` in forwards of at most ``budget`` tokens (sessions that are past their prompt
add one token each to every forward), then every session decodes ``steps`` tokens, then all are flushed. The tokens are given, as in
scoring or in replaying recorded requests, so that a result does not hang on how a near-tie is rounded. ``turn`` cases add the hidden-state
cache: the prompt's hidden states are captured, the session is flushed, restored from them and continued with the next turn's ``turn`` tokens.

Layers have the sizes of the named architectures of ``models/arch.py``; dense models keep their first layers only. Weights are random
and belong to a model, as in a server that is up: one engine per model and configuration serves all inputs. Experts are alike but for a
tenth, as after upcycling, so that a router's near-tie between two of them does no harm.

Configurations are those of ``models/arch.py`` and ``benchmarks/stacks.py``. The results are the logits of every forward (one row per
sequence in it) and, for ``turn`` cases, the captured hidden states.
"""
import itertools
import math
import random
import types

import torch
import torch.nn.functional as F

from hcache_deepspeed_b200.inference.v2 import RaggedInferenceEngineConfig
from hcache_deepspeed_b200.inference.v2.engine_factory import build_engine_from_module

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


# ---- the cases -------------------------------------------------------------------------------------------------------
def _case(name, model, sessions, prompt, steps, budget=4096, dtype="bf16", quant="none", turn=0):
    c = {"model": model, "dtype": dtype, "quant": quant, "sessions": sessions, "prompt": prompt, "steps": steps, "budget": budget, "turn": turn}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user, a short question to the smallest model: launches and latency
        _case("opt-chat", "opt-125m", 1, 19, 8, dtype="fp16"),
        # one user, a question of half a page to a 7B model
        _case("llama7-chat", "llama-2-7b", 1, 501, 24),
        # eight users at once, prompts of up to a thousand tokens: the ordinary load of a small server
        _case("llama7-eight", "llama-2-7b", 8, 1024, 32),
        # a session is saved as hidden states and comes back for its next turn: what the hidden-state cache is for
        _case("llama7-turn", "llama-2-7b", 1, 4093, 8, turn=64),
        # the same model served with 8-bit weights and activations
        _case("llama7-w8a8", "llama-2-7b", 16, 250, 32, quant="wf8af8"),
        # a long document for a model with grouped queries: the largest prefill, in two portions
        _case("llama70-long", "llama-2-70b", 1, 16384, 4, budget=8192),
        # a full batch of short requests to it, prompts entering while others decode
        _case("llama70-batch", "llama-2-70b", 64, 300, 32, budget=2048),
        # a mixture of experts with a shared expert
        _case("qwen2-moe", "qwen2-moe-4096", 16, 700, 32, budget=2048),
        # the four families whose layers mix attention with recurrent state
        _case("nipolorn", "nipolorn-2048", 4, 1500, 24),
        _case("dedelorn", "dedelorn-4096", 1, 4096, 24),
        _case("lotelix", "lotelix-2048", 8, 777, 32),
        _case("relulix", "relulix-4096", 2, 2048, 24),
    ]


def draw(rng):
    """Any of the models, from one short request to a long document or a full batch, up to the cost of the largest listed round."""
    most = max(_cost(c) for c in listed())
    while True:
        model = rng.choice(["opt-125m", "llama-2-7b", "llama-2-7b", "llama-2-70b", "qwen2-moe-4096", "nipolorn-2048", "dedelorn-4096", "lotelix-2048",
                            "relulix-4096"])
        over = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
        sessions, prompt = over(1, 64), over(16, 1900 if model == "opt-125m" else 12000)
        steps, budget = rng.randint(2, 32), rng.choice([2048, 4096, 8192])
        dtype = "fp16" if model == "opt-125m" or (model == "llama-2-7b" and rng.random() < 0.25) else "bf16"
        quant = "wf8af8" if model == "llama-2-7b" and dtype == "bf16" and rng.random() < 0.3 else "none"
        turn = over(8, 256) if model == "llama-2-7b" and quant == "none" and sessions <= 4 and rng.random() < 0.5 else 0
        c = _case(None, model, sessions, prompt, steps, budget, dtype, quant, turn)
        if sessions * prompt <= 24576 and _cost(c) <= most:
            return c


def tolerance(case):
    """Relative error between two correct implementations at the same precision, four times what is seen between kernels that sum and
    round in another order: logits after a few layers of 16-bit activations; 8-bit activations round again in every layer."""
    if case["quant"] != "none":
        return {"rel": 3e-2, "max": 0.5}
    if case["dtype"] == "fp16":
        return {"rel": 5e-3, "max": 0.1}
    return {"rel": 2e-2, "max": 0.4}


# ---- configurations --------------------------------------------------------------------------------------------------
def _stack(kind, width, layers, **kw):
    return dict(model_type=kind, width=width, vocab=32000, layers=layers, norm={"eps": 1e-5}, **kw)


def _config(model):
    """The configuration as a checkpoint folder has it."""
    if model == "opt-125m":
        return dict(model_type="opt", num_hidden_layers=12, hidden_size=768, num_attention_heads=12, ffn_dim=3072, vocab_size=50272,
                    max_position_embeddings=2048, activation_function="relu")
    llama = dict(model_type="llama", vocab_size=32000, rms_norm_eps=1e-5, hidden_act="silu", rope_theta=1e4, max_position_embeddings=1 << 20)
    if model == "llama-2-7b":
        return dict(llama, num_hidden_layers=4, hidden_size=4096, num_attention_heads=32, num_key_value_heads=32, intermediate_size=11008)
    if model == "llama-2-70b":
        return dict(llama, num_hidden_layers=2, hidden_size=8192, num_attention_heads=64, num_key_value_heads=8, intermediate_size=28672)
    if model == "qwen2-moe-4096":
        return dict(llama, model_type="qwen2_moe", num_hidden_layers=4, hidden_size=4096, num_attention_heads=32, num_key_value_heads=8,
                    intermediate_size=3584, num_experts=16, num_experts_per_tok=2, moe_intermediate_size=3584, shared_expert_intermediate_size=3584)
    if model == "nipolorn-2048":
        mixer = {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128**-0.5, "mask": {"size": 1024, "keep_first": 16}},
                 "right": {"heads": 64, "vdim": 64, "state": 128, "groups": 4, "conv": 4, "norm_groups": 4}, "left_scale": 1.0, "right_scale": 0.5}
        return _stack("nipolorn", 2048, [{"type": "parallel", "mixer": mixer, "mlp": {"kind": "dense", "ff": 8192, "limit": 7.0}}] * 4)
    if model == "dedelorn-4096":
        mlp = {"kind": "dense", "ff": 14336}
        delta = {"type": "delta", "mixer": {"heads": 32, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}, "mlp": mlp}
        own = {"heads": 32, "dim": 96, "rot_dim": 32, "vdim": 128, "kv_rank": 512, "scale": 128**-0.5, "rot": {"base": 1e4, "dims": 32}, "mask": {"size": 4096}}
        return _stack("dedelorn", 4096, [delta, {"type": "latent_attention", "mixer": own, "mlp": mlp}, delta,
                                         {"type": "latent_attention", "mixer": dict(own, kv_from=1), "mlp": mlp}])
    if model == "lotelix-2048":
        mlp = {"kind": "moe", "expert": {"ff": 2688}, "router": {"experts": 16, "top": 2}}
        rot = {"base": 1e6, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
        attn = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "mask": {"size": 1024}, "rot": rot, "scale": 128**-0.5,
                                               "v_mix": True}, "mlp": mlp}
        both = {"left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "rot": {"base": 1e6, "dims": 128}, "scale": 128**-0.5},
                "right": {"heads": 16, "dim": 128, "vdim": 128, "tau": 16.0}}
        return _stack("lotelix", 2048, [{"type": "mingru", "mixer": {"width": 2048}, "mlp": mlp}, attn, {"type": "parallel", "mixer": both, "mlp": mlp}, attn],
                      embedding={"scale": 1.0}) | {"norm": {"eps": 1e-5, "groups": 2}}
    if model == "relulix-4096":
        mlp = {"kind": "moe", "expert": {"ff": 3584, "limit": 7.0}, "router": {"experts": 16, "top": 2}}
        ret = {"type": "retention", "mlp": mlp, "mixer": {"heads": 32, "dim": 128, "vdim": 128, "rot": {"base": 1e6, "dims": 128},
                                                         "decay": [1.0 - 2.0**(-5.0 - 7.0 * i / 32) for i in range(32)]}}
        own = {"heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128, "mask": {"size": 2048}, "scale": 128**-0.5, "softcap": 30.0,
               "rot": {"base": 1e6, "dims": 64, "scaling": {"factor": 4.0, "slow": 1.0, "fast": 32.0, "original": 8192}}}
        return _stack("relulix", 4096, [ret, {"type": "attention", "mixer": own, "mlp": mlp}, ret, {"type": "attention", "mixer": dict(own, kv_from=1), "mlp": mlp}],
                      embedding={"scale": 1.0})
    raise KeyError(model)


# ---- weights under their checkpoint names ----------------------------------------------------------------------------
def _weights(model, dtype):
    cfg = _config(model)
    g = torch.Generator(device=DEV).manual_seed(20 + sum(map(ord, model)))

    def rnd(*shape, scale=None):
        return (torch.randn(shape, generator=g, device=DEV) * (shape[-1]**-0.5 if scale is None else scale)).to(dtype)

    def near(n, base=1.0, scale=0.2):
        return (base + torch.randn(n, generator=g, device=DEV) * scale).to(dtype)

    def alike(names, n, shapes):
        """Experts: one set of matrices, each expert a tenth its own."""
        base = {k: rnd(*s) for k, s in shapes.items()}
        for e in range(n):
            for k, t in base.items():
                w[names.format(e=e, k=k)] = t + rnd(*t.shape, scale=0.1 * t.shape[-1]**-0.5)

    w = {}
    if cfg["model_type"] == "opt":
        W, V = cfg["hidden_size"], cfg["vocab_size"]
        d = "model.decoder."
        w[d + "embed_tokens.weight"], w[d + "embed_positions.weight"] = rnd(V, W), rnd(cfg["max_position_embeddings"] + 2, W)
        w[d + "final_layer_norm.weight"], w[d + "final_layer_norm.bias"] = near(W), near(W, 0.0)
        for i in range(cfg["num_hidden_layers"]):
            p = f"{d}layers.{i}."
            for n, (o, k, s) in {"self_attn.q_proj": (W, W, 2.0), "self_attn.k_proj": (W, W, 1.0), "self_attn.v_proj": (W, W, 1.0), "self_attn.out_proj": (W, W, 1.0),
                                 "fc1": (cfg["ffn_dim"], W, 1.0), "fc2": (W, cfg["ffn_dim"], 1.0)}.items():
                w[p + n + ".weight"], w[p + n + ".bias"] = rnd(o, k, scale=s * k**-0.5), near(o, 0.0, 0.1)
            for n in ("self_attn_layer_norm", "final_layer_norm"):
                w[p + n + ".weight"], w[p + n + ".bias"] = near(W), near(W, 0.0, 0.1)
    elif "width" not in cfg:
        W, V, H, G = cfg["hidden_size"], cfg["vocab_size"], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        w["model.embed_tokens.weight"], w["model.norm.weight"], w["lm_head.weight"] = rnd(V, W, scale=1.0), near(W), rnd(V, W)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = near(W), near(W)
            for n, o in (("q", H * 128), ("k", G * 128), ("v", G * 128)):
                w[f"{p}self_attn.{n}_proj.weight"] = rnd(o, W)
                if "num_experts" in cfg:
                    w[f"{p}self_attn.{n}_proj.bias"] = near(o, 0.0)
            w[p + "self_attn.o_proj.weight"] = rnd(W, H * 128)
            glu = lambda ff: {"gate_proj.weight": (ff, W), "up_proj.weight": (ff, W), "down_proj.weight": (W, ff)}  # noqa: E731
            if "num_experts" in cfg:
                w[p + "mlp.gate.weight"], w[p + "mlp.shared_expert_gate.weight"] = rnd(cfg["num_experts"], W, scale=2 * W**-0.5), rnd(1, W)
                alike(p + "mlp.experts.{e}.{k}", cfg["num_experts"], glu(cfg["moe_intermediate_size"]))
                w |= {p + "mlp.shared_expert." + k: rnd(*s) for k, s in glu(cfg["shared_expert_intermediate_size"]).items()}
            else:
                w |= {p + "mlp." + k: rnd(*s) for k, s in glu(cfg["intermediate_size"]).items()}
    else:
        kind, W, V = cfg["model_type"], cfg["width"], cfg["vocab"]
        gain = {"nipolorn": lambda: near(W, 0.0), "relulix": lambda: near(()) }.get(kind, lambda: near(W))
        w["embed"], w["final.norm"], w["head"] = rnd(V, W, scale=1.0), gain(), rnd(V, W)
        if kind == "dedelorn":
            w["embed.norm"] = near(W)
        for i, lc in enumerate(cfg["layers"]):
            p, q, m, f = f"l{i}.", f"l{i}.mix.", lc["mixer"], lc["mlp"]
            w[p + "norm1"] = gain()
            if kind in ("nipolorn", "lotelix"):
                w[p + "norm2"] = gain()
            if kind == "nipolorn":
                w[p + "norm1b"], w[p + "norm2b"] = gain(), gain()
                a, r = m["left"], m["right"]
                inner, gn = r["heads"] * r["vdim"], r["groups"] * r["state"]
                for n, o in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])):
                    w[q + "left." + n] = rnd(o * 128, W)
                w[q + "left.o"] = rnd(W, a["heads"] * 128)
                w[q + "right.in"], w[q + "right.conv"], w[q + "right.conv.b"] = rnd(2 * inner + 2 * gn + r["heads"], W), rnd(inner + 2 * gn, 4, scale=0.6), near(inner + 2 * gn, 0.0)
                w[q + "right.dt_bias"], w[q + "right.A_log"], w[q + "right.D"] = near(r["heads"], -2.0, 1.0), near(r["heads"], 0.0, 0.7), near(r["heads"], 0.0, 1.0)
                w[q + "right.norm"], w[q + "right.o"] = near(inner), rnd(W, inner)
            elif lc["type"] == "delta":
                kd, vd = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
                for n, o in (("q", kd), ("k", kd), ("v", vd)):
                    w[q + n], w[q + n + ".conv"] = rnd(o, W), rnd(o, m["conv"], scale=0.6)
                w[q + "g"], w[q + "b"], w[q + "a"] = rnd(vd, W), rnd(m["heads"], W), rnd(m["heads"], W)
                w[q + "A_log"], w[q + "dt_bias"] = near(m["heads"], -1.0, 1.0), near(m["heads"], -2.0, 1.0)
                w[q + "norm"], w[q + "o"] = near(m["vdim"]), rnd(W, vd)
            elif lc["type"] == "latent_attention":
                w[q + "q"] = rnd(m["heads"] * (m["dim"] + m["rot_dim"]), W, scale=2 * W**-0.5)
                if m.get("kv_from") is None:
                    w[q + "dkv"], w[q + "dkv.norm"] = rnd(m["kv_rank"] + m["rot_dim"], W), near(m["kv_rank"])
                w[q + "uk"], w[q + "uv"], w[q + "o"] = rnd(m["heads"] * m["dim"], m["kv_rank"]), rnd(m["heads"] * m["vdim"], m["kv_rank"]), rnd(W, m["heads"] * m["vdim"])
            elif lc["type"] == "mingru":
                C = m["width"]
                w[q + "z"], w[q + "z.b"], w[q + "x"], w[q + "x.b"] = rnd(C, W), near(C, -1.0, 0.5), rnd(C, W), near(C, 0.0, 0.5)
                w[q + "g"], w[q + "o"] = rnd(C, W), rnd(W, C, scale=2 * C**-0.5)
            elif lc["type"] == "parallel":
                a, r = m["left"], m["right"]
                for n, o in (("q", a["heads"]), ("k", a["kv_heads"]), ("v", a["kv_heads"])):
                    w[q + "left." + n], w[q + "left." + n + ".b"] = rnd(o * 128, W), near(o * 128, 0.0, 0.3)
                w[q + "left.q.norm"], w[q + "left.k.norm"], w[q + "left.pb"] = near(a["heads"] * 128), near(a["kv_heads"] * 128), near(a["heads"], -2.0, 1.0)
                w[q + "left.o"], w[q + "left.o.b"], w[q + "left.out"] = rnd(W, a["heads"] * 128), near(W, 0.0, 0.1), near(W)
                kd, vd = r["heads"] * r["dim"], r["heads"] * r["vdim"]
                for n, o in (("q", kd), ("k", kd), ("v", vd), ("g", vd), ("a1", 16)):
                    w[q + "right." + n] = rnd(o, W)
                w[q + "right.a2"], w[q + "right.a2.b"] = rnd(kd, 16, scale=1.0), near(kd, 1.0, 1.0)
                w[q + "right.norm"], w[q + "right.o"], w[q + "right.out"] = near(r["vdim"]), rnd(W, vd), near(W)
            elif lc["type"] == "retention":
                n_o = m["heads"] * m["vdim"]
                for n, o in (("q", m["heads"] * m["dim"]), ("k", m["heads"] * m["dim"]), ("v", n_o), ("g", n_o)):
                    w[q + n] = rnd(o, W)
                w[q + "k"] = (0.8 * w[q + "q"].float() + 0.6 * w[q + "k"].float()).to(dtype)     # a token's own key answers its query
                w[q + "o"] = rnd(W, n_o, scale=2 * n_o**-0.5)
            else:
                for n, o in (("q", m["heads"]), ) + ((("k", m["kv_heads"]), ("v", m["kv_heads"])) if m.get("kv_from") is None else ()):
                    w[q + n] = rnd(o * 128, W)
                    if kind == "relulix":
                        w[q + n + ".b"] = near(o * 128, 0.0, 0.3)
                w[q + "o"] = rnd(W, m["heads"] * 128, scale=2 * (m["heads"] * 128)**-0.5)
                if kind == "lotelix":
                    w[q + "g"], w[q + "sink"], w[q + "vmix"] = rnd(m["heads"] * 128, W), near(m["heads"], 1.0, 1.0), near(1, 0.5)[0]
            q = p + "mlp."
            if f["kind"] == "dense":
                w[q + "gate"], w[q + "up"], w[q + "down"] = rnd(f["ff"], W), rnd(f["ff"], W), rnd(W, f["ff"])
            else:
                n, ff = f["router"]["experts"], f["expert"]["ff"]
                w[q + "router"] = rnd(n, W, scale=2 * W**-0.5)
                if kind == "relulix":
                    w[q + "router.b"] = near(n, 0.0, 0.5)
                alike(q + "e{e}.{k}", n, {k: s for k, s in (("gate", (ff, W)), ("up", (ff, W)), ("down", (W, ff))) if k != "gate" or kind == "relulix"})
    return w


# ---- a round of serving ----------------------------------------------------------------------------------------------
class _Checkpoint:
    """A model object as ``build_engine_from_module`` takes it: a configuration and named weights."""

    def __init__(self, cfg, weights):
        self.config, self.weights = types.SimpleNamespace(**cfg), weights

    def state_dict(self):
        return self.weights


_engine = {}           # the engine that is up: one at a time
_uids = itertools.count(1)


def _engine_of(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _engine:
        _engine.clear()
        n, most = case["sessions"], case["prompt"] + case["turn"] + case["steps"] + 64
        cfg = RaggedInferenceEngineConfig(
            state_manager={"max_tracked_sequences": n + 2, "max_ragged_batch_size": max(case["budget"], n, case["prompt"] if case["turn"] else 0) + 8,
                           "max_ragged_sequence_count": n + 1, "max_context": most, "max_state_slots": n + 2,
                           "memory_config": {"mode": "tokens", "size": (n + 1) * (most + 128)}},
            hcache={"enabled": bool(case["turn"]), "capture": "sync" if case["turn"] else "off"},
            quantization={"quantization_mode": None if case["quant"] == "none" else case["quant"]})
        dt = DTYPES[case["dtype"]]
        _engine[key] = build_engine_from_module(_Checkpoint(_config(case["model"]), _weights(case["model"], dt)), cfg, dtype=dt, device=torch.device(DEV))
    return _engine[key]


def _lengths(case, seed):
    """Prompt lengths: one session has the full one, further sessions between half and all of it."""
    r = random.Random(seed * 7 + 1 if case["sessions"] > 1 else 0)
    return [case["prompt"]] + [r.randint(max(1, case["prompt"] // 2), case["prompt"]) for _ in range(case["sessions"] - 1)]


def _tokens(case, seed):
    cfg = _config(case["model"])
    g = torch.Generator().manual_seed(seed)
    vocab = cfg.get("vocab", cfg.get("vocab_size"))
    return [torch.randint(0, vocab, (n + case["turn"] + case["steps"], ), generator=g) for n in _lengths(case, seed)]


def _forwards(case, lengths):
    """The forwards of a round: lists of (session, first token, past the last one)."""
    out, n = [], len(lengths)
    if case["turn"]:
        for i, p in enumerate(lengths):
            out.append([(i, 0, p)])                             # captured; the session is flushed, then restored
        out.append([(i, p, p + case["turn"]) for i, p in enumerate(lengths)])
        at, goal = [p + case["turn"] for p in lengths], [p + case["turn"] for p in lengths]
    else:
        at, goal = [0] * n, list(lengths)
    done = [0] * n
    while any(d < case["steps"] for d in done) or any(a < g for a, g in zip(at, goal)):
        fwd, room = [], case["budget"]
        for i in range(n):                                      # sessions that decode come first
            if at[i] >= goal[i] and done[i] < case["steps"] and room:
                fwd.append((i, at[i], at[i] + 1))
                room -= 1
        for i in range(n):
            if at[i] < goal[i] and room:
                take = min(room, goal[i] - at[i])
                fwd.append((i, at[i], at[i] + take))
                room -= take
        for i, a, b in fwd:
            done[i] += at[i] >= goal[i]
            at[i] = b
        out.append(fwd)
    return out


def prepare(case, seed):
    eng = _engine_of(case)
    toks, lengths = _tokens(case, seed), _lengths(case, seed)
    uids = [next(_uids) for _ in toks]
    fwds = _forwards(case, lengths)
    cfg = _config(case["model"])
    logits = torch.empty(sum(map(len, fwds)), cfg.get("vocab", cfg.get("vocab_size")), dtype=DTYPES[case["dtype"]], device=DEV)
    plan = [([uids[i] for i, _, _ in f], [toks[i][a:b].pin_memory() for i, a, b in f]) for f in fwds]
    return {"engine": eng, "uids": uids, "plan": plan, "logits": logits, "turn": bool(case["turn"])}


def run(state):
    eng, out, row = state["engine"], state["logits"], 0
    saved = []
    for k, (uids, tokens) in enumerate(state["plan"]):
        first = state["turn"] and k < len(state["uids"])
        if state["turn"] and k == len(state["uids"]):           # the sessions come back
            for uid, (_, prompt), hidden in zip(uids, state["plan"], saved):
                eng.restore_kv([uid], prompt, [hidden])
        logits, hidden = eng.put(uids, tokens, capture_latents=first)
        out[row:row + len(uids)].copy_(logits)
        row += len(uids)
        if first:
            saved.append(hidden[0])
            eng.flush(uids[0])
    for uid in state["uids"]:
        eng.flush(uid)
    return {"logits": out, "hidden": saved} if state["turn"] else {"logits": out}


# ---- what a round cannot do without ----------------------------------------------------------------------------------
def _sizes(model):
    """(parameters that every forward reads, parameters that a token is multiplied with, (parameters of one expert, experts, top, layers),
    attention layers as (query heads, cached values per token, dim of scores and values, window), fp32 state values per session, width)."""
    cfg = _config(model)
    if "width" not in cfg:
        W, L = cfg["hidden_size"], cfg["num_hidden_layers"]
        V, H = cfg["vocab_size"], cfg["num_attention_heads"]
        G, d = cfg.get("num_key_value_heads", H), W // H
        mlp = 2 * W * cfg["ffn_dim"] if "ffn_dim" in cfg else 3 * W * cfg.get("shared_expert_intermediate_size", cfg["intermediate_size"])
        base = L * (W * (H + 2 * G) * d + H * d * W + mlp) + V * W
        ex = (3 * W * cfg["moe_intermediate_size"], cfg["num_experts"], cfg["num_experts_per_tok"], L) if "num_experts" in cfg else (0, 0, 0, 0)
        return base, base - V * W, ex, [(H, 2 * G * d, 2 * d, 0)] * L, 0, W
    W, V = cfg["width"], cfg["vocab"]
    base, ex, attn, state = 0, (0, 0, 0, 0), [], 0
    for lc in cfg["layers"]:
        m, f = lc["mixer"], lc["mlp"]
        if f["kind"] == "dense":
            base += 3 * W * f["ff"]
        else:
            ex = ((3 if cfg["model_type"] == "relulix" else 2) * W * f["expert"]["ff"], f["router"]["experts"], f["router"]["top"], len(cfg["layers"]))
        for a in ([m] if "kv_heads" in m and lc["type"] == "attention" else [m["left"]] if "left" in m else []):
            H, G, own = a["heads"], a["kv_heads"], a.get("kv_from") is None
            base += W * 128 * (2 * H + 2 * G * own + H * (cfg["model_type"] == "lotelix" and lc["type"] == "attention"))
            attn.append((H, 2 * G * 128, 256, (a.get("mask") or {}).get("size", 0)))
        if lc["type"] == "latent_attention":
            H, R, r = m["heads"], m["kv_rank"], m["rot_dim"]
            base += W * H * (m["dim"] + r) + (W * (R + r) if m.get("kv_from") is None else 0) + H * R * (m["dim"] + m["vdim"]) + W * H * m["vdim"]
            attn.append((H, R + r, m["dim"] + r + m["vdim"], m["mask"]["size"]))
        if lc["type"] == "delta":
            kd, vd = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
            base, state = base + W * (2 * kd + 3 * vd), state + vd * m["dim"]
        if lc["type"] == "retention":
            base, state = base + 5 * W * m["heads"] * 128, state + m["heads"] * 128 * 128
        if lc["type"] == "mingru":
            base, state = base + 4 * W * m["width"], state + m["width"]
        if "right" in m:
            r = m["right"]
            inner = r["heads"] * r["vdim"]
            if "state" in r:
                base, state = base + W * (3 * inner + 2 * r["groups"] * r["state"]), state + inner * r["state"]
            else:
                base, state = base + 5 * W * inner, state + inner * r["dim"]
    return base + V * W, base, ex, attn, state, W


def work(case):
    """Per forward: the weights once (of the experts those that are met), the cached keys and values that are seen and the recurrent states
    once; a pair of products per score; the embedded tokens and the logits."""
    read, used, (ep, en, top, layers), attn, state, W = _sizes(case["model"])
    cfg = _config(case["model"])
    V = cfg.get("vocab", cfg.get("vocab_size"))
    wb = 1 if case["quant"] != "none" else 2
    lengths = [case["prompt"]] + [case["prompt"] * 3 // 4] * (case["sessions"] - 1)
    total, flops = 0.0, 0.0
    for fwd in _forwards(case, lengths):
        n = sum(b - a for _, a, b in fwd)
        met = en * (1 - (1 - top / en)**n) if en else 0
        total += (read - V * W) * wb + V * W * 2 + met * ep * layers * 2 + n * W * 2 + len(fwd) * (V * 2 + 2 * state * 4)
        flops += 2.0 * n * (used + top * ep * layers) + 2.0 * len(fwd) * V * W
        for H, kv, dims, window in attn:
            for _, a, b in fwd:
                total += 2 * kv * (min(b, window + b - a) if window else b) + 2 * kv * (b - a)
                seen = (b * (b + 1) - a * (a + 1)) / 2 if not window else sum(min(t + 1, window) for t in (a, b - 1)) / 2 * (b - a)
                flops += 2.0 * H * dims * seen
        flops += 6.0 * n * state
    if case["turn"]:                                            # hidden states out, in, and through the K / V projection
        n = sum(lengths)
        total += 2 * len(attn) * n * W * 2 + sum(W * kv * 2 + n * kv * 2 for _, kv, _, _ in attn)
        flops += sum(2.0 * n * W * kv for _, kv, _, _ in attn)
    return {"bytes": total, "flops": flops}


def _cost(case):
    w = work(case)
    return w["bytes"] / 6.5e12 + w["flops"] / 1.5e15


# ---- the same in 64 bits, in plain torch -----------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window=0, keep=0, weigh=None):
    """q [n, heads, .], k and v [n, kv_heads, .] -> [n, heads * vdim]; ``weigh(head, scores, visible)`` in place of the softmax."""
    n, H = q.shape[:2]
    group, out = H // k.shape[1], torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
    for lo in range(0, n, 4096):
        hi = min(n, lo + 4096)
        i, j = torch.arange(lo, hi, device=q.device)[:, None], torch.arange(hi, device=q.device)[None, :]
        see = j <= i
        if window:
            see &= (i - j < window) | (j < keep)
        for a in range(H):
            s = (q[lo:hi, a] @ k[:hi, a // group].T) * scale
            p = torch.softmax(s.masked_fill_(~see, -math.inf), -1) if weigh is None else weigh(a, s, see)
            out[lo:hi, a] = p @ v[:hi, a // group]
    return out.reshape(n, -1)


def _turned(x, freq, adjacent=False, factor=1.0):
    """x [n, heads, dims]: pairs turned by position * freq; pair i is (i, i + half), or (2 i, 2 i + 1); values past the pairs stay."""
    half = freq.numel()
    ang = (torch.arange(x.shape[0], dtype=x.dtype, device=x.device)[:, None] * freq)[:, None]
    c, s = torch.cos(ang) * factor, torch.sin(ang) * factor
    if adjacent:
        u, v = x[..., 0:2 * half:2], x[..., 1:2 * half:2]
        return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., 2 * half:]], -1)
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def _frequencies(rot):
    """(angles per position, factor): plain, slowed by wavelength (low, high), or slowed by a ramp over the pairs (slow, fast)."""
    dims, base, sc = rot["dims"], float(rot["base"]), rot.get("scaling")
    f, factor = [base**(-2 * i / dims) for i in range(dims // 2)], 1.0
    if sc and "low" in sc:
        def slowed(x):
            share = (sc["original"] * x / (2 * math.pi) - sc["low"]) / (sc["high"] - sc["low"])
            share = min(max(share, 0.0), 1.0)
            return (1 - share) * x / sc["factor"] + share * x
        f = [slowed(x) for x in f]
    elif sc:
        index = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(index(sc["fast"])), 0), min(math.ceil(index(sc["slow"])), dims - 1)
        ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
        f, factor = [x / sc["factor"] * r + x * (1 - r) for x, r in zip(f, ramp)], 0.1 * math.log(sc["factor"]) + 1
    return torch.tensor(f, dtype=torch.float64, device=DEV), factor


def _conv(u, taps):
    n, K = u.shape[0], taps.shape[1]
    padded = torch.cat([u.new_zeros(K - 1, u.shape[1]), u])
    return sum(padded[j:j + n] * taps[:, j] for j in range(K))


def _glu(h, w, p, act=F.silu, names=("gate", "up", "down")):
    return w.times(act(w.times(h, p + names[0])) * w.times(h, p + names[1]), p + names[2])


def _mixture(h, chosen, weight, expert):
    """Every token's chosen experts; ``expert(e, rows, weights)`` is what rows get from expert e."""
    out = torch.zeros_like(h)
    for e in range(int(chosen.max()) + 1):
        t, j = torch.where(chosen == e)
        if t.numel():
            out.index_add_(0, t, expert(e, h[t], weight[t, j, None]))
    return out


def _eight_bit(x):
    """Rows as 8-bit floats times a scale each, the largest value of a row at 448: what 8-bit serving multiplies."""
    scale = x.abs().amax(-1, keepdim=True).clamp(min=1e-300) / 448.0
    return (x / scale).float().to(torch.float8_e4m3fn).double() * scale


class _Wide:
    """Weights in 64 bits, one at a time; ``quant``: products of a layer take 8-bit rows on both sides."""

    def __init__(self, w, quant):
        self.w, self.quant = w, quant

    def __getitem__(self, name):
        return self.w[name].double()

    def times(self, h, name):
        return _eight_bit(h) @ _eight_bit(self[name]).T if self.quant else h @ self[name].T


def _stream(cfg, w, tokens, hidden=None):
    """The normed last residual stream [n, width] of one whole session and the matrix of the logits; ``hidden``: gets every layer's normed input."""
    kind = cfg["model_type"]
    if kind == "opt":
        d, n = "model.decoder.", tokens.numel()
        W, H = cfg["hidden_size"], cfg["num_attention_heads"]
        ln = lambda x, p: F.layer_norm(x, (W, ), w[p + ".weight"], w[p + ".bias"], 1e-5)  # noqa: E731
        lin = lambda x, p: x @ w[p + ".weight"].T + w[p + ".bias"]  # noqa: E731
        x = w[d + "embed_tokens.weight"][tokens] + w[d + "embed_positions.weight"][2:2 + n]
        for i in range(cfg["num_hidden_layers"]):
            p = f"{d}layers.{i}."
            h = ln(x, p + "self_attn_layer_norm")
            q, k, v = (lin(h, f"{p}self_attn.{c}_proj").reshape(n, H, -1) for c in "qkv")
            x = x + lin(_attend(q, k, v, (W // H)**-0.5), p + "self_attn.out_proj")
            x = x + lin(torch.relu(lin(ln(x, p + "final_layer_norm"), p + "fc1")), p + "fc2")
        return ln(x, d + "final_layer_norm"), w[d + "embed_tokens.weight"]
    if "width" not in cfg:
        eps, n, moe = cfg["rms_norm_eps"], tokens.numel(), "num_experts" in cfg
        freq, _ = _frequencies({"dims": 128, "base": cfg["rope_theta"]})
        hf = ("gate_proj.weight", "up_proj.weight", "down_proj.weight")
        x = w["model.embed_tokens.weight"][tokens]
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            h = _rms(x, eps) * w[p + "input_layernorm.weight"]
            if hidden is not None:
                hidden.append(h)
            q, k, v = (w.times(h, f"{p}self_attn.{c}_proj.weight") for c in "qkv")
            if moe:
                q, k, v = (t + w[f"{p}self_attn.{c}_proj.bias"] for c, t in zip("qkv", (q, k, v)))
            q, k, v = (t.reshape(n, -1, 128) for t in (q, k, v))
            x = x + w.times(_attend(_turned(q, freq), _turned(k, freq), v, 128**-0.5), p + "self_attn.o_proj.weight")
            h = _rms(x, eps) * w[p + "post_attention_layernorm.weight"]
            if moe:
                weight, chosen = torch.softmax(h @ w[p + "mlp.gate.weight"].T, -1).topk(cfg["num_experts_per_tok"], -1)
                x = x + _mixture(h, chosen, weight, lambda e, r, f: f * _glu(r, w, f"{p}mlp.experts.{e}.", names=hf))
                x = x + torch.sigmoid(h @ w[p + "mlp.shared_expert_gate.weight"].T) * _glu(h, w, p + "mlp.shared_expert.", names=hf)
            else:
                x = x + _glu(h, w, p + "mlp.", names=hf)
        return _rms(x, eps) * w["model.norm.weight"], w["lm_head.weight"]
    eps, n, top = cfg["norm"]["eps"], tokens.numel(), "final.norm"
    if kind == "nipolorn":
        norm = lambda x, name: _rms(x, eps) * (1 + w[name])  # noqa: E731
    elif kind == "lotelix":
        norm = lambda x, name: _rms(x.reshape(n, cfg["norm"]["groups"], -1), eps).reshape(n, -1) * w[name]  # noqa: E731
    else:
        norm = lambda x, name: _rms(x, eps) * w[name]  # noqa: E731
    x = w["embed"][tokens]
    x = norm(x, "embed.norm") if kind == "dedelorn" else x * cfg.get("embedding", {}).get("scale", 1.0)
    cached, v_first = {}, None
    for i, lc in enumerate(cfg["layers"]):
        p, q_, m, f = f"l{i}.", f"l{i}.mix.", lc["mixer"], lc["mlp"]
        h = norm(x, p + "norm1")
        heads = lambda name, bias=False: (h @ w[name].T + (w[name + ".b"] if bias else 0)).reshape(n, -1, 128)  # noqa: E731
        if kind == "nipolorn":
            a, l, r = m["left"], q_ + "left.", q_ + "right."
            y = m["left_scale"] * _attend(heads(l + "q"), heads(l + "k"), heads(l + "v"), a["scale"], a["mask"]["size"], a["mask"]["keep_first"]) @ w[l + "o"].T
            a = m["right"]
            H, P, N, G = a["heads"], a["vdim"], a["state"], a["groups"]
            inner = H * P
            z, xbc, dt = (h @ w[r + "in"].T).split([inner, inner + 2 * G * N, H], -1)
            xs, B, C = F.silu(_conv(xbc, w[r + "conv"]) + w[r + "conv.b"]).split([inner, G * N, G * N], -1)
            xs, B, C = xs.reshape(n, H, P), B.reshape(n, G, N).repeat_interleave(H // G, 1), C.reshape(n, G, N).repeat_interleave(H // G, 1)
            dt = F.softplus(dt + w[r + "dt_bias"], threshold=40)
            o = _recur(C, B, xs * dt[..., None], decay=torch.exp(-torch.exp(w[r + "A_log"]) * dt)) + w[r + "D"][:, None] * xs
            o = (o.reshape(n, -1) * F.silu(z)).reshape(n, a["norm_groups"], -1)
            y = y + m["right_scale"] * ((_rms(o, eps).reshape(n, -1) * w[r + "norm"]) @ w[r + "o"].T)
            y = norm(y, p + "norm1b")
        elif lc["type"] == "delta":
            H, G = m["heads"], m["kv_heads"]
            q, k, v = (F.silu(_conv(h @ w[q_ + c].T, w[q_ + c + ".conv"])) for c in "qkv")
            unit = lambda t: (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)  # noqa: E731
            q, k = unit(q.reshape(n, G, -1)) * m["dim"]**-0.5, unit(k.reshape(n, G, -1))
            decay = torch.exp(-torch.exp(w[q_ + "A_log"]) * F.softplus(h @ w[q_ + "a"].T + w[q_ + "dt_bias"], threshold=40))
            o = _recur(q, k, v.reshape(n, H, -1), decay=decay, beta=torch.sigmoid(h @ w[q_ + "b"].T))
            y = ((_rms(o, eps) * w[q_ + "norm"]).reshape(n, -1) * F.silu(h @ w[q_ + "g"].T)) @ w[q_ + "o"].T
        elif lc["type"] == "latent_attention":
            H, R, freq = m["heads"], m["kv_rank"], _frequencies(m["rot"])[0]
            if m.get("kv_from") is None:
                c = h @ w[q_ + "dkv"].T
                cached[i] = _rms(c[:, :R], eps) * w[q_ + "dkv.norm"], _turned(c[:, None, R:], freq, True)
            c, kr = cached[i if m.get("kv_from") is None else m["kv_from"]]
            q = (h @ w[q_ + "q"].T).reshape(n, H, -1)
            q = torch.cat([q[..., :m["dim"]], _turned(q[..., m["dim"]:], freq, True)], -1)
            k = torch.cat([(c @ w[q_ + "uk"].T).reshape(n, H, -1), kr.expand(n, H, m["rot_dim"])], -1)
            y = _attend(q, k, (c @ w[q_ + "uv"].T).reshape(n, H, -1), m["scale"], m["mask"]["size"]) @ w[q_ + "o"].T
        elif lc["type"] == "mingru":
            z, u = torch.sigmoid(h @ w[q_ + "z"].T + w[q_ + "z.b"]), h @ w[q_ + "x"].T + w[q_ + "x.b"]
            add, S, o = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), torch.zeros_like(z[0]), torch.empty_like(z)
            for t in range(n):
                S = torch.addcmul(add[t], 1 - z[t], S)
                o[t] = S
            y = (o * F.silu(h @ w[q_ + "g"].T)) @ w[q_ + "o"].T
        elif lc["type"] == "parallel":
            a, l, r = m["left"], q_ + "left.", q_ + "right."
            freq = _frequencies(a["rot"])[0]
            q, k = ((_rms(h @ w[l + c].T + w[l + c + ".b"], eps) * w[l + c + ".norm"]).reshape(n, -1, 128) for c in "qk")
            pb = w[l + "pb"]
            left = _attend(_turned(q, freq, True), _turned(k, freq, True), heads(l + "v", True), a["scale"],
                           weigh=lambda hd, s, see: torch.sigmoid(s + pb[hd]) * see) @ w[l + "o"].T + w[l + "o.b"]
            a = m["right"]
            q, k, v = ((h @ w[r + c].T).reshape(n, a["heads"], -1) for c in "qkv")
            alpha = torch.sigmoid((h @ w[r + "a1"].T) @ w[r + "a2"].T + w[r + "a2.b"])**(1 / a["tau"])
            o = _recur(q * a["dim"]**-0.5, k, v, fade=alpha.reshape(n, a["heads"], -1))
            right = ((_rms(o, eps) * w[r + "norm"]).reshape(n, -1) * F.silu(h @ w[r + "g"].T)) @ w[r + "o"].T
            y = (_rms(left, eps) * w[l + "out"] + _rms(right, eps) * w[r + "out"]) / 2
        elif lc["type"] == "retention":
            freq = _frequencies(m["rot"])[0]
            k, decay = _turned(heads(q_ + "k"), freq) * m["dim"]**-0.5, torch.tensor(m["decay"], dtype=x.dtype, device=DEV).expand(n, -1)
            o = _rms(_recur(_turned(heads(q_ + "q"), freq), k, heads(q_ + "v"), decay=decay), eps).reshape(n, -1)
            y = (o * F.silu(h @ w[q_ + "g"].T)) @ w[q_ + "o"].T
        else:
            freq, factor = _frequencies(m["rot"])
            biased = kind == "relulix"
            q = _turned(heads(q_ + "q", biased), freq, False, factor)
            if m.get("kv_from") is None:
                cached[i] = _turned(heads(q_ + "k", biased), freq, False, factor), heads(q_ + "v", biased)
            k, v = cached[i if m.get("kv_from") is None else m["kv_from"]]
            if kind == "lotelix":
                if v_first is None:
                    v_first = v
                else:
                    v = (1 - w[q_ + "vmix"]) * v + w[q_ + "vmix"] * v_first
                sink = w[q_ + "sink"]

                def weigh(hd, s, see):
                    e = torch.cat([s.masked_fill(~see, -math.inf), sink[hd].expand(s.shape[0], 1)], -1)
                    return torch.softmax(e, -1)[:, :-1]
            else:
                def weigh(hd, s, see):
                    s = (m["softcap"] * torch.tanh(s / m["softcap"])).masked_fill(~see, -math.inf)
                    return torch.softmax(torch.cat([s, s.new_zeros(s.shape[0], 1)], -1), -1)[:, :-1]
            o = _attend(q, k, v, m["scale"], m["mask"]["size"], weigh=weigh)
            y = (o * torch.sigmoid(h @ w[q_ + "g"].T) if kind == "lotelix" else o) @ w[q_ + "o"].T
        q_ = p + "mlp."
        if kind in ("nipolorn", "lotelix"):
            x, y = x + y, 0.0
            h = norm(x, p + "norm2")
        if kind == "nipolorn":
            g = torch.clamp(h @ w[q_ + "gate"].T, max=f["limit"])
            g = g * torch.sigmoid(1.702 * g) * (torch.clamp(h @ w[q_ + "up"].T, -f["limit"], f["limit"]) + 1)
            x = x + norm(g @ w[q_ + "down"].T, p + "norm2b")
        elif kind == "dedelorn":
            x = x + y + _glu(h, w, q_, act=lambda t: F.gelu(t, approximate="tanh"))
        elif kind == "lotelix":
            weight, chosen = torch.sigmoid(h @ w[q_ + "router"].T).topk(f["router"]["top"], -1)
            x = x + _mixture(h, chosen, weight, lambda e, r, s: torch.relu((s * r) @ w[f"{q_}e{e}.up"].T)**2 @ w[f"{q_}e{e}.down"].T)
        else:
            best, chosen = (h @ w[q_ + "router"].T + w[q_ + "router.b"]).topk(f["router"]["top"], -1)
            lim = f["expert"]["limit"]

            def expert(e, r, s):
                g = torch.clamp(r @ w[f"{q_}e{e}.gate"].T, max=lim)
                return s * ((g * torch.sigmoid(1.702 * g) * (torch.clamp(r @ w[f"{q_}e{e}.up"].T, -lim, lim) + 1)) @ w[f"{q_}e{e}.down"].T)
            x = x + y + _mixture(h, chosen, torch.softmax(best, -1), expert)
    return norm(x, top), w["head"]


def _recur(q, k, v, decay=None, fade=None, beta=None):
    """Read-outs [n, heads, vdim] of S <- decay S + k v^T token by token; ``decay`` [n, heads] or ``fade`` [n, heads, dim]; ``beta`` [n, heads]:
    S moves by that share from what k reads towards v. q, k [n, heads, dim], v [n, heads, vdim]."""
    n, H, P = v.shape
    S, out = q.new_zeros(H, q.shape[2], P), torch.empty_like(v)
    factor = decay[:, :, None, None] if fade is None else fade[:, :, :, None]
    for t in range(n):
        S = S * factor[t]
        u = v[t][:, None] if beta is None else beta[t][:, None, None] * (v[t][:, None] - k[t][:, None] @ S)
        S = torch.baddbmm(S, k[t][:, :, None], u)
        out[t] = (q[t][:, None] @ S)[:, 0]
    return out


def exact(case, seed):
    cfg, lengths = _config(case["model"]), _lengths(case, seed)
    w = _Wide(_weights(case["model"], DTYPES[case["dtype"]]), case["quant"] != "none")
    wants = [[] for _ in lengths]                               # (row of the result, token) of every session
    for row, (i, _, b) in enumerate(x for f in _forwards(case, lengths) for x in f):
        wants[i].append((row, b - 1))
    logits = torch.empty(sum(map(len, wants)), cfg.get("vocab", cfg.get("vocab_size")), dtype=torch.float64, device=DEV)
    saved = []
    for toks, length, want in zip(_tokens(case, seed), lengths, wants):
        hidden = [] if case["turn"] else None
        x, head = _stream(cfg, w, toks.to(DEV), hidden)
        logits[[r for r, _ in want]] = x[[t for _, t in want]] @ head.T
        if hidden is not None:
            saved.append(torch.stack([h[:length] for h in hidden]))
    return {"logits": logits, "hidden": saved} if case["turn"] else {"logits": logits}
