"""What the engine is measured on: steps and requests of the decoders it serves, through its public entry points.

Five kinds of case:

* ``decode``    the dense decoder (Llama / Qwen3 layers), one decode step of ``rows`` requests whose contexts are cached: what
                a server runs most of its time.
* ``portions``  the dense decoder, one step that brings prompt portions, alone or beside decoding requests: what a server
                runs when prompts arrive (``a@p`` is a portion of a tokens behind p cached ones, as chunked prefill makes).
* ``request``   whole requests of one of the other decoders: open, prompts in one step, ``new`` decoded tokens, close.
                Recurrences keep their state in the request, so a request is the unit that can be run again.
* ``generate``  ``Engine.generate`` in float32 (scheduler, sampler with log-probabilities, the 32-bit kernels).

Sizes are those of ``lily_b200/bench`` ("small": width 2048, "mid": the layer sizes of an 8 B model) with fewer layers, as there.
Of the decoders beside the dense one those are here whose layers hold what it has not: a state-space scan (Zirurax), a
linear attention with decay, latent attention and routed experts (Godotar), the delta rule, a selective scan and mixed heads
(Kinanex), a matrix memory, squashing norms and ungated experts in groups (Tugodra).
"""

from __future__ import annotations

import hashlib
import math

import torch
import torch.nn.functional as F

SIZES = {
    "small": dict(width=2048, ff=8192, heads=16, kv_heads=4, head=128, window=1024),
    "mid": dict(width=4096, ff=12288, heads=32, kv_heads=8, head=128, window=2048),
}
VOCAB = 32000
DESIGNS = ("zirurax", "kinanex", "godotar", "tugodra")
PAGE = 64


def listed():
    return [
        # one user of a small model, short context: the smallest call, all launches and latency
        {"name": "decode-1", "kind": "decode", "size": "small", "layers": 4, "rows": 1, "low": 900, "high": 900},
        # the benchmark's own decode step: eight users of an 8 B model's layers at 4,096 positions
        {"name": "decode-8", "kind": "decode", "size": "mid", "layers": 8, "rows": 8, "low": 4096, "high": 4096},
        # a busy server: 64 users with contexts of very different lengths
        {"name": "decode-64", "kind": "decode", "size": "mid", "layers": 8, "rows": 64, "low": 250, "high": 1750},
        # one prompt, the benchmark's own prefill
        {"name": "prefill-2048", "kind": "portions", "size": "mid", "layers": 8, "rows": 0, "low": 0, "high": 0, "portions": "2048"},
        # continuous batching: two ragged prompts and a later portion of a long one beside 19 decoding users
        {"name": "mixed", "kind": "portions", "size": "mid", "layers": 8, "rows": 19, "low": 400, "high": 2900, "portions": "1103,333,640@3072"},
        # a long prompt with a short answer, and many short prompts with longer ones, of the state-space decoder
        {"name": "zirurax-long", "kind": "request", "design": "zirurax", "size": "small", "layers": 4, "prompts": "2048", "new": 8},
        {"name": "zirurax-many", "kind": "request", "design": "zirurax", "size": "small", "layers": 4, "prompts": "70,391,128,33,250,181,64,97", "new": 24},
        # the same of the decoder with the delta rule and the selective scan
        {"name": "kinanex-long", "kind": "request", "design": "kinanex", "size": "small", "layers": 4, "prompts": "1999", "new": 8},
        {"name": "kinanex-many", "kind": "request", "design": "kinanex", "size": "small", "layers": 4, "prompts": "300,45,211,127,512", "new": 24},
        # two prompts of the decoder with linear attention, latent attention and routed experts
        {"name": "godotar", "kind": "request", "design": "godotar", "size": "small", "layers": 4, "prompts": "1500,420", "new": 12},
        # three prompts of the decoder with matrix memory, latent attention and experts in groups
        {"name": "tugodra", "kind": "request", "design": "tugodra", "size": "small", "layers": 4, "prompts": "1200,700,148", "new": 12},
        # checking a checkpoint in 32-bit: greedy tokens with their log-probabilities
        {"name": "generate-fp32", "kind": "generate", "size": "small", "layers": 4, "prompts": "150,61,240", "new": 12},
    ]


def _log(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def _lengths(rng, count, low, high, most):
    out, left = [], most
    for _ in range(count):
        n = min(_log(rng, low, high), left)
        if n < low:
            break
        out.append(n)
        left -= n
    return out


def draw(rng):
    kind = rng.choice(["decode", "portions", "request", "request", "request", "request", "generate"])
    if kind == "decode":
        rows = _log(rng, 1, 64)
        high = min(_log(rng, 200, 4096), 65000 // rows)
        return {"kind": kind, "size": rng.choice(["small", "mid"]), "layers": 4, "rows": rows, "low": max(16, int(high * rng.uniform(0.2, 1.0))), "high": high}
    if kind == "portions":
        size = rng.choice(["small", "mid"])
        portions = [str(n) for n in _lengths(rng, rng.randint(1, 4), 24, 2048, 2048)]
        if rng.random() < 0.4:
            portions[-1] += f"@{_log(rng, 100, 3500)}"
        rows = rng.choice([0, 0, rng.randint(1, 20)])
        high = _log(rng, 100, 3000)
        return {"kind": kind, "size": size, "layers": 4, "rows": rows, "low": 64 if rows else 0, "high": high if rows else 0,
                "portions": ",".join(portions)}
    if kind == "request":
        prompts = _lengths(rng, rng.choice([1, 1, 2, 4, 8, 12]), 24, 2048, 2048)
        return {"kind": kind, "design": rng.choice(DESIGNS), "size": "small", "layers": 4, "prompts": ",".join(map(str, prompts)), "new": _log(rng, 4, 24)}
    return {"kind": kind, "size": "small", "layers": rng.randint(2, 4), "prompts": ",".join(map(str, _lengths(rng, rng.randint(1, 4), 16, 250, 450))),
            "new": rng.randint(4, 12)}


# --------------------------------------------------------------------------- configurations, as in lily_b200/bench

def config(case):
    z, layers = SIZES[case["size"]], case["layers"]
    width, heads, head, ff = z["width"], z["heads"], z["head"], z["ff"]
    if case["kind"] != "request":
        return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": layers, "hidden_size": width,
                "num_attention_heads": heads, "num_key_value_heads": z["kv_heads"], "head_dim": head, "intermediate_size": ff,
                "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": True,
                "max_position_embeddings": 8192, "hidden_act": "silu", "torch_dtype": "bfloat16"}
    base = {"vocab": VOCAB, "width": width, "norm": {"eps": 1e-6}}
    rot = lambda dims: {"dims": dims, "base": 1000000.0}
    gqa = {"heads": heads, "kv_heads": z["kv_heads"], "dim": head, "vdim": head}
    latent = {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "rot": rot(64)}
    design = case["design"]
    if design == "zirurax":
        left = dict(gqa, scale=head ** -0.5, softcap=30.0, mask={"size": z["window"]}, rot=rot(head))
        right = {"heads": width // 32, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}
        kinds = [{"type": "parallel", "mixer": {"left": left, "right": right}, "mlp": {"kind": "dense", "ff": ff}}]
        return dict(base, architecture="Zirurax", embedding={"scale": 1.0}, layers=[kinds[0]] * layers)
    if design == "kinanex":
        delta = dict(gqa, conv=4)
        scan = {"inner": 2 * width, "state": 16, "dt_rank": width // 16, "conv": 4}
        att = dict(gqa, scale=head ** -0.5, v_mix=True,
                   rot=dict(rot(head // 2), scaling={"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}))
        mlp = {"kind": "dense", "ff": ff, "limit": 7.0}
        kinds = [("delta", delta, None), ("attention", att, mlp), ("mamba1", scan, None), ("attention", att, mlp)]
        return dict(base, architecture="Kinanex", logit_scale=1.0,
                    layers=[{"type": t, "mixer": m, "mlp": f} for t, m, f in (kinds[i % 4] for i in range(layers))])
    if design == "godotar":
        wkv = {"heads": width // 64, "dim": 64, "decay_rank": 64}
        lat = dict(latent, q_rank=3 * width // 8, mask={"size": z["window"]})
        moe = {"kind": "moe", "expert": {"ff": ff // 4, "limit": 7.0}, "router": {"experts": 16, "identity": 2, "top": 4}}
        kinds = [("wkv", wkv, {"kind": "dense", "ff": ff}), ("latent_attention", lat, moe), ("wkv", wkv, moe), ("wkv", wkv, moe)]
        return dict(base, architecture="Godotar", logit_scale=1.0,
                    layers=[{"type": t, "mixer": m, "mlp": f} for t, m, f in (kinds[i % 4] for i in range(layers))])
    moe = {"kind": "moe", "expert": {"ff": ff // 4}, "router": {"experts": 16, "top": 3, "groups": {"count": 4, "keep": 2}}, "shared": {"ff": ff // 4}}
    att = dict(gqa, scale=head ** -0.5, mask={"size": z["window"]}, rot=rot(head))
    mem = {"heads": width // 512, "dim": 256, "vdim": 512, "gate_cap": 15.0}
    kinds = [("attention", att), ("latent_attention", latent), ("mlstm", mem), ("attention", dict(att, kv_from=0))]
    return dict(base, architecture="Tugodra", embedding={"scale": 1.0},
                layers=[{"type": kinds[i % 4][0], "mixer": kinds[i % 4][1], "mlp": moe} for i in range(layers)])


def shapes(cfg):
    """Every tensor of the checkpoint: name -> shape."""
    out = {}
    if "architectures" in cfg:
        w, ff, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
        out.update({"model.embed_tokens.weight": (cfg["vocab_size"], w), "model.norm.weight": (w,)})
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}"
            q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
            for name, shape in (("input_layernorm", (w,)), ("post_attention_layernorm", (w,)), ("self_attn.q_proj", (q, w)),
                                ("self_attn.k_proj", (kv, w)), ("self_attn.v_proj", (kv, w)), ("self_attn.o_proj", (w, q)),
                                ("self_attn.q_norm", (d,)), ("self_attn.k_norm", (d,)), ("mlp.gate_proj", (ff, w)),
                                ("mlp.up_proj", (ff, w)), ("mlp.down_proj", (w, ff))):
                out[f"{p}.{name}.weight"] = shape
        return out
    arch, w = cfg["architecture"], cfg["width"]
    put = lambda prefix, **named: out.update({f"{prefix}.{n.replace('__', '.')}": s for n, s in named.items()})
    squash = lambda name: out.update({name: (w,), f"{name}.b": (w,), f"{name}.alpha": ()})
    out["embed"] = (cfg["vocab"], w)
    if arch == "Tugodra":
        out["head"] = (cfg["vocab"], w)
        squash("final.norm")
    else:
        out["final.norm"] = (w,)
    if arch in ("Kinanex", "Godotar"):
        out["embed.norm"] = (w,)
    for i, ly in enumerate(cfg["layers"]):
        kind, m, p, mlp = ly["type"], ly["mixer"], f"l{i}", ly["mlp"]
        for name in ("norm1", "norm1b", "norm2", "norm2b") if arch == "Tugodra" else ():
            squash(f"{p}.{name}")
        if arch != "Tugodra":
            out[f"{p}.norm1"] = (w,)
            if mlp and arch != "Zirurax":
                out[f"{p}.norm2"] = (w,)
        x = f"{p}.mix"
        if kind == "parallel":
            a, s = m["left"], m["right"]
            inner = s["heads"] * s["vdim"]
            channels = inner + 2 * s["groups"] * s["state"]
            hv = a["heads"] * a["vdim"]
            put(x + ".left", q=(a["heads"] * a["dim"], w), k=(a["kv_heads"] * a["dim"], w), v=(a["kv_heads"] * a["vdim"], w), g=(hv, w), o=(w, hv), out=(w,))
            put(x + ".right", **{"in": (inner + channels + s["heads"], w)}, conv=(channels, s["conv"]), conv__b=(channels,), dt_bias=(s["heads"],),
                A_log=(s["heads"],), D=(s["heads"],), norm=(inner,), o=(w, inner), out=(w,))
        elif kind == "delta":
            qk, v = m["kv_heads"] * m["dim"], m["heads"] * m["vdim"]
            put(x, q=(qk, w), k=(qk, w), v=(v, w), q__conv=(qk, m["conv"]), k__conv=(qk, m["conv"]), v__conv=(v, m["conv"]), b=(m["heads"], w),
                a=(m["heads"], w), A_log=(m["heads"],), dt_bias=(m["heads"],), norm=(m["vdim"],), g=(v, w), o=(w, v))
        elif kind == "mamba1":
            n, s, r = m["inner"], m["state"], m["dt_rank"]
            put(x, **{"in": (2 * n, w)}, conv=(n, m["conv"]), conv__b=(n,), x=(r + 2 * s, n), dt=(n, r), dt__b=(n,), A_log=(n, s), D=(n,), o=(w, n))
        elif kind == "wkv":
            hd, r = m["heads"] * m["dim"], m["decay_rank"]
            put(x, **{f"mu__{s}": (w,) for s in "rkvgw"}, **{s: (hd, w) for s in "rkvg"}, w1=(r, w), w2=(hd, r), w0=(hd,), u=(m["heads"], m["dim"]),
                norm=(hd,), o=(w, hd))
        elif kind == "latent_attention":
            h, q_in = m["heads"], m.get("q_rank", w)
            put(x, **({"dq": (q_in, w), "dq__norm": (q_in,), "uq": (h * (m["dim"] + m["rot_dim"]), q_in), "g": (h, w)} if arch == "Godotar" else
                      {"q": (h * (m["dim"] + m["rot_dim"]), w), "sink": (h,)}),
                dkv=(m["kv_rank"] + m["rot_dim"], w), dkv__norm=(m["kv_rank"],), uk=(h * m["dim"], m["kv_rank"]), uv=(h * m["vdim"], m["kv_rank"]),
                o=(w, h * m["vdim"]))
        elif kind == "mlstm":
            h = m["heads"]
            put(x, q=(h * m["dim"], w), k=(h * m["dim"], w), v=(h * m["vdim"], w), g=(h * m["vdim"], w), i=(h, w), f=(h, w), i__b=(h,), f__b=(h,),
                norm=(h * m["vdim"],), o=(w, h * m["vdim"]))
        else:
            q, k, v = m["heads"] * m["dim"], m["kv_heads"] * m["dim"], m["kv_heads"] * m["vdim"]
            put(x, q=(q, w), o=(w, m["heads"] * m["vdim"]))
            if m.get("kv_from") is None:
                put(x, k=(k, w), v=(v, w))
            if arch == "Tugodra":
                put(x, g=(m["heads"], w))
            else:
                put(x, q__b=(q,), k__b=(k,), v__b=(v,), q__norm=(m["dim"],), k__norm=(m["dim"],), talk=(m["heads"], m["heads"]), vmix=())
        if arch == "Kinanex":
            out[f"{p}.ls1"] = (w,)
            if mlp:
                out[f"{p}.ls2"] = (w,)
        if mlp and mlp["kind"] == "dense":
            put(f"{p}.mlp", gate=(mlp["ff"], w), up=(mlp["ff"], w), down=(w, mlp["ff"]))
        elif mlp:
            r, gated = mlp["router"], arch == "Godotar"
            n = r["experts"] + r.get("identity", 0)
            put(f"{p}.mlp", router=(n, w), correction=(n,))
            parts = [(f"e{e}", mlp["expert"]["ff"]) for e in range(r["experts"])]
            if mlp.get("shared"):
                parts.append(("shared", mlp["shared"]["ff"]))
                out[f"{p}.mlp.shared.sg"] = (1, w)
            for name, ff in parts:
                put(f"{p}.mlp.{name}", up=(ff, w), down=(w, ff), **({"gate": (ff, w)} if gated else {}))
    return out


class Weights:
    """A checkpoint drawn from a seed, tensor by tensor: projections of unit gain, gains around one, decays from slow to fast,
    router scores that spread.  What a sublayer adds to the stream is kept well below the stream, as in a trained
    model, so that an expert chosen by a hair's breadth moves a token little."""

    model_dir = "<drawn>"

    def __init__(self, cfg, seed, dtype):
        self.arch, self.seed, self.dtype = cfg.get("architecture", "dense"), seed, dtype
        self.shapes = shapes(cfg)

    def entries(self):
        return {n: (self.dtype, s) for n, s in self.shapes.items()}

    def get(self, name):
        shape, arch = self.shapes[name], self.arch
        seed = int.from_bytes(hashlib.sha256(f"{self.seed}:{name}".encode()).digest()[:7], "little")
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = torch.randn(shape, generator=g, device="cuda")
        u = torch.rand(shape, generator=g, device="cuda") if n.numel() < 1 << 20 else None
        last = name.rsplit(".", 1)[-1]
        if arch == "dense":
            t = 1.0 + 0.1 * n if len(shape) == 1 else n * 0.02
        elif name == "embed":
            t = n
        elif last == "alpha":
            t = 0.7 + 0.2 * u
        elif arch == "Godotar" and (last in ("norm1", "norm2") or name in ("embed.norm", "final.norm")):
            t = 0.1 * n
        elif last == "norm2b":
            t = 0.03 * (1.0 + 0.1 * n)
        elif last in ("norm", "norm1", "norm1b", "norm2", "out", "D"):
            t = 1.0 + 0.1 * n
        elif last in ("ls1", "ls2"):
            t = 0.3 + 0.1 * n
        elif last == "talk":
            t = torch.eye(shape[0], device="cuda") + 0.1 * n
        elif last == "vmix":
            t = torch.sigmoid(n)
        elif last == "A_log":
            t = 4.0 * u - 4.0 if len(shape) == 1 else torch.log(torch.arange(1, shape[1] + 1, device="cuda").float()).expand(shape) + 0.1 * n
        elif last == "dt_bias" or name.endswith("dt.b"):
            t = 0.5 * n - 1.0
        elif ".mu." in name:
            t = u
        elif last == "w0":
            t = 5.0 * u - 5.5
        elif last == "u" and ".mix." in name:
            t = 0.5 * n
        elif name.endswith("i.b"):
            t = n - 0.5
        elif name.endswith("f.b"):
            t = 2.5 + n
        elif last == "sink":
            t = 1.0 + n
        elif last in ("b", "correction"):
            t = 0.05 * n
        elif last == "conv":
            t = 0.5 * n
        elif last == "router":
            t = 3.0 * n / math.sqrt(shape[-1])
        else:
            small = {"o": 0.3, "down": 0.05}.get(last, 1.0) if arch == "Godotar" else 1.0
            t = n * (small / math.sqrt(shape[-1]))
        return t.to(self.dtype)


# --------------------------------------------------------------------------- what a program has in hand, and one pass

def _numbers(text):
    """"1103,640@3072" -> [(1103, 0), (640, 3072)]: (tokens, positions cached before them)."""
    return [tuple(int(x) for x in (item + "@0").split("@")[:2]) for item in text.split(",")]


def _contexts(case):
    """Positions cached before a decode step, request by request, spread between ``low`` and ``high``."""
    return [case["low"] + int((case["high"] - case["low"]) * ((i * 0.6180339887) % 1.0)) for i in range(case["rows"])]


def _sequences(case, seed):
    """For each request of the case: (tokens before the pass, tokens the pass brings)."""
    if case["kind"] in ("request", "generate"):
        plan = [(0, n + (case["new"] if case["kind"] == "request" else 0)) for n, _ in _numbers(case["prompts"])]
    else:
        plan = [(c, 1) for c in _contexts(case)] + [(p, n) for n, p in (_numbers(case["portions"]) if case["kind"] == "portions" else [])]
    g = torch.Generator().manual_seed(seed * 7919 + 17)
    ids = [torch.randint(0, VOCAB, (p + n,), generator=g).tolist() for p, n in plan]
    return [(t[:p], t[p:]) for t, (p, _) in zip(ids, plan)]


def prepare(case, seed):
    from lily_b200 import Engine, EngineConfig, SamplingParams, ServerArgs
    from lily_b200.config.registry import architecture_names, resolve_architecture
    from lily_b200.engine.batch import StepEntry
    from lily_b200.engine.runner import ModelRunner

    cfg = config(case)
    arch = resolve_architecture(architecture_names(cfg))
    dtype = "float32" if case["kind"] == "generate" else "bfloat16"
    seqs = _sequences(case, seed)
    longest = max(len(a) + len(b) for a, b in seqs) + case.get("new", 0) + 2
    count = len(seqs)
    args = dict(dtype=dtype, device="cuda:0", context_length=-(-longest // 256) * 256, max_running_requests=count,
                max_total_tokens=sum(-(-(len(a) + len(b) + case.get("new", 0) + 2) // PAGE) * PAGE for a, b in seqs) + PAGE * count)
    more = dict(page_size=PAGE, random_seed=0)
    source = Weights(cfg, seed, torch.float32 if dtype == "float32" else torch.bfloat16)
    runner = ModelRunner(arch.build_spec(arch.config_from_dict(cfg, {}, architecture=arch.name)), source, ServerArgs(**args, **more))
    state = {"kind": case["kind"], "runner": runner}
    if case["kind"] != "portions":
        runner.capture_decode_graphs([count])
    if case["kind"] == "generate":
        state["engine"] = Engine(EngineConfig("<drawn>", **args, server_args=more), runner=runner)
        state["prompts"] = [b for _, b in seqs]
        state["params"] = SamplingParams(max_new_tokens=case["new"], ignore_eos=True, logprobs=True)
    elif case["kind"] == "request":
        state["prompts"] = [b[:len(b) - case["new"]] for _, b in seqs]
        state["answers"] = [b[len(b) - case["new"]:] for _, b in seqs]
    else:
        slots = [runner.open_request() for _ in seqs]
        for slot, (before, _) in zip(slots, seqs):
            if before:
                runner.step([StepEntry(slot, before, [])])
        state["entries"] = [StepEntry(slot, now, [len(now) - 1]) for slot, (_, now) in zip(slots, seqs)]
        state["at"] = {slot: len(before) for slot, (before, _) in zip(slots, seqs)}
    return state


@torch.inference_mode()
def run(state):
    from lily_b200.engine.batch import StepEntry

    runner = state["runner"]
    if state["kind"] == "generate":
        outs = state["engine"].generate(state["prompts"], state["params"])
        return {"tokens": torch.tensor([o["output_ids"] for o in outs]), "logprobs": torch.tensor([o["logprobs"] for o in outs])}
    if state["kind"] == "request":
        slots = [runner.open_request() for _ in state["prompts"]]
        logits = [runner.step([StepEntry(s, p, [len(p) - 1]) for s, p in zip(slots, state["prompts"])])]
        for tokens in zip(*state["answers"]):
            logits.append(runner.step([StepEntry(s, [t], [0]) for s, t in zip(slots, tokens)]).clone())
        for s in slots:
            runner.close_request(s)
        return torch.stack(logits)
    logits = runner.step(state["entries"])
    # the step's tokens are let go of again: the next pass stands where this one stood
    runner.seq_lens.update(state["at"])
    return logits


# --------------------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Weights read once a step (experts: those that the step's tokens can touch), cached rows and states read and written once a
    step, logits written; products of every token with the weights it meets, attention over the keys it sees, state updates."""
    cfg, item = config(case), 4 if case["kind"] == "generate" else 2
    seqs = [(len(a), len(b)) for a, b in _sequences(case, 0)]
    new = case.get("new", 0)
    if case["kind"] == "request":
        steps = [[(0, n - new) for _, n in seqs]] + [[(n - new + k, 1) for _, n in seqs] for k in range(new)]
    elif case["kind"] == "generate":
        steps = [[(0, n) for _, n in seqs]] + [[(n + k, 1) for _, n in seqs] for k in range(new - 1)]
    else:
        steps = [seqs]
    layers = cfg["layers"] if "layers" in cfg else [{"type": "gqa", "mixer": dict(
        heads=cfg["num_attention_heads"], kv_heads=cfg["num_key_value_heads"], dim=cfg["head_dim"], vdim=cfg["head_dim"]), "mlp": {"kind": "dense"}}
    ] * cfg["num_hidden_layers"]
    width = cfg.get("width") or cfg["hidden_size"]
    sizes = {n: math.prod(s) for n, s in shapes(cfg).items()}
    fixed = sum(v for n, v in sizes.items() if ".mlp.e" not in n and not n.endswith(("embed", "embed_tokens.weight", "head")))
    table = VOCAB * width
    bytes_, flops = 0.0, 0.0
    for step in steps:
        tokens = sum(n for _, n in step)
        bytes_ += (fixed + table) * item + tokens * width * item + len(step) * VOCAB * 4
        flops += 2.0 * fixed * tokens + 2.0 * table * len(step)
        for i, ly in enumerate(layers):
            mlp = ly.get("mlp")
            if mlp and mlp["kind"] == "moe":
                one = sum(v for n, v in sizes.items() if n.startswith(f"l{i}.mlp.e0."))
                bytes_ += one * item * min(mlp["router"]["experts"], tokens * mlp["router"]["top"])
                flops += 2.0 * one * tokens * mlp["router"]["top"]
            m = ly["mixer"]
            mixers = [m["left"], dict(m["right"], ssd=True)] if ly["type"] == "parallel" else [m]
            for mix in mixers:
                if mix.get("ssd"):
                    state = mix["heads"] * mix["vdim"] * mix["state"]
                elif ly["type"] == "mamba1":
                    state = mix["inner"] * mix["state"]
                elif ly["type"] in ("delta", "wkv", "mlstm"):
                    state = mix["heads"] * mix["dim"] * mix.get("vdim", mix["dim"])
                else:
                    row = mix["kv_rank"] + mix["rot_dim"] if "kv_rank" in mix else mix["kv_heads"] * (mix["dim"] + mix["vdim"])
                    per = mix["heads"] * (mix["dim"] + mix.get("rot_dim", 0) + mix["vdim"])
                    window = (mix.get("mask") or {}).get("size") or 1 << 30
                    for before, n in step:
                        bytes_ += row * item * min(before + n, window + n)
                        flops += 2.0 * per * sum(min(before + j + 1, window) for j in range(n))
                    continue
                bytes_ += 8.0 * state * len(step)
                flops += 6.0 * state * tokens
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    # bfloat16: every projection, activation and cached row is rounded to 8 bits.  Against 64 bits the logits of the dense
    # decoder (whose stream is all sublayers and little embedding) are 1.1 to 2.0 % off in the 2-norm, those of the
    # others 0.2 to 0.6 %; float32 is 4e-7 off.
    if case["kind"] == "generate":
        return {"rel": 2e-6, "max": 2e-5, "differ": 0.0}
    return {"rel": 3e-2 if case["kind"] != "request" else 2e-2, "max": 0.3}


# --------------------------------------------------------------------------- the same in 64 bits

def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _halves(x, rot, start=0):
    """x [t, heads, n]: column i < dims/2 turns with column i + dims/2 by position * f_i (float32 angles)."""
    dims = rot["dims"]
    f = float(rot["base"]) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=x.device) / dims)
    sc = rot.get("scaling")
    if sc:
        wave = 2.0 * math.pi / f
        s = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
        f = torch.where(wave < sc["original"] / sc["high"], f, torch.where(wave > sc["original"] / sc["low"], f / sc["factor"], (1 - s) * f / sc["factor"] + s * f))
    ang = torch.arange(x.shape[0], device=x.device).float()[:, None] * f.float()[None]
    cos, sin = ang.cos().double()[:, None], ang.sin().double()[:, None]
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * cos - v * sin, v * cos + u * sin, x[..., dims:]], -1)


def _neighbours(x, rot):
    """The same with columns 2i and 2i + 1 as pairs."""
    dims = rot["dims"]
    order = torch.cat([torch.arange(0, dims, 2), torch.arange(1, dims, 2), torch.arange(dims, x.shape[-1])]).to(x.device)
    return _halves(x[..., order], rot)[..., torch.argsort(order)]


def _attend(q, k, v, scale, window=None, cap=None, sink=None):
    """q [t, H, d], k [t, G, d], v [t, G, dv] -> [t, H, dv], causal, some heads and queries at a time."""
    t, heads = q.shape[:2]
    share = heads // k.shape[1]
    out = q.new_empty(t, heads, v.shape[-1])
    at = torch.arange(t, device=q.device)
    for i in range(0, t, 1024):
        rows = at[i:i + 1024]
        keys = at[:rows[-1] + 1]
        back = rows[:, None] - keys[None]
        hidden = (back < 0) | (back >= (window or 1 << 30))
        for h in range(heads):
            s = (q[rows, h] @ k[keys, h // share].t()) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            s = s.masked_fill(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(len(rows), 1)], -1)
            out[i:i + 1024, h] = torch.softmax(s, -1)[:, :len(keys)] @ v[keys, h // share]
    return out


def _conv(x, taps, bias=None):
    n = taps.shape[1]
    padded = torch.cat([x.new_zeros(n - 1, x.shape[1]), x])
    y = sum(padded[j:j + len(x)] * taps[:, j] for j in range(n))
    return y if bias is None else y + bias


def _heads(x, n):
    return x.view(x.shape[0], n, -1)


def _ssd(h, w, p, c):
    heads, n, groups = c["heads"], c["state"], c["groups"]
    inner = heads * c["vdim"]
    proj = h @ w(f"{p}.in").t()
    z, xbc, dt = proj.split([inner, inner + 2 * groups * n, heads], -1)
    x, b, cc = F.silu(_conv(xbc, w(f"{p}.conv"), w(f"{p}.conv.b"))).split([inner, groups * n, groups * n], -1)
    x = _heads(x, heads)
    b, cc = (_heads(y, groups).repeat_interleave(heads // groups, 1) for y in (b, cc))
    dt = F.softplus(dt + w(f"{p}.dt_bias"))
    decay = torch.exp(-torch.exp(w(f"{p}.A_log")) * dt)
    S, y = x.new_zeros(heads, n, c["vdim"]), torch.empty_like(x)
    for t in range(len(h)):
        S = decay[t][:, None, None] * S + (dt[t][:, None] * b[t])[:, :, None] * x[t][:, None]
        y[t] = torch.einsum("hnp,hn->hp", S, cc[t])
    y = (y + w(f"{p}.D")[:, None] * x).reshape(len(h), inner) * F.silu(z)
    return (_rms(_heads(y, c["norm_groups"])).reshape(len(h), inner) * w(f"{p}.norm")) @ w(f"{p}.o").t()


def _delta(h, w, p, c):
    heads, groups, d = c["heads"], c["kv_heads"], c["dim"]
    act = lambda name, n: _heads(F.silu(_conv(h @ w(f"{p}.{name}").t(), w(f"{p}.{name}.conv"))), n)
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q, k = (unit(act(name, groups)).repeat_interleave(heads // groups, 1) for name in "qk")
    v = act("v", heads)
    b = torch.sigmoid(h @ w(f"{p}.b").t())
    a = torch.exp(-torch.exp(w(f"{p}.A_log")) * F.softplus(h @ w(f"{p}.a").t() + w(f"{p}.dt_bias")))
    S, o = h.new_zeros(heads, d, c["vdim"]), torch.empty_like(v)
    for t in range(len(h)):
        S = a[t][:, None, None] * S
        u = b[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None]
        o[t] = torch.einsum("hdv,hd->hv", S, q[t]) * d ** -0.5
    o = _rms(o) * w(f"{p}.norm") * _heads(F.silu(h @ w(f"{p}.g").t()), heads)
    return o.reshape(len(h), -1) @ w(f"{p}.o").t()


def _selective(h, w, p, c):
    x, z = (h @ w(f"{p}.in").t()).chunk(2, -1)
    x = F.silu(_conv(x, w(f"{p}.conv"), w(f"{p}.conv.b")))
    low, B, C = (x @ w(f"{p}.x").t()).split([c["dt_rank"], c["state"], c["state"]], -1)
    dt = F.softplus(low @ w(f"{p}.dt").t() + w(f"{p}.dt.b"))
    A = -torch.exp(w(f"{p}.A_log"))
    S, y = torch.zeros_like(A), torch.empty_like(x)
    for t in range(len(h)):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * x[t])[:, None] * B[t]
        y[t] = S @ C[t]
    return ((y + w(f"{p}.D") * x) * F.silu(z)) @ w(f"{p}.o").t()


def _wkv(h, w, p, c):
    heads, d = c["heads"], c["dim"]
    before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
    mixed = lambda s: h + (before - h) * w(f"{p}.mu.{s}")
    r, k, v = (_heads(mixed(s) @ w(f"{p}.{s}").t(), heads) for s in "rkv")
    gate = F.silu(mixed("g") @ w(f"{p}.g").t())
    decay = _heads(torch.exp(-torch.exp(torch.tanh(mixed("w") @ w(f"{p}.w1").t()) @ w(f"{p}.w2").t() + w(f"{p}.w0"))), heads)
    u, S, o = w(f"{p}.u"), h.new_zeros(heads, d, d), torch.empty_like(v)
    for t in range(len(h)):
        kv = k[t][:, :, None] * v[t][:, None]
        o[t] = torch.einsum("hi,hij->hj", r[t], S + u[:, :, None] * kv)
        S = decay[t][:, :, None] * S + kv
    return (_rms(o).reshape(len(h), -1) * w(f"{p}.norm") * gate) @ w(f"{p}.o").t()


def _mlstm(h, w, p, c):
    heads, d = c["heads"], c["dim"]
    q, k, v = (_heads(h @ w(f"{p}.{s}").t(), heads) for s in "qkv")
    soft = lambda s: c["gate_cap"] * torch.tanh((h @ w(f"{p}.{s}").t() + w(f"{p}.{s}.b")) / c["gate_cap"])
    i, f = soft("i"), F.logsigmoid(soft("f"))
    S, n, m, o = h.new_zeros(heads, d, c["vdim"]), h.new_zeros(heads, d), h.new_zeros(heads), torch.empty_like(v)
    for t in range(len(h)):
        new = torch.maximum(f[t] + m, i[t])
        keep, write = torch.exp(f[t] + m - new), torch.exp(i[t] - new)
        S = keep[:, None, None] * S + (write[:, None] * k[t])[:, :, None] * v[t][:, None]
        n = keep[:, None] * n + write[:, None] * k[t]
        m = new
        qt = q[t] * d ** -0.5
        o[t] = torch.einsum("hdv,hd->hv", S, qt) / (torch.maximum((n * qt).sum(-1).abs(), torch.exp(-m)) + 1e-6)[:, None]
    return (_rms(o).reshape(len(h), -1) * w(f"{p}.norm") * torch.sigmoid(h @ w(f"{p}.g").t())) @ w(f"{p}.o").t()


def _latent(h, w, p, c, godotar):
    heads, d = c["heads"], c["dim"]
    q = (_rms(h @ w(f"{p}.dq").t()) * w(f"{p}.dq.norm")) @ w(f"{p}.uq").t() if godotar else h @ w(f"{p}.q").t()
    q = _heads(q, heads)
    down = h @ w(f"{p}.dkv").t()
    latent = _rms(down[:, :c["kv_rank"]]) * w(f"{p}.dkv.norm")
    turned = _halves(down[:, None, c["kv_rank"]:], c["rot"]).expand(-1, heads, -1)
    k = torch.cat([_heads(latent @ w(f"{p}.uk").t(), heads), turned], -1)
    q = torch.cat([q[..., :d], _halves(q[..., d:], c["rot"])], -1)
    o = _attend(q, k, _heads(latent @ w(f"{p}.uv").t(), heads), c["scale"], (c.get("mask") or {}).get("size"),
                sink=None if godotar else w(f"{p}.sink"))
    if godotar:
        o = o * torch.sigmoid(h @ w(f"{p}.g").t())[..., None]
    return o.reshape(len(h), -1) @ w(f"{p}.o").t()


def _mixed_heads(h, w, p, c, v):
    heads = c["heads"]
    share = heads // c["kv_heads"]
    q, k = (_halves(_rms(_heads(h @ w(f"{p}.{s}").t() + w(f"{p}.{s}.b"), n)) * w(f"{p}.{s}.norm"), c["rot"])
            for s, n in (("q", heads), ("k", c["kv_heads"])))
    at, out = torch.arange(len(h), device=h.device), []
    for i in range(0, len(h), 512):
        rows = at[i:i + 512]
        s = torch.einsum("ihd,jhd->hij", q[rows], k.repeat_interleave(share, 1)) * c["scale"]
        s = s.masked_fill(rows[:, None] < at[None], -math.inf)
        weights = torch.softmax(torch.cat([s, s.new_zeros(heads, len(rows), 1)], -1), -1)[..., :-1]
        weights = torch.einsum("hg,gij->hij", w(f"{p}.talk"), weights)
        out.append(torch.einsum("hij,jhe->ihe", weights, v.repeat_interleave(share, 1)))
    return torch.cat(out).reshape(len(h), -1) @ w(f"{p}.o").t()


def _experts(h, w, p, c, godotar):
    r = c["router"]
    logits = h @ w(f"{p}.router").t()
    s = torch.softmax(logits, -1) if godotar else torch.sigmoid(logits)
    choice = s + w(f"{p}.correction")
    if r.get("groups"):
        g = choice.view(len(h), r["groups"]["count"], -1)
        kept = torch.topk(torch.topk(g, 2, dim=-1).values.sum(-1), r["groups"]["keep"], dim=-1).indices
        choice = g.masked_fill(torch.ones_like(g[..., 0], dtype=torch.bool).scatter_(1, kept, False)[..., None], -math.inf).flatten(1)
    chosen = torch.topk(choice, r["top"], dim=-1).indices
    weight = s.gather(1, chosen)
    weight = torch.zeros_like(s).scatter_(1, chosen, weight / (weight.sum(-1, keepdim=True) + 1e-20))
    plain = lambda x, name: torch.relu(x @ w(f"{p}.{name}.up").t()) ** 2 @ w(f"{p}.{name}.down").t()

    def clamped(x, name):
        g = torch.clamp(x @ w(f"{p}.{name}.gate").t(), max=c["expert"]["limit"])
        u = torch.clamp(x @ w(f"{p}.{name}.up").t(), -c["expert"]["limit"], c["expert"]["limit"])
        return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(f"{p}.{name}.down").t()
    out = torch.zeros_like(h)
    for e in range(s.shape[1]):
        rows = torch.nonzero(weight[:, e]).flatten()
        y = h[rows] if e >= r["experts"] else (clamped if godotar else plain)(h[rows], f"e{e}")
        out[rows] += weight[rows, e:e + 1] * y
    return out if not c.get("shared") else out + plain(h, "shared") * torch.sigmoid(h @ w(f"{p}.shared.sg").t())


def _forward(cfg, w, ids):
    """Logits of one whole sequence at the places ``ids[1]``, in float64."""
    tokens, wanted = torch.tensor(ids[0], device="cuda"), ids[1]
    if "architectures" in cfg:
        E = w("model.embed_tokens.weight")
        x, heads, kv = E[tokens], cfg["num_attention_heads"], cfg["num_key_value_heads"]
        rot = {"dims": cfg["head_dim"], "base": cfg["rope_theta"]}
        for i in range(cfg["num_hidden_layers"]):
            g = lambda name, p=f"model.layers.{i}": w(f"{p}.{name}.weight")
            h = _rms(x) * g("input_layernorm")
            q = _halves(_rms(_heads(h @ g("self_attn.q_proj").t(), heads)) * g("self_attn.q_norm"), rot)
            k = _halves(_rms(_heads(h @ g("self_attn.k_proj").t(), kv)) * g("self_attn.k_norm"), rot)
            o = _attend(q, k, _heads(h @ g("self_attn.v_proj").t(), kv), cfg["head_dim"] ** -0.5)
            x = x + o.reshape(len(x), -1) @ g("self_attn.o_proj").t()
            h = _rms(x) * g("post_attention_layernorm")
            x = x + (F.silu(h @ g("mlp.gate_proj").t()) * (h @ g("mlp.up_proj").t())) @ g("mlp.down_proj").t()
        return (_rms(x[wanted]) * w("model.norm.weight")) @ E.t()
    arch, E, kept, first = cfg["architecture"], w("embed"), {}, None
    x = E[tokens]
    if arch == "Godotar":
        x = _rms(x) * (1 + w("embed.norm"))
    elif arch == "Kinanex":
        x = _rms(x) * w("embed.norm")

    def norm(y, name):
        if arch == "Tugodra":
            return torch.tanh(y * w(f"{name}.alpha")) * w(name) + w(f"{name}.b")
        return _rms(y) * ((1 if arch == "Godotar" else 0) + w(name))
    for i, ly in enumerate(cfg["layers"]):
        kind, c, p, mlp = ly["type"], ly["mixer"], f"l{i}", ly["mlp"]
        m = f"{p}.mix"
        h = norm(x, f"{p}.norm1")
        if kind == "parallel":
            a = c["left"]
            q, k = (_neighbours(_heads(h @ w(f"{m}.left.{s}").t(), n), a["rot"]) for s, n in (("q", a["heads"]), ("k", a["kv_heads"])))
            o = _attend(q, k, _heads(h @ w(f"{m}.left.v").t(), a["kv_heads"]), a["scale"], a["mask"]["size"], a["softcap"]).reshape(len(x), -1)
            left = (o * torch.sigmoid(h @ w(f"{m}.left.g").t())) @ w(f"{m}.left.o").t()
            y = 0.5 * (_rms(left) * w(f"{m}.left.out") + _rms(_ssd(h, w, f"{m}.right", c["right"])) * w(f"{m}.right.out"))
            gate = F.gelu(h @ w(f"{p}.mlp.gate").t(), approximate="tanh")
            x = x + y + (gate * (h @ w(f"{p}.mlp.up").t())) @ w(f"{p}.mlp.down").t()
            continue
        if kind == "latent_attention":
            y = _latent(h, w, m, c, arch == "Godotar")
        elif kind == "attention" and arch == "Kinanex":
            v = _rms(_heads(h @ w(f"{m}.v").t() + w(f"{m}.v.b"), c["kv_heads"]))
            if first is None:
                first = v
            else:
                v = (1 - w(f"{m}.vmix")) * v + w(f"{m}.vmix") * first
            y = _mixed_heads(h, w, m, c, v)
        elif kind == "attention":
            q = _rms(_neighbours(_heads(h @ w(f"{m}.q").t(), c["heads"]), c["rot"]))
            src = c.get("kv_from", i)
            if src == i:
                kept[i] = (_rms(_neighbours(_heads(h @ w(f"{m}.k").t(), c["kv_heads"]), c["rot"])), _heads(h @ w(f"{m}.v").t(), c["kv_heads"]))
            o = _attend(q, *kept[src], c["scale"], c["mask"]["size"]) * torch.sigmoid(h @ w(f"{m}.g").t())[..., None]
            y = o.reshape(len(x), -1) @ w(f"{m}.o").t()
        else:
            y = {"delta": _delta, "mamba1": _selective, "wkv": _wkv, "mlstm": _mlstm}[kind](h, w, m, c)
        if arch == "Godotar":
            h = norm(x, f"{p}.norm2")
            if mlp["kind"] == "dense":
                y = y + (F.silu(h @ w(f"{p}.mlp.gate").t()) * (h @ w(f"{p}.mlp.up").t())) @ w(f"{p}.mlp.down").t()
            else:
                y = y + _experts(h, w, f"{p}.mlp", mlp, True)
            x = x + y
        elif arch == "Tugodra":
            x = x + norm(y, f"{p}.norm1b")
            x = x + norm(_experts(norm(x, f"{p}.norm2"), w, f"{p}.mlp", mlp, False), f"{p}.norm2b")
        else:
            x = x + w(f"{p}.ls1") * y
            if mlp:
                h = norm(x, f"{p}.norm2")
                g = torch.clamp(h @ w(f"{p}.mlp.gate").t(), max=mlp["limit"])
                u = torch.clamp(h @ w(f"{p}.mlp.up").t(), -mlp["limit"], mlp["limit"])
                x = x + w(f"{p}.ls2") * ((g * torch.sigmoid(1.702 * g) * (u + 1)) @ w(f"{p}.mlp.down").t())
    return norm(x[wanted], "final.norm") @ (w("head") if arch == "Tugodra" else E).t()


@torch.no_grad()
def exact(case, seed):
    cfg = config(case)
    source = Weights(cfg, seed, torch.float32 if case["kind"] == "generate" else torch.bfloat16)
    held = {n: source.get(n).double() for n in source.shapes}
    seqs, new = _sequences(case, seed), case.get("new", 0)
    if case["kind"] == "generate":
        probs = []
        for _, prompt in seqs:
            ids, row = list(prompt), []
            for _ in range(new):
                logp = torch.log_softmax(_forward(cfg, held.__getitem__, (ids, [-1]))[0], -1)
                ids.append(int(logp.argmax()))
                row.append(float(logp.max()))
            probs.append(row)
        return {"tokens": None, "logprobs": torch.tensor(probs, dtype=torch.float64)}
    places = [list(range(len(b) - new - 1, len(b))) if case["kind"] == "request" else [-1] for _, b in seqs]
    logits = [_forward(cfg, held.__getitem__, (a + b, at)) for (a, b), at in zip(seqs, places)]
    if case["kind"] == "request":
        return torch.stack(logits, 1)
    return torch.cat(logits)
