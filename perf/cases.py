"""What a user of this framework has it do, as cases that can be timed and compared.

A case names a model (the Llama shapes of `config.py`, or a layer-list family at the layer shapes of `bench.py --arch`), a
call and the sizes.  Calls, all through the public Python surface with ids on the host, as a program makes them:

* "step":   one `Llama.forward_f32` of one token per sequence behind a cached prefix - a program that samples for itself;
* "prompt": a whole prompt - `Llama.forward_f32` (logits of the last token) or `StackDecoder.forward_rows` (logits of 16
            rows per sequence, as a scoring program asks for);
* "greedy": `generate_all`, then the logits of the next position for up to four of the sequences.

Models are cut to a few layers, so that `exact` can restate them in 64 bits.  Weights are values that bfloat16 holds, as a
checkpoint has them; the output projection favours one token by a wide margin, as a trained model's does, so that greedy
tokens do not hang on the last bit.  Mixtures of experts sit in the first layer of parallel-sublayer models, where the router
reads nothing that was rounded to 16 bits: which experts are chosen is then the same in every correct implementation.
"""
import math

import numpy as np
import torch

import llama3_np_b200  # noqa: F401
from llama3_np_b200 import Debuzen, Gifudra, Llama, Mabedra, ModelArgs, Risalix, Vupitar

FAMILIES = {"risalix": Risalix, "mabedra": Mabedra, "debuzen": Debuzen, "gifudra": Gifudra, "vupitar": Vupitar}
ROWS = 16   # rows per sequence whose logits a "prompt" call of a layer-list model asks for


# ---------------------------------------------------------------------------------------------------------- the cases
def _llama(call, dtype, width, heads, kv_heads, ff, layers, vocab, batch, prompt, new=0):
    return {"model": "llama", "call": call, "dtype": dtype, "width": width, "heads": heads, "kv_heads": kv_heads, "ff": ff,
            "layers": layers, "vocab": vocab, "batch": batch, "prompt": prompt, "new": new}


def _small(call, batch, prompt, new=0):    # the stories15M shape, whole
    return _llama(call, "float32", 288, 6, 6, 768, 6, 32000, batch, prompt, new)


def _1b(call, batch, prompt, new=0):       # Llama-3.2-1B layers
    return _llama(call, "bfloat16", 2048, 32, 8, 8192, 2, 16384, batch, prompt, new)


def _8b(call, batch, prompt, new=0):       # Llama-3-8B layers
    return _llama(call, "bfloat16", 4096, 32, 8, 14336, 2, 16384, batch, prompt, new)


def _family(model, call, dtype, width, batch, prompt, new=0):
    return {"model": model, "call": call, "dtype": dtype, "width": width, "vocab": 8192, "batch": batch, "prompt": prompt, "new": new}


def listed():
    return [
        # the smallest call: one token of one sequence, host ids in, host logits out
        dict(_small("step", 1, 100), name="small-step-b1"),
        # the reference's own run: a five-token prompt, fifty tokens in all, fp32
        dict(_small("greedy", 1, 5, 45), name="small-greedy-b1"),
        # serving many users of the small model: the framework's headline, fp32
        dict(_small("greedy", 256, 64, 64), name="small-greedy-b256"),
        # two prompts of an odd length at the 1B layer shape
        dict(_1b("prompt", 2, 731), name="1b-prompt"),
        # a long prompt at the 8B layer shape: the largest call
        dict(_8b("prompt", 1, 4096), name="8b-prompt"),
        # one user / thirty-two users of the 8B layer shape
        dict(_8b("greedy", 1, 200, 40), name="8b-greedy-b1"),
        dict(_8b("greedy", 32, 40, 40), name="8b-greedy-b32"),
        # prompts of the layer-list families: each layer kind once, one sequence or ragged portions of several
        dict(_family("risalix", "prompt", "bfloat16", 2048, 1, 2048), name="risalix-prompt"),
        dict(_family("mabedra", "prompt", "bfloat16", 2048, 1, 2000), name="mabedra-prompt"),
        dict(_family("debuzen", "prompt", "bfloat16", 2048, 3, 701), name="debuzen-prompt"),
        # the default dtype at a middling size
        dict(_family("gifudra", "prompt", "float32", 1024, 1, 600), name="gifudra-prompt-f32"),
        # batched decode of a layer-list family
        dict(_family("vupitar", "greedy", "bfloat16", 2048, 8, 96, 32), name="vupitar-greedy-b8"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "small", "bf16-prompt", "bf16-greedy", "family", "family", "family", "family-greedy"])
    if kind == "small":
        call = rng.choice(["step", "greedy", "prompt"])
        b = _log(rng, 1, 256 if call == "greedy" else 32)
        p = _log(rng, 2, 60 if b > 64 else 150)
        return _small(call, b, p, _log(rng, 4, 64) if call == "greedy" else 0)
    if kind == "bf16-prompt":
        n = _log(rng, 10, 3500)
        return rng.choice([_1b, _8b])("prompt", rng.randint(1, max(1, min(4, 3500 // n))), n)
    if kind == "bf16-greedy":
        return rng.choice([_1b, _8b])("greedy", _log(rng, 1, 32), _log(rng, 5, 120), _log(rng, 4, 40))
    model, width = rng.choice(sorted(FAMILIES)), 128 * rng.choice([4, 8, 12, 16])
    if kind == "family-greedy":
        return _family(model, "greedy", "bfloat16", width, _log(rng, 1, 12), _log(rng, 5, 150), _log(rng, 4, 32))
    if rng.random() < 0.25:
        return _family(model, "prompt", "float32", 128 * rng.choice([4, 6, 8]), rng.randint(1, 2), _log(rng, 20, 400))
    n = _log(rng, 20, 1900)
    return _family(model, "prompt", "bfloat16", width, rng.randint(1, max(1, min(4, 1900 // n))), n)


# ------------------------------------------------------------------------------------------------- shapes and weights
def _config(case):
    """config.json of a layer-list model."""
    W, model = case["width"], case["model"]
    H = W // 128
    kv = max(1, H // 4)
    base = {"architecture": model.capitalize(), "vocab": case["vocab"], "width": W, "norm": {"eps": 1e-5}}
    if model == "risalix":
        decays = [float(1.0 - 2.0 ** (-(2 + 6 * i / max(1, H - 1)))) for i in range(H)]
        lin = {"type": "lightning", "mixer": {"heads": H, "dim": 128, "vdim": 128, "decay": decays}, "mlp": None}
        dlt = {"type": "channel_delta", "mlp": None,
               "mixer": {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4, "rank_decay": W // 16, "rank_gate": W // 16}}
        att = {"type": "attention", "mixer": {"heads": H, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5},
               "mlp": {"kind": "dense", "ff": 4 * W}}
        return dict(base, layers=[lin, dlt, att], residual_mult=0.5, token_side={"dim": 256})
    if model == "mabedra":
        mixer = {"heads": H, "kv_heads": kv, "dim": 64, "vdim": 128, "diff": 0.3, "scale": 64 ** -0.5, "mask": {"size": 1024},
                 "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
        moe = {"kind": "moe", "expert": {"ff": W // 2}, "router": {"experts": 16, "top": 2}, "shared": {"ff": W}}
        return dict(base, canon={"taps": 4}, layers=[{"type": "attention", "mixer": mixer, "mlp": moe},
                                                     {"type": "attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": 4 * W}}])
    if model == "debuzen":
        mlp = {"kind": "dense", "ff": 4 * W}
        a1 = {"heads": H, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 0.2, "mask": {"size": 1024, "keep_first": 4},
              "rot": {"base": 1000000.0, "dims": 64}}
        a2 = dict(a1, scale=128 ** -0.5, mask={"size": 1024}, rot={"base": 500000.0, "dims": 64})
        par = {"type": "parallel", "mlp": mlp,
               "mixer": {"left": a1, "left_scale": 1.0, "right_scale": 1.0,
                         "right": {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4, "rank_decay": W // 16, "rank_gate": W // 16}}}
        par2 = {"type": "parallel_2", "mlp": mlp,
                "mixer": {"left": a2, "left_scale": 1.0, "right_scale": 1.0,
                          "right": {"heads": W // 64, "groups": 2, "state": 128, "vdim": 64, "conv": 4, "norm_groups": 2}}}
        gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": W // 256, "dim": 128, "vdim": 256, "tau": 16.0, "rank_decay": 16}}
        return dict(base, norm={"eps": 1e-6, "groups": 4}, layers=[par, par2, gla], logit_softcap=30.0)
    if model == "gifudra":
        mixer = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": 3 * W // 4, "kv_rank": 512, "scale": 192 ** -0.5,
                 "rot": {"base": 10000.0, "dims": 64}}
        mlp = {"kind": "dense", "ff": 4 * W}
        return dict(base, streams=4, embedding={"scale": 1.0}, logit_scale=W ** -0.5,
                    layers=[{"type": "latent_attention", "mixer": mixer, "mlp": mlp},
                            {"type": "latent_attention", "mixer": dict(mixer, kv_from=0), "mlp": mlp}])
    mixer = {"left": {"heads": H, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024},
                      "rot": {"base": 500000.0, "dims": 64}},
             "right": {"heads": max(1, W // 256), "dim": 128, "vdim": 256, "gate_cap": 15.0}, "left_scale": 1.0, "right_scale": 1.0}
    moe = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": W // 2}, "shared": {"ff": W}}
    return dict(base, norm={"eps": 1e-6}, embedding={"scale": 1.0},
                layers=[{"type": "parallel", "mixer": mixer, "mlp": moe},
                        {"type": "parallel", "mixer": mixer, "mlp": {"kind": "dense", "ff": 4 * W, "limit": 7.0}}])


def _spec(case):
    """[(tensor name, shape, spread, mean)]; spread None: 1 / sqrt(columns)."""
    W, V, t = case["width"], case["vocab"], []

    def mat(name, n, k, gain=1.0):
        t.append((name, (n, k), gain / math.sqrt(k), 0.0))

    def vec(name, n, mean=0.0, spread=0.1):
        t.append((name, (n,), spread, mean))

    if case["model"] == "llama":
        hd = W // case["heads"]
        t.append(("model.embed_tokens.weight", (V, W), 1.0, 0.0))
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            for nm, n, k in (("self_attn.q_proj", W, W), ("self_attn.k_proj", case["kv_heads"] * hd, W),
                             ("self_attn.v_proj", case["kv_heads"] * hd, W), ("self_attn.o_proj", W, W),
                             ("mlp.up_proj", case["ff"], W), ("mlp.gate_proj", case["ff"], W), ("mlp.down_proj", W, case["ff"])):
                mat(p + nm + ".weight", n, k, 0.85)
            vec(p + "input_layernorm.weight", W, 1.0)
            vec(p + "post_attention_layernorm.weight", W, 1.0)
        vec("model.norm.weight", W, 1.0)
        return t
    cfg, model = _config(case), case["model"]
    t.append(("embed", (V, W), 1.0, 0.0))

    def unit(p, ff, gain=1.0):
        mat(p + "gate", ff, W, gain)
        mat(p + "up", ff, W, gain)
        mat(p + "down", W, ff)

    def delta(p, m):
        H, dk, dv, C = m["heads"], m["dim"], m["vdim"], m["conv"]
        for nm, n in (("q", m["kv_heads"] * dk), ("k", m["kv_heads"] * dk), ("v", H * dv)):
            mat(p + nm, n, W, 2.0)
            mat(p + nm + ".conv", n, C)
        mat(p + "b", H, W)
        vec(p + "A_log", H, 0.3, 0.5)
        vec(p + "norm", dv, 1.0)
        mat(p + "a1", m["rank_decay"], W)
        mat(p + "a2", H * dk, m["rank_decay"])
        vec(p + "dt_bias", H * dk, -1.5, 0.8)
        mat(p + "g1", m["rank_gate"], W)
        mat(p + "g2", H * dv, m["rank_gate"])
        mat(p + "o", W, H * dv)

    for i, lc in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", lc["mixer"], lc["mlp"]
        if model == "vupitar":
            for nm in ("norm1", "norm2"):
                vec(p + nm, W, 1.0, 0.2)
                vec(p + nm + ".b", W)
                vec(p + nm + ".alpha", 1, 0.7)
        else:
            centre = 0.0 if model == "risalix" else 1.0
            vec(p + "norm1", W, centre)
            if mlp is not None and model != "mabedra":
                vec(p + "norm2", W, centre)
        if model == "risalix":
            H, dk, dv = m["heads"], m["dim"], m["vdim"]
            if lc["type"] == "lightning":
                for nm, n, g in (("q", H * dk, 2.0), ("k", H * dk, 2.0), ("v", H * dv, 2.0), ("g", H * dv, 1.0)):
                    mat(p + "mix." + nm, n, W, g)
                mat(p + "mix.o", W, H * dv)
                vec(p + "mix.norm", H * dv, 1.0)
            elif lc["type"] == "channel_delta":
                delta(p + "mix.", m)
            else:
                mat(p + "mix.q", H * dk, W)
                mat(p + "mix.k", m["kv_heads"] * dk, W)
                vec(p + "mix.q.norm", H * dk, 1.0)
                vec(p + "mix.k.norm", m["kv_heads"] * dk, 1.0)
                mat(p + "mix.g", H, W)
                mat(p + "mix.o", W, H * dk)
            sd = cfg["token_side"]["dim"]
            mat(p + "side.gate", sd, W)
            mat(p + "side.proj", W, sd)
            vec(p + "side.norm", W, 1.0)
        elif model == "mabedra":
            H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for nm, n in (("q", 2 * H * dk), ("k", 2 * G * dk), ("v", G * dv)):
                mat(p + "mix." + nm, n, W, 2.0)
                vec(p + "mix." + nm + ".b", n, 0.0, 0.3)
            vec(p + "mix.q.norm", dk, 1.0, 0.2)
            vec(p + "mix.k.norm", dk, 1.0, 0.2)
            for nm in ("lq1", "lk1", "lq2", "lk2"):
                vec(p + "mix." + nm, dk, 0.0, 0.2)
            mat(p + "mix.o", W, H * dv)
            for nm in ("ls1", "ls2"):
                vec(p + nm, W, 0.5, 0.2)
            for nm in ("canon1", "canon2"):
                mat(p + nm, W, 4, 0.8)
            vec(p + "dwa", i + 2, 0.5, 0.2)
        elif model == "debuzen":
            t.append((p + "shift", (W,), 0.25, 0.5))
            if lc["type"] == "gla":
                H, dk, dv = m["heads"], m["dim"], m["vdim"]
                for nm, n, g in (("q", H * dk, 2.0), ("k", H * dk, 2.0), ("v", H * dv, 1.0), ("g", H * dv, 1.0)):
                    mat(p + "mix." + nm, n, W, g)
                mat(p + "mix.a1", m["rank_decay"], W)
                mat(p + "mix.a2", H * dk, m["rank_decay"], 2.0)
                vec(p + "mix.a2.b", H * dk, 2.0, 1.0)
                vec(p + "mix.norm", dv, 1.0)
                mat(p + "mix.o", W, H * dv)
            else:
                a, q = m["left"], p + "mix.left."
                mat(q + "q", a["heads"] * a["dim"], W, 2.0)
                mat(q + "k", a["kv_heads"] * a["dim"], W, 2.0)
                mat(q + "v", a["kv_heads"] * a["vdim"], W)
                mat(q + "o", W, a["heads"] * a["vdim"])
                if lc["type"] == "parallel":
                    vec(q + "pb", a["heads"], -4.0, 0.5)
                    delta(p + "mix.right.", m["right"])
                else:
                    vec(q + "sink", a["heads"], 0.5, 0.5)
                    r, q = m["right"], p + "mix.right."
                    inner, gn = r["heads"] * r["vdim"], r["groups"] * r["state"]
                    mat(q + "in", 2 * inner + 2 * gn + r["heads"], W, 1.5)
                    mat(q + "conv", inner + 2 * gn, r["conv"])
                    vec(q + "conv.b", inner + 2 * gn, 0.0, 0.2)
                    vec(q + "dt_bias", r["heads"], -0.5, 0.5)
                    vec(q + "A_log", r["heads"], 0.0, 0.5)
                    vec(q + "D", r["heads"], 1.0, 0.3)
                    vec(q + "norm", inner, 1.0)
                    mat(q + "o", W, inner)
        elif model == "gifudra":
            H, dn, dr, dv, rk = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            mat(p + "mix.dq", m["q_rank"], W)
            vec(p + "mix.dq.norm", m["q_rank"], 1.0)
            mat(p + "mix.uq", H * (dn + dr), m["q_rank"], 1.2)
            if "kv_from" not in m:
                mat(p + "mix.dkv", rk + dr, W, 1.2)
                vec(p + "mix.dkv.norm", rk, 1.0)
            mat(p + "mix.uk", H * dn, rk, 1.2)
            mat(p + "mix.uv", H * dv, rk)
            vec(p + "mix.sink", H, 0.5, 1.0)
            mat(p + "mix.g", H * dv, W)
            mat(p + "mix.o", W, H * dv)
            for s in (1, 2):
                vec(p + f"ls{s}", W, 0.7, 0.2)
                vec(p + f"hc{s}.in", 4, 0.25, 0.07)
                vec(p + f"hc{s}.out", 4, 1.0, 0.4)
                t.append((p + f"hc{s}.mix", (4, 4), 0.08, 0.2))
            mat(p + "mlp.up", mlp["ff"], W)
            mat(p + "mlp.down", W, mlp["ff"])
        else:
            a, r = m["left"], m["right"]
            for nm, n in (("q", a["heads"] * a["dim"]), ("k", a["kv_heads"] * a["dim"]), ("v", a["kv_heads"] * a["vdim"])):
                mat(p + "mix.left." + nm, n, W)
                vec(p + "mix.left." + nm + ".b", n, 0.0, 0.3)
            vec(p + "mix.left.q.norm", a["dim"], 1.2, 0.3)
            vec(p + "mix.left.k.norm", a["dim"], 1.2, 0.3)
            mat(p + "mix.left.g", a["heads"], W)
            mat(p + "mix.left.o", W, a["heads"] * a["vdim"])
            vec(p + "mix.left.o.b", W, 0.0, 0.2)
            for nm, n in (("q", r["dim"]), ("k", r["dim"]), ("v", r["vdim"]), ("g", r["vdim"])):
                mat(p + "mix.right." + nm, r["heads"] * n, W)
            mat(p + "mix.right.i", r["heads"], W, 2.0)
            mat(p + "mix.right.f", r["heads"], W, 2.0)
            mat(p + "mix.right.o", W, r["heads"] * r["vdim"])
            vec(p + "mix.right.norm", r["heads"] * r["vdim"], 1.0, 0.2)
            vec(p + "mix.right.i.b", r["heads"], -1.0, 0.5)
            vec(p + "mix.right.f.b", r["heads"], 2.5, 1.0)
        if mlp is not None and model in ("risalix", "debuzen"):
            unit(p + "mlp.", mlp["ff"])
        if model in ("mabedra", "vupitar"):
            if mlp["kind"] == "moe":
                mat(p + "mlp.router", mlp["router"]["experts"], W, 3.0)
                for e in range(mlp["router"]["experts"]):
                    unit(p + f"mlp.e{e}.", mlp["expert"]["ff"], 1.3)
                unit(p + "mlp.shared.", mlp["shared"]["ff"], 1.3)
                if model == "vupitar":
                    mat(p + "mlp.shared.sg", 1, W)
            elif model == "vupitar":
                unit(p + "mlp.", mlp["ff"])
            else:
                mat(p + "mlp.up", mlp["ff"], W)
                mat(p + "mlp.down", W, mlp["ff"])
                vec(p + "mlp.act", 4, 0.3, 0.1)
    if model == "risalix":
        t.append(("side.embed", (V, 256 * len(cfg["layers"])), 1.0, 0.0))
    if model == "debuzen":
        vec("embed.norm", W, 1.0)
    if model == "vupitar":
        vec("final.norm.b", W)
        vec("final.norm.alpha", 1, 0.7)
    vec("final.norm", W, 0.0 if model == "risalix" else 1.0)
    return t


def _weights(case, seed):
    """(name -> float32 tensor on the GPU, successor of every token).  The output projection points from a token's
    embedding to its successor's logit (the token itself where the projection is the embedding table)."""
    g = torch.Generator(device="cuda").manual_seed(1000003 * seed + 17)
    V, W, out = case["vocab"], case["width"], {}
    for name, shape, spread, mean in _spec(case):
        a = torch.randn(shape, generator=g, device="cuda")
        out[name] = a.mul_(spread).add_(mean).bfloat16().float()
    if case["model"] == "gifudra":
        return out, torch.arange(V, device="cuda")
    succ = torch.randperm(V, generator=g, device="cuda")
    llama = case["model"] == "llama"
    head = torch.randn((V, W), generator=g, device="cuda").mul_(0.4)
    head[succ] += out["model.embed_tokens.weight" if llama else "embed"].mul(0.7)
    out["lm_head.weight" if llama else "head"] = head.mul_(W ** -0.5).bfloat16().float()
    return out, succ


def _ids(case, seed):
    return np.random.default_rng(seed).integers(0, case["vocab"], (case["batch"], case["prompt"]))


def _rows(case):
    n = min(ROWS, case["prompt"])
    t = [case["prompt"] - 1 - (i * case["prompt"]) // n for i in range(n)][::-1]
    return [b * case["prompt"] + x for b in range(case["batch"]) for x in t]


# ------------------------------------------------------------------------------------------------------ what is timed
def prepare(case, seed):
    w, _ = _weights(case, seed)
    host = {k: v.cpu().numpy() for k, v in w.items()}
    del w
    n, B = case["prompt"] + case["new"] + 8, case["batch"]
    if case["model"] == "llama":
        args = ModelArgs(dim=case["width"], n_layers=case["layers"], n_heads=case["heads"], n_kv_heads=case["kv_heads"],
                         vocab_size=case["vocab"], max_seq_len=max(256, n), norm_eps=1e-6, max_batch_size=B, dtype=case["dtype"])
        m = Llama(host, args)
    else:
        m = FAMILIES[case["model"]](_config(case), host, max_seq_len=max(256, n), max_batch_size=B, dtype=case["dtype"])
    ids = _ids(case, seed)
    s = {"model": m, "call": case["call"], "llama": case["model"] == "llama", "ids": ids, "prompt": case["prompt"], "new": case["new"],
         "rows": _rows(case)}
    if case["call"] == "step":   # the prefix is in the cache already
        m.forward_f32(ids[:, :-1], 0)
    return s


def run(s):
    m, ids, L, n = s["model"], s["ids"], s["prompt"], s["new"]
    if s["call"] == "step":
        return m.forward_f32(ids[:, -1:], L - 1)
    if s["call"] == "prompt":
        return m.forward_f32(ids, 0) if s["llama"] else m.forward_rows(ids, 0, s["rows"])
    if s["llama"]:   # `generate` counts the whole length and decodes at positions L + 1, L + 2, ... (slot L stays empty)
        tokens = m.generate_all(ids, L + n)
        return {"tokens": tokens, "logits": m.forward_f32(tokens[:4, -1:], L + n)}
    tokens = m.generate_all(ids, n)
    return {"tokens": tokens, "logits": m.forward(tokens[:, -1:], L + n - 1)}


# --------------------------------------------------------------------------------------------------- bytes and operations
def work(case):
    """Weights read once per model pass (a prompt is one pass, every greedy step another; of a mixture of experts what the
    tokens at hand can choose at most), caches and states read once per step, logits written; products, visible query-key
    pairs and state updates as operations."""
    es = 2 if case["dtype"] == "bfloat16" else 4
    B, L, n, W, V = case["batch"], case["prompt"], case["new"], case["width"], case["vocab"]
    llama = case["model"] == "llama"
    dense = experts = 0
    top = of = 1
    cfg = None if llama else _config(case)
    for name, shape, _, _ in _spec(case):
        if len(shape) < 2 or "embed" in name or name.endswith("conv"):
            continue
        if ".mlp.e" in name:
            experts += shape[0] * shape[1]
        else:
            dense += shape[0] * shape[1]
    if experts:
        rc = next(lc["mlp"]["router"] for lc in cfg["layers"] if lc["mlp"] and lc["mlp"]["kind"] == "moe")
        top, of = rc["top"], rc["experts"]
    pair, keep, state = 0, 0, 0          # per pair: operations; per cached token: values; state values (read and written)
    span = 1 << 30
    if llama:
        pair, keep = 4 * W * case["layers"], 2 * case["kv_heads"] * (W // case["heads"]) * case["layers"]
    else:
        for lc in cfg["layers"]:
            for m in (lc["mixer"], lc["mixer"].get("left"), lc["mixer"].get("right")):
                if not m or "heads" not in m:
                    continue
                H, dv = m["heads"], m["vdim"]
                dk = m.get("dim") or m["state"]
                if "q_rank" in m:
                    pair += 2 * H * (dk + m["rot_dim"] + dv)
                    keep += m["kv_rank"] + m["rot_dim"]
                elif "scale" in m:
                    k = 2 if "diff" in m else 1
                    pair += 2 * H * k * (dk + dv)
                    keep += m["kv_heads"] * (k * dk + dv)
                    span = min(span, (m.get("mask") or {}).get("size", 1 << 30))
                else:
                    state += H * dk * dv

    def seen(a, b):                      # visible keys summed over the queries a .. b - 1
        return sum(min(i + 1, span) for i in range(a, b))

    passes = 1 if case["call"] != "greedy" else n + 1
    tokens = B * (1 if case["call"] == "step" else L + n if case["call"] == "greedy" else L)
    rows = B if case["call"] != "prompt" or llama else len(_rows(case))
    read = experts * min(1.0, B * (L if case["call"] == "prompt" else 1) * top / of)
    bytes_ = passes * es * (dense + read + V * W) + tokens * W * es + 4 * rows * V
    first = L - 1 if case["call"] == "step" else 0
    pairs = B * seen(first, L + (n if case["call"] == "greedy" else 0))
    if case["call"] == "greedy":
        bytes_ += es * keep * B * seen(L, L + n) + 8 * state * B * n
    elif case["call"] == "step":
        bytes_ += es * keep * B * L
    else:
        bytes_ += es * keep * B * L + 4 * state * B
    flops = 2.0 * tokens * (dense + experts * top / of) + pairs * pair + 4.0 * tokens * state
    flops += 2.0 * V * W * (rows if case["call"] != "greedy" else B * (n + 1))
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(case):
    """About four times what the listed and drawn cases show against `exact`: fp32 sums 4e-7 (Llama) and 1.8e-6 (layer lists);
    bfloat16 operands 1.4e-3 (one kind of layer) and 4.9e-3 (recurrences and attention side by side)."""
    llama = case["model"] == "llama"
    if case["dtype"] == "float32":
        return {"rel": 2e-6 if llama else 8e-6}
    return {"rel": 6e-3 if llama else 2e-2}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rot(x, pos, dims, base, halves, scaling=None):
    """Rotary positions on the first `dims` entries of the last axis; x [B, L, heads, dim], pos [L]."""
    i = torch.arange(dims // 2, device="cuda", dtype=torch.float64)
    f = base ** (-2.0 * i / dims)
    if scaling:
        ratio = scaling["original"] * f / (2 * math.pi)       # original / wavelength
        s = (ratio - scaling["low"]) / (scaling["high"] - scaling["low"])
        f = torch.where(ratio > scaling["high"], f, torch.where(ratio < scaling["low"], f / scaling["factor"], (1 - s) * f / scaling["factor"] + s * f))
    ang = pos.double()[:, None] * f
    c, s = torch.cos(ang)[None, :, None], torch.sin(ang)[None, :, None]
    y = x.clone()
    if halves:
        a, b = x[..., : dims // 2], x[..., dims // 2: dims]
        y[..., : dims // 2], y[..., dims // 2: dims] = a * c - b * s, b * c + a * s
    else:
        a, b = x[..., 0:dims:2], x[..., 1:dims:2]
        y[..., 0:dims:2], y[..., 1:dims:2] = a * c - b * s, b * c + a * s
    return y


def _attend(q, k, v, scale, mask, sink=None, sigmoid=None):
    """q [B, L, H, d], k [B, T, G, d], v [B, T, G, dv], mask [L, T]; head by head."""
    B, L, H, _ = q.shape
    out = torch.zeros(B, L, H, v.shape[-1], device="cuda", dtype=torch.float64)
    rep = H // k.shape[2]
    for b in range(B):
        for h in range(H):
            z = (q[b, :, h] @ k[b, :, h // rep].T) * scale
            if sigmoid is not None:
                p = torch.where(mask, torch.sigmoid(z + sigmoid[h]), 0.0)
            else:
                z = z.masked_fill(~mask, -math.inf)
                if sink is not None:
                    z = torch.cat([z, sink[h].expand(L, 1)], 1)
                p = torch.softmax(z, -1)[:, : mask.shape[1]]
            out[b, :, h] = p @ v[b, :, h // rep]
    return out


def _causal(L, size=0, keep=0, chunked=False):
    i = torch.arange(L, device="cuda")
    m = i[:, None] >= i[None]
    if size and chunked:
        m = m & (i[:, None] // size == i[None] // size)
    elif size:
        m = m & ((i[:, None] - i[None] < size) | (i[None] < keep))
    return m


def _conv(x, w, bias=None):
    """Causal convolution over time per channel; the last tap multiplies the current token."""
    T = w.shape[1]
    pad = torch.cat([x.new_zeros(x.shape[0], T - 1, x.shape[2]), x], 1)
    y = sum(pad[:, j: j + x.shape[1]] * w[:, j] for j in range(T))
    return y if bias is None else y + bias


def _recur(q, k, v, g=None, beta=None):
    """S <- g S (+ beta (v - S^T k) or v) written with k; o = S^T q, token by token; q, k [B, L, H, dk], v [B, L, H, dv]."""
    B, L, H, dk = q.shape
    S = q.new_zeros(B, H, dk, v.shape[-1])
    out = q.new_zeros(B, L, H, v.shape[-1])
    for t in range(L):
        S = S * g[:, t]
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - torch.einsum("bhkv,bhk->bhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None]
        out[:, t] = torch.einsum("bhkv,bhk->bhv", S, q[:, t])
    return out


def _delta(h, P, m, eps):
    B, L, _ = h.shape
    H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    silu, unit = torch.nn.functional.silu, lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q, k, v = (silu(_conv(h @ P[n].T, P[n + ".conv"])) for n in "qkv")
    q, k = unit(q.view(B, L, G, dk)) * dk ** -0.5, unit(k.view(B, L, G, dk))
    q, k = (x.repeat_interleave(H // G, 2) for x in (q, k))
    dt = torch.nn.functional.softplus(h @ P["a1"].T @ P["a2"].T + P["dt_bias"]).view(B, L, H, dk)
    g = torch.exp(-torch.exp(P["A_log"])[:, None] * dt)
    o = _recur(q, k, v.view(B, L, H, dv), g[..., None], torch.sigmoid(h @ P["b"].T))
    o = _rms(o, eps) * P["norm"] * torch.sigmoid(h @ P["g1"].T @ P["g2"].T).view(B, L, H, dv)
    return o.flatten(2) @ P["o"].T


def _sub(P, prefix):
    return {k[len(prefix):]: v for k, v in P.items() if k.startswith(prefix)}


def _unit(x, P, act):
    return (act(x @ P["gate"].T) * (x @ P["up"].T)) @ P["down"].T


def _exact_llama(case, w, ids, pos):
    W, H, G = case["width"], case["heads"], case["kv_heads"]
    hd = W // H
    B, L = ids.shape
    x = w["model.embed_tokens.weight"][ids]
    mask = pos[:, None] >= pos[None]
    gap = bool((pos[1:] - pos[:-1] > 1).any())     # an empty cache slot that later queries see as a zero row
    if gap:
        hole = int(pos[(pos[1:] - pos[:-1] > 1).nonzero()[0]]) + 1
        mask = torch.cat([mask, (pos > hole)[:, None]], 1)
    for i in range(case["layers"]):
        P = _sub(w, f"model.layers.{i}.")
        h = _rms(x, 1e-6) * P["input_layernorm.weight"]
        q, k, v = ((h @ P[f"self_attn.{n}_proj.weight"].T).view(B, L, -1, hd) for n in "qkv")
        q, k = _rot(q, pos, hd, 10000.0, False), _rot(k, pos, hd, 10000.0, False)
        if gap:
            k, v = (torch.cat([a, a.new_zeros(B, 1, G, hd)], 1) for a in (k, v))
        x = x + _attend(q, k, v, hd ** -0.5, mask).flatten(2) @ P["self_attn.o_proj.weight"].T
        h = _rms(x, 1e-6) * P["post_attention_layernorm.weight"]
        x = x + _unit(h, {"gate": P["mlp.gate_proj.weight"], "up": P["mlp.up_proj.weight"], "down": P["mlp.down_proj.weight"]},
                      torch.nn.functional.silu)
    return lambda r: (_rms(x[r], 1e-6) * w["model.norm.weight"]) @ w["lm_head.weight"].T


def _exact_family(case, w, ids):
    cfg, model, F = _config(case), case["model"], torch.nn.functional
    B, L = ids.shape
    eps = cfg["norm"]["eps"]
    pos = torch.arange(L, device="cuda")
    x = w["embed"][ids]
    W = x.shape[-1]

    def norm(x, name):
        if model == "risalix":
            return _rms(x, eps) * (1.0 + w[name])
        if model == "mabedra":
            return _rms(x - x.mean(-1, keepdim=True), eps) * w[name]
        if model == "debuzen":
            return _rms(x.unflatten(-1, (4, W // 4)), eps).flatten(-2) * w[name]
        if model == "vupitar":
            return torch.tanh(w[name + ".alpha"] * x) * w[name] + w[name + ".b"]
        return _rms(x, eps) * w[name]

    def windowed(h, P, m, halves, bias=False, **kw):
        q, k, v = (h @ P[n].T + (P[n + ".b"] if bias else 0.0) for n in "qkv")
        q, k, v = (a.view(B, L, n, -1) for a, n in ((q, m["heads"]), (k, m["kv_heads"]), (v, m["kv_heads"])))
        if bias:
            q, k = _rms(q, eps) * P["q.norm"], _rms(k, eps) * P["k.norm"]
        q, k = (_rot(a, pos, m["rot"]["dims"], m["rot"]["base"], halves) for a in (q, k))
        if "sigmoid" in kw:
            q, k = _rms(q, eps), _rms(k, eps)
        mk = _causal(L, m["mask"]["size"], m["mask"].get("keep_first", 0), chunked=bias)
        o = _attend(q, k, v, m["scale"], mk, **kw)
        if bias:
            o = o * torch.sigmoid(h @ P["g"].T)[..., None]
        return o.flatten(2) @ P["o"].T + (P["o.b"] if bias else 0.0)

    if model == "debuzen":
        x = norm(x, "embed.norm")
    every = [x]
    X = x[:, :, None].expand(B, L, 4, W) if model == "gifudra" else None
    rows = {}
    for i, lc in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", lc["mixer"], lc["mlp"]
        P, M = _sub(w, p), _sub(w, f"l{i}.mix.")
        if model == "risalix":
            H = m["heads"]
            if lc["type"] == "lightning":
                q, k, v = (F.silu(x @ M[n].T).view(B, L, H, 128) for n in "qkv")
                lam = torch.tensor(m["decay"], device="cuda", dtype=torch.float32).double()[None, None, :, None, None].expand(B, L, H, 1, 1)
                o = _rms(_recur(q, k, v, lam).flatten(2), eps) * M["norm"]
                y = (o * torch.sigmoid(x @ M["g"].T)) @ M["o"].T
            elif lc["type"] == "channel_delta":
                y = _delta(x, M, m, eps)
            else:
                q, k = x @ M["q"].T, x @ M["k"].T
                v = k.view(B, L, m["kv_heads"], -1)
                q, k = (_rms(q, eps) * M["q.norm"]).view(B, L, H, -1), (_rms(k, eps) * M["k.norm"]).view(B, L, m["kv_heads"], -1)
                o = _attend(q, k, v, m["scale"], _causal(L)) * torch.sigmoid(x @ M["g"].T)[..., None]
                y = o.flatten(2) @ M["o"].T
            gelu = lambda z: F.gelu(z, approximate="tanh")  # noqa: E731
            x = x + 0.5 * norm(y, p + "norm1")
            if mlp is not None:
                x = x + 0.5 * norm(_unit(x, _sub(P, "mlp."), gelu), p + "norm2")
            e = w["side.embed"][ids][..., i * 256:(i + 1) * 256]
            x = x + 0.5 * _rms((gelu(x @ P["side.gate"].T) * e) @ P["side.proj"].T, eps) * P["side.norm"]
        elif model == "mabedra":
            h = norm(x, p + "norm1")
            u = h + _conv(h, P["canon1"])
            H, G, dk = m["heads"], m["kv_heads"], m["dim"]
            q, k, v = (u @ M[n].T + M[n + ".b"] for n in "qkv")
            q, k = _rms(q.view(B, L, 2 * H, dk), eps) * M["q.norm"], _rms(k.view(B, L, 2 * G, dk), eps) * M["k.norm"]
            q, k = (_rot(a, pos, dk, m["rot"]["base"], True, m["rot"]["scaling"]) for a in (q, k))
            lam = torch.exp(M["lq1"] @ M["lk1"]) - torch.exp(M["lq2"] @ M["lk2"]) + m["diff"]
            mk, v = _causal(L, m["mask"]["size"]), v.view(B, L, G, -1)
            a1, a2 = (_attend(q[:, :, j::2], k[:, :, j::2], v, m["scale"], mk) for j in (0, 1))
            o = _rms(a1 - lam * a2, eps) * (1.0 - m["diff"])
            y = x + P["ls1"] * (o.flatten(2) @ M["o"].T)
            u, Q = h + _conv(h, P["canon2"]), _sub(P, "mlp.")
            if mlp["kind"] == "moe":
                s, e = torch.topk(torch.sigmoid(u @ Q["router"].T), mlp["router"]["top"])
                f = _unit(u, _sub(Q, "shared."), F.silu)
                for j in range(mlp["router"]["experts"]):
                    b, t, r = (e == j).nonzero(as_tuple=True)
                    f[b, t] += _unit(u[b, t] * s[b, t, r][:, None], _sub(Q, f"e{j}."), F.silu)
            else:
                z, c = u @ Q["up"].T, Q["act"]
                f = (c[0] * _rms(z, eps) + c[1] * _rms(z ** 2, eps) + c[2] * _rms(z ** 3, eps) + c[3]) @ Q["down"].T
            every.append(y + P["ls2"] * f)
            x = sum(a * b for a, b in zip(P["dwa"], every))
        elif model == "debuzen":
            h = norm(x, p + "norm1")
            h = h + (torch.cat([h.new_zeros(B, 1, W), h[:, :-1]], 1) - h) * P["shift"]
            if lc["type"] == "gla":
                H, dk, dv = m["heads"], m["dim"], m["vdim"]
                q, k, v = (h @ M["q"].T).view(B, L, H, dk) * dk ** -0.5, (h @ M["k"].T).view(B, L, H, dk), (h @ M["v"].T).view(B, L, H, dv)
                al = torch.sigmoid(h @ M["a1"].T @ M["a2"].T + M["a2.b"]) ** (1.0 / m["tau"])
                o = _rms(_recur(q, k, v, al.view(B, L, H, dk, 1)), eps) * M["norm"]
                y = (o.flatten(2) * F.silu(h @ M["g"].T)) @ M["o"].T
            elif lc["type"] == "parallel":
                A = _sub(M, "left.")
                y = windowed(h, A, m["left"], False, sigmoid=A["pb"]) + _delta(h, _sub(M, "right."), m["right"], eps)
            else:
                A, R, r = _sub(M, "left."), _sub(M, "right."), m["right"]
                H, dv, N, G = r["heads"], r["vdim"], r["state"], r["groups"]
                z, xbc, dt = (h @ R["in"].T).split([H * dv, H * dv + 2 * G * N, H], -1)
                xs, bm, cm = F.silu(_conv(xbc, R["conv"], R["conv.b"])).split([H * dv, G * N, G * N], -1)
                xs, dt = xs.view(B, L, H, dv), F.softplus(dt + R["dt_bias"])
                bm, cm = (a.view(B, L, G, N).repeat_interleave(H // G, 2) for a in (bm, cm))
                a = torch.exp(-torch.exp(R["A_log"]) * dt)
                o = _recur(cm, bm, dt[..., None] * xs, a[..., None, None]) + R["D"][:, None] * xs
                o = (o.flatten(2) * F.silu(z)).unflatten(-1, (2, H * dv // 2))
                y = windowed(h, A, m["left"], True, sink=A["sink"]) + (_rms(o, eps).flatten(2) * R["norm"]) @ R["o"].T
            x = x + y
            x = x + _unit(norm(x, p + "norm2"), _sub(P, "mlp."), F.silu)
        elif model == "gifudra":
            def mix(X, y, s):
                y = y * P[f"ls{s}"]
                return torch.einsum("blsw,st->bltw", X, P[f"hc{s}.mix"]) + y[:, :, None] * P[f"hc{s}.out"][:, None]

            def read(X, s):
                return norm(torch.einsum("blsw,s->blw", X, P[f"hc{s}.in"]), p + f"norm{s}")

            h = read(X, 1)
            H, dn, dr, rk = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
            q = ((_rms(h @ M["dq"].T, eps) * M["dq.norm"]) @ M["uq"].T).view(B, L, H, dn + dr)
            q = torch.cat([q[..., :dn], _rot(q[..., dn:], pos, dr, m["rot"]["base"], True)], -1)
            if "kv_from" not in m:
                c = h @ M["dkv"].T
                rows[i] = _rms(c[..., :rk], eps) * M["dkv.norm"], _rot(c[..., None, rk:], pos, dr, m["rot"]["base"], True)
            c, kr = rows[m.get("kv_from", i)]
            k = torch.cat([(c @ M["uk"].T).view(B, L, H, dn), kr.expand(B, L, H, dr)], -1)
            o = _attend(q, k, (c @ M["uv"].T).view(B, L, H, -1), m["scale"], _causal(L), sink=M["sink"]).flatten(2)
            X = mix(X, (o * torch.sigmoid(h @ M["g"].T)) @ M["o"].T, 1)
            X = mix(X, (torch.relu(read(X, 2) @ P["mlp.up"].T) ** 2) @ P["mlp.down"].T, 2)
            x = X.sum(2)
        else:
            h, A, R, r = norm(x, p + "norm1"), _sub(M, "left."), _sub(M, "right."), m["right"]
            y = windowed(h, A, m["left"], True, bias=True)
            H, dk, dv = r["heads"], r["dim"], r["vdim"]
            q, k, v = (h @ R["q"].T).view(B, L, H, dk) * dk ** -0.5, (h @ R["k"].T).view(B, L, H, dk), (h @ R["v"].T).view(B, L, H, dv)
            cap = lambda z: r["gate_cap"] * torch.tanh(z / r["gate_cap"])  # noqa: E731
            gi, gf = cap(h @ R["i"].T + R["i.b"]), F.logsigmoid(cap(h @ R["f"].T + R["f.b"]))
            mm, n, S, o = gi.new_zeros(B, H), gi.new_zeros(B, H, dk), gi.new_zeros(B, H, dk, dv), gi.new_zeros(B, L, H, dv)
            for t in range(L):
                m2 = torch.maximum(gf[:, t] + mm, gi[:, t])
                a, b = torch.exp(gf[:, t] + mm - m2)[..., None], torch.exp(gi[:, t] - m2)[..., None]
                n, mm = a * n + b * k[:, t], m2
                S = a[..., None] * S + (b * k[:, t])[..., None] * v[:, t, :, None]
                den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-mm)) + 1e-6
                o[:, t] = torch.einsum("bhkv,bhk->bhv", S, q[:, t]) / den[..., None]
            y = y + (_rms(o, eps).flatten(2) * R["norm"] * torch.sigmoid(h @ R["g"].T)) @ R["o"].T
            u, Q = norm(x, p + "norm2"), _sub(P, "mlp.")
            if mlp["kind"] == "moe":
                s, e = torch.topk(torch.softmax(u @ Q["router"].T, -1), mlp["router"]["top"])
                s = s / (s.sum(-1, keepdim=True) + 1e-20)
                f = torch.sigmoid(u @ Q["shared.sg"].T) * _unit(u, _sub(Q, "shared."), F.silu)
                for j in range(mlp["router"]["experts"]):
                    b, t, c = (e == j).nonzero(as_tuple=True)
                    f[b, t] += s[b, t, c][:, None] * _unit(u[b, t], _sub(Q, f"e{j}."), F.silu)
            else:
                g, c = torch.clamp(u @ Q["gate"].T, max=7.0), torch.clamp(u @ Q["up"].T, -7.0, 7.0)
                f = (g * torch.sigmoid(1.702 * g) * (c + 1.0)) @ Q["down"].T
            x = x + y + f

    def logits(r):
        z = norm(x[r], "final.norm") @ (w["embed"] if model == "gifudra" else w["head"]).T
        if model == "gifudra":
            z = z * cfg["logit_scale"]
        return 30.0 * torch.tanh(z / 30.0) if model == "debuzen" else z

    return logits


def exact(case, seed):
    w, succ = _weights(case, seed)
    ids = torch.from_numpy(_ids(case, seed)).cuda()
    B, L, n = case["batch"], case["prompt"], case["new"]
    llama = case["model"] == "llama"
    keep = 4 if llama else B
    if case["call"] == "greedy":   # feed the successors; that they are what the logits choose is read off below
        seq = [ids[:, -1]]
        for _ in range(n):
            seq.append(succ[seq[-1]])
        ids = torch.cat([ids, torch.stack(seq[1:], 1)], 1)
    N = ids.shape[1]
    pos = torch.arange(N, device="cuda")
    if llama and case["call"] == "greedy":
        pos = torch.cat([pos[:L], pos[L:] + 1])
    w = {k: v.double() for k, v in w.items()}
    parts = []
    step = max(1, 20000 // N)      # sequences at a time
    for b in range(0, B, step):
        part = ids[b:b + step]
        of = _exact_llama(case, w, part, pos) if llama else _exact_family(case, w, part)
        if case["call"] == "prompt" and not llama:
            parts.append(of((slice(None), [r for r in _rows(case) if r < L])).flatten(0, 1))
        elif case["call"] == "greedy":
            parts.append((torch.stack([of((slice(None), t)).argmax(-1) for t in range(L - 1, N - 1)], 1), of((slice(None), -1))))
        else:
            parts.append(of((slice(None), -1)))
    if case["call"] == "greedy":
        return {"tokens": torch.cat([p[0] for p in parts]).cpu().numpy(), "logits": torch.cat([p[1] for p in parts])[:keep].cpu().numpy()}
    return torch.cat(parts).cpu().numpy()
