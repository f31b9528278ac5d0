"""The work that users of this framework have it do, as cases that can be timed and compared.

Two families: pipeline stages of litGPT-style transformers (one token of one sample, or a whole prompt, per call) and the
hybrid models (one mixing layer over a step's packed prompts, or a whole one-token step of several streams).  Weights and
inputs are random, made on the GPU from the seed; sizes are those of the registered Llama-3-8B, TinyLlama-1.1B and
Mixtral-8x7B configurations and of the side benchmark's hybrid models.

``listed()`` names twelve cases, ``draw(rng)`` makes more of the same ranges, ``prepare`` builds what a program holds before the
call, ``run`` is one call, ``work`` what it cannot do without, ``exact`` the same in 64 bits with plain torch, ``tolerance`` what
another correct implementation at the same precision may differ by.
"""
import math

import torch
import torch.nn.functional as F

DEV = "cuda"
BF = torch.bfloat16

#: width, heads, key/value groups, head size, feed-forward, vocabulary, rotary base, layer norm's epsilon
MODELS = {
    "Llama-3-8B": (4096, 32, 8, 128, 14336, 128256, 500000, 1e-5),
    "tiny-llama-1.1b": (2048, 32, 4, 64, 5632, 32000, 10000, 1e-5),
    "Mixtral-8x7B-v0.1": (4096, 32, 8, 128, 14336, 32000, 1000000, 1e-5),
}
EXPERTS, TOP = 8, 2


# =============================================================================================
# the cases
# =============================================================================================
def listed():
    return [
        # the smallest call: one token through the five layers that a node of a four-node TinyLlama ring owns
        dict(name="decode tiny", path="decode", model="tiny-llama-1.1b", role="secondary", layers=5, context=300, weights="bf16"),
        # a whole call on a starter node: embedding, its layers, final norm and output head, at a long context; returns logits
        dict(name="decode 8b logits", path="decode", model="Llama-3-8B", role="starter", layers=2, context=1803, weights="bf16"),
        # one token through a node of an eight-node ring that serves block-scaled fp8 weights, at 2048 positions
        dict(name="decode 8b fp8", path="decode", model="Llama-3-8B", role="secondary", layers=4, context=2047, weights="fp8"),
        # the headline benchmark's prompt length on a node's layers
        dict(name="prompt 8b", path="prompt", model="Llama-3-8B", layers=2, tokens=448, weights="bf16"),
        # the fp8 configuration's prompt length
        dict(name="prompt 8b fp8", path="prompt", model="Llama-3-8B", layers=2, tokens=1024, weights="fp8"),
        # the routed feed-forward of a mixture-of-experts model over a prompt of odd length (a stage that starts at it)
        dict(name="prompt mixture", path="mixture", model="Mixtral-8x7B-v0.1", tokens=997),
        # rotation, cache write and causal attention of a long prompt
        dict(name="attention 8b", path="attention", heads=32, groups=8, head_size=128, tokens=4096),
        # hybrid models: the gated delta rule over one long prompt
        dict(name="delta prompt", path="mixer", design="Badapel", kind="channel_delta", width=2048, lengths="2048", start=0),
        # gated linear attention over prompts of unequal lengths packed into one step
        dict(name="gla prompts", path="mixer", design="Badapel", kind="gla", width=2048, lengths="1282,700,65,1", start=0),
        # grouped-query attention with a cap on the scores and learned sinks over one prompt
        dict(name="grouped attention prompt", path="mixer", design="Zudovik", kind="attention", width=2048, lengths="2048", start=0),
        # windowed latent attention over unequal prompts
        dict(name="latent prompts", path="mixer", design="Ratesun", kind="latent_attention", width=2048, lengths="1411,501,136", start=0),
        # a whole call: one token for each of eight streams through a four-layer hybrid model; returns logits
        dict(name="hybrid step", path="step", width=2048, streams=8, context=2048),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lengths(rng, most):
    """One to five sequences that bring up to ``most`` tokens together."""
    total, parts = _log(rng, 64, most), rng.choice((1, 1, 2, 3, 5))
    cuts = sorted(rng.randrange(1, total) for _ in range(parts - 1))
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]) if b > a)


def draw(rng):
    path = rng.choice(("decode", "decode", "prompt", "prompt", "mixture", "attention", "mixer", "mixer", "mixer", "mixer", "step"))
    if path == "decode":
        model = rng.choice(("Llama-3-8B", "tiny-llama-1.1b"))
        return dict(path=path, model=model, role=rng.choice(("starter", "secondary")), layers=rng.randint(1, 3 if "8B" in model else 8),
                    context=_log(rng, 16, 8000 if "8B" in model else 2040), weights=rng.choice(("bf16", "bf16", "fp8")))
    if path == "prompt":
        model = rng.choice(("Llama-3-8B", "tiny-llama-1.1b"))
        return dict(path=path, model=model, layers=rng.randint(1, 2 if "8B" in model else 4),
                    tokens=_log(rng, 33, 1024 if "8B" in model else 2040), weights=rng.choice(("bf16", "bf16", "fp8")))
    if path == "mixture":
        return dict(path=path, model="Mixtral-8x7B-v0.1", tokens=_log(rng, 33, 997))
    if path == "attention":
        heads, groups, size = rng.choice(((32, 8, 128), (32, 4, 64), (32, 32, 128)))
        return dict(path=path, heads=heads, groups=groups, head_size=size, tokens=_log(rng, 33, 4096))
    if path == "mixer":
        design, kind = rng.choice((("Badapel", "channel_delta"), ("Badapel", "gla"), ("Zudovik", "attention"), ("Labepel", "attention"),
                                   ("Vudelix", "attention"), ("Dufelix", "attention"), ("Ratesun", "latent_attention"),
                                   ("Badapel", "latent_attention"), ("Dufelix", "latent_attention")))
        return dict(path=path, design=design, kind=kind, width=rng.choice((1024, 2048)), lengths=_lengths(rng, 2048),
                    start=rng.choice((0, 0, rng.randrange(1, 500))))
    return dict(path="step", width=rng.choice((1024, 2048)), streams=rng.randint(1, 8), context=_log(rng, 16, 2048))


# =============================================================================================
# inputs and weights, from the seed alone
# =============================================================================================
class _Gen:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(seed * 7919 + 17)

    def n(self, *shape, std=1.0, mean=0.0):
        return (torch.randn(*shape, generator=self.g, device=DEV) * std + mean).to(BF)

    def mat(self, rows, cols):
        return self.n(rows, cols, std=cols ** -0.5)

    def ids(self, n, below):
        return torch.randint(0, below, (n,), generator=self.g, device=DEV)


def _stage_weights(case, gen):
    """A stage's tensors under their checkpoint names."""
    C, H, G, hs, I, vocab, _, _ = MODELS[case["model"]]
    w = {}
    for i in range(case.get("layers", 1)):
        p = "transformer.h.%d." % i
        if case["path"] != "mixture":
            w[p + "norm_1.weight"] = gen.n(C, std=0.1, mean=1.0)
            w[p + "attn.attn.weight"] = gen.mat((H + 2 * G) * hs, C)
            w[p + "attn.proj.weight"] = gen.mat(C, H * hs)
        w[p + "norm_2.weight"] = gen.n(C, std=0.1, mean=1.0)
        if case["path"] == "mixture":
            w[p + "mlp.gate.weight"] = gen.mat(EXPERTS, C)
        for e in (["mlp.experts.%d." % j for j in range(EXPERTS)] if case["path"] == "mixture" else ["mlp."]):
            w[p + e + "fc_1.weight"], w[p + e + "fc_2.weight"], w[p + e + "proj.weight"] = gen.mat(I, C), gen.mat(I, C), gen.mat(C, I)
    if case.get("role") == "starter":
        w["transformer.wte.weight"], w["transformer.ln_f.weight"] = gen.n(vocab, C), gen.n(C, std=0.1, mean=1.0)
        w["lm_head.weight"] = gen.mat(vocab, C)
    return w


def _stage_inputs(case, gen):
    C, H, G, hs, _, vocab, _, _ = MODELS[case["model"]]
    if case["path"] != "decode":
        return gen.n(1, case["tokens"], C), None
    x = gen.ids(1, vocab).view(1, 1).cpu() if case["role"] == "starter" else gen.n(1, 1, C)
    return x, gen.n(case["layers"], 2, G, case["context"], hs)  # the keys and values of the tokens before this one


def _hybrid_config(design, kind, width):
    """The layer of the side benchmark's model of that design, without its feed-forward."""
    h = width // 128
    att = dict(heads=h, kv_heads=max(1, h // 4), dim=128, vdim=128, scale=128 ** -0.5)
    lat = dict(heads=h, dim=128, rot_dim=64, vdim=128, kv_rank=512, q_rank=min(1536, width), scale=192 ** -0.5, rot=dict(dims=64, base=10000.0))
    if kind == "attention":
        m = dict(att, **{"Vudelix": dict(mask=dict(size=1024), rot=dict(dims=128, base=500000.0)), "Labepel": dict(mask=dict(size=1024)),
                         "Zudovik": dict(softcap=50.0, rot=dict(dims=64, base=500000.0)), "Dufelix": dict(rot=dict(dims=64, base=500000.0))}[design])
    elif kind == "latent_attention":
        m = dict(lat, mask=dict(size=1024)) if design == "Ratesun" else lat
    elif kind == "gla":
        m = dict(heads=h, dim=64, vdim=128, tau=16.0)
    else:
        m = dict(heads=h, kv_heads=max(1, h // 2), dim=128, vdim=128, conv=4)
    return m


def _mixer_weights(design, kind, m, C, gen):
    """A mixing layer's tensors under their checkpoint names; its low-rank projections have rank 16."""
    h, g = m["heads"], m.get("kv_heads", m["heads"])
    if kind == "attention":
        D, V = m["dim"], m["vdim"]
        w = dict(q=gen.mat(h * D, C), k=gen.mat(g * D, C), v=gen.mat(g * V, C), o=gen.mat(C, h * V),
                 g=gen.mat(h * V if design == "Labepel" else h, C))
        if design in ("Labepel", "Zudovik"):
            w.update({"q.b": gen.n(h * D, std=0.5), "k.b": gen.n(g * D, std=0.5), "v.b": gen.n(g * V, std=0.5)})
            full = design == "Zudovik"
            w.update({"q.norm": gen.n(h * D if full else D, std=0.1, mean=1.0), "k.norm": gen.n(g * D if full else D, std=0.1, mean=1.0)})
        if design == "Zudovik":
            w["sink"] = gen.n(h, std=0.5)
        return w
    if kind == "latent_attention":
        D, R, V, L, Q = m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
        w = {"dq": gen.mat(Q, C), "dq.norm": gen.n(Q, std=0.1, mean=1.0), "uq": gen.mat(h * (D + R), Q), "dkv": gen.mat(L + R, C),
             "dkv.norm": gen.n(L, std=0.1, mean=1.0), "uk": gen.mat(h * D, L), "uv": gen.mat(h * V, L), "o": gen.mat(C, h * V)}
        if design == "Badapel":
            w["g"] = gen.mat(h * V, C)
        if design == "Dufelix":
            w["sink"] = gen.n(h, std=0.5)
        return w
    D, V = m["dim"], m["vdim"]
    if kind == "gla":
        return {"q": gen.mat(h * D, C), "k": gen.mat(h * D, C), "v": gen.mat(h * V, C), "g": gen.mat(h * V, C), "o": gen.mat(C, h * V),
                "norm": gen.n(V, std=0.1, mean=1.0), "a1": gen.mat(16, C), "a2": gen.mat(h * D, 16), "a2.b": gen.n(h * D, std=0.5)}
    return {"q": gen.mat(g * D, C), "q.conv": gen.n(g * D, 4, std=0.5), "k": gen.mat(g * D, C), "k.conv": gen.n(g * D, 4, std=0.5),
            "v": gen.mat(h * V, C), "v.conv": gen.n(h * V, 4, std=0.5), "b": gen.mat(h, C), "A_log": gen.n(h, std=0.5),
            "norm": gen.n(V, std=0.1, mean=1.0), "a1": gen.mat(16, C), "a2": gen.mat(h * D, 16), "dt_bias": gen.n(h * D, std=0.5),
            "g1": gen.mat(16, C), "g2": gen.mat(h * V, 16), "o": gen.mat(C, h * V)}


def _mixer_state(kind, m, slots, seq, start, gen):
    """What a slot holds after ``start`` tokens: cache rows, or the recurrent state and the convolution's last inputs."""
    h, g = m["heads"], m.get("kv_heads", m["heads"])
    if kind in ("attention", "latent_attention"):
        row = g * (m["dim"] + m["vdim"]) if kind == "attention" else m["kv_rank"] + m["rot_dim"]
        c = torch.zeros(slots, seq, row, device=DEV, dtype=BF)
        c[:, :start] = gen.n(slots, start, row)
        return {"cache": c}
    st = {"state": gen.n(slots, h, m["dim"], m["vdim"], std=0.2 if start else 0.0).float()}
    if kind == "channel_delta":
        st["conv"] = gen.n(slots, 3, 2 * g * m["dim"] + h * m["vdim"], std=1.0 if start else 0.0)
    return st


STEP_KINDS = ("latent_attention", "channel_delta", "gla", "latent_attention")
STEP_VOCAB = 32000


def _step_weights(case, gen):
    """The four-layer hybrid model's tensors under their checkpoint names, and the state of its streams."""
    C, w, states = case["width"], {}, []
    w["embed"], w["final.norm"], w["final.norm.b"] = gen.n(STEP_VOCAB, C), gen.n(C, std=0.1, mean=1.0), gen.n(C, std=0.1)
    for i, kind in enumerate(STEP_KINDS):
        m = _hybrid_config("Badapel", kind, C)
        for k, t in _mixer_weights("Badapel", kind, m, C, gen).items():
            w["l%d.mix.%s" % (i, k)] = t
        for k in ("norm1", "norm1b", "norm2", "norm2b"):
            w["l%d.%s" % (i, k)], w["l%d.%s.b" % (i, k)] = gen.n(C, std=0.1, mean=1.0), gen.n(C, std=0.1)
        w["l%d.mlp.up" % i], w["l%d.mlp.down" % i] = gen.mat(4 * C, C), gen.mat(C, 4 * C)
        states.append(_mixer_state(kind, m, case["streams"], case["context"] + 8, case["context"], gen))
    return w, states


# =============================================================================================
# what a program holds before the call, and the call
# =============================================================================================
def prepare(case, seed):
    gen = _Gen(seed)
    path = case["path"]
    if path in ("decode", "prompt", "mixture"):
        return _prepare_stage(case, gen)
    if path == "attention":
        from mdi_llm_b200 import ops
        from mdi_llm_b200.models.gpt import build_rope_cache

        ops.require()
        H, G, hs, T = case["heads"], case["groups"], case["head_size"], case["tokens"]
        cos, sin = build_rope_cache(T + 8, hs, device=torch.device(DEV))
        kv = torch.zeros(1, 2, G, T + 8, hs, device=DEV, dtype=BF)
        qkv = gen.n(T, (H + 2 * G) * hs)
        args = dict(n_head=H, n_groups=G, head_size=hs, rope_n_elem=hs)
        return dict(path=path, call=lambda: ops.attn_prefill(qkv, cos.float().contiguous(), sin.float().contiguous(), kv, 0, **args), kv=kv)
    from mdi_llm_b200.models.config import HybridConfig
    from mdi_llm_b200.models.hybrid import HybridLM
    from mdi_llm_b200.ops.hybrid import BatchPlan

    if path == "mixer":
        design, kind, C, start = case["design"], case["kind"], case["width"], case["start"]
        lengths = [int(n) for n in case["lengths"].split(",")]
        m = _hybrid_config(design, kind, C)
        raw = dict(architecture=design, vocab=64, width=C, layers=[dict(type=kind, mixer=m)], norm=dict(eps=1e-6))
        if design == "Labepel":
            raw["max_positions"] = 4096
        if design == "Ratesun":
            raw.update(embedding=dict(bigram=dict(buckets=16, mul_prev=3, mul_cur=5)), canon=dict(taps=4))
        model = HybridLM(HybridConfig.from_dict(raw), {"l0.mix.a1": 16, "l0.mix.g1": 16}).eval()
        w = _mixer_weights(design, kind, m, C, gen)
        small = {n: gen.n(*p.shape) if p.dim() else gen.n(1) for n, p in model.tensor_map().items() if not n.startswith("l0.mix.")}
        model.load_tensors({**small, **{"l0.mix." + k: t for k, t in w.items()}}, DEV, BF)
        x = gen.n(sum(lengths), C)
        first = _mixer_state(kind, m, len(lengths), start + max(lengths) + 8, start, gen)
        state = model.new_pool(len(lengths), start + max(lengths) + 8).runs[0]
        for k, t in first.items():
            state[k].copy_(t)
        plan = BatchPlan.make(lengths, list(range(len(lengths))), [start] * len(lengths), torch.device(DEV))
        moved = {k: t for k, t in first.items() if k != "cache"}  # what a pass carries forward
        return dict(path=path, mixer=model.blocks[0].mix, x=x, plan=plan, state=state, first=moved)
    from mdi_llm_b200.parallel.hybrid_runner import HybridRunner

    layers = [dict(type=k, mixer=_hybrid_config("Badapel", k, case["width"]), mlp=dict(kind="dense", ff=4 * case["width"])) for k in STEP_KINDS]
    raw = dict(architecture="Badapel", vocab=STEP_VOCAB, width=case["width"], layers=layers, norm=dict(eps=1e-6), logit_softcap=30.0)
    w, states = _step_weights(case, gen)
    ranks = {n: 16 for n in w if n.endswith((".a1", ".g1"))}
    model = HybridLM(HybridConfig.from_dict(raw), ranks).load_tensors(w, DEV, BF)
    n = case["streams"]
    runner = HybridRunner(model, case["context"] + 8, n_slots=n)
    ids = gen.ids(n, STEP_VOCAB).tolist()
    entries = [(i, [ids[i]]) for i in range(n)]
    runner.step(entries)  # the first steps of a batch size warm up and capture, as they do in a serving loop
    runner.step(entries)
    for run_, st in zip(runner.pool.runs, states):
        for k, t in st.items():
            run_[k].copy_(t)
    return dict(path=path, runner=runner, entries=entries, context=case["context"])


def _prepare_stage(case, gen):
    from mdi_llm_b200.models.config import Config
    from mdi_llm_b200.models.stage import build_stage
    from mdi_llm_b200.parallel.engine import FusedStage, FusedStageRunner

    path, layers = case["path"], case.get("layers", 1)
    w = _stage_weights(case, gen)
    x, past = _stage_inputs(case, gen)
    seq = (case["context"] if path == "decode" else case["tokens"]) + 8
    cfg = Config.from_name(case["model"], n_layer=layers)
    role = case.get("role", "secondary")
    more = dict(first_parts="mlp") if path == "mixture" else {}
    stage = build_stage(cfg, role if role == "starter" else role + ":0", layers, meta=True, **more)
    stage.load_weights(w)
    s = dict(path=path, x=x)
    if path == "decode" and case["weights"] == "bf16":
        s["runner"] = FusedStageRunner(stage, max_seq_length=seq, n_slots=1)
        s["runner"].begin_sample(0)
        fused = s["runner"].stage
    else:
        fused = FusedStage(stage, n_slots=1, max_seq_length=seq, weight_dtype=case.get("weights", "bf16"))
    s.update(stage=fused, kv=fused.kv, starter=role == "starter")
    if path == "decode":
        fused.kv[:, 0, :, :, : case["context"]] = past
        s.update(slot_pos=case["context"], pos=torch.tensor([case["context"]]))
        run(s)  # the first call captures the step, as it does in a serving loop
    else:
        s["pos"] = torch.arange(case["tokens"], device=DEV)
    return s


def run(s):
    path = s["path"]
    if path == "decode":
        return _run_decode(s)
    if path in ("prompt", "mixture"):
        return dict(y=s["stage"].prefill(s["x"], s["pos"], 0), **({"kv": s["kv"]} if path == "prompt" else {}))
    if path == "attention":
        return dict(y=s["call"](), kv=s["kv"])
    if path == "mixer":
        s["plan"].shared.clear()  # as the model does when a step starts
        for k, t in s["first"].items():
            s["state"][k].copy_(t)
        with torch.inference_mode():
            y = s["mixer"](s["x"], s["plan"], s["state"])
        return dict(y=y, state=dict(s["state"]))
    r = s["runner"]
    for slot in r.pool.length:  # the same step again: every stream back at its position
        r.pool.length[slot] = s["context"]
    return dict(logits=r.step(s["entries"]), state=[dict(st) for st in r.pool.runs])


def _run_decode(s):
    if "runner" in s:
        y = s["runner"].forward(0, s["x"], s["pos"])
        return dict(logits=s["runner"].head(y), hidden=y, kv=s["kv"]) if s["starter"] else dict(hidden=y, kv=s["kv"])
    st = s["stage"]  # fp8 weights: the stage itself, step by step
    if s["starter"]:
        st.set_ctx(0, s["slot_pos"], token=int(s["x"]))
        st.graph("token", lambda: (st.enqueue_embed(from_tokens=False), st.enqueue_blocks(None, False))).launch()
        st.hidden_in[0].copy_(st.out_local[0])
        st.graph("head", lambda: st.enqueue_head(wait=False, stats=False)).launch()
        return dict(logits=st.logits.view(1, 1, -1).clone(), hidden=st.out_local[0].view(1, 1, -1).clone(), kv=s["kv"])
    st.hidden_in[0].copy_(s["x"].view(-1))
    st.set_ctx(0, s["slot_pos"])
    st.graph("token", lambda: st.enqueue_blocks(None, False)).launch()
    return dict(hidden=st.out_local[0].view(1, 1, -1).clone(), kv=s["kv"])


# =============================================================================================
# what a call cannot do without
# =============================================================================================
def work(case):
    path = case["path"]
    if path in ("decode", "prompt", "mixture"):
        C, H, G, hs, I, vocab, _, _ = MODELS[case["model"]]
        per = 1 if case.get("weights") == "fp8" else 2
        n, L = (1 if path == "decode" else case["tokens"]), case.get("layers", 1)
        attn = ((H + 2 * G) * hs + H * hs) * C
        if path == "mixture":
            used = min(EXPERTS, n * TOP)
            return dict(bytes=2.0 * (used * 3 * I * C + EXPERTS * C) + 4.0 * n * C, flops=2.0 * n * TOP * 3 * I * C)
        mats = L * (attn + 3 * I * C)
        seen = case["context"] + 1 if path == "decode" else (n + 1) / 2
        keys = L * (2 * 2 * G * hs * (case["context"] + 1 if path == "decode" else n))
        head = vocab * C if case.get("role") == "starter" else 0
        return dict(bytes=float(per * (mats + head) + keys + 4.0 * n * C + (4 * vocab if head else 0)),
                    flops=2.0 * n * (mats + head) + 4.0 * L * H * hs * n * seen)
    if path == "attention":
        H, G, hs, T = case["heads"], case["groups"], case["head_size"], case["tokens"]
        return dict(bytes=2.0 * T * hs * (2 * H + 4 * G), flops=2.0 * H * hs * T * (T + 1))
    if path == "mixer":
        lengths, C, kind, start = [int(x) for x in case["lengths"].split(",")], case["width"], case["kind"], case["start"]
        m, n = _hybrid_config(case["design"], kind, C), sum(int(x) for x in case["lengths"].split(","))
        mats = _mixer_mats(case["design"], kind, m, C)
        b, f = 2.0 * mats + 4.0 * n * C, 2.0 * n * mats
        h, g = m["heads"], m.get("kv_heads", m["heads"])
        if kind in ("attention", "latent_attention"):
            W = (m.get("mask") or {}).get("size", 0)
            row = g * (m["dim"] + m["vdim"]) if kind == "attention" else m["kv_rank"] + m["rot_dim"]
            first = (lambda p: p // W * W) if case["design"] == "Labepel" else (lambda p: max(0, p - W + 1) if W else 0)
            pairs = sum(start + i + 1 - first(start + i) for ln in lengths for i in range(ln))
            dk = m["dim"] + m.get("rot_dim", 0)
            b += 2.0 * row * sum(ln + start + ln - first(start) for ln in lengths)
            return dict(bytes=b, flops=f + 2.0 * h * pairs * (dk + m["vdim"]))
        b += 8.0 * len(lengths) * h * m["dim"] * m["vdim"]
        return dict(bytes=b, flops=f + (8.0 if kind == "channel_delta" else 5.0) * n * h * m["dim"] * m["vdim"])
    C, n, ctx, b, f = case["width"], case["streams"], case["context"] + 1, 2.0 * STEP_VOCAB * case["width"], 2.0 * case["streams"] * STEP_VOCAB * case["width"]
    for kind in STEP_KINDS:
        m = _hybrid_config("Badapel", kind, C)
        mats = _mixer_mats("Badapel", kind, m, C) + 8 * C * C
        b, f = b + 2.0 * mats, f + 2.0 * n * mats
        if kind == "latent_attention":
            row = m["kv_rank"] + m["rot_dim"]
            b, f = b + 2.0 * n * ctx * row, f + 2.0 * n * ctx * m["heads"] * (row + m["kv_rank"])
        else:
            b, f = b + 8.0 * n * m["heads"] * m["dim"] * m["vdim"], f + 8.0 * n * m["heads"] * m["dim"] * m["vdim"]
    return dict(bytes=b + 4.0 * n * STEP_VOCAB, flops=f)


def _mixer_mats(design, kind, m, C):
    h, g = m["heads"], m.get("kv_heads", m["heads"])
    D, V = m["dim"], m["vdim"]
    if kind == "attention":
        return C * (h * D + g * (D + V) + h * V + (h * V if design == "Labepel" else h))
    if kind == "latent_attention":
        L, R, Q = m["kv_rank"], m["rot_dim"], m["q_rank"]
        return C * (Q + L + R + h * V + (h * V if design == "Badapel" else 0)) + Q * h * (D + R) + L * h * (D + V)
    if kind == "gla":
        return C * (2 * h * D + 3 * h * V + 16) + 16 * h * D
    return C * (2 * g * D + 2 * h * V + h + 32) + 16 * h * (D + V)


def tolerance(case):
    """Every path keeps its activations in bf16 and sums in 32 bits: about four times what a run differs from 64 bits (0.003 for
    rotation and attention, 0.005 for a mixing layer, 0.006 for two layers of a prompt, 0.01 for a token through several layers,
    0.02 where two nearly equal experts change places, 0.03 with activations rounded to fp8), and at most 0.03."""
    if case["path"] == "attention":
        return {"rel": 0.012, "max": 0.2}
    if case["path"] == "mixer":
        return {"rel": 0.02, "max": 0.3}
    if case["path"] == "prompt" and case["weights"] == "bf16":
        return {"rel": 0.024, "max": 0.3}
    return {"rel": 0.03, "max": 0.9 if case["path"] == "mixture" else 0.4}


# =============================================================================================
# the same in 64 bits
# =============================================================================================
def exact(case, seed):
    gen = _Gen(seed)
    with torch.no_grad():
        if case["path"] in ("decode", "prompt", "mixture"):
            return _exact_stage(case, gen)
        if case["path"] == "attention":
            H, G, hs, T = case["heads"], case["groups"], case["head_size"], case["tokens"]
            qkv = gen.n(T, (H + 2 * G) * hs).double()
            kv = torch.zeros(1, 2, G, T + 8, hs, device=DEV, dtype=torch.float64)
            return dict(y=_causal(qkv, kv[0], 0, H, G, hs, 10000), kv=kv)
        if case["path"] == "mixer":
            design, kind, C, start = case["design"], case["kind"], case["width"], case["start"]
            lengths = [int(n) for n in case["lengths"].split(",")]
            m = _hybrid_config(design, kind, C)
            w = {k: t.double() for k, t in _mixer_weights(design, kind, m, C, gen).items()}
            for shape in _small_shapes(design, C):
                gen.n(*shape)
            x = gen.n(sum(lengths), C).double()
            st = {k: t.double() for k, t in _mixer_state(kind, m, len(lengths), start + max(lengths) + 8, start, gen).items()}
            y, r = torch.empty(sum(lengths), C, device=DEV, dtype=torch.float64), 0
            for i, n in enumerate(lengths):
                y[r:r + n] = _mix(design, kind, m, w, x[r:r + n], {k: t[i] for k, t in st.items()}, start)
                r += n
            return dict(y=y, state=st)
        return _exact_step(case, gen)


def _small_shapes(design, C):
    """Shapes of the one-layer model's other tensors, in the order they are made in."""
    out = [(64, C), (C,)]
    if design == "Badapel":
        out.append((C,))
    if design == "Ratesun":
        out += [(C,), (17, C)]
    if design == "Labepel":
        out.append((4096, C))
    if design in ("Vudelix", "Zudovik", "Dufelix"):
        out.append((64, C))
    out.append((C,))
    if design in ("Badapel", "Ratesun"):
        out += [(C,), (C,), (C,)]
    if design == "Dufelix":
        out.append((C,))
    if design == "Ratesun":
        out += [(C, 4), (2,)]
    if design == "Labepel":
        out.append((C,))
    return out


def _rms(x, eps):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, first, dims, base, pairs):
    """``x [tokens, heads, size]``: the first ``dims`` entries of each head rotated by position."""
    n = x.size(0)
    f = float(base) ** (-torch.arange(0, dims, 2, device=DEV, dtype=torch.float64) / dims)
    a = torch.arange(first, first + n, device=DEV, dtype=torch.float64)[:, None] * f
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    i, j = (slice(0, dims, 2), slice(1, dims, 2)) if pairs else (slice(0, dims // 2), slice(dims // 2, dims))
    y = x.clone()
    y[..., i], y[..., j] = x[..., i] * c - x[..., j] * s, x[..., j] * c + x[..., i] * s
    return y


def _attend(q, k, v, scale, hidden, cap=0.0, sink=None):
    """``q [n, H, D]``, ``k [keys, G, D]``, ``v [keys, G, V]``: softmax attention, a few heads at a time."""
    n, H, _ = q.shape
    rep = H // k.size(1)
    out = torch.empty(n, H, v.size(2), device=DEV, dtype=torch.float64)
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink[h].expand(n, 1)), 1)
        out[:, h] = torch.softmax(s, 1)[:, :k.size(0)] @ v[:, h // rep]
    return out


def _causal(qkv, kv, first, H, G, hs, base):
    """Rotation, cache write and attention of a transformer layer; ``kv [2, G, positions, hs]`` is written."""
    n = qkv.size(0)
    x = qkv.view(n, G, H // G + 2, hs)
    q = _rotate(x[:, :, :-2].reshape(n, H, hs), first, hs, base, False)
    kv[0][:, first:first + n] = _rotate(x[:, :, -2], first, hs, base, False).transpose(0, 1)
    kv[1][:, first:first + n] = x[:, :, -1].transpose(0, 1)
    keys = first + n
    hidden = torch.arange(keys, device=DEV)[None] > torch.arange(first, keys, device=DEV)[:, None]
    return _attend(q, kv[0][:, :keys].transpose(0, 1), kv[1][:, :keys].transpose(0, 1), hs ** -0.5, hidden).reshape(n, H * hs)


def _fp8(w):
    """A block-scaled weight as it is served: e4m3 values and a scale for each 128 of a row."""
    b = w.float().view(w.size(0), -1, 128)
    s = (b.abs().amax(-1, keepdim=True) / 448.0).clamp_min(1e-12)
    return ((b / s).clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double() * s.double()).view(w.shape)


def _exact_stage(case, gen):
    C, H, G, hs, I, vocab, base, eps = MODELS[case["model"]]
    w, path = _stage_weights(case, gen), case["path"]
    x, past = _stage_inputs(case, gen)
    first = case["context"] if path == "decode" else 0
    n, L = (1 if path == "decode" else case["tokens"]), case.get("layers", 1)
    served = (lambda k: _fp8(w[k])) if case.get("weights") == "fp8" else (lambda k: w[k].double())
    kv = torch.zeros(L, 1, 2, G, first + n + 8, hs, device=DEV, dtype=torch.float64)
    if past is not None:
        kv[:, 0, :, :, :first] = past.double()
    x = w["transformer.wte.weight"][x.view(-1).to(DEV)].double() if case.get("role") == "starter" else x[0].double()
    for i in range(L):
        p = "transformer.h.%d." % i
        if path == "mixture":
            x = x + _mixture(_rms(x, eps) * w[p + "norm_2.weight"].double(), w, p + "mlp.")
            continue
        h = _rms(x, eps) * w[p + "norm_1.weight"].double()
        x = x + _causal(h @ served(p + "attn.attn.weight").T, kv[i, 0], first, H, G, hs, base) @ served(p + "attn.proj.weight").T
        h = _rms(x, eps) * w[p + "norm_2.weight"].double()
        x = x + (F.silu(h @ served(p + "mlp.fc_1.weight").T) * (h @ served(p + "mlp.fc_2.weight").T)) @ served(p + "mlp.proj.weight").T
    if path != "decode":
        return dict(y=x[None], **({"kv": kv} if path == "prompt" else {}))
    out = dict(hidden=x[None], kv=kv)
    if case["role"] == "starter":
        out["logits"] = ((_rms(x, eps) * w["transformer.ln_f.weight"].double()) @ served("lm_head.weight").T)[None]
    return out


def _mixture(h, w, p):
    z, e = torch.topk(h @ w[p + "gate.weight"].double().T, TOP, -1)
    s, y = torch.softmax(z, -1), torch.zeros_like(h)
    for j in range(EXPERTS):
        tok, k = torch.where(e == j)
        a, b, c = (w["%sexperts.%d.%s.weight" % (p, j, t)].double() for t in ("fc_1", "fc_2", "proj"))
        y.index_add_(0, tok, s[tok, k, None] * ((F.silu(h[tok] @ a.T) * (h[tok] @ b.T)) @ c.T))
    return y


def _mix(design, kind, m, w, x, st, start):
    """One mixing layer over one sequence; ``st`` is its slot's state, which is written."""
    n, h, g = x.size(0), m["heads"], m.get("kv_heads", m["heads"])
    D, V, eps = m["dim"], m["vdim"], 1e-6
    if kind in ("attention", "latent_attention"):
        keys, pos = start + n, torch.arange(start, start + n, device=DEV)[:, None]
        j, W = torch.arange(keys, device=DEV)[None], (m.get("mask") or {}).get("size", 0)
        hidden = j > pos
        if W:
            hidden = hidden | ((j < pos // W * W) if design == "Labepel" else (pos - j >= W))
    if kind == "attention":
        q, k, v = (x @ w[t].T + w.get(t + ".b", 0.0) for t in "qkv")
        if design == "Zudovik":
            q, k = _rms(q, eps) * w["q.norm"], _rms(k, eps) * w["k.norm"]
        q, k = q.view(n, h, D), k.view(n, g, D)
        if "rot" in m:
            q, k = (_rotate(t, start, m["rot"]["dims"], m["rot"]["base"], design != "Dufelix") for t in (q, k))
        if design in ("Vudelix", "Labepel"):
            q, k = _rms(q, eps) * w.get("q.norm", 1.0), _rms(k, eps) * w.get("k.norm", 1.0)
        st["cache"][start:keys] = torch.cat((k.reshape(n, g * D), v), 1)
        k, v = st["cache"][:keys, :g * D].view(keys, g, D), st["cache"][:keys, g * D:].view(keys, g, V)
        sink = {"Labepel": torch.zeros(h, device=DEV, dtype=torch.float64), "Zudovik": w.get("sink")}.get(design)
        o, gate = _attend(q, k, v, m["scale"], hidden, m.get("softcap", 0.0), sink), torch.sigmoid(x @ w["g"].T)
        return (o * gate.view(n, h, -1)).reshape(n, h * V) @ w["o"].T
    if kind == "latent_attention":
        R, L, rot, pairs = m["rot_dim"], m["kv_rank"], m["rot"], design != "Badapel"
        q = ((_rms(x @ w["dq"].T, eps) * w["dq.norm"]) @ w["uq"].T).view(n, h, D + R)
        q = torch.cat((q[..., :D], _rotate(q[..., D:], start, rot["dims"], rot["base"], pairs)), -1)
        c = x @ w["dkv"].T
        st["cache"][start:keys] = torch.cat((_rms(c[:, :L], eps) * w["dkv.norm"],
                                             _rotate(c[:, None, L:], start, rot["dims"], rot["base"], pairs)[:, 0]), 1)
        lat, kr = st["cache"][:keys, :L], st["cache"][:keys, L:]
        k = torch.cat(((lat @ w["uk"].T).view(keys, h, D), kr[:, None].expand(keys, h, R)), -1)
        o = _attend(q, k, (lat @ w["uv"].T).view(keys, h, V), m["scale"], hidden, 0.0, w.get("sink")).reshape(n, h * V)
        return (o * torch.sigmoid(x @ w["g"].T) if "g" in w else o) @ w["o"].T
    S = st["state"]
    if kind == "gla":
        q, k, v, gate = (x @ w[t].T for t in "qkvg")
        q, k, v, gate = q.view(n, h, D) * D ** -0.5, k.view(n, h, D), v.view(n, h, V), F.silu(gate)
        a = torch.exp(F.logsigmoid((x @ w["a1"].T) @ w["a2"].T + w["a2.b"]) / m["tau"]).view(n, h, D)
        b = None
    else:
        p = torch.cat((st["conv"], torch.cat([x @ w[t].T for t in "qkv"], 1)), 0)
        taps = torch.cat([w[t + ".conv"] for t in "qkv"], 0)
        c = F.silu(sum(p[i:i + n] * taps[:, i] for i in range(4)))
        st["conv"].copy_(p[-3:])
        q, k, v = c.split((g * D, g * D, h * V), 1)
        q, k = (t.reshape(n, g, D) for t in (q, k))
        q, k = (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6) for t in (q, k))
        q, k = (t.repeat_interleave(h // g, 1) for t in (q * D ** -0.5, k))
        v, gate, b = v.reshape(n, h, V), torch.sigmoid((x @ w["g1"].T) @ w["g2"].T), torch.sigmoid(x @ w["b"].T)
        a = torch.exp(-torch.exp(w["A_log"])[:, None] * F.softplus((x @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(n, h, D))
    o = torch.empty(n, h, V, device=DEV, dtype=torch.float64)
    for t in range(n):
        S.mul_(a[t][:, :, None])
        u = v[t] if b is None else b[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S.add_(k[t][:, :, None] * u[:, None])
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return ((_rms(o, eps) * w["norm"]).reshape(n, h * V) * gate) @ w["o"].T


def _layer_norm(x, w, b):
    return F.layer_norm(x, (x.size(-1),), w, b, 1e-6)


def _exact_step(case, gen):
    w, states = _step_weights(case, gen)
    ids = gen.ids(case["streams"], STEP_VOCAB)
    w = {k: t.double() for k, t in w.items()}
    x, left = w["embed"][ids], []
    for i, kind in enumerate(STEP_KINDS):
        p, m, st = "l%d." % i, _hybrid_config("Badapel", kind, case["width"]), {k: t.double() for k, t in states[i].items()}
        mix = {k[len(p) + 4:]: t for k, t in w.items() if k.startswith(p + "mix.")}
        h = _layer_norm(x, w[p + "norm1"], w[p + "norm1.b"])
        y = torch.cat([_mix("Badapel", kind, m, mix, h[j:j + 1], {k: t[j] for k, t in st.items()}, case["context"]) for j in range(x.size(0))], 0)
        left.append(st)
        x = x + _layer_norm(y, w[p + "norm1b"], w[p + "norm1b.b"])
        h = _layer_norm(x, w[p + "norm2"], w[p + "norm2.b"])
        x = x + _layer_norm(F.gelu(h @ w[p + "mlp.up"].T) @ w[p + "mlp.down"].T, w[p + "norm2b"], w[p + "norm2b.b"])
    z = _layer_norm(x, w["final.norm"], w["final.norm.b"]) @ w["embed"].T
    return dict(logits=30.0 * torch.tanh(z / 30.0), state=left)
