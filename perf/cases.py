"""Timed cases: the work that serving the registered decoder designs consists of.

Most cases are one layer's part (a feed-forward, an attention or recurrent mixer, routed experts), called the way the engine's
blocks call it: a part bound to its weights, the step's context, the layer's cache.  One case is a whole model behind the step
function.  Layer sizes are those of bench.py's comparisons of the designs (widths 2048 and 4096, heads of 128, feed-forwards of
three times the width), batches and contexts those of its decode and prompt workloads.

A case is a dict; `kind` says which part it is:

    ff        gated feed-forward (silu)                                  all dense layers of the Qwen3 decoder
    gqa       grouped-query attention with per-head norms and rotation    the same
    hgrn2     gated linear recurrence                                     Riruzen
    decay     linear attention with a fixed decay a head                  Bonolorn ("lightning"), Venitar ("retention")
    delta     gated delta rule, a decay a head or (rank > 0) a channel    Nelovik, Venitar
    ssm       selective state space                                       Nelovik
    experts   routed experts, softmax over the chosen                     Kifezen
    latent    latent attention with a rotated part and sinks              Kifezen
    serve     a Qwen3 decoder of a few layers: prompts, then decode steps, through ModelRunner.step

`seqs` requests share `tokens` new tokens (seqs == tokens: a decode step); `behind` tokens of each are in the cache already.
"""
import math

import torch

DEV = "cuda:0"
EPS = 1e-6
THETA = 1e6
PAGE = 16


def listed():
    return [
        # one decoded token through the smaller design's feed-forward: the smallest call, launches and latency
        dict(name="feed-forward 1 token", kind="ff", width=2048, ff=6144, tokens=1, dtype="bfloat16"),
        # a prompt of 2048 tokens through the larger one's: the largest product there is
        dict(name="feed-forward 2048 tokens", kind="ff", width=4096, ff=12288, tokens=2048, dtype="bfloat16"),
        # decode attention of bench.py's headline: 8 requests at 8192 cached tokens, 32 heads on 8
        dict(name="attention decode 8x8192", kind="gqa", width=4096, heads=32, kv_heads=8, seqs=8, tokens=8, behind=8191, dtype="bfloat16"),
        # a whole prompt of 2048 tokens
        dict(name="attention prompt 2048", kind="gqa", width=4096, heads=32, kv_heads=8, seqs=1, tokens=2048, behind=0, dtype="bfloat16"),
        # Riruzen's recurrence over one prompt
        dict(name="hgrn2 prompt 2048", kind="hgrn2", width=2048, heads=16, dim=128, vdim=128, seqs=1, tokens=2048, continued=False),
        # Bonolorn's recurrence over four prompts of different lengths in one step
        dict(name="lightning 4 prompts", kind="decay", width=4096, heads=16, dim=128, vdim=128, form="lightning", seqs=4, tokens=1654, continued=False),
        # Nelovik's delta rule over one prompt
        dict(name="delta prompt 2048", kind="delta", width=2048, heads=16, kv_heads=8, dim=128, vdim=128, rank=0, seqs=1, tokens=2048, continued=False),
        # Venitar's delta rule with channel decays: 64 requests decode
        dict(name="channel delta decode 64", kind="delta", width=4096, heads=16, kv_heads=8, dim=128, vdim=128, rank=64, seqs=64, tokens=64, continued=True),
        # Nelovik's state space: a later portion of a prompt, of odd length
        dict(name="state space portion 333", kind="ssm", width=2048, heads=32, vdim=64, state=128, groups=2, seqs=1, tokens=333, continued=True),
        # Kifezen's experts: 8 requests decode, every expert's weights are streamed
        dict(name="experts decode 8", kind="experts", width=4096, experts=16, top=4, ff=1536, tokens=8),
        # Kifezen's latent attention: 64 requests decode at 2016 cached tokens
        dict(name="latent decode 64x2016", kind="latent", width=4096, heads=32, seqs=64, tokens=64, behind=2015),
        # a whole decoder: 8 requests bring prompts of different lengths and then decode 8 tokens each, logits of every step
        dict(name="serve 8 requests", kind="serve", width=2048, heads=16, kv_heads=4, ff=6144, layers=4, vocab=32000, seqs=8, tokens=512, new=8),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def batch(most=2048):
        """(seqs, tokens): a decode step, one portion, or several"""
        r = rng.random()
        if r < 0.35:
            n = log(1, 64)
            return n, n
        if r < 0.7:
            return 1, log(17, most)
        n = rng.randint(2, 6)
        return n, max(8 * n, log(64, most))

    kind = rng.choice(["ff", "ff", "gqa", "gqa", "hgrn2", "decay", "delta", "delta", "ssm", "experts", "latent", "serve"])
    width = rng.choice([2048, 4096])
    heads = width // 128
    if kind == "ff":
        f32 = rng.random() < 0.2
        return dict(kind=kind, width=width, ff=3 * width, tokens=log(1, 48 if f32 else 2048), dtype="float32" if f32 else "bfloat16")
    if kind == "gqa":
        f32 = rng.random() < 0.2
        seqs, tokens = batch(64 if f32 else 2048)
        behind = log(16, 8191 if seqs <= 8 else 65528 // seqs) - 1 if seqs == tokens else rng.choice([0, log(64, 2048)])
        behind = min(behind, 512) if f32 else behind
        return dict(kind=kind, width=width, heads=heads, kv_heads=heads // 4, seqs=seqs, tokens=tokens, behind=behind, dtype="float32" if f32 else "bfloat16")
    seqs, tokens = batch()
    again = seqs == tokens or rng.random() < 0.3
    if kind == "hgrn2":
        d = rng.choice([64, 128, 128])
        return dict(kind=kind, width=width, heads=heads, dim=d, vdim=128, seqs=seqs, tokens=tokens, continued=again)
    if kind == "decay":
        form = rng.choice(["lightning", "retention"])
        return dict(kind=kind, width=width, heads=heads // 2 if form == "lightning" else heads, dim=rng.choice([64, 128, 128]), vdim=128, form=form,
                    seqs=seqs, tokens=tokens, continued=again)
    if kind == "delta":
        h = heads // rng.choice([1, 2])
        return dict(kind=kind, width=width, heads=h, kv_heads=h // rng.choice([1, 2]), dim=128, vdim=128, rank=rng.choice([0, 0, 64]), seqs=seqs,
                    tokens=tokens, continued=again)
    if kind == "ssm":
        return dict(kind=kind, width=width, heads=width // 64, vdim=64, state=rng.choice([64, 128, 128]), groups=2, seqs=seqs, tokens=tokens, continued=again)
    if kind == "experts":
        return dict(kind=kind, width=width, experts=16, top=4, ff=3 * width // 8, tokens=tokens)
    if kind == "latent":
        behind = log(16, 2048) - 1 if seqs == tokens else rng.choice([0, log(64, 2048)])
        return dict(kind=kind, width=width, heads=heads, seqs=seqs, tokens=tokens, behind=behind)
    seqs = rng.randint(1, 16)
    return dict(kind="serve", width=2048, heads=16, kv_heads=4, ff=6144, layers=rng.randint(2, 4), vocab=32000, seqs=seqs,
                tokens=max(4 * seqs, log(64, 1024)), new=rng.randint(2, 8))


# ---- sizes -----------------------------------------------------------------------------------------------------

def lengths(case):
    """New tokens of each request: all one, or shares that grow from request to request."""
    n, s = case["tokens"], case["seqs"]
    if n == s:
        return [1] * s
    total = s * (s + 1) // 2
    out = [max(1, n * (i + 1) // total) for i in range(s)]
    out[-1] += n - sum(out)
    return out


def decays(case):
    h = case["heads"]
    return [1.0 - 2.0 ** -(3 + 8 * i / max(h - 1, 1)) for i in range(h)]


LATENT = dict(dim=128, rot_dim=64, vdim=128, kv_rank=512, rot_base=1e4)


def shapes(case):
    """Tensor name -> shape, for the part of the case."""
    k, w = case["kind"], case["width"]
    if k == "ff":
        return {"m.gate_proj.weight": (case["ff"], w), "m.up_proj.weight": (case["ff"], w), "m.down_proj.weight": (w, case["ff"])}
    if k == "gqa":
        q, kv = case["heads"] * 128, case["kv_heads"] * 128
        return {"m.q_proj.weight": (q, w), "m.k_proj.weight": (kv, w), "m.v_proj.weight": (kv, w), "m.o_proj.weight": (w, q),
                "m.q_norm.weight": (128,), "m.k_norm.weight": (128,)}
    if k == "hgrn2":
        n, m = case["heads"] * case["dim"], case["heads"] * case["vdim"]
        return {"m.q": (n, w), "m.f": (n, w), "m.v": (m, w), "m.o": (w, m), "m.f.b": (n,), "m.lower": (n,), "m.norm": (case["vdim"],)}
    if k == "decay":
        n, m = case["heads"] * case["dim"], case["heads"] * case["vdim"]
        t = {"m.q": (n, w), "m.k": (n, w), "m.v": (m, w), "m.g": (m, w), "m.o": (w, m)}
        return dict(t, **({"m.norm": (m,)} if case["form"] == "lightning" else {}))
    if k == "delta":
        h, n, m, r = case["heads"], case["kv_heads"] * case["dim"], case["heads"] * case["vdim"], case["rank"]
        t = {"m.q": (n, w), "m.k": (n, w), "m.v": (m, w), "m.b": (h, w), "m.o": (w, m), "m.q.conv": (n, 4), "m.k.conv": (n, 4), "m.v.conv": (m, 4),
             "m.A_log": (h,), "m.dt_bias": (h * case["dim"] if r else h,), "m.norm": (case["vdim"],)}
        return dict(t, **({"m.a1": (r, w), "m.g1": (r, w), "m.a2": (h * case["dim"], r), "m.g2": (m, r)} if r else {"m.a": (h, w), "m.g": (m, w)}))
    if k == "ssm":
        h, m, bc = case["heads"], case["heads"] * case["vdim"], case["groups"] * case["state"]
        return {"m.in": (2 * m + 2 * bc + h, w), "m.conv": (m + 2 * bc, 4), "m.conv.b": (m + 2 * bc,), "m.o": (w, m), "m.A_log": (h,), "m.dt_bias": (h,),
                "m.D": (h,), "m.norm": (m,)}
    if k == "experts":
        t = {"m.router": (case["experts"], w)}
        for j in range(case["experts"]):
            t.update({f"m.e{j}.gate": (case["ff"], w), f"m.e{j}.up": (case["ff"], w), f"m.e{j}.down": (w, case["ff"])})
        return t
    if k == "latent":
        h, L = case["heads"], LATENT
        return {"m.q": (h * (L["dim"] + L["rot_dim"]), w), "m.dkv": (L["kv_rank"] + L["rot_dim"], w), "m.g": (h, w), "m.o": (w, h * L["vdim"]),
                "m.dkv.norm": (L["kv_rank"],), "m.uk": (h * L["dim"], L["kv_rank"]), "m.uv": (h * L["vdim"], L["kv_rank"]), "m.sink": (h,)}
    t = {"model.embed_tokens.weight": (case["vocab"], w), "model.norm.weight": (w,), "lm_head.weight": (case["vocab"], w)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        sub = {n.replace("m.", p + "self_attn.", 1): s for n, s in shapes(dict(case, kind="gqa")).items()}
        sub.update({n.replace("m.", p + "mlp.", 1): s for n, s in shapes(dict(case, kind="ff")).items()})
        t.update(sub, **{p + "input_layernorm.weight": (w,), p + "post_attention_layernorm.weight": (w,)})
    return t


F32 = ("A_log", "dt_bias", ".D", ".lower")          # tensors that checkpoints keep in 32-bit


def tensors(case, seed):
    """The weights, from the seed alone: maps N(0, 0.02), norms 1 + N(0, 0.1), rates as the designs initialise them."""
    g = torch.Generator(device=DEV)
    g.manual_seed(2 * seed + 1)
    f32 = case.get("dtype") == "float32"
    out = {}
    for name, shape in shapes(case).items():
        if name.endswith("A_log"):                                   # rates 1 .. 16
            x = torch.log(1.0 + 15.0 * torch.rand(shape, generator=g, device=DEV))
        elif name.endswith("dt_bias"):                               # steps of 0.001 .. 0.1 before the softplus
            dt = torch.exp(math.log(1e-3) + torch.rand(shape, generator=g, device=DEV) * math.log(100.0))
            x = dt + torch.log(-torch.expm1(-dt))
        elif name.endswith("lower"):
            x = torch.rand(shape, generator=g, device=DEV)
        else:
            x = torch.randn(shape, generator=g, device=DEV)
            norm = name.endswith(("norm", "norm.weight", ".D"))
            if norm:
                x = 1.0 + 0.1 * x
            elif name.endswith("conv"):
                x = 0.5 * x
            elif name.endswith((".in", ".a", ".b", ".a1")) and case["kind"] in ("delta", "ssm"):
                x = 0.01 * x
            else:
                x = 0.02 * x
        out[name] = x if f32 or name.endswith(F32) else x.to(torch.bfloat16)
    return out


def inputs(case, seed):
    """What a call brings: the normed stream, and what earlier steps have left in the caches."""
    g = torch.Generator(device=DEV)
    g.manual_seed(2 * seed)
    k = case["kind"]
    act = torch.float32 if case.get("dtype") == "float32" else torch.bfloat16
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    got = {}
    if k == "serve":
        n = case["tokens"] + case["seqs"] * case["new"]
        got["ids"] = torch.randint(0, case["vocab"], (n,), generator=g, device=DEV).cpu().tolist()
        return got
    got["h"] = rnd(case["tokens"], case["width"]).to(act)
    if k in ("gqa", "latent"):
        lens = lengths(case)
        pages = [-(-(case["behind"] + n) // PAGE) for n in lens]
        P, total = max(pages), sum(pages)
        order = torch.randperm(total, generator=g, device=DEV).to(torch.int32)
        table, at = torch.full((case["seqs"], P), -1, dtype=torch.int32, device=DEV), 0
        for i, n in enumerate(pages):
            table[i, :n] = order[at:at + n]
            at += n
        got["table"] = table
        if k == "gqa":
            got["k"], got["v"] = (rnd(total, case["kv_heads"], PAGE, 128).to(act) for _ in range(2))
        else:
            got["k"] = rnd(total, 1, PAGE, LATENT["kv_rank"] + LATENT["rot_dim"]).to(act)
    if k in ("hgrn2", "decay", "delta", "ssm"):
        rows = case["dim"] if "dim" in case else case["state"]
        scale = 0.3 if case["continued"] else 0.0
        got["state"] = scale * rnd(case["seqs"] + 1, case["heads"], rows, case["vdim"])
        if k == "delta":
            got["conv"] = scale * rnd(case["seqs"] + 1, 3, 2 * case["kv_heads"] * case["dim"] + case["heads"] * case["vdim"])
        if k == "ssm":
            got["conv"] = scale * rnd(case["seqs"] + 1, 3, case["heads"] * case["vdim"] + 2 * case["groups"] * case["state"])
    return got


# ---- the framework's side ------------------------------------------------------------------------------------------

def make_part(rt, case):
    from lucciola_b200 import parts as P
    k, w = case["kind"], case["width"]
    f32 = torch.float32
    if k == "ff":
        return P.SwiGLUFeedForward(rt, "m", w, case["ff"])
    if k == "gqa":
        return P.GQAttention(rt, "m", w, case["heads"], case["kv_heads"], 128, P.RotaryEmbedding(rt, 128, THETA), qk_norm_eps=EPS)
    if k == "hgrn2":
        return P.GatedLinearRecurrence(rt, "m", w, case["heads"], case["dim"], case["vdim"], EPS)
    if k == "decay" and case["form"] == "lightning":
        return P.DecayLinearAttention(rt, "m", w, case["heads"], case["dim"], case["vdim"], decays(case), EPS)
    if k == "decay":
        return P.DecayLinearAttention(rt, "m", w, case["heads"], case["dim"], case["vdim"], decays(case), EPS, act=None, k_scale=case["dim"] ** -0.5,
                                      position_encoding=P.RotaryEmbedding(rt, case["dim"], THETA), head_norm=True, norm_weight=False, gate_act="silu",
                                      out_dtype=f32)
    if k == "delta":
        from lucciola_b200.parts.delta_rule import GatedDeltaRule
        return GatedDeltaRule(rt, "m", w, case["heads"], case["kv_heads"], case["dim"], case["vdim"], 4, EPS, decay_rank=case["rank"],
                              gate_rank=case["rank"], gate_act="sigmoid" if case["rank"] else "silu")
    if k == "ssm":
        from lucciola_b200.parts.state_space import SelectiveStateSpace
        return SelectiveStateSpace(rt, "m", w, case["heads"], case["vdim"], case["state"], case["groups"], 2, 4, EPS)
    if k == "experts":
        return P.RoutedExperts(rt, "m", w, case["experts"], case["top"], case["ff"], "silu", 0.0, 1.0, correction=False, out_dtype=f32, scores="softmax")
    L = LATENT
    return P.RotaryLatentAttention(rt, "m", w, case["heads"], L["dim"], L["rot_dim"], L["vdim"], L["kv_rank"], (L["dim"] + L["rot_dim"]) ** -0.5,
                                   P.RotaryEmbedding(rt, L["rot_dim"], L["rot_base"]), EPS, out_dtype=f32)


def prepare_serve(case, seed):
    from lucciola_b200 import EngineOptions
    from lucciola_b200.config.registry import resolve_architecture
    from lucciola_b200.engine.step import ModelRunner
    from lucciola_b200.parts import Runtime
    from lucciola_b200.weights.loader import bind_weights
    cfg = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=case["width"], num_hidden_layers=case["layers"],
               num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], head_dim=128, intermediate_size=case["ff"],
               vocab_size=case["vocab"], max_position_embeddings=8192, rope_theta=THETA, rms_norm_eps=EPS, tie_word_embeddings=False,
               attention_bias=False, hidden_act="silu", use_sliding_window=False)
    given = tensors(case, seed)

    class Source:
        def names(self):
            return list(given)

        def shape_dtype(self, name):
            return tuple(given[name].shape), given[name].dtype

        def get(self, name):
            return given[name]

    torch.cuda.set_device(0)
    rt = Runtime(DEV, torch.bfloat16)
    arch = resolve_architecture(cfg)
    model = arch.build(arch.config_from_dict(cfg), rt)
    bind_weights(model, Source(), rt.act_dtype, rt.device)
    options = EngineOptions(max_blocks=512, block_size=PAGE, max_tokens_per_step=4096, max_num_seqs=32, max_model_len=2048)
    runner = ModelRunner(model, rt, options)
    ids, plan, at = inputs(case, seed)["ids"], [], 0
    for n in lengths(case):
        plan.append((ids[at:at + n], ids[at + n:at + n + case["new"]]))
        at += n + case["new"]
    return dict(case=case, runner=runner, requests=plan)


def prepare(case, seed):
    if case["kind"] == "serve":
        return prepare_serve(case, seed)
    from lucciola_b200.parts import BatchShape, KVCacheView, PlanView, Runtime, StateCacheView, StepContext
    torch.cuda.set_device(0)
    rt = Runtime(DEV, torch.float32 if case.get("dtype") == "float32" else torch.bfloat16)
    rt.stream = torch.cuda.current_stream().cuda_stream
    part = make_part(rt, case)
    weights = tensors(case, seed)
    part.bind_all(lambda name: weights[name])
    given = inputs(case, seed)
    state = dict(case=case, part=part, h=given["h"])
    if case["kind"] == "ff" or case["kind"] == "experts":
        return state
    lens, behind = lengths(case), case.get("behind", 0)
    starts = [behind] * case["seqs"]
    T, S, longest = sum(lens), len(lens), max(lens)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    plans, key = {}, part.plan_key()
    if key is not None:
        made = part.plan(BatchShape(lens, starts, longest, behind + longest, behind + longest))
        plans[key] = PlanView({n: torch.from_numpy(a).to(DEV) for n, a in made.arrays.items()}, made.host)
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    state["step"] = StepContext(
        num_tokens=T, num_seqs=S, positions=i32([behind + t for n in lens for t in range(n)]), token_seq=i32([i for i, n in enumerate(lens) for _ in range(n)]),
        cu_tokens=i32(cu), context_lens=i32([behind + n for n in lens]), block_tables=[given["table"]] if "table" in given else [],
        state_slots=torch.arange(S, dtype=torch.int32, device=DEV), q_lens=lens, start_positions=starts, max_q_len=longest,
        max_context_len=behind + longest, span_hint=behind + longest, plans=plans)
    if case["kind"] == "gqa":
        state["cache"] = KVCacheView(given["k"], given["v"], 0, PAGE)
        state["kept"] = [given["k"], given["v"]]
    elif case["kind"] == "latent":
        state["cache"] = KVCacheView(given["k"], given["k"], 0, PAGE)
        state["kept"] = [given["k"]]
    else:
        state["kept"] = [given[n] for n in ("conv", "state") if n in given]
        views = tuple(StateCacheView(t) for t in state["kept"])
        state["cache"] = views if case["kind"] in ("delta", "ssm") else views[0]
        state["fresh"] = not case["continued"]
    return state


def run(state):
    if "runner" in state:
        return run_serve(state)
    if "step" not in state:
        return state["part"].forward(state["h"], None)
    if state.get("fresh"):                          # requests that are admitted with this step start from zeros
        for t in state["kept"]:
            t.zero_()
    out = state["part"].forward(state["h"], state["step"], state["cache"])
    return [out, *state["kept"]]


def run_serve(state):
    """The requests' prompts in one step, then a step a token; returns every step's logits."""
    from lucciola_b200.engine.step import StepEntry
    runner, requests, out = state["runner"], state["requests"], []
    out.append(runner.step([StepEntry(i, p, (len(p) - 1,)) for i, (p, _) in enumerate(requests)]).clone())
    for j in range(state["case"]["new"]):
        out.append(runner.step([StepEntry(i, new[j:j + 1], (0,)) for i, (_, new) in enumerate(requests)]).clone())
    for i in range(len(requests)):
        runner.finish(i)
    return torch.stack(out)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------

def work(case):
    k, T = case["kind"], case["tokens"]
    size = 4 if case.get("dtype") == "float32" else 2
    sizes = {n: math.prod(s) for n, s in shapes(case).items()}
    maps = {n: c for n, c in sizes.items() if len(shapes(case)[n]) == 2 and not n.endswith("conv")}
    lens = lengths(case) if "seqs" in case else [T]
    if k == "serve":
        body = sum(c for n, c in maps.items() if "embed" not in n and n != "lm_head.weight")
        head = maps["lm_head.weight"]
        steps, S = 1 + case["new"], case["seqs"]
        n = T + S * case["new"]
        rows = sum(x * (x + 1) / 2 + sum(x + j for j in range(1, case["new"] + 1)) for x in lens)
        kv = 4 * case["kv_heads"] * 128 * case["layers"]
        return {"bytes": size * steps * (body + head) + kv * (n + sum(x + j for x in lens for j in range(case["new"]))) + 4.0 * S * steps * case["vocab"],
                "flops": 2.0 * body * n + 2.0 * head * S * steps + 4.0 * 128 * case["heads"] * case["layers"] * rows}
    if k == "experts":
        used = min(case["experts"], T * case["top"])
        one = 3 * case["width"] * case["ff"]
        return {"bytes": 2.0 * (used * one + sizes["m.router"]) + 6.0 * T * case["width"], "flops": 2.0 * T * (case["top"] * one + sizes["m.router"])}
    bytes_ = size * sum(sizes.values()) + (size + (4 if k in ("delta", "latent") or case.get("form") == "retention" else size)) * T * case["width"]
    flops = 2.0 * T * sum(maps.values())
    if k in ("gqa", "latent"):
        seen = sum(sum(case["behind"] + t + 1 for t in range(n)) for n in lens)
        if k == "gqa":
            bytes_ += size * 2 * case["kv_heads"] * 128 * (case["seqs"] * case["behind"] + T)
            flops += 4.0 * case["heads"] * 128 * seen
        else:
            # every head's own keys and values, or the latent space: whichever is less work
            bytes_ += 2 * 576 * (case["seqs"] * case["behind"] + T)
            apart = 2.0 * case["heads"] * (192 + 128) * seen + 2.0 * case["heads"] * 256 * 512 * case["seqs"] * case["behind"]
            flops += min(apart, 2.0 * case["heads"] * (576 + 512) * seen)
    elif k in ("hgrn2", "decay", "delta", "ssm"):
        rows = case.get("dim") or case["state"]
        cell = case["heads"] * rows * case["vdim"]
        bytes_ += 4.0 * cell * case["seqs"] * (2 if case["continued"] else 1)
        flops += (6.0 if k == "delta" else 4.0) * cell * T
    return {"bytes": float(bytes_), "flops": float(flops)}


def tolerance(case):
    """Measured against `exact`: parts whose values are rounded to 16 bits a few times on the way 0.0016 .. 0.0042, the whole decoder
    0.011, parts in 32 bits throughout 1.3e-6."""
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    return {"rel": 3e-2, "max": 0.3} if case["kind"] == "serve" else {"rel": 1e-2, "max": 0.2}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------

def _silu(x):
    return x * torch.sigmoid(x)


def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _rotate(x, pos, base):
    """Half-rotation of all of x [T, heads, n]."""
    n = x.shape[-1]
    f = base ** (-torch.arange(0, n, 2, dtype=torch.float64, device=DEV) / n)
    a = pos.double()[:, None, None] * f
    u, v = x[..., :n // 2], x[..., n // 2:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)


def _attend(q, k, v, start, scale, sinks=None):
    """q [T, H, D] at positions start .. over k [n, G, D], v [n, G, V]."""
    T, H, _ = q.shape
    n, G, _ = k.shape
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    k, v = k.permute(1, 2, 0), v.transpose(0, 1)
    for t0 in range(0, T, 256):
        m = min(256, T - t0)
        s = q[t0:t0 + m].reshape(m, G, H // G, -1).permute(1, 2, 0, 3).reshape(G, H // G * m, -1) @ k * scale
        s = s.view(G, H // G, m, n)
        s.masked_fill_(torch.arange(n, device=DEV)[None, :] > (start + t0 + torch.arange(m, device=DEV))[:, None], -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks.view(G, H // G, 1, 1).expand(G, H // G, m, 1)], -1)
        p = torch.softmax(s, -1)[..., :n].reshape(G, -1, n) @ v
        out[t0:t0 + m] = p.view(G, H // G, m, -1).permute(2, 0, 1, 3).reshape(m, H, -1)
    return out


def _conv(x, past, w, lens, bias=None):
    """silu of the causal convolution of each request's rows; returns (y, the last inputs of each)."""
    out, last, at = [], [], 0
    for i, n in enumerate(lens):
        z = torch.cat([past[i], x[at:at + n]])
        y = sum(z[j:j + n] * w[:, j] for j in range(w.shape[1]))
        out.append(_silu(y if bias is None else y + bias))
        last.append(z[n:])
        at += n
    return torch.cat(out), torch.stack(last)


def _walk(lens, state, step):
    """step(t, S) for every token in order; returns the outputs and the states."""
    outs, states, t = [], [], 0
    for i, n in enumerate(lens):
        S = state[i]
        for _ in range(n):
            S, o = step(t, S)
            outs.append(o)
            t += 1
        states.append(S)
    return torch.stack(outs), torch.stack(states + [state[len(lens)]])


def exact(case, seed):
    w = {n: t.double() for n, t in tensors(case, seed).items()}
    given = inputs(case, seed)
    k = case["kind"]
    if k == "serve":
        return exact_serve(case, w, given["ids"])
    x = given["h"].double()
    T = x.shape[0]
    p = lambda name: x @ w["m." + name].T
    if k == "ff":
        return (_silu(p("gate_proj.weight")) * p("up_proj.weight")) @ w["m.down_proj.weight"].T
    if k == "experts":
        z = p("router")
        top = z.topk(case["top"], -1)
        weight = torch.softmax(top.values, -1)
        out = torch.zeros_like(x)
        for j in range(case["experts"]):
            t, c = (top.indices == j).nonzero(as_tuple=True)
            h = x[t]
            out[t] += weight[t, c, None] * ((_silu(h @ w[f"m.e{j}.gate"].T) * (h @ w[f"m.e{j}.up"].T)) @ w[f"m.e{j}.down"].T)
        return out
    lens, H = lengths(case), case["heads"]
    if k in ("gqa", "latent"):
        b, out, at = case["behind"], [], 0
        if k == "gqa":
            G = case["kv_heads"]
            q, kk, v = p("q_proj.weight").view(T, H, 128), p("k_proj.weight").view(T, G, 128), p("v_proj.weight").view(T, G, 128)
            q, kk = _rms(q) * w["m.q_norm.weight"], _rms(kk) * w["m.k_norm.weight"]
        else:
            q, dkv = p("q").view(T, H, 192), p("dkv")
            c, kr = _rms(dkv[:, :512]) * w["m.dkv.norm"], dkv[:, 512:]
        for i, n in enumerate(lens):
            rows, pos = slice(at, at + n), torch.arange(b, b + n, device=DEV)
            pages = given["table"][i, :-(-(b + n) // PAGE)].long()
            past = given["k"][pages].double().transpose(1, 2).flatten(0, 1)[:b]
            if k == "gqa":
                vpast = given["v"][pages].double().transpose(1, 2).flatten(0, 1)[:b]
                keys, values = torch.cat([past, _rotate(kk[rows], pos, THETA)]), torch.cat([vpast, v[rows]])
                out.append(_attend(_rotate(q[rows], pos, THETA), keys, values, b, 128 ** -0.5))
            else:
                lat = torch.cat([past[:, 0, :512], c[rows]])
                rot = torch.cat([past[:, 0, 512:], _rotate(kr[rows, None], pos, LATENT["rot_base"])[:, 0]])
                m = lat.shape[0]
                keys = torch.cat([(lat @ w["m.uk"].T).view(m, H, 128), rot[:, None].expand(m, H, 64)], -1)
                qq = torch.cat([q[rows, :, :128], _rotate(q[rows, :, 128:], pos, LATENT["rot_base"])], -1)
                out.append(_attend(qq, keys, (lat @ w["m.uv"].T).view(m, H, 128), b, 192 ** -0.5, w["m.sink"]))
            at += n
        o = torch.cat(out)
        if k == "gqa":
            return [o.reshape(T, -1) @ w["m.o_proj.weight"].T, None, None]
        return [(o * torch.sigmoid(p("g"))[:, :, None]).reshape(T, -1) @ w["m.o"].T, None]
    state, V = given["state"].double(), case["vdim"]
    if k == "hgrn2":
        D = case["dim"]
        q, v = _silu(p("q")).view(T, H, D, 1), p("v").view(T, H, 1, V)
        low = w["m.lower"]
        f = (low + (1 - low) * torch.sigmoid(p("f") + w["m.f.b"])).view(T, H, D, 1)

        def step(t, S):
            S = f[t] * S + (1 - f[t]) * v[t]
            return S, (S * q[t]).sum(1)
        o, states = _walk(lens, state, step)
        return [(_rms(o) * w["m.norm"]).reshape(T, -1) @ w["m.o"].T, states]
    if k == "decay":
        D, light = case["dim"], case["form"] == "lightning"
        q, kk, v, g = p("q").view(T, H, D), p("k").view(T, H, D), p("v").view(T, H, 1, V), p("g")
        if light:
            q, kk, v = _silu(q), _silu(kk), _silu(v)
        else:
            pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
            q, kk = _rotate(q, pos, THETA), _rotate(kk, pos, THETA) * D ** -0.5
        d = torch.tensor(decays(case), dtype=torch.float64, device=DEV)[:, None, None]
        q, kk = q[..., None], kk[..., None]

        def step(t, S):
            S = d * S + kk[t] * v[t]
            return S, (S * q[t]).sum(1)
        o, states = _walk(lens, state, step)
        o = _rms(o.reshape(T, -1)) * w["m.norm"] * torch.sigmoid(g) if light else _rms(o).reshape(T, -1) * _silu(g)
        return [o @ w["m.o"].T, states]
    if k == "delta":
        D, G, r = case["dim"], case["kv_heads"], case["rank"]
        pre = torch.cat([p("q"), p("k"), p("v")], -1)
        y, last = _conv(pre, given["conv"].double(), torch.cat([w[f"m.{n}.conv"] for n in "qkv"]), lens)
        unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
        q, kk, v = y[:, :G * D].view(T, G, D), y[:, G * D:2 * G * D].view(T, G, D), y[:, 2 * G * D:].view(T, H, V)
        q, kk = (unit(z).repeat_interleave(H // G, 1) for z in (q, kk))
        q, kk = (q * D ** -0.5)[..., None], kk[..., None]
        beta = torch.sigmoid(p("b"))
        rate = -torch.exp(w["m.A_log"])
        soft = torch.nn.functional.softplus
        if r:
            a = (p("a1") @ w["m.a2"].T + w["m.dt_bias"]).view(T, H, D)
            decay, gate = torch.exp(rate[:, None] * soft(a))[..., None], torch.sigmoid(p("g1") @ w["m.g2"].T)
        else:
            decay, gate = torch.exp(rate * soft(p("a") + w["m.dt_bias"]))[..., None, None], _silu(p("g"))

        def step(t, S):
            S = decay[t] * S
            u = beta[t][:, None] * (v[t] - (S * kk[t]).sum(1))
            S = S + kk[t] * u[:, None]
            return S, (S * q[t]).sum(1)
        o, states = _walk(lens, state, step)
        last = torch.cat([last, given["conv"].double()[-1:]])
        return [((_rms(o) * w["m.norm"]).reshape(T, -1) * gate) @ w["m.o"].T, last, states]
    N, G = case["state"], case["groups"]
    m, bc = H * V, G * N
    pre = p("in")
    z, xbc, dt = pre[:, :m], pre[:, m:2 * m + 2 * bc], torch.nn.functional.softplus(pre[:, 2 * m + 2 * bc:] + w["m.dt_bias"])
    y, last = _conv(xbc, given["conv"].double(), w["m.conv"], lens, w["m.conv.b"])
    v = y[:, :m].view(T, H, V)
    B, C = (y[:, m + i * bc:m + (i + 1) * bc].view(T, G, N).repeat_interleave(H // G, 1)[..., None] for i in (0, 1))
    decay = torch.exp(-torch.exp(w["m.A_log"]) * dt)[..., None, None]

    def step(t, S):
        S = decay[t] * S + B[t] * (dt[t][:, None] * v[t])[:, None]
        return S, (S * C[t]).sum(1) + w["m.D"][:, None] * v[t]
    o, states = _walk(lens, state, step)
    o = o.reshape(T, m) * _silu(z)
    o = _rms(o.view(T, 2, -1)).reshape(T, m) * w["m.norm"]
    return [o @ w["m.o"].T, torch.cat([last, given["conv"].double()[-1:]]), states]


def exact_serve(case, w, ids):
    """Every request's whole sequence at once; the logits of its prompt's last token and of each token after it."""
    H, G, rows, at = case["heads"], case["kv_heads"], [], 0
    for n in lengths(case):
        n += case["new"]
        x = w["model.embed_tokens.weight"][torch.tensor(ids[at:at + n], device=DEV)]
        pos = torch.arange(n, device=DEV)
        for i in range(case["layers"]):
            t = lambda name: w[f"model.layers.{i}.{name}.weight"]
            h = _rms(x) * t("input_layernorm")
            q, k, v = ((h @ t(f"self_attn.{s}_proj").T).view(n, c, 128) for s, c in (("q", H), ("k", G), ("v", G)))
            q, k = _rotate(_rms(q) * t("self_attn.q_norm"), pos, THETA), _rotate(_rms(k) * t("self_attn.k_norm"), pos, THETA)
            x = x + _attend(q, k, v, 0, 128 ** -0.5).reshape(n, -1) @ t("self_attn.o_proj").T
            h = _rms(x) * t("post_attention_layernorm")
            x = x + (_silu(h @ t("mlp.gate_proj").T) * (h @ t("mlp.up_proj").T)) @ t("mlp.down_proj").T
        tail = _rms(x[n - case["new"] - 1:]) * w["model.norm.weight"]
        rows.append(tail @ w["lm_head.weight"].T)
        at += n
    return torch.stack(rows, 1)
