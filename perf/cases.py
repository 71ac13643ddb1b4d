"""The calls that the framework's speed is judged by: what a program that serves or evaluates these models has it do.

A case is a model, a call and sizes:
    model  "gptj-6b" (28 layers, width 4096), "gptj-tiny" (2 layers, width 256), "keselix", "bavutar" (6 layer runs; ``width``)
    call   "reply"   CausalTransformer.generate with the logits, one call from host ids to host tokens
           "batch"   the per-GPU program: CausalTransformerShard.generate_initial and generate_scan on device ids
           "serve"   continuous batching: prompts of unequal length admitted into the slots of a running batch, then steps
           "replay"  TraceRunner: portions of several requests in turn, logits behind every portion (layer stacks)
           "eval"    CausalTransformer.eval: loss and hits of every position
``batch`` sequences or slots, ``prompt`` the (longest) prompt, ``steps`` decoded tokens or replayed steps.

Weights have the shape of a trained model's where it matters for comparing results: the head prefers one successor of every
token by a clear margin, as a trained model does on most positions, so that a decoded sequence does not depend on the rounding
of near-ties; everything else is random.  A model is made once and kept, as a program that serves it would.
"""
import os
import random
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.getcwd(), "mesh-transformer-jax_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

WINDOW = 2048                                        # longest prompt of every model but the tiny one
TINY_WINDOW = 128
MOST_ROWS = 32 * 1024                                # prompt tokens of the largest call


def listed():
    return [
        # the smallest model and shortest steps: what a call costs besides its arithmetic
        dict(name="tiny_reply", model="gptj-tiny", width=256, dtype="bfloat16", call="reply", batch=2, prompt=100, steps=32, sampled=False),
        # one user's turn: a short question, a short answer
        dict(name="gptj_reply", model="gptj-6b", width=4096, dtype="bfloat16", call="reply", batch=1, prompt=137, steps=16, sampled=False),
        # a full context behind one sequence: prefill of the whole window, decode with eviction
        dict(name="gptj_window", model="gptj-6b", width=4096, dtype="bfloat16", call="batch", batch=1, prompt=2048, steps=16, sampled=False),
        # a few users at once, prompts as they come
        dict(name="gptj_serve_5", model="gptj-6b", width=4096, dtype="bfloat16", call="serve", batch=5, prompt=701, steps=12, sampled=True),
        # a full serving batch, nucleus sampling
        dict(name="gptj_batch_32", model="gptj-6b", width=4096, dtype="bfloat16", call="batch", batch=32, prompt=1024, steps=16, sampled=True),
        # perplexity over whole windows, and over short documents of odd length
        dict(name="gptj_eval_8x2048", model="gptj-6b", width=4096, dtype="bfloat16", call="eval", batch=8, prompt=2048, steps=0, sampled=False),
        dict(name="gptj_eval_3x333", model="gptj-6b", width=4096, dtype="bfloat16", call="eval", batch=3, prompt=333, steps=0, sampled=False),
        # state-space and latent-attention layers: one long conversation; a batch of short ones
        dict(name="keselix_reply", model="keselix", width=4096, dtype="bfloat16", call="reply", batch=1, prompt=1500, steps=32, sampled=False),
        dict(name="keselix_batch_24", model="keselix", width=2048, dtype="bfloat16", call="batch", batch=24, prompt=300, steps=32, sampled=True),
        # requests that grow by a few tokens at a time, in 32 bits
        dict(name="keselix_replay_f32", model="keselix", width=2048, dtype="float32", call="replay", batch=3, prompt=21, steps=12, sampled=False),
        # matrix-state and grouped-attention layers: one conversation; users of very different length
        dict(name="bavutar_reply", model="bavutar", width=4096, dtype="bfloat16", call="reply", batch=1, prompt=900, steps=32, sampled=False),
        dict(name="bavutar_serve_8", model="bavutar", width=4096, dtype="bfloat16", call="serve", batch=8, prompt=2000, steps=24, sampled=True),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    model = rng.choice(["gptj-6b"] * 5 + ["keselix"] * 4 + ["bavutar"] * 4 + ["gptj-tiny"])
    gptj = model.startswith("gptj")
    call = rng.choice(["reply", "batch", "serve", "eval"] + ([] if gptj else ["replay"]))
    width = {"gptj-6b": 4096, "gptj-tiny": 256}.get(model) or rng.choice([2048, 4096])
    dtype = "float32" if call == "replay" and rng.random() < 0.5 else "bfloat16"
    window = TINY_WINDOW if model == "gptj-tiny" else WINDOW
    batch = {"reply": spread(1, 4), "batch": spread(1, 32), "serve": spread(2, 16), "replay": spread(1, 6), "eval": spread(1, 8)}[call]
    prompt = spread(1, 150) if call == "replay" else spread(17, window)
    prompt = max(1, min(prompt, (MOST_ROWS if gptj else MOST_ROWS // 2) // batch))
    steps = 0 if call == "eval" else spread(8, 16 if call == "replay" or model == "gptj-6b" else 48)
    return dict(model=model, width=width, dtype=dtype, call=call, batch=batch, prompt=prompt, steps=steps,
                sampled=call in ("batch", "serve") and rng.random() < 0.6)


# ------------------------------------------------------------------ models ----
def config(case):
    """The configuration of a case's model, with the proportions that bench.py gives layer stacks at a width."""
    d, model = case["width"], case["model"]
    if model == "gptj-6b":
        return {"layers": 28, "d_model": 4096, "n_heads": 16, "n_vocab": 50400, "norm": "layernorm", "pe": "rotary",
                "pe_rotary_dims": 64, "seq": WINDOW, "cores_per_replica": 1, "per_replica_batch": 1}
    if model == "gptj-tiny":
        return {"layers": 2, "d_model": 256, "n_heads": 4, "n_vocab": 512, "norm": "layernorm", "pe": "rotary",
                "pe_rotary_dims": 16, "seq": TINY_WINDOW, "cores_per_replica": 1, "per_replica_batch": 1}
    if model == "keselix":
        attn = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": d * 11 // 4},
                "mixer": {"heads": d // 128, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                          "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 64}}}
        ssm = {"type": "mamba1", "mixer": {"inner": 2 * d, "state": 16, "conv": 4, "dt_rank": d // 16}, "mlp": None}
        return {"architecture": "Keselix", "vocab": 32768, "width": d, "layers": [ssm, attn, ssm, attn], "norm": {"eps": 1e-5},
                "loop": {"start": 1, "stop": 3, "times": 2}, "residual_mult": 0.5, "seq": WINDOW, "mtj_dtype": case["dtype"]}
    mlp = {"kind": "dense", "ff": 3 * d}
    attn = {"type": "attention", "mlp": mlp,
            "mixer": {"heads": d // 128, "kv_heads": d // 512, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                      "q_temp": {"coef": 0.1, "every": 8192}}}
    delta = {"type": "channel_delta", "mlp": mlp,
             "mixer": {"heads": d // 128, "kv_heads": d // 128, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 128, "gate_rank": 128}}
    ssd = {"type": "mamba2", "mlp": mlp,
           "mixer": {"heads": d // 32, "vdim": 64, "state": 128, "groups": 8, "norm_groups": 8, "conv": 4}}
    late = dict(attn, mixer=dict(attn["mixer"], kv_from=1))
    return {"architecture": "Bavutar", "vocab": 32768, "width": d, "layers": [delta, attn, ssd, delta, late, ssd], "norm": {"eps": 1e-5},
            "postln_alpha": 2.0, "embedding": {"scale": 1.0}, "logit_softcap": 30.0, "seq": WINDOW, "mtj_dtype": case["dtype"]}


def layer_runs(cfg):
    """[(layer index, first of a pass of the loop)] in the order the layers run."""
    n, loop = len(cfg["layers"]), cfg.get("loop")
    if not loop:
        return [(i, False) for i in range(n)]
    a, b = loop["start"], loop["stop"]
    return ([(i, False) for i in range(a)] + [(i, i == a) for _ in range(loop["times"]) for i in range(a, b)] +
            [(i, False) for i in range(b, n)])


def successors(vocab):
    """The token that the model prefers behind each token."""
    return np.random.default_rng(7).permutation(vocab)


def random_params(cfg):
    """The two-level parameter tree, bf16 on the GPU."""
    from mesh_transformer import registry
    from mesh_transformer._runtime import param_shapes
    full = registry.prepare(cfg)
    d, V = full["d_model"], full["n_vocab"]
    gen = torch.Generator(device="cuda")
    succ = torch.from_numpy(successors(V)).cuda()
    params, embed, at = {}, None, 0

    def normal(shape, std, mean=0.0):
        return torch.randn(shape, generator=gen, device="cuda") * std + mean

    def head(shape):
        """Rows along the embedding of the token they follow, long enough for a clear preference, and noise."""
        rows = torch.empty((V, d), device="cuda")
        e = embed.float()
        rows[succ] = e / e.norm(dim=-1, keepdim=True)
        rows = rows * {"gptj": 0.6 if V > 1000 else 1.0, "Keselix": 0.5, "Bavutar": 2.0}[cfg.get("architecture", "gptj")] + normal((V, d), 0.002)
        return rows if shape == (V, d) else rows.T

    for mod, leaves in param_shapes(full).items():
        out = {}
        for leaf, shape in leaves.items():
            at += 1
            gen.manual_seed(1000 + at)
            name = leaf.split(".", 1)[1] if leaf[0] == "l" and leaf[1:2].isdigit() else leaf
            if mod.endswith("embedding_shard/~/linear") and leaf == "w" or name == "embed":
                t = embed = normal(shape, 1.0).to(torch.bfloat16)
            elif mod.endswith("projection_shard/~/linear") and leaf == "w" or name == "head":
                t = None if embed is None else head(tuple(shape))
            elif name in ("scale", "norm1", "norm1b", "norm2", "norm2b", "final.norm") or name.endswith(".norm") or name == "mix.D":
                t = normal(shape, 0.1, 1.0)
            elif name in ("offset", "b") or name.endswith("norm.b") or name in ("norm1.b", "norm2.b", "mix.conv.b"):
                t = normal(shape, 0.1)
            elif name == "mix.A_log":
                t = (1 + 15 * torch.rand(shape, generator=gen, device="cuda")).log()
            elif name in ("mix.dt.b", "mix.dt_bias"):
                dt = torch.exp(torch.rand(shape, generator=gen, device="cuda") * np.log(100.0) + np.log(1e-3))
                t = dt + torch.log(-torch.expm1(-dt))               # step sizes from 0.001 to 0.1
            elif name == "loop.in":                                 # keeps both halves, mixes a little
                eye = 0.7 * torch.eye(d, device="cuda")
                t = torch.cat([eye, eye], 1) + normal(shape, 0.1 * shape[-1] ** -0.5)
            elif name == "w":                                       # GPT-J: its usual 0.02, sublayers scaled by depth
                t = normal(shape, 0.02 * ((2 * cfg["layers"]) ** -0.5 if mod.endswith(("linear_3", "linear_5")) else 1.0))
            else:
                t = normal(shape, shape[-1] ** -0.5)
            out[leaf] = t if t is None else t.to(torch.bfloat16)[None]
        params[mod] = out
    for leaves in params.values():                                  # a head that is listed before the embedding
        for leaf, t in leaves.items():
            if t is None:
                gen.manual_seed(999)
                leaves[leaf] = head((V, d)).to(torch.bfloat16)[None]
    return params


_kept = {}                                            # the last model, and what was opened for its last kind of call


def network(case):
    """The case's CausalTransformer: made once and kept until another model is asked for."""
    from mesh_transformer.transformer_shard import CausalTransformer
    key = (case["model"], case["width"], case["dtype"])
    if _kept.get("model") != key:
        forget()
        net = CausalTransformer(config(case), init_weights=False)
        net.state = {"params": random_params(config(case)), "step": np.array(0), "opt_state": None}
        _kept.update(model=key, net=net)
    return _kept["net"]


def forget(opened_only=False):
    for name in ("opened", "net"):
        if name == "net" and opened_only:
            continue
        thing = _kept.pop(name, None)
        if thing is not None:
            thing.close()
    _kept.pop("capacity", None)
    if not opened_only:
        _kept.pop("model", None)
    torch.cuda.empty_cache()


def runtime(case):
    """A per-GPU runtime with the capacity of the case's batch, as the device-level programs open it."""
    from mesh_transformer._runtime import ShardRuntime
    net = network(case)
    key = (case["batch"], case["steps"])
    if _kept.get("capacity") != key:
        forget(opened_only=True)
        net.close()
        rt = ShardRuntime(net.config, max_batch=case["batch"], max_gen=case["steps"])
        rt.load_params(net.state["params"])
        _kept.update(opened=rt, capacity=key)
    return _kept["opened"]


# ----------------------------------------------------------------- passes ----
def inputs(case, seed):
    """What is asked of the model, from the seed alone: prompts, portions or documents, as host arrays."""
    rng = np.random.default_rng([seed, 5])
    cfg = config(case)
    V = cfg.get("n_vocab") or cfg["vocab"]
    B, P = case["batch"], case["prompt"]
    out = {"key": int(rng.integers(1, 2 ** 60))}
    if case["call"] == "replay":
        portions = [[int(n) for n in rng.integers(1, P + 1, size=B)] for _ in range(case["steps"])]
        portions[0] = [P] * B                                      # every request opens with its longest portion
        out["steps"] = [[rng.integers(0, V, size=n) for n in step] for step in portions]
        return out
    lengths = np.full(B, P)
    if case["call"] == "serve":
        lengths = np.maximum(1, (P * np.linspace(1.0, 0.08, B)).astype(int))
    elif case["call"] == "reply" and B > 1:
        lengths = np.maximum(1, (P * np.linspace(1.0, 0.5, B)).astype(int))
    out["prompts"] = [rng.integers(0, V, size=n) for n in lengths]
    if case["call"] == "eval":
        obs = np.stack(out["prompts"])
        likely = successors(V)[obs]
        out["obs"] = obs
        out["target"] = np.where(rng.random(obs.shape) < 0.5, likely, rng.integers(0, V, size=obs.shape))
        out["ctx_length"] = np.maximum(1, (P * np.linspace(1.0, 0.7, B)).astype(int))
    return out


def prepare(case, seed):
    x = inputs(case, seed)
    state = {"case": case, "net": network(case), "key": x["key"]}
    B, call = case["batch"], case["call"]
    seq = state["net"].config["seq"]
    if call == "eval":
        forget(opened_only=True)
        state["sample"] = {k: x[k].astype(np.uint32) for k in ("obs", "target")}
        state["sample"]["ctx_length"] = x["ctx_length"]
        return state
    if call == "replay":
        from mesh_transformer.trace import TraceRunner
        forget(opened_only=True)
        state["runner"] = TraceRunner(state["net"], B)
        state["trace"] = [{"step": i, "entries": [{"id": str(r), "tokens": [int(t) for t in tokens], "want": [len(tokens) - 1]}
                                                  for r, tokens in enumerate(step)], "end": []} for i, step in enumerate(x["steps"])]
        state["trace"][-1]["end"] = [str(r) for r in range(B)]
        return state
    if call == "serve":
        state["rt"] = runtime(case)
        state["prompts"] = [torch.from_numpy(p.astype(np.int32)).cuda() for p in x["prompts"]]
    else:
        ctx = np.zeros((B, seq), np.uint32)
        for row, p in zip(ctx, x["prompts"]):
            row[seq - len(p):] = p
        state["lengths"] = np.array([len(p) for p in x["prompts"]], np.uint32)
        if call == "reply":
            forget(opened_only=True)
            state["ctx"] = ctx
        else:
            from mesh_transformer.transformer_shard import CausalTransformerShard
            state["rt"] = runtime(case)
            state["shard"] = CausalTransformerShard(state["net"].config, runtime=state["rt"])
            state["ctx"] = torch.from_numpy(ctx.view(np.int32)).cuda()
    state["sampler"] = {"greedy": True}
    if case["sampled"]:
        state["sampler"] = {"greedy": False, "top_p": torch.full((B,), 0.9, device="cuda"), "temp": torch.ones(B, device="cuda")}
    return state


def run(state):
    case = state["case"]
    B, steps = case["batch"], case["steps"]
    if case["call"] == "eval":
        return state["net"].eval(state["sample"])
    if case["call"] == "replay":
        return torch.cat([state["runner"].step(step) for step in state["trace"]])
    if case["call"] == "reply":
        random.seed(state["key"])
        greedy = {"top_p": np.zeros(B), "temp": np.ones(B)}
        _, (tokens, _, logits) = state["net"].generate(state["ctx"], state["lengths"], steps, greedy, return_logits=True)
        return {"tokens": tokens.astype(np.int64)[:, :, 0].T, "logits": logits[:, :, 0].swapaxes(0, 1)}
    rt = state["rt"]
    tokens = torch.empty((steps, B), dtype=torch.int32, device="cuda")
    logits = torch.empty((steps, B, rt.config["n_vocab"]), dtype=torch.float32, device="cuda")
    if case["sampled"]:
        rt.set_seed(state["key"])
    if case["call"] == "batch":
        state["shard"].generate_initial(state["ctx"], state["lengths"])
        state["shard"].generate_scan(steps, tokens, logits, **state["sampler"])
    else:
        rt.start_batch(B)
        for slot, prompt in enumerate(state["prompts"]):
            rt.admit(slot, prompt)
        for t in range(steps):
            rt.decode_step(None, tokens[t], logits[t], **state["sampler"])
    return {"tokens": tokens, "logits": logits}


# ------------------------------------------------------------------- sizes ----
def sequences(case):
    """[(prompt rows computed, decoded rows, rows with logits)] of every sequence; seed-independent up to a replay's portions."""
    x = inputs(case, 0)
    if case["call"] == "replay":
        return [(sum(len(step[r]) for step in x["steps"]), 0, case["steps"]) for r in range(case["batch"])]
    if case["call"] == "eval":
        return [(case["prompt"], 0, case["prompt"])] * case["batch"]
    return [(len(p) - 1, case["steps"], case["steps"]) for p in x["prompts"]]


def work(case):
    """Flops of every row; bytes: each weight once per forward pass that has to follow another one, caches and states as they
    are read and written, activations only where they are inputs or outputs."""
    cfg = config(case)
    V = cfg.get("n_vocab") or cfg["vocab"]
    d = case["width"]
    seqs = sequences(case)
    passes = {"eval": 1, "replay": case["steps"]}.get(case["call"], case["steps"] + 1)
    act = 4 if case["dtype"] == "float32" else 2
    weights = flops = cache = 0
    if "n_heads" in cfg:
        weights = cfg["layers"] * 12 * d * d
        for rows, dec, _ in seqs:
            n = rows + dec
            flops += cfg["layers"] * 2 * d * n * (n + 1)
            cache += cfg["layers"] * 4 * d * (n + sum(min(rows + 1 + t, cfg["seq"] - 1) for t in range(dec)))
    else:
        from mesh_transformer import registry
        from mesh_transformer.layer_stack import tensor_shapes
        shapes = tensor_shapes(registry.prepare(cfg))
        for i, first in layer_runs(cfg):
            weights += sum(int(np.prod(s)) for k, s in shapes.items() if k.startswith(f"l{i}.") and len(s) > 1 and "conv" not in k and "A_log" not in k)
            weights += int(np.prod(shapes["loop.in"])) if first else 0
            kind, m = cfg["layers"][i]["type"], cfg["layers"][i]["mixer"]
            for rows, dec, _ in seqs:
                n = rows + dec
                if kind == "latent_attention":
                    w = m["mask"]["size"]
                    flops += 2 * sum(min(t + 1, w) for t in range(n)) * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
                    cache += act * (m["kv_rank"] + m["rot_dim"]) * (n + sum(min(rows + 1 + t, w) for t in range(dec)))
                elif kind == "attention":
                    flops += n * (n + 1) * m["heads"] * (m["dim"] + m["vdim"])
                    cache += act * m["kv_heads"] * (m["dim"] + m["vdim"]) * (n + sum(rows + 1 + t for t in range(dec)))
                elif kind == "mamba1":
                    flops += 6 * n * m["inner"] * m["state"]
                    cache += 8 * (1 + dec) * m["inner"] * (m["state"] + m["conv"] - 1)
                else:
                    k = m["state"] if kind == "mamba2" else m["dim"]
                    flops += (6 if kind == "mamba2" else 8) * n * m["heads"] * k * m["vdim"]
                    cache += 8 * (1 + dec) * m["heads"] * k * m["vdim"]
    flops += 2 * weights * sum(r + n for r, n, _ in seqs)
    scored = sum(n for _, _, n in seqs)
    flops += 2 * V * d * scored
    outputs = 5 * scored if case["call"] == "eval" else 4 * V * scored
    return {"bytes": 2 * weights * passes + 2 * V * d * max(1, passes - 1) + cache + outputs, "flops": flops}


def tolerance(case):
    """About four times what the outputs were measured to be off from ``exact``: 5e-7 in 32 bits; in bf16 8e-4 (logits of GPT-J),
    2.3e-4 (its losses) and 6e-3 (layer stacks, whose recurrences carry rounding on)."""
    if case["dtype"] == "float32":
        return {"rel": 4e-6}
    if case["model"].startswith("gptj"):
        return {"rel": 1e-3 if case["call"] == "eval" else 4e-3, "differ": 2e-3}
    return {"rel": 2.5e-2, "differ": 2e-3}


# ------------------------------------------------------------------- exact ----
def exact(case, seed):
    """The same outputs in 64-bit floating point, plain torch."""
    cfg = config(case)
    x = inputs(case, seed)
    params = network(case).state["params"]
    if _kept.get("opened") is not None:
        forget(opened_only=True)
    forward = gptj_forward if "n_heads" in cfg else stack_forward
    with torch.no_grad():
        if case["call"] == "eval":
            obs, target = (torch.from_numpy(x[k].astype(np.int64)).cuda() for k in ("obs", "target"))
            ranges = [(0, case["prompt"])] * case["batch"]
            loss, hit = [], []
            limit = torch.from_numpy(x["ctx_length"]).cuda()
            for b, logits in forward(cfg, params, obs, ranges, limit):
                at = logits.gather(-1, target[b][:, None])[:, 0]
                loss.append(torch.logsumexp(logits, -1) - at)
                hit.append(at == logits.max(-1).values)
            loss = torch.stack(loss)
            return {"loss": loss.mean(-1), "last_loss": loss[:, -1], "all_loss": loss, "correct": torch.stack(hit)}
        if case["call"] == "replay":
            B, steps = case["batch"], case["steps"]
            tokens = [np.concatenate([step[r] for step in x["steps"]]) for r in range(B)]
            ends = [np.cumsum([len(step[r]) for step in x["steps"]]) - 1 for r in range(B)]
            out = [None] * B
            for b, logits in forward(cfg, params, padded(tokens), [(0, len(t)) for t in tokens], None):
                out[b] = logits[torch.from_numpy(ends[b]).cuda()]
            return torch.stack(out, 1).reshape(steps * B, -1)
        succ = successors(cfg.get("n_vocab") or cfg["vocab"])
        steps, tokens = case["steps"], []
        for p in x["prompts"]:
            p = list(p)
            for _ in range(steps - 1):
                p.append(succ[p[-1]])
            tokens.append(np.array(p))
        ranges = [(len(t) - steps, len(t)) for t in tokens]
        out = [None] * case["batch"]
        for b, logits in forward(cfg, params, padded(tokens), ranges, None):
            out[b] = logits
            want = torch.from_numpy(np.append(tokens[b][len(tokens[b]) - steps + 1:], succ[tokens[b][-1]])).cuda()
            if not torch.equal(logits.argmax(-1), want):
                raise RuntimeError("the model does not follow its successors: these weights cannot be compared")
        logits = torch.stack(out, 1)
        return {"tokens": logits.argmax(-1), "logits": logits}


def padded(tokens):
    """Sequences side by side, filled up behind their ends (nothing looks forward)."""
    out = np.zeros((len(tokens), max(len(t) for t in tokens)), np.int64)
    for row, t in zip(out, tokens):
        row[:len(t)] = t
    return torch.from_numpy(out).cuda()


def linear(x, w):
    """x [..., in] times a bf16 weight [in, out], in 64 bits."""
    return x @ w.double()


def in_rows(f, x, rows=8192):
    flat = x.reshape(-1, x.shape[-1])
    return torch.cat([f(c) for c in flat.split(rows)]).reshape(*x.shape[:-1], -1)


def normed(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double() + b.double()


def rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()


def rotated(x, base, n):
    """The first n of the last axis of x [B, T, H, .] turned pairwise by the position's angles."""
    pos = torch.arange(x.shape[1], device=x.device, dtype=torch.float64)
    freq = float(base) ** (-torch.arange(0, n, 2, device=x.device, dtype=torch.float64) / n)
    ang = (pos[:, None] * freq)[:, None, :]
    u, v = x[..., 0:n:2], x[..., 1:n:2]
    turned = torch.stack([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin()], -1).flatten(-2)
    return torch.cat([turned, x[..., n:]], -1)


def attend(q, k, v, scale, window, limit=None):
    """q [B, T, H, n], k [B, T, G, n], v [B, T, G, m]: softmax over the visible keys, a few heads at a time."""
    B, T, H, _ = q.shape
    group = H // k.shape[2]
    i = torch.arange(T, device=q.device)
    seen = (i[:, None] >= i[None, :]) & (i[:, None] - i[None, :] < window)
    out = torch.empty(B, T, H, v.shape[-1], dtype=torch.float64, device=q.device)
    for b in range(B):
        ok = seen if limit is None else seen & (i[None, :] <= limit[b])
        for h0 in range(0, H, 8):
            hs = list(range(h0, min(H, h0 + 8)))
            kv = [h // group for h in hs]
            s = torch.einsum("thn,jhn->htj", q[b][:, hs], k[b][:, kv]) * scale
            out[b][:, hs] = torch.einsum("htj,jhm->thm", s.masked_fill_(~ok, -torch.inf).softmax(-1), v[b][:, kv])
    return out


def gptj_forward(cfg, params, tokens, ranges, limit):
    """Yields (sequence, logits of its rows in the range)."""
    part = {k.split("/~/", 1)[1]: {n: t[0] for n, t in v.items()} for k, v in params.items()}
    H = cfg["n_heads"]
    x = part["embedding_shard/~/linear"]["w"][tokens].double() + part["embedding_shard/~/linear"]["b"].double()
    B, T, d = x.shape
    for i in range(cfg["layers"]):
        w = {n: part[f"layer_{i}/~/{n}"] for n in ("replicated_layer_norm", "linear", "linear_1", "linear_2", "linear_3", "linear_4", "linear_5")}
        h = normed(x, w["replicated_layer_norm"]["scale"], w["replicated_layer_norm"]["offset"], 1e-5)
        q, v, k = (linear(h, w[n]["w"]).view(B, T, H, d // H) for n in ("linear", "linear_1", "linear_2"))
        R = cfg["pe_rotary_dims"]
        a = attend(rotated(q, 10000, R), rotated(k, 10000, R), v, (d // H) ** -0.5, cfg["seq"] - 1, limit)
        up, down, ub, db = w["linear_4"]["w"].double(), w["linear_5"]["w"].double(), w["linear_4"]["b"].double(), w["linear_5"]["b"].double()
        x = x + linear(a.view(B, T, d), w["linear_3"]["w"])
        x += in_rows(lambda c: torch.nn.functional.gelu(c @ up + ub, approximate="tanh") @ down + db, h)
    p = part["projection_shard/~/linear"]
    ln, head = part["projection_shard/~/replicated_layer_norm"], p["w"].double()
    for b, (lo, hi) in enumerate(ranges):
        yield b, normed(x[b, lo:hi], ln["scale"], ln["offset"], 1e-5) @ head + p["b"].double()


def causal_conv(x, taps, bias):
    K = taps.shape[1]
    xp = torch.nn.functional.pad(x, (0, 0, K - 1, 0))
    return sum(xp[:, j:j + x.shape[1]] * taps[:, j].double() for j in range(K)) + bias


def latent_attention(h, w, m, eps):
    B, T, _ = h.shape
    H, n, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
    q = linear(h, w["q"].T).view(B, T, H, n + r)
    base = m["rot"]["base"]
    q = torch.cat([q[..., :n], rotated(q[..., n:], base, r)], -1)
    down = linear(h, w["dkv"].T)
    c = rms(down[..., :rank], w["dkv.norm"], eps)
    kr = rotated(down[..., None, rank:], base, r)
    k = torch.cat([linear(c, w["uk"].T).view(B, T, H, n), kr.expand(B, T, H, r)], -1)
    v = linear(c, w["uv"].T).view(B, T, H, m["vdim"])
    return linear(attend(q, k, v, m["scale"], m["mask"]["size"]).flatten(2), w["o"].T)


def mamba1(h, w, m):
    n, rank, N = m["inner"], m["dt_rank"], m["state"]
    xz = linear(h, w["in"].T)
    u = torch.nn.functional.silu(causal_conv(xz[..., :n], w["conv"], w["conv.b"].double()))
    p = linear(u, w["x"].T)
    dt = torch.nn.functional.softplus(linear(p[..., :rank], w["dt"].T) + w["dt.b"].double(), threshold=100.0)
    A, D = -w["A_log"].double().exp(), w["D"].double()
    S = torch.zeros(h.shape[0], n, N, dtype=torch.float64, device=h.device)
    y = torch.empty_like(u)
    du = dt * u
    for t in range(h.shape[1]):
        S = torch.exp(dt[:, t, :, None] * A).mul_(S).add_(du[:, t, :, None] * p[:, t, None, rank:rank + N])
        y[:, t] = torch.einsum("bcn,bn->bc", S, p[:, t, rank + N:])
    return linear((y + D * u) * torch.nn.functional.silu(xz[..., n:]), w["o"].T)


def grouped_attention(h, w, m, eps, kv):
    B, T, _ = h.shape
    q = rms(linear(h, w["q"].T), w["q.norm"], eps).view(B, T, m["heads"], m["dim"])
    pos = torch.arange(T, device=h.device, dtype=torch.float64)
    q = q * (1 + m["q_temp"]["coef"] * torch.log(torch.floor((pos + 1) / m["q_temp"]["every"]) + 1))[:, None, None]
    if kv is None:
        kv = (rms(linear(h, w["k"].T), w["k.norm"], eps).view(B, T, m["kv_heads"], m["dim"]),
              linear(h, w["v"].T).view(B, T, m["kv_heads"], m["vdim"]))
    return linear(attend(q, *kv, m["scale"], 1 << 30).flatten(2), w["o"].T), kv


def channel_delta(h, w, m, eps):
    B, T, _ = h.shape
    H, G, n, nv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    conv = lambda name: torch.nn.functional.silu(causal_conv(linear(h, w[name].T), w[name + ".conv"], 0.0))  # noqa: E731
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)                                    # noqa: E731
    q, k = (unit(conv(c).view(B, T, G, n).repeat_interleave(H // G, 2)) for c in ("q", "k"))
    q, v = q * n ** -0.5, conv("v").view(B, T, H, nv)
    beta = torch.sigmoid(linear(h, w["b"].T))
    raw = (linear(linear(h, w["a1"].T), w["a2"].T) + w["dt_bias"].double()).view(B, T, H, n)
    g = torch.exp(-w["A_log"].double().exp()[:, None] * torch.nn.functional.softplus(raw, threshold=100.0))
    S = torch.zeros(B, H, n, nv, dtype=torch.float64, device=h.device)
    o = torch.empty_like(v)
    for t in range(T):
        S = S * g[:, t, :, :, None]
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhnm,bhn->bhm", S, k[:, t]))
        S += k[:, t, :, :, None] * u[:, :, None, :]
        o[:, t] = torch.einsum("bhnm,bhn->bhm", S, q[:, t])
    gate = torch.sigmoid(linear(linear(h, w["g1"].T), w["g2"].T)).view(B, T, H, nv)
    return linear((rms(o, w["norm"], eps) * gate).flatten(2), w["o"].T)


def mamba2(h, w, m, eps):
    B, T, _ = h.shape
    H, nv, N, G = m["heads"], m["vdim"], m["state"], m["groups"]
    inner = H * nv
    p = linear(h, w["in"].T)
    z, u, dt = p[..., :inner], p[..., inner:2 * inner + 2 * G * N], p[..., 2 * inner + 2 * G * N:]
    u = torch.nn.functional.silu(causal_conv(u, w["conv"], w["conv.b"].double()))
    x = u[..., :inner].view(B, T, H, nv)
    b, c = (u[..., inner + i * G * N:inner + (i + 1) * G * N].view(B, T, G, N).repeat_interleave(H // G, 2) for i in (0, 1))
    dt = torch.nn.functional.softplus(dt + w["dt_bias"].double(), threshold=100.0)
    g = torch.exp(-w["A_log"].double().exp() * dt)
    S = torch.zeros(B, H, N, nv, dtype=torch.float64, device=h.device)
    y = torch.empty_like(x)
    for t in range(T):
        S = S * g[:, t, :, None, None] + (dt[:, t, :, None] * b[:, t])[..., None] * x[:, t, :, None, :]
        y[:, t] = torch.einsum("bhnm,bhn->bhm", S, c[:, t])
    y = (y + w["D"].double()[:, None] * x).flatten(2) * torch.nn.functional.silu(z)
    y = y.view(B, T, m["norm_groups"], -1)
    y = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + eps)).flatten(2) * w["norm"].double()
    return linear(y, w["o"].T)


def stack_forward(cfg, params, tokens, ranges, limit):
    """Yields (sequence, logits of its rows in the range).  Layer stacks do not read ``limit``."""
    W = {k: t[0] for k, t in next(iter(params.values())).items()}
    eps = cfg["norm"]["eps"]
    post = cfg["architecture"] == "Bavutar"
    x = W["embed"][tokens].double() * (cfg["embedding"]["scale"] if post else 1.0)
    x0, kept = x, {}
    silu = torch.nn.functional.silu
    for i, first in layer_runs(cfg):
        if first:
            x = linear(torch.cat([x, x0], -1), W["loop.in"].T)
        layer, p = cfg["layers"][i], f"l{i}."
        w = {k[len(p) + 4:]: t for k, t in W.items() if k.startswith(p + "mix.")}
        m, kind = layer["mixer"], layer["type"]
        h = x if post else rms(x, W[p + "norm1"], eps)
        if kind == "attention":
            y, kept[i] = grouped_attention(h, w, m, eps, kept.get(m.get("kv_from")))
        else:
            y = {"latent_attention": lambda: latent_attention(h, w, m, eps), "mamba1": lambda: mamba1(h, w, m),
                 "mamba2": lambda: mamba2(h, w, m, eps), "channel_delta": lambda: channel_delta(h, w, m, eps)}[kind]()
        if post:
            x = normed(cfg["postln_alpha"] * x + y, W[p + "norm1"], W[p + "norm1.b"], eps)
            up, down = W[p + "mlp.up"].T.double(), W[p + "mlp.down"].T.double()
            y = in_rows(lambda c: (c @ up).clamp_min(0).square() @ down, x)
            x = normed(cfg["postln_alpha"] * x + y, W[p + "norm2"], W[p + "norm2.b"], eps)
            continue
        x = x + cfg["residual_mult"] * rms(y, W[p + "norm1b"], eps)
        if layer["mlp"] is not None:
            gate, up, down = (W[p + n].T.double() for n in ("mlp.gate", "mlp.up", "mlp.down"))
            y = in_rows(lambda c: (silu(c @ gate) * (c @ up)) @ down, rms(x, W[p + "norm2"], eps))
            x = x + cfg["residual_mult"] * rms(y, W[p + "norm2b"], eps)
    head = W["head"].T.double()
    for b, (lo, hi) in enumerate(ranges):
        rows = x[b, lo:hi]
        if not post:
            yield b, rms(rows, W["final.norm"], eps) @ head
            continue
        cap = cfg["logit_softcap"]
        yield b, cap * torch.tanh(normed(rows, W["final.norm"], W["final.norm.b"], eps) @ head / cap)
