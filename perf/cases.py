"""The work that programs have this framework do, as cases to time.

Every case runs through the public entry points: a model made from a configuration and tensors, ``Inference`` with its cache, and
``Engine.step`` (whole prompts, logits of every token, as scoring and trace replay ask for them) or ``Engine.decode_step`` (one token
for every sequence, from a CUDA graph, as the generation loop runs); a mixture of experts is called as the part it is.  Sizes are
those of the framework's own benchmark (the Llama shapes, and the layers of the other designs at the same widths).  Most cases
are one layer, or one of each kind of a design, between an embedding table and a small vocabulary; one is the whole 1B-shaped
Llama decoder with its real vocabulary.
"""
import math

import torch

from kuiperllama_b200 import Inference, SequenceInput
from kuiperllama_b200.config import PartSpec, config_from_dict
from kuiperllama_b200.engine import DecoderModel, parse_dtype
from kuiperllama_b200.parts import MoEFeedForward, Runtime, StepContext

DEV = "cuda:0"
F64 = torch.float64
WIDTHS = (1024, 2048, 4096)
INTER = {1024: 4096, 2048: 8192, 4096: 14336}          # the feed-forward's size beside each width
EXPERTS, TOP = 16, 4
LIMIT, ALPHA, SHIFT = 7.0, 1.702, 1.0
WINDOW, KEEP = 1024, 64


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # One sequence at a time in true 32-bit arithmetic, as a replay that is compared number by number runs: the smallest call.
        dict(name="f32_token", layer="llama", dtype="float32", width=2048, layers=2, vocab=2048, step="token", seqs=1, tokens=300),
        # The same model reading a prompt.
        dict(name="f32_prompt", layer="llama", dtype="float32", width=2048, layers=2, vocab=2048, step="prompt", seqs=1, tokens=777),
        # The whole 1B-shaped decoder serving 64 conversations: the logits of the next token of each.
        dict(name="llama_1b_token_64", layer="llama", dtype="bfloat16", width=2048, layers=16, vocab=128256, step="token", seqs=64, tokens=700),
        # Layers of the 8B shape decoding a small batch: the benchmark's headline, bound by the weights' bytes.
        dict(name="llama_8b_token_8", layer="llama", dtype="bfloat16", width=4096, layers=2, vocab=4096, step="token", seqs=8, tokens=520),
        # A layer of the 8B shape reading a long prompt: bound by the products.
        dict(name="llama_8b_prompt", layer="llama", dtype="bfloat16", width=4096, layers=1, vocab=512, step="prompt", seqs=1, tokens=2048),
        # Terolix: the gated delta rule over one prompt.
        dict(name="delta_prompt", layer="delta", dtype="bfloat16", width=2048, layers=1, vocab=512, step="prompt", seqs=1, tokens=2048),
        # Bededra: the state-space layer over three prompts of uneven lengths.
        dict(name="ssm_prompts", layer="ssm", dtype="bfloat16", width=2048, layers=1, vocab=512, step="prompt", seqs=3, tokens=4001),
        # Bededra: attention with mixed heads beside gated linear attention over one prompt, the largest case of a layer.
        dict(name="parallel_prompt", layer="parallel", dtype="bfloat16", width=2048, layers=1, vocab=512, step="prompt", seqs=1, tokens=2048),
        # Bededra: both kinds of layer decoding 64 sequences; every sequence's states are read and written.
        dict(name="hybrid_token_64", layer="hybrid", dtype="bfloat16", width=2048, layers=2, vocab=512, step="token", seqs=64, tokens=200),
        # Munadra: attention over the shared latent, a long prompt.
        dict(name="latent_prompt", layer="latent", dtype="bfloat16", width=2048, layers=1, vocab=512, step="prompt", seqs=1, tokens=2048),
        # Dofevik: attention over a window with a sink, several prompts in one step.
        dict(name="window_prompts", layer="window", dtype="bfloat16", width=2048, layers=1, vocab=512, step="prompt", seqs=4, tokens=6000),
        # Munadra: the experts of a layer for the tokens of a prompt.
        dict(name="experts_prompt", layer="experts", dtype="bfloat16", width=2048, layers=1, vocab=0, step="prompt", seqs=1, tokens=2048),
    ]


def draw(rng):
    """Another case of the same ranges: any layer, width and number of sequences that the listed cases' kinds have in use, prompts of
    17 to a few thousand tokens, contexts of 20 to 1,000, batches of 1 to 64."""
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    layer = rng.choice(["llama", "llama", "llama", "f32", "delta", "ssm", "parallel", "hybrid", "latent", "window", "experts"])
    if layer == "f32":
        step = rng.choice(["token", "prompt"])
        return dict(layer="llama", dtype="float32", width=rng.choice((1024, 2048)), layers=2, vocab=2048, step=step,
                    seqs=spread(1, 8) if step == "token" else 1, tokens=spread(20, 700))
    width = rng.choice(WIDTHS if layer in ("llama", "latent", "window", "experts") else WIDTHS[:2])
    step = rng.choice(["token", "prompt"]) if layer == "llama" else "token" if layer == "hybrid" else "prompt"
    if step == "token":
        return dict(layer=layer, dtype="bfloat16", width=width, layers=2, vocab=rng.choice((512, 2048, 4096)), step=step,
                    seqs=spread(1, 64), tokens=spread(20, 1000) if layer == "llama" else spread(20, 200))
    most = {"parallel": 2048, "delta": 3000, "experts": 3000, "latent": 2500}.get(layer, 4500 if width < 4096 else 2500)
    tokens = spread(1 if layer == "experts" else 17, most)
    return dict(layer=layer, dtype="bfloat16", width=width, layers=1, vocab=0 if layer == "experts" else rng.choice((512, 1000)), step=step,
                seqs=1 if layer == "experts" else min(spread(1, 8), tokens), tokens=tokens)


def lengths(case):
    """Tokens of every sequence: for a prompt step they add up to ``tokens``, for a token step the longest has ``tokens``."""
    n, total = case["seqs"], case["tokens"]
    if case["step"] == "token":
        return [max(1, total - (i * 37) % (total // 2 + 1)) for i in range(n)]
    share = [1 + (i * 7) % 5 for i in range(n)]
    out = [max(1, total * s // sum(share)) for s in share]
    out[0] += total - sum(out)
    return out


# ------------------------------------------------------------------------------------------------ configurations

def heads_of(width):
    """(heads, key/value heads, head size) of the Llama shape of that width."""
    return {1024: (16, 4, 64), 2048: (32, 8, 64), 4096: (32, 8, 128)}[width]


def mixer(kind, width):
    H, G, d = heads_of(width)
    if kind == "delta":
        return {"heads": width // 128, "kv_heads": max(1, width // 512), "dim": 128, "vdim": 128, "conv": 4}
    if kind == "ssm":
        return {"heads": 2 * width // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
    if kind == "parallel":
        return {"left": {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "softcap": 50.0, "mask": {"size": WINDOW, "keep_first": KEEP}},
                "right": {"heads": width // 128, "dim": 64, "vdim": 128, "tau": 16.0, "rank": 16}, "left_scale": 1.0, "right_scale": 1.0}
    if kind == "latent":
        return {"heads": H, "dim": d, "rot_dim": d // 2, "vdim": d, "kv_rank": 256, "scale": (1.5 * d) ** -0.5,
                "rot": {"base": 500000.0, "dims": d // 2, "scaling": {"factor": 8.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}
    return {"heads": H, "kv_heads": G, "dim": d, "vdim": d, "scale": d ** -0.5, "mask": {"size": WINDOW},
            "rot": {"base": 500000.0, "dims": d // 2, "scaling": {"factor": 8.0}}}


def kinds(case):
    return ["ssm", "parallel"] if case["layer"] == "hybrid" else [case["layer"]] * case["layers"]


def config(case):
    W, vocab = case["width"], case["vocab"]
    if case["layer"] == "llama":
        H, G, d = heads_of(W)
        return {"architectures": ["LlamaForCausalLM"], "hidden_size": W, "intermediate_size": INTER[W], "num_hidden_layers": case["layers"],
                "num_attention_heads": H, "num_key_value_heads": G, "head_dim": d, "vocab_size": vocab, "max_position_embeddings": 8192,
                "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "rope_scaling": None, "tie_word_embeddings": True, "hidden_act": "silu"}
    names = {"delta": "delta", "ssm": "mamba2", "parallel": "parallel", "latent": "latent_attention", "window": "attention"}
    layers = [{"type": names[k], "mixer": mixer(k, W), "mlp": None} for k in kinds(case)]
    common = {"vocab": vocab, "width": W, "norm": {"eps": 1e-5}, "max_positions": 8192, "layers": layers}
    if case["layer"] == "delta":
        return {"architecture": "Terolix", **common}
    if case["layer"] == "latent":
        return {"architecture": "Munadra", "embedding": {"scale": 45.0}, "logit_scale": 1.0, **common}
    if case["layer"] == "window":
        return {"architecture": "Dofevik", **common}
    return {"architecture": "Bededra", "canon": {"taps": 4}, **common}


# ------------------------------------------------------------------------------------------------ weights

def weights(case, seed):
    """Tensor name -> bfloat16 values on the device, as a checkpoint holds them: matrices N(0, 1 / inputs), norm weights near 1, decays
    and step sizes in the ranges such layers are initialised with."""
    W, g = case["width"], torch.Generator(device=DEV).manual_seed(seed)
    t = {}

    def normal(name, *shape, std=None, mean=0.0):
        x = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(0.0, shape[-1] ** -0.5 if std is None else std, generator=g)
        t[name] = (x + mean if mean else x).bfloat16()

    def uniform(name, n, lo, hi, f):
        t[name] = f(lo + (hi - lo) * torch.rand(n, device=DEV, generator=g)).bfloat16()

    def rate(p, n):          # exp(A_log) in [1, 16], softplus(dt_bias) in [0.001, 0.1]
        uniform(p + "A_log", n, 1.0, 16.0, torch.log)
        uniform(p + "dt_bias", n, math.log(0.001), math.log(0.1), lambda u: torch.log(torch.expm1(torch.exp(u))))

    if case["layer"] == "experts":
        ff = INTER[W] // 4
        normal("router", EXPERTS, W)
        for e in range(EXPERTS):
            normal(f"e{e}.gate", ff, W)
            normal(f"e{e}.up", ff, W)
            normal(f"e{e}.down", W, ff)
        return t
    if case["layer"] == "llama":
        H, G, d = heads_of(W)
        normal("model.embed_tokens.weight", case["vocab"], W, std=0.02)
        normal("model.norm.weight", W, std=0.1, mean=1.0)
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            normal(p + "input_layernorm.weight", W, std=0.1, mean=1.0)
            normal(p + "post_attention_layernorm.weight", W, std=0.1, mean=1.0)
            normal(p + "self_attn.q_proj.weight", H * d, W)
            normal(p + "self_attn.k_proj.weight", G * d, W)
            normal(p + "self_attn.v_proj.weight", G * d, W)
            normal(p + "self_attn.o_proj.weight", W, H * d)
            normal(p + "mlp.gate_proj.weight", INTER[W], W)
            normal(p + "mlp.up_proj.weight", INTER[W], W)
            normal(p + "mlp.down_proj.weight", W, INTER[W])
        return t
    normal("embed", case["vocab"], W, std=0.02)
    for i, kind in enumerate(kinds(case)):
        p, m = f"l{i}.mix.", mixer(kind, W)
        if kind == "delta":
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for name in ("norm1", "norm1b"):
                normal(f"l{i}.{name}", W, std=0.1, mean=1.0)
                normal(f"l{i}.{name}.b", W, std=0.02)
            normal(f"l{i}.rg1", W, W)
            normal(f"l{i}.rg1.b", W, std=0.1)
            for name, n in (("q", G * d), ("k", G * d), ("v", H * dv), ("g", H * dv), ("b", H)):
                normal(p + name, n, W)
            normal(p + "a", H, W, std=0.2 * W ** -0.5)
            for name, n in (("q", G * d), ("k", G * d), ("v", H * dv)):
                normal(p + name + ".conv", n, m["conv"])
            rate(p, H)
            normal(p + "norm", dv, std=0.1, mean=1.0)
            normal(p + "o", W, H * dv)
        elif kind == "latent":
            H, d, rd, dv, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            normal(f"l{i}.norm1", W, std=0.1)
            normal(p + "q", H * (d + rd), W)
            normal(p + "dkv", r + rd, W)
            normal(p + "dkv.norm", r, std=0.1, mean=1.0)
            normal(p + "uk", H * d, r)
            normal(p + "uv", H * dv, r)
            normal(p + "sink", H, std=1.0)
            normal(p + "g", H, W)
            normal(p + "o", W, H * dv)
        elif kind == "window":
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            normal(f"l{i}.norm1", 1, std=0.1, mean=1.0)
            for name, n in (("q", H * d), ("k", G * d), ("v", G * d)):
                normal(p + name, n, W)
                normal(p + name + ".b", n, std=0.1)
            normal(p + "sink", H, std=1.0)
            normal(p + "o", W, H * d)
        else:
            normal(f"l{i}.norm1", W, std=0.1, mean=1.0)
            normal(f"l{i}.canon1", W, 4, std=0.2)
            if kind == "ssm":
                H, P, N = m["heads"], m["vdim"], m["state"]
                inner, C = H * P, H * P + 2 * N
                normal(p + "in", inner + C + H, W)
                t[p + "in"][inner + C:] *= 0.2
                normal(p + "conv", C, 4)
                normal(p + "conv.b", C, std=0.1)
                rate(p, H)
                normal(p + "D", H, std=0.1, mean=1.0)
                normal(p + "norm", inner, std=0.1, mean=1.0)
                normal(p + "o", W, inner)
            else:
                q, (H, G, d, dv) = p + "left.", (m["left"][k] for k in ("heads", "kv_heads", "dim", "vdim"))
                for name, n in (("q", H * d), ("k", G * d), ("v", G * dv), ("g", H)):
                    normal(q + name, n, W)
                normal(q + "r1", H, std=0.1, mean=0.5)
                normal(q + "r2", H, std=0.01, mean=0.1)
                normal(q + "talk", H, H, std=0.1)
                t[q + "talk"] += torch.eye(H, device=DEV, dtype=torch.bfloat16)
                normal(q + "o", W, H * dv)
                q, (H, d, dv, rank) = p + "right.", (m["right"][k] for k in ("heads", "dim", "vdim", "rank"))
                for name, n in (("q", H * d), ("k", H * d), ("v", H * dv), ("g", H * dv), ("a1", rank)):
                    normal(q + name, n, W)
                normal(q + "a2", H * d, rank)
                normal(q + "a2.b", H * d, std=1.0)
                normal(q + "norm", dv, std=0.1, mean=1.0)
                normal(q + "o", W, H * dv)
    normal("final.norm", 1 if case["layer"] == "window" else W, std=0.1, mean=0.0 if case["layer"] == "latent" else 1.0)
    if case["layer"] == "delta":
        normal("final.norm.b", W, std=0.02)
    elif case["layer"] != "latent":
        normal("head", case["vocab"], W)
    return t


def token_ids(case, seed):
    """The sequences' tokens; a token step's sequences end with one token that ``prepare`` decodes and one that ``run`` decodes."""
    g = torch.Generator().manual_seed(seed + 1)
    more = 2 if case["step"] == "token" else 0
    return [torch.randint(0, case["vocab"], (n + more,), generator=g).tolist() for n in lengths(case)]


def expert_rows(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    return torch.empty((case["tokens"], case["width"]), dtype=torch.float32, device=DEV).normal_(0.0, 1.0, generator=g).bfloat16()


# ------------------------------------------------------------------------------------------------ what a program does

def prepare(case, seed):
    if case["layer"] == "experts":
        W, n = case["width"], case["tokens"]
        spec = PartSpec("moe", {"hidden_size": W, "experts": EXPERTS, "top": TOP, "expert_size": INTER[W] // 4, "limit": LIMIT, "alpha": ALPHA,
                                "shift": SHIFT, "renormalise": False,
                                "names": {"router": "router", "gate": "e{e}.gate", "up": "e{e}.up", "down": "e{e}.down"}})
        part = MoEFeedForward(spec, "", weights(case, seed), Runtime(device=torch.device(DEV), dtype=torch.bfloat16))
        ids = torch.arange(n, dtype=torch.int32, device=DEV)
        one = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
        step = StepContext(n_tokens=n, n_seqs=1, token_ids=ids, positions=ids, token_slot=torch.zeros_like(ids), seq_slots=one([0]), seq_starts=one([0]),
                           seq_new=one([n]), cu_tokens=one([0, n]), is_decode=n == 1, max_new=n, max_context=n, host_slots=[0], host_starts=[0], host_new=[n])
        return {"part": part, "step": step, "rows": expert_rows(case, seed)}
    spec = config_from_dict(config(case)).to_model_spec()
    model = DecoderModel(spec, weights(case, seed), Runtime(device=torch.device(DEV), dtype=parse_dtype(case["dtype"])))
    ids = token_ids(case, seed)
    held = sum(-(-(len(t) + 1) // 64) * 64 for t in ids)
    infer = Inference(model, max_tokens=held, max_batch=len(ids), max_seq_len=max(len(t) for t in ids) + 1)
    state = {"infer": infer, "ids": ids}
    with torch.inference_mode():
        if case["step"] == "token":
            eng = infer.engine
            slots = [eng.alloc_slot() for _ in ids]
            eng.step([SequenceInput(s, t[:-2], []) for s, t in zip(slots, ids)])
            eng.decode_step(slots, [t[-2] for t in ids])            # the step whose launches are captured for the ones that follow
            state.update(slots=slots, last=[t[-1] for t in ids], held=[len(t) - 1 for t in ids])
        elif sum(len(t) for t in ids) <= infer.engine.SMALL_STEP_TOKENS:
            run(state)                                              # a small step is captured likewise
    return state


@torch.inference_mode()
def run(state):
    if "part" in state:
        out = state["part"].forward(state["rows"], state["step"])
        return out.sum(dim=0) if out.dim() == 3 else out            # pieces whose sum is the result
    eng = state["infer"].engine
    if "slots" in state:
        for s, n in zip(state["slots"], state["held"]):
            eng.cache.lengths[s] = n                                # the same place of every sequence again
        return eng.decode_step(state["slots"], state["last"])
    slots = [eng.alloc_slot() for _ in state["ids"]]
    logits = eng.step([SequenceInput(s, t, range(len(t))) for s, t in zip(slots, state["ids"])])
    for s in slots:
        eng.free_slot(s)
    return logits


# ------------------------------------------------------------------------------------------------ bytes and operations

def pairs(lens, window=None, keep=0):
    """Visible (query, key) pairs of prompts."""
    n = 0
    for t in lens:
        if window is None or t <= window:
            n += t * (t + 1) // 2
        else:
            n += window * (window + 1) // 2 + (t - window) * window
            n += sum(min(keep, i - window + 1) for i in range(window, t))
    return n


def work(case):
    W, lens = case["width"], lengths(case)
    rows = sum(lens) if case["step"] == "prompt" else len(lens)
    size = 4 if case["dtype"] == "float32" else 2
    if case["layer"] == "experts":
        ff = INTER[W] // 4
        used = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** rows)      # experts that some row chooses
        return {"bytes": used * 3 * W * ff * 2 + EXPERTS * W * 2 + rows * W * 6, "flops": 2 * rows * (TOP * 3 * W * ff + EXPERTS * W)}
    matrix = cache = state = 0          # elements of matrices, elements of keys and values, bytes of states
    flops = 0
    ctx = [t + 2 for t in lens] if case["step"] == "token" else lens
    for kind in kinds(case):
        m = mixer(kind, W)
        seen = pairs(lens, *((WINDOW, KEEP) if kind == "parallel" else (WINDOW,) if kind == "window" else ())) if case["step"] == "prompt" else sum(ctx)
        if kind == "llama":
            H, G, d = heads_of(W)
            matrix += 2 * (H + G) * d * W + 3 * W * INTER[W]
            cache += sum(ctx) * 2 * G * d
            flops += 4 * H * d * seen
        elif kind == "delta":
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            matrix += W * (2 * G * d + 3 * H * dv + 2 * H) + W * W
            state += 2 * len(lens) * H * d * dv * 4
            flops += 6 * H * d * dv * rows
        elif kind == "latent":
            H, d, rd, dv, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            matrix += W * (H * (d + rd) + r + rd + H + H * dv) + r * H * (d + dv)
            cache += sum(ctx) * (r + rd)
            flops += 2 * H * (d + rd + dv) * seen
        elif kind == "window":
            H, G, d = m["heads"], m["kv_heads"], m["dim"]
            matrix += 2 * (H + G) * d * W
            cache += sum(ctx) * 2 * G * d
            flops += 4 * H * d * seen
        elif kind == "ssm":
            H, P, N = m["heads"], m["vdim"], m["state"]
            matrix += W * (3 * H * P + 2 * N + H)
            state += 2 * len(lens) * H * P * N * 4
            flops += 4 * H * P * N * rows
        else:
            H, G, d, dv = (m["left"][k] for k in ("heads", "kv_heads", "dim", "vdim"))
            matrix += W * (H * d + G * (d + dv) + H + H * dv)
            cache += sum(ctx) * G * (d + dv)
            flops += (2 * H * (d + dv) + 2 * H * H) * seen
            H, d, dv, rank = (m["right"][k] for k in ("heads", "dim", "vdim", "rank"))
            matrix += W * (2 * H * d + 3 * H * dv + rank)
            state += 2 * len(lens) * H * d * dv * 4
            flops += 4 * H * d * dv * rows
    matrix += case["vocab"] * W
    return {"bytes": matrix * size + cache * size + state + rows * (case["vocab"] * 4 + W * size), "flops": flops + 2 * rows * matrix}


def tolerance(case):
    """About four times the distance from the 64-bit results (float32: 5e-6; one bfloat16 layer: 2e-3 to 6.5e-3; 16 Llama layers: 1e-2,
    where the largest value that is taken at all is stated)."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": {"llama": 0.03, "latent": 0.01, "experts": 0.01}.get(case["layer"], 0.02)}


# ------------------------------------------------------------------------------------------------ the same in 64 bits

def rms(x, w, eps=1e-5):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def silu(x):
    return x * torch.sigmoid(x)


def softplus(x):
    return torch.nn.functional.softplus(x, threshold=40.0)


def conv(x, w):
    """Causal, per channel: x [T, C], w [C, taps], the last tap is the current token's."""
    T, taps = x.shape[0], w.shape[1]
    pad = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    return sum(pad[j:j + T] * w[:, j] for j in range(taps))


def turned(x, freqs, factor=1.0, interleaved=False):
    """x [T, heads, d]: its first 2 * len(freqs) elements turn by position times frequency."""
    a = torch.arange(x.shape[0], dtype=F64, device=x.device)[:, None] * torch.tensor(freqs, dtype=F64, device=x.device)
    c, s, n = (torch.cos(a) * factor)[:, None], (torch.sin(a) * factor)[:, None], 2 * len(freqs)
    y = x.clone()
    i, j = (slice(0, n, 2), slice(1, n, 2)) if interleaved else (slice(0, n // 2), slice(n // 2, n))
    y[..., i], y[..., j] = x[..., i] * c - x[..., j] * s, x[..., j] * c + x[..., i] * s
    return y


def attend(q, k, v, scale, window=None, sink=None, score=None, mix=None, keep=0):
    """q [T, H, d], k [T, G, d], v [T, G, dv] -> [T, H, dv], some queries at a time."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    out, j = [], torch.arange(T, device=q.device)
    k, v = (x.permute(1, 0, 2).repeat_interleave(H // G, 0) for x in (k, v))
    for i0 in range(0, T, 256):
        i = torch.arange(i0, min(T, i0 + 256), device=q.device)
        s = torch.matmul(q[i].permute(1, 0, 2), k.transpose(1, 2)) * scale
        dist = i[:, None] - j[None, :]
        if score is not None:
            s = score(s, dist.clamp(min=0))
        hidden = dist < 0
        if window is not None:
            hidden = hidden | ((dist >= window) & (j[None, :] >= keep))
        s = s.masked_fill(hidden, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink[:, None, None])
        e = torch.exp(s - top)
        den = e.sum(-1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[:, None, None] - top))
        e = e / den
        if mix is not None:
            e = torch.matmul(mix, e.reshape(H, -1)).reshape(e.shape)
        out.append(torch.matmul(e, v).permute(1, 0, 2))
    return torch.cat(out)


def plain_frequencies(dims, base, factor=1.0):
    return [base ** (-2.0 * i / dims) / factor for i in range(dims // 2)]


def yarn_frequencies(dims, base, factor, original, fast, slow):
    at = lambda turns: dims * math.log(original / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(at(fast)), 0), min(math.ceil(at(slow)), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [f / factor * r + f * (1.0 - r) for f, r in zip(plain_frequencies(dims, base), ramp)], 0.1 * math.log(factor) + 1.0


def exact_mixer(kind, h, w, m):
    T = h.shape[0]
    if kind == "delta":
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k, v = (silu(conv(h @ w[n].T, w[n + ".conv"])).view(T, -1, 128) for n in "qkv")
        q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        q, k = (q * d ** -0.5).repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
        beta = torch.sigmoid(h @ w["b"].T)
        a = torch.exp(-torch.exp(w["A_log"]) * softplus(h @ w["a"].T + w["dt_bias"]))
        S, o = h.new_zeros(H, d, dv), h.new_empty(T, H, dv)
        for t in range(T):
            S = S * a[t, :, None, None]
            u = beta[t, :, None] * (v[t] - torch.matmul(k[t, :, None], S)[:, 0])
            S = torch.baddbmm(S, k[t, :, :, None], u[:, None])
            o[t] = torch.matmul(q[t, :, None], S)[:, 0]
        return (rms(o, w["norm"]).reshape(T, H * dv) * silu(h @ w["g"].T)) @ w["o"].T
    if kind == "ssm":
        H, P, N = m["heads"], m["vdim"], m["state"]
        inner = H * P
        z, xBC, dt = (h @ w["in"].T).split([inner, inner + 2 * N, H], dim=1)
        xBC = silu(conv(xBC, w["conv"]) + w["conv.b"])
        x, B, C = xBC[:, :inner].reshape(T, H, P), xBC[:, inner:inner + N], xBC[:, inner + N:]
        dt = softplus(dt + w["dt_bias"])
        a, xd = torch.exp(-torch.exp(w["A_log"]) * dt), x * dt[..., None]
        S, y = h.new_zeros(H, N, P), h.new_empty(T, H, P)
        for t in range(T):
            S = S * a[t, :, None, None] + B[t, None, :, None] * xd[t, :, None]
            y[t] = torch.matmul(C[t], S)
        y = (y + w["D"][:, None] * x).reshape(T, inner) * silu(z)
        return rms(y, w["norm"]) @ w["o"].T
    if kind == "parallel":
        l, lw = m["left"], {k[5:]: v for k, v in w.items() if k.startswith("left.")}
        H, G, d, dv = l["heads"], l["kv_heads"], l["dim"], l["vdim"]
        cap, r1, r2 = l["softcap"], lw["r1"][:, None, None], lw["r2"][:, None, None]
        o = attend((h @ lw["q"].T).view(T, H, d), (h @ lw["k"].T).view(T, G, d), (h @ lw["v"].T).view(T, G, dv), l["scale"], WINDOW,
                   score=lambda s, dist: cap * torch.tanh(s / cap) - r1 * torch.log1p(r2 * dist), mix=lw["talk"], keep=KEEP)
        left = (o * torch.sigmoid(h @ lw["g"].T)[..., None]).reshape(T, H * dv) @ lw["o"].T
        r, rw = m["right"], {k[6:]: v for k, v in w.items() if k.startswith("right.")}
        H, d, dv = r["heads"], r["dim"], r["vdim"]
        q, k, v = (h @ rw["q"].T).view(T, H, d) * d ** -0.5, (h @ rw["k"].T).view(T, H, d), (h @ rw["v"].T).view(T, H, dv)
        a = torch.sigmoid((h @ rw["a1"].T) @ rw["a2"].T + rw["a2.b"]).pow(1.0 / r["tau"]).view(T, H, d)
        S, o = h.new_zeros(H, d, dv), h.new_empty(T, H, dv)
        for t in range(T):
            S = S * a[t, :, :, None] + k[t, :, :, None] * v[t, :, None]
            o[t] = torch.matmul(q[t, :, None], S)[:, 0]
        return left + (rms(o, rw["norm"]).reshape(T, H * dv) * silu(h @ rw["g"].T)) @ rw["o"].T
    H, d = m["heads"], m["dim"]
    if kind == "latent":
        rd, dv, r, rot = m["rot_dim"], m["vdim"], m["kv_rank"], m["rot"]
        f, factor = yarn_frequencies(rot["dims"], rot["base"], **rot["scaling"])
        c, kr = (h @ w["dkv"].T).split([r, rd], dim=1)
        c, kr = rms(c, w["dkv.norm"]), turned(kr[:, None], f, factor, True)
        qn, qr = (h @ w["q"].T).view(T, H, d + rd).split([d, rd], dim=2)
        k = torch.cat([(c @ w["uk"].T).view(T, H, d), kr.expand(T, H, rd)], dim=2)
        o = attend(torch.cat([qn, turned(qr, f, factor, True)], dim=2), k, (c @ w["uv"].T).view(T, H, dv), m["scale"], sink=w["sink"])
        return (o * torch.sigmoid(h @ w["g"].T)[..., None]).reshape(T, H * dv) @ w["o"].T
    G, f = m["kv_heads"], plain_frequencies(m["rot"]["dims"], m["rot"]["base"], m["rot"]["scaling"]["factor"])
    q, k = (rms(turned((h @ w[n].T + w[n + ".b"]).view(T, -1, d), f, interleaved=True), None) for n in "qk")
    return attend(q, k, (h @ w["v"].T + w["v.b"]).view(T, G, d), m["scale"], WINDOW, w["sink"]).reshape(T, H * d) @ w["o"].T


def exact_llama(x, w, case):
    H, G, d = heads_of(case["width"])
    T, f = x.shape[0], plain_frequencies(d, 500000.0)
    for i in range(case["layers"]):
        g = lambda name: w[f"model.layers.{i}.{name}.weight"].to(F64)
        h = rms(x, g("input_layernorm"))
        q, k, v = ((h @ g(f"self_attn.{n}_proj").T).view(T, -1, d) for n in "qkv")
        x = x + attend(turned(q, f), turned(k, f), v, d ** -0.5).reshape(T, H * d) @ g("self_attn.o_proj").T
        h = rms(x, g("post_attention_layernorm"))
        x = x + (silu(h @ g("mlp.gate_proj").T) * (h @ g("mlp.up_proj").T)) @ g("mlp.down_proj").T
    return x


def exact(case, seed):
    w = weights(case, seed)
    if case["layer"] == "experts":
        h = expert_rows(case, seed).to(F64)
        s, idx = torch.softmax(h @ w["router"].to(F64).T, dim=-1).topk(TOP, dim=-1)
        out = torch.zeros_like(h)
        for e in range(EXPERTS):
            rows, place = (idx == e).nonzero(as_tuple=True)
            gate, up, down = (w[f"e{e}.{n}"].to(F64) for n in ("gate", "up", "down"))
            g, u = (h[rows] @ gate.T).clamp(max=LIMIT), (h[rows] @ up.T).clamp(-LIMIT, LIMIT)
            out.index_add_(0, rows, s[rows, place][:, None] * ((g * torch.sigmoid(ALPHA * g) * (u + SHIFT)) @ down.T))
        return out
    out = []
    last = case["step"] == "token"
    if case["layer"] == "llama" and case["layers"] * sum(lengths(case)) > 1 << 20:
        return None
    for ids in token_ids(case, seed):
        i = torch.tensor(ids, device=DEV)
        if case["layer"] == "llama":
            x = exact_llama(w["model.embed_tokens.weight"][i].to(F64), w, case)
            x = rms(x[-1:] if last else x, w["model.norm.weight"].to(F64))
            out.append(x @ w["model.embed_tokens.weight"].to(F64).T)
            continue
        W64 = {n: t.to(F64) for n, t in w.items()}
        x = W64["embed"][i]
        if case["layer"] == "latent":
            x = x * 45.0
        for n, kind in enumerate(kinds(case)):
            p = f"l{n}."
            mine = {k[len(p) + 4:]: t for k, t in W64.items() if k.startswith(p + "mix.")}
            norm = W64[p + "norm1"]
            if kind == "delta":
                h = torch.nn.functional.layer_norm(x, (case["width"],), norm, W64[p + "norm1.b"], 1e-5)
                y = exact_mixer(kind, h, mine, mixer(kind, case["width"])) * torch.sigmoid(h @ W64[p + "rg1"].T + W64[p + "rg1.b"])
                x = x + torch.nn.functional.layer_norm(y, (case["width"],), W64[p + "norm1b"], W64[p + "norm1b.b"], 1e-5)
            elif kind == "latent":
                x = x + rms(exact_mixer(kind, x, mine, mixer(kind, case["width"])), 1.0 + norm)
            else:
                h = rms(x, norm)
                if kind != "window":
                    h = h + conv(h, W64[p + "canon1"])
                x = x + exact_mixer(kind, h, mine, mixer(kind, case["width"]))
        x = x[-1:] if last else x
        if case["layer"] == "delta":
            x = torch.nn.functional.layer_norm(x, (case["width"],), W64["final.norm"], W64["final.norm.b"], 1e-5)
        else:
            x = rms(x, W64["final.norm"] + (1.0 if case["layer"] == "latent" else 0.0))
        out.append(x @ (W64["head"] if "head" in W64 else W64["embed"]).T)
    return torch.cat(out)
